// fft64_any1.cu -- the any-length FP64 transforms, one signal to a block.
#include "fft64_any.cuh"

namespace nadia {
namespace plain {

void rows_any1(RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    rows_any_modes<1>(mode, fwd, A, p, threads, smem, st);
}

void cols_any1(ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    cols_any_modes<1>(mode, fwd, A, p, threads, smem, st);
}

} // namespace plain
} // namespace nadia
