// fft64_any8.cu -- the any-length FP64 transforms, 8 signals to a block.
#include "fft64_any.cuh"

namespace nadia {
namespace plain {

void rows_any8(RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    rows_any_modes<8>(mode, fwd, A, p, threads, smem, st);
}

void cols_any8(ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    cols_any_modes<8>(mode, fwd, A, p, threads, smem, st);
}

} // namespace plain
} // namespace nadia
