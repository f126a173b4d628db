// fft64_any4.cu -- the any-length FP64 transforms, 4 signals to a block.
#include "fft64_any.cuh"

namespace nadia {
namespace plain {

void rows_any4(RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    rows_any_modes<4>(mode, fwd, A, p, threads, smem, st);
}

void cols_any4(ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
               int threads, size_t smem, cudaStream_t st)
{
    cols_any_modes<4>(mode, fwd, A, p, threads, smem, st);
}

} // namespace plain
} // namespace nadia
