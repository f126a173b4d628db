// fft64_p2_64.cu -- FP64 transforms of 64 points.
#include "fft64_p2.cuh"

namespace nadia {
namespace plain {

bool rows_p2_64(int L, RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (L) {
    case 4: return rows_modes<64, 4>(mode, fwd, A, st);
    default: return false;
    }
}

bool cols_p2_64(int L, ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (L) {
    case 4: return cols_modes<64, 4>(mode, fwd, A, st);
    default: return false;
    }
}

} // namespace plain
} // namespace nadia
