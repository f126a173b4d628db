// fft64_p2_256.cu -- FP64 transforms of 256 points.
#include "fft64_p2.cuh"

namespace nadia {
namespace plain {

bool rows_p2_256(int L, RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (L) {
    case 1: return rows_modes<256, 1>(mode, fwd, A, st);
    case 2: return rows_modes<256, 2>(mode, fwd, A, st);
    case 4: return rows_modes<256, 4>(mode, fwd, A, st);
    default: return false;
    }
}

bool cols_p2_256(int L, ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (L) {
    case 2: return cols_modes<256, 2>(mode, fwd, A, st);
    case 4: return cols_modes<256, 4>(mode, fwd, A, st);
    default: return false;
    }
}

} // namespace plain
} // namespace nadia
