// fft64_p2.cuh -- row and column transforms of 64 ... 4096 points (powers of
// two), with every index a compile-time constant.
//
// A thread holds 8 values (16 where the plan ends in an 8 and a 2, which it
// then does without an exchange between them).  The first pass's inputs come
// straight from global memory and the last pass's outputs go straight back,
// so a length of np passes costs np-1 trips through shared memory.  The
// signals of a tile are interleaved there: neighbouring lanes hold the same
// position of neighbouring signals, which makes the twiddles of a warp one or
// two lines and the bank pattern independent of the span.
#pragma once

#include "fft64.cuh"

namespace nadia {
namespace plain {
namespace {

// The passes of a length: 8s, then the remaining 4 or 2.  At 1024 points the 2 is
// joined to the last 8 (sixteen values a thread, one exchange less: HIO 1024^2
// 53.3 us against 56.3); at 128 points the grid is too small for half as many
// threads (128^2 23 us joined, 15.5 not).
template <int N>
struct P2 {
    static constexpr int lg = N <= 64 ? 6 : N <= 128 ? 7 : N <= 256 ? 8 : N <= 512 ? 9
                            : N <= 1024 ? 10 : N <= 2048 ? 11 : 12;
    static constexpr bool join = lg == 10;
    static constexpr int np = lg / 3 + (lg % 3 != 0 && !join);
    static constexpr int EPT = join ? 16 : 8;
    static constexpr int r1(int p) { return p < lg / 3 ? 8 : lg % 3 == 2 ? 4 : 2; }
    static constexpr int r2(int p) { return join && p == np - 1 ? 2 : 1; }
    static constexpr int span(int p) { return p == 0 ? 1 : span(p - 1) * r1(p - 1) * r2(p - 1); }
    static constexpr int tw(int p) // offset of the pass's twiddles: the first pass has none
    {
        return p <= 1 ? 0 : tw(p - 1) + (r1(p - 1) - 1) * span(p - 1);
    }
};

// Position of value `pos` of signal `sig` in the exchange buffer: the signals
// of a tile are interleaved; the exclusive or spreads the first pass's writes
// (stride 8) over the banks.
template <int L>
__device__ __forceinline__ int slot64(int pos, int sig)
{
    constexpr int mask = 8 / L - 1;
    return (pos ^ ((pos >> 3) & mask)) * L + sig;
}

// Pass P of the tile, from `v` to the next pass's inputs, or to `store` after
// the last.  A thread holds EPT values: NB butterflies of radix R.
template <int N, int L, int NT, bool FWD, int P, class Store>
__device__ __forceinline__ void passes(double2 *v, double2 *sm, const double2 *__restrict__ tw,
                                       Store &&store)
{
    using PL = P2<N>;
    constexpr int R1 = PL::r1(P), R2 = PL::r2(P), R = R1 * R2, NB = PL::EPT / R, Ns = PL::span(P);
    const double2 *t1 = tw + PL::tw(P), *t2 = t1 + (P > 0 ? (R1 - 1) * Ns : 0);
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int b = threadIdx.x + q * NT, j = b / L;
        super<R1, R2, FWD>(v + q * R, P == 0 ? 0 : j % Ns, Ns, t1, t2, nullptr, nullptr);
    }
    if constexpr (P == PL::np - 1) {
        let_next_start();
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int b = threadIdx.x + q * NT, sig = b % L, j = b / L;
            store(sig, (j / Ns) * Ns * R + j % Ns, v + q * R);
        }
    } else {
        if (P > 0) __syncthreads(); // every value of the last exchange has been read
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int b = threadIdx.x + q * NT, sig = b % L, j = b / L;
            const int base = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r)
                sm[slot64<L>(base + out_offset<R1, R2>(r) * Ns, sig)] = v[q * R + r];
        }
        __syncthreads();
        constexpr int Rn = PL::r1(P + 1) * PL::r2(P + 1), NBn = PL::EPT / Rn, m = N / Rn;
#pragma unroll
        for (int q = 0; q < NBn; ++q) {
            const int b = threadIdx.x + q * NT, sig = b % L, j = b / L;
#pragma unroll
            for (int r = 0; r < Rn; ++r) v[q * Rn + r] = sm[slot64<L>(j + r * m, sig)];
        }
        passes<N, L, NT, FWD, P + 1>(v, sm, tw, store);
    }
}

template <int N, int L>
struct Tile64 {
    static constexpr int nt = N * L / P2<N>::EPT;
    // registers for two blocks of 512 threads or their like on an SM; a
    // sixteen-value thread needs twice as many
    static constexpr int minb = (P2<N>::EPT == 16 ? 512 : 1024) / nt > 8 ? 8
                              : (P2<N>::EPT == 16 ? 512 : 1024) / nt < 1 ? 1
                              : (P2<N>::EPT == 16 ? 512 : 1024) / nt;
    static constexpr size_t smem = (size_t)N * L * sizeof(double2);
};

// Rows first .. first+count-1, L to a block.
template <int N, int L, int MODE, bool FWD>
__global__ void __launch_bounds__(Tile64<N, L>::nt, Tile64<N, L>::minb) k_rows_p2(const Fft64Args A)
{
    extern __shared__ double2 sm[];
    after_previous();
    constexpr int NT = Tile64<N, L>::nt, R = P2<N>::r1(0), NB = P2<N>::EPT / R, m = N / R;
    const int r0 = A.first + blockIdx.x * L, end = A.first + A.count;
    if (A.pairs && r0 >= end) {
        add_errors(A, sm);
        return;
    }
    double2 v[P2<N>::EPT];
    double diff = 0, mag = 0;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int b = threadIdx.x + q * NT, i = r0 + b % L, j = b / L;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[q * R + r] = i < end ? row_load<MODE>(A, i, j + r * m, diff, mag)
                                   : make_double2(0.0, 0.0);
    }
    passes<N, L, NT, FWD, 0>(v, sm, A.tw, [&](int sig, int base, const double2 *o) {
        constexpr int P = P2<N>::np - 1, R1 = P2<N>::r1(P), R2 = P2<N>::r2(P), Ns = P2<N>::span(P);
        const int i = r0 + sig;
        if (i < end) {
#pragma unroll
            for (int r = 0; r < R1 * R2; ++r)
                A.dst[(size_t)i * N + base + out_offset<R1, R2>(r) * Ns] = o[r];
        }
    });
}

// Columns first .. first+count-1, L to a block.
template <int N, int L, int MODE, bool FWD>
__global__ void __launch_bounds__(Tile64<N, L>::nt, Tile64<N, L>::minb) k_cols_p2(const Fft64Args A)
{
    extern __shared__ double2 sm[];
    after_previous();
    constexpr int NT = Tile64<N, L>::nt, R = P2<N>::r1(0), NB = P2<N>::EPT / R, m = N / R;
    const int c0 = A.first + blockIdx.x * L, end = A.first + A.count;
    if (A.pairs && c0 >= end) {
        add_errors(A, sm);
        return;
    }
    double2 v[P2<N>::EPT];
    double diff = 0, mag = 0;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int b = threadIdx.x + q * NT, c = c0 + b % L, j = b / L;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[q * R + r] = c < end ? A.src[(size_t)(j + r * m) * A.ny + c] : make_double2(0.0, 0.0);
    }
    passes<N, L, NT, FWD, 0>(v, sm, A.tw, [&](int sig, int base, const double2 *o) {
        constexpr int P = P2<N>::np - 1, R1 = P2<N>::r1(P), R2 = P2<N>::r2(P), Ns = P2<N>::span(P);
        constexpr int R_ = R1 * R2, G = R_ < 4 ? R_ : 4;
        const int c = c0 + sig;
        if (c < end) {
#pragma unroll
            for (int g = 0; g < R_; g += G) {
                Aux x[G];
#pragma unroll
                for (int r = 0; r < G; ++r)
                    x[r] = col_fetch<MODE>(A, base + out_offset<R1, R2>(g + r) * Ns, c);
#pragma unroll
                for (int r = 0; r < G; ++r)
                    col_store<MODE>(A, base + out_offset<R1, R2>(g + r) * Ns, c, o[g + r], x[r],
                                    diff, mag);
            }
        }
    });
    if constexpr (MODE == C_MOD || MODE == C_FRESNEL) leave_error(A, diff, mag, sm);
}

template <int N, int L, int MODE, bool FWD>
void rows_p2(const Fft64Args &A, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_rows_p2<N, L, MODE, FWD>, Tile64<N, L>::smem, done);
    launch_pass(k_rows_p2<N, L, MODE, FWD>, (A.count + L - 1) / L + (A.pairs > 0), Tile64<N, L>::nt,
                Tile64<N, L>::smem, st, A);
}

template <int N, int L, int MODE, bool FWD>
void cols_p2(const Fft64Args &A, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_cols_p2<N, L, MODE, FWD>, Tile64<N, L>::smem, done);
    launch_pass(k_cols_p2<N, L, MODE, FWD>, (A.count + L - 1) / L + (A.pairs > 0), Tile64<N, L>::nt,
                Tile64<N, L>::smem, st, A);
}

// every compiled mode of one length and tile width
template <int N, int L>
bool rows_modes(RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (mode) {
    case R_PLAIN: fwd ? rows_p2<N, L, R_PLAIN, true>(A, st) : rows_p2<N, L, R_PLAIN, false>(A, st); return true;
    case R_SWAP: rows_p2<N, L, R_SWAP, true>(A, st); return true;
    case R_WF_FROM: rows_p2<N, L, R_WF_FROM, false>(A, st); return true;
    case R_WF_TO: rows_p2<N, L, R_WF_TO, true>(A, st); return true;
    default: return false;
    }
}

template <int N, int L>
bool cols_modes(ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (mode) {
    case C_PLAIN: fwd ? cols_p2<N, L, C_PLAIN, true>(A, st) : cols_p2<N, L, C_PLAIN, false>(A, st); return true;
    case C_MOD: cols_p2<N, L, C_MOD, true>(A, st); return true;
    case C_FRESNEL: cols_p2<N, L, C_FRESNEL, true>(A, st); return true;
    case C_COMB: cols_p2<N, L, C_COMB, false>(A, st); return true;
    default: return false;
    }
}

} // namespace
} // namespace plain
} // namespace nadia
