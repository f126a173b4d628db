// fft64_any.cuh -- row and column transforms of any plan (lengths that are not
// one of fft64_p2.cuh's), tile by tile through two shared-memory buffers.
//
// Neighbouring small radices are joined (2*3, 2*5, 3*3), which saves a trip
// through shared memory each, but no further: the passes are bound by latency,
// and with 16 and 15 values a thread (128 registers) an SM held half as many
// blocks (HIO 1000x1200 150 us; with at most 10 values and the block's shape
// fitted to the plan 123 us).  The arithmetic and its order
// stay those of the separate passes.  A large prime p costs 8p operations a
// value; with four outputs a thread the sums run from one value and four shared
// twiddles a step.
#pragma once

#include "fft64.cuh"

namespace nadia {
namespace plain {
namespace {


// position of value `pos` of signal `sig`; swz spreads the first pass's
// writes (stride 2^swz times an odd number) over the banks
template <int L>
__device__ __forceinline__ int slot_any(int pos, int sig, int swz)
{
    constexpr int mask = 8 / L - 1;
    return (swz ? pos ^ ((pos >> swz) & mask) : pos) * L + sig;
}

// One pass from `src` to `dst`.
template <int L, int R1, int R2, bool FWD>
__device__ __forceinline__ void any_pass(const double2 *src, double2 *dst, int swz,
                                         const Fft64Pass &s, const double2 *__restrict__ tw)
{
    constexpr int R = R1 * R2;
    const int m = (int)s.dm.d, Ns = s.Ns, total = L * m;
    for (int b = threadIdx.x; b < total; b += (int)blockDim.x) {
        const int sig = b % L, j = b / L;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[slot_any<L>(j + r * m, sig, swz)];
        const int g = s.dNs.div(j), k = j - g * Ns;
        super<R1, R2, FWD>(v, k, Ns, tw + s.tw1, tw + s.tw2, tw + s.wq1, tw + s.wq2);
        const int base = g * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r)
            dst[slot_any<L>(base + out_offset<R1, R2>(r) * Ns, sig, swz)] = v[r];
    }
}

// A prime radix above 7: the inputs are twiddled in place, then each item of
// work is C outputs of one butterfly, summed over the inputs in increasing
// order (lanes of a warp take neighbouring butterflies and share the C
// twiddles W[t * n / R]).  ZERO: the items of outputs 0 .. C-1; output 0 is the
// plain sum.
constexpr int kPrimeOut = 4;
template <int L, bool FWD, bool IN_SM, bool ZERO>
__device__ __forceinline__ void prime_item(const double2 *__restrict__ x, double2 *dst,
                                           const double2 *__restrict__ w, int R, int m, int Ns,
                                           int j, int sig, int g, int s0, int swz)
{
    constexpr int C = kPrimeOut;
    double2 acc[C];
    int id[C], st[C];
    const double2 x0 = x[slot_any<L>(j, sig, swz)];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        acc[c] = x0;
        id[c] = 0;
        st[c] = s0 + c < R ? s0 + c : 0;
    }
#pragma unroll 2
    for (int r = 1; r < R; ++r) {
        const double2 v = x[slot_any<L>(j + r * m, sig, swz)];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            double2 y = v;
            if (!(ZERO && c == 0)) {
                id[c] += st[c];
                id[c] -= id[c] >= R ? R : 0;
                y = cmul(v, IN_SM ? w[id[c]] : twid<FWD>(w + id[c]));
            }
            acc[c].x = acc[c].x + y.x;
            acc[c].y = acc[c].y + y.y;
        }
    }
    const int base = g * Ns * R + (j - g * Ns);
#pragma unroll
    for (int c = 0; c < C; ++c)
        if (s0 + c < R) dst[slot_any<L>(base + (s0 + c) * Ns, sig, swz)] = acc[c];
}

template <int L, bool FWD, bool IN_SM>
__device__ __forceinline__ void any_prime(double2 *src, double2 *dst, double2 *w, int n, int swz,
                                          const Fft64Pass &s, const double2 *__restrict__ tw)
{
    constexpr int C = kPrimeOut;
    const int R = s.r1, m = (int)s.dm.d, Ns = s.Ns, lm = L * m, nt = (int)blockDim.x;
    if (IN_SM)
        for (int t = threadIdx.x; t < R; t += nt) w[t] = twid<FWD>(tw + s.wq1 + t);
    if (Ns > 1) {
        for (int e = threadIdx.x + lm; e < L * n; e += nt) {
            const int sig = e % L, pos = e / L, r = s.dm.div(pos), j = pos - r * m;
            const int k = j - s.dNs.div(j) * Ns;
            if (k > 0) {
                double2 &x = src[slot_any<L>(pos, sig, swz)];
                x = cmul(x, twid<FWD>(tw + s.tw1 + (r - 1) * Ns + k));
            }
        }
    }
    __syncthreads();
    const double2 *tab = IN_SM ? w : tw + s.wq1;
    for (int it = threadIdx.x; it < (R + C - 1) / C * lm; it += nt) {
        const int sb = it / lm, b = it - sb * lm, sig = b % L, j = b / L, g = s.dNs.div(j);
        if (sb == 0)
            prime_item<L, FWD, IN_SM, true>(src, dst, tab, R, m, Ns, j, sig, g, 0, swz);
        else
            prime_item<L, FWD, IN_SM, false>(src, dst, tab, R, m, Ns, j, sig, g, C * sb, swz);
    }
}

// All passes of the tile in `a`; returns the buffer that holds the result.
template <int L, bool FWD>
__device__ __forceinline__ double2 *any_passes(double2 *a, const Fft64Plan &p,
                                               const double2 *__restrict__ tw)
{
    double2 *b = a + any_values(p.n, L, p.swz), *w = b + any_values(p.n, L, p.swz);
    for (int ip = 0; ip < p.np; ++ip) {
        const Fft64Pass &s = p.pass[ip];
        switch (s.r1 * 16 + s.r2) {
#define NADIA_PASS(r, q) \
    case (r) * 16 + (q): any_pass<L, r, q, FWD>(a, b, p.swz, s, tw); break;
            NADIA_PASS(2, 1)
            NADIA_PASS(3, 1)
            NADIA_PASS(4, 1)
            NADIA_PASS(5, 1)
            NADIA_PASS(7, 1)
            NADIA_PASS(8, 1)
            NADIA_PASS(2, 3)
            NADIA_PASS(2, 5)
            NADIA_PASS(3, 3)
#undef NADIA_PASS
        default:
            if (p.prime_sm)
                any_prime<L, FWD, true>(a, b, w, p.n, p.swz, s, tw);
            else
                any_prime<L, FWD, false>(a, b, w, p.n, p.swz, s, tw);
        }
        __syncthreads();
        double2 *t = a;
        a = b;
        b = t;
    }
    return a;
}

template <int L, int MODE, bool FWD>
__global__ void __launch_bounds__(kAnyMaxThreads, 3) k_rows_any(const Fft64Args A, const Fft64Plan p)
{
    extern __shared__ double2 sm[];
    after_previous();
    const int r0 = A.first + blockIdx.x * L, end = A.first + A.count;
    if (A.pairs && r0 >= end) {
        add_errors(A, sm);
        return;
    }
    double diff = 0, mag = 0;
#pragma unroll 4
    for (int e = threadIdx.x; e < L * p.n; e += blockDim.x) {
        const int i = r0 + e % L, j = e / L;
        if (i < end) sm[slot_any<L>(j, e % L, p.swz)] = row_load<MODE>(A, i, j, diff, mag);
    }
    __syncthreads();
    const double2 *res = any_passes<L, FWD>(sm, p, A.tw);
    let_next_start();
#pragma unroll 4
    for (int e = threadIdx.x; e < L * p.n; e += blockDim.x) {
        const int i = r0 + e % L, j = e / L;
        if (i < end) A.dst[(size_t)i * p.n + j] = res[slot_any<L>(j, e % L, p.swz)];
    }
    if constexpr (MODE == R_POLY) leave_error(A, diff, mag, sm);
}

template <int L, int MODE, bool FWD>
__global__ void __launch_bounds__(kAnyMaxThreads, 3) k_cols_any(const Fft64Args A, const Fft64Plan p)
{
    extern __shared__ double2 sm[];
    after_previous();
    const int c0 = A.first + blockIdx.x * L, end = A.first + A.count;
    if (A.pairs && c0 >= end) {
        add_errors(A, sm);
        return;
    }
    double diff = 0, mag = 0;
#pragma unroll 4
    for (int e = threadIdx.x; e < L * p.n; e += blockDim.x) {
        const int c = c0 + e % L, i = e / L;
        double2 v = make_double2(0.0, 0.0);
        if (c < end && i >= A.lo && i < A.hi) v = A.src[(size_t)i * A.ny + c];
        sm[slot_any<L>(i, e % L, p.swz)] = v;
    }
    __syncthreads();
    const double2 *res = any_passes<L, FWD>(sm, p, A.tw);
    let_next_start();
#pragma unroll 4
    for (int e = threadIdx.x; e < L * p.n; e += blockDim.x) {
        const int c = c0 + e % L, i = e / L;
        if (c < end) {
            const Aux x = col_fetch<MODE>(A, i, c);
            col_store<MODE>(A, i, c, res[slot_any<L>(i, e % L, p.swz)], x, diff, mag);
        }
    }
    if constexpr (MODE == C_MOD || MODE == C_FRESNEL) leave_error(A, diff, mag, sm);
}

template <int L, int MODE, bool FWD>
void rows_any(const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_rows_any<L, MODE, FWD>, smem, done);
    launch_pass(k_rows_any<L, MODE, FWD>, (A.count + L - 1) / L + (A.pairs > 0), threads, smem, st, A, p);
}

template <int L, int MODE, bool FWD>
void cols_any(const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_cols_any<L, MODE, FWD>, smem, done);
    launch_pass(k_cols_any<L, MODE, FWD>, (A.count + L - 1) / L + (A.pairs > 0), threads, smem, st, A, p);
}

template <int L>
void rows_any_modes(RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem,
                    cudaStream_t st)
{
    switch (mode) {
    case R_PLAIN:
        fwd ? rows_any<L, R_PLAIN, true>(A, p, threads, smem, st) : rows_any<L, R_PLAIN, false>(A, p, threads, smem, st);
        break;
    case R_SWAP: rows_any<L, R_SWAP, true>(A, p, threads, smem, st); break;
    case R_WF_FROM: rows_any<L, R_WF_FROM, false>(A, p, threads, smem, st); break;
    case R_WF_TO: rows_any<L, R_WF_TO, true>(A, p, threads, smem, st); break;
    case R_PAD: rows_any<L, R_PAD, true>(A, p, threads, smem, st); break;
    case R_POLY: rows_any<L, R_POLY, false>(A, p, threads, smem, st); break;
    }
}

template <int L>
void cols_any_modes(ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem,
                    cudaStream_t st)
{
    switch (mode) {
    case C_PLAIN:
        fwd ? cols_any<L, C_PLAIN, true>(A, p, threads, smem, st) : cols_any<L, C_PLAIN, false>(A, p, threads, smem, st);
        break;
    case C_MOD: cols_any<L, C_MOD, true>(A, p, threads, smem, st); break;
    case C_FRESNEL: cols_any<L, C_FRESNEL, true>(A, p, threads, smem, st); break;
    case C_COMB: cols_any<L, C_COMB, false>(A, p, threads, smem, st); break;
    case C_POLYQ: cols_any<L, C_POLYQ, true>(A, p, threads, smem, st); break;
    }
}

} // namespace
} // namespace plain
} // namespace nadia
