// fft64_any.cuh -- row and column transforms of any plan (lengths that are not
// one of fft64_p2.cuh's), tile by tile through two shared-memory buffers.
//
// Neighbouring small radices are joined (2*3, 2*5, 3*3), which saves a trip
// through shared memory each, but no further: the passes are bound by latency,
// and with 16 and 15 values a thread (128 registers) an SM held half as many
// blocks (HIO 1000x1200 150 us; with at most 10 values and the block's shape
// fitted to the plan 116 us).  The first pass reads global memory and, where
// nothing else is to be fetched, the last one writes it (96 us).  The arithmetic
// and its order stay those of the separate passes.  A large prime p costs 8p
// operations a value.
#pragma once

#include "fft64.cuh"

namespace nadia {
namespace plain {
namespace {


// Value `pos` of signal `sig` in a buffer: the signals of a tile are interleaved,
// and where the first pass writes at a stride of 8 or 4 values its outputs are
// permuted within groups of eight (sh = 3 or 2; 31: not), which spreads them
// over the banks.
template <int L>
__device__ __forceinline__ int slot_any(int pos, int sig, int sh)
{
    return (pos ^ ((pos >> sh) & (8 / L - 1))) * L + sig;
}

// The first pass (span 1, no twiddles on its inputs): in(sig, pos) to `dst`.
template <int L, int R1, int R2, bool FWD, class In>
__device__ __forceinline__ void any_first(In &&in, double2 *dst, bool swizzled, const Fft64Pass &s,
                                          const double2 *__restrict__ tw)
{
    constexpr int R = R1 * R2;
    const int flip = (R == 8 || R == 4) && swizzled ? 8 / L - 1 : 0;
    const int m = (int)s.dm.d, total = L * m;
    for (int b = threadIdx.x; b < total; b += (int)blockDim.x) {
        const int sig = b % L, j = b / L;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = in(sig, j + r * m);
        super<R1, R2, FWD>(v, 0, 1, tw, tw + s.tw2, tw + s.wq1, tw + s.wq2);
        const int base = R * j;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int pos = base + out_offset<R1, R2>(r);
            // (pos / R) is j
            dst[((R == 8 || R == 4) ? pos ^ (j & flip) : pos) * L + sig] = v[r];
        }
    }
}

// A pass from `src` to `dst`.
template <int L, int R1, int R2, bool FWD>
__device__ __forceinline__ void any_pass(const double2 *src, double2 *dst, int sh,
                                         const Fft64Pass &s, const double2 *__restrict__ tw)
{
    constexpr int R = R1 * R2;
    const int m = (int)s.dm.d, Ns = s.Ns, total = L * m;
    for (int b = threadIdx.x; b < total; b += (int)blockDim.x) {
        const int sig = b % L, j = b / L;
        const int g = s.dNs.div(j), k = j - g * Ns;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[slot_any<L>(j + r * m, sig, sh)];
        super<R1, R2, FWD>(v, k, Ns, tw + s.tw1, tw + s.tw2, tw + s.wq1, tw + s.wq2);
        double2 *d = dst + (g * Ns * R + k) * L + sig;
        const int step = Ns * L;
#pragma unroll
        for (int r = 0; r < R; ++r) d[out_offset<R1, R2>(r) * step] = v[r];
    }
}

// The last pass: from `src` to out(sig, first position, distance, values), the
// value at q standing at first + out_offset(q) * distance.
template <int L, int R1, int R2, bool FWD, class Out>
__device__ __forceinline__ void any_last(const double2 *src, int sh, const Fft64Pass &s,
                                         const double2 *__restrict__ tw, Out &&out)
{
    constexpr int R = R1 * R2;
    const int m = (int)s.dm.d, Ns = s.Ns, total = L * m; // m = Ns: k = j
    for (int b = threadIdx.x; b < total; b += (int)blockDim.x) {
        const int sig = b % L, j = b / L;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[slot_any<L>(j + r * m, sig, sh)];
        super<R1, R2, FWD>(v, j, Ns, tw + s.tw1, tw + s.tw2, tw + s.wq1, tw + s.wq2);
#pragma unroll
        for (int r = 0; r < R; ++r) out(sig, j + out_offset<R1, R2>(r) * Ns, v[r]);
    }
}

// A prime radix above 7.  The inputs, twiddled, go to the other buffer in plain
// order; then each item of work is C outputs of one butterfly, summed over the
// inputs in increasing order (lanes of a warp take neighbouring butterflies and
// share the C twiddles W[t * n / R]) and written back to `src`, in which the
// result is.  A step of the sum is one value, C twiddles and 8C operations; the
// twiddles' offsets count up and wrap, and the value's address counts up.
// ZERO: the items of outputs 0 .. C-1; output 0 is the plain sum.
constexpr int kPrimeOut = 4;
template <bool FWD, bool IN_SM, bool ZERO>
__device__ __forceinline__ void prime_sums(const double2 *x, int xstep,
                                           const double2 *__restrict__ w, int R, int s0,
                                           double2 *acc)
{
    constexpr int C = kPrimeOut;
    unsigned id[C], st[C];
    const double2 x0 = *x;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        acc[c] = x0;
        id[c] = 0;
        st[c] = s0 + c < R ? s0 + c : 0;
    }
#pragma unroll 2
    for (int r = 1; r < R; ++r) {
        x += xstep;
        const double2 v = *x;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            double2 y = v;
            if (!(ZERO && c == 0)) {
                id[c] += st[c];
                id[c] = min(id[c], id[c] - (unsigned)R); // back below R
                y = cmul(v, IN_SM ? w[id[c]] : twid<FWD>(w + id[c]));
            }
            acc[c].x = acc[c].x + y.x;
            acc[c].y = acc[c].y + y.y;
        }
    }
}

template <int L, bool FWD, bool IN_SM>
__device__ __forceinline__ void any_prime(double2 *src, double2 *dst, double2 *w, int n, int sh,
                                          const Fft64Pass &s, const double2 *__restrict__ tw)
{
    constexpr int C = kPrimeOut;
    const int R = s.r1, m = (int)s.dm.d, Ns = s.Ns, lm = L * m, nt = (int)blockDim.x;
    if (IN_SM)
        for (int t = threadIdx.x; t < R; t += nt) w[t] = twid<FWD>(tw + s.wq1 + t);
#pragma unroll 4
    for (int e = threadIdx.x; e < L * n; e += nt) {
        const int sig = e % L, pos = e / L;
        double2 v = src[slot_any<L>(pos, sig, sh)];
        if (Ns > 1 && pos >= m) {
            const int r = s.dm.div(pos), j = pos - r * m, k = j - s.dNs.div(j) * Ns;
            if (k > 0) v = cmul(v, twid<FWD>(tw + s.tw1 + (r - 1) * Ns + k));
        }
        dst[e] = v;
    }
    __syncthreads();
    const double2 *tab = IN_SM ? w : tw + s.wq1;
    for (int it = threadIdx.x; it < (R + C - 1) / C * lm; it += nt) {
        const int sb = it / lm, b = it - sb * lm, s0 = C * sb;
        double2 acc[C];
        if (sb == 0)
            prime_sums<FWD, IN_SM, true>(dst + b, lm, tab, R, s0, acc);
        else
            prime_sums<FWD, IN_SM, false>(dst + b, lm, tab, R, s0, acc);
        const int sig = b % L, j = b / L, g = s.dNs.div(j);
        double2 *d = src + (g * Ns * R + (j - g * Ns) + s0 * Ns) * L + sig;
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (s0 + c < R) d[c * Ns * L] = acc[c];
    }
}

#define NADIA_RADICES(X) X(8, 1) X(4, 1) X(2, 1) X(3, 1) X(5, 1) X(7, 1) X(2, 3) X(2, 5) X(3, 3)

// The whole transform of a tile, from in(sig, pos) to out(sig, pos, value).
// DIRECT: the last pass hands its values on from registers; otherwise they go
// through shared memory, for an `out` that has loads of its own to wait for
// (a thread then has four of them under way).
template <int L, bool FWD, bool DIRECT, class In, class Out>
__device__ __forceinline__ void any_transform(double2 *sm, const Fft64Plan &p,
                                              const double2 *__restrict__ tw, In &&in, Out &&out)
{
    double2 *a = sm, *b = sm + any_values(p.n, L, p.swz), *w = b + any_values(p.n, L, p.swz);
    int sh = 31, ip = 0, last = p.np - 1;
    // the first pass, from global memory; a large prime starts from a copy
    {
        const Fft64Pass &s = p.pass[0];
        switch (p.np ? s.r1 * 16 + s.r2 : 0) {
#define NADIA_FIRST(r, q) \
    case (r) * 16 + (q): any_first<L, r, q, FWD>(in, a, p.swz < 31, s, tw); ip = 1; break;
            NADIA_RADICES(NADIA_FIRST)
#undef NADIA_FIRST
        default:
#pragma unroll 4
            for (int e = threadIdx.x; e < L * p.n; e += (int)blockDim.x) a[e] = in(e % L, e / L);
        }
        if (ip) sh = p.swz;
    }
    __syncthreads();
    for (; ip < last + !DIRECT; ++ip) {
        const Fft64Pass &s = p.pass[ip];
        switch (s.r1 * 16 + s.r2) {
#define NADIA_PASS(r, q) \
    case (r) * 16 + (q): any_pass<L, r, q, FWD>(a, b, sh, s, tw); break;
            NADIA_RADICES(NADIA_PASS)
#undef NADIA_PASS
        default:
            if (p.prime_sm)
                any_prime<L, FWD, true>(a, b, w, p.n, sh, s, tw);
            else
                any_prime<L, FWD, false>(a, b, w, p.n, sh, s, tw);
            double2 *t = a; // its result is in `a`
            a = b;
            b = t;
        }
        __syncthreads();
        sh = 31;
        double2 *t = a;
        a = b;
        b = t;
    }
    if (DIRECT && ip == last) {
        const Fft64Pass &s = p.pass[ip];
        switch (s.r1 * 16 + s.r2) {
#define NADIA_LAST(r, q) \
    case (r) * 16 + (q): \
        let_next_start(); \
        any_last<L, r, q, FWD>(a, sh, s, tw, out); \
        return;
            NADIA_RADICES(NADIA_LAST)
#undef NADIA_LAST
        default:
            if (p.prime_sm)
                any_prime<L, FWD, true>(a, b, w, p.n, sh, s, tw);
            else
                any_prime<L, FWD, false>(a, b, w, p.n, sh, s, tw);
        }
        __syncthreads();
        sh = 31;
    }
    let_next_start();
    out.all(a, L * p.n, sh);
}
#undef NADIA_RADICES

// Rows go out as they come.
template <int L>
struct RowsOut {
    const Fft64Args &A;
    int r0, end, n;
    __device__ __forceinline__ void operator()(int sig, int j, double2 v) const
    {
        if (r0 + sig < end) A.dst[(size_t)(r0 + sig) * n + j] = v;
    }
    __device__ __forceinline__ void all(const double2 *a, int values, int sh) const
    {
#pragma unroll 4
        for (int e = threadIdx.x; e < values; e += (int)blockDim.x)
            (*this)(e % L, e / L, a[slot_any<L>(e / L, e % L, sh)]);
    }
};

// Columns pass through their epilogue, G values of a thread at a time: what it
// reads is fetched for all G before the first is used.
template <int L, int MODE>
struct ColsOut {
    static constexpr int G = 4;
    const Fft64Args &A;
    int c0, end;
    double diff = 0, mag = 0;
    __device__ __forceinline__ void operator()(int sig, int i, double2 v)
    {
        if (c0 + sig < end) col_store<MODE>(A, i, c0 + sig, v, Aux{}, diff, mag);
    }
    __device__ __forceinline__ void all(const double2 *a, int values, int sh)
    {
        const int nt = (int)blockDim.x;
#pragma unroll 1
        for (int e0 = threadIdx.x; e0 < values; e0 += G * nt) {
            Aux x[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int e = e0 + g * nt;
                if (e < values && c0 + e % L < end) x[g] = col_fetch<MODE>(A, e / L, c0 + e % L);
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int e = e0 + g * nt;
                if (e < values && c0 + e % L < end)
                    col_store<MODE>(A, e / L, c0 + e % L, a[slot_any<L>(e / L, e % L, sh)], x[g],
                                    diff, mag);
            }
        }
    }
};

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
    any_transform<L, FWD, true>(
        sm, p, A.tw,
        [&](int sig, int j) {
            return r0 + sig < end ? row_load<MODE>(A, r0 + sig, j, diff, mag) : make_double2(0.0, 0.0);
        },
        RowsOut<L>{A, r0, end, p.n});
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
    ColsOut<L, MODE> out{A, c0, end};
    any_transform<L, FWD, MODE == C_PLAIN>(
        sm, p, A.tw,
        [&](int sig, int i) {
            return c0 + sig < end && i >= A.lo && i < A.hi ? A.src[(size_t)i * A.ny + c0 + sig]
                                                           : make_double2(0.0, 0.0);
        },
        out);
    if constexpr (MODE == C_MOD || MODE == C_FRESNEL) leave_error(A, out.diff, out.mag, sm);
}

template <int L, int MODE, bool FWD>
void rows_any(const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_rows_any<L, MODE, FWD>, smem, done, kAnyCarveKB * 100 / 228);
    launch_pass(k_rows_any<L, MODE, FWD>, (A.count + L - 1) / L + (A.pairs > 0), threads, smem, st, A, p);
}

template <int L, int MODE, bool FWD>
void cols_any(const Fft64Args &A, const Fft64Plan &p, int threads, size_t smem, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    allow_smem(k_cols_any<L, MODE, FWD>, smem, done, kAnyCarveKB * 100 / 228);
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
    case R_ODD: rows_any<L, R_ODD, false>(A, p, threads, smem, st); break;
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
