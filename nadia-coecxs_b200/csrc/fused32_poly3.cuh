// fused32_poly3.cuh -- PolyCDI's transform passes on tiles whose threads hold one
// butterfly per pass.
//
// A tile of L = 4 signals (one panel of columns, or four rows) of N = RA*RB*RC
// points runs three Stockham passes; pass p has N*L/R butterflies and the first
// N*L/R of the tile's threads take one each.  The radices need not divide a
// common number of values per thread, so 1080 points are 10*12*9 with 12 values
// and 64 registers a thread -- thirty warps an SM -- where tiles that hold every
// value of a thread through all passes need 6*6*6*5 with 30 values, 168
// registers and ten warps, too few to hide the loads and the exchanges.
// B200, PolyCDI 1024^2 padded to 1080^2, an iteration: one reconstruction 49.9 us
// with those tiles and 39.1 with these, four 189 and 135, eight 359 and 271.
// Forming two thirds of the twiddles as products, as the other tiles do, took
// four from 138 to 134 us but leaves the estimate 1.9e-6 from 64 bits after 32 HIO
// iterations, against 1.7e-6 for those tiles and 1.0e-6 with every twiddle from
// the table.
//
// The inverse order is RA, RB, RC and the forward order RC, RB, RA, so that the
// values leaving one transform are the inputs of the other's first pass.
#pragma once

#include "fused32_poly.cuh"

namespace nadia {
namespace f32 {

// 9 = 3 x 3 Cooley-Tukey: X[k1 + 3 k2] = DFT3_q( W9^(q k1) * DFT3_m(v[q + 3m])[k1] )[k2]
template <bool FWD, bool PK>
struct Dft<9, FWD, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        const float sg = FWD ? -1.f : 1.f;
        const float2 w1 = make_float2(0.76604444311897804f, sg * 0.64278760968653933f); // 2 pi / 9
        const float2 w2 = make_float2(0.17364817766693035f, sg * 0.98480775301220806f); // 4 pi / 9
        const float2 w4 = make_float2(-0.93969262078590838f, sg * 0.34202014332566873f); // 8 pi / 9
        float2 a[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            float2 t[3] = {v[q], v[q + 3], v[q + 6]};
            Dft<3, FWD, PK>::run(t);
#pragma unroll
            for (int k = 0; k < 3; ++k) a[q][k] = t[k];
        }
        a[1][1] = cmul(a[1][1], w1);
        a[1][2] = cmul(a[1][2], w2);
        a[2][1] = cmul(a[2][1], w2);
        a[2][2] = cmul(a[2][2], w4);
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            float2 t[3] = {a[0][k1], a[1][k1], a[2][k1]};
            Dft<3, FWD, PK>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = t[k2];
        }
    }
};

template <int N_, int RA_, int RB_, int RC_, int MINB_>
struct Tile3 {
    static constexpr int N = N_, L = 4, RA = RA_, RB = RB_, RC = RC_, MINB = MINB_;
    static constexpr int imax(int a, int b) { return a > b ? a : b; }
    static constexpr int E = imax(RA, imax(RB, RC)); // values a thread holds at most
    static constexpr int NT = N * L / (RA < RB ? (RA < RC ? RA : RC) : (RB < RC ? RB : RC));
    static constexpr size_t smem = (size_t)N * L * sizeof(float2);
    static_assert(RA * RB * RC == N && NT <= 1024 && NT % 32 == 0, "three passes");
    // passes that touch global memory deal rows in panels of four positions
    static_assert((N / RA) % kPanel == 0 && (N / RC) % kPanel == 0, "whole panels");
};

// butterfly `beta` of a pass: its signal and its index in the signal.  EDGE: a
// pass that touches global memory, dealt for the panel layout (rows: 4
// positions x 4 rows of a panel; columns: the panel's 4 columns).
template <int MAP, bool EDGE>
__device__ __forceinline__ void deal3(int beta, int &s, int &j)
{
    if (MAP == kRowMap && EDGE) {
        s = (beta / kPanel) % 4;
        j = beta / 16 * kPanel + beta % kPanel;
    } else {
        s = beta % 4;
        j = beta / 4;
    }
}

// v[r] *= W^(t1 r), every twiddle from the table (no products of twiddles, whose
// rounding would add to the transform's)
template <int R, bool FWD>
__device__ __forceinline__ void twiddle3(float2 *v, int t1, const float2 *__restrict__ tw)
{
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twiddle<FWD>(tw, t1 * r));
}

// The butterflies of a pass of radix R at span Ns, and their outputs to the tile.
template <class T, int MAP, bool FWD, int R, int Ns, bool EDGE>
__device__ __forceinline__ void pass3(float2 *v, float2 *sm, const float2 *__restrict__ tw)
{
    if (threadIdx.x < T::N * T::L / R) {
        int s, j;
        deal3<MAP, EDGE>(threadIdx.x, s, j);
        if (Ns > 1) twiddle3<R, FWD>(v, (j % Ns) * (T::N / (Ns * R)), tw);
        Dft<R, FWD, true>::run(v);
        if (Ns * R < T::N) {
            const int base = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) sm[(base + r * Ns) * T::L + s] = v[r];
        }
    }
}

// the inputs of the next pass (radix R) from the tile
template <class T, int MAP, int R, bool EDGE>
__device__ __forceinline__ void fetch3(float2 *v, const float2 *sm)
{
    __syncthreads();
    if (threadIdx.x < T::N * T::L / R) {
        int s, j;
        deal3<MAP, EDGE>(threadIdx.x, s, j);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = sm[(j + r * (T::N / R)) * T::L + s];
    }
    __syncthreads();
}

// The whole transform: v holds the inputs of the first pass before and the
// outputs of the last one after.
template <class T, int MAP, bool FWD>
__device__ __forceinline__ void transform3(float2 *v, float2 *sm, const float2 *__restrict__ tw)
{
    constexpr int R0 = FWD ? T::RC : T::RA, R1 = T::RB, R2 = FWD ? T::RA : T::RC;
    pass3<T, MAP, FWD, R0, 1, true>(v, sm, tw);
    fetch3<T, MAP, R1, false>(v, sm);
    pass3<T, MAP, FWD, R1, R0, false>(v, sm, tw);
    fetch3<T, MAP, R2, true>(v, sm);
    pass3<T, MAP, FWD, R2, R0 * R1, true>(v, sm, tw);
}

// f(value, signal, position) for the values a thread holds at the radix-R pass
template <class T, int MAP, int R, class F>
__device__ __forceinline__ void each3(F &&f)
{
    if (threadIdx.x < T::N * T::L / R) {
        int s, j;
        deal3<MAP, true>(threadIdx.x, s, j);
#pragma unroll
        for (int r = 0; r < R; ++r) f(r, s, j + r * (T::N / R));
    }
}

// forward column transforms of the estimate's rows (see k_poly_col_fwd)
template <class T>
__global__ void __launch_bounds__(T::NT, T::MINB) k_poly3_col_fwd(const Slot *const *slots,
                                                                   const float2 *__restrict__ tw)
{
    extern __shared__ float2 sm[];
    after_previous();
    const Slot &S = *slots[blockIdx.y];
    float2 *__restrict__ P = S.P;
    const int mx = S.mx, my = S.my, r0 = S.px, r1 = S.mx - S.px;
    const int y0 = blockIdx.x * kPanel;
    float2 v[T::E];
    each3<T, kColMap, T::RC>([&](int e, int s, int pos) {
        v[e] = (pos >= r0 && pos < r1) ? P[paddr(pos, y0 + s, mx)] : make_float2(0.f, 0.f);
    });
    transform3<T, kColMap, true>(v, sm, tw);
    let_next_start();
    const float s02 = S.s0 * S.s0;
    float *__restrict__ q = S.q;
    each3<T, kColMap, T::RA>([&](int e, int s, int kx) {
        const float2 X = v[e];
        P[paddr(kx, y0 + s, mx)] = X;
        q[paddr(centred(kx, mx), centred(y0 + s, my), mx)] = s02 * (X.x * X.x + X.y * X.y);
    });
}

// Psi times the ratio, inverse column transforms (see k_poly_col_inv)
template <class T>
__global__ void __launch_bounds__(T::NT, T::MINB) k_poly3_col_inv(const Slot *const *slots,
                                                                   const float2 *__restrict__ tw)
{
    extern __shared__ float2 sm[];
    after_previous();
    const Slot &S = *slots[blockIdx.y];
    float2 *__restrict__ P = S.P;
    const int mx = S.mx, my = S.my, px = S.px, py = S.py;
    const int nx = mx - 2 * px, ny = my - 2 * py;
    const float *__restrict__ ratio = S.ratio;
    const int y0 = blockIdx.x * kPanel;
    const float s02 = S.s0 * S.s0;
    float2 v[T::E];
    each3<T, kColMap, T::RA>([&](int e, int s, int kx) {
        const int i = centred(kx, mx) - px, j = centred(y0 + s, my) - py;
        float r = 1.f;
        if (i >= 0 && i < nx && j >= 0 && j < ny) r = __ldg(&ratio[paddr(i, j, nx)]);
        v[e] = cscale(P[paddr(kx, y0 + s, mx)], s02 * r);
    });
    transform3<T, kColMap, false>(v, sm, tw);
    let_next_start();
    each3<T, kColMap, T::RC>([&](int e, int s, int pos) {
        if (pos >= px && pos < px + nx) P[paddr(pos, y0 + s, mx)] = v[e];
    });
}

// the exchange tile, then the tile's rows of x and of the support
template <class T>
constexpr size_t poly3_row_smem()
{
    return T::smem + (size_t)T::N * T::L * 12;
}

// inverse row transforms, combine, forward row transforms (see k_poly_row)
template <class T, int MODE>
__global__ void __launch_bounds__(T::NT, T::MINB) k_poly3_row(const Slot *const *slots,
                                                               const float2 *__restrict__ tw)
{
    extern __shared__ float2 sm[];
    after_previous();
    const Slot &S = *slots[blockIdx.y];
    float2 *__restrict__ P = S.P;
    float2 *__restrict__ x = S.x;
    const int mx = S.mx, my = S.my, px = S.px, py = S.py;
    const int nx = mx - 2 * px, ny = my - 2 * py;
    const int i0 = blockIdx.x * T::L; // unpadded row of the tile's first signal
    float2 v[T::E];
    if (MODE == kRowFull) {
        float2 *xs = sm + T::N * T::L;
        float *ss = reinterpret_cast<float *>(xs + T::N * T::L);
        const bool er = S.er;
        // the tile's rows of a panel are one run of 16 elements (ny is a multiple
        // of four in this form)
        const int nseg = ny / kPanel;
        const float2 *__restrict__ xg = x + (size_t)i0 * kPanel;
        const float *__restrict__ sg = S.sup + (size_t)i0 * kPanel;
        if (!er)
            for (int c = threadIdx.x; c < nseg * 8; c += T::NT)
                cp_async16(xs + c * 2, xg + (size_t)(c / 8) * nx * kPanel + 2 * (c % 8));
        for (int c = threadIdx.x; c < nseg * 4; c += T::NT)
            cp_async16(ss + c * 4, sg + (size_t)(c / 4) * nx * kPanel + 4 * (c % 4));
        if (blockIdx.x == 0 && S.project) {
            double t = 0.0;
            for (int b = threadIdx.x; b < S.ncol; b += T::NT) t += S.partials[b];
            t = block_sum<T::NT>(t);
            if (threadIdx.x == 0) {
                const double e = t * S.inv_norm2;
                const long long it = *S.iter;
                *S.err = e;
                S.ring[it % S.ring_len] = e;
                *S.iter = it + 1;
            }
        } else if (blockIdx.x == 0 && threadIdx.x == 0) {
            const long long it = *S.iter;
            S.ring[it % S.ring_len] = *S.err;
            *S.iter = it + 1;
        }
        each3<T, kRowMap, T::RA>([&](int e, int s, int pos) {
            v[e] = P[paddr(px + i0 + s, pos, mx)];
        });
        transform3<T, kRowMap, false>(v, sm, tw);
        cp_async_wait_all();
        __syncthreads();
        const float wid = S.w_id, wpf = S.w_pf, wps = S.w_ps, wpsf = S.w_psf;
        each3<T, kRowMap, T::RC>([&](int e, int s, int pos) {
            const int j = pos - py;
            float2 xn = make_float2(0.f, 0.f);
            if (j >= 0 && j < ny) {
                const size_t a = paddr(i0 + s, j, nx);
                const int b = (j / kPanel * T::L + s) * kPanel + j % kPanel; // staged index
                const float f = support_factor(ss[b]);
                if (er)
                    xn = cscale(v[e], f);
                else
                    xn = combine2(xs[b], v[e], f, wid, wpf, wps, wpsf);
                x[a] = xn;
            }
            v[e] = xn;
        });
    } else {
        each3<T, kRowMap, T::RC>([&](int e, int s, int pos) {
            const int j = pos - py;
            v[e] = (j >= 0 && j < ny) ? x[paddr(i0 + s, j, nx)] : make_float2(0.f, 0.f);
        });
    }
    transform3<T, kRowMap, true>(v, sm, tw);
    let_next_start();
    each3<T, kRowMap, T::RA>([&](int e, int s, int pos) {
        P[paddr(px + i0 + s, pos, mx)] = v[e];
    });
}

template <class K>
void allow3(K kernel, size_t bytes)
{
    NADIA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

template <class T>
PolyVariant make_poly3(const char *radices)
{
    PolyVariant t;
    t.n = T::N;
    t.nt = T::NT;
    t.L = T::L;
    t.radices = radices;
    t.prepare = [] {
        allow3(k_poly3_col_fwd<T>, T::smem);
        allow3(k_poly3_col_inv<T>, T::smem);
        allow3(k_poly3_row<T, kRowFull>, poly3_row_smem<T>());
        allow3(k_poly3_row<T, kRowPrime>, T::smem);
    };
    t.col_fwd = [](const Slot *const *slots, int nslots, int tiles, cudaStream_t st, const float2 *tw) {
        launch_pass(k_poly3_col_fwd<T>, dim3(tiles, nslots), T::NT, T::smem, st, slots, tw);
    };
    t.col_inv = [](const Slot *const *slots, int nslots, int tiles, cudaStream_t st, const float2 *tw) {
        launch_pass(k_poly_expand, dim3(kExpandBlocks, nslots), kExpandThreads, 0, st, slots);
        launch_pass(k_poly3_col_inv<T>, dim3(tiles, nslots), T::NT, T::smem, st, slots, tw);
    };
    t.row = [](int mode, const Slot *const *slots, int nslots, int tiles, cudaStream_t st,
               const float2 *tw) {
        if (mode == kRowFull)
            launch_pass(k_poly3_row<T, kRowFull>, dim3(tiles, nslots), T::NT, poly3_row_smem<T>(), st,
                        slots, tw);
        else
            launch_pass(k_poly3_row<T, kRowPrime>, dim3(tiles, nslots), T::NT, T::smem, st, slots, tw);
    };
    return t;
}

} // namespace f32
} // namespace nadia
