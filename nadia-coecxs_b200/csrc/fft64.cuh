// fft64.cuh -- device code of the FP64 transforms (see fft64.h).  Compiled
// with --fmad=false.
#pragma once

#include "fft64.h"

namespace nadia {
namespace plain {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 w)
{
    return make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}

// a twiddle for the direction: conjugated backward
template <bool FWD>
__device__ __forceinline__ double2 twid(const double2 *__restrict__ p)
{
    double2 w = __ldg(p);
    if (!FWD) w.y = -w.y;
    return w;
}

template <bool FWD>
__device__ __forceinline__ void bfly4(double2 &v0, double2 &v1, double2 &v2, double2 &v3)
{
    double2 a, b, c, d;
    a.x = v0.x + v2.x; a.y = v0.y + v2.y;
    b.x = v0.x - v2.x; b.y = v0.y - v2.y;
    c.x = v1.x + v3.x; c.y = v1.y + v3.y;
    d.x = v1.x - v3.x; d.y = v1.y - v3.y;
    v0.x = a.x + c.x; v0.y = a.y + c.y;
    v2.x = a.x - c.x; v2.y = a.y - c.y;
    if (FWD) {
        v1.x = b.x + d.y; v1.y = b.y - d.x;
        v3.x = b.x - d.y; v3.y = b.y + d.x;
    } else {
        v1.x = b.x - d.y; v1.y = b.y + d.x;
        v3.x = b.x + d.y; v3.y = b.y - d.x;
    }
}

// The butterfly of radix R on v[0], v[S], v[2S], ...: 2, 4 and 8 written out,
// odd R the direct sum in increasing input order with wq[t] = W[t * n / R].
template <int R, int S, bool FWD>
__device__ __forceinline__ void bfly(double2 *v, const double2 *__restrict__ wq)
{
    if constexpr (R == 2) {
        const double2 a = v[0], c = v[S];
        v[0].x = a.x + c.x; v[0].y = a.y + c.y;
        v[S].x = a.x - c.x; v[S].y = a.y - c.y;
    } else if constexpr (R == 4) {
        bfly4<FWD>(v[0], v[S], v[2 * S], v[3 * S]);
    } else if constexpr (R == 8) {
        const double c8 = 0.70710678118654752440;
        double2 a[4], b[4], t;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const double2 p = v[r * S], q = v[(r + 4) * S];
            a[r].x = p.x + q.x; a[r].y = p.y + q.y;
            b[r].x = p.x - q.x; b[r].y = p.y - q.y;
        }
        if (FWD) {
            t = b[1]; b[1].x = (t.x + t.y) * c8; b[1].y = (t.y - t.x) * c8;
            t = b[2]; b[2].x = t.y;              b[2].y = -t.x;
            t = b[3]; b[3].x = (t.y - t.x) * c8; b[3].y = -((t.x + t.y) * c8);
        } else {
            t = b[1]; b[1].x = (t.x - t.y) * c8; b[1].y = (t.y + t.x) * c8;
            t = b[2]; b[2].x = -t.y;             b[2].y = t.x;
            t = b[3]; b[3].x = -((t.x + t.y) * c8); b[3].y = (t.x - t.y) * c8;
        }
        bfly4<FWD>(a[0], a[1], a[2], a[3]);
        bfly4<FWD>(b[0], b[1], b[2], b[3]);
#pragma unroll
        for (int r = 0; r < 4; ++r) { v[2 * r * S] = a[r]; v[(2 * r + 1) * S] = b[r]; }
    } else {
        double2 y[R];
        y[0] = v[0];
#pragma unroll
        for (int r = 1; r < R; ++r) { y[0].x = y[0].x + v[r * S].x; y[0].y = y[0].y + v[r * S].y; }
#pragma unroll
        for (int s = 1; s < R; ++s) y[s] = v[0];
#pragma unroll
        for (int r = 1; r < R; ++r)
#pragma unroll
            for (int s = 1; s < R; ++s) {
                const double2 p = cmul(v[r * S], twid<FWD>(wq + (r * s) % R));
                y[s].x = y[s].x + p.x;
                y[s].y = y[s].y + p.y;
            }
#pragma unroll
        for (int s = 0; s < R; ++s) v[s * S] = y[s];
    }
}

// Twiddles and butterflies of a pass on the R1*R2 values of one thread: v[q]
// is input j + q * n/R and, afterwards, the output at base + out_offset(q)*Ns
// with base = (j / Ns) * Ns * R + k, k = j % Ns.  The first element of a group
// (k = 0) is not multiplied.
template <int R1, int R2>
constexpr __host__ __device__ int out_offset(int q)
{
    return q / R2 + (q % R2) * R1;
}

template <int R1, int R2, bool FWD>
__device__ __forceinline__ void super(double2 *v, int k, int Ns, const double2 *__restrict__ tw1,
                                      const double2 *__restrict__ tw2,
                                      const double2 *__restrict__ wq1,
                                      const double2 *__restrict__ wq2)
{
    if (k > 0) {
#pragma unroll
        for (int r = 1; r < R1; ++r) {
            const double2 w = twid<FWD>(tw1 + (r - 1) * Ns + k);
#pragma unroll
            for (int c = 0; c < R2; ++c) v[r * R2 + c] = cmul(v[r * R2 + c], w);
        }
    }
#pragma unroll
    for (int c = 0; c < R2; ++c) bfly<R1, R2, FWD>(v + c, wq1);
    if constexpr (R2 > 1) {
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            if (r > 0 || k > 0) {
#pragma unroll
                for (int c = 1; c < R2; ++c)
                    v[r * R2 + c] = cmul(v[r * R2 + c],
                                         twid<FWD>(tw2 + ((c - 1) * R1 + r) * Ns + k));
            }
            bfly<R2, 1, FWD>(v + r * R2, wq2);
        }
    }
}

// ---------------------------------------------------------- element steps

__device__ __forceinline__ double mag_of(double2 c) { return sqrt(c.x * c.x + c.y * c.y); }

// Complex_2D::set_mag with the magnitude already known
__device__ __forceinline__ double2 set_mag(double2 c, double mag, double value)
{
    if (mag == 0) return make_double2(value, 0.0);
    const double q = value / mag;
    return make_double2(c.x * q, c.y * q);
}

// the quadrant swap's partner of index i on an even axis
__device__ __forceinline__ int partner(int i, int m) { return i < m / 2 ? i + m / 2 : i - m / 2; }

// FresnelCDI::multiply_factors at (i, j): the quarter table's folded index
__device__ __forceinline__ double2 factor(double2 o, const double2 *__restrict__ coef, int i, int j,
                                          int nx, int ny, int direction)
{
    const int i_ = min(i, nx - 1 - i), j_ = min(j, ny - 1 - j);
    const double2 cf = __ldg(&coef[(size_t)i_ * (ny / 2) + j_]);
    const double cr = cf.x, ci = direction * cf.y;
    return make_double2(o.x * cr - o.y * ci, o.y * cr + o.x * ci);
}

// the support constraint on one value
__device__ __forceinline__ double2 supported64(double2 v, double sv)
{
    if (sv == 0) return make_double2(0.0, 0.0);
    if (sv < 1) return make_double2(v.x * sv, v.y * sv);
    return v;
}

// The value a row transform starts from.  MODE R_POLY adds to the error sums.
template <int MODE>
__device__ __forceinline__ double2 row_load(const Fft64Args &A, int i, int j, double &diff,
                                            double &mag)
{
    if constexpr (MODE == R_PLAIN) {
        return A.src[(size_t)i * A.ny + j];
    } else if constexpr (MODE == R_ODD) {
        const size_t k = (size_t)i * A.ny + j;
        double2 v = A.src[__ldg(&A.from[k])];
        for (int c = __ldg(&A.cnt[k]); c > 0; --c) v = make_double2(v.x * A.s, v.y * A.s);
        return v;
    } else if constexpr (MODE == R_PAD) {
        // i: row of the estimate; the transform's row is i + px
        const int c = j - A.py;
        return c >= 0 && c < A.wny ? A.src[(size_t)i * A.wny + c] : make_double2(0.0, 0.0);
    } else if constexpr (MODE == R_POLY) {
        const double2 u = A.src[(size_t)i * A.ny + j];
        double2 v = make_double2(u.x * A.s, u.y * A.s);
        const int r = partner(i, A.nx) - A.px, c = partner(j, A.ny) - A.py;
        if (r >= 0 && r < A.wnx && c >= 0 && c < A.wny) {
            const size_t e = (size_t)r * A.wny + c;
            if (A.bs == nullptr || A.bs[e] > 0) {
                const double calc = A.calc[e], meas = A.isqrt[e];
                const double m = mag_of(v);
                const double scaled = calc == 0.0 ? 0.0 : m * meas / calc;
                v = set_mag(v, m, scaled);
                mag += meas * meas;
                diff += (meas - calc) * (meas - calc);
            }
        }
        return make_double2(v.x * A.s, v.y * A.s);
    } else {
        const int ip = partner(i, A.nx), jp = partner(j, A.ny);
        double2 u = A.src[(size_t)ip * A.ny + jp];
        if (MODE == R_WF_TO) u = factor(u, A.coef, ip, jp, A.nx, A.ny, -1);
        u = make_double2(u.x * A.s, u.y * A.s);
        if (MODE == R_WF_FROM) u = factor(u, A.coef, i, j, A.nx, A.ny, +1);
        return u;
    }
}

// What a column transform's epilogue reads beside its value, fetched for
// several outputs before the first is used.
struct Aux {
    double a, b;
    double2 c, d;
};

template <int MODE>
__device__ __forceinline__ Aux col_fetch(const Fft64Args &A, int i, int j)
{
    Aux x{};
    if constexpr (MODE == C_MOD) {
        const int ip = A.swapped ? partner(i, A.nx) : i, jp = A.swapped ? partner(j, A.ny) : j;
        const size_t d = (size_t)ip * A.ny + jp;
        x.a = __ldg(&A.isqrt[d]);
        x.b = A.bs ? __ldg(&A.bs[d]) : 1.0;
    } else if constexpr (MODE == C_FRESNEL) {
        const size_t d = (size_t)i * A.ny + j;
        x.a = __ldg(&A.isqrt[d]);
        x.b = A.bs ? __ldg(&A.bs[d]) : 1.0;
        x.c = __ldg(&A.ill[d]);
        const int i_ = min(i, A.nx - 1 - i), j_ = min(j, A.ny - 1 - j);
        x.d = __ldg(&A.coef[(size_t)i_ * (A.ny / 2) + j_]);
    } else if constexpr (MODE == C_COMB) {
        const int ip = A.swapped ? partner(i, A.nx) : i, jp = A.swapped ? partner(j, A.ny) : j;
        const int r = ip - A.px, c = jp - A.py;
        if (r >= 0 && r < A.wnx) {
            const size_t d = (size_t)r * A.wny + c;
            x.a = __ldg(&A.sup[d]);
            if (!A.er) x.c = A.x[d];
        }
    }
    return x;
}

// Finishes output (i, j) of a column transform.
template <int MODE>
__device__ __forceinline__ void col_store(const Fft64Args &A, int i, int j, double2 v, const Aux &x,
                                          double &diff, double &mag)
{
    const size_t e = (size_t)i * A.ny + j;
    if constexpr (MODE == C_PLAIN) {
        A.dst[e] = v;
    } else if constexpr (MODE == C_MOD) {
        // PlanarCDI.c++:65-73 around BaseCDI::scale_intensity (BaseCDI.c++:163-189)
        v = make_double2(v.x * A.s, v.y * A.s);
        if (x.b > 0) {
            const double cis = x.a, cm = mag_of(v);
            v = set_mag(v, cm, cis);
            mag += cis * cis;
            diff += (cm - cis) * (cm - cis);
        }
        A.dst[e] = make_double2(v.x * A.s, v.y * A.s);
    } else if constexpr (MODE == C_FRESNEL) {
        // FresnelCDI.c++:217-250
        const double2 t = x.c, cf = x.d;
        double cr = cf.x, ci = -1 * cf.y;
        double2 o = make_double2(v.x * cr - v.y * ci, v.y * cr + v.x * ci);
        o = make_double2(o.x + 1.0 * t.x, o.y + 1.0 * t.y);
        if (x.b > 0) {
            const double cis = x.a, cm = mag_of(o);
            o = set_mag(o, cm, cis);
            mag += cis * cis;
            diff += (cm - cis) * (cm - cis);
        }
        o = make_double2(o.x + -1.0 * t.x, o.y + -1.0 * t.y);
        ci = 1 * cf.y;
        A.dst[e] = make_double2(o.x * cr - o.y * ci, o.y * cr + o.x * ci);
    } else if constexpr (MODE == C_COMB) {
        const int ip = A.swapped ? partner(i, A.nx) : i, jp = A.swapped ? partner(j, A.ny) : j;
        const int r = ip - A.px, c = jp - A.py;
        if (r < 0 || r >= A.wnx) return;
        if (A.swapped) v = make_double2(v.x * A.s, v.y * A.s);
        const size_t d = (size_t)r * A.wny + c;
        if (A.er) {
            A.x[d] = supported64(v, x.a);
            return;
        }
        // the combine of BaseCDI.c++:346-383
        const double2 o = x.c;
        double vr = A.id * o.x, vi = A.id * o.y;
        vr += A.w[3] * v.x;
        vi += A.w[3] * v.y;
        if (A.use_ps) {
            const double2 t = supported64(o, x.a);
            vr += A.w[2] * t.x;
            vi += A.w[2] * t.y;
        }
        if (A.use_psf) {
            const double2 t = supported64(v, x.a);
            vr += A.w[0] * t.x;
            vi += A.w[0] * t.y;
        }
        A.x[d] = make_double2(vr, vi);
    } else { // C_POLYQ: expand_wl's m * m, once per element (PolyCDI.c++:296-334)
        A.dst[e] = v;
        v = make_double2(v.x * A.s, v.y * A.s);
        const double m = mag_of(v);
        A.q[(size_t)partner(i, A.nx) * A.ny + partner(j, A.ny)] = m * m;
    }
}

// ------------------------------------------------------------ error metric

// Sums a pair over the block (a fixed tree: shuffles, then the warps in
// order); thread 0 has the result.
__device__ __forceinline__ void block_pair(double &a, double &b, double *sm)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
    }
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) { sm[2 * w] = a; sm[2 * w + 1] = b; }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < nw; ++k) { a += sm[2 * k]; b += sm[2 * k + 1]; }
}

// The block's error sums to its pair.  `buf`: the block's exchange buffer (at
// least 64 values), no longer needed.
__device__ __forceinline__ void leave_error(const Fft64Args &A, double diff, double mag,
                                            double2 *buf)
{
    __syncthreads();
    block_pair(diff, mag, reinterpret_cast<double *>(buf));
    if (threadIdx.x == 0) {
        A.partials[2 * blockIdx.x] = diff;
        A.partials[2 * blockIdx.x + 1] = mag;
    }
}

// The error metric from the pairs of the pass before, in an order of its own
// fixed by the block size (one block of the following pass).
__device__ __forceinline__ void add_errors(const Fft64Args &A, double2 *buf)
{
    double diff = 0, mag = 0;
    for (int b = threadIdx.x; b < A.pairs; b += blockDim.x) {
        diff += A.partials[2 * b];
        mag += A.partials[2 * b + 1];
    }
    block_pair(diff, mag, reinterpret_cast<double *>(buf));
    if (threadIdx.x == 0) {
        const double e = diff / mag;
        *A.err = e;
        if (A.ring) {
            A.ring[*A.iter % A.ring_len] = e;
            *A.iter += 1;
        }
    }
}

// A pass starts while the one before it drains: its blocks take the places that
// free up and wait here until everything before is complete and visible
// (programmatic dependent launch).  HIO on B200 without and with: 128^2 26.8 ->
// 14.7 us, 256^2 23.8 -> 16.1, 512^2 32.9 -> 23.4, 1024^2 60.1 -> 51.4; with the
// next pass let go at the start of a block instead, 512^2 took 43.7 us.
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// called when a block has only its epilogue left: sooner, and the next pass's
// blocks crowd onto the SMs that happen to have room
__device__ __forceinline__ void let_next_start()
{
    asm volatile("griddepcontrol.launch_dependents;");
}

} // namespace
} // namespace plain
} // namespace nadia
