// plain64.cu -- kernels of the plain FP64 path (see plain64.h).  Compiled
// with --fmad=false: every product and sum below rounds separately, as in
// the reference's double build compiled without contraction.
#include "plain64.h"

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace nadia {
namespace plain {

namespace {

constexpr int kThreads = 256;

inline int blocks_for(size_t n, int per = kThreads)
{
    size_t b = (n + per - 1) / per;
    return (int)std::min<size_t>(std::max<size_t>(b, 1), 1u << 30);
}

__global__ void k_invert(double2 *a, int nx, int ny, double s)
{
    const int mx = nx / 2, my = ny / 2;
    const size_t total = (size_t)nx * my;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        int i = (int)(e / my), j = (int)(e - (size_t)i * my);
        int jn = j + my, in = i + mx;
        if (i >= mx) in = in - 2 * mx;
        double2 *pp = a + (size_t)in * ny + jn, *qq = a + (size_t)i * ny + j;
        double2 t = *pp, u = *qq;
        *pp = make_double2(u.x * s, u.y * s);
        *qq = make_double2(t.x * s, t.y * s);
    }
}

// Block sum of two doubles with a fixed tree; thread 0 gets the result.
__device__ void block_sum2(double &a, double &b)
{
    __shared__ double sa[kThreads], sb[kThreads];
    sa[threadIdx.x] = a;
    sb[threadIdx.x] = b;
    __syncthreads();
    for (int off = kThreads / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
            sa[threadIdx.x] += sa[threadIdx.x + off];
            sb[threadIdx.x] += sb[threadIdx.x + off];
        }
        __syncthreads();
    }
    a = sa[0];
    b = sb[0];
}

__device__ __forceinline__ double mag_of(double2 c) { return sqrt(c.x * c.x + c.y * c.y); }

__device__ __forceinline__ double2 set_mag(double2 c, double value)
{
    double mag = mag_of(c);
    if (mag == 0) return make_double2(value, 0.0);
    double q = value / mag;
    return make_double2(c.x * q, c.y * q);
}

__global__ void k_scale_intensity(double2 *c, const double *__restrict__ isqrt,
                                  const double *__restrict__ bs, size_t n, double *partials)
{
    double diff = 0, mag = 0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        if (bs == nullptr || bs[k] > 0) {
            double cis = isqrt[k];
            double2 v = c[k];
            double cm = mag_of(v);
            c[k] = set_mag(v, cis);
            mag += cis * cis;
            diff += (cm - cis) * (cm - cis);
        }
    }
    block_sum2(diff, mag);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = diff;
        partials[2 * blockIdx.x + 1] = mag;
    }
}

__global__ void k_finish_error(const double *partials, int nblocks, double *err)
{
    double diff = 0, mag = 0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        diff += partials[2 * b];
        mag += partials[2 * b + 1];
    }
    block_sum2(diff, mag);
    if (threadIdx.x == 0) *err = (diff / mag);
}

// the error metric into the history, as the fused kernels do it themselves
__global__ void k_record(const double *err, double *ring, int ring_len, long long *iter)
{
    ring[*iter % ring_len] = *err;
    *iter += 1;
}

__global__ void k_support(double2 *c, const double *__restrict__ sup, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double sv = sup[k];
        if (sv == 0) {
            c[k] = make_double2(0.0, 0.0);
        } else if (sv < 1) {
            double2 v = c[k];
            c[k] = make_double2(v.x * sv, v.y * sv);
        }
    }
}

struct Weights { double w[5]; double id; };

__global__ void k_combine(double2 *x, const double2 *__restrict__ pfs,
                          const double2 *__restrict__ pf, const double2 *__restrict__ ps,
                          const double2 *__restrict__ psf, Weights W, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = x[k];
        double vr = W.id * v.x, vi = W.id * v.y;
        if (pfs) { double2 t = pfs[k]; vr += W.w[1] * t.x; vi += W.w[1] * t.y; }
        if (pf) { double2 t = pf[k]; vr += W.w[3] * t.x; vi += W.w[3] * t.y; }
        if (ps) { double2 t = ps[k]; vr += W.w[2] * t.x; vi += W.w[2] * t.y; }
        if (psf) { double2 t = psf[k]; vr += W.w[0] * t.x; vi += W.w[0] * t.y; }
        x[k] = make_double2(vr, vi);
    }
}

// k_support's operation on one value
__device__ __forceinline__ double2 supported(double2 v, double sv)
{
    if (sv == 0) return make_double2(0.0, 0.0);
    if (sv < 1) return make_double2(v.x * sv, v.y * sv);
    return v;
}

// The combine loop with Ps x = support(x) formed on the fly (no transmission
// constraint, no other projection); the same sums in the same order as copying,
// projecting and combining separately.
__global__ void k_combine_support(double2 *x, const double *__restrict__ sup, int use_ps, Weights W,
                                  size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        const double2 v = x[k];
        double vr = W.id * v.x, vi = W.id * v.y;
        if (use_ps) {
            const double2 t = supported(v, sup[k]);
            vr += W.w[2] * t.x;
            vi += W.w[2] * t.y;
        }
        x[k] = make_double2(vr, vi);
    }
}

__global__ void k_multiply_factors(double2 *c, const double2 *__restrict__ coef, int nx, int ny,
                                   int direction)
{
    const double x_mid = (nx - 1) / 2.0, y_mid = (ny - 1) / 2.0;
    const int qy = ny / 2;
    const size_t n = (size_t)nx * ny;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        int i = (int)(e / ny), j = (int)(e - (size_t)i * ny);
        double2 o = c[e];
        int i_ = (int)(x_mid - fabs(x_mid - i));
        int j_ = (int)(y_mid - fabs(y_mid - j));
        double2 cf = coef[(size_t)i_ * qy + j_];
        double cr = cf.x, ci = direction * cf.y;
        c[e] = make_double2(o.x * cr - o.y * ci, o.y * cr + o.x * ci);
    }
}

__global__ void k_add_scaled(double2 *c, const double2 *__restrict__ b, double sc, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = c[k], t = b[k];
        c[k] = make_double2(v.x + sc * t.x, v.y + sc * t.y);
    }
}

__global__ void k_scale(double2 *c, double f, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = c[k];
        c[k] = make_double2(v.x * f, v.y * f);
    }
}

__global__ void k_pad(const double2 *__restrict__ x, int nx, int ny, double2 *p, int px, int py)
{
    const int mx = nx + 2 * px, my = ny + 2 * py;
    const size_t n = (size_t)mx * my;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        int i = (int)(e / my) - px, j = (int)(e % my) - py;
        p[e] = (i >= 0 && i < nx && j >= 0 && j < ny) ? x[(size_t)i * ny + j]
                                                      : make_double2(0.0, 0.0);
    }
}

__global__ void k_unpad(const double2 *__restrict__ p, int nx, int ny, int px, int py,
                        double2 *x)
{
    const int my = ny + 2 * py;
    const size_t n = (size_t)nx * ny;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        int i = (int)(e / ny), j = (int)(e - (size_t)i * ny);
        x[e] = p[(size_t)(i + px) * my + j + py];
    }
}

__global__ void k_poly_expand(const double2 *__restrict__ c, const double *__restrict__ spec,
                              int nl, double lambdac, int nx, int ny, int px, int py,
                              double *isc)
{
    const int mx = nx + 2 * px, my = ny + 2 * py;
    const size_t n = (size_t)nx * ny;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        int i = (int)(e / ny) + px, j = (int)(e % ny) + py; // padded coordinates
        double acc = 0.0;
        for (int sn = 0; sn < nl; ++sn) {
            double lambda = spec[2 * sn], weightl = spec[2 * sn + 1];
            double lf = lambda / lambdac;
            double xval = lf * (i - nx / 2.0) + nx / 2.0;
            double yval = lf * (j - ny / 2.0) + ny / 2.0;
            if (((xval >= 0) && (xval < mx)) && ((yval >= 0) && (yval < my))) {
                double m = mag_of(c[(size_t)(int)xval * my + (int)yval]);
                acc = acc + weightl * (m * m);
            }
        }
        isc[e] = sqrt(acc);
    }
}

// expand_wl on the squared magnitudes of the centred field, through the
// sample rows and columns of each line (set_spectrum forms them as
// k_poly_expand does; -1: outside)
__global__ void k_poly_gather(const double *__restrict__ q, const double *__restrict__ spec, int nl,
                              const int *__restrict__ rows, const int *__restrict__ cols, int nx,
                              int ny, int my, double *isc)
{
    for (int i = blockIdx.y; i < nx; i += gridDim.y) {
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ny; j += gridDim.x * blockDim.x) {
            double acc = 0.0;
            for (int l = 0; l < nl; ++l) {
                const int r = __ldg(&rows[l * nx + i]), c = __ldg(&cols[l * ny + j]);
                if (r >= 0 && c >= 0)
                    acc = acc + __ldg(&spec[2 * l + 1]) * __ldg(&q[(size_t)r * my + c]);
            }
            isc[(size_t)i * ny + j] = sqrt(acc);
        }
    }
}

__global__ void k_poly_scale(double2 *c, const double *__restrict__ isc,
                             const double *__restrict__ isqrt, const double *__restrict__ bs,
                             int nx, int ny, int px, int py, double *partials)
{
    const int my = ny + 2 * py;
    const size_t n = (size_t)nx * ny;
    double diff = 0, mag = 0;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        if (bs == nullptr || bs[e] > 0) {
            int i = (int)(e / ny), j = (int)(e - (size_t)i * ny);
            double calc = isc[e], meas = isqrt[e], scaled;
            double2 *pp = c + (size_t)(i + px) * my + j + py;
            double2 v = *pp;
            if (calc == 0.0)
                scaled = 0.0;
            else
                scaled = mag_of(v) * meas / calc;
            *pp = set_mag(v, scaled);
            mag += meas * meas;
            diff += (meas - calc) * (meas - calc);
        }
    }
    block_sum2(diff, mag);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = diff;
        partials[2 * blockIdx.x + 1] = mag;
    }
}

__global__ void k_magnitude(const double2 *__restrict__ c, double *out, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        out[k] = mag_of(c[k]);
}

// The largest value of an array of non-negative doubles, kept as its bits (which
// order like the values) in Shrink::max: NaNs are passed over as
// Real_2D::get_max does, unless the first element is one (then the maximum is
// NaN, whose bits lie above every number's).
__device__ __forceinline__ unsigned long long max_bits(double v, bool first)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return v != v ? (first ? 0x7ff8000000000000ull : 0ull) : b;
}
__device__ __forceinline__ void block_max(unsigned long long m, bool nan, Shrink *w)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, m, off);
        m = o > m ? o : m;
    }
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(&w->max, m);
    if (nan) w->nan = 1;
}

// BaseCDI::convolve (BaseCDI.c++:432-474) by tiles: the input (|x| for a complex
// one) with a halo of CUT in shared memory, zero outside the grid (adding
// 0 * g leaves a sum as it is, so the order and the value of every sum are the
// reference's), four outputs down a column to a thread so that a value read
// from shared memory serves up to four sums.  The window and the order of its
// terms are not separable in rounding, so the 81 (121) products stay; they bound
// the kernel from 1024^2 on (162 operations a pixel, 38 us at 2048^2).
// Measured on B200, whole apply_shrinkwrap: 256^2 190 us, 2048^2 550 us before
// (one thread finishing each maximum, seven kernels and copies).
constexpr int kBlurTile = 32;
struct BlurTable { double g[36]; };

template <int CUT, bool CPLX>
__global__ void __launch_bounds__(kThreads) k_blur64(const void *in, double *out, int nx, int ny,
                                                     const BlurTable T, Shrink *w)
{
    constexpr int H = kBlurTile + 2 * CUT, ROWS = 4;
    __shared__ double t[H][H + 1];
    const int i0 = blockIdx.y * kBlurTile, j0 = blockIdx.x * kBlurTile;
    for (int e = threadIdx.x; e < H * H; e += kThreads) {
        const int a = e / H, b = e - a * H, i = i0 + a - CUT, j = j0 + b - CUT;
        double v = 0;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
            const size_t k = (size_t)i * ny + j;
            v = CPLX ? mag_of(((const double2 *)in)[k]) : ((const double *)in)[k];
        }
        t[a][b] = v;
    }
    __syncthreads();
    const int b = threadIdx.x % kBlurTile, a0 = threadIdx.x / kBlurTile * ROWS;
    double acc[ROWS] = {0, 0, 0, 0};
#pragma unroll
    for (int r = 0; r < ROWS + 2 * CUT; ++r) {
        // row a0 + r of the tile is row r - q of output a0 + q's window
#pragma unroll
        for (int c = 0; c <= 2 * CUT; ++c) {
            const double v = t[a0 + r][b + c];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const int d = r - q;
                if (d >= 0 && d <= 2 * CUT) {
                    const int di = d < CUT ? CUT - d : d - CUT, dj = c < CUT ? CUT - c : c - CUT;
                    acc[q] += v * T.g[di * (CUT + 1) + dj];
                }
            }
        }
    }
    unsigned long long m = 0;
    bool nan = false;
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int i = i0 + a0 + q, j = j0 + b;
        if (i < nx && j < ny) {
            out[(size_t)i * ny + j] = acc[q];
            const unsigned long long o = max_bits(acc[q], i == 0 && j == 0);
            m = o > m ? o : m;
            nan = nan || acc[q] != acc[q];
        }
    }
    if (w) block_max(m, nan, w);
}

__global__ void __launch_bounds__(kThreads) k_max64(const double *__restrict__ a, size_t n, Shrink *w)
{
    unsigned long long m = 0;
    bool nan = false;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        const double v = a[k];
        const unsigned long long o = max_bits(v, k == 0);
        m = o > m ? o : m;
        nan = nan || v != v;
    }
    block_max(m, nan, w);
}

// Square grids visit every element once in apply_threshold, so its values are 0
// and 1 and their maximum is known: the threshold and set_support's division
// by that maximum in one pass.  Clears the words of the next shrinkwrap.
__global__ void k_threshold_divide64(const double *__restrict__ in, double *out, size_t n, double t,
                                     const Shrink *w, Shrink *next)
{
    const double mx = __longlong_as_double((long long)w->max), lim = t * mx;
    const double max2 = !(mx < lim) || w->nan ? 1.0 : 0.0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        out[k] = ((in[k] < lim) ? 0.0 : 1.0) / max2;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        next->max = 0;
        next->nan = 0;
    }
}

// apply_threshold with the reference's loop bounds (i < nx, j < nx) and
// Real_2D::get's (x > nx, y > ny) test: an element at linear index L is
// visited once per pair (i, j = L - i*ny) with 0 <= j < nx, in increasing i.
__global__ void k_threshold(double *a, int nx, int ny, double t, const Shrink *w)
{
    const double lim = t * __longlong_as_double((long long)w->max);
    const size_t n = (size_t)nx * ny;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        long long L = (long long)e;
        long long ilo = (L - nx + 1 + ny - 1) / ny; // ceil((L-nx+1)/ny) for L-nx+1 >= 0
        if (L - nx + 1 < 0) ilo = 0;
        long long ihi = L / ny;
        if (ihi > nx - 1) ihi = nx - 1;
        if (ilo > ihi) continue;
        double cur = a[e];
        for (long long i = ilo; i <= ihi; ++i) {
            long long j = L - i * ny;
            double v = (j > ny) ? 0.0 : cur;
            cur = (v < lim) ? 0.0 : 1.0;
        }
        a[e] = cur;
    }
}

__global__ void k_divide_by_max(const double *__restrict__ in, double *out, size_t n,
                                const Shrink *w)
{
    const double m = __longlong_as_double((long long)w->max);
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        out[k] = in[k] / m;
}

__global__ void k_fresnel_set_t(const double2 *__restrict__ t, const double2 *__restrict__ ill,
                                double2 *esw, int nx, int ny)
{
    const size_t n = (size_t)nx * ny;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
         e += (size_t)gridDim.x * blockDim.x) {
        int j = (int)(e % ny);
        if (ny >= nx && j >= nx) continue;
        double2 l = ill[e], tt = t[e];
        esw[e] = make_double2(l.x * tt.x - l.y * tt.y - l.x, l.x * tt.y + l.y * tt.x - l.y);
    }
}

__global__ void k_fresnel_get_t(const double2 *__restrict__ esw, const double2 *__restrict__ ill,
                                double2 *out, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 l = ill[k];
        double denom = l.x * l.x + l.y * l.y;
        if (denom != 0) {
            double2 e = esw[k];
            double rn = l.x * (e.x + l.x) + l.y * (e.y + l.y);
            double in = l.x * (e.y + l.y) - l.y * (e.x + l.x);
            out[k] = make_double2(rn / denom, in / denom);
        } else {
            out[k] = make_double2(1.0, 0.0);
        }
    }
}

__global__ void k_autocorr_fill(const double *__restrict__ isqrt, double2 *t, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double comp = (1.0 / sqrt(2.0)) * (isqrt[k] * isqrt[k]);
        t[k] = make_double2(comp, comp);
    }
}

inline int grid_of(size_t n) { return std::min(blocks_for(n), 148 * 16); }

} // namespace

// Odd grids: Complex_2D::invert's swap loop (Complex_2D.c++:318-353) then
// visits some elements twice and never moves the last column (for odd ny),
// so its result depends on the loop order.  The loop is replayed once on the
// host over element indices: out[k] = in[src[k]] multiplied cnt[k] times by
// the scale factor, one multiplication after the other as the loop does.
__global__ void k_invert_gather(const double2 *__restrict__ in, double2 *__restrict__ out,
                                const int *__restrict__ src, const unsigned char *__restrict__ cnt,
                                size_t n, double s)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = in[src[k]];
        for (int c = cnt[k]; c > 0; --c) v = make_double2(v.x * s, v.y * s);
        out[k] = v;
    }
}

const OddInvert &odd_invert(int nx, int ny)
{
    static std::mutex mu;
    static std::map<std::tuple<int, int, int>, OddInvert> cache;
    int dev = 0;
    NADIA_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    OddInvert &t = cache[std::make_tuple(dev, nx, ny)];
    if (!t.src) {
        const size_t n = (size_t)nx * ny;
        std::vector<int> src(n);
        std::vector<unsigned char> cnt(n, 0);
        for (size_t k = 0; k < n; ++k) src[k] = (int)k;
        const int mx = nx / 2, my = ny / 2;
        for (int i = 0; i < nx; ++i)
            for (int j = 0; j < my; ++j) {
                int jn = j + my, in = i + mx;
                if (i >= mx) in = in - 2 * mx;
                const size_t p = (size_t)in * ny + jn, q = (size_t)i * ny + j;
                const int ts = src[p];
                const unsigned char tc = cnt[p];
                src[p] = src[q];
                cnt[p] = (unsigned char)(cnt[q] + 1);
                src[q] = ts;
                cnt[q] = (unsigned char)(tc + 1);
            }
        NADIA_CUDA(cudaMalloc(&t.src, n * sizeof(int)));
        NADIA_CUDA(cudaMalloc(&t.cnt, n));
        upload_now(t.src, src.data(), n * sizeof(int));
        upload_now(t.cnt, cnt.data(), n);
    }
    return t;
}

// Odd grids: the swap and scale_intensity (BaseCDI.c++:163-189) of the detector
// side, from the transform `in` to the centred field `out`, with the error sums.
__global__ void k_odd_modulus(const double2 *__restrict__ in, double2 *__restrict__ out,
                              const int *__restrict__ src, const unsigned char *__restrict__ cnt,
                              size_t n, double s, const double *__restrict__ isqrt,
                              const double *__restrict__ bs, double *partials)
{
    double diff = 0, mag = 0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = in[src[k]];
        for (int c = cnt[k]; c > 0; --c) v = make_double2(v.x * s, v.y * s);
        if (bs == nullptr || bs[k] > 0) {
            const double cis = isqrt[k], cm = mag_of(v);
            v = set_mag(v, cis);
            mag += cis * cis;
            diff += (cm - cis) * (cm - cis);
        }
        out[k] = v;
    }
    block_sum2(diff, mag);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = diff;
        partials[2 * blockIdx.x + 1] = mag;
    }
}

int odd_modulus(const double2 *in, double2 *out, const OddInvert &t, size_t n, const Fft64Args &A,
                cudaStream_t s)
{
    const int blocks = std::min(grid_of(n), kRedBlocks);
    k_odd_modulus<<<blocks, kThreads, 0, s>>>(in, out, t.src, t.cnt, n, A.s, A.isqrt, A.bs, A.partials);
    return blocks;
}

void invert(double2 *a, int nx, int ny, bool sc, cudaStream_t s, double2 *scratch)
{
    double f = 1;
    if (sc) f = 1.0 / (sqrt((double)(nx * ny)));
    if ((nx | ny) & 1) {
        NADIA_REQUIRE(scratch != nullptr, NADIA_ERR_INVALID, "odd grids need a scratch array");
        const OddInvert &t = odd_invert(nx, ny);
        const size_t n = (size_t)nx * ny;
        k_invert_gather<<<grid_of(n), kThreads, 0, s>>>(a, scratch, t.src, t.cnt, n, f);
        NADIA_CUDA(cudaMemcpyAsync(a, scratch, n * sizeof(double2), cudaMemcpyDeviceToDevice, s));
        return;
    }
    k_invert<<<grid_of((size_t)nx * (ny / 2)), kThreads, 0, s>>>(a, nx, ny, f);
}

void scale_intensity(double2 *c, const double *isqrt, const double *bs, size_t n,
                     double *partials, double *err, cudaStream_t s)
{
    k_scale_intensity<<<kRedBlocks, kThreads, 0, s>>>(c, isqrt, bs, n, partials);
    k_finish_error<<<1, kThreads, 0, s>>>(partials, kRedBlocks, err);
}

void support_constraint(double2 *c, const double *sup, size_t n, cudaStream_t s)
{
    k_support<<<grid_of(n), kThreads, 0, s>>>(c, sup, n);
}

void combine(double2 *x, const double2 *pfs, const double2 *pf, const double2 *ps,
             const double2 *psf, const double w[5], size_t n, cudaStream_t s)
{
    Weights W;
    for (int i = 0; i < 5; ++i) W.w[i] = w[i];
    W.id = 1 + w[4];
    k_combine<<<grid_of(n), kThreads, 0, s>>>(x, pfs, pf, ps, psf, W, n);
}

void combine_support(double2 *x, const double *support, bool use_ps, const double w[5], size_t n,
                     cudaStream_t s)
{
    Weights W;
    for (int i = 0; i < 5; ++i) W.w[i] = w[i];
    W.id = 1 + w[4];
    k_combine_support<<<grid_of(n), kThreads, 0, s>>>(x, support, use_ps ? 1 : 0, W, n);
}

void multiply_factors(double2 *c, const double2 *coef, int nx, int ny, int direction,
                      cudaStream_t s)
{
    k_multiply_factors<<<grid_of((size_t)nx * ny), kThreads, 0, s>>>(c, coef, nx, ny, direction);
}

void add_scaled(double2 *c, const double2 *b, double sc, size_t n, cudaStream_t s)
{
    k_add_scaled<<<grid_of(n), kThreads, 0, s>>>(c, b, sc, n);
}

void scale(double2 *c, double f, size_t n, cudaStream_t s)
{
    k_scale<<<grid_of(n), kThreads, 0, s>>>(c, f, n);
}

void pad(const double2 *x, int nx, int ny, double2 *p, int px, int py, cudaStream_t s)
{
    size_t n = (size_t)(nx + 2 * px) * (ny + 2 * py);
    k_pad<<<grid_of(n), kThreads, 0, s>>>(x, nx, ny, p, px, py);
}

void unpad(const double2 *p, int nx, int ny, int px, int py, double2 *x, cudaStream_t s)
{
    k_unpad<<<grid_of((size_t)nx * ny), kThreads, 0, s>>>(p, nx, ny, px, py, x);
}

void poly_expand(const double2 *c, const double *spec, int nl, double lambdac, int nx, int ny,
                 int px, int py, double *isc, cudaStream_t s)
{
    k_poly_expand<<<grid_of((size_t)nx * ny), kThreads, 0, s>>>(c, spec, nl, lambdac, nx, ny,
                                                               px, py, isc);
}

void poly_gather(const double *q, const double *spec, int nl, const int *rows, const int *cols,
                 int nx, int ny, int my, double *isc, cudaStream_t s)
{
    dim3 grid((ny + 127) / 128, std::min(nx, 65535));
    k_poly_gather<<<grid, 128, 0, s>>>(q, spec, nl, rows, cols, nx, ny, my, isc);
}

// the error metric where no pass follows the one with the modulus
__global__ void k_finish_pairs(const Fft64Args A)
{
    double diff = 0, mag = 0;
    for (int b = threadIdx.x; b < A.pairs; b += blockDim.x) {
        diff += A.partials[2 * b];
        mag += A.partials[2 * b + 1];
    }
    block_sum2(diff, mag);
    if (threadIdx.x == 0) {
        const double e = diff / mag;
        *A.err = e;
        if (A.ring) {
            A.ring[*A.iter % A.ring_len] = e;
            *A.iter += 1;
        }
    }
}

void finish_error(const Fft64Args &A, cudaStream_t s) { k_finish_pairs<<<1, kThreads, 0, s>>>(A); }

void record_error(const double *err, double *ring, int ring_len, long long *iter, cudaStream_t s)
{
    k_record<<<1, 1, 0, s>>>(err, ring, ring_len, iter);
}

void poly_scale(double2 *c, const double *isc, const double *isqrt, const double *bs, int nx,
                int ny, int px, int py, double *partials, double *err, cudaStream_t s)
{
    k_poly_scale<<<kRedBlocks, kThreads, 0, s>>>(c, isc, isqrt, bs, nx, ny, px, py, partials);
    k_finish_error<<<1, kThreads, 0, s>>>(partials, kRedBlocks, err);
}

void magnitude(const double2 *c, double *out, size_t n, cudaStream_t s)
{
    k_magnitude<<<grid_of(n), kThreads, 0, s>>>(c, out, n);
}

namespace {
template <int CUT>
void blur64(const void *in, bool cplx, double *out, int nx, int ny, const std::vector<double> &g,
            Shrink *w, cudaStream_t s)
{
    BlurTable T{};
    std::copy(g.begin(), g.end(), T.g);
    const dim3 grid((ny + kBlurTile - 1) / kBlurTile, (nx + kBlurTile - 1) / kBlurTile);
    if (cplx)
        k_blur64<CUT, true><<<grid, kThreads, 0, s>>>(in, out, nx, ny, T, w);
    else
        k_blur64<CUT, false><<<grid, kThreads, 0, s>>>(in, out, nx, ny, T, w);
}
} // namespace

void convolve(const double *in, double *out, int nx, int ny, const std::vector<double> &g,
              cudaStream_t s)
{
    blur64<5>(in, false, out, nx, ny, g, nullptr, s);
}

void shrinkwrap(const double2 *x, double *blurred, double *support, int nx, int ny,
                const std::vector<double> &g, double t, Shrink *w, int turn, cudaStream_t s)
{
    const size_t n = (size_t)nx * ny;
    Shrink *now = w + 2 * (turn & 1), *next = w + 2 * ((turn + 1) & 1);
    blur64<4>(x, true, blurred, nx, ny, g, now, s);
    if (nx == ny) {
        k_threshold_divide64<<<grid_of(n), kThreads, 0, s>>>(blurred, support, n, t, now, next);
        return;
    }
    k_threshold<<<grid_of(n), kThreads, 0, s>>>(blurred, nx, ny, t, now);
    k_max64<<<grid_of(n), kThreads, 0, s>>>(blurred, n, now + 1);
    k_divide_by_max<<<grid_of(n), kThreads, 0, s>>>(blurred, support, n, now + 1);
    // the next turn's words
    NADIA_CUDA(cudaMemsetAsync(next, 0, 2 * sizeof(Shrink), s));
}

void fresnel_set_transmission(const double2 *t, const double2 *ill, double2 *esw, int nx, int ny,
                              cudaStream_t s)
{
    k_fresnel_set_t<<<grid_of((size_t)nx * ny), kThreads, 0, s>>>(t, ill, esw, nx, ny);
}

void fresnel_get_transmission(const double2 *esw, const double2 *ill, double2 *out, size_t n,
                              cudaStream_t s)
{
    k_fresnel_get_t<<<grid_of(n), kThreads, 0, s>>>(esw, ill, out, n);
}

// TransmissionConstraint::apply_constraint, TransmissionConstraint.c++:76-172
// region sums of |ln|t|| and |arg t| per block, in a fixed order: each
// thread walks its pixels four at a time (one int4 of the region map, so the
// map streams at full width) and accumulates region pixels in order
__global__ void k_tc_sums(const double2 *__restrict__ t, const int *__restrict__ region, size_t n,
                          int R, double *partials)
{
    double lnA[kMaxRegions], ph[kMaxRegions];
    for (int r = 0; r < R; ++r) lnA[r] = ph[r] = 0;
    const int4 *reg4 = reinterpret_cast<const int4 *>(region);
    const size_t n4 = n / 4; // n = nx*ny with even nx and ny
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n4;
         q += (size_t)gridDim.x * blockDim.x) {
        const int4 rr = __ldg(&reg4[q]);
        const int rv[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int r = rv[c];
            if (r > 0) {
                const double2 v = t[4 * q + c];
                ph[r - 1] += fabs(atan2(v.y, v.x));
                lnA[r - 1] += fabs(log(mag_of(v)));
            }
        }
    }
    for (int r = 0; r < R; ++r) {
        double a = lnA[r], b = ph[r];
        block_sum2(a, b);
        if (threadIdx.x == 0) {
            partials[2 * ((size_t)blockIdx.x * R + r)] = a;
            partials[2 * ((size_t)blockIdx.x * R + r) + 1] = b;
        }
        __syncthreads();
    }
}

// one block per region: the block partials summed by a fixed tree
__global__ void k_tc_cmean(const double *partials, int nblocks, int R, const double *params,
                           double *cmean)
{
    const int r = blockIdx.x;
    double a = 0, b = 0;
    for (int blk = threadIdx.x; blk < nblocks; blk += blockDim.x) {
        a += partials[2 * ((size_t)blk * R + r)];
        b += partials[2 * ((size_t)blk * R + r) + 1];
    }
    block_sum2(a, b);
    if (threadIdx.x == 0) cmean[r] = params[4 * r + 2] != 0 ? params[4 * r + 3] : a / b;
}

__global__ void k_tc_apply(double2 *t, const int *__restrict__ region, size_t n, int R,
                           const double *__restrict__ params, const double *__restrict__ cmean,
                           int flip, int flip_sign, int unity)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x) {
        double2 v = t[k];
        double mag_old = mag_of(v);
        const int r = R > 0 ? region[k] : 0;
        if (r > 0) {
            const double phase_old = atan2(v.y, v.x);
            const double a1 = params[4 * (r - 1)], a2 = params[4 * (r - 1) + 1];
            const double cm = cmean[r - 1];
            const double mag_new = exp((1 - a1) * log(mag_old) + a1 * cm * phase_old);
            const double phase_new = (1 - a2) * phase_old + a2 * log(mag_old) / cm;
            v = set_mag(v, mag_new);
            const double m = mag_of(v); // Complex_2D::set_phase keeps the current magnitude
            v = make_double2(m * cos(phase_new), m * sin(phase_new));
            mag_old = mag_new;
        }
        if (flip && flip_sign * v.y > 0) v.y = -1 * v.y;
        if (unity && mag_old > 1) v = set_mag(v, 1);
        t[k] = v;
    }
}

void autocorr_fill(const double *isqrt, double2 *t, size_t n, cudaStream_t s)
{
    k_autocorr_fill<<<grid_of(n), kThreads, 0, s>>>(isqrt, t, n);
}

void transmission_constraint(double2 *t, const int *region, size_t n, int nregions,
                             const double *params, double *partials, double *cmean,
                             int charge_flip, int flip_sign, int enforce_unity, cudaStream_t s)
{
    if (nregions > 0) {
        k_tc_sums<<<kRedBlocks, kThreads, 0, s>>>(t, region, n, nregions, partials);
        k_tc_cmean<<<nregions, kThreads, 0, s>>>(partials, kRedBlocks, nregions, params, cmean);
    }
    if (nregions > 0 || charge_flip || enforce_unity)
        k_tc_apply<<<grid_of(n), kThreads, 0, s>>>(t, region, n, nregions, params, cmean,
                                                    charge_flip, flip_sign, enforce_unity);
}

} // namespace plain
} // namespace nadia
