// fft64.h -- the FP64 transforms and the element-wise steps fused with them.
//
// A 2-D transform is the canonical schedule (every row, then every column;
// radix plan and twiddles of plan_radices/twiddles, no fused multiply-add), so
// rows and columns of one transform cannot share a kernel with those of the
// next: an iteration of PlanarCDI or FresnelCDI is four kernels -- rows
// forward, columns forward with the modulus, rows backward, columns backward
// with the support and the combine.  Each 1-D transform reads and writes
// global memory once and everything the reference does between two transforms
// happens on the values in registers: 160 bytes a pixel for an HIO iteration
// (32 + 40 + 32 + 56), where one kernel per loop moved about 370.
//
// Measured on B200, one HIO iteration, one kernel per loop against this form:
// 128^2 52 -> 16 us, 256^2 52 -> 17, 1024^2 138 -> 45, 2048^2 468 -> 222,
// 4096^2 2547 -> 916, 1000x1200 355 -> 96, 645x475 (odd) 380 -> 84, 515x387
// (primes 103 and 43) 2095 -> 123.  What bounds them now: up to 256^2 the four
// dependent launches; to 1024^2 the latency of one wave of blocks; at 2048^2 the
// load and store pipe (32-byte pieces of lines in the column passes) and the
// square root and division of the modulus beside 670 MB of traffic (103 us).
#pragma once

#include "common.h"

namespace nadia {
namespace plain {

// what a row transform reads
enum RowMode {
    R_PLAIN,   // src[i, j]
    R_SWAP,    // s * src[p(i, j)]: Complex_2D::invert before FresnelCDI's transform
    R_WF_FROM, // factor(+1) of s * src[p(i, j)] (FresnelCDI_WF::propagate_from_detector)
    R_WF_TO,   // s * factor(-1)(src[p(i, j)])   (FresnelCDI_WF::propagate_to_detector)
    R_ODD,     // odd grids: the swap loop's replay, s^cnt[k] * src[from[k]]
    R_PAD,     // PolyCDI: row i of the estimate, zero outside columns py..py+ny-1
    R_POLY     // PolyCDI: scale_intensity on s * src, times s; error partials
};
// what happens to a column transform's outputs
enum ColMode {
    C_PLAIN,
    C_MOD,     // s * set_mag(s * v, sqrt(I)) at measured pixels; error partials
    C_FRESNEL, // factors, white field, modulus, white field, factors; error partials
    C_COMB,    // v = Pf x (swapped and scaled if `swapped`): support and combine into x
    C_POLYQ    // v in place, |s v|^2 of the centred field to q
};

// a divisor below 2^16 of dividends below 2^16: x / d by one multiplication
struct FastDiv {
    unsigned d, mul;
    __host__ __device__ FastDiv() : d(1), mul(0) {}
    explicit FastDiv(unsigned v) : d(v), mul(v > 1 ? (unsigned)(((1ull << 32) + v - 1) / v) : 0) {}
    __device__ __forceinline__ int div(int x) const
    {
        return d == 1 ? x : (int)__umulhi((unsigned)x, mul);
    }
};

// One pass of a plan: the radix-r1 pass at span Ns and, when r2 > 1, the
// radix-r2 pass at span Ns*r1 on the same r1*r2 values in registers.
struct Fft64Pass {
    int r1, r2, Ns, tw1, tw2, wq1, wq2; // offsets of the twiddles and prime-radix tables
    FastDiv dNs, dm;                     // division by Ns and by n / (r1 * r2)
};

// the any-length kernels' launch bounds
constexpr int kAnyMaxThreads = 256, kAnyRegisters = 80;
// KB of shared memory that their blocks take of an SM's 228 (of which the rest
// is L1): the twiddles live in L1, and with all 228 taken 1000x1200 took 110 us
// an iteration and 1080^2 104, with 196 97 and 93, with 132 105 and 109
constexpr int kAnyCarveKB = 196;

constexpr int kMaxSuper = 14;
struct Fft64Plan {
    int n, np, swz; // swz: 3 or 2 where the first pass is of radix 8 or 4, else 31
    int prime_sm;   // the prime radices' table fits in shared memory
    Fft64Pass pass[kMaxSuper];
};

// values of one shared-memory buffer of the any-length kernels: the swizzle
// permutes positions within groups of eight
__host__ __device__ inline int any_values(int n, int L, int swz)
{
    return (swz < 31 ? (n + 7) & ~7 : n) * L;
}

struct Fft64Args {
    const double2 *src = nullptr;
    double2 *dst = nullptr;
    int nx = 0, ny = 0;         // the grid the transform runs on
    int first = 0, count = 0;   // rows or columns first .. first+count-1
    int lo = 0, hi = 0;         // column transforms: rows outside [lo, hi) read as zero
    const double2 *tw = nullptr;
    double s = 1;
    const double *isqrt = nullptr, *bs = nullptr, *sup = nullptr;
    const double2 *coef = nullptr, *ill = nullptr;
    const int *from = nullptr;  // R_ODD
    const unsigned char *cnt = nullptr;
    int swapped = 0;            // C_MOD: sqrt(I) at p(q); C_COMB: the value belongs to p(q)
    double2 *x = nullptr;       // C_COMB
    double w[5] = {0, 0, 0, 0, 0}, id = 0;
    int er = 0, use_ps = 0, use_psf = 0;
    int wnx = 0, wny = 0, px = 0, py = 0; // PolyCDI: the unpadded grid and its offset
    const double *calc = nullptr;         // PolyCDI: sqrt of the expanded intensity
    double *q = nullptr;
    // error metric: a pass with a modulus leaves one pair of sums per block in
    // `partials`; the next pass, given their number in `pairs`, has one block
    // more than its tiles, which adds them up into *err and
    // ring[*iter % ring_len] beside the transforms
    double *partials = nullptr, *err = nullptr, *ring = nullptr;
    int pairs = 0;
    long long *iter = nullptr;
    int ring_len = 1;
};

// The transforms along one axis: plan, twiddles (per pass, in the order a
// block reads them) and launch shape.
struct Fft64Axis {
    Fft64Plan plan{};
    DevBuf<double2> tw;
    bool p2 = false; // 64 ... 4096, a power of two
    int max_prime = 0;
    void init(int n);
    int tile_p2(int count, bool cols) const; // signals to a block
    void shape_any(int count, bool cols, int *L, int *threads) const;
    size_t smem_any(int L) const;
};

// fft64_p2_*.cu: N = 64 ... 4096; false where the combination is not compiled
bool launch_rows_p2(int N, int L, RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st);
bool launch_cols_p2(int N, int L, ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st);
// fft64_any*.cu
void launch_rows_any(int L, RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
                     int threads, size_t smem, cudaStream_t st);
void launch_cols_any(int L, ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
                     int threads, size_t smem, cudaStream_t st);

// In-place unnormalised 2-D DFT of an nx-by-ny row-major double2 array with
// the canonical Stockham schedule: every row (length ny), then every column.
struct Fft2d {
    int nx = 0, ny = 0;
    Fft64Axis X, Y; // columns (length nx), rows (length ny)
    void init(int nx, int ny);
    void exec(double2 *a, bool forward, cudaStream_t s) const;
    // rows/columns A.first .. +A.count-1 in a fused mode; nx, ny and tw are
    // filled in.  Returns the number of blocks (pairs of error sums).
    int rows(RowMode mode, bool forward, Fft64Args A, cudaStream_t s) const;
    int cols(ColMode mode, bool forward, Fft64Args A, cudaStream_t s) const;
};

// the error metric from `pairs` pairs of sums, where no pass follows
void finish_error(const Fft64Args &A, cudaStream_t s);

// the largest dynamic shared memory a kernel may have, raised once per device
template <class K>
void allow_smem(K kernel, size_t bytes, std::atomic<unsigned long long> &done, int carveout = 0)
{
    if (bytes <= 48 * 1024 && !carveout) return;
    int dev = 0;
    NADIA_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    NADIA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    if (carveout)
        NADIA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, carveout));
    done.fetch_or(bit, std::memory_order_release);
}

} // namespace plain
} // namespace nadia
