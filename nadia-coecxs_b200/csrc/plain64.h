// plain64.h -- the plain FP64 path: one kernel per loop of the reference
// (NADIA/src/Complex_2D.c++, BaseCDI.c++, PlanarCDI.c++, FresnelCDI.c++,
// PolyCDI.c++), each performing the same sequence of IEEE-754 double
// operations per element as the reference's double build, so results agree
// bit for bit except for the order of the error-metric sums.  The steps of an
// iteration that lie next to a transform run inside it (fft64.h); the kernels
// here serve everything else.  Compiled with --fmad=false so no multiply-add
// is contracted.
#pragma once

#include "common.h"
#include "fft64.h"

#include <vector>

namespace nadia {
namespace plain {

// Number of blocks used by the two-stage reductions (fixed, so the summation
// order is the same on every call).
constexpr int kRedBlocks = 592;

// Complex_2D::invert(scale), Complex_2D.c++:318-353 (even sizes).
// scratch: nx*ny values, needed for odd sizes (the swap loop's replay is a
// gather into it), unused otherwise
void invert(double2 *a, int nx, int ny, bool scale, cudaStream_t s, double2 *scratch = nullptr);

// The swap loop replayed for an odd grid: out[k] = in[src[k]] times the scale
// cnt[k] times.  Read-only tables, one per device and size, kept for the life
// of the process (like the twiddle tables).
struct OddInvert {
    int *src = nullptr;
    unsigned char *cnt = nullptr;
};
const OddInvert &odd_invert(int nx, int ny);
// the swap and scale_intensity on an odd grid (A: s, isqrt, bs, partials);
// returns the number of pairs of error sums
int odd_modulus(const double2 *in, double2 *out, const OddInvert &t, size_t n, const Fft64Args &A,
                cudaStream_t s);

// BaseCDI::scale_intensity, BaseCDI.c++:163-189.  beam_stop may be null.
// Writes diff/mag to *err (device).
void scale_intensity(double2 *c, const double *isqrt, const double *beam_stop, size_t n,
                     double *partials, double *err, cudaStream_t s);

// BaseCDI::support_constraint, BaseCDI.c++:136-154.
void support_constraint(double2 *c, const double *support, size_t n, cudaStream_t s);

// The combine loop of BaseCDI::iterate, BaseCDI.c++:346-383.  Null term
// pointers are skipped, as the reference skips zero weights.
void combine(double2 *x, const double2 *pfs, const double2 *pf, const double2 *ps,
             const double2 *psf, const double w[5], size_t n, cudaStream_t s);

// The combine of an algorithm whose only projection is Ps, formed on the fly
// from the support (valid without a transmission constraint).
void combine_support(double2 *x, const double *support, bool use_ps, const double w[5], size_t n,
                     cudaStream_t s);

// FresnelCDI::multiply_factors, FresnelCDI.c++:98-126 (quarter table coef).
void multiply_factors(double2 *c, const double2 *coef, int nx, int ny, int direction,
                      cudaStream_t s);

// Complex_2D::add(c2, scale), Complex_2D.c++:184-199.
void add_scaled(double2 *c, const double2 *b, double scale, size_t n, cudaStream_t s);

// Complex_2D::scale, Complex_2D.c++:170-180.
void scale(double2 *c, double f, size_t n, cudaStream_t s);

// get_padded / get_unpadded, Complex_2D.c++:403-460 (zero padding).
void pad(const double2 *x, int nx, int ny, double2 *p, int px, int py, cudaStream_t s);
void unpad(const double2 *p, int nx, int ny, int px, int py, double2 *x, cudaStream_t s);

// PolyCDI::expand_wl, PolyCDI.c++:296-334, evaluated on the central window
// (the only part the reference reads back).  spec: nlambda (wavelength,
// normalised weight) pairs on the device.
void poly_expand(const double2 *c, const double *spec, int nlambda, double lambdac, int nx,
                 int ny, int px, int py, double *isqrt_calc, cudaStream_t s);

// The same from the centred field's squared magnitudes q (rows of my values),
// through per-line tables of sample rows and columns (-1: outside).
void poly_gather(const double *q, const double *spec, int nlambda, const int *rows,
                 const int *cols, int nx, int ny, int my, double *isqrt_calc, cudaStream_t s);

// *err into the history: ring[*iter % ring_len], and *iter counted on.
void record_error(const double *err, double *ring, int ring_len, long long *iter, cudaStream_t s);

// PolyCDI::scale_intensity, PolyCDI.c++:255-292 (c is the padded field).
void poly_scale(double2 *c, const double *isqrt_calc, const double *isqrt,
                const double *beam_stop, int nx, int ny, int px, int py, double *partials,
                double *err, cudaStream_t s);

// get_2d(MAG), Complex_2D.c++:159-165.
void magnitude(const double2 *c, double *out, size_t n, cudaStream_t s);

// BaseCDI::convolve with a cut-off of 5 (set_support's soften), BaseCDI.c++:
// 432-474; g: the (cut+1)^2 weights.
void convolve(const double *in, double *out, int nx, int ny, const std::vector<double> &g,
              cudaStream_t s);

// the maximum of a non-negative array as its bits, and whether a NaN was seen
struct Shrink {
    unsigned long long max;
    int nan;
};

// BaseCDI::apply_shrinkwrap, BaseCDI.c++:416-429: |x| convolved with a cut-off
// of 4 (weights g), thresholded at t of its maximum with apply_threshold's
// `j < nx` bound (BaseCDI.c++:477-492), divided by the maximum of that
// (set_support, BaseCDI.c++:95-102).  w: four words, zero before the first call;
// turn: the number of earlier calls with them.
void shrinkwrap(const double2 *x, double *blurred, double *support, int nx, int ny,
                const std::vector<double> &g, double t, Shrink *w, int turn, cudaStream_t s);

// FresnelCDI::set_transmission_function, FresnelCDI.c++:253-283 (with its
// `j < nx` inner bound).
void fresnel_set_transmission(const double2 *t, const double2 *ill, double2 *esw, int nx,
                              int ny, cudaStream_t s);

// FresnelCDI::get_transmission_function, FresnelCDI.c++:298-355.
void fresnel_get_transmission(const double2 *esw, const double2 *ill, double2 *out, size_t n,
                              cudaStream_t s);

// PlanarCDI::get_intensity_autocorrelation, first loop (PlanarCDI.c++:18-25).
void autocorr_fill(const double *isqrt, double2 *t, size_t n, cudaStream_t s);

// TransmissionConstraint::apply_constraint (TransmissionConstraint.c++:76-172)
// on the device.  region[k] is 0 or the 1-based region of pixel k; params
// holds (alpha1, alpha2, c fixed?, fixed c) per region.  Region sums are
// reduced in a fixed order (kRedBlocks blocks, then one thread per region).
constexpr int kMaxRegions = 16;
void transmission_constraint(double2 *t, const int *region, size_t n, int nregions,
                             const double *params, double *partials, double *cmean,
                             int charge_flip, int flip_sign, int enforce_unity, cudaStream_t s);

} // namespace plain
} // namespace nadia
