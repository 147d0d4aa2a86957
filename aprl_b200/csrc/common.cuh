// common.cuh -- device-side views, constants and helpers shared by the field
// and particle kernels of the B200 PIC step.
//
// Memory layout in HBM (one run):
//   * Yee components in the reference's SoA layout, x fastest,
//     index (k*ny_c + j)*nx_c + i (src/eb_field.h:134-141), but E and B are
//     z RING BUFFERS: logical plane k lives at physical plane
//     (k + zbase_c) mod nz_c.  The moving-window shift
//     (src/moving_window_fields.cpp:439-518) then only decrements zbase and
//     rewrites the one inserted plane instead of moving the volume.
//   * Two E buffers: E^n ("old") and E* ("star", the zero-current preview
//     with its boundary applied).  The trial candidate E* - dt/eps0 J is never
//     stored.
//   * The wide part of the particle shapes lives on the grid.  A deposit or
//     gather weight of either shape is a narrow weight (linear in x, y, z for
//     linear-binomial3; linear in x, y and the plain B-spline in z for
//     quintic-compensated) convolved with a fixed filter: [1/4, 1/2, 1/4] in
//     x and in z, or the seven compensation coefficients in z.  Particles
//     therefore deposit the narrow weights into the RAW current (12 nodes a
//     piece instead of 64, 44 instead of 92) and gather from the FILTERED
//     orbit sum and B; grid passes apply the filter (J = filter(raw)).  Both
//     are plain (not ring-buffered) arrays of one geometry, padded by the
//     filter's reach: one node on either side in x, jpad planes in z.
//   * CPML convolution histories keep the reference's [slot][k][row] order
//     (src/eb_cpml.cpp:42-96) with the same z ring as their component.
#pragma once

#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace aprl_gpu {

constexpr double kC = 299792458.0;          // src/eb_field.cpp:15-19
constexpr double kEpsilon0 = 8.8541878128e-12;
constexpr double kMu0 = 1.25663706212e-6;
constexpr double kEpsilon = 2.220446049250313080847e-16;  // DBL_EPSILON
constexpr double kDblMin = 2.2250738585072013830903e-308;
constexpr double kPi = 3.14159265358979323846;

// Device error codes (first error wins; the host maps them to statuses).
enum DeviceError : unsigned {
  kErrNone = 0,
  kErrCrossingBudget = 1,     // weights(): more than 64 cuts
  kErrOrbitOutside = 2,       // clipOpenOrbit found no in-domain part
  kErrDepositOutside = 3,     // depositor endpoint outside the E/B domain
  kErrSupportX = 4,           // quintic transverse support outside x grid
  kErrSupportY = 5,           // transverse support outside y grid
  kErrRootNonphysical = 6,    // momentum(): nonphysical mean-gamma root
  kErrRootNoConvergence = 7,  // momentum(): 12 Newton steps exhausted
  kErrNonFinite = 8,          // non-finite particle coordinate
  kErrStartInCpml = 9,        // active particle starts in the CPML region
  kErrStartOutside = 10,      // trajectory starts outside the domain
  kErrBeyondExit = 11,        // active particle started beyond the exit
  kErrUpstream = 12,          // active particle upstream of the inlet
  kErrCarrierWeight = 13,     // invalid carrier weight
  kErrFellBehind = 14,        // particle/carrier behind the moving inlet
  kErrReferenceRange = 15,    // inlet reference query outside the table
  kErrHitLocate = 16,         // boundary hit fraction outside [0,1]
  kErrEarlyRelease = 17,      // held particle released before entering the window
  kErrAdmission = 18,         // invalid upstream admission of a held particle
  kErrHeldBoundary = 19,      // held segment crossed a particle boundary
  kErrInletSource = 20,       // non-finite charge-matched inlet source
  kErrInletField = 21,        // non-finite charge-matched inlet field
  kErrFixedRange = 22,        // deterministic deposit: contribution beyond the fixed-point range
  kErrBounds = 23,            // bounds-checked build: an index outside its array
  kErrSurfaceCurrent = 24,    // non-finite equivalent boundary current of the reference
  kErrReferenceSupport = 25,  // shaped reference source on or outside the zero-potential box
  kErrReferenceSource = 26,   // shaped reference source: non-finite longitudinal coordinate
  kErrReferenceCharge = 27,   // shaped reference source: non-finite charge
  kErrCount
};

struct DeviceStatus {
  unsigned code;
  unsigned long long where;  // particle or element index of the first error
};

__device__ __forceinline__ void raise_error(DeviceStatus* s, unsigned code,
                                            unsigned long long where) {
  if (atomicCAS(&s->code, 0u, code) == 0u) s->where = where;
}

// The bounds-checked build (-DAPRL_GPU_BOUNDS_CHECK, libaprl_b200_checked.so):
// every field, current, orbit-sum, CPML-history and inlet-plane index of the
// step's kernels is tested against its array before the access.  An index
// outside raises kErrBounds in the run's status word with `site` (which
// access) in the top 16 bits of the recorded element and the index below,
// and the access goes to element 0 instead: the kernel never touches memory
// outside its arrays and never traps.  In the normal build the checks
// compile to nothing.  Sites, plus the component: 1 E, 4 B, 7 raw current and
// filtered sum by node, 10 Cowan tile, 16 history, 22 plane 0 before the inlet,
// 24 filtered sum by offset, 27 filtered B by node, 30 chord deposit, 33 raw
// current, 36 S0, 39 E* and 42 filtered sum of a filter pass, 45 B of the
// magnetic filter, 48 visitor's deposit, 51 S0 of the wide gather, 54 B of the
// wide gather, 57 output of the magnetic filter, 60 J read-out, 63 raw current
// or its fixed-point pairs by marked column, 66 column marks, 67 E* and 70 S0 of
// the preview.
#ifdef APRL_GPU_BOUNDS_CHECK
__device__ __forceinline__ size_t bounded(DeviceStatus* s, size_t index, size_t extent,
                                          unsigned site) {
  if (index < extent) return index;
  if (s) raise_error(s, kErrBounds, ((unsigned long long)site << 48) | (index & 0xffffffffffffull));
  return 0;
}
#define APRL_BOUNDED(status, index, extent, site) \
  ::aprl_gpu::bounded((status), (size_t)(index), (size_t)(extent), (site))
#else
#define APRL_BOUNDED(status, index, extent, site) (index)
#endif

// One magnet of SIFieldSourceSet (src/eb_sources.h:103-140).
struct DMagnet {
  int type;  // 0 undulator, 1 dipole, 2 quadrupole
  int gaussian_fringe;
  double center[3];
  double length, period, peak_field;
  double quadrupole_gradient, wave_number, fringe_extent;
  double cos_angle, sin_angle;
};

struct DFrame {  // BoostFrameTransform
  double gamma, beta, gamma_beta;
  double lab_time_origin, lab_z_origin, box_z_origin;
};

// Everything the kernels need about the grid; passed by value.  E and B are
// binary64 in every mode.  F is the type of the current J and of the
// particle-side weight arithmetic: double for the FP64 drop-in, float for
// the FP32-mixed mode.
template <class F>
struct GridT {
  int nx, ny, nz;
  double dx, dy, dz, dt;
  double origin[3];      // localOriginBox_ of the current window
  double* e_old[3];      // E^n  (ring)
  double* e_star[3];     // E*   (ring)
  double* b[3];          // B    (ring)
  F* j[3];               // raw current (plain, padded)
  int jpad;              // its z padding: 1 (linear-binomial3) or 3 (quintic)
  // Columns of the raw current that hold deposits of this step: one byte per
  // row j and eight x nodes (mark_column).  Unmarked columns are zero, so the
  // clears and the filter passes skip them: a bunch reaches about half of a
  // window's columns (and all of their z), and the marks fit in one SM's L1.
  unsigned char* mark;
  int mark_pitch;
  double inv_h[3];       // 1/dx, 1/dy, 1/dz, each rounded once
  int zb_e[3];           // ring bases of Ex Ey Ez
  int zb_b[3];           // ring bases of Bx By Bz
  F jcoef;               // (-1*dt)/eps0, applyCurrentSource(-1) scale
  // Deterministic mode: the deposit adds into these (lo, hi) word pairs
  // (fixed_add, scale jq_scale) instead of J, and a conversion pass writes J
  // from them once per trial.  Null in the default mode.
  unsigned long long* jq[3];
  double jq_scale;
  // Set for the kernels of a fixed-point trial issued ahead of the verdict
  // on the previous one: nonzero once an earlier trial of the step has
  // converged, and the trial's kernels then return at once.
  const int* stop;
  DeviceStatus* status;  // the run's status word (the bounds-checked build reports here)
};

// True when the trial this grid view belongs to was made unnecessary.
template <class F>
__device__ __forceinline__ bool trial_skipped(const GridT<F>& g) {
  return g.stop != nullptr && *g.stop != 0;
}
using DGrid = GridT<double>;

template <class F>
__device__ __forceinline__ int e_nx(const GridT<F>& g, int c) { return g.nx + (c != 0); }
template <class F>
__device__ __forceinline__ int e_ny(const GridT<F>& g, int c) { return g.ny + (c != 1); }
template <class F>
__device__ __forceinline__ int e_nz(const GridT<F>& g, int c) { return g.nz + (c != 2); }
template <class F>
__device__ __forceinline__ int b_nx(const GridT<F>& g, int c) { return g.nx + (c == 0); }
template <class F>
__device__ __forceinline__ int b_ny(const GridT<F>& g, int c) { return g.ny + (c == 1); }
template <class F>
__device__ __forceinline__ int b_nz(const GridT<F>& g, int c) { return g.nz + (c == 2); }

__device__ __forceinline__ int ring(int k, int base, int n) {
  int p = k + base;
  return p >= n ? p - n : p;
}

#ifdef APRL_GPU_BOUNDS_CHECK
// (i, j, k) inside an nx x ny x nz component, else kErrBounds and node 0.
__device__ __forceinline__ bool node_inside(DeviceStatus* s, int i, int j, int k, int nx, int ny,
                                            int nz, unsigned site) {
  if (i >= 0 && i < nx && j >= 0 && j < ny && k >= 0 && k < nz) return true;
  if (s) raise_error(s, kErrBounds, ((unsigned long long)site << 48) |
                                        ((unsigned long long)(unsigned)k << 24) |
                                        (((unsigned long long)(unsigned)j & 0xfffull) << 12) |
                                        ((unsigned long long)(unsigned)i & 0xfffull));
  return false;
}
#define APRL_NODE_CHECK(g, i, j, k, nx, ny, nz, site) \
  if (!node_inside((g).status, (i), (j), (k), (nx), (ny), (nz), (site))) return 0
#else
#define APRL_NODE_CHECK(g, i, j, k, nx, ny, nz, site)
#endif

// Array offsets are formed in 32 bits: a run holds more than fifteen arrays of
// a component's size, so no component that fits a GPU has 2^32 elements.  In
// 64 bits the index arithmetic was over half of the grid kernels'
// instructions.
template <class F>
__device__ __forceinline__ unsigned e_index(const GridT<F>& g, int c, int i, int j, int k) {
  const int nzc = e_nz(g, c);
  APRL_NODE_CHECK(g, i, j, k, e_nx(g, c), e_ny(g, c), nzc, 1 + c);
  return (unsigned)((ring(k, g.zb_e[c], nzc) * e_ny(g, c) + j) * (unsigned)e_nx(g, c) + i);
}

template <class F>
__device__ __forceinline__ unsigned b_index(const GridT<F>& g, int c, int i, int j, int k) {
  const int nzc = b_nz(g, c);
  APRL_NODE_CHECK(g, i, j, k, b_nx(g, c), b_ny(g, c), nzc, 4 + c);
  return (unsigned)((ring(k, g.zb_b[c], nzc) * b_ny(g, c) + j) * (unsigned)b_nx(g, c) + i);
}

// The raw current and the filtered orbit sum of E component c: nodes
// -1 <= i <= e_nx, 0 <= j < e_ny, -jpad <= k < e_nz + jpad.
template <class F>
__device__ __forceinline__ unsigned j_index(const GridT<F>& g, int c, int i, int j, int k) {
  APRL_NODE_CHECK(g, i + 1, j, k + g.jpad, e_nx(g, c) + 2, e_ny(g, c), e_nz(g, c) + 2 * g.jpad,
                  7 + c);
  return (unsigned)(((k + g.jpad) * e_ny(g, c) + j) * (unsigned)(e_nx(g, c) + 2) + (i + 1));
}
template <class F>
__device__ __forceinline__ size_t j_count(const GridT<F>& g, int c) {
  return (size_t)(e_nx(g, c) + 2) * e_ny(g, c) * (e_nz(g, c) + 2 * g.jpad);
}

// Marks raw column (i, j), -1 <= i <= nx + 1, 0 <= j <= ny.  The read spares
// the store of a byte that is already set; a stale read only repeats it.
constexpr int kMarkNodes = 8;
__host__ __device__ __forceinline__ int mark_block(int i) { return (i + 1) / kMarkNodes; }
template <class F>
__device__ __forceinline__ size_t mark_index(const GridT<F>& g, int i, int j) {
  return APRL_BOUNDED(g.status, (size_t)j * g.mark_pitch + mark_block(i),
                      (size_t)(g.ny + 1) * g.mark_pitch, 66);
}
template <class F>
__device__ __forceinline__ void mark_column(const GridT<F>& g, int i, int j) {
  unsigned char* const m = g.mark + mark_index(g, i, j);
  if (!*m) *m = 1;
}
template <class F>
__device__ __forceinline__ bool column_marked(const GridT<F>& g, int i, int j) {
  return g.mark[mark_index(g, i, j)] != 0;
}

// The filtered B of component c: nodes -1 <= i <= b_nx, 0 <= j < b_ny,
// -1 <= k <= b_nz.
template <class F>
__device__ __forceinline__ unsigned bf_index(const GridT<F>& g, int c, int i, int j, int k) {
  APRL_NODE_CHECK(g, i + 1, j, k + 1, b_nx(g, c) + 2, b_ny(g, c), b_nz(g, c) + 2, 27 + c);
  return (unsigned)(((k + 1) * b_ny(g, c) + j) * (unsigned)(b_nx(g, c) + 2) + (i + 1));
}

// Elements of E component c and of B component c.
template <class F>
__device__ __forceinline__ size_t e_count(const GridT<F>& g, int c) {
  return (size_t)e_nx(g, c) * e_ny(g, c) * e_nz(g, c);
}
template <class F>
__device__ __forceinline__ size_t b_count(const GridT<F>& g, int c) {
  return (size_t)b_nx(g, c) * b_ny(g, c) * b_nz(g, c);
}

template <class F>
__device__ __forceinline__ size_t bf_count(const GridT<F>& g, int c) {
  return (size_t)(b_nx(g, c) + 2) * b_ny(g, c) * (b_nz(g, c) + 2);
}

// applyCurrentSource's interior mask (src/source_coupling.cpp:87) at one rank.
template <class F>
__device__ __forceinline__ bool current_mask(const GridT<F>& g, int c, int i, int j, int k) {
  if (c == 0) return j > 0 && j < g.ny && k != 0 && k != g.nz;
  if (c == 1) return i > 0 && i < g.nx && k != 0 && k != g.nz;
  return i > 0 && i < g.nx && j > 0 && j < g.ny;
}

// x / h for a divisor whose reciprocal `inv` = RN(1/h) is at hand: Markstein's
// correction (P. W. Markstein, IBM J. Res. Dev. 34, 1990).  q = x * inv is
// within 1.5 ulp of the quotient; q + (x - q h) inv, each step fused, is
// Q + (Q - q) e for the exact quotient Q and the reciprocal's relative error e,
// an error below 2^-52 ulp before its one rounding.  Markstein's theorem
// gives the correctly rounded quotient for a q within one ulp.  For the q here,
// every pair of significands was compared at each precision from 3 to 13 bits,
// and every binary32 significand over the splines' divisors, without a miss; a
// miss would be one ulp.  So x / h's bits, away from overflow and the subnormal
// range, in three operations instead of the division's loop.
__device__ __forceinline__ double divide_by(double x, double h, double inv) {
  const double q = x * inv;
  return fma(fma(-q, h, x), inv, q);
}
__device__ __forceinline__ float divide_by(float x, float h, float inv) {
  const float q = x * inv;
  return fmaf(fmaf(-q, h, x), inv, q);
}

// ---------------------------------------------------------------------------
// Order-free summation of binary64 contributions (the deterministic mode).
// An addend v -- one contribution, or a warp's sum of up to 32 of them --
// becomes the integer n = round(v * scale), split into lo = n mod 2^32
// (0 <= lo < 2^32) and hi = floor(n / 2^32), and both parts are added with
// 64-bit integer reductions into a (lo, hi) word pair.  Integer addition is
// associative, so after any interleaving of the adds the pair holds the exact
// sum of the rounded addends, hi * 2^32 + lo (hi two's complement), and so
// does every other run: the pair's value does not depend on the order of the
// adds (which lanes a warp sums is a function of the storage order, itself
// reproducible).  `scale` is a power of two chosen by the host so that the
// largest contribution a run can make maps below 2^62, so a warp's sum stays
// below 2^67.  lo stays below 2^64 for fewer than 2^32 adds, and hi, which
// grows by less than 2^30 a contribution and 1 an add, below 2^63 in magnitude
// for fewer than 2^32 contributions to one node.
constexpr double kFixedLimit = 4611686018427387904.0;  // 2^62

// MERGED: v is a warp's sum (the limit leaves room for that sum's rounding).
// Returns false (and adds nothing) for a value outside the range.
template <bool MERGED = false>
__device__ __forceinline__ bool fixed_add(unsigned long long* pair, double v, double scale) {
  const double s = v * scale;
  if (!(fabs(s) < (MERGED ? 64.0 * kFixedLimit : kFixedLimit))) return false;
  unsigned long long lo;
  long long hi;
  // From 2^53 on s is a whole number, so floor and remainder split it exactly
  // without an int64.
  if (!MERGED || fabs(s) < kFixedLimit) {
    const long long n = __double2ll_rn(s);
    lo = (unsigned long long)n & 0xffffffffull;
    hi = n >> 32;
  } else {
    const double h = floor(s * 0x1p-32);
    lo = (unsigned long long)(s - h * 0x1p32);
    hi = (long long)h;
  }
  if (lo) atomicAdd(&pair[0], lo);
  if (hi) atomicAdd(&pair[1], (unsigned long long)hi);
  return true;
}

// The pair's value hi * 2^32 + lo, rounded once to binary64 and multiplied
// by `unscale` (1/scale, a power of two, so that product is exact).
__device__ __forceinline__ double fixed_value(unsigned long long lo, unsigned long long hi_word,
                                              double unscale) {
  const long long hi = (long long)hi_word;
  // 128-bit two's complement (vh:vl) = hi * 2^32 + lo.
  const unsigned long long shifted = (unsigned long long)hi << 32;
  unsigned long long vl = shifted + lo;
  long long vh = (hi >> 32) + (vl < shifted ? 1 : 0);
  const bool negative = vh < 0;
  unsigned long long mh = (unsigned long long)vh, ml = vl;
  if (negative) {  // magnitude: two's complement negation of the 128-bit value
    ml = ~ml + 1ull;
    mh = ~mh + (ml == 0ull ? 1ull : 0ull);
  }
  double m;
  if (mh == 0ull) {
    m = __ull2double_rn(ml);
  } else {
    // The leading 64 bits, with every bit below them folded into bit 0 (a
    // sticky bit under the 11 bits the conversion drops), round once.
    const int lz = __clzll((long long)mh);
    unsigned long long top = lz ? (mh << lz) | (ml >> (64 - lz)) : mh;
    const unsigned long long rest = lz ? ml << lz : ml;
    top |= rest != 0ull ? 1ull : 0ull;
    m = ldexp(__ull2double_rn(top), 64 - lz);
  }
  return (negative ? -m : m) * unscale;
}

// ---------------------------------------------------------------------------
// The quintic-compensated node and edge bases, shared by the deposit, the
// gathers, the charge-matched inlet and the Gauss-law node density.
template <class F>
struct Basis {
  long long first;
  int count;
  F v[12];
};

// The seven compensation coefficients of the p = 5 spline
// (src/longitudinal_shape.h:48-54), each formed in binary64 and rounded once
// to the arithmetic type.
namespace quintic_detail {
constexpr double p = 5., a = p / 6., b = 3 * p / 40. + p * (p - 1) / 72.,
                 d = 5 * p / 112. + p * (p - 1) / 80. + p * (p - 1) * (p - 2) / 1296.;
constexpr double c[7] = {-d / 64.,
                         b / 16. + 3 * d / 32.,
                         -a / 4. - b / 4. - 15 * d / 64.,
                         1 + a / 2. + 3 * b / 8. + 5 * d / 16.,
                         -a / 4. - b / 4. - 15 * d / 64.,
                         b / 16. + 3 * d / 32.,
                         -d / 64.};
}  // namespace quintic_detail

static __constant__ double kQuinticC64[7] = {
    quintic_detail::c[0], quintic_detail::c[1], quintic_detail::c[2], quintic_detail::c[3],
    quintic_detail::c[4], quintic_detail::c[5], quintic_detail::c[6]};
template <class F>
__device__ __forceinline__ F quintic_coefficient(int k) {
  return F(kQuinticC64[k]);
}

// basis(z, edge, QuinticCompensated) (src/longitudinal_shape.h:48-54): the
// cell in binary64, the B-spline and compensation arithmetic in F on the
// cell-relative offset.  The compensation of the degree-`degree` spline
// values n[0..degree]:
template <class F>
__device__ __forceinline__ void quintic_compensate(const F* n, unsigned degree, double cell,
                                                   Basis<F>& r) {
  r.first = (long long)cell - 5;
  r.count = degree + 7;
  for (int q = 0; q < 12; ++q) r.v[q] = F(0.);
  for (unsigned j = 0; j <= degree; ++j)
    for (unsigned k = 0; k < 7; ++k) r.v[j + k] += n[j] * quintic_coefficient<F>(k);
}

// The B-spline recursion on f = z - floor(z) up to `degree`.
template <class F>
__device__ __forceinline__ void quintic_spline_level(F n[6], F f, unsigned j) {
  F saved = F(0.);
#pragma unroll
  for (unsigned k = 0; k < j; ++k) {
    const F t = divide_by(n[k], F(j), F(1.) / F(j));
    n[k] = saved + (F(k + 1) - f) * t;
    saved = (f + F(j) - F(k) - F(1)) * t;
  }
  n[j] = saved;
}

template <class F>
__device__ __forceinline__ void quintic_basis(double z, bool edge, Basis<F>& r) {
  const unsigned degree = edge ? 4 : 5;
  const double cell = floor(z);
  const F f = F(z - cell);
  F n[6] = {F(1.), F(0.), F(0.), F(0.), F(0.), F(0.)};
#pragma unroll
  for (unsigned j = 1; j <= 5; ++j)
    if (j <= degree) quintic_spline_level(n, f, j);
  quintic_compensate(n, degree, cell, r);
}

// BoostFrameTransform::gammaFromProperVelocity (src/boostframe.cpp:74-87).
__device__ __forceinline__ double gamma_u(double ux, double uy, double uz) {
  const double scale = fmax(1.0, fmax(fabs(ux), fmax(fabs(uy), fabs(uz))));
  const double inv = 1.0 / scale;
  const double a = ux * inv, b = uy * inv, c = uz * inv;
  return scale * sqrt(inv * inv + a * a + b * b + c * c);
}

// repeatHeldAddition (src/pending_particle_queue.cpp:38-88): `count`
// separately rounded binary64 additions, with runs of constant spacing
// skipped by integer ULP arithmetic.  Host and device share this code.
__host__ __device__ __forceinline__ unsigned long long held_bits(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(v);
#else
  unsigned long long b;
  memcpy(&b, &v, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double held_from_bits(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}
__host__ __device__ __forceinline__ unsigned long long held_ordered(unsigned long long v) {
  return (v & 0x8000000000000000ull) ? ~v : v ^ 0x8000000000000000ull;
}
__host__ __device__ __forceinline__ double held_from_ordered(unsigned long long v) {
  return held_from_bits((v & 0x8000000000000000ull) ? v ^ 0x8000000000000000ull : ~v);
}
__host__ __device__ __forceinline__ bool held_same_spacing(unsigned long long a,
                                                           unsigned long long b) {
  const unsigned long long m = 0x8000000000000000ull | 0x7ff0000000000000ull;
  return (a & m) == (b & m);
}
__host__ __device__ __forceinline__ double held_repeat_positive(double x, double increment,
                                                                unsigned long long count) {
  while (count) {
    const double y = x + increment;
    if (!isfinite(y)) return y;
    if (count == 1 || y == x) return y;
    const double z = y + increment;
    const unsigned long long bx = held_bits(x), by = held_bits(y), bz = held_bits(z);
    if (isfinite(z) && held_same_spacing(bx, by) && held_same_spacing(by, bz)) {
      const unsigned long long ox = held_ordered(bx), oy = held_ordered(by), oz = held_ordered(bz);
      const unsigned long long stride = oy - ox;
      if (stride && oz - oy == stride) {
        const unsigned long long last_bits =
            (bx & 0x8000000000000000ull) ? bx & (0x8000000000000000ull | 0x7ff0000000000000ull)
                                         : bx | 0x000fffffffffffffull;
        const unsigned long long available = (held_ordered(last_bits) - ox) / stride;
        const unsigned long long safe = available ? available - 1 : 0;
        const unsigned long long jump = safe < count ? safe : count;
        if (jump) {
          x = held_from_ordered(ox + jump * stride);
          count -= jump;
          continue;
        }
      }
    }
    x = y;
    --count;
  }
  return x;
}
__host__ __device__ __forceinline__ double repeat_held_addition(double initial, double increment,
                                                                unsigned long long count) {
  if (!count) return initial;
  if (increment < 0.) {
    const double result = -held_repeat_positive(-initial, -increment, count);
    return result == 0. ? 0. : result;
  }
  return held_repeat_positive(initial, increment, count);
}

// labZFromBoxZT (src/boostframe.cpp:241-245).
__device__ __forceinline__ double lab_z_from_box_zt(const DFrame& f, double z, double t) {
  return f.lab_z_origin + fma(f.gamma_beta * kC, t, f.gamma * (z - f.box_z_origin));
}

}  // namespace aprl_gpu
