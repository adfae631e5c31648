// Romein-strategy convolutional gridder for GB300 (sm_103a).
//
// Work decomposition.  One CTA grids one *track*: the visibilities of one (facet, baseline,
// channel) in time order (rows of a baseline are contiguous after repack_input_data, as in
// bullseye/mo/gpu_algorithm/wrapper.cu:367-454).  Consecutive samples of a track move slowly
// across the uv grid, which is what Romein's ownership scheme exploits (J. W. Romein, "An
// efficient work-distribution strategy for gridding radio-telescope data on GPUs", ICS 2012).
//
// Ownership.  For full support W, the W x W cells under any visibility's kernel footprint
// contain exactly one cell of every (x mod W, y mod W) class.  Thread (du, strip) owns the
// classes x = du (mod W) and y in {strip*J .. strip*J+J-1} (mod W): for each visibility it
// updates exactly the J cells of its classes inside the footprint, accumulating in registers
// while the owned cell stays the same and flushing with a global atomic when it changes.  The
// reference GPU kernel instead binds each thread to a fixed footprint offset
// (bullseye/mo/gpu_algorithm/templated_gridder.h:59-69), which flushes on every cell move.
//
// Per-visibility work (the prologue) is done once per CTA, not once per thread: threads each
// prepare one visibility (correlation selection, weights x flags, Jones J_p^-1 V J_q^-H, facet
// phase rotation, planar uv transform, cell and tap-offset selection) into shared memory (the
// persistent batched kernel stages records that the record kernel prepared, by TMA bulk copies).
// The staged chunk is then merged into groups of visibilities with a common tap row, and the
// owner threads add each group to their cells (see "merged gridding" below).
//
// Numerics (matching the reference CPU library, bullseye/mo/cpu_algorithm/*):
//  * uvw / lambda, the phase argument 2 pi (u dl + v dm + w dn), the uv transform and the
//    cell/tap selection are evaluated in FP64 in both libraries;
//  * 1-D AA kernels select cells and taps with floor (the reference sets FE_DOWNWARD,
//    convolution_policies.h:73-75); w-projection uses round-half-even (FE_TONEAREST, :233);
//  * tap index = trunc((1 - u + round(u)) * os) + j*os; a visibility is dropped when
//    disc + W + 2 >= n or disc < 0 (convolution_policies.h:86-97);
//  * single-precision library: visibilities, taps and the register accumulation are FP32,
//    the phase is evaluated by sincospif on the argument reduced in FP64 to turns; cells are
//    added to the grid in FP64 (two FP64 planes in the place of an FP32 grid and its rounding
//    errors), or in plain FP32 when compensation is off;
//  * normalisation: sum over taps of the real tap weight times weight x flag
//    (templated_gridder.h:97 and store_normalization_term), computed per visibility as
//    Re(sum_j k_u[j] * sum_i k_v[i]) from kernel row sums precomputed in FP64, accumulated per
//    staging slot (FP32 with Kahan compensation in the single library, FP64 in the double one)
//    and reduced per warp into FP64.
#pragma once
#include <algorithm>
#include <type_traits>

#include "common.h"

namespace bz {

#if defined(BULLSEYE_SINGLE)
typedef float acc_real;
#else
typedef double acc_real;
#endif

struct cplx {
  acc_real re, im;
};
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
  cplx r;
  r.re = a.re * b.re - a.im * b.im;
  r.im = a.re * b.im + a.im * b.re;
  return r;
}

enum CorrMode { CORR_SINGLE = 0, CORR_DUAL = 1, CORR_QUAD = 2, CORR_QUAD_JONES = 3, CORR_SAMPLING = 4 };

// Per-facet transform constants in FP64
// (phase_transform_policies.h:110-134, baseline_transform_policies.h:117-149).
struct FacetXform {
  double u_term, v_term;  // planar uv transform: u -= w u_term, v -= w v_term
  double dl, dm, dn;      // phase rotation offsets
  // the facet's grid: uv scale (pixels per wavelength), footprint-corner offsets nx/2 - s and
  // ny/2 - s, the complex-element offset of its [groups][NC][ny][nx] block, and its size
  double u_scale, v_scale, gcx, gcy;
  long long grid_base;
  int nx, ny;
};

// The transform to a facet centre (arcsec), with its phase rotation and its uv transform each on or off: the
// one place where host and device code form it.  At the phase centre both are exactly the identity: where
// multiply-adds are contracted the differences of products below would leave their rounding errors (1e-17),
// which move a sample that lies on a cell boundary.
__host__ __device__ inline FacetXform facet_transform(double ra0, double dec0, double ra, double dec, bool phase,
                                                      bool uvx) {
  FacetXform x = {};
  if (ra == ra0 && dec == dec0) return x;
  const double k = (double)kArcsecToRad;
  const double d_ra = (ra - ra0) * k, n_dec = dec * k, o_dec = dec0 * k;
  const double c_d_ra = cos(d_ra), s_d_ra = sin(d_ra), c_n = cos(n_dec), s_n = sin(n_dec), c_o = cos(o_dec),
               s_o = sin(o_dec);
  if (uvx) {
    const double li0 = c_n * s_d_ra, mi0 = s_n * c_o - c_n * s_o * c_d_ra, ni0 = s_n * s_o + c_n * c_o * c_d_ra;
    x.u_term = li0 / ni0;
    x.v_term = mi0 / ni0;
  }
  if (phase) {
    x.dl = -c_n * s_d_ra;
    x.dm = -(s_n * c_o - c_n * s_o * c_d_ra);
    x.dn = 1.0 - sqrt(1.0 - x.dl * x.dl - x.dm * x.dm);
  }
  return x;
}

struct GridArgs {
  // row inputs (device)
  const vis_complex *vis;
  const vis_real *weights;
  const uint8_t *flags;
  const vis_real *uvw;
  const uint8_t *flagged_rows;
  const unsigned *field;
  const unsigned *spw;
  const unsigned *ant1;
  const unsigned *ant2;
  const size_t *time_ids;
  const vis_complex *jones_inv;  // inverted 2x2 terms [T][A][F][S][Ch][4]
  const vis_complex *jones_inv_t;  // the same terms time-innermost, [A][S][Ch][F][T][4], or null (record kernel)
  const size_t *starts;          // baseline row starts [slots + 1] or null (fixed segments)
  // per-run tables (device)
  const vis_real *wavelengths;
  const uint8_t *enabled;
  const size_t *cgi;
  const void *conv;              // real [K] or complex [P][K]
  const double *tap_sums;        // FP64 complex [P][tap_f] row sums of the kernel, or null
  const float *tap_sums_f;       // the same rounded to FP32 (the single-precision record kernel), or null
  int tap_f;
  const void *conv_t;            // kernel regrouped by tap offset [P][tap_f][W], or null
  const void *conv_w;            // support-window rows [P][tap_f][conv_w_stride], or null (see
                                 // the batched planner)
  int conv_w_stride;
  const uint8_t *facet_row_mask; // [facets][rows]: 0 leaves the row out of that facet, or null
  const FacetXform *facets;
  // outputs
  vis_complex *grid;             // slices [(f*groups + g)*NC + k][ny][nx]
  vis_complex *grid_lo;          // second word of the wide accumulation (same layout) or null
  double *norm;                  // [f][groups][NC] or null (sampling function)
  int *error;                    // sticky device error word
  // sizes and scalars
  long long nrows;
  int nchan, npol, pol0, pol1, nspw, nant, ntimes;
  int facet_base;                // facet index of launch facet 0 in the ABI facet list
  int nfacets_total;             // ABI num_facet_centres (Jones indexing)
  int groups;                    // cube channels (or sampling-function channels)
  int nx, ny, W, os, K, P;
  int W_full;                    // the ABI's full support (visibility acceptance test); 0 means W
  int mode;                      // CorrMode
  int phase, uvx;                // faceting phase rotation / planar uv transform
  int nslots, seg;               // track slots (baselines or fixed segments), segment length
  int V, GB;                     // visibilities staged per chunk, groups merged at a time
  const int *plane_lo;           // per w plane: first tap of its nonzero window (support-aware), or null
  const int4 *segments;          // persistent mode: {row_begin, row_end, channel, -} per segment, or null
  const int *work_count;         // persistent mode: number of segments of this launch (device)
  const int *segment_base;       // persistent mode: index of this launch's first segment (device)
  long long segment_capacity;    // persistent mode: entries in segments
  int *work_next;                // persistent mode: work-item counter (device, zeroed before launch)
  // persistent mode with precomputed visibility records (or null: records are computed in place)
  const void *records;           // GridRec<NC> of every work item, item (si, f) at rec_off[si] x F + f x len
  const long long *rec_off;      // per scheduled segment: records of the segments before it
  const int2 *item_range;        // per work item si x F + f: its valid records [x, y) (x >= y: none)
  long long rec_capacity;        // records the buffer holds (a segment past it is gridded in place)
  long long range_capacity;      // entries of item_range (items past it grid all their records)
  unsigned imaging_field;
  double u_scale, v_scale, gcx, gcy, wmax;
};

// Error bits written to GridArgs::error (host decodes them)
enum DeviceError {
  DEV_ERR_GRID_INDEX = 1,
  DEV_ERR_JONES_INDEX = 2,
  DEV_ERR_SINGULAR = 4,
  DEV_ERR_POL_INDEX = 8,
  DEV_ERR_WAIT_TIMEOUT = 16,  // a bounded wait for staged records ran out
  DEV_ERR_ANTENNA = 32        // an antenna pair outside baseline_count (row sort)
};

template <bool WPROJ>
struct TapT;
template <>
struct TapT<false> {
  typedef acc_real type;
};
template <>
struct TapT<true> {
  typedef cplx type;
};

// One staged visibility, prepared by the prologue (16-byte aligned header for vector loads).
template <int NC>
struct __align__(16) VisRec {
  int u0, v0, ru, rv;      // footprint corner and its residues mod W
  int g, valid, fu, fv;    // grid group, validity, tap offsets
  int plane, fu0, fv0, pad0;  // w plane; tap offsets before the support-window shift
  cplx vis[NC];            // weighted, corrected, rotated visibility
  acc_real cw[NC];         // weight x flag per correlation (normalisation)
};

// What the multiply-add loop reads of a staged visibility: a VisRec without its normalisation
// fields.  The visibility-record kernel writes one per (row, facet, channel) of a call; the
// persistent segment kernel then stages them by bulk copies (sizes a multiple of 16 bytes).
template <int NC>
struct __align__(16) GridRec {
  int u0, v0, ru, rv;      // footprint corner and its residues mod the class width
  int g, valid, fu, fv;    // grid group, validity, support-window table rows
  cplx vis[NC];            // weighted, corrected, rotated visibility
};

// 2x2 complex products on row-major [a b; c d] stored as 4 cplx
__device__ __forceinline__ void jmul(const cplx *A, const cplx *B, cplx *O) {
  cplx t0 = cmul(A[0], B[0]), t1 = cmul(A[1], B[2]);
  cplx t2 = cmul(A[0], B[1]), t3 = cmul(A[1], B[3]);
  cplx t4 = cmul(A[2], B[0]), t5 = cmul(A[3], B[2]);
  cplx t6 = cmul(A[2], B[1]), t7 = cmul(A[3], B[3]);
  O[0].re = t0.re + t1.re; O[0].im = t0.im + t1.im;
  O[1].re = t2.re + t3.re; O[1].im = t2.im + t3.im;
  O[2].re = t4.re + t5.re; O[2].im = t4.im + t5.im;
  O[3].re = t6.re + t7.re; O[3].im = t6.im + t7.im;
}

// Phase factor e^{i x} for an FP64 argument (double-precision library; the single-precision
// library evaluates sincospif on the argument reduced to turns, in choose_cells).
#if !defined(BULLSEYE_SINGLE)
__device__ __forceinline__ cplx phase_factor(double x) {
  cplx r;
  double s, c;
  sincos(x, &s, &c);
  r.re = c;
  r.im = s;
  return r;
}
#endif

// Flush one owned cell's register accumulator into the grid (cell: the grid element of correlation 0).
//
// WIDE accumulation (the 32-bit library's default): while a call grids, the 8 bytes of a cell in `grid`
// hold the FP64 real part of its value and those in `grid_lo` the FP64 imaginary part
// (kernels_misc.cuh converts).  The additions return nothing, so a thread never waits for
// one.  Recovering each FP32 addition's rounding error from the value that a returning atomic gives
// (TwoSum into the second grid) moves the same bytes at about the same rate (coalesced additions into L2:
// 3.1e11 cells a second here, 3.6e11 there; beyond L2 1.4e11 against 1.2e11), but each flush then waits a
// round trip, and the registers, queues and instructions around it cost more than the additions.
#if defined(BULLSEYE_SINGLE)
// x as FP64, on the integer pipe: the exponent rebiased by 1023 - 127, the fraction moved from 23 to 52
// bits.  (The conversion instruction runs on the FP64 pipe, at 1/64 of the FP32 rate, and bounded the class
// launches at 92 % of it.)  Denormals, infinities and NaN take the instruction, under a predicate.
__device__ __forceinline__ double to_double(float x) {
  const unsigned u = __float_as_uint(x), t = u & 0x7fffffffu;
  const int hi = (((int)u >> 3) & (int)0x8fffffff) + 0x38000000;
  double d = __hiloint2double(t ? hi : (int)u, (int)(u << 29));
  if (t - 1u < 0x007fffffu || t >= 0x7f800000u) d = (double)x;
  return d;
}
#endif

// PAIR accumulation (the 32-bit library's form for caller-owned grids that are large for the call, see
// pair_accumulation): a cell keeps its FP32 value in `grid`, and what an addition rounded off goes to `grid_lo` (TwoSum
// of the value that the returning addition gives).  It converts nothing around the call.
enum Acc { ACC_PLAIN = 0, ACC_WIDE = 1, ACC_PAIR = 2 };

// The form of a call with or without second words (FP64 accumulation needs none).
inline Acc acc_form(bool second_words) {
#if defined(BULLSEYE_SINGLE)
  return second_words ? ACC_WIDE : ACC_PLAIN;
#else
  (void)second_words;
  return ACC_PLAIN;
#endif
}

#if defined(BULLSEYE_SINGLE)
__device__ __forceinline__ float2 pair_add(const GridArgs &a, long long at, cplx x) {
  return atomicAdd(reinterpret_cast<float2 *>(a.grid + at), make_float2(x.re, x.im));
}
__device__ __forceinline__ void pair_rest(const GridArgs &a, long long at, cplx x, float2 old) {
  const float s0 = __fadd_rn(old.x, x.re), b0 = __fsub_rn(s0, old.x);
  const float s1 = __fadd_rn(old.y, x.im), b1 = __fsub_rn(s1, old.y);
  const float e0 = __fadd_rn(__fsub_rn(old.x, __fsub_rn(s0, b0)), __fsub_rn(x.re, b0));
  const float e1 = __fadd_rn(__fsub_rn(old.y, __fsub_rn(s1, b1)), __fsub_rn(x.im, b1));
  const bool r0 = e0 != 0.f && isfinite(s0), r1 = e1 != 0.f && isfinite(s1);  // (an infinity has no second word)
  if (r0 || r1) atomicAdd(reinterpret_cast<float2 *>(a.grid_lo + at), make_float2(r0 ? e0 : 0.f, r1 ? e1 : 0.f));
}
#endif

template <int NC, int ACC>
__device__ __forceinline__ void flush_cell(const GridArgs &a, long long cell, long long nxy, cplx (&acc)[NC]) {
#if defined(BULLSEYE_SINGLE)
  if (ACC != ACC_PLAIN) {
    unsigned any = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) any |= __float_as_uint(acc[k].re) | __float_as_uint(acc[k].im);
    if (!(any & 0x7fffffffu)) return;  // a zero cell: nothing to add (taps outside a plane's window are zero)
  }
  if (ACC == ACC_WIDE) {
    double *re = reinterpret_cast<double *>(a.grid) + cell, *im = reinterpret_cast<double *>(a.grid_lo) + cell;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      atomicAdd(re + k * nxy, to_double(acc[k].re));
      atomicAdd(im + k * nxy, to_double(acc[k].im));
    }
  } else if (ACC == ACC_PAIR) {
    float2 old[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) old[k] = pair_add(a, cell + k * nxy, acc[k]);
#pragma unroll
    for (int k = 0; k < NC; ++k) pair_rest(a, cell + k * nxy, acc[k], old[k]);
  } else {
#pragma unroll
    for (int k = 0; k < NC; ++k)
      atomicAdd(reinterpret_cast<float2 *>(a.grid + k * nxy + cell), make_float2(acc[k].re, acc[k].im));
  }
#else
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    atomicAdd(&a.grid[k * nxy + cell].re, acc[k].re);
    atomicAdd(&a.grid[k * nxy + cell].im, acc[k].im);
  }
#endif
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    acc[k].re = 0;
    acc[k].im = 0;
  }
}

// Per-visibility normalisation partial sums of a staged chunk (8 bytes per correlation either way).
// The single-precision library accumulates them in FP32 with Kahan compensation and widens to
// FP64 only when a partial sum leaves the CTA; the double library accumulates in FP64.
#if defined(BULLSEYE_SINGLE)
struct NormAcc {
  float s, c;
};
__device__ __forceinline__ void norm_zero(NormAcc &n) { n.s = 0.f; n.c = 0.f; }
__device__ __forceinline__ void norm_add(NormAcc &n, float x) {
  const float y = x - n.c;
  const float t = n.s + y;
  n.c = (t - n.s) - y;
  n.s = t;
}
__device__ __forceinline__ double norm_value(const NormAcc &n) { return (double)n.s - (double)n.c; }
typedef float NormTerm;
#else
typedef double NormAcc;
__device__ __forceinline__ void norm_zero(NormAcc &n) { n = 0.0; }
__device__ __forceinline__ void norm_add(NormAcc &n, double x) { n += x; }
__device__ __forceinline__ double norm_value(const NormAcc &n) { return n; }
typedef double NormTerm;
#endif
static_assert(sizeof(NormAcc) == sizeof(double), "normalisation partial sums keep the shared-memory layout");

// Per-channel constants of the prologue, recomputed only when the spw changes along a track.
struct ChanCache {
  unsigned spw = 0xffffffffu;
  double inv = 0;     // 1 / lambda
  double su = 0, sv = 0, sw = 0;  // (1 / lambda) x u_scale, v_scale, plane scale
};

// Cells, taps, w plane and phase factor of one visibility in one facet: the geometry shared by
// the gridder and its adjoint, so both select exactly the same footprint.
struct CellChoice {
  int du, dv;    // footprint corner (full support)
  int fu, fv;    // tap offsets into the plane's kernel row
  int plane;     // w plane
  bool flip;     // w < 0 with w-projection: grid the conjugate at (-u, -v)
};

// Returns false when the footprint leaves the grid or the w plane is out of range (the reference's
// acceptance test: corner >= 0 and corner + W + 2 < n, convolution_policies.h:81-83,241-243).
template <bool WPROJ>
__device__ __forceinline__ bool choose_cells(double um, double vm, double wm, const ChanCache &cc,
                                             const FacetXform &fx, bool phase, bool uvx, double u_scale,
                                             double v_scale, double plane_scale, double gcx, double gcy, int nx,
                                             int ny, int Wf, int P, int os, cplx &ph, CellChoice &out) {
  ph.re = 1;
  ph.im = 0;
#if defined(BULLSEYE_SINGLE)
  // Single-precision library: the same mathematics with fewer FP64 operations (GB300 issues FP64
  // at 1/64 of FP32).  FP64 is kept for the phase argument, reduced in turns:
  //   t = (u dl + v dm + w dn) / lambda (metres x 1/lambda),  phase = e^{2 pi i (t - rint(t))},
  // and for the pixel coordinates, scaled from metres by the per-channel constants
  // (1/lambda) x u_scale and (1/lambda) x v_scale, and the tap offsets.
  (void)u_scale;
  (void)v_scale;
  (void)plane_scale;
  if (phase) {
    const double t = (um * fx.dl + vm * fx.dm + wm * fx.dn) * cc.inv;
    const float f = (float)(t - rint(t));
    float sn, cs;
    sincospif(2.0f * f, &sn, &cs);
    ph.re = cs;
    ph.im = sn;
  }
  double u = um, v = vm;
  if (uvx) {
    u = fma(-wm, fx.u_term, um);
    v = fma(-wm, fx.v_term, vm);
  }
  u *= cc.su;
  v *= cc.sv;
  double wabs = wm;
  out.flip = WPROJ && wm < 0;
  if (out.flip) {
    u = -u; v = -v; wabs = -wm;
  }
  const double ru_ = WPROJ ? rint(u) : floor(u);
  const double rv_ = WPROJ ? rint(v) : floor(v);
  // the corner offsets nx/2 - s are integers, so round(u + gcx) = round(u) + gcx
  const double du_d = ru_ + gcx;
  const double dv_d = rv_ + gcy;
  long long plane = 0;
  if (WPROJ) {
    double pl = rint(fabs(wabs) * cc.sw);
    plane = (pl >= 0.0 && pl < (double)P) ? (long long)pl : -1;  // NaN and out of range -> dropped
  }
  if (!(du_d >= 0.0 && dv_d >= 0.0 && du_d + (Wf + 2) < (double)nx && dv_d + (Wf + 2) < (double)ny && plane >= 0 &&
        plane < P))
    return false;
  // tap offsets in FP64: an FP32 fraction moves a tap by one oversampled step about once in 1e5
  // samples, which shows in the dirty image at the 1e-5 level
  out.fu = (int)((1.0 - (u - ru_)) * (double)os);
  out.fv = (int)((1.0 - (v - rv_)) * (double)os);
#else
  // Double-precision library: the reference's operation order (parity at 1e-12 needs the same
  // cells and taps): uvw / lambda, phase, uv transform, scale, round, tap offsets.
  double u = um * cc.inv, v = vm * cc.inv, w = wm * cc.inv;
  if (phase) ph = phase_factor(6.283185307179586476925286766559 * (u * fx.dl + v * fx.dm + w * fx.dn));
  if (uvx) {
    u = u - w * fx.u_term;
    v = v - w * fx.v_term;
  }
  u *= u_scale;
  v *= v_scale;
  out.flip = WPROJ && w < 0;
  if (out.flip) {
    u = -u; v = -v; w = -w;
  }
  const double ru_ = WPROJ ? rint(u) : floor(u);
  const double rv_ = WPROJ ? rint(v) : floor(v);
  const double du_d = WPROJ ? rint(u + gcx) : floor(u + gcx);
  const double dv_d = WPROJ ? rint(v + gcy) : floor(v + gcy);
  long long plane = 0;
  if (WPROJ) {
    double pl = rint(fabs(w) * plane_scale);
    plane = (pl >= 0.0 && pl < (double)P) ? (long long)pl : -1;  // NaN and out of range -> dropped
  }
  if (!(du_d >= 0.0 && dv_d >= 0.0 && du_d + (Wf + 2) < (double)nx && dv_d + (Wf + 2) < (double)ny && plane >= 0 &&
        plane < P))
    return false;
  out.fu = (int)((1.0 - u + ru_) * (double)os);
  out.fv = (int)((1.0 - v + rv_) * (double)os);
#endif
  out.du = (int)du_d;
  out.dv = (int)dv_d;
  out.plane = (int)plane;
  return true;
}

// ------------------------------------------------------------ double-float cell choice
// Single-precision library, record kernel: the cell, tap and phase choice of choose_cells with
// pairs of floats in place of FP64 (GB300 issues FP64 at 1/64 of FP32, and the FP64 pipe bounds a
// prologue that keeps about 40 FP64 operations per visibility and facet).  A pair hi + lo
// (|lo| <= ulp(hi) / 2) carries about 48 significant bits; sums use Knuth's error-free TwoSum,
// products the FMA form of Dekker's TwoProduct (products by __fmul_rn, which is never contracted
// into an FMA).  Per facet and spw the FP64 constants are split into pairs once (DfFacet); each
// visibility then needs FP32 arithmetic only.  Roundings decide on the exact high part and use
// the low part at ties, so cells and taps agree with the FP64 choice except where the two
// computations round a value within about 1e-12 pixel of a boundary differently.
struct DF {
  float hi, lo;
};
struct DfFacet {
  DF pu, pv, pw;  // phase: dl / lambda, dm / lambda, dn / lambda (turns per metre)
  DF su, sv;      // pixels per metre: (1 / lambda) x u_scale, (1 / lambda) x v_scale
  DF ut, vt;      // planar uv transform terms
  int gcx, gcy;   // footprint-corner offsets nx/2 - s, ny/2 - s
  float osf;      // oversampling factor
};
#if defined(BULLSEYE_SINGLE)
__device__ __forceinline__ DF df_split(double x) {
  DF r;
  r.hi = (float)x;
  r.lo = (float)(x - (double)r.hi);
  return r;
}
__device__ __forceinline__ DF df_quick(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return DF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const DF s = df_two_sum(a.hi, b.hi);
  return df_quick(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ DF df_mul_f(DF a, float b) {
  const float p = __fmul_rn(a.hi, b);
  const float e = fmaf(a.lo, b, fmaf(a.hi, b, -p));
  return df_quick(p, e);
}
__device__ __forceinline__ DF df_mul(DF a, DF b) {
  const float p = __fmul_rn(a.hi, b.hi);
  const float e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p)));
  return df_quick(p, e);
}

// Round half to even, and the int of an integer-valued float, for |x| < 2^22: adding 1.5 x 2^23
// leaves unit spacing, so the sum is the rounded value and its bits count it (FP32 adds on the
// FMA pipe instead of the rounding and conversion instructions).
__device__ __forceinline__ float rint22(float x) { return __fsub_rn(__fadd_rn(x, 12582912.f), 12582912.f); }
__device__ __forceinline__ int int22(float k) { return __float_as_int(__fadd_rn(k, 12582912.f)) - 0x4B400000; }
__device__ __forceinline__ float floor22(float x) {
  const float r = rint22(x);
  return r > x ? __fsub_rn(r, 1.f) : r;
}

__device__ __forceinline__ void df_facet(const FacetXform &fx, double inv, int os, DfFacet &k) {
  k.osf = (float)os;
  k.pu = df_split(fx.dl * inv);
  k.pv = df_split(fx.dm * inv);
  k.pw = df_split(fx.dn * inv);
  k.su = df_split(inv * fx.u_scale);
  k.sv = df_split(inv * fx.v_scale);
  k.ut = df_split(fx.u_term);
  k.vt = df_split(fx.v_term);
  k.gcx = (int)fx.gcx;
  k.gcy = (int)fx.gcy;
}

// Rounds x (|x| < 2^22) to the nearest integer, halves to even like rint (round = true), or down
// like floor; d = x - r as a pair.  hi - r is exact (Sterbenz), and a low part cannot carry x past
// the next rounding boundary unless hi sits on it.
__device__ __forceinline__ void df_round(DF x, bool round, float &r, DF &d) {
  if (round) {
    r = rint22(x.hi);
    const float h = __fsub_rn(x.hi, r);
    if (h == 0.5f && x.lo > 0.f) {
      r = __fadd_rn(r, 1.f);
      d = DF{-0.5f, x.lo};
    } else if (h == -0.5f && x.lo < 0.f) {
      r = __fsub_rn(r, 1.f);
      d = DF{0.5f, x.lo};
    } else {
      d = DF{h, x.lo};
    }
  } else {
    r = floor22(x.hi);
    const float h = __fsub_rn(x.hi, r);
    if (h == 0.f && x.lo < 0.f) {
      r = __fsub_rn(r, 1.f);
      d = DF{1.f, x.lo};
    } else {
      d = DF{h, x.lo};
    }
  }
}

// trunc((1 - d) x os) for 1 - d > 0 (the tap offset), with the low part deciding at integers.
__device__ __forceinline__ int df_tap(DF d, float osf) {
  DF e = df_two_sum(1.f, -d.hi);
  e = df_quick(e.hi, __fsub_rn(e.lo, d.lo));
  e = df_mul_f(e, osf);
  float k = floor22(e.hi);
  if (e.hi == k && e.lo < 0.f) k = __fsub_rn(k, 1.f);
  return int22(k);
}

// choose_cells with the facet's pairs k and the row's w plane (computed per row in FP64: it does
// not depend on the facet; -1 when out of range).
template <bool WPROJ>
__device__ __forceinline__ bool choose_cells_df(float um, float vm, float wm, const DfFacet &k, int plane, bool phase,
                                                bool uvx, int nx, int ny, int Wf, int P, int os, cplx &ph,
                                                CellChoice &out) {
  ph.re = 1;
  ph.im = 0;
  if (phase) {
    const DF t = df_add(df_add(df_mul_f(k.pu, um), df_mul_f(k.pv, vm)), df_mul_f(k.pw, wm));
    const float r = fabsf(t.hi) < 4194304.f ? rint22(t.hi) : rintf(t.hi);
    const float f = __fadd_rn(__fsub_rn(t.hi, r), t.lo);
    float sn, cs;
    sincospif(2.0f * f, &sn, &cs);
    ph.re = cs;
    ph.im = sn;
  }
  DF u, v;
  if (uvx) {
    const DF pu = df_mul_f(k.ut, wm), pv = df_mul_f(k.vt, wm);
    u = df_mul(df_add(DF{um, 0.f}, DF{-pu.hi, -pu.lo}), k.su);
    v = df_mul(df_add(DF{vm, 0.f}, DF{-pv.hi, -pv.lo}), k.sv);
  } else {
    u = df_mul_f(k.su, um);
    v = df_mul_f(k.sv, vm);
  }
  out.flip = WPROJ && wm < 0;
  if (out.flip) {
    u = DF{-u.hi, -u.lo};
    v = DF{-v.hi, -v.lo};
  }
  // corners far off the grid (or not finite) are rejected before rounding
  if (!(fabsf(u.hi) < 4194304.f && fabsf(v.hi) < 4194304.f)) return false;
  float ru, rv;
  DF du_f, dv_f;
  df_round(u, WPROJ, ru, du_f);
  df_round(v, WPROJ, rv, dv_f);
  const int du = int22(ru) + k.gcx, dv = int22(rv) + k.gcy;
  if (!(du >= 0 && dv >= 0 && du + (Wf + 2) < nx && dv + (Wf + 2) < ny && plane >= 0 && plane < P)) return false;
  out.fu = df_tap(du_f, k.osf);
  out.fv = df_tap(dv_f, k.osf);
  out.du = du;
  out.dv = dv;
  out.plane = plane;
  return true;
}
#endif

// The facet-independent part of a visibility's prologue: one (row, channel)'s checks and inputs.
// Four consecutive values starting at a multiple of four elements (a 2x2 Jones term; a row's four
// correlations, weights or flags): vector loads when the array's base allows them (`vec`, the same
// for every thread of a launch), element loads otherwise (a caller's device array may sit at any
// element boundary).
__device__ __forceinline__ bool vec16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
__device__ __forceinline__ void load_c4(const vis_complex *p, bool vec, cplx out[4]) {
  if (vec) {
#if defined(BULLSEYE_SINGLE)
    const float4 x = __ldg(reinterpret_cast<const float4 *>(p)), y = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    out[0].re = x.x; out[0].im = x.y; out[1].re = x.z; out[1].im = x.w;
    out[2].re = y.x; out[2].im = y.y; out[3].re = y.z; out[3].im = y.w;
#else
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double2 v = __ldg(reinterpret_cast<const double2 *>(p) + k);
      out[k].re = v.x; out[k].im = v.y;
    }
#endif
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      out[k].re = p[k].re;
      out[k].im = p[k].im;
    }
  }
}
__device__ __forceinline__ void load_r4(const vis_real *p, bool vec, acc_real out[4]) {
  if (vec) {
#if defined(BULLSEYE_SINGLE)
    const float4 x = __ldg(reinterpret_cast<const float4 *>(p));
    out[0] = x.x; out[1] = x.y; out[2] = x.z; out[3] = x.w;
#else
    const double2 x = __ldg(reinterpret_cast<const double2 *>(p)), y = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    out[0] = x.x; out[1] = x.y; out[2] = y.x; out[3] = y.y;
#endif
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = (acc_real)p[k];
  }
}
__device__ __forceinline__ void load_f4(const uint8_t *p, bool vec, bool out[4]) {
  if (vec) {
    const unsigned x = __ldg(reinterpret_cast<const unsigned *>(p));
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = ((x >> (8 * k)) & 0xffu) != 0;  // little-endian byte k
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = p[k] != 0;
  }
}

template <int NC>
struct RowInputs {
  bool use;            // in range, channel enabled, spw and grid group valid, Jones indices valid
  bool row_ok;         // not flagged, in the imaging field
  unsigned spw;
  int g;               // grid group (cube channel)
  long long sc;        // spw x nchan + channel
  long long jt1, jt2;  // Jones rows t x nant + antenna; with jones_inv_t, ((antenna x S + spw) x Ch + channel) x F
  long long tt;        // the row's time index (with jones_inv_t)
  vis_real uvw_in[3];  // as stored (the double-float cell choice starts from them)
  cplx vis[NC];
  acc_real wt[NC];
  bool fl[NC];
};

template <int NC>
__device__ __forceinline__ void load_row(const GridArgs &a, int chan, long long row, bool in_range, RowInputs<NC> &ri) {
  ri.use = false;
  if (!in_range) return;
  const int c = chan;
  const unsigned spw = a.spw[row];
  if (spw >= (unsigned)a.nspw) {
    atomicOr(a.error, DEV_ERR_GRID_INDEX);
    return;
  }
  const long long sc = (long long)spw * a.nchan + c;
  if (!a.enabled[sc]) return;
  const size_t g = a.cgi[sc];
  if (g >= (size_t)a.groups) {
    atomicOr(a.error, DEV_ERR_GRID_INDEX);
    return;
  }
  ri.spw = spw;
  ri.sc = sc;
  ri.g = (int)g;
  ri.uvw_in[0] = a.uvw[3 * row];
  ri.uvw_in[1] = a.uvw[3 * row + 1];
  ri.uvw_in[2] = a.uvw[3 * row + 2];
  ri.row_ok = !a.flagged_rows[row] && (a.field[row] == a.imaging_field);
  const long long base = ((long long)row * a.nchan + c) * a.npol;
  if (a.mode == CORR_SAMPLING) {
#pragma unroll
    for (int k = 0; k < NC; ++k) { ri.vis[k].re = 1; ri.vis[k].im = 0; ri.wt[k] = 1; ri.fl[k] = false; }
  } else if constexpr (NC == 4) {
    // a row's 4 correlations start at a multiple of 4 elements when npol = 4
    const bool v4 = a.npol == 4;
    load_c4(a.vis + base, v4 && vec16(a.vis), ri.vis);
    load_r4(a.weights + base, v4 && vec16(a.weights), ri.wt);
    load_f4(a.flags + base, v4 && (reinterpret_cast<uintptr_t>(a.flags) & 3) == 0, ri.fl);
  } else {
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      int pi = (k == 0) ? a.pol0 : a.pol1;
      vis_complex vv = a.vis[base + pi];
      ri.vis[k].re = vv.re; ri.vis[k].im = vv.im;
      ri.wt[k] = (acc_real)a.weights[base + pi];
      ri.fl[k] = a.flags[base + pi] != 0;
    }
  }
  ri.jt1 = ri.jt2 = ri.tt = 0;
  if (NC == 4 && a.mode == CORR_QUAD_JONES) {
    const long long t = (long long)a.time_ids[row];
    const unsigned a1 = a.ant1[row], a2 = a.ant2[row];
    if (t < 0 || t >= a.ntimes || a1 >= (unsigned)a.nant || a2 >= (unsigned)a.nant) {
      atomicOr(a.error, DEV_ERR_JONES_INDEX);
      return;
    }
    if (a.jones_inv_t) {
      ri.jt1 = (((long long)a1 * a.nspw + spw) * a.nchan + c) * a.nfacets_total;
      ri.jt2 = (((long long)a2 * a.nspw + spw) * a.nchan + c) * a.nfacets_total;
      ri.tt = t;
    } else {
      ri.jt1 = t * a.nant + a1;
      ri.jt2 = t * a.nant + a2;
    }
  }
  ri.use = true;
}

// The facet part of the prologue: the row's Jones correction for facet f_local, weights and flags,
// cells, taps, phase rotation and flip, into rec (valid = 0 when the row is left out of the facet
// or its footprint is off the grid).  inv = 1 / lambda of the row's channel.
template <int NC, bool WPROJ>
__device__ __forceinline__ void facet_record(const GridArgs &a, int f_local, int chan, long long row,
                                             const RowInputs<NC> &ri, double inv, VisRec<NC> &rec,
                                             const double plane_scale, const DfFacet *dk = nullptr,
                                             int plane_df = -1) {
  rec.valid = 0;
  if (!ri.use) return;
  const int c = chan;
  const int fglob = a.facet_base + f_local;
  // a row left out of this facet (uneven facet layouts) is skipped like an off-grid visibility
  if (a.facet_row_mask && !a.facet_row_mask[(long long)fglob * a.nrows + row]) return;
  const FacetXform &fx = a.facets[f_local];
  cplx vis[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) vis[k] = ri.vis[k];
  if (NC == 4 && a.mode == CORR_QUAD_JONES) {
    // V <- J_p^-1 (V J_q^-H)   (correlation_gridding_policies.h:523-542; terms pre-inverted).
    // With the time-innermost copy, the 32 rows of a warp (consecutive times of one baseline and
    // channel) read one contiguous run of terms per antenna and facet.
    cplx P[4], Q[4], T[4], O[4];
    if (a.jones_inv_t) {
      const bool jv = vec16(a.jones_inv_t);
      load_c4(a.jones_inv_t + ((ri.jt1 + fglob) * a.ntimes + ri.tt) * 4, jv, P);
      load_c4(a.jones_inv_t + ((ri.jt2 + fglob) * a.ntimes + ri.tt) * 4, jv, Q);
    } else {
      const long long i1 = (((ri.jt1 * a.nfacets_total + fglob) * a.nspw + ri.spw) * a.nchan + c) * 4;
      const long long i2 = (((ri.jt2 * a.nfacets_total + fglob) * a.nspw + ri.spw) * a.nchan + c) * 4;
      const bool jv = vec16(a.jones_inv);
      load_c4(a.jones_inv + i1, jv, P);
      load_c4(a.jones_inv + i2, jv, Q);
    }
    // hermitian transpose of Q
    cplx qh[4];
    qh[0].re = Q[0].re; qh[0].im = -Q[0].im;
    qh[1].re = Q[2].re; qh[1].im = -Q[2].im;
    qh[2].re = Q[1].re; qh[2].im = -Q[1].im;
    qh[3].re = Q[3].re; qh[3].im = -Q[3].im;
    jmul(vis, qh, T);
    jmul(P, T, O);
#pragma unroll
    for (int k = 0; k < 4; ++k) vis[k] = O[k];
  }
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    bool keep = !(ri.fl[k] || !ri.row_ok);
    acc_real cw = keep ? ri.wt[k] : (acc_real)0;
    rec.cw[k] = cw;
    vis[k].re *= cw;
    vis[k].im *= cw;
  }
  CellChoice cell;
  cplx ph;
#if defined(BULLSEYE_SINGLE)
  if (dk) {
    if (!choose_cells_df<WPROJ>((float)ri.uvw_in[0], (float)ri.uvw_in[1], (float)ri.uvw_in[2], *dk, plane_df,
                                a.phase != 0, a.uvx != 0, fx.nx, fx.ny, a.W_full ? a.W_full : a.W, a.P, a.os, ph,
                                cell))
      return;
  } else
#endif
  {
    ChanCache cc;
    cc.spw = ri.spw;
    cc.inv = inv;
    cc.su = inv * fx.u_scale;
    cc.sv = inv * fx.v_scale;
    cc.sw = inv * plane_scale;
    if (!choose_cells<WPROJ>((double)ri.uvw_in[0], (double)ri.uvw_in[1], (double)ri.uvw_in[2], cc, fx, a.phase != 0, a.uvx != 0, fx.u_scale, fx.v_scale,
                             plane_scale, fx.gcx, fx.gcy, fx.nx, fx.ny, a.W_full ? a.W_full : a.W, a.P, a.os, ph, cell))
      return;
  }
  if (a.phase) {
#pragma unroll
    for (int k = 0; k < NC; ++k) vis[k] = cmul(vis[k], ph);
  }
  if (cell.flip) {
#pragma unroll
    for (int k = 0; k < NC; ++k) vis[k].im = -vis[k].im;
  }
  const long long plane = cell.plane;
  int du = cell.du, dv = cell.dv;
  rec.fu = cell.fu;
  rec.fv = cell.fv;
  rec.fu0 = cell.fu;
  rec.fv0 = cell.fv;
  int lo = 0;
  if (a.plane_lo) {
    // support-aware: grid only the plane's nonzero window of a.W taps (the taps outside it are
    // exactly zero), shifting the footprint corner and the tap offsets by the window start
    lo = a.plane_lo[plane];
    du += lo;
    dv += lo;
    rec.fu += lo * a.os;
    rec.fv += lo * a.os;
  }
  if (a.conv_w) {
    // start of the (plane, tap offset) row of the support-window table (window start included)
    rec.fu = (int)(((long long)plane * a.tap_f + cell.fu) * a.conv_w_stride);
    rec.fv = (int)(((long long)plane * a.tap_f + cell.fv) * a.conv_w_stride);
  } else if (a.conv_t) {
    // index of the first staged tap in the regrouped table
    const int Wfull = a.W_full ? a.W_full : a.W;
    rec.fu = (int)(((long long)plane * a.tap_f + cell.fu) * Wfull + lo);
    rec.fv = (int)(((long long)plane * a.tap_f + cell.fv) * Wfull + lo);
  } else {
    // index of the first tap in the ABI's table
    rec.fu += (int)(plane * a.K);
    rec.fv += (int)(plane * a.K);
  }
  rec.plane = (int)plane;
  rec.u0 = du;
  rec.v0 = dv;
  rec.ru = du % a.W;
  rec.rv = dv % a.W;
  rec.g = ri.g;
#pragma unroll
  for (int k = 0; k < NC; ++k) rec.vis[k] = vis[k];
  rec.valid = 1;
}

// One visibility's prologue in one facet, in one piece for the in-place gridder (fewer values live
// at once than load_row + facet_record, which the record kernel uses; both make the same record
// from the same arithmetic).  cc keeps the per-channel constants while the spw stays the same.
template <int NC, bool WPROJ>
__device__ __forceinline__ void prologue(const GridArgs &a, int f_local, int chan, long long row, bool in_range,
                                         VisRec<NC> &rec, ChanCache &cc, const double plane_scale) {
  rec.valid = 0;
  if (!in_range) return;
  const int c = chan;
  unsigned spw = a.spw[row];
  if (spw >= (unsigned)a.nspw) {
    atomicOr(a.error, DEV_ERR_GRID_INDEX);
    return;
  }
  long long sc = (long long)spw * a.nchan + c;
  if (!a.enabled[sc]) return;
  size_t g = a.cgi[sc];
  if (g >= (size_t)a.groups) {
    atomicOr(a.error, DEV_ERR_GRID_INDEX);
    return;
  }
  const int fglob = a.facet_base + f_local;
  // a row left out of this facet (uneven facet layouts) is skipped like an off-grid visibility
  if (a.facet_row_mask && !a.facet_row_mask[(long long)fglob * a.nrows + row]) return;
  const FacetXform &fx = a.facets[f_local];
  if (spw != cc.spw) {  // 1/lambda is constant along a track unless the spw changes
    cc.spw = spw;
    cc.inv = 1.0 / (double)a.wavelengths[sc];
    cc.su = cc.inv * fx.u_scale;
    cc.sv = cc.inv * fx.v_scale;
    cc.sw = cc.inv * plane_scale;
  }
  const double um = (double)a.uvw[3 * row], vm = (double)a.uvw[3 * row + 1], wm = (double)a.uvw[3 * row + 2];
  bool row_ok = !a.flagged_rows[row] && (a.field[row] == a.imaging_field);

  cplx vis[NC];
  acc_real wt[NC];
  bool fl[NC];
  const long long base = ((long long)row * a.nchan + c) * a.npol;
  if (a.mode == CORR_SAMPLING) {
#pragma unroll
    for (int k = 0; k < NC; ++k) { vis[k].re = 1; vis[k].im = 0; wt[k] = 1; fl[k] = false; }
  } else if (NC == 1 || NC == 2) {
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      int pi = (k == 0) ? a.pol0 : a.pol1;
      vis_complex vv = a.vis[base + pi];
      vis[k].re = vv.re; vis[k].im = vv.im;
      wt[k] = (acc_real)a.weights[base + pi];
      fl[k] = a.flags[base + pi] != 0;
    }
  } else {
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      vis_complex vv = a.vis[base + k];
      vis[k].re = vv.re; vis[k].im = vv.im;
      wt[k] = (acc_real)a.weights[base + k];
      fl[k] = a.flags[base + k] != 0;
    }
  }
  if (NC == 4 && a.mode == CORR_QUAD_JONES) {
    // V <- J_p^-1 (V J_q^-H)   (correlation_gridding_policies.h:523-542; terms pre-inverted)
    long long t = (long long)a.time_ids[row];
    unsigned a1 = a.ant1[row], a2 = a.ant2[row];
    if (t < 0 || t >= a.ntimes || a1 >= (unsigned)a.nant || a2 >= (unsigned)a.nant) {
      atomicOr(a.error, DEV_ERR_JONES_INDEX);
      return;
    }
    long long i1 = ((((t * a.nant + a1) * a.nfacets_total + fglob) * a.nspw + spw) * a.nchan + c) * 4;
    long long i2 = ((((t * a.nant + a2) * a.nfacets_total + fglob) * a.nspw + spw) * a.nchan + c) * 4;
    cplx P[4], Q[4], T[4], O[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      vis_complex p = a.jones_inv[i1 + k], q = a.jones_inv[i2 + k];
      P[k].re = p.re; P[k].im = p.im;
      Q[k].re = q.re; Q[k].im = q.im;
    }
    // hermitian transpose of Q
    cplx qh[4];
    qh[0].re = Q[0].re; qh[0].im = -Q[0].im;
    qh[1].re = Q[2].re; qh[1].im = -Q[2].im;
    qh[2].re = Q[1].re; qh[2].im = -Q[1].im;
    qh[3].re = Q[3].re; qh[3].im = -Q[3].im;
    jmul(vis, qh, T);
    jmul(P, T, O);
#pragma unroll
    for (int k = 0; k < 4; ++k) vis[k] = O[k];
  }
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    bool keep = !(fl[k] || !row_ok);
    acc_real cw = keep ? wt[k] : (acc_real)0;
    rec.cw[k] = cw;
    vis[k].re *= cw;
    vis[k].im *= cw;
  }
  CellChoice cell;
  cplx ph;
  if (!choose_cells<WPROJ>(um, vm, wm, cc, fx, a.phase != 0, a.uvx != 0, fx.u_scale, fx.v_scale, plane_scale, fx.gcx,
                           fx.gcy, fx.nx, fx.ny, a.W_full ? a.W_full : a.W, a.P, a.os, ph, cell))
    return;
  if (a.phase) {
#pragma unroll
    for (int k = 0; k < NC; ++k) vis[k] = cmul(vis[k], ph);
  }
  if (cell.flip) {
#pragma unroll
    for (int k = 0; k < NC; ++k) vis[k].im = -vis[k].im;
  }
  const long long plane = cell.plane;
  int du = cell.du, dv = cell.dv;
  rec.fu = cell.fu;
  rec.fv = cell.fv;
  rec.fu0 = cell.fu;
  rec.fv0 = cell.fv;
  int lo = 0;
  if (a.plane_lo) {
    // support-aware: grid only the plane's nonzero window of a.W taps (the taps outside it are
    // exactly zero), shifting the footprint corner and the tap offsets by the window start
    lo = a.plane_lo[plane];
    du += lo;
    dv += lo;
    rec.fu += lo * a.os;
    rec.fv += lo * a.os;
  }
  if (a.conv_w) {
    // start of the (plane, tap offset) row of the support-window table (window start included)
    rec.fu = (int)(((long long)plane * a.tap_f + cell.fu) * a.conv_w_stride);
    rec.fv = (int)(((long long)plane * a.tap_f + cell.fv) * a.conv_w_stride);
  } else if (a.conv_t) {
    // index of the first staged tap in the regrouped table
    const int Wfull = a.W_full ? a.W_full : a.W;
    rec.fu = (int)(((long long)plane * a.tap_f + cell.fu) * Wfull + lo);
    rec.fv = (int)(((long long)plane * a.tap_f + cell.fv) * Wfull + lo);
  } else {
    // index of the first tap in the ABI's table
    rec.fu += (int)(plane * a.K);
    rec.fv += (int)(plane * a.K);
  }
  rec.plane = (int)plane;
  rec.u0 = du;
  rec.v0 = dv;
  rec.ru = du % a.W;
  rec.rv = dv % a.W;
  rec.g = (int)g;
#pragma unroll
  for (int k = 0; k < NC; ++k) rec.vis[k] = vis[k];
  rec.valid = 1;
}

// ------------------------------------------------------------------ merged gridding of staged chunks
//
// Taps are products: footprint cell (u, v) of a visibility gets vis x ku(u) x kv(v).  Consecutive
// visibilities of a track sit a fraction of an oversampling step apart, so a stretch of them often
// shares the footprint corner and one of the two tap rows.  Such a *group* is summed along the other
// axis first; with a common ku,
//     T(v) = sum over the group of vis x kv(v)            (W multiply-adds per visibility)
//     cell(u, v) += ku(u) x T(v)                            (W^2 multiply-adds per group, not per visibility)
// which is the same sum with its common factor taken out (and the other way round with a common kv).
// On Earth-rotation tracks sampled every 14 s (27 EVLA antennas, 1024-cell grids 1.4 degrees wide,
// oversampling 15) groups hold 4.6 visibilities on average when each work item merges along the axis on
// which its track moves more in tap steps; fixed to one axis they hold 2.3 (v) or 3.9 (u), and merging
// only identical footprints gives 1.9.
//
// An item's axes are (a, b): b is the merge axis, (a, b) = (u, v) or (v, u).  A warp's lanes own columns
// along a, a thread's J rows run along b, so that the frequent moves (along b) flush one row of a strip
// with all its lanes.  A chunk of V records in shared memory is taken in two steps, in batches of GB groups:
//   merge_groups  thread (i, part) forms T(i) of every nparts-th group of the batch, reading the taps
//                 from the kernel table through L1, and copies the group's common tap row;
//   grid_groups   the Romein owner threads add their column's tap x T(row) to their J cells.
//
// What the merge and the split of the builds measured (GB300, 27 antennas x 100 times x 64 channels,
// 16 facets, whole batched call with copy-back): 36.0 -> 27.2 ms in single precision; 64-bit library,
// 40 times x 16 channels x 4 facets: 27.3 -> 7.7 ms (its FP64 pipe bounded the multiply-adds).

// Most records of a chunk: group lists are built from 64-bit masks.
constexpr int kMaxChunk = 64;

// Merged values are stored as 16-byte vectors [group][NC / N][column], so that a warp's columns read
// consecutive 16-byte words (no bank conflicts).
template <int NC>
struct MergeVec {
  static constexpr int N = NC * sizeof(cplx) >= 16 ? (int)(16 / sizeof(cplx)) : NC;
  static constexpr int H = NC / N;
  struct __align__(N * sizeof(cplx)) type {
    cplx v[N];
  };
};

// Bytes before the merged values, rounded up to 16: computed in place, V staged records and their
// normalisation state (partial sums, grid group); from precomputed records, two buffers of V GridRecs
// (one filled while the other is gridded).  A launch reserves the larger, so each work item may take
// either form.
template <int NC>
__host__ __device__ inline size_t stage_head_bytes(int V) {
  const size_t own = sizeof(VisRec<NC>) + sizeof(NormAcc) * NC + sizeof(int);
  const size_t pre = 2 * sizeof(GridRec<NC>);
  return ((own > pre ? own : pre) * (size_t)V + 15) / 16 * 16;
}
// Merged values (W + J - 1: the first J - 1 are repeated after the last, so that a thread's J consecutive
// owned rows read consecutive entries without a wrap) and the common tap row of one group.
template <int NC, bool WPROJ>
__host__ __device__ inline size_t merge_group_bytes(int W, int J) {
  return sizeof(cplx) * NC * (size_t)(W + J - 1) + sizeof(typename TapT<WPROJ>::type) * (size_t)W;
}
// Per warp: the group list, and one column's values (flush_column).
template <int NC>
__host__ __device__ inline size_t warp_scratch_bytes(int J) {
  return kMaxChunk * sizeof(unsigned short) + sizeof(cplx) * NC * (size_t)J;
}

// Staged records V, groups per batch GB and dynamic shared memory of a launch.
struct ChunkShape {
  int V, GB;
  size_t smem;
};

// The chunk shape for CTAs of nthreads with regs registers per thread: as many CTAs per SM as the
// register file allows within 195 KB (the next split between shared memory and L1 is 196 KB, which
// leaves 60 KB to the kernel table; 199 KB and the 28 KB of the last split cost 1 % of a batched call of 27
// antennas x 400 times x 64 channels, and 163 KB with shorter batches 6 % of a 64-antenna snapshot step),
// fewer when a batch of six groups does not fit.  64 records per chunk where they take at most half of the CTA's share (a
// chunk's end also ends a group), 32 otherwise.
constexpr size_t kStaticSmem = 640;  // at most, of the segment kernel
template <int NC, bool WPROJ>
__host__ inline ChunkShape chunk_shape(int W, int nthreads, int J, int regs = 128) {
  const int nwarps = (nthreads + 31) / 32;
  const size_t fixed = warp_scratch_bytes<NC>(J) * nwarps + 64;
  const size_t per = merge_group_bytes<NC, WPROJ>(W, J);
  ChunkShape s{32, 1, 0};
  for (int ctas = std::max(1, std::min(24, 65536 / (nthreads * regs)));; --ctas) {
    const size_t budget = std::min<size_t>(200 * 1024, (size_t)195 * 1024 / ctas - 1024 - kStaticSmem);
    for (int V : {64, 32}) {
      const size_t head = stage_head_bytes<NC>(V) + fixed;
      if (V > 32 && 2 * head > budget) continue;
      const int gb = budget > head ? (int)std::min<size_t>((size_t)V, (budget - head) / per) : 0;
      if (gb >= 6 || ctas == 1) {
        s.V = V;
        s.GB = std::max(1, gb);
        s.smem = head + per * s.GB;
        return s;
      }
    }
  }
}

// premultiplied visibility times the column tap
__device__ __forceinline__ void mac(cplx &acc, cplx a, acc_real t) {
  acc.re = fma(a.re, t, acc.re);
  acc.im = fma(a.im, t, acc.im);
}
__device__ __forceinline__ void mac(cplx &acc, cplx a, cplx t) {
  acc.re = fma(a.re, t.re, acc.re);
  acc.re = fma(-a.im, t.im, acc.re);
  acc.im = fma(a.re, t.im, acc.im);
  acc.im = fma(a.im, t.re, acc.im);
}

// Thread -> owned (column, strip) map.  WIDE pads the columns to a multiple of 32 so that every
// warp covers one strip: the row taps it reads are then warp-uniform (shared-memory broadcast).
template <bool WIDE>
__device__ __forceinline__ void owner_map(int tid, int W, int J, int &du, int &strip, bool &owner) {
  const int nstrips = (W + J - 1) / J;
  if (WIDE) {
    const int wpr = (W + 31) >> 5;  // warps per strip
    const int warp = tid >> 5, lane = tid & 31;
    du = (warp % wpr) * 32 + lane;
    strip = warp / wpr;
    owner = du < W && strip < nstrips;
  } else {
    du = tid % W;
    strip = tid / W;
    owner = strip < nstrips;
  }
}

// Register state of a Romein owner thread: the accumulators of its J cells and the footprint they
// belong to.  For the last footprint corner (pa0, pb0) the owned cells are
// (pa0 + oa, pb0 + wrap(ob0 + j)), wrap(i) = i - W when i >= W.
template <int NC, int J>
struct OwnerState {
  cplx acc[J][NC];
  unsigned dirty;
  int cg, pa0, pb0, oa, ob0;
};

template <int NC, int J>
__device__ __forceinline__ void owner_reset(OwnerState<NC, J> &st) {
#pragma unroll
  for (int j = 0; j < J; ++j) {
#pragma unroll
    for (int k = 0; k < NC; ++k) { st.acc[j][k].re = 0; st.acc[j][k].im = 0; }
  }
  st.dirty = 0;
  st.cg = -1;
  st.pa0 = -1;
  st.pb0 = -1;
  st.oa = 0;
  st.ob0 = 0;
}

// Prologue of one staging slot: the visibility of `row` staged into recs[slot].
template <int NC, bool WPROJ>
__device__ __forceinline__ void stage_slot(const GridArgs &a, int f_local, int chan, long long row, bool in_range,
                                           int slot, VisRec<NC> *recs, ChanCache &cc, double plane_scale) {
  VisRec<NC> rec;
  prologue<NC, WPROJ>(a, f_local, chan, row, in_range, rec, cc, plane_scale);
  recs[slot] = rec;
}

// Normalisation term of a staged visibility from the precomputed kernel row sums, added to its
// slot's running sums (which go to the global normalisation when the slot's grid group changes).
template <int NC>
__device__ __forceinline__ void norm_slot(const GridArgs &a, const VisRec<NC> &rec, int slot, NormAcc *s_nacc,
                                          int *s_ng, long long fslice) {
  if (!rec.valid) return;
  const double *su = a.tap_sums + 2 * ((long long)rec.plane * a.tap_f + rec.fu0);
  const double *sv = a.tap_sums + 2 * ((long long)rec.plane * a.tap_f + rec.fv0);
  const NormTerm nt = (NormTerm)(su[0] * sv[0] - su[1] * sv[1]);
  NormAcc *na = s_nacc + slot * NC;
  if (s_ng[slot] != rec.g) {
    if (s_ng[slot] >= 0) {
#pragma unroll
      for (int k = 0; k < NC; ++k)
        if (norm_value(na[k]) != 0.0) atomicAdd(&a.norm[(fslice + s_ng[slot]) * NC + k], norm_value(na[k]));
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) norm_zero(na[k]);
    s_ng[slot] = rec.g;
  }
#pragma unroll
  for (int k = 0; k < NC; ++k) norm_add(na[k], (NormTerm)rec.cw[k] * nt);
}

// The kernel table that a staged record's fu and fv index: the support-window table or the table
// regrouped by tap offset (taps of a row adjacent), or the ABI's own (taps os elements apart).  The
// table is read one tap per lane, a row's taps by consecutive lanes.  A caller-owned ABI table may
// start at any element part: it is read in parts then.
template <bool WPROJ>
struct TapTable {
  const void *p;
  int step;
  bool whole;
};
template <bool WPROJ>
__device__ __forceinline__ TapTable<WPROJ> tap_table(const GridArgs &a) {
  TapTable<WPROJ> t;
  t.p = a.conv_w ? a.conv_w : a.conv_t ? a.conv_t : a.conv;
  t.step = a.conv_w || a.conv_t ? 1 : a.os;
  t.whole = (reinterpret_cast<uintptr_t>(t.p) & (sizeof(typename TapT<WPROJ>::type) - 1)) == 0;
  return t;
}
__device__ __forceinline__ acc_real read_tap(const TapTable<false> &t, int first, int j) {
  return __ldg(reinterpret_cast<const acc_real *>(t.p) + first + j * t.step);
}
__device__ __forceinline__ cplx read_tap(const TapTable<true> &t, int first, int j) {
  const int at = first + j * t.step;
  cplx r;
  if (t.whole) {
#if defined(BULLSEYE_SINGLE)
    const float2 v = __ldg(reinterpret_cast<const float2 *>(t.p) + at);
#else
    const double2 v = __ldg(reinterpret_cast<const double2 *>(t.p) + at);
#endif
    r.re = v.x;
    r.im = v.y;
  } else {
    r.re = __ldg(reinterpret_cast<const acc_real *>(t.p) + 2 * (long long)at);
    r.im = __ldg(reinterpret_cast<const acc_real *>(t.p) + 2 * (long long)at + 1);
  }
  return r;
}

// Barriers of the record staging.  Waits are bounded.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long *bar) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_arrive_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// Non-blocking test of the phase of the given parity.
__device__ __forceinline__ bool bar_test(unsigned long long *bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait for the phase of the given parity (polls, then polls with short sleeps: about 0.2 s
// at most); false when the bound ran out.
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity) {
  for (int i = 0; i < (1 << 22); ++i) {
    if (bar_test(bar, parity)) return true;
    if (i >= 64) __nanosleep(32);
  }
  return false;
}
// Orders this thread's earlier shared-memory accesses (and those a CTA barrier published to it)
// before its following bulk copies into shared memory.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// One bulk (TMA) copy global -> shared of `bytes` (16-byte aligned addresses, a multiple of 16
// bytes) that completes its bytes on the barrier.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Normalisation without precomputed row sums (the allocation-free entries), four lanes per staged
// visibility: Re(sum_u k_u * sum_v k_v) x weight x flag (loop bounds are warp-uniform so the
// shuffles always see full warps); lane 4i owns the running sums of staged slot i.
template <int NC, bool WPROJ>
__device__ __forceinline__ void norm_from_taps(const GridArgs &a, const VisRec<NC> *recs, int nv,
                                               const TapTable<WPROJ> &table, NormAcc *s_nacc, int *s_ng,
                                               long long fslice) {
  const int W = a.W;
  const int tid = threadIdx.x;
  for (int b4 = tid & ~31; b4 < 4 * nv; b4 += blockDim.x) {
    const int q = b4 + (tid & 31);
    const int vi = q >> 2, part = q & 3;
    const bool act = vi < nv && recs[vi].valid;
    // tap sums in the library's working precision (FP64 units are scarce on this GPU)
    acc_real sur = 0, sui = 0, svr = 0, svi = 0;
    if (act) {
      const int fu = recs[vi].fu, fv = recs[vi].fv;
      for (int j = part; j < W; j += 4) {
        const typename TapT<WPROJ>::type u = read_tap(table, fu, j), v = read_tap(table, fv, j);
        if constexpr (WPROJ) {
          sur += u.re; sui += u.im; svr += v.re; svi += v.im;
        } else {
          sur += u; svr += v;
        }
      }
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
      sur += __shfl_xor_sync(0xffffffffu, sur, off);
      sui += __shfl_xor_sync(0xffffffffu, sui, off);
      svr += __shfl_xor_sync(0xffffffffu, svr, off);
      svi += __shfl_xor_sync(0xffffffffu, svi, off);
    }
    if (act && part == 0) {
      const VisRec<NC> &r = recs[vi];
      const NormTerm nt = (NormTerm)sur * (NormTerm)svr - (NormTerm)sui * (NormTerm)svi;
      NormAcc *na = s_nacc + vi * NC;
      if (s_ng[vi] != r.g) {
        if (s_ng[vi] >= 0) {
#pragma unroll
          for (int k = 0; k < NC; ++k)
            if (norm_value(na[k]) != 0.0) atomicAdd(&a.norm[(fslice + s_ng[vi]) * NC + k], norm_value(na[k]));
        }
#pragma unroll
        for (int k = 0; k < NC; ++k) norm_zero(na[k]);
        s_ng[vi] = r.g;
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) norm_add(na[k], (NormTerm)r.cw[k] * nt);
    }
  }
}

// Group starts among slots [32 b, 32 b + 32) of a chunk, merging along u (a group shares its v tap row)
// and along v, the first slots of runs (one footprint corner and grid group) and the valid slots, as
// warp masks (whole-warp call).
struct SlotMasks {
  unsigned valid, run, along_u, along_v;
};
template <class Rec>
__device__ __forceinline__ SlotMasks slot_masks(const Rec *recs, int nv, int b) {
  const int t = b * 32 + (threadIdx.x & 31);
  bool valid = false, run = false, au = false, av = false;
  if (t < nv) {
    const int4 c0 = *reinterpret_cast<const int4 *>(&recs[t].u0);
    const int4 c1 = *reinterpret_cast<const int4 *>(&recs[t].g);
    valid = c1.y != 0;
    run = valid;
    if (valid && t > 0) {
      const int4 p0 = *reinterpret_cast<const int4 *>(&recs[t - 1].u0);
      const int4 p1 = *reinterpret_cast<const int4 *>(&recs[t - 1].g);
      run = !p1.y || p0.x != c0.x || p0.y != c0.y || p1.x != c1.x;
      au = p1.w != c1.w;
      av = p1.z != c1.z;
    }
    au = valid && (au || run);
    av = valid && (av || run);
  }
  SlotMasks m;
  m.valid = __ballot_sync(0xffffffffu, valid);
  m.run = __ballot_sync(0xffffffffu, run);
  m.along_u = __ballot_sync(0xffffffffu, au);
  m.along_v = __ballot_sync(0xffffffffu, av);
  return m;
}

// A group list entry: first slot (7 bits), visibilities (7 bits), whether a run starts there.
constexpr int kGroupRun = 1 << 14;

// The groups of a staged chunk, written by the calling warp (whole-warp call; any warp finds the same
// groups).  `pick` first decides the item's merge axis from this chunk: the one that leaves fewer groups.
template <class Rec>
__device__ __forceinline__ int find_groups(const Rec *recs, int nv, bool pick, bool &along_v, unsigned short *list) {
  typedef unsigned long long u64;
  const SlotMasks m0 = slot_masks(recs, nv, 0);
  SlotMasks m1{0, 0, 0, 0};
  if (nv > 32) m1 = slot_masks(recs, nv, 1);
  if (pick) along_v = __popc(m0.along_v) + __popc(m1.along_v) < __popc(m0.along_u) + __popc(m1.along_u);
  const u64 start = along_v ? (u64)m1.along_v << 32 | m0.along_v : (u64)m1.along_u << 32 | m0.along_u;
  const u64 run = (u64)m1.run << 32 | m0.run;
  const u64 edge = start | ~((u64)m1.valid << 32 | m0.valid);  // slots that do not continue a group
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = lane + 32 * h;
    if (start >> t & 1) {
      const u64 rest = t < 63 ? edge >> (t + 1) : 0;
      const int len = rest ? __ffsll(rest) : 64 - t;
      list[__popcll(start & ((1ull << t) - 1))] = (unsigned short)(t | len << 7 | ((run >> t & 1) ? kGroupRun : 0));
    }
  }
  __syncwarp();
  return __popcll(start);
}

// T and the common tap row of groups [g0, g1) of a chunk: thread (entry i, part of nparts).
template <int NC, bool WPROJ, class Rec>
__device__ __forceinline__ void merge_groups(const TapTable<WPROJ> &table, const Rec *recs, const unsigned short *list,
                                             int g0, int g1, bool along_v, int W, int J, int i, int part, int nparts,
                                             typename MergeVec<NC>::type *T, typename TapT<WPROJ>::type *tb) {
  typedef typename TapT<WPROJ>::type tap_t;
  typedef MergeVec<NC> M;
  if (part >= nparts) return;
  const int S = W + J - 1;
  for (int gi = g0 + part; gi < g1; gi += nparts) {
    const int e = list[gi], s = e & 127, end = s + ((e >> 7) & 127);
    const tap_t ka0 = read_tap(table, along_v ? recs[s].fu : recs[s].fv, i);
    cplx t[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) { t[k].re = 0; t[k].im = 0; }
    // four table loads in flight (past the end: the last one again)
    for (int v = s; v < end; v += 4) {
      tap_t kb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = min(v + q, end - 1);
        kb[q] = read_tap(table, along_v ? recs[r].fv : recs[r].fu, i);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v + q < end) {
          const typename M::type *x = reinterpret_cast<const typename M::type *>(recs[v + q].vis);
#pragma unroll
          for (int h = 0; h < M::H; ++h) {
            const typename M::type y = x[h];
#pragma unroll
            for (int n = 0; n < M::N; ++n) mac(t[h * M::N + n], y.v[n], kb[q]);
          }
        }
    }
    typename M::type *Tg = T + (gi - g0) * M::H * S;
#pragma unroll
    for (int h = 0; h < M::H; ++h) {
      typename M::type y;
#pragma unroll
      for (int n = 0; n < M::N; ++n) y.v[n] = t[h * M::N + n];
      for (int j = i; j < S; j += W) Tg[h * S + j] = y;
    }
    tb[(gi - g0) * W + i] = ka0;
  }
}

// Adds one real component (part 0 real, 1 imaginary) of correlation k of a cell.
template <int ACC>
__device__ __forceinline__ void add_component(const GridArgs &a, long long at, int part, acc_real x) {
#if defined(BULLSEYE_SINGLE)
  if (ACC == ACC_WIDE)
    atomicAdd(reinterpret_cast<double *>(part ? a.grid_lo : a.grid) + at, to_double(x));
  else
    atomicAdd(reinterpret_cast<float *>(a.grid + at) + part, x);
#else
  atomicAdd(reinterpret_cast<double *>(a.grid + at) + part, x);
#endif
}

// Flushes the J cells of lane l of the calling warp (whole-warp call): the lane puts them in shared
// memory and the warp's lanes add one component each.  By itself the lane would add its 2 NC J components
// one after the other while the warp waits, which took a third of the class launches.  cell0: the grid
// element of correlation 0 at row coordinate 0 of the lane's column.
template <int NC, int J, int ACC>
__device__ __forceinline__ void flush_column(const GridArgs &a, int l, int W, long long cell0, long long nxy, int sb,
                                             cplx *buf, OwnerState<NC, J> &st) {
  const int lane = threadIdx.x & 31;
  const unsigned dirty = __shfl_sync(0xffffffffu, st.dirty, l);
  const int ob0 = __shfl_sync(0xffffffffu, st.ob0, l);
  cell0 = __shfl_sync(0xffffffffu, cell0, l);
  if (lane == l) {
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        buf[j * NC + k] = st.acc[j][k];
        st.acc[j][k].re = 0;
        st.acc[j][k].im = 0;
      }
    st.dirty = 0;
  }
  __syncwarp();
#if defined(BULLSEYE_SINGLE)
  if constexpr (ACC == ACC_PAIR) {  // whole cells: both components come back with one addition
#pragma unroll
    for (int c0 = 0; c0 < J * NC; c0 += 32) {
      const int c = c0 + lane, j = c / NC, k = c % NC;
      if (c < J * NC && (dirty >> j & 1)) {
        const cplx x = buf[c];
        const int ob = ob0 + j >= W ? ob0 + j - W : ob0 + j;
        const long long at = cell0 + (long long)(st.pb0 + ob) * sb + k * nxy;
        if (x.re != 0.f || x.im != 0.f) pair_rest(a, at, x, pair_add(a, at, x));
      }
    }
    __syncwarp();
    return;
  }
#endif
#pragma unroll
  for (int c0 = 0; c0 < J * NC * 2; c0 += 32) {
    const int c = c0 + lane, j = c / (2 * NC), k = (c >> 1) % NC;
    if (c < J * NC * 2 && (dirty >> j & 1)) {
      const int ob = ob0 + j >= W ? ob0 + j - W : ob0 + j;
      add_component<ACC>(a, cell0 + (long long)(st.pb0 + ob) * sb + k * nxy, c & 1,
                          reinterpret_cast<const acc_real *>(buf)[c]);
    }
  }
  __syncwarp();
}

// Multiply-adds of groups [g0, g1) of a chunk into an owner thread's cells (whole-warp call).  When the
// footprint moves, the owned cells are recomputed and those that changed are flushed: rows that moved by
// every lane of their strip, one or two columns that moved by flush_column.  Cells lie sa (along a) and
// sb (along b) elements apart.
template <int NC, bool WPROJ, int J, int ACC, class Rec>
__device__ __forceinline__ void grid_groups(const GridArgs &a, const Rec *recs, const unsigned short *list, int g0, int g1,
                                            bool along_v, const typename MergeVec<NC>::type *T,
                                            const typename TapT<WPROJ>::type *tb, int du, int strip, unsigned rows_mask,
                                            long long fbase, long long nxy, int gnx, cplx *col_buf,
                                            OwnerState<NC, J> &st) {
  typedef typename TapT<WPROJ>::type tap_t;
  typedef MergeVec<NC> M;
  const int W = a.W, S = W + J - 1;
  for (int gi = g0; gi < g1; ++gi) {
    const int e = list[gi];
    if (e & kGroupRun) {
      const int rs = e & 127;
      const int4 h = *reinterpret_cast<const int4 *>(&recs[rs].u0);
      const int g = recs[rs].g;
      const int a0 = along_v ? h.x : h.y, b0 = along_v ? h.y : h.x;
      if (a0 != st.pa0 || b0 != st.pb0 || g != st.cg) {
        const int sa = along_v ? 1 : gnx, sb = along_v ? gnx : 1;
        int o = du - (along_v ? h.z : h.w);
        o += (o < 0) ? W : 0;
        int nob0 = strip * J - (along_v ? h.w : h.z);
        nob0 += (nob0 < 0) ? W : 0;
        const long long cell0 = fbase + (long long)st.cg * NC * nxy + (long long)(st.pa0 + st.oa) * sa;
        bool out = st.dirty && (a0 + o != st.pa0 + st.oa || g != st.cg);  // the column moved
        const unsigned m = __ballot_sync(0xffffffffu, out);
        if (m && __popc(m) <= 2) {
          flush_column<NC, J, ACC>(a, __ffs(m) - 1, W, cell0, nxy, sb, col_buf, st);
          if (m & (m - 1)) flush_column<NC, J, ACC>(a, 31 - __clz(m), W, cell0, nxy, sb, col_buf, st);
        }
        if (st.dirty) {
#pragma unroll
          for (int j = 0; j < J; ++j) {
            const int ob = st.ob0 + j >= W ? st.ob0 + j - W : st.ob0 + j;
            const int nb = nob0 + j >= W ? nob0 + j - W : nob0 + j;
            if ((st.dirty & (1u << j)) && (out || b0 + nb != st.pb0 + ob)) {
              flush_cell<NC, ACC>(a, cell0 + (long long)(st.pb0 + ob) * sb, nxy, st.acc[j]);
              st.dirty &= ~(1u << j);
            }
          }
        }
        st.cg = g;
        // columns beyond W (padding lanes) read in-bounds values and are never flushed
        st.oa = o < W ? o : W - 1;
        st.ob0 = nob0 < W ? nob0 : 0;  // lanes past the last strip own nothing: keep their reads in bounds
        st.pa0 = a0;
        st.pb0 = b0;
      }
    }
    // branch-free multiply-adds over the J owned rows (offsets modulo W; rows of non-owning lanes stay
    // in bounds and are never flushed)
    const typename M::type *Tg = T + (gi - g0) * M::H * S + st.ob0;
    const tap_t k = tb[(gi - g0) * W + st.oa];
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
      for (int h = 0; h < M::H; ++h) {
        const typename M::type y = Tg[h * S + j];
#pragma unroll
        for (int n = 0; n < M::N; ++n) mac(st.acc[j][h * M::N + n], y.v[n], k);
      }
    st.dirty |= rows_mask;
  }
}

// What a CTA keeps for one work item: its shared-memory pieces, owner mapping and facet geometry.
template <int NC, bool WPROJ>
struct ItemSetup {
  typename MergeVec<NC>::type *T;        // [GB][H][W + J - 1]
  typename TapT<WPROJ>::type *tb;        // [GB][W]
  unsigned short *list;                  // this warp's group list
  cplx *col_buf;                         // this warp's column buffer [J][NC]
  TapTable<WPROJ> table;
  int du, strip, ax, ap, nparts, gnx;
  unsigned rows_mask;
  bool grids;
  long long nxy, fbase;
};
template <int NC, bool WPROJ, int J, int ACC, bool WIDE>
__device__ __forceinline__ void item_setup(const GridArgs &a, int f_local, unsigned char *smem, ItemSetup<NC, WPROJ> &s) {
  typedef typename MergeVec<NC>::type vec_t;
  typedef typename TapT<WPROJ>::type tap_t;
  const int W = a.W, GB = a.GB, tid = threadIdx.x;
  const int warp_id = tid >> 5;
  unsigned char *p = smem + stage_head_bytes<NC>(a.V);
  s.T = reinterpret_cast<vec_t *>(p);
  p += sizeof(cplx) * NC * (size_t)(W + J - 1) * GB;
  s.tb = reinterpret_cast<tap_t *>(p);
  p += sizeof(tap_t) * (size_t)W * GB;
  p = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
  p += warp_scratch_bytes<NC>(J) * warp_id;
  s.col_buf = reinterpret_cast<cplx *>(p);
  s.list = reinterpret_cast<unsigned short *>(s.col_buf + J * NC);
  s.table = tap_table<WPROJ>(a);
  bool owner;
  owner_map<WIDE>(tid, W, J, s.du, s.strip, owner);
  s.rows_mask = 0;
#pragma unroll
  for (int j = 0; j < J; ++j)
    if (s.strip * J + j < W) s.rows_mask |= 1u << j;
  if (!owner) s.rows_mask = 0;
  s.grids = __any_sync(0xffffffffu, s.rows_mask != 0);
  s.ap = tid / W;
  s.ax = tid - s.ap * W;
  s.nparts = (int)blockDim.x / W;
  const FacetXform &fx = a.facets[f_local];
  s.gnx = fx.nx;
  s.nxy = (long long)fx.nx * fx.ny;
  s.fbase = fx.grid_base;  // element offset of this facet's grid block
}

// The ng groups of one staged chunk (block-wide call; ends with the CTA's barrier, after which the
// records may be overwritten).  Before that barrier, next() prepares what follows the chunk.
template <int NC, bool WPROJ, int J, int ACC, class Rec, class Next>
__device__ __forceinline__ void grid_chunk(const GridArgs &a, const Rec *recs, const unsigned short *list, int ng,
                                           bool along_v, const ItemSetup<NC, WPROJ> &s, OwnerState<NC, J> &st, Next next) {
  int g0 = 0;
  do {
    const int g1 = min(ng, g0 + a.GB);
    merge_groups<NC, WPROJ>(s.table, recs, list, g0, g1, along_v, a.W, J, s.ax, s.ap, s.nparts, s.T, s.tb);
    __syncthreads();
    if (s.grids)
      grid_groups<NC, WPROJ, J, ACC>(a, recs, list, g0, g1, along_v, s.T, s.tb, s.du, s.strip, s.rows_mask, s.fbase,
                                      s.nxy, s.gnx, s.col_buf, st);
    if (g1 == ng) next();
    __syncthreads();
    g0 = g1;
  } while (g0 < ng);
}

// End of a work item (or of a stretch of its rows): the owned cells are flushed and start at zero again.
template <int NC, bool WPROJ, int J, int ACC>
__device__ __forceinline__ void item_flush(const GridArgs &a, const ItemSetup<NC, WPROJ> &s, bool along_v,
                                           OwnerState<NC, J> &st) {
  if (!st.dirty) return;
  const int sa = along_v ? 1 : s.gnx, sb = along_v ? s.gnx : 1;
  const long long cell0 = s.fbase + (long long)st.cg * NC * s.nxy + (long long)(st.pa0 + st.oa) * sa;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int ob = st.ob0 + j >= a.W ? st.ob0 + j - a.W : st.ob0 + j;
    if (st.dirty & (1u << j)) flush_cell<NC, ACC>(a, cell0 + (long long)(st.pb0 + ob) * sb, s.nxy, st.acc[j]);
  }
  st.dirty = 0;
}

// How long the owned cells of an item may stay in registers, over segments: cells of slow tracks never leave the
// footprint, and plain accumulation over ever more channels would lose what the flushes hold.  `segs`
// segments with `rows` rows in `groups` merged groups are in; one more may follow while that makes four at most, no
// more than the visibilities per group (each group is one addition to a cell, so that a cell takes no more
// additions than it has visibilities in one segment), and one per 30 rows of a segment (short segments end
// their groups early).  The bar is the error against 64 bits of a segment gridded visibility by visibility and
// flushed without loss at its end.  Parts of it with 1, 2, 3 and 4 segments in every stay: 100 rows of 14 s 0.51 0.63 0.69
// 0.80, 200 rows 0.42 0.53 0.63 0.72; 16 rows 0.87 1.00 1.09 1.14; 100 fast rows (0.8 degrees each, groups of one or two)
// 0.80 1.02 1.17 1.37.  (With stays of 512 rows whatever the track, arrays of ten antennas were 1.2 to 2.3 times past
// it.)  The rule costs 27 antennas x 100 times x 64 channels in 16 facets 19.7 -> 21.6 ms, 400 times 61.1 -> 61.8, a
// snapshot of 16 times 632 -> 723 us.
constexpr int kStaySegs = 4, kStayRows = 30;
__device__ __forceinline__ bool may_stay(int segs, int rows, int groups) {
  return segs < kStaySegs && (segs + 1) * groups <= rows && (segs + 1) * segs * kStayRows <= rows;
}

// Whether the rows of a channel's segments are taken last to first: a work item's segments are
// consecutive channels of one baseline, and turning round at each channel continues where the channel
// before it ended, a cell or less away, so that the owned cells stay in registers.
__device__ __forceinline__ bool rows_backwards(int chan) { return chan & 1; }

// What one CTA grids in place: its running state, and one row range (a channel's rows [r0, r1)) at a
// time, staged V rows at a time (prologue) and gridded chunk by chunk.
template <int NC, bool WPROJ, int J, int ACC, bool WIDE>
struct InPlace {
  VisRec<NC> *recs;  // [V]
  NormAcc *nacc;     // [V][NC]
  int *ng;           // [V]
  ItemSetup<NC, WPROJ> s;
  OwnerState<NC, J> st;
  long long fslice;
  bool along_v, first;
  int segs, stay, groups;  // since the owned cells last went out: segments, their rows and groups

  __device__ __forceinline__ void begin(const GridArgs &a, int f_local) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    recs = reinterpret_cast<VisRec<NC> *>(smem_raw);
    nacc = reinterpret_cast<NormAcc *>(smem_raw + sizeof(VisRec<NC>) * (size_t)a.V);
    ng = reinterpret_cast<int *>(nacc + (size_t)a.V * NC);
    item_setup<NC, WPROJ, J, ACC, WIDE>(a, f_local, smem_raw, s);
    fslice = (long long)(a.facet_base + f_local) * a.groups;
    if (a.norm)
      for (int i = threadIdx.x; i < a.V; i += blockDim.x) {
#pragma unroll
        for (int k = 0; k < NC; ++k) norm_zero(nacc[i * NC + k]);
        ng[i] = -1;
      }
    owner_reset(st);
    along_v = false;
    first = true;
    segs = stay = groups = 0;
  }

  __device__ __forceinline__ void rows(const GridArgs &a, int f_local, int chan, long long r0, long long r1) {
    if (r1 > a.nrows) r1 = a.nrows;
    const int tid = threadIdx.x, nt = blockDim.x;
    ChanCache cc;
    const double plane_scale = WPROJ ? (double)(a.P - 1) / a.wmax : 0.0;
    const bool back = rows_backwards(chan);
    for (long long base = r0; base < r1; base += a.V) {
      const int nv = (int)min((long long)a.V, r1 - base);
      for (int i = tid; i < nv; i += nt)
        stage_slot<NC, WPROJ>(a, f_local, chan, back ? r1 - 1 - (base - r0) - i : base + i, true, i, recs, cc, plane_scale);
      __syncthreads();
      if (a.norm) {
        if (a.tap_sums) {
          for (int i = tid; i < nv; i += nt) norm_slot<NC>(a, recs[i], i, nacc, ng, fslice);
        } else {
          norm_from_taps<NC, WPROJ>(a, recs, nv, s.table, nacc, ng, fslice);
        }
      }
      const int ngroups = find_groups(recs, nv, first, along_v, s.list);  // every warp its own list
      grid_chunk<NC, WPROJ, J, ACC>(a, recs, s.list, ngroups, along_v, s, st, [] {});
      first = false;
      groups += ngroups;
    }
    stay += (int)(r1 - r0);
    ++segs;
  }
  __device__ __forceinline__ void flush(const GridArgs &a) {
    item_flush<NC, WPROJ, J, ACC>(a, s, along_v, st);
    segs = stay = groups = 0;
  }

  // Normalisation, after the last rows.
  __device__ __forceinline__ void end(const GridArgs &a) {
    if (!a.norm || first) return;
    // the slots' current partial sums (earlier grid groups went out when the group
    // changed), summed over each warp by shuffles when its slots share one group (one atomic per
    // correlation and warp), added slot by slot otherwise.  The slots' state was last written before
    // the chunk loop's final barrier.
    for (int b = threadIdx.x & ~31; b < a.V; b += blockDim.x) {
      const int i = b + (threadIdx.x & 31);
      const bool has = i < a.V && ng[i] >= 0;
      const int my_g = has ? ng[i] : -1;
      const unsigned m = __ballot_sync(0xffffffffu, has);
      if (!m) continue;
      const int g0 = __shfl_sync(0xffffffffu, my_g, __ffs(m) - 1);
      const NormAcc *na = nacc + (has ? i : 0) * NC;
      if (__all_sync(0xffffffffu, !has || my_g == g0)) {
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          double v = has ? norm_value(na[k]) : 0.0;
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
          if ((threadIdx.x & 31) == 0 && v != 0.0) atomicAdd(&a.norm[(fslice + g0) * NC + k], v);
        }
      } else if (has) {
#pragma unroll
        for (int k = 0; k < NC; ++k)
          if (norm_value(na[k]) != 0.0) atomicAdd(&a.norm[(fslice + my_g) * NC + k], norm_value(na[k]));
      }
    }
  }
};

// Most segments of one work item.
constexpr int kMaxItemSegs = 16;

// The records of a work item's segments, in the order that they are gridded: piece i holds records
// [first[i], first[i + 1]) at src[i] (in shared memory, written by the CTA's first warp).
template <int NC>
struct RecordPieces {
  const GridRec<NC> *src[kMaxItemSegs];
  int first[kMaxItemSegs + 1];
};

// One work item from precomputed records: its pieces' records are staged V at a time by bulk copies
// (one per piece that a chunk touches) into two buffers used in turn, the next chunk's copies in flight
// while the current chunk is gridded.  No prologue and no normalisation here (the record kernel did
// both).  rbar are the two record barriers (one arrival each), rphase their phase parities (bit b for
// buffer b); copies are only issued for a chunk of this item, so none is in flight when the item ends.
template <int NC, bool WPROJ, int J, int ACC, bool WIDE>
__device__ __forceinline__ void grid_records(const GridArgs &a, const int f_local, const RecordPieces<NC> &pc, int npieces,
                                             unsigned long long *rbar, unsigned &rphase) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int V = a.V;
  GridRec<NC> *rb = reinterpret_cast<GridRec<NC> *>(smem_raw);  // [2][V]
  const int n = pc.first[npieces];
  if (n <= 0) return;
  const int tid = threadIdx.x;
  // Chunks hold V records.  Where not even two segments may stay in registers together (see may_stay) they end with
  // their segments, so that the cells go out exactly there: a chunk that runs on into the next segment adds its
  // rows to cells that have taken a whole segment already (64 records over segments of 45 rows: grids 1.2 times
  // as far off).  The first chunk ends with its segment; its groups tell for the next ones.  Thread 0 keeps the
  // books in shared memory, where they cost the owner threads no registers.
  __shared__ struct {
    int count[2], last[2];         // the staged chunks' records; whether no other chunk follows
    int at, piece, brief, cut;     // the next chunk's first record, and the piece that the one before it started in
    int ended, segs, stay, groups;  // pieces that ended; since the cells last went out: segments, rows and groups
    int out;                       // the cells go out after this chunk
  } s_ck;
  auto issue = [&](int buf) {
    const int lo = s_ck.at;
    int p = s_ck.piece;
    while (pc.first[p + 1] <= lo) ++p;
    s_ck.piece = p;
    const int hi = min(min(n, lo + V), s_ck.cut ? pc.first[p + 1] : n);
    s_ck.at = hi;
    s_ck.count[buf] = hi - lo;
    s_ck.last[buf] = hi == n;
    // the buffer may last have been written by plain stores (an item prepared in place)
    fence_proxy_async();
    bar_arrive_tx(&rbar[buf], (unsigned)(sizeof(GridRec<NC>) * (hi - lo)));  // (and publishes the above)
    GridRec<NC> *dst = rb + buf * V;
    for (int at = lo; at < hi;) {
      while (pc.first[p + 1] <= at) ++p;
      const int k = min(hi, pc.first[p + 1]) - at;
      bulk_copy(dst + (at - lo), pc.src[p] + (at - pc.first[p]), (unsigned)(sizeof(GridRec<NC>) * k), &rbar[buf]);
      at += k;
    }
  };
  if (tid == 0) {
    s_ck.at = s_ck.piece = s_ck.ended = s_ck.segs = s_ck.stay = s_ck.groups = 0;
    s_ck.brief = n < 2 * kStayRows * npieces;
    s_ck.cut = 1;
    issue(0);
  }
  ItemSetup<NC, WPROJ> s;
  item_setup<NC, WPROJ, J, ACC, WIDE>(a, f_local, smem_raw, s);
  OwnerState<NC, J> st;
  owner_reset(st);
  bool along_v = false;
  // Where the strips are long (J > 4), the group lists of chunks after the first are found by the last warp
  // (it has the fewest owners) for the CTA while the other warps still grid the chunk before; found by
  // every warp ahead of the chunk's merge they cost 2 % of a batched call of 27 antennas x 400 times x 64
  // channels.  The first chunk's list has nothing to hide behind, and the launches with J = 4 (small
  // supports, few warps) lost 3 % of a 16-time snapshot's class launches by it.
  constexpr bool kOneFinder = J > 4;
  __shared__ unsigned short s_list[2][kMaxChunk];
  __shared__ int s_ngroups[2];
  auto landed = [&](int buf) {
    const unsigned par = (rphase >> buf) & 1u;
    if (!bar_wait(&rbar[buf], par)) {
      atomicOr(a.error, DEV_ERR_WAIT_TIMEOUT);
      bar_wait(&rbar[buf], par);
    }
  };
  bool first = true;
  for (int cur = 0;; cur ^= 1) {
    landed(cur);
    rphase ^= 1u << cur;
    const int nv = s_ck.count[cur];
    const bool last = s_ck.last[cur];
    const unsigned short *list = s.list;
    int ng = 0;
    if (first) {
      ng = find_groups(rb + cur * V, nv, true, along_v, s.list);
      if (tid == 0) s_ck.cut = s_ck.brief || 2 * ng > nv;
    }
    // the other buffer was last read by the previous chunk, which every thread has finished
    if (tid == 0 && !last) issue(cur ^ 1);
    if (!first) {
      if (kOneFinder) {
        list = s_list[cur];
        ng = s_ngroups[cur];
      } else {
        ng = find_groups(rb + cur * V, nv, false, along_v, s.list);
      }
    }
    first = false;
    grid_chunk<NC, WPROJ, J, ACC>(a, rb + cur * V, list, ng, along_v, s, st, [&] {
      if (kOneFinder && !last && threadIdx.x >= blockDim.x - 32) {
        landed(cur ^ 1);
        const int found = find_groups(rb + (cur ^ 1) * V, s_ck.count[cur ^ 1], false, along_v, s_list[cur ^ 1]);
        if ((tid & 31) == 0) s_ngroups[cur ^ 1] = found;
      }
      // the owned cells go out at the end, and before it when a segment ended in the chunk and may_stay says so
      if (tid == 0) {
        const int stay = s_ck.stay + nv, groups = s_ck.groups + ng;
        int segs = s_ck.segs, out = last;
        if (!last) {
          const int hi = s_ck.at - s_ck.count[cur ^ 1], was = segs;
          int e = s_ck.ended;
          for (; pc.first[e + 1] <= hi; ++e) segs += pc.first[e + 1] > pc.first[e];
          s_ck.ended = e;
          if (segs != was) {
            out = !may_stay(segs, stay, groups);
            s_ck.cut = s_ck.brief || 2 * groups > stay;
          }
        }
        s_ck.segs = out ? 0 : segs;
        s_ck.stay = out ? 0 : stay;
        s_ck.groups = out ? 0 : groups;
        s_ck.out = out;
      }
    });
    if (s_ck.out) item_flush<NC, WPROJ, J, ACC>(a, s, along_v, st);
    if (last) break;
  }
}

// Register caps of the persistent segment kernel: the J rows' accumulators (8 J values), the merge
// step's values and the footprint state, without spills in the loops.
template <int J>
constexpr int kSegRegs = J <= 4 && sizeof(acc_real) == 4 ? 96 : J == 6 ? 112 : 128;

// One CTA per track: blockIdx -> (facet, baseline slot or row segment, channel).
template <int NC, bool WPROJ, int J, int ACC, bool WIDE>
__global__ void __launch_bounds__(512, 1) romein_grid_kernel(const GridArgs a) {
  long long track = blockIdx.x;
  const int chan = (int)(track % a.nchan);
  track /= a.nchan;
  const int slot = (int)(track % a.nslots);
  const int f_local = (int)(track / a.nslots);
  long long r0, r1;
  if (a.starts) {
    r0 = (long long)a.starts[slot];
    r1 = (long long)a.starts[slot + 1];
  } else {
    r0 = (long long)slot * a.seg;
    r1 = min(a.nrows, r0 + a.seg);
  }
  InPlace<NC, WPROJ, J, ACC, WIDE> work;
  work.begin(a, f_local);
  work.rows(a, f_local, chan, r0, r1);
  work.flush(a);
  work.end(a);
}

// Persistent form: a fixed grid of CTAs takes work items from a device counter until the device-side
// item count is exhausted.  Every segment is a run of one track's rows whose w planes share this
// launch's support class (a.W), in the order (baseline, channel, rows), the rows of odd channels
// backwards; an item is a block of consecutive segments in one facet, gridded as one stretch: the owned
// cells go out when the footprint leaves them, and all of them only where may_stay ends a stay.  The block is
// as long as leaves eight items per CTA, kMaxItemSegs at most (gridding 27 antennas x 100 times x 64
// channels into 16 facets, one segment per item spends a quarter of the class launches on the ends).  From
// records without w kernels it is one segment (supports of 7 and 15, 8 facets: 200 slow times 2678 -> 2651 and 4383 ->
// 4398 us, fast tracks 4724 -> 4494 and 8274 -> 7759, and errors below those of several).
// Items of one block are adjacent, so the facets of a segment are gridded while its rows are hot in L2.
// The loop ends on the count, never waits on other CTAs.  Two builds share the segments of a launch:
// PRE grids those that the record kernel had room for, the other build the rest (every segment when
// there are no records); the prologue of the latter would cost the former registers.
template <int NC, bool WPROJ, int J, int ACC, bool WIDE, bool PRE, int REGS = kSegRegs<J>>
__global__ void __launch_bounds__(512, 1) __maxnreg__(REGS) romein_segment_kernel(const GridArgs a, const int nfacets) {
  __shared__ int s_item;
  __shared__ int s_first, s_last;  // unmasked row range of a segment (facet row masks)
  __shared__ __align__(8) unsigned long long s_rec_bar[2];
  __shared__ RecordPieces<NC> s_pieces;
  unsigned rphase = 0;
  if (PRE && threadIdx.x == 0) {
    bar_init(&s_rec_bar[0], 1);
    bar_init(&s_rec_bar[1], 1);
  }
  const int count = *a.work_count;
  const long long base = *a.segment_base;
  int per = (int)max(1ll, min((long long)kMaxItemSegs, (long long)count * nfacets / (8ll * gridDim.x)));
  if (PRE && !WPROJ) per = 1;
  const long long total = (long long)((count + per - 1) / per) * nfacets;
  // a segment of the schedule; false (reported) when it lies outside the schedule or the rows
  auto segment = [&](long long si, int4 &sg) -> bool {
    if (si < 0 || si >= a.segment_capacity) {
      atomicOr(a.error, DEV_ERR_GRID_INDEX);
      return false;
    }
    sg = a.segments[si];
    if (sg.x < 0 || sg.x > sg.y || (long long)sg.y > a.nrows || sg.z < 0 || sg.z >= a.nchan) {
      atomicOr(a.error, DEV_ERR_GRID_INDEX);
      return false;
    }
    return true;
  };
  auto recorded = [&](long long si, int len) {
    return a.records && (a.rec_off[si] + len) * nfacets <= a.rec_capacity;
  };
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(a.work_next, 1);
    __syncthreads();
    const long long item = s_item;
    if (item >= total) break;
    const int block = (int)(item / nfacets);
    const int f_local = (int)(item - (long long)block * nfacets);
    const long long s0 = base + (long long)block * per;
    const int nseg = min(per, count - block * per);
    if constexpr (PRE) {
      // one lane per segment: its first to last valid record (all of them past the range table)
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int n = 0;
        int4 sg;
        if (lane < nseg && segment(s0 + lane, sg) && recorded(s0 + lane, sg.y - sg.x)) {
          const long long si = s0 + lane, it = si * nfacets + f_local;
          const int len = sg.y - sg.x;
          int lo = 0, hi = len;
          if (it < a.range_capacity) {
            const int2 rg = a.item_range[it];
            lo = rg.x;
            hi = rg.y;
          }
          n = max(0, hi - lo);
          s_pieces.src[lane] = reinterpret_cast<const GridRec<NC> *>(a.records) + a.rec_off[si] * nfacets +
                               (long long)f_local * len + lo;
        }
        int sum = n;
#pragma unroll
        for (int off = 1; off < kMaxItemSegs; off <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, sum, off);
          if (lane >= off) sum += x;
        }
        if (lane == 0) s_pieces.first[0] = 0;
        if (lane < nseg) s_pieces.first[lane + 1] = sum;
      }
      __syncthreads();
      grid_records<NC, WPROJ, J, ACC, WIDE>(a, f_local, s_pieces, nseg, s_rec_bar, rphase);
    } else {
      InPlace<NC, WPROJ, J, ACC, WIDE> work;
      work.begin(a, f_local);
      for (int i = 0;; ++i) {
        if (i == nseg || (work.segs && !may_stay(work.segs, work.stay, work.groups))) work.flush(a);
        if (i == nseg) break;
        int4 sg;
        if (!segment(s0 + i, sg) || recorded(s0 + i, sg.y - sg.x)) continue;
        long long r0 = sg.x, r1 = sg.y;
        if (a.facet_row_mask) {
          // a facet that leaves rows out grids only the segment's first to last row it keeps, and skips
          // the segment when it keeps none (the rows in between are still tested in the prologue)
          __syncthreads();
          if (threadIdx.x == 0) {
            s_first = 0x7fffffff;
            s_last = -1;
          }
          __syncthreads();
          const uint8_t *m = a.facet_row_mask + (long long)(a.facet_base + f_local) * a.nrows;
          int first = 0x7fffffff, last = -1;
          for (int r = sg.x + (int)threadIdx.x; r < sg.y; r += (int)blockDim.x)
            if (m[r]) {
              first = min(first, r);
              last = max(last, r);
            }
          if (last >= 0) {
            atomicMin(&s_first, first);
            atomicMax(&s_last, last);
          }
          __syncthreads();
          if (s_last < 0) continue;  // uniform: every thread reads the same shared values
          r0 = s_first;
          r1 = (long long)s_last + 1;
        }
        work.rows(a, f_local, sg.z, r0, r1);
      }
      work.end(a);
    }
  }
}

}  // namespace bz

// Queues the conversion of n cells of a narrow grid to the wide form of the 32-bit library's accumulation
// (have_lo: its second word holds a value; else it is written), and back, in place or to `out` as one word
// (kernels_misc.cuh); no work in the 64-bit library.
bool bz_widen_grid(vis_complex *hi, vis_complex *lo, long long n, bool have_lo, cudaStream_t st);
bool bz_narrow_grid(vis_complex *hi, vis_complex *lo, vis_complex *out, long long n, cudaStream_t st);
