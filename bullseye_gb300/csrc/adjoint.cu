// Adjoint of facet gridding (a degridder): gradients of a real loss with respect to the
// visibilities and the per-antenna 2x2 Jones terms, given the gradient with respect to the grids.
//
// Forward (per facet f, visibility (row, channel), correlation c, footprint cell (x, y)):
//   M   = J_p^-1 V J_q^-H                       (Jones correction, 2x2)
//   V'  = s M,  s = weight x flag x e^{i phi_f} (phase rotation to the facet centre)
//   y   = V' (w >= 0) or conj(V') (w < 0, gridded at (-u, -v))
//   G  += y tap(x - u0, y - v0)
// With the real-inner-product convention dL = Re <g_z, dz> (torch's complex gradient):
//   g_y  = sum over the footprint of g_G conj(tap)         (a gather: no atomics)
//   g_V' = g_y or conj(g_y)
//   g_M  = conj(s) g_V'
//   g_V  = P^H g_M Q                                      (P = J_p^-1, Q = J_q^-1)
//   g_Jp = -P^H g_M M^H,   g_Jq = -Q^H g_M^H M            (d(J^-1) = -J^-1 dJ J^-1)
// Cells, taps, w plane and phase come from the gridder's own choose_cells (floor for 1-D AA
// kernels, round-half-even for w-projection, full-support acceptance), so the adjoint reads exactly
// the footprint the gridder wrote.  The normalisation sums depend only on weights and taps, so they
// carry no gradient.
//
// Prediction (bullseye_predict) is the physical forward model of the same measurement, on the same
// gather: from model grids G_f (the model images divided by the gridding correction, transformed
// with the reference's shifts, or given as grids),
//   D   = sum over the footprint of G_f conj(tap)            [/ Re sum tap: the normalised form of
//                                                              the reference's prototype degridder,
//                                                              Resampling.ipynb cell 17]
//   V'  = D (w >= 0) or conj(D) (w < 0),   M = e^{-i phi_f} V'
//   V  += J_p M J_q^H   (the gains applied forward; no weights, no flags), summed over facets.
//
// Work layout: a warp takes 32 consecutive rows of one channel; each lane resolves its own row's Jones
// terms and geometry.  Rows are consecutive times of a baseline when they come baseline by baseline, so
// stretches of them share the footprint corner, the w plane and the row taps kv: such a *group* gathers the
// grid once,
//   R(u) = sum over v of g_G(u, v) conj(kv(v))      (W^2 grid reads per group, lanes along u),
//   D    = sum over u of R(u) conj(ku(u))            (W per visibility, reduced over the warp),
// which is each visibility's footprint sum with its common factor taken out.  EVLA tracks with 14 s samples
// (oversampling 15) give 3.9 visibilities per group.  Rows in any other order give groups of one.
//
// Prediction with w kernels keeps every visibility's own order of additions: its model grids come from
// images divided by the taper, whose large edge values cancel in each footprint sum by factors of 1e3 and
// more, so that sums taken in another order differ by as much as they are off.  There, up to four
// visibilities of a stretch that shares corner, w plane and grid (a *run*, 14 visibilities on the tracks
// above) read each grid cell once and keep their own products and sums.
// The visibility result (summed over facets) is written once; Jones gradients are accumulated with
// atomics because every antenna appears on many baselines.
#include <cufft.h>

#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "common.h"
#include "gridder.cuh"

using namespace bz;

namespace {

struct AdjointArgs {
  const vis_complex *vis;
  const vis_real *weights;
  const uint8_t *flags;
  const vis_real *uvw;
  const uint8_t *flagged_rows;
  const unsigned *field;
  const unsigned *spw;
  const unsigned *ant1, *ant2;
  const size_t *time_ids;
  const vis_complex *jones;  // raw terms [T][A][F][S][Ch][4], or null (no correction)
  const vis_real *wavelengths;
  const uint8_t *enabled;
  const size_t *cgi;
  const void *conv;
  const vis_real *facet_centres;  // [F][2] arcsec, or null (no faceting)
  const vis_complex *grad_grid;   // [F][cube][4][ny][nx], or [F][cube][ny][nx][4] with grid_interleaved
  vis_complex *grad_vis;          // [R][Ch][4]
  vis_complex *grad_jones;        // like jones, accumulated; or null
  long long nrows;
  int nchan, nspw, nant, ntimes, nfacets, cube, nx, ny, W, os, K, P, faceting;
  int normalise;  // prediction: divide each facet's gathered value by the real part of its tap sum
  int row_bytes;  // shared memory of a warp's staged kernel row, 0: taps are read from the table
  int grid_interleaved;  // prediction from its own model grids: a cell's 4 correlations are adjacent
  unsigned imaging_field;
  double u_scale, v_scale, gcx, gcy, wmax, ra0, dec0;
};

// Dynamic shared memory of the gather kernel: the facet transforms, the w planes' windows, then
// (16-byte aligned) per warp the rows' sums [32][8] and, when there is room, one plane's kernel row [K].
__host__ __device__ inline size_t degrid_warps_offset(int nfacets, int P) {
  return (sizeof(FacetXform) * (size_t)nfacets + sizeof(int2) * (size_t)P + 15) / 16 * 16;
}
constexpr int kDegridWarps = 4;
constexpr size_t kDegridSums = 32 * 9 * sizeof(acc_real);  // 8 components and the tap sum per row
// The kernel row is staged up to this size per warp (with four warps per CTA, four CTAs on an SM).
constexpr size_t kDegridRowMax = 11 * 1024;
template <bool WPROJ>
__host__ __device__ inline size_t degrid_row_bytes(int K) {
  const size_t b = (sizeof(typename TapT<WPROJ>::type) * (size_t)K + 15) / 16 * 16;
  return b <= kDegridRowMax ? b : 0;
}

// The 4 adjacent correlations of one cell (32 bytes in single precision, 16-byte aligned): two
// 16-byte loads.
__device__ __forceinline__ void load_cell4(const vis_complex *p, cplx out[4]) {
#if defined(BULLSEYE_SINGLE)
  const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 2);
  out[0].re = a.x; out[0].im = a.y;
  out[1].re = a.z; out[1].im = a.w;
  out[2].re = b.x; out[2].im = b.y;
  out[3].re = b.z; out[3].im = b.w;
#else
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    out[k].re = p[k].re;
    out[k].im = p[k].im;
  }
#endif
}

__device__ __forceinline__ cplx cconj(cplx a) {
  a.im = -a.im;
  return a;
}
__device__ __forceinline__ cplx cadd(cplx a, cplx b) {
  a.re += b.re;
  a.im += b.im;
  return a;
}
// 2x2 products with optional hermitian transposes: O = op(A) op(B)
__device__ __forceinline__ void mat2(const cplx *A, bool ha, const cplx *B, bool hb, cplx *O) {
  cplx a[4], b[4];
  if (ha) { a[0] = cconj(A[0]); a[1] = cconj(A[2]); a[2] = cconj(A[1]); a[3] = cconj(A[3]); }
  else { a[0] = A[0]; a[1] = A[1]; a[2] = A[2]; a[3] = A[3]; }
  if (hb) { b[0] = cconj(B[0]); b[1] = cconj(B[2]); b[2] = cconj(B[1]); b[3] = cconj(B[3]); }
  else { b[0] = B[0]; b[1] = B[1]; b[2] = B[2]; b[3] = B[3]; }
  jmul(a, b, O);
}

__device__ __forceinline__ bool inv2(cplx *m) {
  cplx det;
  det.re = (m[0].re * m[3].re - m[0].im * m[3].im) - (m[1].re * m[2].re - m[1].im * m[2].im);
  det.im = (m[0].re * m[3].im + m[0].im * m[3].re) - (m[1].re * m[2].im + m[1].im * m[2].re);
  if (det.re == (acc_real)0 && det.im == (acc_real)0) return false;
  const acc_real n2 = det.re * det.re + det.im * det.im;
  cplx inv;
  inv.re = det.re / n2;
  inv.im = -det.im / n2;
  cplx neg;
  neg.re = -inv.re;
  neg.im = -inv.im;
  const cplx a0 = m[0];
  m[0] = cmul(m[3], inv);
  m[3] = cmul(a0, inv);
  m[1] = cmul(m[1], neg);
  m[2] = cmul(m[2], neg);
  return true;
}

__device__ __forceinline__ acc_real tap_at(const void *conv, long long idx, acc_real) {
  return (acc_real)((const vis_real *)conv)[idx];
}
__device__ __forceinline__ cplx tap_at(const void *conv, long long idx, cplx) {
  const vis_complex c = ((const vis_complex *)conv)[idx];
  cplx t;
  t.re = (acc_real)c.re;
  t.im = (acc_real)c.im;
  return t;
}
__device__ __forceinline__ bool tap_zero(acc_real t) { return t == (acc_real)0; }
__device__ __forceinline__ bool tap_zero(cplx t) { return t.re == (acc_real)0 && t.im == (acc_real)0; }
// acc += g conj(t), with one rounding of the sum per term (two fused multiply-adds on it are an instruction less and
// two roundings)
__device__ __forceinline__ void mac_conj(cplx &acc, cplx g, acc_real t) {
  acc.re = fma(g.re, t, acc.re);
  acc.im = fma(g.im, t, acc.im);
}
__device__ __forceinline__ void mac_conj(cplx &acc, cplx g, cplx t) {
  acc.re += fma(g.re, t.re, g.im * t.im);
  acc.im += fma(g.im, t.re, -(g.re * t.im));
}
__device__ __forceinline__ cplx tap_value(acc_real t) { cplx c; c.re = t; c.im = 0; return c; }
__device__ __forceinline__ cplx tap_value(cplx t) { return t; }
__device__ __forceinline__ acc_real real_part(acc_real t) { return t; }
__device__ __forceinline__ acc_real real_part(cplx t) { return t.re; }

// The footprint sums of B visibilities of one run (each in the order of a visibility by itself: lane l takes
// cells l, l + 32, ... of the window, then a butterfly over the lanes), cells read once.  fu, fv: the
// visibilities' first taps in the window.
template <int B, class Tap, class Cell>
__device__ __forceinline__ void gather_run(const int (&fu)[B], const int (&fv)[B], int ww, int os, long long nx,
                                           const Tap &tap, const Cell &cell, acc_real (&v)[B][8], acc_real (&ts)[B]) {
  cplx D[B][4];
#pragma unroll
  for (int b = 0; b < B; ++b) {
#pragma unroll
    for (int k = 0; k < 4; ++k) { D[b][k].re = 0; D[b][k].im = 0; }
    ts[b] = 0;
  }
  const int lane = threadIdx.x & 31;
  const int ncell = ww * ww, sju = 32 % ww, sjv = 32 / ww;
  int ru = lane % ww, rv = lane / ww;
  long long off = (long long)rv * nx + ru;
  const long long step = (long long)sjv * nx + sju, wrap = nx - ww;
#pragma unroll(B > 1 ? 1 : 2)
  for (int idx = lane; idx < ncell; idx += 32) {
    cplx gc[4];
    cell(off, gc);
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const cplx t = cmul(tap_value(tap(fu[b] + ru * os)), tap_value(tap(fv[b] + rv * os)));
      const cplx ct = cconj(t);
      ts[b] += t.re;
#pragma unroll
      for (int k = 0; k < 4; ++k) D[b][k] = cadd(D[b][k], cmul(gc[k], ct));
    }
    ru += sju;
    rv += sjv;
    off += step;
    if (ru >= ww) {  // one wrap at most: sju < ww, or ww > 32 and sju = 32
      ru -= ww;
      ++rv;
      off += wrap;
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[b][2 * k] = D[b][k].re;
      v[b][2 * k + 1] = D[b][k].im;
    }
}

// Sums eight values over the warp; lane l returns the sum of value l >> 2 (in each group of four lanes).
// Each of the first three steps halves the values a lane carries: 9 shuffles, not 40.
__device__ __forceinline__ acc_real warp_sum8(const acc_real (&v)[8]) {
  const int lane = threadIdx.x & 31;
  acc_real a[4], b[2], c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const acc_real send = (lane & 16) ? v[i] : v[i + 4], keep = (lane & 16) ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const acc_real send = (lane & 8) ? a[i] : a[i + 2], keep = (lane & 8) ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  {
    const acc_real send = (lane & 4) ? b[0] : b[1], keep = (lane & 4) ? b[1] : b[0];
    c = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// A value as the sum of two words: the tap sum that prediction divides by, so that the quotient is rounded once
// (summed and divided in single words it is off by as much again as the gathered value: 1.19e-7 against 0.89e-7;
// products of taps that are summed as they are gathered share their roundings with it, 1.07e-7).
struct Pair {
  acc_real hi, lo;
};
__device__ __forceinline__ void pair_add(Pair &s, acc_real x) {
  const acc_real t = s.hi + x, b = t - s.hi;
  s.lo += (s.hi - (t - b)) + (x - b);
  s.hi = t;
}
__device__ __forceinline__ Pair pair_product(Pair a, Pair b) {
  const acc_real p = a.hi * b.hi;
  return Pair{p, fma(a.hi, b.hi, -p) + fma(a.hi, b.lo, a.lo * b.hi)};
}
// v / d, inv = 1 / d.hi
__device__ __forceinline__ acc_real pair_quotient(acc_real v, Pair d, acc_real inv) {
  const acc_real q = v * inv, r = fma(fma(-q, d.lo, fma(-q, d.hi, v)), inv, q);
  return r == r ? r : q;  // (an infinity's remainder is not a number)
}

__device__ __forceinline__ void atomic_add_c(vis_complex *dst, cplx v) {
  atomicAdd(&dst->re, (vis_real)v.re);
  atomicAdd(&dst->im, (vis_real)v.im);
}

// PREDICT = false: the adjoint (grad_grid -> grad_vis, grad_jones).  PREDICT = true: prediction
// (model grids in grad_grid -> visibilities in grad_vis).
template <bool WPROJ, bool PREDICT>
__global__ void __launch_bounds__(kDegridWarps * 32, sizeof(acc_real) == 4 ? 4 : 3) degrid_adjoint_kernel(const AdjointArgs a) {
  typedef typename TapT<WPROJ>::type tap_t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FacetXform *fx = reinterpret_cast<FacetXform *>(smem_raw);
  for (int f = threadIdx.x; f < a.nfacets; f += blockDim.x) {
    double ra = a.ra0, dec = a.dec0;
    if (a.faceting && a.facet_centres) {
      ra = (double)a.facet_centres[2 * f];
      dec = (double)a.facet_centres[2 * f + 1];
    }
    // the gridder's own transform, so that a sample takes the same cells
    fx[f] = facet_transform(a.ra0, a.dec0, ra, dec, a.faceting != 0, a.faceting != 0);
  }
  // nonzero window [lo, hi] of every w plane's kernel row, one warp per plane: a footprint cell s
  // reads sample fu + s*os with fu in [floor(os/2), floor(3 os/2)] (w-projection, round to nearest)
  // or [0, os] (AA, floor); cells that cannot reach a nonzero sample carry a zero tap and are skipped
  int2 *win = reinterpret_cast<int2 *>(smem_raw + sizeof(FacetXform) * a.nfacets);
  {
    const int ln = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int fu_min = WPROJ ? (int)floor(0.5 * a.os - 1e-6) : 0;
    const int fu_max = WPROJ ? (int)floor(1.5 * a.os + 1e-6) : a.os;
    for (int pl = wid; pl < a.P; pl += nw) {
      int lo = 0x7fffffff, hi = -1;
      for (int i = ln; i < a.K; i += 32) {
        if (!tap_zero(tap_at(a.conv, (long long)pl * a.K + i, tap_t()))) {
          lo = min(lo, i);
          hi = max(hi, i);
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      if (ln == 0) {
        int2 w2 = make_int2(0, -1);  // empty window: an all-zero row
        if (hi >= 0) {
          w2.x = max(0, (int)ceil((double)(lo - fu_max) / a.os));
          w2.y = min(a.W - 1, (int)floor((double)(hi - fu_min) / a.os));
        }
        win[pl] = w2;
      }
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const size_t row_bytes = (size_t)a.row_bytes;
  unsigned char *mine = smem_raw + degrid_warps_offset(a.nfacets, a.P) + (kDegridSums + row_bytes) * (threadIdx.x >> 5);
  acc_real *s_sum = reinterpret_cast<acc_real *>(mine);              // [32][8], then [32] tap sums
  tap_t *s_row = reinterpret_cast<tap_t *>(mine + kDegridSums);      // the kernel row of plane staged
  int staged = -1;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int W = a.W;
  const long long nxy = (long long)a.nx * a.ny;
  const double plane_scale = WPROJ ? (double)(a.P - 1) / a.wmax : 0.0;
  const bool jones_vec = vec16(a.jones);  // 16-byte loads of the 2x2 terms (every term starts at 4 x 8 bytes)

  // Each warp takes 32 consecutive rows of one channel at a time (the channels of a row block by
  // neighbouring warps).  Lane i does the scalar work of row i: its loads, the FP64 geometry, the Jones
  // inverses and the chain rule, so that FP64 and the 2x2 algebra run 32 rows per instruction (GB300
  // issues FP64 at 1/64 of FP32).  The warp then gathers the footprints group by group with every lane,
  // and each row's sums land in its own lane.
  const long long blocks = (a.nrows + 31) / 32, total = blocks * a.nchan;
  for (long long task = warp; task < total; task += nwarps) {
    const int c = (int)(task % a.nchan);
    const long long row = task / a.nchan * 32 + lane;
    bool live = row < a.nrows;
    long long sc = 0;
    unsigned spw = 0;
    size_t g = 0;
    if (live) {
      spw = a.spw[row];
      live = spw < (unsigned)a.nspw;
    }
    if (live) {
      sc = (long long)spw * a.nchan + c;
      live = a.enabled[sc] != 0;
    }
    if (live) {
      g = a.cgi[sc];
      live = g < (size_t)a.cube;
    }
    ChanCache cc;
    double um = 0, vm = 0, wm = 0;
    if (live) {
      cc.spw = spw;
      cc.inv = 1.0 / (double)a.wavelengths[sc];
      cc.su = cc.inv * a.u_scale;
      cc.sv = cc.inv * a.v_scale;
      cc.sw = cc.inv * plane_scale;
      um = (double)a.uvw[3 * row];
      vm = (double)a.uvw[3 * row + 1];
      wm = (double)a.uvw[3 * row + 2];
    }
    const long long base = (row * a.nchan + c) * 4;
    cplx gV[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { gV[k].re = 0; gV[k].im = 0; }

    for (int f = 0; f < a.nfacets; ++f) {
      // this lane's item: Jones indices and the geometry (the gridder's own cell choice: same
      // cells, taps, plane and phase)
      long long i1 = 0, i2 = 0;
      CellChoice cell;
      cell.du = cell.dv = cell.fu = cell.fv = cell.plane = 0;
      cell.flip = false;
      cplx ph;
      ph.re = 1;
      ph.im = 0;
      bool ok = live;
      if (ok && a.jones) {
        const long long t = (long long)a.time_ids[row];
        const unsigned a1 = a.ant1[row], a2 = a.ant2[row];
        if (t < 0 || t >= a.ntimes || a1 >= (unsigned)a.nant || a2 >= (unsigned)a.nant) {
          ok = false;
        } else {
          i1 = ((((t * a.nant + a1) * a.nfacets + f) * a.nspw + spw) * a.nchan + c) * 4;
          i2 = ((((t * a.nant + a2) * a.nfacets + f) * a.nspw + spw) * a.nchan + c) * 4;
        }
      }
      if (ok)
        ok = choose_cells<WPROJ>(um, vm, wm, cc, fx[f], a.faceting != 0, a.faceting != 0, a.u_scale, a.v_scale,
                                 plane_scale, a.gcx, a.gcy, a.nx, a.ny, W, a.P, a.os, ph, cell);
      // gather, group by group: D_k = sum over the footprint of g_G conj(tap)
      const bool want_ts = PREDICT && a.normalise;
      int prev_fv = __shfl_up_sync(0xffffffffu, cell.fv, 1), prev_u = __shfl_up_sync(0xffffffffu, cell.du, 1);
      int prev_v = __shfl_up_sync(0xffffffffu, cell.dv, 1), prev_pl = __shfl_up_sync(0xffffffffu, cell.plane, 1);
      const int gi = (int)g, prev_g = __shfl_up_sync(0xffffffffu, gi, 1);
      const unsigned oks = __ballot_sync(0xffffffffu, ok);
      constexpr bool kRuns = PREDICT && WPROJ;  // see the work layout above
      const bool begins = ok && !(lane > 0 && (oks >> (lane - 1) & 1) && (kRuns || prev_fv == cell.fv) &&
                                  prev_u == cell.du && prev_v == cell.dv && prev_pl == cell.plane && prev_g == gi);
      const unsigned starts = __ballot_sync(0xffffffffu, begins);
      unsigned todo = starts;
      __syncwarp();  // every lane has read the previous facet's sums
      while (todo) {
        const int it = __ffs(todo) - 1;
        todo &= todo - 1;
        // the group's rows [it, end): up to the next group or row without a footprint
        const unsigned edge = (starts | ~oks) & (it < 31 ? ~0u << (it + 1) : 0u);
        const int end = edge ? __ffs(edge) - 1 : 32;
        const int u0 = __shfl_sync(0xffffffffu, cell.du, it), v0 = __shfl_sync(0xffffffffu, cell.dv, it);
        const int plane = __shfl_sync(0xffffffffu, cell.plane, it), fv = __shfl_sync(0xffffffffu, cell.fv, it);
        const long long git = __shfl_sync(0xffffffffu, gi, it);
        const long long slice0 = ((long long)f * a.cube + git) * 4;
        const long long cube0 = ((long long)f * a.cube + git) * nxy;  // interleaved layout
        const int2 w2 = win[plane];
        const int ww = w2.y - w2.x + 1;
        // the plane's kernel row (the w plane does not depend on the facet: it changes once or twice in
        // a warp's rows)
        if (row_bytes && staged != plane) {
          __syncwarp();
          for (int i = lane; i < a.K; i += 32) s_row[i] = tap_at(a.conv, (long long)plane * a.K + i, tap_t());
          __syncwarp();
          staged = plane;
        }
        auto tap = [&](int at) { return row_bytes ? s_row[at] : tap_at(a.conv, (long long)plane * a.K + at, tap_t()); };
        if (ww <= 0) {  // an all-zero kernel row: the sums are zero
          for (int i = it * 8 + lane; i < end * 8; i += 32) s_sum[i] = 0;
          if (want_ts && lane >= it && lane < end) s_sum[256 + lane] = 0;
          continue;
        }
        if constexpr (kRuns) {
          const long long corner = (long long)(v0 + w2.x) * a.nx + (u0 + w2.x);
          const int w0 = w2.x * a.os;
          const bool packed = a.grid_interleaved != 0;
          const vis_complex *p = packed ? a.grad_grid + (cube0 + corner) * 4 : a.grad_grid + slice0 * nxy + corner;
          auto cells = [&](long long off, cplx (&gc)[4]) {
            if (packed) {
              load_cell4(p + off * 4, gc);
            } else {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const vis_complex gg = p[k * nxy + off];
                gc[k].re = gg.re;
                gc[k].im = gg.im;
              }
            }
          };
          auto some = [&](auto nb, int i0) {
            constexpr int B = decltype(nb)::value;
            int fus[B], fvs[B];
            acc_real v[B][8], ts[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
              fus[b] = __shfl_sync(0xffffffffu, cell.fu, i0 + b) + w0;
              fvs[b] = __shfl_sync(0xffffffffu, cell.fv, i0 + b) + w0;
            }
            gather_run<B>(fus, fvs, ww, a.os, a.nx, tap, cells, v, ts);
#pragma unroll
            for (int b = 0; b < B; ++b) {
              const acc_real sum = warp_sum8(v[b]);
              if ((lane & 3) == 0) s_sum[(i0 + b) * 8 + (lane >> 2)] = sum;
              if (want_ts) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ts[b] += __shfl_xor_sync(0xffffffffu, ts[b], o);
                if (lane == 0) s_sum[256 + i0 + b] = ts[b];
              }
            }
          };
          int i = it;
          for (; i + 4 <= end; i += 4) some(std::integral_constant<int, 4>{}, i);
          if (i + 2 <= end) {
            some(std::integral_constant<int, 2>{}, i);
            i += 2;
          }
          if (i < end) some(std::integral_constant<int, 1>{}, i);
          continue;
        }
        // lanes along u (32 columns at a time); a narrow window's rows are dealt to 32 / xw lane sets
        const int xw = ww > 16 ? 32 : ww > 8 ? 16 : 8, ys = 32 / xw, y0 = lane / xw;
        const long long corner = (long long)(v0 + w2.x) * a.nx + (u0 + w2.x);
        const int fvw = fv + w2.x * a.os;
        for (int xb = 0; xb < ww; xb += 32) {
          const int xl = xb + (lane & (xw - 1));
          const bool in = xl < ww;
          const int x = in ? xl : ww - 1;  // lanes past the window read its last column and count zero
          // even and odd rows in two sums, so that a chain of additions is no longer than that of a visibility
          // gathered by itself (W^2 / 32 terms per lane).  Error of random gradients' gathered values, as part of that
          // of single visibilities, with one sum and two roundings per term: 1.02 to 1.18; so: 0.95 to 0.99.
          cplx R[2][4];
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int k = 0; k < 4; ++k) { R[q][k].re = 0; R[q][k].im = 0; }
          const bool packed = PREDICT && a.grid_interleaved;
          const vis_complex *p = packed ? a.grad_grid + (cube0 + corner + x) * 4 : a.grad_grid + slice0 * nxy + corner + x;
          auto row = [&](int y, cplx (&sum)[4]) {
            cplx gc[4];
            if (packed) {
              load_cell4(p + (long long)y * a.nx * 4, gc);
            } else {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const vis_complex gg = p[k * nxy + (long long)y * a.nx];
                gc[k].re = gg.re;
                gc[k].im = gg.im;
              }
            }
            const tap_t t = tap(fvw + y * a.os);
#pragma unroll
            for (int k = 0; k < 4; ++k) mac_conj(sum[k], gc[k], t);
          };
          int y = y0;
#pragma unroll 1
          for (; y + ys < ww; y += 2 * ys) {
            row(y, R[0]);
            row(y + ys, R[1]);
          }
          if (y < ww) row(y, R[0]);
#pragma unroll
          for (int k = 0; k < 4; ++k) R[0][k] = cadd(R[0][k], R[1][k]);
          for (int i = it; i < end; ++i) {
            const int at = __shfl_sync(0xffffffffu, cell.fu, i) + (w2.x + x) * a.os;
            tap_t t = tap(at);
            cplx D[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              D[k].re = 0;
              D[k].im = 0;
              mac_conj(D[k], R[0][k], t);
            }
            acc_real v[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              v[2 * k] = in ? D[k].re : (acc_real)0;
              v[2 * k + 1] = in ? D[k].im : (acc_real)0;
            }
            const acc_real sum = warp_sum8(v);
            if ((lane & 3) == 0) {
              acc_real *d = s_sum + i * 8 + (lane >> 2);
              *d = xb ? *d + sum : sum;
            }
          }
        }
      }
      __syncwarp();
      cplx myD[4];
      acc_real myTS = 0;
      if (ok) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          myD[k].re = s_sum[lane * 8 + 2 * k];
          myD[k].im = s_sum[lane * 8 + 2 * k + 1];
        }
        if (kRuns && want_ts) myTS = s_sum[256 + lane];
      }
      Pair ts{0, 0};
      if (PREDICT && !kRuns && want_ts && ok) {
        // sum of ku x sum of kv of the lane's own row (real taps, one plane: w kernels are predicted by runs)
        const int2 w2 = win[cell.plane];
        Pair su{0, 0}, sv{0, 0};
        for (int s = w2.x; s <= w2.y; ++s) {
          const int u = cell.fu + s * a.os, v = cell.fv + s * a.os;
          const long long row0 = (long long)cell.plane * a.K;
          pair_add(su, real_part(row_bytes ? s_row[u] : tap_at(a.conv, row0 + u, tap_t())));
          pair_add(sv, real_part(row_bytes ? s_row[v] : tap_at(a.conv, row0 + v, tap_t())));
        }
        ts = pair_product(su, sv);
        myTS = ts.hi;
      }
      if (!ok) continue;
      if (PREDICT) {
        // V' = D or conj(D) (w < 0), normalised by the tap sum; M = e^{-i phi} V'; V += J_p M J_q^H
        const acc_real inv = (want_ts && myTS != (acc_real)0) ? (acc_real)1 / myTS : (acc_real)1;
        const cplx cph = cconj(ph);
        cplx X[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          cplx v = cell.flip ? cconj(myD[k]) : myD[k];
          if (kRuns || !want_ts || myTS == (acc_real)0) {  // (runs keep every visibility's own operations)
            v.re *= inv;
            v.im *= inv;
          } else {
            v.re = pair_quotient(v.re, ts, inv);
            v.im = pair_quotient(v.im, ts, inv);
          }
          X[k] = cmul(cph, v);
        }
        if (a.jones) {
          cplx Pm[4], Qm[4], T[4], O[4];
          load_c4(a.jones + i1, jones_vec, Pm);
          load_c4(a.jones + i2, jones_vec, Qm);
          mat2(Pm, false, X, false, T);  // J_p M
          mat2(T, false, Qm, true, O);   // (J_p M) J_q^H
#pragma unroll
          for (int k = 0; k < 4; ++k) gV[k] = cadd(gV[k], O[k]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) gV[k] = cadd(gV[k], X[k]);
        }
        continue;
      }
      // chain rule back to V (and the Jones terms), each lane for its own item
      cplx Pm[4], Qm[4];
      if (a.jones) {
        load_c4(a.jones + i1, jones_vec, Pm);
        load_c4(a.jones + i2, jones_vec, Qm);
        if (!inv2(Pm) || !inv2(Qm)) continue;  // a singular term: no gradient through it
      }
      const bool row_ok = !a.flagged_rows[row] && a.field[row] == a.imaging_field;
      acc_real cw[4];
      bool fl[4];
      load_r4(a.weights + base, vec16(a.weights), cw);
      load_f4(a.flags + base, (reinterpret_cast<uintptr_t>(a.flags) & 3) == 0, fl);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (!row_ok || fl[k]) cw[k] = (acc_real)0;
      cplx gM[4];
      const cplx cph = cconj(ph);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const cplx gvp = cell.flip ? cconj(myD[k]) : myD[k];
        cplx t = cmul(cph, gvp);
        t.re *= cw[k];
        t.im *= cw[k];
        gM[k] = t;
      }
      if (a.jones) {
        cplx T[4], G1[4];
        mat2(Pm, true, gM, false, T);  // P^H gM
        mat2(T, false, Qm, false, G1);  // (P^H gM) Q
#pragma unroll
        for (int k = 0; k < 4; ++k) gV[k] = cadd(gV[k], G1[k]);
        if (a.grad_jones) {
          cplx V[4];
          load_c4(a.vis + base, vec16(a.vis), V);
          cplx VQ[4], M[4], gp[4], gq[4];
          mat2(V, false, Qm, true, VQ);  // V Q^H
          mat2(Pm, false, VQ, false, M);  // M = P V Q^H
          mat2(T, false, M, true, gp);    // P^H gM M^H
          cplx T2[4];
          mat2(Qm, true, gM, true, T2);   // Q^H gM^H
          mat2(T2, false, M, false, gq);  // Q^H gM^H M
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            gp[k].re = -gp[k].re; gp[k].im = -gp[k].im;
            gq[k].re = -gq[k].re; gq[k].im = -gq[k].im;
            atomic_add_c(a.grad_jones + i1 + k, gp[k]);
            atomic_add_c(a.grad_jones + i2 + k, gq[k]);
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) gV[k] = cadd(gV[k], gM[k]);
      }
    }
    if (live) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        vis_complex o;
        o.re = (vis_real)gV[k].re;
        o.im = (vis_real)gV[k].im;
        a.grad_vis[base + k] = o;
      }
    }
  }
}

// Arguments shared by the adjoint and the prediction (device pointers, sizes from the struct).
AdjointArgs degrid_args(const gridding_parameters &p, int faceting) {
  AdjointArgs a;
  std::memset(&a, 0, sizeof a);
  a.vis = p.visibilities; a.weights = p.visibility_weights; a.flags = (const uint8_t *)p.flags;
  a.uvw = (const vis_real *)p.uvw_coords; a.flagged_rows = (const uint8_t *)p.flagged_rows;
  a.field = p.field_array; a.spw = p.spw_index_array; a.ant1 = p.antenna_1_ids; a.ant2 = p.antenna_2_ids;
  a.time_ids = p.timestamp_ids; a.jones = p.jones_terms;
  a.wavelengths = p.reference_wavelengths; a.enabled = (const uint8_t *)p.enabled_channels; a.cgi = p.channel_grid_indicies;
  a.conv = p.conv; a.facet_centres = p.facet_centres;
  a.nrows = (long long)p.row_count;
  a.nchan = (int)p.channel_count; a.nspw = (int)p.spw_count; a.nant = (int)p.antenna_count;
  a.ntimes = (int)p.no_timestamps_read;
  a.nfacets = (int)(p.num_facet_centres ? p.num_facet_centres : 1);
  a.cube = (int)p.cube_channel_dim_size;
  a.nx = (int)p.nx; a.ny = (int)p.ny;
  a.W = (int)(2 * p.conv_support + 1);
  a.os = (int)p.conv_oversample;
  a.K = (a.W + 2) + (a.W + 1) * (a.os - 1);
  a.P = (int)(p.wplanes > 1 ? p.wplanes : 1);
  a.faceting = faceting ? 1 : 0;
  a.imaging_field = p.imaging_field;
  a.u_scale = (double)p.nx * (double)p.cell_size_x * (double)kArcsecToRad;
  a.v_scale = -((double)p.ny * (double)p.cell_size_y * (double)kArcsecToRad);
  a.gcx = (double)(p.nx / 2 - p.conv_support);
  a.gcy = (double)(p.ny / 2 - p.conv_support);
  a.wmax = (double)(float)p.wmax_est;
  a.ra0 = (double)p.phase_centre_ra;
  a.dec0 = (double)p.phase_centre_dec;
  return a;
}

// Zeroes the output, then one persistent-style launch of the gather (32 rows of a channel per warp pass).
template <bool PREDICT>
int launch_degrid(AdjointArgs a, bool wproj, cudaStream_t st) {
  const size_t head = degrid_warps_offset(a.nfacets, a.P);
  if (head + (size_t)8 * 2 * a.W * sizeof(cplx) > 200 * 1024) return BZ_ERR_UNSUPPORTED;  // facets and planes
  const size_t row = wproj ? degrid_row_bytes<true>(a.K) : degrid_row_bytes<false>(a.K);
  a.row_bytes = head + kDegridWarps * (kDegridSums + row) <= 200 * 1024 ? (int)row : 0;
  const size_t smem = head + kDegridWarps * (kDegridSums + (size_t)a.row_bytes);
  if (cudaMemsetAsync(a.grad_vis, 0, sizeof(vis_complex) * (size_t)a.nrows * a.nchan * 4, st) != cudaSuccess) return BZ_ERR_CUDA;
  if (a.nrows == 0) return BZ_OK;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long warps_needed = (a.nrows + 31) / 32 * a.nchan;  // 32 rows of a channel per warp pass
  const long long blocks = std::min<long long>((warps_needed + kDegridWarps - 1) / kDegridWarps, (long long)sms * 32);
  auto kern = wproj ? degrid_adjoint_kernel<true, PREDICT> : degrid_adjoint_kernel<false, PREDICT>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return BZ_ERR_CUDA;
  kern<<<(unsigned)blocks, kDegridWarps * 32, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? BZ_OK : BZ_ERR_CUDA;
}

// v / c for the single-precision library with c's reciprocal as a pair of floats (r = hi + lo, 48 bits):
// v r in error-free FP32 steps, the FP64 quotient's rounding but for ties.  FP64 divisions, two per value at
// 1/64 of the FP32 rate, took 5.6 ms for 64 slices of 1024^2 (0.16 ms of HBM time).  Values whose product
// is not well inside the normal range are divided in FP64.
#if defined(BULLSEYE_SINGLE)
__device__ __forceinline__ float taper_divide(float v, double c, float hi, float lo, bool pair) {
  const float p = __fmul_rn(v, hi);
  const float m = fabsf(p);
  if (pair && m > 1e-25f && m < 1e37f) return __fadd_rn(p, fmaf(v, lo, fmaf(v, hi, -p)));
  if (v == 0.0f && pair) return p;
  return (float)((double)v / c);
}
#endif

// Model images -> the FFT input: dst[s][y][x] = img[s][(y+ny/2)%ny][(x+nx/2)%nx] / (taper_x[x'] taper_y[y'])
// at the source pixel (x', y') (numpy's ifftshift; the tapers are the gridding correction c(l) c(m)
// that finalize divides by, or null).  A thread takes one pixel of blockIdx.y's slices: its taper once.
__global__ void __launch_bounds__(256) predict_taper_shift_kernel(const vis_complex *__restrict__ img,
                                                                  vis_complex *__restrict__ dst, int nx, int ny,
                                                                  long long slices, const double *__restrict__ taper_x,
                                                                  const double *__restrict__ taper_y) {
  const long long nxy = (long long)nx * ny;
  const long long per = (slices + gridDim.y - 1) / gridDim.y, s0 = blockIdx.y * per, s1 = min(slices, s0 + per);
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < nxy; r += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(r / nx), x = (int)(r - (long long)y * nx);
    const int sy = (y + ny / 2) % ny, sx = (x + nx / 2) % nx;
    const vis_complex *in = img + (long long)sy * nx + sx;
    double c = 1.0;
#if defined(BULLSEYE_SINGLE)
    float hi = 1.f, lo = 0.f;
    bool pair = false;
#endif
    if (taper_x) {
      c = taper_x[sx] * taper_y[sy];
#if defined(BULLSEYE_SINGLE)
      const double q = 1.0 / c;
      hi = (float)q;
      lo = (float)(q - (double)hi);
      pair = fabs(q) > 1e-12 && fabs(q) < 1e12;
#endif
    }
#pragma unroll 4
    for (long long s = s0; s < s1; ++s) {
      vis_complex v = in[s * nxy];
      if (taper_x) {
#if defined(BULLSEYE_SINGLE)
        v.re = taper_divide(v.re, c, hi, lo, pair);
        v.im = taper_divide(v.im, c, hi, lo, pair);
#else
        v.re = v.re / c;
        v.im = v.im / c;
#endif
      }
      dst[s * nxy + r] = v;
    }
  }
}

// After the forward transform: numpy's fftshift, cell (y, x) = src[(y-ny/2)%ny][(x-nx/2)%nx], written
// with the 4 correlations of a cell adjacent, dst[(f cube + g)][y][x][k] for source slice
// (f cube + g) x 4 + k (the gather then reads a cell's correlations with two 16-byte loads).
__global__ void predict_fftshift_kernel(const vis_complex *__restrict__ src, vis_complex *__restrict__ dst, int nx,
                                        int ny, long long slices) {
  const long long nxy = (long long)nx * ny, total = nxy * slices;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i & 3);
    const long long cell = i >> 2, q = cell / nxy, r = cell - q * nxy;
    const int y = (int)(r / nx), x = (int)(r - (long long)y * nx);
    const int sy = (y + ny - ny / 2) % ny, sx = (x + nx - nx / 2) % nx;
    dst[i] = src[(q * 4 + k) * nxy + (long long)sy * nx + sx];
  }
}

// Batched 2-D forward plans, one per (device, ny, nx, batch), kept for the life of the process.
// Plans are shared by host threads: setting the stream and executing happen under the lock.
std::mutex g_plan_mutex;
std::map<std::tuple<int, int, int, int>, cufftHandle> g_plans;

int forward_fft(vis_complex *data, int nx, int ny, int batch, cudaStream_t st) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_plan_mutex);
  const auto key = std::make_tuple(dev, ny, nx, batch);
  auto it = g_plans.find(key);
  if (it == g_plans.end()) {
    cufftHandle plan;
    int dims[2] = {ny, nx};
    const int dist = nx * ny;
#if defined(BULLSEYE_SINGLE)
    const cufftType type = CUFFT_C2C;
#else
    const cufftType type = CUFFT_Z2Z;
#endif
    if (cufftPlanMany(&plan, 2, dims, nullptr, 1, dist, nullptr, 1, dist, type, batch) != CUFFT_SUCCESS) return BZ_ERR_CUFFT;
    it = g_plans.emplace(key, plan).first;
  }
  if (cufftSetStream(it->second, st) != CUFFT_SUCCESS) return BZ_ERR_CUFFT;
#if defined(BULLSEYE_SINGLE)
  const cufftResult r = cufftExecC2C(it->second, (cufftComplex *)data, (cufftComplex *)data, CUFFT_FORWARD);
#else
  const cufftResult r = cufftExecZ2Z(it->second, (cufftDoubleComplex *)data, (cufftDoubleComplex *)data, CUFFT_FORWARD);
#endif
  return r == CUFFT_SUCCESS ? BZ_OK : BZ_ERR_CUFFT;
}

constexpr int kPredictNormalise = 1;
constexpr int kPredictFromGrid = 2;

}  // namespace

// See include/bullseye_gb300.h.  Every pointer is a device pointer (as for the allocation-free
// gridding entry); jones_terms holds the raw (not inverted) terms or is null.
extern "C" int bullseye_grid_adjoint(const gridding_parameters *params, const void *grad_grid, void *grad_vis,
                                     void *grad_jones, int faceting, void *stream) {
  const char *name = "bullseye_grid_adjoint";
  if (!params || !grad_grid || !grad_vis) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: params, grad_grid and grad_vis are required", name);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  const gridding_parameters &p = *params;
  if (p.number_of_polarization_terms != 4 || p.number_of_polarization_terms_being_gridded != 4 || !p.visibilities ||
      !p.uvw_coords || !p.visibility_weights || !p.flags || !p.flagged_rows || !p.field_array || !p.spw_index_array ||
      !p.conv || !p.reference_wavelengths || !p.enabled_channels || !p.channel_grid_indicies ||
      (p.jones_terms && (!p.antenna_1_ids || !p.antenna_2_ids || !p.timestamp_ids))) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: four polarisation terms and the row and table arrays are required", name);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  AdjointArgs a = degrid_args(p, faceting);
  a.grad_grid = (const vis_complex *)grad_grid;
  a.grad_vis = (vis_complex *)grad_vis;
  a.grad_jones = p.jones_terms ? (vis_complex *)grad_jones : nullptr;
  const int rc = launch_degrid<false>(a, p.wplanes > 1, static_cast<cudaStream_t>(stream));
  if (rc != BZ_OK) bz_record_error(rc, "%s: launch failed (status %d)", name, rc);
  return rc;
}

// See include/bullseye_gb300.h.
extern "C" size_t bullseye_predict_ws_bytes(const gridding_parameters *params) {
  if (!params) return 0;
  const gridding_parameters &p = *params;
  const size_t F = p.num_facet_centres ? p.num_facet_centres : 1;
  return 2 * F * p.cube_channel_dim_size * 4 * p.nx * p.ny * sizeof(vis_complex);
}

// See include/bullseye_gb300.h.
extern "C" int bullseye_predict(const gridding_parameters *params, const void *model, const double *taper_x,
                                const double *taper_y, int faceting, int flags, void *vis_out, void *workspace,
                                size_t ws_bytes, void *stream) {
  const char *name = "bullseye_predict";
  if (!params || !model || !vis_out) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: params, model and vis_out are required", name);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  const gridding_parameters &p = *params;
  if (p.number_of_polarization_terms != 4 || p.number_of_polarization_terms_being_gridded != 4 || !p.uvw_coords ||
      !p.spw_index_array || !p.conv || !p.reference_wavelengths || !p.enabled_channels || !p.channel_grid_indicies ||
      (p.jones_terms && (!p.antenna_1_ids || !p.antenna_2_ids || !p.timestamp_ids)) || p.nx == 0 || p.ny == 0 ||
      p.cube_channel_dim_size == 0 || p.conv_oversample == 0 || (flags & ~(kPredictNormalise | kPredictFromGrid))) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: four polarisation terms, uvw, spw and the tables are required", name);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  if ((taper_x == nullptr) != (taper_y == nullptr)) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: give both gridding-correction tapers or neither", name);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  const bool from_grid = (flags & kPredictFromGrid) != 0;
  const size_t need = from_grid ? 0 : bullseye_predict_ws_bytes(params);
  if (need && (!workspace || ws_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))) {
    bz_record_error(BZ_ERR_INVALID_ARGUMENT, "%s: workspace of %zu bytes at %p, need %zu bytes 256-byte aligned", name,
                    ws_bytes, workspace, need);
    return BZ_ERR_INVALID_ARGUMENT;
  }
  const size_t F = p.num_facet_centres ? p.num_facet_centres : 1;
  const long long slices = (long long)(F * p.cube_channel_dim_size * 4);
  if (!from_grid && ((long long)p.nx * (long long)p.ny > 0x7fffffffLL || slices > 0x7fffffffLL)) {
    bz_record_error(BZ_ERR_UNSUPPORTED, "%s: %lld model slices of %zu x %zu exceed one batched transform", name, slices,
                    p.nx, p.ny);
    return BZ_ERR_UNSUPPORTED;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const vis_complex *grids = static_cast<const vis_complex *>(model);
  if (!from_grid) {
    vis_complex *buf = static_cast<vis_complex *>(workspace);
    vis_complex *out = buf + (size_t)slices * p.nx * p.ny;
    // about 300 K threads: pixels, and the slices in as many parts as small images leave room for
    const long long nxy = (long long)p.nx * (long long)p.ny;
    const unsigned pixels = (unsigned)std::min<long long>((nxy + 255) / 256, 4096);
    const unsigned parts = (unsigned)std::max<long long>(1, std::min<long long>(slices, 1216 / pixels));
    predict_taper_shift_kernel<<<dim3(pixels, parts), 256, 0, st>>>(grids, buf, (int)p.nx, (int)p.ny, slices, taper_x, taper_y);
    int rc = cudaGetLastError() == cudaSuccess ? BZ_OK : BZ_ERR_CUDA;
    if (rc == BZ_OK) rc = forward_fft(buf, (int)p.nx, (int)p.ny, (int)slices, st);
    if (rc == BZ_OK) {
      predict_fftshift_kernel<<<2048, 256, 0, st>>>(buf, out, (int)p.nx, (int)p.ny, slices);
      rc = cudaGetLastError() == cudaSuccess ? BZ_OK : BZ_ERR_CUDA;
    }
    if (rc != BZ_OK) {
      bz_record_error(rc, "%s: model transform failed (status %d)", name, rc);
      return rc;
    }
    grids = out;
  }
  AdjointArgs a = degrid_args(p, faceting);
  a.grad_grid = grids;
  a.grid_interleaved = from_grid ? 0 : 1;  // the model grids made above interleave the correlations
  a.grad_vis = static_cast<vis_complex *>(vis_out);
  a.normalise = (flags & kPredictNormalise) ? 1 : 0;
  const int rc = launch_degrid<true>(a, p.wplanes > 1, st);
  if (rc != BZ_OK) bz_record_error(rc, "%s: launch failed (status %d)", name, rc);
  return rc;
}
