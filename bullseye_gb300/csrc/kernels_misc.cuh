// Small device kernels around the gridder: Jones inversion, the grids' two forms,
// and the finalize (shift / real-part packing / gridding correction) passes.
#pragma once
#include "common.h"

namespace bz {

// Time-innermost position of term i of a [T][A][F][S][Ch] table: [A][S][Ch][F][T].
struct JonesDims {
  long long T, A, F, S, C;
};
__device__ __forceinline__ long long jones_time_major(long long i, const JonesDims &d) {
  const long long c = i % d.C;
  long long r = i / d.C;
  const long long s = r % d.S;
  r /= d.S;
  const long long f = r % d.F;
  r /= d.F;
  const long long a = r % d.A;
  const long long t = r / d.A;
  return (((a * d.S + s) * d.C + c) * d.F + f) * d.T + t;
}

// Invert every 2x2 Jones matrix (jones_2x2.h:86-126).  Singular matrices (determinant exactly
// zero) are replaced by zeros and flagged; the reference throws instead.  With out_t, each
// inverse is also written time-innermost (the record kernel's copy).
__global__ void invert_jones_kernel(const vis_complex *__restrict__ in, vis_complex *__restrict__ out,
                                    long long n, int *error, vis_complex *__restrict__ out_t = nullptr,
                                    JonesDims dims = JonesDims{0, 0, 0, 0, 0}) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  vis_complex *o2 = out_t ? out_t + 4 * jones_time_major(i, dims) : nullptr;
  typedef vis_real T;
  vis_complex a = in[4 * i], b = in[4 * i + 1], c = in[4 * i + 2], d = in[4 * i + 3];
  T dr = (a.re * d.re - a.im * d.im) - (b.re * c.re - b.im * c.im);
  T di = (a.re * d.im + a.im * d.re) - (b.re * c.im + b.im * c.re);
  vis_complex z = {0, 0};
  if (dr == (T)0 && di == (T)0) {
    atomicOr(error, 4);
    out[4 * i] = z; out[4 * i + 1] = z; out[4 * i + 2] = z; out[4 * i + 3] = z;
    if (o2) { o2[0] = z; o2[1] = z; o2[2] = z; o2[3] = z; }
    return;
  }
  // 1 / det with scaling (Smith's method) to avoid overflow
  T ir, ii;
  if (fabs((double)dr) >= fabs((double)di)) {
    T r = di / dr, den = dr + di * r;
    ir = (T)1 / den;
    ii = -r / den;
  } else {
    T r = dr / di, den = dr * r + di;
    ir = r / den;
    ii = (T)-1 / den;
  }
  auto mul = [](vis_complex x, T yr, T yi) {
    vis_complex o;
    o.re = x.re * yr - x.im * yi;
    o.im = x.re * yi + x.im * yr;
    return o;
  };
  const vis_complex r0 = mul(d, ir, ii), r1 = mul(b, -ir, -ii), r2 = mul(c, -ir, -ii), r3 = mul(a, ir, ii);
  out[4 * i] = r0;
  out[4 * i + 1] = r1;
  out[4 * i + 2] = r2;
  out[4 * i + 3] = r3;
  if (o2) { o2[0] = r0; o2[1] = r1; o2[2] = r2; o2[3] = r3; }
}

#if defined(BULLSEYE_SINGLE)
// The two forms of a single-precision grid: *narrow*, a value is hi + lo of two FP32 complex words, and
// *wide*, the form that the wide accumulation adds to: the 8 bytes of hi hold the FP64 real part, those of
// lo the imaginary part.  A conversion works in place, on both words of a cell at once.  A zero cell has
// the same bits in both forms and is left alone: most of a grid is zero (the tracks of a bench facet
// cover 6 % of it), the kernels then read 16 bytes a cell (HBM), and the FP64 pipe is kept for the rest.
__device__ __forceinline__ bool widen_cell(uint2 &h, uint2 &l) {
  if ((h.x | h.y | l.x | l.y) == 0) return false;
  // (-0 + 0 is +0: a cell without a second word keeps its sign)
  double re = (double)__uint_as_float(h.x), im = (double)__uint_as_float(h.y);
  if (l.x) re += (double)__uint_as_float(l.x);
  if (l.y) im += (double)__uint_as_float(l.y);
  h = make_uint2((unsigned)__double2loint(re), (unsigned)__double2hiint(re));
  l = make_uint2((unsigned)__double2loint(im), (unsigned)__double2hiint(im));
  return true;
}
__device__ __forceinline__ bool narrow_cell(uint2 &h, uint2 &l) {
  if ((h.x | h.y | l.x | l.y) == 0) return false;
  const double re = __hiloint2double((int)h.y, (int)h.x), im = __hiloint2double((int)l.y, (int)l.x);
  const float a = (float)re, b = (float)im;
  // what is not finite has no second word: inf - inf would turn an infinity that lies in the grid into NaN
  const float a2 = isfinite(a) ? (float)(re - (double)a) : 0.f;
  const float b2 = isfinite(b) ? (float)(im - (double)b) : 0.f;
  h = make_uint2(__float_as_uint(a), __float_as_uint(b));
  l = make_uint2(__float_as_uint(a2), __float_as_uint(b2));
  return true;
}
// Both directions over n cells, eight cells per thread in flight (16-byte loads of two cells when both
// buffers allow them, cell by cell otherwise).
template <bool WIDEN>
__global__ void __launch_bounds__(256) convert_grid_kernel(vis_complex *hi, vis_complex *lo, long long n) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  auto one = [](uint2 &h, uint2 &l) { return WIDEN ? widen_cell(h, l) : narrow_cell(h, l); };
  long long done = 0;
  if (((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15) == 0) {
    uint4 *ph = reinterpret_cast<uint4 *>(hi), *pl = reinterpret_cast<uint4 *>(lo);
    const long long pairs = n / 2;
    // whole warps stay in the loop: a stretch whose cells are all zero is passed by on a vote (on each lane's
    // own test the FP64 path was evaluated ahead of it, 6 FP64 operations for every zero cell: 28.5 us for the
    // 2 million cells of a snapshot's facets, 12.5 for the way back)
    for (long long i0 = tid - (threadIdx.x & 31); i0 < pairs; i0 += 4 * nt) {
      const long long i = i0 + (threadIdx.x & 31);
      uint4 h[4], l[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + q * nt < pairs) {
          h[q] = ph[i + q * nt];
          l[q] = pl[i + q * nt];
        } else {
          h[q] = l[q] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned bits = h[q].x | h[q].y | h[q].z | h[q].w | l[q].x | l[q].y | l[q].z | l[q].w;
        if (!__any_sync(0xffffffffu, bits != 0)) continue;
        uint2 h0 = make_uint2(h[q].x, h[q].y), h1 = make_uint2(h[q].z, h[q].w);
        uint2 l0 = make_uint2(l[q].x, l[q].y), l1 = make_uint2(l[q].z, l[q].w);
        const bool c0 = one(h0, l0), c1 = one(h1, l1);
        if (c0 || c1) {
          ph[i + q * nt] = make_uint4(h0.x, h0.y, h1.x, h1.y);
          pl[i + q * nt] = make_uint4(l0.x, l0.y, l1.x, l1.y);
        }
      }
    }
    done = 2 * pairs;
  }
  for (long long i = done + tid; i < n; i += nt) {
    uint2 h = reinterpret_cast<uint2 *>(hi)[i], l = reinterpret_cast<uint2 *>(lo)[i];
    if (one(h, l)) {
      reinterpret_cast<uint2 *>(hi)[i] = h;
      reinterpret_cast<uint2 *>(lo)[i] = l;
    }
  }
}
// The same for a grid without a second word yet (lo is written).
__global__ void __launch_bounds__(256) widen_grid_new_kernel(vis_complex *hi, vis_complex *lo, long long n) {
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n;
       i0 += (long long)gridDim.x * blockDim.x) {
    const long long i = i0 + lane;
    uint2 h = make_uint2(0, 0);
    if (i < n) h = reinterpret_cast<const uint2 *>(hi)[i];
    double im = 0.0;
    if (__any_sync(0xffffffffu, (h.x | h.y) != 0) && (h.x | h.y)) {
      reinterpret_cast<double *>(hi)[i] = (double)__uint_as_float(h.x);
      im = (double)__uint_as_float(h.y);
    }
    if (i < n) reinterpret_cast<double *>(lo)[i] = im;
  }
}
#endif

// The value of cell i of an accumulated grid: hi + lo, or the rounded wide value.
__device__ __forceinline__ vis_complex grid_value(const vis_complex *hi, const vis_complex *lo, bool wide, long long i) {
  vis_complex h;
#if defined(BULLSEYE_SINGLE)
  if (wide) {
    uint2 a = reinterpret_cast<const uint2 *>(hi)[i], b = reinterpret_cast<const uint2 *>(lo)[i];
    narrow_cell(a, b);
    h.re = __uint_as_float(a.x) + __uint_as_float(b.x);
    h.im = __uint_as_float(a.y) + __uint_as_float(b.y);
    return h;
  }
#endif
  h = hi[i];
  if (lo) {
    h.re += lo[i].re;
    h.im += lo[i].im;
  }
  return h;
}

// out = the accumulated grid's values (out may be hi).  Wide grids go two cells per load, eight in flight,
// and pass by the FP64 path where a warp's cells are all zero (cell by cell, with the conversions evaluated
// for zero cells too, the 16 facets of 1024^2 cells x 4 correlations took 546 us; 239 so, the HBM time).
__global__ void __launch_bounds__(256) resolve_grid_kernel(const vis_complex *hi, const vis_complex *lo, bool wide,
                                                           vis_complex *out, long long n) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  long long done = 0;
#if defined(BULLSEYE_SINGLE)
  if (wide && ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo) | reinterpret_cast<uintptr_t>(out)) &
               15) == 0) {
    const long long pairs = n / 2;
    for (long long i0 = tid - (threadIdx.x & 31); i0 < pairs; i0 += 4 * nt) {
      const long long i = i0 + (threadIdx.x & 31);
      uint4 h[4], l[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        h[q] = l[q] = make_uint4(0, 0, 0, 0);
        if (i + q * nt < pairs) {
          h[q] = reinterpret_cast<const uint4 *>(hi)[i + q * nt];
          l[q] = reinterpret_cast<const uint4 *>(lo)[i + q * nt];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 r = make_uint4(0, 0, 0, 0);
        const unsigned bits = h[q].x | h[q].y | h[q].z | h[q].w | l[q].x | l[q].y | l[q].z | l[q].w;
        if (__any_sync(0xffffffffu, bits != 0)) {
          uint2 h0 = make_uint2(h[q].x, h[q].y), h1 = make_uint2(h[q].z, h[q].w);
          uint2 l0 = make_uint2(l[q].x, l[q].y), l1 = make_uint2(l[q].z, l[q].w);
          narrow_cell(h0, l0);
          narrow_cell(h1, l1);
          r = make_uint4(__float_as_uint(__uint_as_float(h0.x) + __uint_as_float(l0.x)),
                         __float_as_uint(__uint_as_float(h0.y) + __uint_as_float(l0.y)),
                         __float_as_uint(__uint_as_float(h1.x) + __uint_as_float(l1.x)),
                         __float_as_uint(__uint_as_float(h1.y) + __uint_as_float(l1.y)));
        }
        if (i + q * nt < pairs) reinterpret_cast<uint4 *>(out)[i + q * nt] = r;
      }
    }
    done = 2 * pairs;
  }
#endif
  for (long long i = done + tid; i < n; i += nt) out[i] = grid_value(hi, lo, wide, i);
}

// out[f][i] = init[f][i] + the accumulated value of cell i, for f < nf, i < per: a facet-invariant
// contribution added to every facet's initial grid.
__global__ void broadcast_add_kernel(const vis_complex *__restrict__ init, const vis_complex *__restrict__ hi,
                                     const vis_complex *__restrict__ lo, bool wide, vis_complex *__restrict__ out,
                                     long long per, long long nf) {
  const long long total = per * nf;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const vis_complex h = grid_value(hi, lo, wide, i % per);
    vis_complex o = init[i];
    o.re += h.re;
    o.im += h.im;
    out[i] = o;
  }
}

// Gather with the inverse shift of numpy's ifftshift: dst[y][x] = src[(y+ny/2)%ny][(x+nx/2)%nx]
// for each of `slices` planes.  Equivalent to bullseye/mo/cpu_gpu_common/fft_shift_utils.cpp:75-111.
// Stokes (or correlation) term of every (facet, cube slice): dst[f][c] = (src[f][c][a] +
// sign * src[f][c][b]) / 2 over nxy cells, from facet blocks of `cube` x `corr` slices into
// compact [facet][cube] slices (bullseye/data/stokes.py:90-172 combines the same pairs on the host).
__global__ void stokes_combine_kernel(const vis_complex *__restrict__ src, vis_complex *__restrict__ dst, long long nxy,
                                      int facets, int cube, int corr, int a, int b, int sign) {
  const long long total = (long long)facets * cube * nxy;
  const vis_real half = (vis_real)0.5, sg = (vis_real)sign;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long fc = i / nxy, r = i - fc * nxy;
    const long long base = fc * corr * nxy + r;  // slice (f, c, 0) of the facet block
    const vis_complex va = src[base + (long long)a * nxy], vb = src[base + (long long)b * nxy];
    vis_complex o;
    o.re = (va.re + sg * vb.re) * half;
    o.im = (va.im + sg * vb.im) * half;
    dst[i] = o;
  }
}

__global__ void ifftshift_gather_kernel(const vis_complex *__restrict__ src, vis_complex *__restrict__ dst, int nx,
                                        int ny, long long slices) {
  long long nxy = (long long)nx * ny;
  long long total = nxy * slices;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long s = i / nxy, r = i - s * nxy;
    int y = (int)(r / nx), x = (int)(r - (long long)y * nx);
    int sy = (y + ny / 2) % ny, sx = (x + nx / 2) % nx;
    dst[i] = src[s * nxy + (long long)sy * nx + sx];
  }
}

// After the transform: fftshift (dst[y][x] = src[(y-ny/2)%ny][(x-nx/2)%nx]) into `shifted`,
// and the float32 real parts into `packed`, optionally divided by the separable gridding
// correction corr_x[x] * corr_y[y].
__global__ void fftshift_pack_kernel(const vis_complex *__restrict__ src, vis_complex *__restrict__ shifted,
                                     float *__restrict__ packed, int nx, int ny, long long slices,
                                     const double *__restrict__ corr_x, const double *__restrict__ corr_y) {
  long long nxy = (long long)nx * ny;
  long long total = nxy * slices;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long s = i / nxy, r = i - s * nxy;
    int y = (int)(r / nx), x = (int)(r - (long long)y * nx);
    int sy = (y + ny - ny / 2) % ny, sx = (x + nx - nx / 2) % nx;
    vis_complex v = src[s * nxy + (long long)sy * nx + sx];
    if (shifted) shifted[i] = v;
    double re = (double)v.re;
    if (corr_x) re = re / (corr_x[x] * corr_y[y]);
    packed[i] = (float)re;
  }
}

// FP32 FMA throughput probe: kFmaProbeChains independent dependency chains per thread.
constexpr int kFmaProbeChains = 16;
__global__ void fma_probe_kernel(float *out, int iters) {
  float acc[kFmaProbeChains];
#pragma unroll
  for (int k = 0; k < kFmaProbeChains; ++k) acc[k] = (float)(threadIdx.x + k) * 1e-3f;
  const float m = 0.999999f, a = 1e-7f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < kFmaProbeChains; ++k) acc[k] = fmaf(acc[k], m, a);
  }
  float s = 0;
#pragma unroll
  for (int k = 0; k < kFmaProbeChains; ++k) s += acc[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace bz
