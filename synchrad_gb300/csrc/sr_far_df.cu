// Double-float far-field radiation integral for GB300 (sm_103a): spectra of
// FP64 accuracy computed on the FP32 pipe (precision SR_PREC_DF).
//
// The sum is the reference's (synchrad/kernel_farfield.cl:59-107) in the form
// the mixed kernel uses (sr_far_mixed.cu): A carried on theta-hat and phi-hat,
// tau = (t - z) + (1 - cos theta) z - n_x x - n_y y, the |dphase| < pi mask
// decided from |omega| |dtau| with a guard band and the reference's own FP64
// test inside it.  What changes is the arithmetic of every per-point term,
// which here keeps about 48 significant bits (double-float: value = hi + lo):
//  * per (direction, step), in FP64: tau, |dtau|, the amplitude on theta-hat
//    and phi-hat, and the phase d_omega * tau in revolutions, whose whole turns
//    are dropped exactly; the rotations R = exp(i d_omega tau) and R^2 as
//    double-floats;
//  * per lane and step: the phase of its first point, omega_0 tau, from a
//    double-float frequency and tau, whole turns dropped, and exp(2 pi i f) of
//    the fraction f from a 1024-entry double-float table of exp(2 pi i k/1024)
//    times a Taylor step over the remaining |2 pi r| <= pi/1024;
//  * the lane's K points in pairs: rotation of a pair by R^2 and the four
//    accumulations A_theta, A_phi (re, im) as packed double-float arithmetic
//    (FFMA2 / FADD2 / FMUL2 error-free transformations);
//  * per-track |A|^2 (or the comp's components) in FP64 into per-subset
//    partial spectra, added in fixed order: deterministic results.
// The accumulators keep a hi sum with its TwoSum errors, product errors and
// cross terms gathered in a lo sum: after N steps the sum is accurate to about
// N 2^-48 of the terms' magnitudes.
//
// Decomposition: a warp owns 32/L directions and, for each, an omega tile of
// L*K points; a CTA of kDW warps owns kDW consecutive warp tasks and one track
// subset; one CTA per (task group, subset) item.  Every warp reads the FP64
// step records of its subset directly (one record per lane per 32-step chunk,
// coalesced) and broadcasts its per-(direction, step) setup through shared
// memory.  Nothing waits on another CTA or on an asynchronous copy.
//
// On even omega axes the steps that include a whole band are summed by
// transforms (df_spread_kernel, df_transform_kernel) and far_df_kernel adds the
// others.
#include <algorithm>
#include <cmath>

#include "sr_common.cuh"
#include "sr_internal.h"
#include "sr_fast_sum.cuh"
#include "sr_mixed_common.cuh"

namespace sr {
namespace {

constexpr int kDW = 8;           // warps per CTA
constexpr int kTabBits = 10;
constexpr int kTab = 1 << kTabBits;  // exp(2 pi i k / kTab) table entries
constexpr int kDMaxDpw = 4;      // directions per warp
constexpr int kDSetupF4 = 4;     // float4 per (direction, step) in the setup

// Per-step record in FP64 (96 bytes): q = t - z, x, y, z, bbar (3),
// 1 - bbar_z, a (3) as in the mixed records (far_prepass_kernel), unrounded.
struct __align__(16) DfRecord {
  double q, x, y, z, bx, by, bz, omb, ax, ay, az, pad;
};

template <typename TT>
__global__ void df_prepass_kernel(FarMixedParams p, DfRecord *rec) {
  const TT *X = (const TT *)p.x, *Y = (const TT *)p.y, *Z = (const TT *)p.z;
  const TT *UX = (const TT *)p.ux, *UY = (const TT *)p.uy, *UZ = (const TT *)p.uz;
  const double dtInv = 1.0 / p.dt;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < p.total_steps;
       g += (int64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = p.n_tracks;  // track of step g: last t with offsets[t] <= g
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (p.offsets[mid] <= g) lo = mid; else hi = mid;
    }
    const uint32_t t = lo;
    const int64_t base = p.offsets[t];
    const int64_t n = p.offsets[t + 1] - base;
    const int64_t s = g - base;
    DfRecord r;
    if (s + 1 >= n) {
      r.q = r.x = r.y = r.z = r.bx = r.by = r.bz = r.omb = r.ax = r.ay = r.az = r.pad = 0.0;
      rec[g] = r;
      continue;
    }
    const double time = (double)(uint32_t)(p.it_start[t] + (uint32_t)s) * p.dt;
    r.x = (double)X[g];
    r.y = (double)Y[g];
    r.z = (double)Z[g];
    r.q = time - r.z;
    double b0[3], b1[3], omb[2];
    for (int k = 0; k < 2; ++k) {
      const double ux = (double)UX[g + k], uy = (double)UY[g + k], uz = (double)UZ[g + k];
      const double tr = ux * ux + uy * uy;
      const double gam = sqrt(1.0 + (tr + uz * uz));
      const double gi = 1.0 / gam;
      double *b = k ? b1 : b0;
      b[0] = ux * gi; b[1] = uy * gi; b[2] = uz * gi;
      omb[k] = (uz > 0.0) ? (1.0 + tr) / (gam * (gam + uz)) : (gam - uz) * gi;
    }
    r.bx = 0.5 * (b1[0] + b0[0]);
    r.by = 0.5 * (b1[1] + b0[1]);
    r.bz = 0.5 * (b1[2] + b0[2]);
    r.omb = 0.5 * (omb[0] + omb[1]);
    r.ax = (b1[0] - b0[0]) * dtInv;
    r.ay = (b1[1] - b0[1]) * dtInv;
    r.az = (b1[2] - b0[2]) * dtInv;
    r.pad = 0.0;
    rec[g] = r;
  }
}

// tau = t - n.x of a step, the same to the last bit wherever it is formed.
__device__ __forceinline__ double df_tau(double q, double x, double y, double z, double omc,
                                         double n0, double n1) {
  return __fma_rn(-n1, y, __fma_rn(-n0, x, __fma_rn(omc, z, q)));
}

// exp(2 pi i k / kTab) = (cos hi, cos lo, sin hi, sin lo), from FP64 sincospi.
__global__ void df_table_kernel(float4 *tab) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < kTab) {
    double s, c;
    sincospi(2.0 * (double)k / (double)kTab, &s, &c);
    const df ch = df_from_double(c), sh = df_from_double(s);
    tab[k] = make_float4(ch.hi, ch.lo, sh.hi, sh.lo);
  }
}

// exp(2 pi i f) for a double-float fraction |f| <= 1/2 (+ a few ulp):
// table entry k = rint(f kTab) times exp(i theta), theta = 2 pi (f - k/kTab),
// |theta| <= pi/kTab: sin = theta - theta^3/6, cos = 1 - theta^2/2 + theta^4/24
// (the first dropped terms are below 3e-15).
__device__ __forceinline__ void df_cis(const float4 *tab, df f, df &c, df &s) {
  const float kf = rintf(f.hi * (float)kTab);
  const float4 T = tab[((int)kf) & (kTab - 1)];
  const df r = two_sum(f.hi - kf * (1.0f / (float)kTab), f.lo);  // the difference is exact
  const df th = df_mul(df{SR_TWO_PI_HI, SR_TWO_PI_LO}, r);
  const float t2 = th.hi * th.hi;
  float e2 = __fmaf_rn(th.hi, th.hi, -t2);
  e2 = __fmaf_rn(2.0f * th.hi, th.lo, e2);  // theta^2 = t2 + e2
  const df sn = fast_two_sum(th.hi, th.lo - th.hi * t2 * (1.0f / 6.0f));
  df cs = two_sum(1.0f, -0.5f * t2);
  cs.lo += t2 * t2 * (1.0f / 24.0f) - 0.5f * e2;
  cs = fast_two_sum(cs.hi, cs.lo);
  const df Tc{T.x, T.y}, Ts{T.z, T.w};
  c = df_sub(df_mul(Tc, cs), df_mul(Ts, sn));
  s = df_add(df_mul(Tc, sn), df_mul(Ts, cs));
}

// Whole revolutions of a double-float phase dropped: the fraction in about
// [-1/2, 1/2] (hi - rint(hi) is exact).
__device__ __forceinline__ df df_frac(df r) {
  const float n = rintf(r.hi);
  return two_sum(r.hi - n, r.lo);
}

// ---- packed double-float pairs (two points per register pair) ----
struct df2 {
  float2 hi, lo;
};
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {  // a - b, one rounding
  return __ffma2_rn(b, f2(-1.0f), a);
}
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s, float2 &e) {
  s = __fadd2_rn(a, b);
  const float2 bb = sub2(s, a);
  e = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}
// acc += a z for a double-float scalar a = (ah, al) broadcast (nah = -ah).
__device__ __forceinline__ void df2_acc(df2 &acc, float2 ah, float2 al, float2 nah,
                                        const df2 &z) {
  const float2 p = __fmul2_rn(ah, z.hi);
  const float2 ne = __ffma2_rn(nah, z.hi, p);  // p - ah z.hi: the product's error, negated
  const float2 cr = __ffma2_rn(ah, z.lo, __fmul2_rn(al, z.hi));
  float2 s, e;
  two_sum2(acc.hi, p, s, e);
  acc.hi = s;
  acc.lo = __fadd2_rn(acc.lo, __fadd2_rn(e, sub2(cr, ne)));
}
// a x + b y for pairs a, b and per-slot double-floats x, y (nxh = -x.hi,
// nyh = -y.hi), renormalised.
__device__ __forceinline__ df2 df2_dot(const df2 &a, float2 xh, float2 xl, float2 nxh,
                                       const df2 &b, float2 yh, float2 yl, float2 nyh) {
  const float2 p1 = __fmul2_rn(a.hi, xh);
  const float2 ne1 = __ffma2_rn(a.hi, nxh, p1);
  const float2 p2 = __fmul2_rn(b.hi, yh);
  const float2 ne2 = __ffma2_rn(b.hi, nyh, p2);
  float2 s, e;
  two_sum2(p1, p2, s, e);
  float2 cr = __ffma2_rn(a.hi, xl, __fmul2_rn(a.lo, xh));
  cr = __ffma2_rn(b.hi, yl, __ffma2_rn(b.lo, yh, cr));
  const float2 lo = __fadd2_rn(e, sub2(cr, __fadd2_rn(ne1, ne2)));
  df2 r;
  r.hi = __fadd2_rn(s, lo);
  r.lo = sub2(lo, sub2(r.hi, s));
  return r;
}

// Per-direction constants of a work item.
struct DirConstDf {
  double sT, cT, sPh, cPh, n0, n1, omc;  // omc = 1 - cos(theta)
  double tprev;                          // tau of the step before the current chunk
};

// ------------------------------------------------------------------------
// Even frequency axes: the sum over the steps by transforms, as in the mixed
// kernels (sr_fast_sum.cuh) but to this precision: 14 taps of a Kaiser-Bessel
// kernel (aliasing 1e-13) in double-float, the circle and its FFT in FP64.
//   df_spread_kernel: a lane is a direction, a warp walks a segment of a track;
//     the 14 cells around the step stay in registers as double-floats, a cell
//     that the step leaves is added to the circle in FP64.  A tap is its Taylor
//     polynomial about the nearest of 128 nodes a cell, double-float where the
//     term needs it.
//   df_transform_kernel: a block sums the circles of a (track, direction, band),
//     transforms both components and leaves A in place of the circle.
//   far_df_kernel<., true> adds the steps whose band the |dphase| < pi rule cuts.
// ------------------------------------------------------------------------
constexpr int kDTaps = 14, kDPairs = kDTaps / 2;
constexpr int kDNodes = 128;
constexpr int kDRow = 4 * kDPairs + 1;  // float4 per node; odd: lanes at different
                                        // nodes read different banks
constexpr double kDBeta = 32.87;        // pi sqrt((taps / 2)^2 (2 - 1/2)^2 - 0.8)
constexpr int kDSeries = 52;            // terms of I0 at kDBeta
constexpr int kDSpreadWarps = 4;

struct DfFast {
  // [0] the axis is not even, [1] sampled steps that the phase limit cuts
  unsigned int *uneven;
  float4 *taps;          // [kDNodes + 1][kDRow] Taylor coefficients, pairs of taps
  double *deconv;        // [257] 1 / transform of the kernel, |index from the centre|
  double2 *twiddle;      // [M] exp(2 pi i k / M)
  unsigned int *cut;     // [chunks of 32 steps][n_dwb] directions with a cut step
  unsigned int *any;     // [n_tracks][n_dwb]
  double *cells;         // [n_segs][n_dwb][32][M][4] circles, then A
  uint32_t n_bands, nb, M, n_dwb, n_segs, seg_steps;
  uint32_t batch;        // tracks at a time
};

__device__ __forceinline__ uint32_t df_first_segment(const FarMixedParams &p, const DfFast &f,
                                                     uint32_t t) {
  return (uint32_t)((uint64_t)p.offsets[t] / f.seg_steps -
                    (uint64_t)p.offsets[0] / f.seg_steps) + t;
}

// Index of cell (or frequency) j of a track's first circle of a direction.
__device__ __forceinline__ uint64_t df_cell(const FarMixedParams &p, const DfFast &f, uint32_t t,
                                            uint32_t dir, uint32_t band, uint32_t j) {
  const uint64_t unit =
      (uint64_t)df_first_segment(p, f, t) * f.n_dwb + (dir / 32u) * f.n_bands + band;
  return ((unit * 32u + dir % 32u) * f.M + j) * 4u;
}

// Whether the transforms are taken.  Where the |dphase| < pi rule cuts more than a
// sixth of the sampled (direction, step) pairs, the cut steps' kernel would walk
// most chunks anyway and everything is left to the term-by-term kernel (20 tracks,
// 900 steps of which 9 make a period, 144 directions, 100 frequencies: 3.5 ms with the
// transforms, 2.7 without; 40 tracks of 1200 steps, 16 a period, a quarter cut, 144
// directions, 16 frequencies: 4.7 and 3.7).
constexpr uint32_t kDSamples = 1024;
__device__ __forceinline__ bool df_by_transform(const DfFast &f) {
  return f.uneven[0] == 0u && 6u * f.uneven[1] <= kDSamples;
}

// Largest |omega| of a band.
__device__ __forceinline__ float df_band_max(const FarMixedParams &p, const DfFast &f,
                                             uint32_t band) {
  const uint32_t j0 = band * f.nb, j1 = min(j0 + f.nb, p.n_omega) - 1u;
  return (float)fmax(fabs(p.omega[j0]), fabs(p.omega[j1]));
}

// Tables, whether the axis is even (one thread per entry), and the sampled steps (the
// first kDSamples threads).
__global__ void __launch_bounds__(32) df_fast_tables_kernel(FarMixedParams p, DfFast f,
                                                            const DfRecord *rec, double c_last,
                                                            double inv_i0) {
  const uint32_t n = p.n_omega;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kDSamples) {  // whole warps
    const uint32_t nT = p.n_theta, n_dirs = nT * p.n_phi;
    const uint32_t t = (uint32_t)((uint64_t)i * p.n_tracks / kDSamples);
    const uint32_t nb = track_body(p, t);
    bool cut = false;
    if (nb > 1) {
      const uint32_t s = 1u + (i * 2654435761u >> 8) % (nb - 1u), d = (i * 40503u) % n_dirs;
      const uint32_t iT = d % nT, iP = d / nT;
      const double omc = 1.0 - p.cos_theta[iT], n0 = p.sin_theta[iT] * p.cos_phi[iP],
                   n1 = p.sin_theta[iT] * p.sin_phi[iP];
      const DfRecord &a = rec[p.offsets[t] + s], &b = rec[p.offsets[t] + s - 1];
      const float adt = (float)fabs(df_tau(a.q, a.x, a.y, a.z, omc, n0, n1) -
                                    df_tau(b.q, b.x, b.y, b.z, omc, n0, n1));
      const double wa = p.omega[0], wb = p.omega[n - 1u];
      const float wmin = (wa <= 0.0) != (wb <= 0.0) ? 0.f : (float)fmin(fabs(wa), fabs(wb));
      cut = !((float)fmax(fabs(wa), fabs(wb)) * adt < kPiLo) && !(wmin * adt > kPiHi);
    }
    const uint32_t m = __ballot_sync(0xffffffffu, cut);
    if (threadIdx.x == 0 && m) atomicAdd(f.uneven + 1, (uint32_t)__popc(m));
    return;
  }
  i -= kDSamples;
  const uint32_t n_tap = (kDNodes + 1) * kDTaps;
  if (i < n_tap) {
    // I0(beta sqrt(1 - (2x/W)^2)) = F(y), F(y) = sum y^k / k!^2, y quadratic in
    // x: Taylor coefficients of F by Horner's scheme, then of F(y(x + r))
    const int g = (int)(i / kDTaps), l = (int)(i % kDTaps);
    const double x = (double)(g - kDNodes / 2) / kDNodes + (kDTaps / 2 - 0.5) - l;
    const double b2 = kDBeta * kDBeta / (kDTaps * kDTaps);
    const double y = 0.25 * kDBeta * kDBeta - b2 * x * x, y1 = -2.0 * b2 * x, y2 = -b2;
    double F[6] = {0, 0, 0, 0, 0, 0}, c = c_last;
    for (int k = kDSeries; k >= 0; --k) {
#pragma unroll
      for (int j = 5; j > 0; --j) F[j] = F[j] * y + F[j - 1];
      F[0] = F[0] * y + c;
      c *= (double)k * (double)k;
    }
    const double y11 = y1 * y1;
    double a[6];
    a[0] = F[0];
    a[1] = F[1] * y1;
    a[2] = F[1] * y2 + F[2] * y11;
    a[3] = 2.0 * F[2] * y1 * y2 + F[3] * y11 * y1;
    a[4] = F[2] * y2 * y2 + 3.0 * F[3] * y11 * y2 + F[4] * y11 * y11;
    a[5] = 3.0 * F[3] * y1 * y2 * y2 + 4.0 * F[4] * y11 * y1 * y2 + F[5] * y11 * y11 * y1;
    float *o = (float *)(f.taps + (size_t)g * kDRow + 4 * (l / 2)) + (l & 1);
    const df d0 = df_from_double(a[0] * inv_i0), d1 = df_from_double(a[1] * inv_i0);
    o[0] = d0.hi; o[2] = d1.hi; o[4] = d0.lo; o[6] = d1.lo;
    for (int j = 2; j < 6; ++j) o[8 + 2 * (j - 2)] = (float)(a[j] * inv_i0);
  } else if (i < n_tap + f.M) {
    const uint32_t k = i - n_tap;
    double sn, cn;
    sincospi(2.0 * (double)k / (double)f.M, &sn, &cn);
    f.twiddle[k] = make_double2(cn, sn);
  } else if (i <= n_tap + f.M + f.nb / 2u) {
    const uint32_t k = i - n_tap - f.M;
    const double x = kDTaps * M_PI * (double)k / (double)f.M;
    const double s = sqrt(kDBeta * kDBeta - x * x);
    f.deconv[k] = s / (kDTaps * sinh(s) * inv_i0);
  }
  const double w0 = p.omega[0], dw = (p.omega[n - 1] - w0) / (double)(n - 1);
  bool bad = !(fabs(dw) > 0.0) || !isfinite(dw);
  for (uint32_t j = i; j < n; j += gridDim.x * blockDim.x - kDSamples) {
    const double wj = p.omega[j];
    if (!(fabs(wj - (w0 + (double)j * dw)) <= 1e-12 * fabs(wj) + 1e-300)) bad = true;
  }
  if (bad) atomicOr(f.uneven, 1u);
}

// The circles cleared (a memset would write up to 4 GiB also where the cut steps take
// the transforms off, and a warp alone its 32 circles too slowly).
__global__ void __launch_bounds__(256) df_clear_kernel(const DfFast f, uint64_t n) {
  if (!df_by_transform(f)) return;
  double2 *c = reinterpret_cast<double2 *>(f.cells);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    c[i] = make_double2(0.0, 0.0);
}

// Adds a float to a double in memory; the conversion by integer operations
// keeps off the FP64 pipe.
__device__ __forceinline__ void df_red(double *a, float v) {
  const uint32_t b = __float_as_uint(v), m = b & 0x7fffffffu;
  uint32_t hi = (m >> 3) + 0x38000000u;
  if (m < 0x00800000u) hi = 0u;              // zero (and below the normal range)
  if (m >= 0x7f800000u) hi = 0x7ff00000u | (m >> 3);  // infinity, NaN
  const uint32_t lo = m < 0x00800000u ? 0u : b << 29;
  const double d = __hiloint2double((int)(hi | (b & 0x80000000u)), (int)lo);
  asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(a), "d"(d) : "memory");
}

// a b for pairs a and a per-slot double-float (xh, xl), nxh = -xh; not
// renormalised.
__device__ __forceinline__ df2 df2_mul(const df2 &a, float2 xh, float2 xl, float2 nxh) {
  df2 r;
  r.hi = __fmul2_rn(a.hi, xh);
  const float2 ne = __ffma2_rn(a.hi, nxh, r.hi);
  r.lo = sub2(__ffma2_rn(a.hi, xl, __fmul2_rn(a.lo, xh)), ne);
  return r;
}

// f tau less its whole turns, one rounding.
__device__ __forceinline__ df df_turns(double f, double tau) {
  return df_from_double(__fma_rn(f, tau, -rint(f * tau)));
}

struct DfSpreadSmem {
  float4 taps[(kDNodes + 1) * kDRow];
  float4 tab[kTab];
  // of 32 steps: q, x | y, z (FP64), (bx, ax), (by, ay), (bz, az) as
  // (hi, hi, lo, lo), (1 - bz hi, lo, 0, 0)
  float4 rec[kDSpreadWarps][32][6];
};

// Bound by FP32 instructions (about 800 a warp and step, the packed ones two
// cycles each) at 8 warps an SM, the most that 255 registers a lane allow;
// beside them run 300 cycles of table reads and, of FP64, the phases' 350 (in
// double-float the frequencies' 48 bits cost 5e-10 of the spectrum after 1e5
// turns, 5.8 ms; in FP64 1e-11 to 5e-11, 6.3 ms).  32 tracks of 2000 steps, 128
// x 32 x 32 points: 39.2 ms term by term, 6.3 with the transforms.
__global__ void __launch_bounds__(kDSpreadWarps * 32, 2)
    df_spread_kernel(const __grid_constant__ FarMixedParams p, const DfFast f,
                     const DfRecord *__restrict__ rec, const float4 *__restrict__ gtab) {
  if (!df_by_transform(f)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DfSpreadSmem &sm = *reinterpret_cast<DfSpreadSmem *>(smem_raw);
  for (int i = threadIdx.x; i < (kDNodes + 1) * kDRow; i += blockDim.x) sm.taps[i] = f.taps[i];
  for (int i = threadIdx.x; i < kTab; i += blockDim.x) sm.tab[i] = gtab[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t unit = blockIdx.x * kDSpreadWarps + warp;
  if (unit >= f.n_segs * f.n_dwb) return;
  const uint32_t gs = unit / f.n_dwb, dwb = unit % f.n_dwb;
  uint32_t lo = 0, hi = p.n_tracks;  // the segment's track
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (df_first_segment(p, f, mid) <= gs) lo = mid; else hi = mid;
  }
  const uint32_t t = lo;
  SnapState snap;
  snap.init(p.it_start[t], p.it_end[t], p.snap_its + (size_t)t * p.snap_stride, p.n_snaps);
  if (snap.fire_it == SnapState::NEVER) return;  // nothing of the track is written
  const uint64_t last = (uint64_t)min((int64_t)track_body(p, t), snap.fire_it + 1);
  const uint64_t sa = (uint64_t)(gs - df_first_segment(p, f, t)) * f.seg_steps;
  if (sa >= last) return;
  const uint32_t a = (uint32_t)sa, b = (uint32_t)min(last, sa + f.seg_steps);
  const int64_t base = p.offsets[t];

  const uint32_t nT = p.n_theta, n_dirs = nT * p.n_phi;
  const uint32_t band = dwb % f.n_bands, j0 = band * f.nb;
  const uint32_t nb = min(f.nb, p.n_omega - j0);
  const uint32_t dir_raw = (dwb / f.n_bands) * 32u + lane;
  const bool active = dir_raw < n_dirs;
  const uint32_t dir = active ? dir_raw : n_dirs - 1u, iT = dir % nT, iP = dir / nT;
  const double sTd = p.sin_theta[iT], cTd = p.cos_theta[iT];
  const double n0 = sTd * p.cos_phi[iP], n1 = sTd * p.sin_phi[iP], omcd = 1.0 - cTd;
  const df sT = df_from_double(sTd), cT = df_from_double(cTd), omc = df_from_double(omcd);
  const df sP = df_from_double(p.sin_phi[iP]), cP = df_from_double(p.cos_phi[iP]);
  const double inv2pi = 0.15915494309189533577;
  const double w0 = p.omega[0], dw = (p.omega[p.n_omega - 1] - w0) / (double)(p.n_omega - 1);
  const double f_c = (w0 + (double)(j0 + nb / 2u) * dw) * inv2pi, f_d = dw * inv2pi;
  const float wmax = df_band_max(p, f, band);
  const double wa = p.omega[j0], wb = p.omega[j0 + nb - 1u];
  const float wmin = (wa <= 0.0) != (wb <= 0.0) ? 0.f : (float)fmin(fabs(wa), fabs(wb));
  const int M = (int)f.M;
  const float Mf = (float)M;
  double *cells = f.cells + ((uint64_t)unit * 32u + lane) * (uint64_t)M * 4u;
  df2 acc[kDPairs][4];  // cells cur - 6 .. cur + 7 in pairs: theta re, im, phi re, im
#pragma unroll
  for (int j = 0; j < kDPairs; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c].hi = acc[j][c].lo = f2(0.f);
  int cur = 0;
  bool live = false;
  double prev = 0.0;
  if (a > 0) {
    const DfRecord &e = rec[base + a - 1];
    prev = df_tau(e.q, e.x, e.y, e.z, omcd, n0, n1);
  }
  bool any = false;
  float4 (*rc)[6] = sm.rec[warp];
  for (uint32_t s0 = a; s0 < b; s0 += 32u) {
    const uint32_t cnt = min(32u, b - s0);
    __syncwarp();
    if ((uint32_t)lane < cnt) {
      const DfRecord r = rec[base + s0 + lane];
      double2 *o = reinterpret_cast<double2 *>(rc[lane]);
      o[0] = make_double2(r.q, r.x);
      o[1] = make_double2(r.y, r.z);
      const double u[3] = {r.bx, r.by, r.bz}, v[3] = {r.ax, r.ay, r.az};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const df du = df_from_double(u[k]), dv = df_from_double(v[k]);
        rc[lane][2 + k] = make_float4(du.hi, dv.hi, du.lo, dv.lo);
      }
      const df om = df_from_double(r.omb);
      rc[lane][5] = make_float4(om.hi, om.lo, 0.f, 0.f);
    }
    __syncwarp();
    bool cut = false;
#pragma unroll 1
    for (uint32_t i = 0; i < cnt; ++i) {
      const double2 r0 = reinterpret_cast<const double2 *>(rc[i])[0];
      const double2 r1 = reinterpret_cast<const double2 *>(rc[i])[1];
      const double taud = df_tau(r0.x, r0.y, r1.x, r1.y, omcd, n0, n1);
      // the track's first step compares the phase with zero
      // (synchrad/kernel_farfield.cl:49, 65-72)
      const float adt = (float)fabs(s0 + i == 0u ? taud : taud - prev);
      prev = taud;
      if (!(wmax * adt < kPiLo)) {
        cut = cut || (active && !(wmin * adt > kPiHi));
        continue;
      }
      if (!active) continue;
      // amplitudes on theta-hat and phi-hat from the record in the plane of phi
      const float4 qx = rc[i][2], qy = rc[i][3], qz = rc[i][4], qo = rc[i][5];
      const df2 X{make_float2(qx.x, qx.y), make_float2(qx.z, qx.w)};
      const df2 Y{make_float2(qy.x, qy.y), make_float2(qy.z, qy.w)};
      const df2 Z{make_float2(qz.x, qz.y), make_float2(qz.z, qz.w)};
      const df2 R = df2_dot(X, f2(cP.hi), f2(cP.lo), f2(-cP.hi), Y, f2(sP.hi), f2(sP.lo),
                            f2(-sP.hi));  // (b_rho, a_rho)
      const df2 Q = df2_dot(Y, f2(cP.hi), f2(cP.lo), f2(-cP.hi), X, f2(-sP.hi), f2(-sP.lo),
                            f2(sP.hi));  // (b_phi, a_phi)
      const df2 T = df2_dot(R, f2(cT.hi), f2(cT.lo), f2(-cT.hi), Z, f2(-sT.hi), f2(-sT.lo),
                            f2(sT.hi));  // (theta.b, theta.a)
      const df2 E = df2_dot(Z, make_float2(omc.hi, cT.hi), make_float2(omc.lo, cT.lo),
                            make_float2(-omc.hi, -cT.hi), R, make_float2(-sT.hi, sT.hi),
                            make_float2(-sT.lo, sT.lo),
                            make_float2(sT.hi, -sT.hi));  // (1 - n.b - (1 - b_z), n.a)
      const df D = df_add(df{qo.x, qo.y}, df{E.hi.x, E.lo.x});
      const float y = __frcp_rn(D.hi);
      const float res = __fmaf_rn(-D.hi, y, 1.0f) - D.lo * y;
      const df c2 = fast_two_sum(y, y * __fmaf_rn(res, res, res));
      const df c1 = df_mul(df{E.hi.y, E.lo.y}, df_mul(c2, c2));
      const df2 tq{make_float2(T.hi.x, Q.hi.x), make_float2(T.lo.x, Q.lo.x)};
      const df2 ta{make_float2(T.hi.y, Q.hi.y), make_float2(T.lo.y, Q.lo.y)};
      const df2 amp = df2_dot(tq, f2(-c1.hi), f2(-c1.lo), f2(c1.hi), ta, f2(-c2.hi), f2(-c2.lo),
                              f2(c2.hi));  // on (theta-hat, phi-hat)
      // phase of the band's centre; cell: d_omega tau / 2 pi turns of M cells
      // (in FP64: tau may be many turns)
      df zc, zs;
      df_cis(sm.tab, df_turns(f_c, taud), zc, zs);
      const df2 vr = df2_mul(amp, f2(zc.hi), f2(zc.lo), f2(-zc.hi));
      const df2 vi = df2_mul(amp, f2(zs.hi), f2(zs.lo), f2(-zs.hi));
      const df u = df_turns(f_d, taud);
      const float uh = u.hi * Mf, ul = u.lo * Mf;
      const float rm = rintf((uh - 0.5f) + ul);
      const df fa = two_sum(uh, -rm), fb = two_sum(fa.hi, -0.5f);
      const df ff = two_sum(fb.hi, (fa.lo + fb.lo) + ul);  // in [-1/2, 1/2]
      const float gk = rintf(ff.hi * (float)kDNodes);
      const df r = two_sum(ff.hi - gk * (1.0f / (float)kDNodes), ff.lo);
      const float4 *tp = sm.taps + ((int)gk + kDNodes / 2) * kDRow;
      const int m = (int)rm & (M - 1);
      if (live && m != cur) {
        int adv = ((m - cur + M / 2) & (M - 1)) - M / 2;
        auto leave = [&](int cell, int pair, bool second) {
          double *o = cells + (uint64_t)(cell & (M - 1)) * 4u;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            df_red(o + c, second ? acc[pair][c].hi.y : acc[pair][c].hi.x);
            df_red(o + c, second ? acc[pair][c].lo.y : acc[pair][c].lo.x);
          }
        };
        if (adv >= kDTaps || adv <= -kDTaps) {
#pragma unroll
          for (int j = 0; j < kDPairs; ++j) {
            leave(cur - 6 + 2 * j, j, false);
            leave(cur - 5 + 2 * j, j, true);
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[j][c].hi = acc[j][c].lo = f2(0.f);
          }
          cur = m;
          adv = 0;
        }
        while (adv > 0) {
          leave(cur - 6, 0, false);
#pragma unroll
          for (int j = 0; j < kDPairs; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              acc[j][c].hi.x = acc[j][c].hi.y;
              acc[j][c].lo.x = acc[j][c].lo.y;
              acc[j][c].hi.y = j + 1 < kDPairs ? acc[j + 1 < kDPairs ? j + 1 : j][c].hi.x : 0.f;
              acc[j][c].lo.y = j + 1 < kDPairs ? acc[j + 1 < kDPairs ? j + 1 : j][c].lo.x : 0.f;
            }
          ++cur;
          --adv;
        }
        while (adv < 0) {
          leave(cur + 7, kDPairs - 1, true);
#pragma unroll
          for (int j = kDPairs - 1; j >= 0; --j)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              acc[j][c].hi.y = acc[j][c].hi.x;
              acc[j][c].lo.y = acc[j][c].lo.x;
              acc[j][c].hi.x = j > 0 ? acc[j > 0 ? j - 1 : 0][c].hi.y : 0.f;
              acc[j][c].lo.x = j > 0 ? acc[j > 0 ? j - 1 : 0][c].lo.y : 0.f;
            }
          --cur;
          ++adv;
        }
      }
      cur = m;
      live = true;
      const float2 rh = f2(r.hi), rl = f2(r.lo), nrh = f2(-r.hi);
#pragma unroll
      for (int j = 0; j < kDPairs; ++j) {
        const float4 q0 = tp[4 * j], q1 = tp[4 * j + 1], q2 = tp[4 * j + 2], q3 = tp[4 * j + 3];
        const float2 a0 = make_float2(q0.x, q0.y), a1 = make_float2(q0.z, q0.w);
        float2 in = __ffma2_rn(rh, make_float2(q3.z, q3.w), make_float2(q3.x, q3.y));
        in = __ffma2_rn(rh, in, make_float2(q2.z, q2.w));
        in = __ffma2_rn(rh, in, make_float2(q2.x, q2.y));
        const float2 dl = __ffma2_rn(rh, in, make_float2(q1.z, q1.w));
        const float2 pr = __fmul2_rn(rh, a1);
        const float2 ne = __ffma2_rn(nrh, a1, pr);
        float2 tl = __ffma2_rn(rh, dl, make_float2(q1.x, q1.y));
        tl = sub2(__ffma2_rn(rl, a1, tl), ne);
        df2 w;
        w.hi = __fadd2_rn(a0, pr);
        w.lo = __fadd2_rn(tl, sub2(pr, sub2(w.hi, a0)));
        df2_acc(acc[j][0], f2(vr.hi.x), f2(vr.lo.x), f2(-vr.hi.x), w);
        df2_acc(acc[j][1], f2(vi.hi.x), f2(vi.lo.x), f2(-vi.hi.x), w);
        df2_acc(acc[j][2], f2(vr.hi.y), f2(vr.lo.y), f2(-vr.hi.y), w);
        df2_acc(acc[j][3], f2(vi.hi.y), f2(vi.lo.y), f2(-vi.hi.y), w);
      }
    }
    any = any || cut;
    const uint32_t word = __ballot_sync(0xffffffffu, cut);
    if (lane == 0) f.cut[((uint64_t)base / 32u + t + s0 / 32u) * f.n_dwb + dwb] = word;
  }
  if (live) {
#pragma unroll
    for (int j = 0; j < kDTaps; ++j) {
      double *o = cells + (uint64_t)((cur - 6 + j) & (M - 1)) * 4u;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        df_red(o + c, j & 1 ? acc[j / 2][c].hi.y : acc[j / 2][c].hi.x);
        df_red(o + c, j & 1 ? acc[j / 2][c].lo.y : acc[j / 2][c].lo.x);
      }
    }
  }
  const uint32_t word = __ballot_sync(0xffffffffu, any);
  if (lane == 0 && word) atomicOr(f.any + (uint64_t)t * f.n_dwb + dwb, word);
}

// A block per (track, direction, band): the FFT of both components, radix 2
// from one buffer to the other, in FP64.
__global__ void __launch_bounds__(128) df_transform_kernel(const __grid_constant__ FarMixedParams p,
                                                           const DfFast f) {
  if (!df_by_transform(f)) return;
  extern __shared__ __align__(16) double2 tsm[];
  const uint32_t M = f.M, nT = p.n_theta, n_dirs = nT * p.n_phi;
  const uint32_t dir = blockIdx.x % n_dirs, tb = blockIdx.x / n_dirs;
  const uint32_t band = tb % f.n_bands, t = tb / f.n_bands;
  SnapState snap;
  snap.init(p.it_start[t], p.it_end[t], p.snap_its + (size_t)t * p.snap_stride, p.n_snaps);
  if (snap.fire_it == SnapState::NEVER) return;
  const uint64_t last = (uint64_t)min((int64_t)track_body(p, t), snap.fire_it + 1);
  const uint32_t segs = (uint32_t)((last + f.seg_steps - 1) / f.seg_steps);
  double *c0 = f.cells + df_cell(p, f, t, dir, band, 0);
  const uint64_t stride = (uint64_t)f.n_dwb * 32u * M * 4u;
  double2 *x = tsm, *y = tsm + 2 * M;
  for (uint32_t m = threadIdx.x; m < M; m += blockDim.x) {
    double2 u = make_double2(0.0, 0.0), v = u;
    for (uint32_t g = 0; g < segs; ++g) {
      const double2 *q = reinterpret_cast<const double2 *>(c0 + g * stride + 4u * m);
      const double2 q0 = q[0], q1 = q[1];
      u.x += q0.x; u.y += q0.y; v.x += q1.x; v.y += q1.y;
    }
    x[m] = u;
    x[M + m] = v;
  }
  __syncthreads();
  for (uint32_t s = 1; s < M; s *= 2) {
    for (uint32_t i = threadIdx.x; i < M; i += blockDim.x) {  // M/2 butterflies of each
      const uint32_t c = i & (M / 2), k = i & (M / 2 - 1), q = k & (s - 1), ps = k - q;
      const double2 a = x[2 * c + k], b = x[2 * c + k + M / 2];
      const double2 w = f.twiddle[ps];
      const double2 d = make_double2(a.x - b.x, a.y - b.y);
      y[2 * c + 2 * ps + q] = make_double2(a.x + b.x, a.y + b.y);
      y[2 * c + 2 * ps + q + s] = make_double2(d.x * w.x - d.y * w.y, d.x * w.y + d.y * w.x);
    }
    __syncthreads();
    double2 *z = x;
    x = y;
    y = z;
  }
  const uint32_t j0 = band * f.nb, nb = min(f.nb, p.n_omega - j0);
  for (uint32_t j = threadIdx.x; j < nb; j += blockDim.x) {
    const int k = (int)j - (int)(nb / 2u);
    const double dv = f.deconv[k < 0 ? -k : k];
    const double2 u = x[k & (int)(M - 1)], v = x[M + (k & (int)(M - 1))];
    double2 *o = reinterpret_cast<double2 *>(c0 + 4u * j);
    o[0] = make_double2(u.x * dv, u.y * dv);
    o[1] = make_double2(v.x * dv, v.y * dv);
  }
}

template <int K>
struct DfAcc {  // pairs of points, 4 sums each: A_theta re/im, A_phi re/im
  df2 tr[K / 2], ti[K / 2], pr[K / 2], pi[K / 2];
};

// FAST: the steps that include the whole band come from the transforms; this
// kernel adds the cut ones and writes the comps.  Where the transforms are not
// taken the other instance does everything.
template <int K, bool FAST>
__global__ void __launch_bounds__(kDW * 32, 1)
    far_df_kernel(FarMixedParams p, const DfRecord *__restrict__ rec,
                  const float4 *__restrict__ gtab, DfFast df_) {
  static_assert(K == 8, "K (more points per lane spill at 255 registers)");
  if (df_.uneven != nullptr && df_by_transform(df_) != FAST) return;
  constexpr int KP = K / 2;
  __shared__ float4 tab[kTab];
  __shared__ DirConstDf dcs[kDW][kDMaxDpw];
  extern __shared__ float4 setup_all[];  // [kDW][dpw][kDSetupF4][32]
  for (int i = threadIdx.x; i < kTab; i += blockDim.x) tab[i] = gtab[i];

  const int dpw = (int)p.dpw, L = 32 / dpw;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dsub = lane / L, ll = lane % L;
  float4 *setup = setup_all + (size_t)warp * 32 * dpw * kDSetupF4;

  const uint32_t nO = p.n_omega, nT = p.n_theta;
  const uint32_t n_dirs = nT * p.n_phi;
  const uint64_t P = (uint64_t)nO * n_dirs;
  const uint32_t n_groups_dir = (n_dirs + dpw - 1) / dpw;
  const uint32_t n_wt = n_groups_dir * p.n_wtiles;
  const double inv2pi = 0.15915494309189533577;
  const double dw_glob = (nO > 1) ? (p.omega[nO - 1] - p.omega[0]) / (double)(nO - 1) : 0.0;
  const double dw_rev = dw_glob * inv2pi;

  const uint32_t item = blockIdx.x;
  const uint32_t sub = item / p.n_groups, grp = item % p.n_groups;
  const uint32_t wt = grp * kDW + warp;
  const bool active_w = wt < n_wt;
  const uint32_t dgrp = active_w ? wt / p.n_wtiles : 0u;
  const uint32_t tile = active_w ? wt % p.n_wtiles : 0u;
  const uint32_t dir_raw = dgrp * dpw + dsub;
  const bool active = active_w && dir_raw < n_dirs;
  const uint32_t dir = active ? dir_raw : 0u;
  const int j0 = (int)(tile * (uint32_t)(L * K)) + ll * K;
  const int nv = active ? max(0, min(K, (int)nO - j0)) : 0;

  if (ll == 0) {
    const uint32_t iT = dir % nT, iP = dir / nT;
    DirConstDf &d = dcs[warp][dsub];
    d.sT = p.sin_theta[iT];
    d.cT = p.cos_theta[iT];
    d.sPh = p.sin_phi[iP];
    d.cPh = p.cos_phi[iP];
    d.n0 = d.sT * d.cPh;
    d.n1 = d.sT * d.sPh;
    d.omc = 1.0 - d.cT;
    d.tprev = 0.0;
  }
  // lane constants: first frequency in revolutions, uniformity, |omega| range
  const double w0d = nv > 0 ? p.omega[j0] : 0.0;
  const df w0_rev = df_from_double(w0d * inv2pi);
  const float w0f = (float)w0d, dwf = (float)dw_glob;
  const float inv_dwf = (dwf != 0.f) ? 1.0f / dwf : 0.f;
  bool uniform = true;
  float wabs_min = 3.0e38f, wabs_max = 0.f;
  for (int m = 0; m < nv; ++m) {
    const double wm = p.omega[j0 + m];
    if (fabs(wm - (w0d + (double)m * dw_glob)) > 1e-12 * fabs(wm) + 1e-300) uniform = false;
    wabs_min = fminf(wabs_min, (float)fabs(wm));
    wabs_max = fmaxf(wabs_max, (float)fabs(wm));
  }
  if (nv == 0) { wabs_min = 0.f; wabs_max = 0.f; }
  constexpr bool fast = FAST;
  const uint32_t band = FAST ? (uint32_t)min(j0, (int)nO - 1) / df_.nb : 0u;
  const float band_max = FAST ? df_band_max(p, df_, band) : 0.f;
  __syncthreads();  // table and direction constants

  uint32_t t0, t1;
  subset_tracks(p, sub, t0, t1);
  for (uint32_t t = t0; t < t1; ++t) {
    const int64_t base = p.offsets[t];
    const uint32_t n_body = track_body(p, t);
    const uint32_t it_start = p.it_start[t], it_end = p.it_end[t];
    const double wp = p.weight[t];
    const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
    SnapState snap;
    snap.init(it_start, it_end, snaps, p.n_snaps);
    DfAcc<K> acc;
#pragma unroll
    for (int q = 0; q < KP; ++q) {
      acc.tr[q].hi = acc.tr[q].lo = acc.ti[q].hi = acc.ti[q].lo = f2(0.f);
      acc.pr[q].hi = acc.pr[q].lo = acc.pi[q].hi = acc.pi[q].lo = f2(0.f);
    }

    // Snapshot write: A from the double-float sums, per comp, in FP64.
    auto flush = [&](uint32_t ksnap) {
      if (!active) return;
      const DirConstDf &d = dcs[warp][dsub];
      const double wpdt2 = wp * p.dt * p.dt;
      const double wpdt = sqrt(wp) * p.dt;
      const double thxd = d.cT * d.cPh, thyd = d.cT * d.sPh, thzd = -d.sT;
      const double phxd = -d.sPh, phyd = d.cPh;
      double *part = p.partial + ((uint64_t)sub * p.n_out * p.n_snaps) * P;
#pragma unroll
      for (int q = 0; q < KP; ++q) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int m = 2 * q + e;
          if (m >= nv) continue;
          auto val = [&](const df2 &v) {
            return e ? (double)v.hi.y + (double)v.lo.y : (double)v.hi.x + (double)v.lo.x;
          };
          double Ar = val(acc.tr[q]), Ai = val(acc.ti[q]);
          double Br = val(acc.pr[q]), Bi = val(acc.pi[q]);
          if (fast) {
            const double *v = df_.cells + df_cell(p, df_, t, dir, band, j0 + m - band * df_.nb);
            Ar += v[0]; Ai += v[1]; Br += v[2]; Bi += v[3];
          }
          const uint64_t gti = (uint64_t)(j0 + m) + (uint64_t)nO * dir;
          if (p.save_A != nullptr) {  // the adjoint's forward record, per snapshot
            float4 *sa = reinterpret_cast<float4 *>(p.save_A) +
                         ((uint64_t)t * p.n_snaps + ksnap) * P + gti;
            *sa = make_float4((float)Ar, (float)Ai, (float)Br, (float)Bi);
          }
          auto add = [&](int c, double v) {
            part[((uint64_t)c * p.n_snaps + ksnap) * P + gti] += v;
          };
          switch (p.comp) {
            case SR_COMP_TOTAL:
              add(0, wpdt2 * (Ar * Ar + Ai * Ai + Br * Br + Bi * Bi));
              break;
            case SR_COMP_CARTESIAN: {
              const double xr = thxd * Ar + phxd * Br, xi = thxd * Ai + phxd * Bi;
              const double yr = thyd * Ar + phyd * Br, yi = thyd * Ai + phyd * Bi;
              const double zr = thzd * Ar, zi = thzd * Ai;
              add(0, wpdt2 * (xr * xr + xi * xi));
              add(1, wpdt2 * (yr * yr + yi * yi));
              add(2, wpdt2 * (zr * zr + zi * zi));
              break;
            }
            case SR_COMP_CARTESIAN_COMPLEX: {
              const double f = wpdt * p.form_factor[j0 + m];
              add(0, f * (thxd * Ar + phxd * Br));
              add(1, f * (thxd * Ai + phxd * Bi));
              add(2, f * (thyd * Ar + phyd * Br));
              add(3, f * (thyd * Ai + phyd * Bi));
              add(4, f * (thzd * Ar));
              add(5, f * (thzd * Ai));
              break;
            }
            case SR_COMP_SPHERIC:
              add(1, wpdt2 * (Ar * Ar + Ai * Ai));
              add(2, wpdt2 * (Br * Br + Bi * Bi));
              break;
            default:  // SR_COMP_SPHERIC_COMPLEX (FormFactor not applied)
              add(2, wpdt * Ar);
              add(3, wpdt * Ai);
              add(4, wpdt * Br);
              add(5, wpdt * Bi);
              break;
          }
        }
      }
    };

    // the chunks of 32 steps that hold a cut step of the warp's directions
    uint32_t some = 0xffffffffu;
    bool any = true;
    const uint32_t b_lo = tile * (uint32_t)(L * K) / max(1u, df_.nb);
    const uint32_t b_hi = min((tile + 1) * (uint32_t)(L * K), nO) / max(1u, df_.nb);
    const uint32_t g32 = dgrp * dpw / 32u, dmask = ((1u << dpw) - 1u) << (dgrp * dpw % 32u);
    auto cut_word = [&](const uint32_t *row) {
      uint32_t v = 0u;
      for (uint32_t b = b_lo; b <= b_hi && b < df_.n_bands; ++b)
        v |= __ldcg(row + (uint64_t)g32 * df_.n_bands + b);
      return v & dmask;
    };
    if (fast) any = cut_word(df_.any + (uint64_t)t * df_.n_dwb) != 0u;
    for (uint32_t s0 = 0; any && s0 < n_body; s0 += 32) {
      const uint32_t mcnt = min(32u, n_body - s0);
      if (fast) {
        if ((s0 & 1023u) == 0u) {
          const uint32_t c = s0 / 32u + (uint32_t)lane;
          some = __ballot_sync(0xffffffffu,
                               c * 32u < n_body &&
                                   cut_word(df_.cut + ((uint64_t)base / 32u + t + c) * df_.n_dwb) != 0u);
        }
        if (!((some >> (s0 / 32u % 32u)) & 1u)) {
          if (snap.fire_it >= (int64_t)s0 && snap.fire_it < (int64_t)(s0 + mcnt)) {
            flush(snap.k);
            snap.advance(it_start, it_end, snaps, p.n_snaps);
          }
          continue;
        }
      }
      if (active_w) {
        // ---- per-(direction, step) setup: lane l -> step s0 + l ----
        {
          const uint32_t l = (uint32_t)lane < mcnt ? (uint32_t)lane : mcnt - 1;
          const DfRecord r = rec[base + s0 + l];
          const bool first = (s0 + l) == 0;
          for (int dd = 0; dd < dpw; ++dd) {
            DirConstDf &d = dcs[warp][dd];
            const double tau = df_tau(r.q, r.x, r.y, r.z, d.omc, d.n0, d.n1);
            double prev = __shfl_up_sync(0xffffffffu, tau, 1);
            if (lane == 0) {
              prev = d.tprev;
              if (FAST && s0 > 0) {  // the chunk before may have been skipped
                const DfRecord &e = rec[base + s0 - 1];
                prev = df_tau(e.q, e.x, e.y, e.z, d.omc, d.n0, d.n1);
              }
            }
            // the track's first step compares the phase with zero
            // (synchrad/kernel_farfield.cl:49, 65-72)
            const double dtau = first ? tau : tau - prev;
            const double D = r.omb + d.omc * r.bz - d.n0 * r.bx - d.n1 * r.by;
            const double c2 = 1.0 / D;
            const double an = d.n0 * r.ax + d.n1 * r.ay + d.cT * r.az;
            const double c1 = an * c2 * c2;
            const double thx = d.cT * d.cPh, thy = d.cT * d.sPh, thz = -d.sT;
            const double tb = thx * r.bx + thy * r.by + thz * r.bz;
            const double ta = thx * r.ax + thy * r.ay + thz * r.az;
            const double pb = -d.sPh * r.bx + d.cPh * r.by;
            const double pa = -d.sPh * r.ax + d.cPh * r.ay;
            const df at = df_from_double(-(c1 * tb + c2 * ta));
            const df ap = df_from_double(-(c1 * pb + c2 * pa));
            // R = exp(2 pi i dw_rev tau), whole turns dropped in FP64 (exact)
            const double rr = dw_rev * tau;
            df Rc, Rs;
            df_cis(tab, df_from_double(rr - rint(rr)), Rc, Rs);
            const df R2c = df_sub(df_mul(Rc, Rc), df_mul(Rs, Rs));
            const df R2s = df_mul(df{2.f * Rs.hi, 2.f * Rs.lo}, Rc);
            const df tdf = df_from_double(tau);
            float4 *st = setup + (size_t)dd * kDSetupF4 * 32 + lane;
            st[0 * 32] = make_float4(tdf.hi, tdf.lo, (float)fabs(dtau), 0.f);
            st[1 * 32] = make_float4(at.hi, at.lo, ap.hi, ap.lo);
            st[2 * 32] = make_float4(Rc.hi, Rc.lo, Rs.hi, Rs.lo);
            st[3 * 32] = make_float4(R2c.hi, R2c.lo, R2s.hi, R2s.lo);
            const double last = __shfl_sync(0xffffffffu, tau, mcnt - 1);
            __syncwarp();
            if (lane == 0) d.tprev = last;
          }
        }
        __syncwarp();
        // ---- the points: K per lane, in pairs ----
#pragma unroll 1
        for (uint32_t i = 0; i < mcnt; ++i) {
          const uint32_t s = s0 + i;
          const float4 *st = setup + (size_t)dsub * kDSetupF4 * 32 + i;
          const float4 S0 = st[0], S1 = st[32], S2 = st[64], S3 = st[96];
          const float adt = S0.z;
          const bool all_in = wabs_max * adt < kPiLo;
          const bool all_out = wabs_min * adt > kPiHi || (fast && band_max * adt < kPiLo);
          uint32_t mask = (nv == 0 || all_out) ? 0u : (nv >= 32 ? 0xffffffffu : ((1u << nv) - 1u));
          if (nv > 0 && !all_in && !all_out) {
            const DirConstDf &d = dcs[warp][dsub];
            if (uniform) {
              const float inv_adt = __frcp_rn(adt);  // adt > 0 here
              mask = omega_range_bits_r(w0f, dwf, inv_dwf, kPiLo * inv_adt, nv);
              uint32_t unc = omega_range_bits_r(w0f, dwf, inv_dwf, kPiHi * inv_adt, nv) & ~mask;
              while (unc) {
                const int m = __ffs(unc) - 1;
                unc &= unc - 1u;
                if (exact_mask(p, base, s, it_start, p.omega[j0 + m], d.n0, d.n1, d.cT))
                  mask |= 1u << m;
              }
            } else {
              mask = 0;
#pragma unroll 1
              for (int m = 0; m < nv; ++m) {
                const double wm = p.omega[j0 + m];
                const float ph = (float)fabs(wm) * adt;
                bool inc;
                if (ph < kPiLo) inc = true;
                else if (ph > kPiHi) inc = false;
                else inc = exact_mask(p, base, s, it_start, wm, d.n0, d.n1, d.cT);
                mask |= (uint32_t)inc << m;
              }
            }
          }
          if (mask != 0u) {
            const df tau{S0.x, S0.y};
            const float2 ath = f2(S1.x), atl = f2(S1.y), natb = f2(-S1.x);
            const float2 aph = f2(S1.z), apl = f2(S1.w), napb = f2(-S1.z);
            // first pair: (z0, z0 R), z0 = exp(2 pi i omega_0 tau)
            df2 zr, zi;
            {
              df c0, s0v;
              df_cis(tab, df_frac(df_mul_raw(w0_rev, tau)), c0, s0v);
              df2 a, b;
              a.hi = f2(c0.hi); a.lo = f2(c0.lo);
              b.hi = f2(s0v.hi); b.lo = f2(s0v.lo);
              // slot 0: (1, 0); slot 1: R
              const float2 xh = make_float2(1.f, S2.x), xl = make_float2(0.f, S2.y);
              const float2 yh = make_float2(0.f, S2.z), yl = make_float2(0.f, S2.w);
              zr = df2_dot(a, xh, xl, make_float2(-1.f, -S2.x), b, make_float2(0.f, -S2.z),
                           make_float2(0.f, -S2.w), make_float2(0.f, S2.z));
              zi = df2_dot(a, yh, yl, make_float2(0.f, -S2.z), b, xh, xl,
                           make_float2(-1.f, -S2.x));
            }
            const float2 r2ch = f2(S3.x), r2cl = f2(S3.y), nr2ch = f2(-S3.x);
            const float2 r2sh = f2(S3.z), r2sl = f2(S3.w), nr2sh = f2(-S3.z);
#pragma unroll
            for (int q = 0; q < KP; ++q) {
              if (!uniform) {  // non-uniform axis: each point's own phase
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int m = min(2 * q + e, max(nv - 1, 0));
                  df c0, s0v;
                  df_cis(tab, df_frac(df_mul_raw(df_from_double(p.omega[j0 + m] * inv2pi), tau)),
                         c0, s0v);
                  if (e == 0) {
                    zr.hi.x = c0.hi; zr.lo.x = c0.lo; zi.hi.x = s0v.hi; zi.lo.x = s0v.lo;
                  } else {
                    zr.hi.y = c0.hi; zr.lo.y = c0.lo; zi.hi.y = s0v.hi; zi.lo.y = s0v.lo;
                  }
                }
              }
              const float g0 = ((mask >> (2 * q)) & 1u) ? 1.f : 0.f;
              const float g1 = ((mask >> (2 * q + 1)) & 1u) ? 1.f : 0.f;
              const float2 g = make_float2(g0, g1);
              const float2 at_h = __fmul2_rn(ath, g), at_l = __fmul2_rn(atl, g),
                           nat_h = __fmul2_rn(natb, g);
              const float2 ap_h = __fmul2_rn(aph, g), ap_l = __fmul2_rn(apl, g),
                           nap_h = __fmul2_rn(napb, g);
              df2_acc(acc.tr[q], at_h, at_l, nat_h, zr);
              df2_acc(acc.ti[q], at_h, at_l, nat_h, zi);
              df2_acc(acc.pr[q], ap_h, ap_l, nap_h, zr);
              df2_acc(acc.pi[q], ap_h, ap_l, nap_h, zi);
              if (q + 1 < KP && uniform) {
                const df2 nr = df2_dot(zr, r2ch, r2cl, nr2ch, zi, f2(-S3.z), f2(-S3.w), r2sh);
                const df2 ni = df2_dot(zr, r2sh, r2sl, nr2sh, zi, r2ch, r2cl, nr2ch);
                zr = nr;
                zi = ni;
              }
            }
          }
          if ((int64_t)s == snap.fire_it) {  // uniform over the CTA
            flush(snap.k);
            snap.advance(it_start, it_end, snaps, p.n_snaps);
          }
        }
        __syncwarp();
      } else {
        for (uint32_t i = 0; i < mcnt; ++i)
          if ((int64_t)(s0 + i) == snap.fire_it) snap.advance(it_start, it_end, snaps, p.n_snaps);
      }
    }
    while (snap.fire_it != SnapState::NEVER) {  // writes due after the last body step
      flush(snap.k);
      snap.advance(it_start, it_end, snaps, p.n_snaps);
    }
    if (ll == 0) dcs[warp][dsub].tprev = 0.0;  // the next track starts afresh
    __syncwarp();
  }
}

// Whether the transforms are taken, their circles and segments.
//
// The further launches and a segment's serial walk make about 0.24 ms; term by
// term a track's steps take about 1 us each, more where the points fill the
// SMs.  Measured (us, transforms / term by term; 64 frequencies): 4 directions
// on one track of 1500 steps 239 / 1524, of 300 steps about 235 / 357; 576
// directions on 20 tracks 1853 / 6529, of 300 steps 743 / 1504, of 60 steps
// 749 / 407.
DfFast df_fast_layout(const FarMixedConfig &c, int64_t total_steps, uint32_t n_snaps) {
  DfFast f{};
  if (c.direct || n_snaps != 1 || c.n_omega < 16 || c.n_dirs == 0 || c.n_tracks == 0 || total_steps <= 0)
    return f;
  const uint64_t mean = (uint64_t)total_steps / c.n_tracks;
  if (mean < 160 || (mean < 256 && (uint64_t)c.n_omega * c.n_dirs * c.n_tracks < 200000)) return f;
  f.n_bands = (c.n_omega + kFastMaxBand - 1) / kFastMaxBand;
  f.nb = (c.n_omega + f.n_bands - 1) / f.n_bands;
  if (f.n_bands > 1) f.nb = (f.nb + 7) / 8 * 8;  // a lane's 8 frequencies lie in one band
  const uint32_t M = fast_cells(f.nb);
  f.n_dwb = (c.n_dirs + 31) / 32 * f.n_bands;
  // segments that fill the SMs four times over, of 64 steps or more, longer ones
  // where the circles would take over 4 GiB, else whole tracks, batch by batch
  const uint64_t all = (uint64_t)total_steps * f.n_dwb, circle = (uint64_t)f.n_dwb * 32 * M * 32;
  const uint64_t slots = 4ull * c.n_sm * 2 * kDSpreadWarps, room = (4ull << 30) / circle;
  uint64_t seg = std::max<uint64_t>(64, (all / slots + 31) / 32 * 32);
  while ((uint64_t)total_steps / seg + c.n_tracks > room && seg < (1ull << 30)) seg *= 2;
  seg = std::min<uint64_t>(seg, 1ull << 30);
  uint64_t batch = c.n_tracks, n_segs = (uint64_t)total_steps / seg + batch;
  if (n_segs > room) {
    if (total_steps >= (1ll << 30)) return DfFast{};
    batch = room;
    n_segs = batch;
  }
  if (batch == 0 || n_segs * f.n_dwb > 0x7fffffffull ||
      batch * c.n_dirs * f.n_bands > 0x7fffffffull)
    return DfFast{};
  f.seg_steps = (uint32_t)seg;
  f.n_segs = (uint32_t)n_segs;
  f.batch = (uint32_t)batch;
  f.M = M;
  return f;
}

int launch_df_tables(const FarMixedParams &p, const DfFast &f, const DfRecord *rec,
                     cudaStream_t s) {
  double i0 = 0.0, c = 1.0;  // I0(beta) = sum (beta^2 / 4)^k / k!^2
  for (int k = 0; k <= kDSeries; ++k) {
    if (k) c *= 0.25 * kDBeta * kDBeta / ((double)k * k);
    i0 += c;
  }
  double c_last = 1.0;
  for (int k = 1; k <= kDSeries; ++k) c_last /= (double)k * k;
  const uint32_t n = kDSamples + (kDNodes + 1) * kDTaps + f.M + f.nb / 2 + 1;
  df_fast_tables_kernel<<<(n + 31) / 32, 32, 0, s>>>(p, f, rec, c_last, 1.0 / i0);
  cudaError_t e = allow_smem((const void *)df_spread_kernel, (int)sizeof(DfSpreadSmem));
  if (e == cudaSuccess) e = allow_smem((const void *)df_transform_kernel, (int)(4 * 1024 * 16));
  return cuda_fail(e, "far_df smem attribute");
}

// One batch of tracks into their circles and transforms.
int launch_df_fast(const FarMixedParams &p, const DfFast &f, const DfRecord *rec,
                   const float4 *tab, size_t zero_bytes, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(f.any, 0, zero_bytes, s);
  if (e != cudaSuccess) return cuda_fail(e, "cut flags reset");
  const uint64_t units = (uint64_t)f.n_segs * f.n_dwb, pairs = units * 64u * f.M;
  df_clear_kernel<<<(unsigned)std::min<uint64_t>((pairs + 255) / 256, 8ull * device_sm_count()),
                    256, 0, s>>>(f, pairs);
  df_spread_kernel<<<(unsigned)((units + kDSpreadWarps - 1) / kDSpreadWarps), kDSpreadWarps * 32,
                     sizeof(DfSpreadSmem), s>>>(p, f, rec, tab);
  df_transform_kernel<<<p.n_tracks * p.n_theta * p.n_phi * f.n_bands, 128, 4 * f.M * 16, s>>>(p, f);
  return cuda_fail(cudaGetLastError(), "far_df transform launch");
}

struct DfLayout {
  size_t records, partial, table, taps, deconv, twiddle, cut, any, cells, total;
  DfFast f;
};

DfLayout df_layout(int64_t total_steps, uint64_t P, int n_out, uint32_t n_snaps,
                   const FarMixedConfig &cfg) {
  const int n_sub = cfg.n_sub;
  DfLayout l;
  size_t off = 256;  // status word and the axis test's
  l.records = off;
  off += ((size_t)total_steps * sizeof(DfRecord) + 255) / 256 * 256;
  l.partial = off;
  off += ((size_t)n_sub * n_out * n_snaps * P * 8 + 255) / 256 * 256;
  l.table = off;
  off += (size_t)kTab * sizeof(float4);
  l.f = df_fast_layout(cfg, total_steps, n_snaps);
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) / 256 * 256;
    return at;
  };
  if (l.f.M) {
    l.taps = take((size_t)(kDNodes + 1) * kDRow * sizeof(float4));
    l.deconv = take((size_t)(kFastMaxBand / 2 + 1) * 8);
    l.twiddle = take((size_t)l.f.M * 16);
    l.cut = take(((size_t)total_steps / 32 + l.f.batch) * l.f.n_dwb * 4);
    l.any = take((size_t)l.f.batch * l.f.n_dwb * 4);
    l.cells = take((size_t)l.f.n_segs * l.f.n_dwb * 32 * l.f.M * 32);
  }
  l.total = off;
  return l;
}

template <int K, bool FAST>
int launch_df_main(const FarMixedParams &p, const DfRecord *rec, const float4 *tab,
                   const DfFast &f, cudaStream_t s) {
  const size_t smem = (size_t)kDW * 32 * p.dpw * kDSetupF4 * sizeof(float4);
  cudaError_t e = allow_smem((const void *)far_df_kernel<K, FAST>, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "far_df smem attribute");
  far_df_kernel<K, FAST><<<p.n_items, kDW * 32, smem, s>>>(p, rec, tab, f);
  return cuda_fail(cudaGetLastError(), "far_df kernel launch");
}

}  // namespace

// Work shape of the double-float far field: K = 8 points per lane (the 64
// double-float accumulator pairs of 16 points spill at 255 registers), L lanes
// per direction, and track subsets for about four CTAs per SM.
FarMixedConfig far_df_choose(uint32_t n_omega, uint32_t n_dirs, uint32_t n_tracks, int n_sm) {
  FarMixedConfig c;
  c.W = kDW;
  c.ctas_per_sm = 1;
  c.stage = 32;
  c.K = 8;
  int L = 32;
  while (L > 32 / kDMaxDpw && (uint32_t)(L / 2) * c.K >= n_omega) L /= 2;
  c.L = L;
  c.dpw = 32 / L;
  const uint64_t n_wtiles = (n_omega + (uint64_t)L * c.K - 1) / ((uint64_t)L * c.K);
  const uint64_t dgroups = (n_dirs + c.dpw - 1) / c.dpw;
  const uint64_t groups = (dgroups * n_wtiles + c.W - 1) / c.W;
  uint64_t nsub = (4 * (uint64_t)n_sm + groups - 1) / (groups ? groups : 1);
  if (nsub > n_tracks) nsub = n_tracks;
  if (nsub < 1) nsub = 1;
  if (nsub > 64) nsub = 64;
  c.n_sub = (int)nsub;
  c.grid = (int)(groups * nsub);
  c.direct = false;
  c.n_omega = n_omega;
  c.n_dirs = n_dirs;
  c.n_tracks = n_tracks;
  c.n_sm = n_sm;
  return c;
}

size_t far_df_workspace(int64_t total_steps, uint64_t n_points, int n_out, uint32_t n_snaps,
                        const FarMixedConfig &cfg) {
  return df_layout(total_steps, n_points, n_out, n_snaps, cfg).total;
}

int launch_far_df(FarMixedParams p, const FarMixedConfig &shape, void *ws, size_t ws_bytes,
                  cudaStream_t stream) {
  const uint64_t P = (uint64_t)p.n_omega * p.n_theta * p.n_phi;
  if (P == 0 || p.n_tracks == 0 || p.n_snaps == 0) return SR_OK;
  // term by term where the scratch does not hold the transforms' circles
  FarMixedConfig cfg = shape;
  DfLayout lay = df_layout(p.total_steps, P, p.n_out, p.n_snaps, cfg);
  if (ws_bytes < lay.total) {
    cfg.direct = true;
    lay = df_layout(p.total_steps, P, p.n_out, p.n_snaps, cfg);
  }
  if (ws == nullptr || ws_bytes < lay.total)
    return fail(SR_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", lay.total, ws_bytes);
  if (((uintptr_t)ws & 255u) != 0) return fail(SR_ERR_WORKSPACE, "workspace not 256-byte aligned");
  if (cfg.K != 8) return fail(SR_ERR_INVALID, "points per lane %d (8)", cfg.K);
  unsigned char *w = (unsigned char *)ws;
  p.status = (int *)w;
  p.partial = (double *)(w + lay.partial);
  DfRecord *rec = (DfRecord *)(w + lay.records);
  float4 *tab = (float4 *)(w + lay.table);
  p.dpw = (uint32_t)cfg.dpw;
  p.n_wtiles = (p.n_omega + (uint32_t)(cfg.L * cfg.K) - 1) / (uint32_t)(cfg.L * cfg.K);
  const uint32_t n_dirs = p.n_theta * p.n_phi;
  const uint32_t dgroups = (n_dirs + cfg.dpw - 1) / cfg.dpw;
  p.n_groups = (uint32_t)(((uint64_t)dgroups * p.n_wtiles + cfg.W - 1) / cfg.W);
  p.n_sub = (uint32_t)cfg.n_sub;
  p.n_items = p.n_groups * p.n_sub;

  cudaError_t e = cudaMemsetAsync(w, 0, 256, stream);
  if (e != cudaSuccess) return cuda_fail(e, "status reset");
  e = cudaMemsetAsync(p.partial, 0, (size_t)p.n_sub * p.n_out * p.n_snaps * P * 8, stream);
  if (e != cudaSuccess) return cuda_fail(e, "partial reset");
  const int n_sm = device_sm_count();
  df_table_kernel<<<(kTab + 255) / 256, 256, 0, stream>>>(tab);
  if (p.total_steps > 0) {
    int64_t nb = (p.total_steps + 255) / 256;
    if (nb > 8 * (int64_t)n_sm * 16) nb = 8 * (int64_t)n_sm * 16;
    if (p.track_f32)
      df_prepass_kernel<float><<<(int)nb, 256, 0, stream>>>(p, rec);
    else
      df_prepass_kernel<double><<<(int)nb, 256, 0, stream>>>(p, rec);
  }
  int rc = cuda_fail(cudaGetLastError(), "far_df prepass launch");
  if (rc) return rc;
  void *tok = nullptr;
  timing_record(stream, true, &tok);
  if (lay.f.M) {
    DfFast f = lay.f;
    f.uneven = (unsigned int *)(w + 64);
    f.taps = (float4 *)(w + lay.taps);
    f.deconv = (double *)(w + lay.deconv);
    f.twiddle = (double2 *)(w + lay.twiddle);
    f.cut = (unsigned int *)(w + lay.cut);
    f.any = (unsigned int *)(w + lay.any);
    f.cells = (double *)(w + lay.cells);
    rc = launch_df_tables(p, f, rec, stream);
    for (uint32_t t = 0; !rc && t < p.n_tracks; t += f.batch) {
      FarMixedParams q = p;  // the batch's tracks
      q.n_tracks = std::min(f.batch, p.n_tracks - t);
      q.offsets += t;
      q.weight += t;
      q.it_start += t;
      q.it_end += t;
      q.snap_its += (size_t)t * p.snap_stride;
      if (q.save_A) q.save_A += (size_t)t * p.n_snaps * P * 4;
      rc = launch_df_fast(q, f, rec, tab, lay.cells - lay.any, stream);
      if (!rc) rc = launch_df_main<8, true>(q, rec, tab, f, stream);
    }
    if (!rc) rc = launch_df_main<8, false>(p, rec, tab, f, stream);
  } else {
    rc = launch_df_main<8, false>(p, rec, tab, DfFast{}, stream);
  }
  timing_record(stream, false, &tok);
  if (rc) return rc;
  const uint64_t total = (uint64_t)p.n_out * p.n_snaps * P;
  uint64_t nb = (total + 255) / 256;
  if (nb > (uint64_t)n_sm * 64) nb = (uint64_t)n_sm * 64;
  mixed_reduce_kernel<<<(unsigned)nb, 256, 0, stream>>>(p);
  return cuda_fail(cudaGetLastError(), "far_df reduce launch");
}

}  // namespace sr
