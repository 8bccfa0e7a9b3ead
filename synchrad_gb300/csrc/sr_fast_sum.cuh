// Spectral sums over track steps on an evenly spaced omega axis through a
// transform over the steps: the kernels shared by the mixed-precision far and
// near fields.
//
// Both fields need, per direction (screen point) and track,
//     A_j = sum_s v_s exp(i omega_j tau_s),  omega_j = omega_0 + j d_omega,
// a discrete Fourier sum with uneven times tau_s.  Term by term it costs
// N x steps products; here each step is spread with a smooth kernel of kTaps
// cells onto a circle of M >= 2 N cells of the phase d_omega tau mod 2 pi,
// one M-point FFT per (track, direction, component) turns the cells into the
// sums and a division by the kernel's transform undoes the spreading (the
// nonuniform FFT of Dutt & Rokhlin, SIAM J. Sci. Comput. 14 (1993), with the
// Kaiser-Bessel kernel of Jackson et al., IEEE TMI 10 (1991), beta from Beatty
// et al., IEEE TMI 24 (2005)).  The kernel's aliasing is below 3e-8 of the sum
// at kTaps = 8 and M = 2 N, under the rounding of the FP32 terms.
//
// tau grows along a track, so the steps of a direction sweep the circle: a
// lane owns one direction and holds the kTaps cells around the current step
// in registers; when the step moves on by one cell the oldest one is complete
// and leaves for the lane's circle in global memory (red.v4.f32: the lane is
// the only writer of its circle, so the order of the sums is fixed).  The
// per-(direction, step) values (double-float tau, amplitudes) are computed
// once for all frequencies, by the lane itself.
//
// A step enters when omega |dtau| < pi at every frequency of the band with the
// guard band to spare (kPiLo).  A step that the rule cuts inside the band, or
// whose band edge lies in the guard band, goes to a short list per lane; the
// warp empties the lists by direct sums over the included frequencies, with
// the exact FP64 test in the guard band.
#pragma once

#include "sr_mixed_common.cuh"

namespace sr {
namespace {

constexpr int kTaps = 8;
constexpr int kFastList = 512;    // list entries per lane, fewer for short segments
constexpr int kFastWarps = 4;     // warps per CTA
// Per-warp shared memory: step records of the current chunk while spreading,
// the transpose buffer of the FFT otherwise; the first field's outputs; the
// cos/sin phi of the warp's directions.
struct FastSmem {
  union {
    float4 rec[8704 / 16];
    float2 tr[32 * 33];
  };
  float2 out[kFastMaxBand];
  float4 phic[32];
};

// Taps phi(f + 3.5 - l), l = 0..7, for f in [-1/2, 1/2]: degree-8 Chebyshev
// fits of the Kaiser-Bessel kernel on each cell, even and odd parts shared by
// the mirrored taps.
__device__ __forceinline__ void kb_taps(float f, float (&w)[kTaps]) {
  const float g = f * f;
  auto pair = [&](int l, float e0, float o0, float e1, float o1, float e2, float o2, float e3,
                  float o3, float e4) {
    float e = __fmaf_rn(e4, g, e3);
    e = __fmaf_rn(e, g, e2);
    e = __fmaf_rn(e, g, e1);
    e = __fmaf_rn(e, g, e0);
    float o = __fmaf_rn(o3, g, o2);
    o = __fmaf_rn(o, g, o1);
    o = __fmaf_rn(o, g, o0);
    w[l] = __fmaf_rn(o, f, e);
    w[kTaps - 1 - l] = __fmaf_rn(-o, f, e);
  };
  pair(0, 9.660679643e-05f, -7.671282510e-04f, 2.600571373e-03f, -4.920937587e-03f,
       5.659276154e-03f, -3.947199788e-03f, 1.406157040e-03f, 9.299917292e-05f, -2.649927337e-04f);
  pair(1, 1.900451072e-02f, -6.841991097e-02f, 1.010312214e-01f, -7.361625135e-02f,
       1.998347044e-02f, 7.933221757e-03f, -7.344931830e-03f, 9.507333161e-04f, 7.229428156e-04f);
  pair(2, 2.666729093e-01f, -4.878970087e-01f, 2.578946948e-01f, 5.260234699e-02f,
       -9.378349781e-02f, 1.511092298e-02f, 1.341344323e-02f, -4.336146638e-03f,
       -9.862204315e-04f);
  pair(3, 8.674505353e-01f, -4.952890873e-01f, -3.615280092e-01f, 2.447273135e-01f,
       6.815172732e-02f, -5.749912560e-02f, -7.492190693e-03f, 8.106620982e-03f,
       4.874356382e-04f);
}

// One cell's sums added to the lane's circle (no return value, no ordering
// against other lanes: each circle has one writer).
__device__ __forceinline__ void red_f4(float4 *p, float2 a, float2 b) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(
                   __cvta_generic_to_global(p)),
               "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y)
               : "memory");
}

// A term of a partial spectrum (one writer per subset and point: the order of
// the sum is the order of the tracks).
__device__ __forceinline__ void red_f64(double *p, double v) {
  asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "d"(v)
               : "memory");
}
__device__ __forceinline__ df df_square(df a) {
  const float p = a.hi * a.hi;
  return df{p, __fmaf_rn(a.hi + a.hi, a.lo, __fmaf_rn(a.hi, a.hi, -p))};
}
// |x|^2 + |y|^2 of two complex FP32 values, exact to about 2^-46.
__device__ __forceinline__ df df_norm2(float2 x, float2 y) {
  const float a = x.x * x.x, b = x.y * x.y, c = y.x * y.x, d = y.y * y.y;
  const float l = (__fmaf_rn(x.x, x.x, -a) + __fmaf_rn(x.y, x.y, -b)) +
                  (__fmaf_rn(y.x, y.x, -c) + __fmaf_rn(y.y, y.y, -d));
  const df s = two_sum(a, b), t = two_sum(c, d);
  const df r = two_sum(s.hi, t.hi);
  return df{r.hi, r.lo + ((s.lo + t.lo) + l)};
}

// exp(2 pi i w tau) as phasor_rev, with the FP32 library's sin and cos: one
// seed serves every frequency of the band, so the hardware functions' error
// (~4e-7) would not average over seeds as it does term by term.
__device__ __forceinline__ void phasor_exact(float wh, float wl, float th, float tl, float &s,
                                             float &c) {
  const float p = wh * th;
  float e = __fmaf_rn(wh, th, -p);
  e = __fmaf_rn(wh, tl, e);
  e = __fmaf_rn(wl, th, e);
  const float f = (p - rintf(p)) + e;
  sincospif(f + f, &s, &c);
}

// cos(2 pi k / 32) as hi + lo.
__device__ __forceinline__ df cos32(int k) {
  constexpr float h[9] = {1.f, 0.980785251f, 0.923879504f,
                          0.831469595f, 0.707106769f, 0.555570245f,
                          0.382683426f, 0.195090324f, 0.f};
  constexpr float l[9] = {0.f, 2.97394731e-08f, 2.83074897e-08f,
                          1.68702634e-08f, 1.21016175e-08f, -1.17695214e-08f,
                          6.22335072e-09f, -1.67047143e-09f, 0.f};
  k &= 31;
  if (k > 16) k = 32 - k;
  return k <= 8 ? df{h[k], l[k]} : df{-h[16 - k], -l[16 - k]};
}

// d (c + i s), the factor given as hi + lo: the twiddles are the same for
// every track, so their rounding would not average over the tracks.
__device__ __forceinline__ float2 mul_df(float2 d, float ch, float sh, float cl, float sl) {
  return make_float2(__fmaf_rn(d.x, ch, __fmaf_rn(-d.y, sh, __fmaf_rn(d.x, cl, -d.y * sl))),
                     __fmaf_rn(d.x, sh, __fmaf_rn(d.y, ch, __fmaf_rn(d.x, sl, d.y * cl))));
}

// In-place DFT with exp(+2 pi i j k / N) of N = 4, 8, 16 or 32 register
// values, decimation in frequency; output k is left at index bitrev(k).
template <int N>
__device__ __forceinline__ void fft_reg(float2 (&x)[N]) {
#pragma unroll
  for (int len = N; len > 1; len >>= 1) {
#pragma unroll
    for (int b = 0; b < N; b += len) {
#pragma unroll
      for (int j = 0; j < len / 2; ++j) {
        const float2 u = x[b + j], v = x[b + j + len / 2];
        x[b + j] = make_float2(u.x + v.x, u.y + v.y);
        const float2 d = make_float2(u.x - v.x, u.y - v.y);
        const int k = j * (32 / len);  // twiddle exp(2 pi i k / 32)
        float2 r;
        if (k == 0) {
          r = d;
        } else if (k == 8) {
          r = make_float2(-d.y, d.x);
        } else {
          const df c = cos32(k), s = cos32(k - 8);
          r = mul_df(d, c.hi, s.hi, c.lo, s.lo);
        }
        x[b + j + len / 2] = r;
      }
    }
  }
}
template <int N>
__device__ __forceinline__ constexpr int bitrev(int k) {
  int r = 0;
  for (int n = N; n > 1; n >>= 1) {
    r = (r << 1) | (k & 1);
    k >>= 1;
  }
  return r;
}

// The M-point transforms (exp(+2 pi i m k / M)) of NF fields, element
// 32 i + lane of field q in x[q][i]; element a + R1 b of field q comes out in
// y[bitrev(b)] of lane q R1 + a.
template <int R1, int NF>
__device__ __forceinline__ void fft_fields(float2 (&x)[NF][R1], float2 (&y)[32], float2 *tr,
                                           const float4 *tw, int lane) {
  static_assert(R1 * NF == 32, "one warp holds 1024 cells");
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    fft_reg<R1>(x[q]);
#pragma unroll
    for (int a = 0; a < R1; ++a) {
      const float2 v = x[q][bitrev<R1>(a)];
      float2 r = v;
      if (a) {
        const float4 t = __ldg(tw + a * 32 + lane);  // exp(2 pi i a lane / M)
        r = mul_df(v, t.x, t.y, t.z, t.w);
      }
      tr[(q * R1 + a) * 33 + lane] = r;
    }
  }
  __syncwarp();
#pragma unroll
  for (int l = 0; l < 32; ++l) y[l] = tr[lane * 33 + l];
  __syncwarp();
  fft_reg<32>(y);
}

// The N band sums of the fields in x (cells) to dst[q][j], j = frequency index
// + N/2 (not yet divided by the kernel's transform).
template <int R1, int NF>
__device__ __forceinline__ void fft_band(float2 (&x)[NF][R1], float2 *tr, const float4 *tw,
                                         int lane, int n, float2 *dst) {
  float2 y[32];
  fft_fields<R1, NF>(x, y, tr, tw, lane);
  const int q = lane / R1, a = lane % R1;
#pragma unroll
  for (int b = 0; b < 32; ++b) {
    const int k = a + R1 * b;
    const int j = (b < 16 ? k : k - 32 * R1) + n / 2;
    if (j >= 0 && j < n) dst[q * n + j] = y[bitrev<32>(b)];
  }
  __syncwarp();
}

// Values of a direction (far) or screen point (near) that its lane keeps.
template <bool NEAR>
struct LaneDir;
template <>
struct LaneDir<false> {
  float dc_h, dc_l, st_h, st_l;  // 1 - cos(theta), sin(theta) as double-floats
  float f_dc, f_st, f_ct;
};
template <>
struct LaneDir<true> {
  float X_h, X_l, Y_h, Y_l, L_h, L_l;
};

// The part of a warp's scratch slice.
template <bool NEAR>
struct FastSlice {
  static constexpr int NP = NEAR ? 3 : 1;  // pairs of complex fields
  unsigned char *base;
  __device__ FastSlice(const FastParams &f, size_t i) : base(f.scratch + i * f.slice_bytes) {}
  // [NP][32][M] cells (X re, X im, Y re, Y im)
  __device__ float4 *grid() const { return (float4 *)base; }
  // [NP][32][2][nb] direct sums of the listed steps: sums, then low parts
  __device__ float4 *part(const FastParams &f) const { return grid() + (size_t)NP * 32 * f.M; }
  // [32][list] tau.hi, tau.lo, first | last << 16
  __device__ float4 *lhead(const FastParams &f) const {
    return grid() + (size_t)NP * 32 * (f.M + 2 * f.nb);
  }
  // [NP][32][list] amplitudes X, Y
  __device__ float2 *lamp(const FastParams &f) const {
    return (float2 *)(lhead(f) + f.list * 32);
  }
};

// State of one warp's unit of work: 32 directions x one omega band.
template <bool NEAR>
struct FastUnit {
  static constexpr int NP = NEAR ? 3 : 1;
  uint32_t slot0;      // first direction
  uint32_t j0;         // first frequency of the band
  int nb;              // its frequencies
  df f_c, f_d;         // (centre frequency, d_omega) / 2 pi
  float wmax, wmin;    // largest and smallest |omega| of the band
  LaneDir<NEAR> ld;
  uint32_t dir;
  bool active;
  int kphi;            // phi of the lane among the warp's (far)
};

__device__ __forceinline__ void lane_dir(const FarMixedParams &p, uint32_t iT, uint32_t,
                                         LaneDir<false> &ld) {
  const df c = df_from_double(1.0 - p.cos_theta[iT]), s = df_from_double(p.sin_theta[iT]);
  ld.dc_h = c.hi; ld.dc_l = c.lo; ld.st_h = s.hi; ld.st_l = s.lo;
  ld.f_dc = (float)(1.0 - p.cos_theta[iT]);
  ld.f_st = (float)p.sin_theta[iT];
  ld.f_ct = (float)p.cos_theta[iT];
}
__device__ __forceinline__ void lane_dir(const FarMixedParams &p, uint32_t iR, uint32_t iP,
                                         LaneDir<true> &ld) {
  const df x = df_from_double(p.sin_theta[iR] * p.cos_phi[iP]);
  const df y = df_from_double(p.sin_theta[iR] * p.sin_phi[iP]);
  const df L = df_from_double(p.L_screen);
  ld.X_h = x.hi; ld.X_l = x.lo; ld.Y_h = y.hi; ld.Y_l = y.lo;
  ld.L_h = L.hi; ld.L_l = L.lo;
}
__device__ __forceinline__ float4 phi_pairs(const FarMixedParams &p, uint32_t iP) {
  const df c = df_from_double(p.cos_phi[iP]), s = df_from_double(p.sin_phi[iP]);
  return make_float4(c.hi, c.lo, s.hi, s.lo);
}

template <bool NEAR>
__device__ void unit_init(const FarMixedParams &p, uint32_t dwb, int lane, FastSmem &sm,
                          FastUnit<NEAR> &u) {
  const FastParams &f = p.fast;
  const uint32_t nT = p.n_theta, n_dirs = nT * p.n_phi;
  const uint32_t band = dwb % f.n_bands;
  u.slot0 = (dwb / f.n_bands) * 32u;
  u.j0 = band * f.nb;
  u.nb = (int)min(f.nb, p.n_omega - u.j0);
  const double w0 = p.omega[0];
  const double dw = (p.omega[p.n_omega - 1] - w0) / (double)(p.n_omega - 1);
  const double inv2pi = 0.15915494309189533577;
  u.f_c = df_from_double((w0 + (double)(u.j0 + u.nb / 2) * dw) * inv2pi);
  u.f_d = df_from_double(dw * inv2pi);
  const double wa = w0 + (double)u.j0 * dw, wb = w0 + (double)(u.j0 + u.nb - 1) * dw;
  u.wmax = (float)fmax(fabs(wa), fabs(wb));
  u.wmin = (wa <= 0.0) != (wb <= 0.0) ? 0.f : (float)fmin(fabs(wa), fabs(wb));
  u.active = u.slot0 + lane < n_dirs;
  u.dir = u.active ? u.slot0 + lane : n_dirs - 1;
  const uint32_t iT = u.dir % nT, iP = u.dir / nT, iP0 = u.slot0 / nT;
  u.kphi = (int)(iP - iP0);
  lane_dir(p, iT, iP, u.ld);
  if constexpr (!NEAR) {
    if (lane < (int)f.n_phik) sm.phic[lane] = phi_pairs(p, min(iP0 + lane, p.n_phi - 1));
  }
  __syncwarp();
}

// a x + b y for double-floats a, b, rounded once: the rounding of cos and sin
// would be the same at every step of a phi and not average out (spectra of one
// batch of 16 betatron tracks 1.35e-6 from 64 bits with it, 1.19e-6 without; ten
// batches 0.8e-6 to 1.6e-6, mean 1.15e-6, term by term 1.22e-6).  A phi's record
// serves all its directions, so it costs no measurable time.
__device__ __forceinline__ float turned(float a, float al, float x, float b, float bl, float y) {
  const float p = a * x, q = b * y;
  const df s = two_sum(p, q);
  return s.hi + (s.lo + (__fmaf_rn(a, x, -p) + __fmaf_rn(b, y, -q)) + (al * x + bl * y));
}

// The chunk's step records in shared memory.  Far: per (phi of the warp,
// step) the record turned into the plane of that phi, so that a lane's
// tau and amplitudes take its theta alone:
//   (q.hi, q.lo, z.hi, z.lo) (rho.hi, rho.lo, b_rho, b_z) (1 - b_z, b_phi, a_rho, a_z) (a_phi)
// with rho = cos(phi) x + sin(phi) y.  Near: the records as they are.
template <bool NEAR>
__device__ __forceinline__ void stage_records(const FarMixedParams &p, int64_t g, uint32_t cnt,
                                              uint32_t cs, uint32_t n_phik, int lane,
                                              FastSmem &sm) {
  const float4 *src = p.records + g * kRecF4;
  if constexpr (NEAR) {
    if ((uint32_t)lane < cnt) {
#pragma unroll
      for (int k = 0; k < 3; ++k) sm.rec[lane * 3 + k] = __ldg(src + (size_t)lane * kRecF4 + k);
    }
  } else {
    const uint32_t n = cs * n_phik;
    for (uint32_t i = lane; i < n; i += 32u) {
      const uint32_t k = i / cs, s = i % cs;
      if (s >= cnt) continue;
      const float4 *r = src + (size_t)s * kRecF4;
      const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2), r3 = __ldg(r + 3);
      const float4 ph = sm.phic[k];
      const df rho = df_add(df_mul(df{ph.x, ph.y}, df{r0.z, r0.w}),
                            df_mul(df{ph.z, ph.w}, df{r1.x, r1.y}));
      float4 *d = sm.rec + k * (cs * 4u + 1u) + s * 4u;
      d[0] = make_float4(r0.x, r0.y, r1.z, r1.w);
      d[1] = make_float4(rho.hi, rho.lo, turned(ph.x, ph.y, r2.x, ph.z, ph.w, r2.y), r2.z);
      d[2] = make_float4(r2.w, turned(ph.x, ph.y, r2.y, -ph.z, -ph.w, r2.x),
                         turned(ph.x, ph.y, r3.x, ph.z, ph.w, r3.y), r3.z);
      d[3] = make_float4(turned(ph.x, ph.y, r3.y, -ph.z, -ph.w, r3.x), 0.f, 0.f, 0.f);
    }
  }
  __syncwarp();
}

// 1/d to FP32 rounding: the hardware estimate and one Newton step, 5 % of the
// spreading faster than __frcp_rn.  For every d of a binade and every estimate
// within its 1 ulp of error the step ends at the correctly rounded value or, once
// in a million, beside it (0.5 ulp + 1e-7).
__device__ __forceinline__ float rcp_newton(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float e = __fmaf_rn(-d, r, 1.0f);
  // an overflowed or zero estimate (d subnormal, 0 or infinite) stands as it is
  return fabsf(e) < 1.0f ? __fmaf_rn(r, e, r) : r;
}

// tau (near: tau - L) of step i of the chunk for the lane's direction, and
// its amplitudes: far X = A_theta, Y = A_phi; near X_c, Y_c of component c
// with A_c = Y_c + i omega X_c.
template <bool NEAR>
__device__ __forceinline__ df step_values(const LaneDir<NEAR> &ld, const FastSmem &sm,
                                          uint32_t rec0, uint32_t i, float (&X)[NEAR ? 3 : 1],
                                          float (&Y)[NEAR ? 3 : 1]) {
  if constexpr (!NEAR) {
    const float4 *r = sm.rec + rec0 + i * 4u;
    const float4 a = r[0], b = r[1], c = r[2];
    const float aphi = r[3].x;
    // tau = q + (1 - cos th) z - sin th rho  (double-float)
    const df p1 = df_mul_raw(df{ld.dc_h, ld.dc_l}, df{a.z, a.w});
    const df p2 = df_mul_raw(df{ld.st_h, ld.st_l}, df{b.x, b.y});
    const df s1 = two_sum(a.x, p1.hi);
    const df s2 = two_sum(s1.hi, -p2.hi);
    const df tau = fast_two_sum(s2.hi, ((a.y + p1.lo) - p2.lo) + (s1.lo + s2.lo));
    const float D = c.x + ld.f_dc * b.w - ld.f_st * b.z;
    const float c2 = rcp_newton(D);
    const float an = ld.f_st * c.z + ld.f_ct * c.w;
    const float c1 = an * c2 * c2;
    const float tb = ld.f_ct * b.z - ld.f_st * b.w;
    const float ta = ld.f_ct * c.z - ld.f_st * c.w;
    X[0] = -(c1 * tb + c2 * ta);
    Y[0] = -(c1 * c.y + c2 * aphi);
    return tau;
  } else {
    const float4 *r = sm.rec + i * 3u;
    const float4 r0 = r[0], r1 = r[1], r2 = r[2];
    // tau - L = (t - z) + rho^2 / (r + L - z)
    const df ddx = df_sub(df{ld.X_h, ld.X_l}, df{r0.z, r0.w});
    const df ddy = df_sub(df{ld.Y_h, ld.Y_l}, df{r1.x, r1.y});
    const df D = df_sub(df{ld.L_h, ld.L_l}, df{r1.z, r1.w});
    const df rho2 = df_add(df_mul(ddx, ddx), df_mul(ddy, ddy));
    const df rr = df_sqrt(df_add(rho2, df_mul(D, D)));
    const df F = (D.hi > 0.f) ? df_div(rho2, df_add(rr, D)) : df_sub(rr, D);
    const float rinv = __frcp_rn(rr.hi + rr.lo);
    const float nx = (ddx.hi + ddx.lo) * rinv, ny = (ddy.hi + ddy.lo) * rinv;
    const float nz = (D.hi + D.lo) * rinv;
    const float omn = (F.hi + F.lo) * rinv;  // 1 - n_z
    X[0] = (r2.x - nx) * rinv;
    X[1] = (r2.y - ny) * rinv;
    X[2] = (omn - r2.w) * rinv;
    const float q = rinv * rinv;
    Y[0] = nx * q; Y[1] = ny * q; Y[2] = nz * q;
    return df_add(df{r0.x, r0.y}, F);
  }
}

// Per-lane sweep state along one track.
template <bool NEAR>
struct Sweep {
  static constexpr int NP = NEAR ? 3 : 1;
  float2 gx[NP][kTaps], gy[NP][kTaps];  // cells cur-3 .. cur+4
  int cur;          // cell of the last included step (mod M)
  bool live;        // the window holds something
  float tp_h, tp_l; // tau of the previous step
  int n_list;       // entries of the lane's list
  bool dirty;       // the lane's direct sums hold something
};

template <bool NEAR>
__device__ __forceinline__ void window_clear(Sweep<NEAR> &w) {
#pragma unroll
  for (int c = 0; c < Sweep<NEAR>::NP; ++c)
#pragma unroll
    for (int l = 0; l < kTaps; ++l) w.gx[c][l] = w.gy[c][l] = make_float2(0.f, 0.f);
}

// The whole window to the lane's circle.
template <bool NEAR>
__device__ __forceinline__ void window_flush(Sweep<NEAR> &w, float4 *cells, int M) {
#pragma unroll
  for (int c = 0; c < Sweep<NEAR>::NP; ++c)
#pragma unroll
    for (int l = 0; l < kTaps; ++l)
      red_f4(cells + (size_t)c * 32 * M + ((w.cur - 3 + l) & (M - 1)), w.gx[c][l], w.gy[c][l]);
  window_clear(w);
}

// The included frequencies [jf, jl] of a step whose rule cuts the band: the
// certain interval (kPiLo), extended by the exact FP64 test through the
// guard band (up to kPiHi), as jf | jl << 16.  Empty: jf > jl.
template <bool NEAR>
__device__ __forceinline__ uint32_t cut_interval(const FarMixedParams &p, uint32_t j0, int nb,
                                              float w0f, float dwf, uint32_t dir, int64_t base, uint32_t s,
                                              uint32_t it_start, float adt) {
  const float inv_dw = 1.0f / dwf, inv_adt = __frcp_rn(adt);
  const uint32_t iT = dir % p.n_theta, iP = dir / p.n_theta;
  auto inside = [&](int j) -> bool {
    const double w = p.omega[j0 + j];
    if constexpr (NEAR)
      return exact_mask_near(p, base, s, it_start, w, p.sin_theta[iT] * p.cos_phi[iP],
                             p.sin_theta[iT] * p.sin_phi[iP]);
    else
      return exact_mask(p, base, s, it_start, w, p.sin_theta[iT] * p.cos_phi[iP],
                        p.sin_theta[iT] * p.sin_phi[iP], p.cos_theta[iT]);
  };
  int uf, ul, jf, jl;
  omega_interval(w0f, dwf, inv_dw, kPiLo * inv_adt, nb, jf, jl);
  omega_interval(w0f, dwf, inv_dw, kPiHi * inv_adt, nb, uf, ul);
  if (jf > jl) {  // no certain point: the first and last that pass the test
    jf = 1;
    jl = 0;
    for (int j = uf; j <= ul; ++j)
      if (inside(j)) {
        if (jf > jl) jf = j;
        jl = j;
      }
    return (uint32_t)jf | ((uint32_t)jl << 16);
  }
  while (jl + 1 <= ul && inside(jl + 1)) ++jl;
  while (jf - 1 >= uf && inside(jf - 1)) --jf;
  return (uint32_t)jf | ((uint32_t)jl << 16);
}

// Direct sums of the n listed steps of lane d (direction slot0 + d), by the whole
// warp: point j = lane + 32 k, seeded by sin/cos and rotated by exp(32 i d_omega
// tau), added to the lane's sums where they hold something (`add`).
// Pairs of entries share the packed FP32 operations, and two pairs run side by
// side: bound by the instructions of short dependent chains at 12 warps an SM
// (16 betatron tracks, half of their steps listed, 256 frequencies: one pair
// 35.8 ms, two 33.6, four 46.4, out of registers; the entries' values handed
// round by shuffles 38.5 where shared memory takes 35.8).  At most 8 blocks of
// 32 points per pass, so that the pair sums stay in registers.
constexpr int kPairF = 20;  // floats a staged pair takes (14, padded)
template <bool NEAR, int NK>
__device__ __forceinline__ void drain_one(const FarMixedParams &p, FastSlice<NEAR> sl,
                                          uint32_t slot0, uint32_t j0, int nb, double dw,
                                          int64_t base, uint32_t it_start, int d, int n, bool add,
                                          float *pairs, int lane) {
  constexpr int NP = NEAR ? 3 : 1;
  constexpr int KB = NK < 8 ? NK : 8;
  const double w0 = p.omega[0];
  const double inv2pi = 0.15915494309189533577;
  const df f32 = df_from_double(32.0 * dw * inv2pi);
  const float w0f = (float)(w0 + (double)j0 * dw), dwf = (float)dw;
  float4 *lhead = sl.lhead(p.fast) + (size_t)d * p.fast.list, *part = sl.part(p.fast);
  const float2 *lamp = sl.lamp(p.fast) + (size_t)d * p.fast.list;
  constexpr int kPairs = 2;
  // the included frequencies of each entry, in place of its |dtau|
  for (int e = lane; e < n; e += 32) {
    float4 *h = lhead + e;
    const float adt = __ldcg(&h->z);
    const uint32_t s = __float_as_uint(__ldcg(&h->w));
    h->z = __uint_as_float(
        cut_interval<NEAR>(p, j0, nb, w0f, dwf, slot0 + d, base, s, it_start, adt));
  }
  __syncwarp();
#pragma unroll 1
  for (int h0 = 0; h0 < NK; h0 += KB) {
    if (32 * h0 >= nb) break;
    const df fl = df_from_double((w0 + (double)(j0 + 32 * h0 + lane) * dw) * inv2pi);
#pragma unroll 1
    for (int c = 0; c < NP; ++c) {
      float2 xr[KB], xi[KB], yr[KB], yi[KB];  // .x: even entries, .y: odd entries
#pragma unroll
      for (int k = 0; k < KB; ++k) xr[k] = xi[k] = yr[k] = yi[k] = make_float2(0.f, 0.f);
      for (int e0 = 0; e0 < n; e0 += 32) {
        // a lane loads one entry and its rotation; the warp then takes the
        // entries in order
        const int ne = min(32, n - e0), el = e0 + min(lane, ne - 1);
        const float4 h = __ldcg(lhead + el);
        float2 am = __ldcg(lamp + (size_t)c * 32 * p.fast.list + el);
        const bool own = lane < ne;
        if (!own) am = make_float2(0.f, 0.f);
        float hs, hc;
        phasor_rev(f32.hi, f32.lo, h.x, h.y, hs, hc);
        __syncwarp();
        {
          float *q = pairs + (lane >> 1) * kPairF + (lane & 1);
          q[0] = h.x; q[2] = h.y; q[4] = own ? h.z : __uint_as_float(1u); q[6] = am.x;
          q[8] = am.y; q[10] = hc; q[12] = hs;
        }
        __syncwarp();
        for (int e = 0; e < ne; e += 2 * kPairs) {
          // kPairs chains of rotations side by side; entries past the last of
          // the list have no amplitude and end at block 0
          float2 vx[kPairs], vy[kPairs], rc[kPairs], rs[kPairs], zc[kPairs], zs[kPairs];
          int fa[kPairs], la[kPairs], fb[kPairs], lb[kPairs];
          int last = -1, whole = 0x7fff;
#pragma unroll
          for (int i = 0; i < kPairs; ++i) {
            const float4 *q =
                reinterpret_cast<const float4 *>(pairs + ((e >> 1) + i) * kPairF);
            const float4 q0 = q[0], q1 = q[1], q2 = q[2];
            rs[i] = *reinterpret_cast<const float2 *>(q + 3);
            vx[i] = make_float2(q1.z, q1.w);
            vy[i] = make_float2(q2.x, q2.y);
            rc[i] = make_float2(q2.z, q2.w);
            const uint32_t ra = __float_as_uint(q1.x), rb = __float_as_uint(q1.y);
            fa[i] = (int)(ra & 0xffffu) - 32 * h0;
            la[i] = (int)(ra >> 16) - 32 * h0;
            fb[i] = (int)(rb & 0xffffu) - 32 * h0;
            lb[i] = (int)(rb >> 16) - 32 * h0;
            // an entry without frequencies (fa > la) adds nothing below: its
            // block range is empty or masked
            last = max(last, max(la[i], lb[i]));
            whole = min(whole, max(fa[i], fb[i]) <= 0 ? min(la[i], lb[i]) + 1 : 0);
            phasor_rev(fl.hi, fl.lo, q0.x, q0.z, zs[i].x, zc[i].x);
            phasor_rev(fl.hi, fl.lo, q0.y, q0.w, zs[i].y, zc[i].y);
          }
          const int kw = whole >> 5;  // blocks below are included whole by all
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            if (32 * k > last) break;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
              float2 px = vx[i], py = vy[i];
              if (k >= kw) {
                const int j = lane + 32 * k;
                if (j < fa[i] || j > la[i]) px.x = py.x = 0.f;
                if (j < fb[i] || j > lb[i]) px.y = py.y = 0.f;
              }
              xr[k] = __ffma2_rn(px, zc[i], xr[k]);
              xi[k] = __ffma2_rn(px, zs[i], xi[k]);
              yr[k] = __ffma2_rn(py, zc[i], yr[k]);
              yi[k] = __ffma2_rn(py, zs[i], yi[k]);
              rot2p(zc[i], zs[i], rc[i], rs[i], make_float2(-rs[i].x, -rs[i].y), zc[i], zs[i]);
            }
          }
        }
      }
      // compensated: a track can empty its lists a thousand times
      float4 *a = part + ((size_t)c * 32 + d) * 2 * p.fast.nb + 32 * h0;
      float4 *al = a + p.fast.nb;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int j = lane + 32 * k;
        if (j + 32 * h0 < nb) {
          float4 v = make_float4(xr[k].x + xr[k].y, xi[k].x + xi[k].y, yr[k].x + yr[k].y,
                                 yi[k].x + yi[k].y);
          float4 l = make_float4(0.f, 0.f, 0.f, 0.f);
          if (add) {
            const float4 o = a[j];
            l = al[j];
            df t = two_sum(o.x, v.x);
            v.x = t.hi; l.x += t.lo;
            t = two_sum(o.y, v.y);
            v.y = t.hi; l.y += t.lo;
            t = two_sum(o.z, v.z);
            v.z = t.hi; l.z += t.lo;
            t = two_sum(o.w, v.w);
            v.w = t.hi; l.w += t.lo;
          }
          a[j] = v;
          al[j] = l;
        }
      }
    }
  }
  __syncwarp();
}

// d_omega (an FP64 division: once for all lists that a warp empties; the lists'
// kernel forms it per list, kept in registers there it cost 8 %).
__device__ __forceinline__ double axis_step(const FarMixedParams &p) {
  return (p.omega[p.n_omega - 1] - p.omega[0]) / (double)(p.n_omega - 1);
}

// The lists of every lane of the warp.
template <bool NEAR, int NK>
__device__ __forceinline__ void drain_lists(const FarMixedParams &p, FastSlice<NEAR> sl,
                                            uint32_t slot0, uint32_t j0, int nb, int64_t base,
                                            uint32_t it_start, int n_list, bool dirty, FastSmem &sm,
                                            int lane) {
  __syncwarp();
  const uint32_t old = __ballot_sync(0xffffffffu, dirty);
  const double dw = axis_step(p);
#pragma unroll 1
  for (uint32_t m = __ballot_sync(0xffffffffu, n_list > 0); m; m &= m - 1) {
    const int d = __ffs(m) - 1;
    drain_one<NEAR, NK>(p, sl, slot0, j0, nb, dw, base, it_start, d,
                        __shfl_sync(0xffffffffu, n_list, d), (old >> d) & 1u,
                        reinterpret_cast<float *>(sm.rec), lane);
  }
  __syncwarp();
}

// Spread steps [a, b) of a track into the lane's circle (steps before `from`
// only give the previous tau).
template <bool NEAR, int NK>
__device__ __forceinline__ void spread_steps(const FarMixedParams &p, const FastUnit<NEAR> &u,
                                             const FastSlice<NEAR> &sl, FastSmem &sm,
                                             Sweep<NEAR> &w, int64_t base, uint32_t it_start,
                                             uint32_t a, uint32_t b, uint32_t from, int lane) {
  constexpr int NP = NEAR ? 3 : 1;
  const int M = (int)p.fast.M;
  const float Mf = (float)M;
  const uint32_t cs = p.fast.chunk;
  float4 *cells = sl.grid() + (size_t)lane * M;
  const uint32_t rec0 = NEAR ? 0u : (uint32_t)u.kphi * (cs * 4u + 1u);
  for (uint32_t s0 = a, cnt = 0; s0 < b; s0 += cnt) {
    // the step before `from` stands alone, so that chunks start at `from`
    cnt = s0 < from ? 1u : min(cs, b - s0);
    __syncwarp();
    stage_records<NEAR>(p, base + s0, cnt, cs, p.fast.n_phik, lane, sm);
#pragma unroll 1
    for (uint32_t i = 0; i < cnt; ++i) {
      const uint32_t s = s0 + i;
      float X[NP], Y[NP];
      const df tau = step_values<NEAR>(u.ld, sm, rec0, i, X, Y);
      // the track's first step compares its whole phase with zero
      // (synchrad/kernel_farfield.cl:49, kernel_nearfield.cl:48)
      float dt0 = (tau.hi - w.tp_h) + (tau.lo - w.tp_l);
      if (s == 0) {
        dt0 = tau.hi + tau.lo;
        if constexpr (NEAR) dt0 += u.ld.L_h + u.ld.L_l;
      }
      const float adt = fabsf(dt0);
      w.tp_h = tau.hi;
      w.tp_l = tau.lo;
      const bool mine = u.active && s >= from;
      if (mine && u.wmax * adt < kPiLo) {
        // phase of the band's centre, whole turns dropped
        float zs, zc;
        phasor_exact(u.f_c.hi, u.f_c.lo, tau.hi, tau.lo, zs, zc);
        // cell of the step: d_omega tau / 2 pi turns of M cells
        const float pr = u.f_d.hi * tau.hi;
        float e = __fmaf_rn(u.f_d.hi, tau.hi, -pr);
        e = __fmaf_rn(u.f_d.hi, tau.lo, e);
        e = __fmaf_rn(u.f_d.lo, tau.hi, e);
        const float uh = (pr - rintf(pr)) * Mf, ul = e * Mf;
        const float rm = rintf((uh - 0.5f) + ul);
        const float f = ((uh - rm) - 0.5f) + ul;
        const int m = (int)rm;
        int adv = ((m - w.cur + M / 2) & (M - 1)) - M / 2;
        float t[kTaps];
        kb_taps(f, t);
        const float2 z = make_float2(zc, zs);
        // more than one cell on: all but the last plainly (each cell leaves once)
        while (w.live && adv > 1 && adv < kTaps) {
#pragma unroll
          for (int c = 0; c < NP; ++c) {
            red_f4(cells + (size_t)c * 32 * M + ((w.cur - 3) & (M - 1)), w.gx[c][0], w.gy[c][0]);
#pragma unroll
            for (int l = 0; l + 1 < kTaps; ++l) {
              w.gx[c][l] = w.gx[c][l + 1];
              w.gy[c][l] = w.gy[c][l + 1];
            }
            w.gx[c][kTaps - 1] = w.gy[c][kTaps - 1] = make_float2(0.f, 0.f);
          }
          ++w.cur;
          --adv;
        }
        if (w.live && adv == 1) {
#pragma unroll
          for (int c = 0; c < NP; ++c) {
            red_f4(cells + (size_t)c * 32 * M + ((w.cur - 3) & (M - 1)), w.gx[c][0], w.gy[c][0]);
            const float2 vx = __fmul2_rn(make_float2(X[c], X[c]), z);
            const float2 vy = __fmul2_rn(make_float2(Y[c], Y[c]), z);
#pragma unroll
            for (int l = 0; l + 1 < kTaps; ++l) {
              w.gx[c][l] = __ffma2_rn(make_float2(t[l], t[l]), vx, w.gx[c][l + 1]);
              w.gy[c][l] = __ffma2_rn(make_float2(t[l], t[l]), vy, w.gy[c][l + 1]);
            }
            w.gx[c][kTaps - 1] = __fmul2_rn(make_float2(t[kTaps - 1], t[kTaps - 1]), vx);
            w.gy[c][kTaps - 1] = __fmul2_rn(make_float2(t[kTaps - 1], t[kTaps - 1]), vy);
          }
          w.cur = m;
        } else {
          if (!w.live) {
            w.cur = m;
            w.live = true;
          } else if (adv != 0) {
            if (adv == -1) {
#pragma unroll
              for (int c = 0; c < NP; ++c) {
                red_f4(cells + (size_t)c * 32 * M + ((w.cur + 4) & (M - 1)), w.gx[c][kTaps - 1],
                       w.gy[c][kTaps - 1]);
#pragma unroll
                for (int l = kTaps - 1; l > 0; --l) {
                  w.gx[c][l] = w.gx[c][l - 1];
                  w.gy[c][l] = w.gy[c][l - 1];
                }
                w.gx[c][0] = w.gy[c][0] = make_float2(0.f, 0.f);
              }
            } else {
              window_flush(w, cells, M);
            }
            w.cur = m;
          }
#pragma unroll
          for (int c = 0; c < NP; ++c) {
            const float2 vx = __fmul2_rn(make_float2(X[c], X[c]), z);
            const float2 vy = __fmul2_rn(make_float2(Y[c], Y[c]), z);
#pragma unroll
            for (int l = 0; l < kTaps; ++l) {
              w.gx[c][l] = __ffma2_rn(make_float2(t[l], t[l]), vx, w.gx[c][l]);
              w.gy[c][l] = __ffma2_rn(make_float2(t[l], t[l]), vy, w.gy[c][l]);
            }
          }
        }
      } else if (mine && !(u.wmin * adt > kPiHi)) {
        const int k = w.n_list++;
        sl.lhead(p.fast)[lane * p.fast.list + k] =
            make_float4(tau.hi, tau.lo, adt, __uint_as_float(s));
#pragma unroll
        for (int c = 0; c < NP; ++c)
          sl.lamp(p.fast)[((size_t)c * 32 + lane) * p.fast.list + k] = make_float2(X[c], Y[c]);
      }
    }
    // cells that stay in the window for long would gather hundreds of terms:
    // started afresh every 128 steps (fewer where a sweep would lap the circle), their FP32 sums round a fifth as much
    const bool drain = __any_sync(0xffffffffu, w.n_list > (int)p.fast.list - 32);
    if (drain || ((s0 + cnt - from) & (p.fast.block - 1u)) == 0u) {
      if (w.live) window_flush(w, cells, M);
      if (drain) {
        drain_lists<NEAR, NK>(p, sl, u.slot0, u.j0, u.nb, base, it_start, w.n_list, w.dirty, sm, lane);
        w.dirty = w.dirty || w.n_list > 0;
        w.n_list = 0;
        window_clear(w);
      }
    }
  }
}

// Steps [a, b) of a track into the warp's circles and direct sums, nothing
// left in registers; returns whether the lane's direct sums hold something.
// LATER: the lists that are left are handed to fast_lists_kernel.
template <bool NEAR, int NK, bool LATER>
__device__ __forceinline__ bool spread_range(const FarMixedParams &p, const FastUnit<NEAR> &uref,
                                          FastSlice<NEAR> sl, FastSmem &sm, int64_t base,
                                          uint32_t it_start, uint32_t a, uint32_t b, bool dirty,
                                          uint32_t unit, int lane) {
  const FastUnit<NEAR> u = uref;
  Sweep<NEAR> w;
  window_clear(w);
  w.cur = 0;
  w.live = false;
  w.dirty = dirty;
  w.tp_h = w.tp_l = 0.f;
  w.n_list = 0;
  spread_steps<NEAR, NK>(p, u, sl, sm, w, base, it_start, a ? a - 1 : 0u, b, a, lane);
  if (w.live) window_flush(w, sl.grid() + (size_t)lane * p.fast.M, (int)p.fast.M);
  const uint32_t left = __ballot_sync(0xffffffffu, w.n_list > 0);
  if (LATER) {
    uint32_t at = 0;
    if (left && lane == 0) at = atomicAdd(p.fast.n_work, (uint32_t)__popc(left));
    at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(left & ((1u << lane) - 1u));
    if (w.n_list > 0) p.fast.work[at] = make_uint2(unit * 32u + lane, (uint32_t)w.n_list);
  } else if (left) {
    drain_lists<NEAR, NK>(p, sl, u.slot0, u.j0, u.nb, base, it_start, w.n_list, w.dirty, sm, lane);
    w.dirty = w.dirty || w.n_list > 0;
  }
  __threadfence();
  __syncwarp();
  return w.dirty;
}

// One pair of amplitudes A (X), B (Y) at frequency j of a direction, as the
// comp wants it, added to the partial spectrum `out`; A is also kept for the
// adjoints where asked.
template <bool NEAR>
__device__ __forceinline__ void emit_point(const FarMixedParams &p, uint32_t dir, int c, uint32_t j,
                                           uint32_t t, uint32_t ksnap, double wpdt2, double wpdt,
                                           double *out, double Ar, double Ai, double Br,
                                           double Bi) {
  const uint64_t P = (uint64_t)p.n_omega * p.n_theta * p.n_phi;
  const uint64_t gti = (uint64_t)j + (uint64_t)p.n_omega * dir;
  const uint32_t iT = dir % p.n_theta, iP = dir / p.n_theta;
  auto add = [&](int o, double v) {
    red_f64(out + ((uint64_t)o * p.n_snaps + ksnap) * P + gti, v);
  };
  if constexpr (!NEAR) {
    if (p.save_A != nullptr)
      reinterpret_cast<float4 *>(p.save_A)[((uint64_t)t * p.n_snaps + ksnap) * P + gti] =
          make_float4((float)Ar, (float)Ai, (float)Br, (float)Bi);
    if (p.comp == SR_COMP_TOTAL) {
      add(0, wpdt2 * (Ar * Ar + Ai * Ai + Br * Br + Bi * Bi));
    } else if (p.comp == SR_COMP_SPHERIC) {
      add(1, wpdt2 * (Ar * Ar + Ai * Ai));
      add(2, wpdt2 * (Br * Br + Bi * Bi));
    } else if (p.comp == SR_COMP_SPHERIC_COMPLEX) {
      add(2, wpdt * Ar);
      add(3, wpdt * Ai);
      add(4, wpdt * Br);
      add(5, wpdt * Bi);
    } else {
      const double cT = p.cos_theta[iT], sT = p.sin_theta[iT];
      const double cP = p.cos_phi[iP], sP = p.sin_phi[iP];
      const double hx = cT * cP, hy = cT * sP;
      const double xr = hx * Ar - sP * Br, xi = hx * Ai - sP * Bi;
      const double yr = hy * Ar + cP * Br, yi = hy * Ai + cP * Bi;
      const double zr = -sT * Ar, zi = -sT * Ai;
      if (p.comp == SR_COMP_CARTESIAN) {
        add(0, wpdt2 * (xr * xr + xi * xi));
        add(1, wpdt2 * (yr * yr + yi * yi));
        add(2, wpdt2 * (zr * zr + zi * zi));
      } else {
        const double f = wpdt * p.form_factor[j];
        add(0, f * xr);
        add(1, f * xi);
        add(2, f * yr);
        add(3, f * yi);
        add(4, f * zr);
        add(5, f * zi);
      }
    }
  } else {
    const double w = p.omega[j];
    const double Er = Br - w * Ai, Ei = Bi + w * Ar;  // Y + i omega X
    if (p.save_A != nullptr) {
      float *sa = p.save_A + 8 * (((uint64_t)t * p.n_snaps + ksnap) * P + gti);
      reinterpret_cast<float2 *>(sa)[c] = make_float2((float)Er, (float)Ei);
      if (c == 2) reinterpret_cast<float2 *>(sa)[3] = make_float2(0.f, 0.f);
    }
    if (p.comp == SR_COMP_TOTAL) {
      add(0, wpdt2 * (Er * Er + Ei * Ei));
    } else if (p.comp == SR_COMP_CARTESIAN) {
      add(c, wpdt2 * (Er * Er + Ei * Ei));
    } else {  // cartesian_complex (FormFactor not applied)
      double sL, cL;
      sincos(w * p.L_screen, &sL, &cL);
      add(2 * c, wpdt * (Er * cL - Ei * sL));
      add(2 * c + 1, wpdt * (Er * sL + Ei * cL));
    }
  }
}

// The band sums xs, ys (undivided) of one pair of fields added to the
// compensated sums `part` beside its circle, which they open where `add` is
// false.
template <bool NEAR>
__device__ __forceinline__ void fold_pair(const FarMixedParams &p, const FastUnit<NEAR> &u,
                                          const float2 *xs, const float2 *ys, float4 *part,
                                          bool add, int lane) {
  for (int m = lane; m < u.nb; m += 32) {
    const df dv = df_from_double(p.fast.deconv[m - u.nb / 2 + kFastMaxBand / 2]);
    const float2 x = xs[m], y = ys[m];
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), l = o;
    if (add) {
      o = part[m];
      l = part[p.fast.nb + m];
    }
    auto put = [&](float v, float &hi, float &lo) {
      const float h = v * dv.hi;
      const df s = two_sum(hi, h);
      hi = s.hi;
      lo += s.lo + (__fmaf_rn(v, dv.hi, -h) + v * dv.lo);
    };
    put(x.x, o.x, l.x);
    put(x.y, o.y, l.y);
    put(y.x, o.z, l.z);
    put(y.y, o.w, l.w);
    part[m] = o;
    part[p.fast.nb + m] = l;
  }
}

// The spectrum of one pair of fields, X and Y (band sums xs, ys, undivided),
// with the compensated sums of n_seg slices beside them (`dirty`: the directions
// for which they hold something, with FOLD `held` for the first slice), added to
// the partial spectrum of track subset `sub`.
// MANY: several slices.
template <bool NEAR, bool FOLD, bool MANY>
__device__ __forceinline__ void emit_pair(const FarMixedParams &p, const FastUnit<NEAR> &u,
                                          uint32_t dir, int d, int c, const float2 *xs,
                                          const float2 *ys, const float4 *part, int n_seg,
                                          uint32_t held, const uint32_t *dirty, uint32_t t,
                                          uint32_t ksnap, uint32_t sub, int lane) {
  const uint64_t P = (uint64_t)p.n_omega * p.n_theta * p.n_phi;
  const double wp = p.weight[t];
  const double wpdt2 = wp * p.dt * p.dt, wpdt = sqrt(wp) * p.dt;
  double *out = p.partial + (uint64_t)sub * p.n_out * p.n_snaps * P;
  auto holds = [&](int i) {
    return (((FOLD && i == 0 ? held : dirty[(size_t)i * p.fast.n_dwb]) >> d) & 1u) != 0u;
  };
  bool listed = false;
  for (int i = 0; i < n_seg; ++i) listed = listed || holds(i);
  const uint64_t g0 = (uint64_t)u.j0 + (uint64_t)p.n_omega * dir;
  const bool plain = p.comp == SR_COMP_TOTAL && p.save_A == nullptr;
  if (!listed && plain) {
    // |A|^2 from the FP32 sums in double-float (exact products), scaled and
    // added in FP64: a third of the FP64 operations of the general form below
    double *o = out + (uint64_t)ksnap * P + g0;
    for (int m = lane; m < u.nb; m += 32) {
      const double dv = p.fast.deconv[m - u.nb / 2 + kFastMaxBand / 2];
      const float2 x = xs[m], y = ys[m];
      df q;
      if constexpr (!NEAR) {
        q = df_norm2(x, y);
      } else {
        const double w = p.omega[u.j0 + m];
        const df wd = df_from_double(w);
        const df a = df_mul_raw(wd, df{-x.y, 0.f}), b = df_mul_raw(wd, df{x.x, 0.f});
        q = df_add(df_square(df_add(df{y.x, 0.f}, a)), df_square(df_add(df{y.y, 0.f}, b)));
      }
      red_f64(o + m, (wpdt2 * dv * dv) * ((double)q.hi + (double)q.lo));
    }
    return;
  }
  if (!MANY || !listed) {
    for (int m = lane; m < u.nb; m += 32) {
      const double dv = p.fast.deconv[m - u.nb / 2 + kFastMaxBand / 2];
      const float2 x = xs[m], y = ys[m];
      double Ar = (double)x.x * dv, Ai = (double)x.y * dv;
      double Br = (double)y.x * dv, Bi = (double)y.y * dv;
      if (!MANY && listed) {
        const float4 v = part[m], l = part[p.fast.nb + m];
        Ar += (double)v.x + (double)l.x;
        Ai += (double)v.y + (double)l.y;
        Br += (double)v.z + (double)l.z;
        Bi += (double)v.w + (double)l.w;
      }
      emit_point<NEAR>(p, dir, c, u.j0 + m, t, ksnap, wpdt2, wpdt, out, Ar, Ai, Br, Bi);
    }
    return;
  }
  // with direct sums of several slices: in double-float as well.  In FP64, two
  // operations per value and slice, the transforms of 20 near tracks of 600 steps, 10
  // a period, 140 directions, 512 frequencies took 0.87 ms, with 4 % of the
  // steps cut, and 0.37 with none; now 0.61.
  for (int m = lane; m < u.nb; m += 32) {
    const df dv = df_from_double(p.fast.deconv[m - u.nb / 2 + kFastMaxBand / 2]);
    const float2 x = xs[m], y = ys[m];
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    auto gather = [](float v, float vl, float &hi, float &lo) {
      const df e = two_sum(hi, v);
      hi = e.hi;
      lo += e.lo + vl;
    };
    for (int i = 0; i < n_seg; ++i)
      if (holds(i)) {  // direct sums of the listed steps, circles folded before
        const float4 *q = part + (size_t)i * (p.fast.slice_bytes * p.fast.n_dwb / 16) + m;
        const float4 v = q[0], vl = q[p.fast.nb];
        gather(v.x, vl.x, h.x, l.x);
        gather(v.y, vl.y, h.y, l.y);
        gather(v.z, vl.z, h.z, l.z);
        gather(v.w, vl.w, h.w, l.w);
      }
    auto amplitude = [&](float v, float hi, float lo) {
      const float q = v * dv.hi;
      const df e = two_sum(q, hi);
      return fast_two_sum(e.hi, e.lo + (lo + (__fmaf_rn(v, dv.hi, -q) + v * dv.lo)));
    };
    const df Ar = amplitude(x.x, h.x, l.x), Ai = amplitude(x.y, h.y, l.y);
    const df Br = amplitude(y.x, h.z, l.z), Bi = amplitude(y.y, h.w, l.w);
    if (plain) {
      df q;
      if constexpr (!NEAR) {
        q = df_add(df_add(df_square(Ar), df_square(Ai)), df_add(df_square(Br), df_square(Bi)));
      } else {
        const df wd = df_from_double(p.omega[u.j0 + m]);
        q = df_add(df_square(df_sub(Br, df_mul(wd, Ai))), df_square(df_add(Bi, df_mul(wd, Ar))));
      }
      red_f64(out + (uint64_t)ksnap * P + g0 + m, wpdt2 * ((double)q.hi + (double)q.lo));
    } else {
      emit_point<NEAR>(p, dir, c, u.j0 + m, t, ksnap, wpdt2, wpdt, out,
                       (double)Ar.hi + (double)Ar.lo, (double)Ai.hi + (double)Ai.lo,
                       (double)Br.hi + (double)Br.lo, (double)Bi.hi + (double)Bi.lo);
    }
  }
}

// Transforms the pairs [pr0, pr1) (pair = local direction x NP + c) of one
// track, the circles of n_circ slices from `circles` on added up, and folds them
// into the first slice's sums (FOLD and `fold`) or emits them with the sums of
// n_seg slices from `slice0` on.
template <bool NEAR, int R1, bool FOLD, bool MANY>
__device__ __forceinline__ void transform_pairs(const FarMixedParams &p, const FastUnit<NEAR> &u,
                                                const unsigned char *circles, int n_circ,
                                                unsigned char *slice0, int n_seg, uint32_t held,
                                                const uint32_t *dirty, bool fold, FastSmem &sm,
                                                int pr0, int pr1, uint32_t t, uint32_t ksnap,
                                                uint32_t sub, int lane) {
  constexpr int NP = NEAR ? 3 : 1;
  constexpr int NF = 32 / R1, M = 32 * R1;
  const uint32_t n_dirs = p.n_theta * p.n_phi;
  const size_t stride = p.fast.slice_bytes * p.fast.n_dwb;  // between a track's segments
  const float4 *grid = (const float4 *)circles;
  float4 *parts = (float4 *)slice0 + (size_t)NP * 32 * M;
  auto emit = [&](int pr, const float2 *xs, const float2 *ys) {
    const int d = pr / NP, c = pr % NP;
    float4 *part = parts + ((size_t)c * 32 + d) * 2 * p.fast.nb;
    if (FOLD && fold)
      fold_pair<NEAR>(p, u, xs, ys, part, (held >> d) & 1u, lane);
    else
      emit_pair<NEAR, FOLD, MANY>(p, u, u.slot0 + d, d, c, xs, ys, part, n_seg, held, dirty, t, ksnap, sub,
                      lane);
  };
  if constexpr (R1 == 32) {
    for (int pr = pr0; pr < pr1; ++pr) {
      const int d = pr / NP, c = pr % NP;
      if (u.slot0 + d >= n_dirs) break;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {  // field X, then Y
        float2 x[1][32];
        const float2 *g = (const float2 *)(grid + ((size_t)c * 32 + d) * M) + h;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[0][i] = __ldcg(g + 2 * (32 * i + lane));
        for (int sg = 1; sg < n_circ; ++sg) {
          const float2 *gs = g + (size_t)sg * (stride / 8);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float2 v = __ldcg(gs + 2 * (32 * i + lane));
            x[0][i].x += v.x;
            x[0][i].y += v.y;
          }
        }
        fft_band<32, 1>(x, sm.tr, p.fast.twiddle, lane, u.nb, h ? sm.tr : sm.out);
      }
      emit(pr, sm.out, sm.tr);
      __syncwarp();
    }
  } else {
    for (int q0 = pr0; q0 < pr1; q0 += NF / 2) {
      if (u.slot0 + q0 / NP >= n_dirs) break;
      float2 x[NF][R1];
#pragma unroll
      for (int k = 0; k < NF / 2; ++k) {
        const int pr = min(q0 + k, pr1 - 1), d = pr / NP, c = pr % NP;
        const float4 *g = grid + ((size_t)c * 32 + d) * M;
#pragma unroll
        for (int i = 0; i < R1; ++i) {
          const float4 v = __ldcg(g + 32 * i + lane);
          x[2 * k][i] = make_float2(v.x, v.y);
          x[2 * k + 1][i] = make_float2(v.z, v.w);
        }
        for (int sg = 1; sg < n_circ; ++sg) {
          const float4 *gs = g + (size_t)sg * (stride / 16);
#pragma unroll
          for (int i = 0; i < R1; ++i) {
            const float4 v = __ldcg(gs + 32 * i + lane);
            x[2 * k][i].x += v.x;
            x[2 * k][i].y += v.y;
            x[2 * k + 1][i].x += v.z;
            x[2 * k + 1][i].y += v.w;
          }
        }
      }
      fft_band<R1, NF>(x, sm.tr, p.fast.twiddle, lane, u.nb, sm.out);
#pragma unroll 1
      for (int k = 0; k < NF / 2; ++k) {
        const int pr = q0 + k;
        if (pr >= pr1 || u.slot0 + pr / NP >= n_dirs) break;
        emit(pr, sm.out + (2 * k) * u.nb, sm.out + (2 * k + 1) * u.nb);
      }
      __syncwarp();
    }
  }
}

// Tracks of subset `sub`: one each when there are as many subsets as tracks.
__device__ __forceinline__ void fast_tracks_of(const FarMixedParams &p, uint32_t sub, uint32_t &t0,
                                               uint32_t &t1) {
  if (p.fast.n_sub == p.n_tracks) {
    t0 = sub;
    t1 = sub + 1;
  } else {
    subset_range(p, sub, p.fast.n_sub, t0, t1);
  }
}

template <bool NEAR>
__device__ __forceinline__ void clear_circles(const FastSlice<NEAR> &sl, uint32_t M, int lane) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t i = lane; i < FastSlice<NEAR>::NP * 32u * M; i += 32u) __stcg(sl.grid() + i, zero);
  __threadfence();
  __syncwarp();
}

// Whole tracks: a warp takes (32 directions x band, track subset) items from
// a queue, and for each track spreads its steps, transforms the 32 circles
// and adds the spectra at every snapshot.
//
// Bound by the spreading loop's instructions, about 150 a step and warp (df tau
// and amplitudes 60, taps 45, sums 32 packed, the window's moves) at 12 warps an
// SM (near 8): far 48 % of the issue slots, ALU and FMA pipes 30 % each; 168
// registers inlined are twice as fast as 128 or as a called transform.  32
// tracks of 4000 steps, 512 x 64 x 64 points: 85.8 ms term by term, 6.6 here;
// near, 16 tracks of 8000 steps, 256 x 64 x 64: 83.8 and 13.7 ms.  1024 tracks,
// 512 x 64 x 64: 2.71 s and 183 ms.
// FOLD: the tracks of more than fold_steps(M) steps (a launch of their own, only
// where there can be any: with the fold in one kernel the spreading loop of all
// tracks lost 1.5 % to the registers it takes).
template <bool NEAR, int R1, bool FOLD>
__global__ void __launch_bounds__(kFastWarps * 32, NEAR ? 2 : 3)
fast_tracks_kernel(const __grid_constant__ FarMixedParams p) {
  if (*p.fast.uneven || (FOLD && !p.fast.uneven[1])) return;
  constexpr int NP = NEAR ? 3 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FastSmem &sm = reinterpret_cast<FastSmem *>(smem_raw)[warp];
  const FastParams &f = p.fast;
  const uint32_t wid = blockIdx.x * kFastWarps + warp;
  const FastSlice<NEAR> sl(f, wid);
  const uint32_t n_items = f.n_dwb * f.n_sub;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(f.queue + FOLD, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n_items) return;
    const uint32_t sub = item / f.n_dwb;
    FastUnit<NEAR> u;
    __syncwarp();
    unit_init<NEAR>(p, item % f.n_dwb, lane, sm, u);
    uint32_t t0, t1;
    fast_tracks_of(p, sub, t0, t1);
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t n_body = track_body(p, t);
      if (FOLD != (n_body > fold_steps(32 * R1))) continue;
      const uint32_t it_start = p.it_start[t], it_end = p.it_end[t];
      const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
      SnapState snap;
      snap.init(it_start, it_end, snaps, p.n_snaps);
      if (snap.fire_it == SnapState::NEVER) continue;  // nothing of the track is written
      clear_circles<NEAR>(sl, 32 * R1, lane);
      bool dirty_l = false;
      const int64_t base = p.offsets[t];
      uint32_t s = 0;
      // steps up to each snapshot's write; those due after the last body step
      // repeat the same amplitudes; steps after the last write enter nothing
      while (snap.fire_it != SnapState::NEVER) {
        const uint32_t due = (uint32_t)min((int64_t)n_body, snap.fire_it + 1);
        const uint32_t full = (s & ~(fold_steps(32 * R1) - 1u)) + fold_steps(32 * R1);
        const bool fold = FOLD && due > full;
        const uint32_t e = fold ? full : due;
        if (e > s) {
          dirty_l = spread_range<NEAR, R1 / 2, false>(p, u, sl, sm, base, it_start, s, e, dirty_l,
                                                      0u, lane);
          s = e;
        }
        const uint32_t held = __ballot_sync(0xffffffffu, dirty_l);
        transform_pairs<NEAR, R1, FOLD, false>(p, u, sl.base, 1, sl.base, 1, held, &held, fold, sm,
                                               0, 32 * NP, t, snap.k, sub, lane);
        if (fold) {
          clear_circles<NEAR>(sl, 32 * R1, lane);
          dirty_l = true;
        } else {
          snap.advance(it_start, it_end, snaps, p.n_snaps);
        }
      }
    }
  }
}

// Few tracks: first the steps, each unit into its own slice, so that every SM
// has work.  A unit is a segment of f.seg_steps steps (one snapshot; track t's
// segments start at first_segment(t), one number spare per track) or the
// steps between two snapshots (f.seg_steps = 0) ...
__device__ __forceinline__ uint32_t first_segment(const FarMixedParams &p, uint32_t t) {
  return (uint32_t)((uint64_t)p.offsets[t] / p.fast.seg_steps) + t;
}
// The track's k-th snapshot write, and the first step that the one before it
// does not enter; false if there is none.
__device__ __forceinline__ bool nth_snapshot(const FarMixedParams &p, uint32_t t, uint32_t k,
                                             SnapState &snap, uint64_t &from) {
  const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
  snap.init(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  from = 0;
  for (uint32_t i = 0; i < k && snap.fire_it != SnapState::NEVER; ++i) {
    from = (uint64_t)snap.fire_it + 1;
    snap.advance(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  }
  return snap.fire_it != SnapState::NEVER;
}

// Track of unit gs / n_dwb.
__device__ __forceinline__ uint32_t unit_track(const FarMixedParams &p, uint32_t gs) {
  if (p.fast.seg_steps == 0) return gs / p.n_snaps;
  uint32_t lo = 0, hi = p.n_tracks;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (first_segment(p, mid) <= gs) lo = mid; else hi = mid;
  }
  return lo;
}

// FOLD: the units of more than fold_steps(M).
template <bool NEAR, int R1, bool FOLD>
__global__ void __launch_bounds__(kFastWarps * 32, NEAR ? 2 : 3)
fast_spread_kernel(const __grid_constant__ FarMixedParams p) {
  if (*p.fast.uneven || (FOLD && !p.fast.uneven[1])) return;
  constexpr int NP = NEAR ? 3 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FastSmem &sm = reinterpret_cast<FastSmem *>(smem_raw)[warp];
  const FastParams &f = p.fast;
  const uint32_t unit = blockIdx.x * kFastWarps + warp;
  if (unit >= f.n_segs * f.n_dwb) return;
  const uint32_t gs = unit / f.n_dwb, dwb = unit % f.n_dwb;
  const uint32_t t = unit_track(p, gs);
  uint64_t a, b;
  if (f.seg_steps == 0) {  // the steps between two snapshots
    SnapState snap;
    if (!nth_snapshot(p, t, gs % p.n_snaps, snap, a)) return;
    b = (uint64_t)min((int64_t)track_body(p, t), snap.fire_it + 1);
    a = min(a, b);
  } else {
    a = (uint64_t)(gs - first_segment(p, t)) * f.seg_steps;
    SnapState snap;
    uint64_t from;
    if (!nth_snapshot(p, t, 0, snap, from)) return;
    const uint64_t n = (uint64_t)min((int64_t)track_body(p, t), snap.fire_it + 1);
    if (a >= n && a > 0) return;  // no segment of the track
    b = min(n, a + f.seg_steps);
  }
  if (FOLD != (b > a && b - a > fold_steps(32 * R1))) return;
  const FastSlice<NEAR> sl(f, unit);
  FastUnit<NEAR> u;
  unit_init<NEAR>(p, dwb, lane, sm, u);
  clear_circles<NEAR>(sl, f.M, lane);
  bool dirty_l = false;
  while (b > a) {
    const uint64_t e = FOLD ? min(b, a + fold_steps(32 * R1)) : b;
    dirty_l = spread_range<NEAR, R1 / 2, !FOLD>(p, u, sl, sm, p.offsets[t], p.it_start[t],
                                                (uint32_t)a, (uint32_t)e, dirty_l, unit, lane);
    a = e;
    if (FOLD && a < b) {
      const uint32_t held = __ballot_sync(0xffffffffu, dirty_l);
      transform_pairs<NEAR, R1, true, false>(p, u, sl.base, 1, sl.base, 1, held, nullptr, true, sm,
                                             0, 32 * NP, t, 0u, 0u, lane);
      clear_circles<NEAR>(sl, f.M, lane);
      dirty_l = true;
    }
  }
  const uint32_t dirty = __ballot_sync(0xffffffffu, dirty_l);
  if (lane == 0) f.dirty[unit] = dirty;
}

// ... then the lists of cut steps that the segments are left with, a warp per list:
// cut steps crowd in some directions and segments, and a warp that had to empty all
// of its lanes' lists kept the others waiting (87 betatron tracks of 456 to 918
// steps, 354 x 70 x 2 points: 2.66 ms, term by term 2.04, now 1.33; far, 87 tracks
// of 300 steps, 8 a period, 512 x 140: 2.95, 1.36, 1.30; near, 20 tracks of 600 steps,
// 8 a period, 300 x 140: 2.09, 1.17, 1.01) ...
template <bool NEAR, int R1>
__global__ void __launch_bounds__(kFastWarps * 32, 4)
fast_lists_kernel(const __grid_constant__ FarMixedParams p) {
  if (*p.fast.uneven) return;
  __shared__ __align__(16) float pairs[kFastWarps][16 * kPairF];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const FastParams &f = p.fast;
  const uint32_t n_work = f.n_work[0];
  if (n_work == 0u) return;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(f.n_work + 1, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n_work) return;
    const uint2 w = f.work[item];
    const uint32_t unit = w.x / 32u, d = w.x % 32u, dwb = unit % f.n_dwb;
    const uint32_t t = unit_track(p, unit / f.n_dwb);
    const uint32_t j0 = dwb % f.n_bands * f.nb;
    const bool add = (__ldcg(f.dirty + unit) >> d) & 1u;
    drain_one<NEAR, R1 / 2>(p, FastSlice<NEAR>(f, unit), dwb / f.n_bands * 32u, j0,
                            (int)min(f.nb, p.n_omega - j0), axis_step(p), p.offsets[t],
                            p.it_start[t], (int)d, (int)w.y, add, pairs[warp], lane);
    if (lane == 0) atomicOr(f.dirty + unit, 1u << d);
  }
}

// ... then, a few directions per warp and its track subset, the transforms of
// the summed circles.  FOLD: of the tracks whose segments are more than one circle
// may sum.
template <bool NEAR, int R1, bool FOLD>
__global__ void __launch_bounds__(kFastWarps * 32, 4)
fast_transform_kernel(const __grid_constant__ FarMixedParams p) {
  if (*p.fast.uneven || (FOLD && !p.fast.uneven[1])) return;
  constexpr int NP = NEAR ? 3 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FastSmem &sm = reinterpret_cast<FastSmem *>(smem_raw)[warp];
  const FastParams &f = p.fast;
  uint32_t item = blockIdx.x * kFastWarps + warp;
  const uint32_t per = f.dirs_per_warp, n_g = 32u / per;
  if (item >= f.n_dwb * n_g * f.n_sub * p.n_snaps) return;
  const uint32_t g = item % n_g;
  item /= n_g;
  const uint32_t dwb = item % f.n_dwb;
  item /= f.n_dwb;
  const uint32_t k = item % p.n_snaps, sub = item / p.n_snaps;
  FastUnit<NEAR> u;
  unit_init<NEAR>(p, dwb, lane, sm, u);
  uint32_t t0, t1;
  fast_tracks_of(p, sub, t0, t1);
  for (uint32_t t = t0; t < t1; ++t) {
    SnapState snap;
    uint64_t from;
    if (!nth_snapshot(p, t, k, snap, from)) continue;
    size_t unit0;
    int n_seg;
    if (f.seg_steps == 0) {
      unit0 = (size_t)t * p.n_snaps;
      n_seg = (int)k + 1;
    } else {
      const uint64_t n = (uint64_t)min((int64_t)track_body(p, t), snap.fire_it + 1);
      unit0 = first_segment(p, t);
      n_seg = n ? (int)((n + f.seg_steps - 1) / f.seg_steps) : 1;
    }
    unit0 = unit0 * f.n_dwb + dwb;
    unsigned char *slice0 = f.scratch + unit0 * f.slice_bytes;
    uint32_t held = FOLD ? f.dirty[unit0] : 0u;
    // circles of segments: plain sums of up to fold_steps(M) steps, as one
    // circle would hold them
    const int many =
        f.seg_steps == 0 ? n_seg : (int)max(1u, fold_steps(32 * R1) / f.seg_steps);
    if (FOLD != (n_seg > many)) continue;
    for (int c0 = 0; c0 < (FOLD ? n_seg : 1); c0 += many) {
      const bool fold = FOLD && c0 + many < n_seg;
      transform_pairs<NEAR, R1, FOLD, true>(p, u, slice0 + (size_t)c0 * f.n_dwb * f.slice_bytes,
                                      FOLD ? min(many, n_seg - c0) : n_seg, slice0, n_seg, held,
                                      f.dirty + unit0, fold, sm, (int)(g * per) * NP,
                                      (int)((g + 1) * per) * NP, t, snap.k, sub, lane);
      held = 0xffffffffu;
    }
  }
}

// Axes that are not evenly spaced: a sine and a cosine per point and step.  A
// warp takes (direction, 32 K frequencies, track subset) items; its lanes
// compute tau and the amplitudes of 32 steps, one each, then every lane sums
// its K frequencies lane + 32 m over them (the frequencies as double-floats in
// registers; the FP32 sums fold into compensated pairs every 1024 steps).
// Bound by the XU pipe: two hardware functions per point and step, 0.125
// cycles per SM.
template <bool NEAR, int K>
__global__ void __launch_bounds__(kFastWarps * 32, 3)
uneven_axis_kernel(const __grid_constant__ FarMixedParams p) {
  if (*p.fast.uneven == 0u) return;
  constexpr int NP = NEAR ? 3 : 1, NV = 4 * NP;  // pairs, real sums per point
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FastSmem &sm = reinterpret_cast<FastSmem *>(smem_raw)[warp];
  float4 *sv = sm.rec + 160;                           // tau.hi, tau.lo, |dtau| of a step
  float2 *sa = reinterpret_cast<float2 *>(sm.rec + 192);  // [NP][32] amplitudes X, Y
  const uint32_t n_dirs = p.n_theta * p.n_phi, nO = p.n_omega;
  const uint64_t P = (uint64_t)nO * n_dirs;
  const uint32_t tiles = (nO + 32 * K - 1) / (32 * K);
  const uint64_t n_items = (uint64_t)n_dirs * tiles * p.n_sub;
  const double inv2pi = 0.15915494309189533577;
  for (;;) {
    uint32_t item32 = 0;
    if (lane == 0) item32 = atomicAdd(p.queue, 1u);
    const uint64_t item = __shfl_sync(0xffffffffu, item32, 0);
    if (item >= n_items) return;
    const uint32_t sub = (uint32_t)(item / ((uint64_t)n_dirs * tiles));
    const uint32_t rest = (uint32_t)(item % ((uint64_t)n_dirs * tiles));
    const uint32_t dir = rest / tiles, j0 = (rest % tiles) * 32u * K + lane;
    const uint32_t iT = dir % p.n_theta, iP = dir / p.n_theta;
    LaneDir<NEAR> ld;
    lane_dir(p, iT, iP, ld);
    __syncwarp();
    if constexpr (!NEAR) {
      if (lane == 0) sm.phic[0] = phi_pairs(p, iP);
    }
    __syncwarp();
    float wh[K], wl[K], wa[K];
    float wmax = 0.f;
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const double w = p.omega[min(j0 + 32u * m, nO - 1u)];
      const df r = df_from_double(w * inv2pi);
      wh[m] = r.hi;
      wl[m] = r.lo;
      wa[m] = (float)fabs(w);
      wmax = wa[m] <= 3.0e38f ? fmaxf(wmax, wa[m]) : INFINITY;  // NaN and infinity too
    }
    double *out = p.partial + (uint64_t)sub * p.n_out * p.n_snaps * P;
    uint32_t t0, t1;
    subset_tracks(p, sub, t0, t1);
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t n_body = track_body(p, t);
      const uint32_t it_start = p.it_start[t], it_end = p.it_end[t];
      const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
      SnapState snap;
      snap.init(it_start, it_end, snaps, p.n_snaps);
      if (snap.fire_it == SnapState::NEVER) continue;
      const int64_t base = p.offsets[t];
      const double wpdt2 = p.weight[t] * p.dt * p.dt, wpdt = sqrt(p.weight[t]) * p.dt;
      float acc[K][NV], hi[K][NV], lo[K][NV];
#pragma unroll
      for (int m = 0; m < K; ++m)
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[m][v] = hi[m][v] = lo[m][v] = 0.f;
      auto fold = [&]() {
#pragma unroll
        for (int m = 0; m < K; ++m)
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            const df e = two_sum(hi[m][v], acc[m][v]);
            hi[m][v] = e.hi;
            lo[m][v] += e.lo;
            acc[m][v] = 0.f;
          }
      };
      auto flush = [&]() {
        fold();
#pragma unroll
        for (int m = 0; m < K; ++m) {
          const uint32_t j = j0 + 32u * m;
          if (j < nO) {
#pragma unroll
            for (int c = 0; c < NP; ++c) {
              auto val = [&](int v) { return (double)hi[m][4 * c + v] + (double)lo[m][4 * c + v]; };
              emit_point<NEAR>(p, dir, c, j, t, snap.k, wpdt2, wpdt, out, val(0), val(1), val(2),
                               val(3));
            }
          }
        }
        snap.advance(it_start, it_end, snaps, p.n_snaps);
      };
      float tp_h = 0.f, tp_l = 0.f;
      for (uint32_t s0 = 0; s0 < n_body && snap.fire_it != SnapState::NEVER; s0 += 32) {
        const uint32_t cnt = min(32u, n_body - s0);
        __syncwarp();
        stage_records<NEAR>(p, base + s0, cnt, 32u, 1u, lane, sm);
        {
          const uint32_t l = min((uint32_t)lane, cnt - 1);
          float X[NP], Y[NP];
          const df tau = step_values<NEAR>(ld, sm, 0u, l, X, Y);
          float ph = __shfl_up_sync(0xffffffffu, tau.hi, 1);
          float pl = __shfl_up_sync(0xffffffffu, tau.lo, 1);
          if (lane == 0) { ph = tp_h; pl = tp_l; }
          float dt0 = (tau.hi - ph) + (tau.lo - pl);
          if (s0 + l == 0) {  // the first step's whole phase is compared with zero
            dt0 = tau.hi + tau.lo;
            if constexpr (NEAR) dt0 += ld.L_h + ld.L_l;
          }
          tp_h = __shfl_sync(0xffffffffu, tau.hi, cnt - 1);
          tp_l = __shfl_sync(0xffffffffu, tau.lo, cnt - 1);
          sv[lane] = make_float4(tau.hi, tau.lo, fabsf(dt0), 0.f);
#pragma unroll
          for (int c = 0; c < NP; ++c) sa[c * 32 + lane] = make_float2(X[c], Y[c]);
        }
        __syncwarp();
#pragma unroll 1
        for (uint32_t i = 0; i < cnt; ++i) {
          const float4 q = sv[i];
          float2 am[NP];
#pragma unroll
          for (int c = 0; c < NP; ++c) am[c] = sa[c * 32 + i];
          const bool all_in = __all_sync(0xffffffffu, wmax * q.z < kPiLo);
#pragma unroll
          for (int m = 0; m < K; ++m) {
            bool in = true;
            if (!all_in) {
              const float ph = wa[m] * q.z;
              if (ph < kPiLo) {
                in = true;
              } else if (ph > kPiHi) {
                in = false;
              } else {
                const double w = p.omega[min(j0 + 32u * m, nO - 1u)];
                const double n0 = p.sin_theta[iT] * p.cos_phi[iP];
                const double n1 = p.sin_theta[iT] * p.sin_phi[iP];
                in = NEAR ? exact_mask_near(p, base, s0 + i, it_start, w, n0, n1)
                          : exact_mask(p, base, s0 + i, it_start, w, n0, n1, p.cos_theta[iT]);
              }
            }
            float sn, cs;
            phasor_rev(wh[m], wl[m], q.x, q.y, sn, cs);
            if (!in) sn = cs = 0.f;
#pragma unroll
            for (int c = 0; c < NP; ++c) {
              acc[m][4 * c + 0] = __fmaf_rn(am[c].x, cs, acc[m][4 * c + 0]);
              acc[m][4 * c + 1] = __fmaf_rn(am[c].x, sn, acc[m][4 * c + 1]);
              acc[m][4 * c + 2] = __fmaf_rn(am[c].y, cs, acc[m][4 * c + 2]);
              acc[m][4 * c + 3] = __fmaf_rn(am[c].y, sn, acc[m][4 * c + 3]);
            }
          }
          if ((int64_t)(s0 + i) == snap.fire_it) flush();  // uniform over the warp
        }
        if (((s0 + 32) & 1023u) == 0) fold();
      }
      while (snap.fire_it != SnapState::NEVER) flush();  // due after the last body step
    }
  }
}

// ------------------------------------------------------------------ host side
inline uint32_t fast_cells(uint32_t nb) {
  uint32_t M = 128;
  while (M < 2 * nb) M *= 2;
  return M;
}
constexpr size_t kFastTables = (kFastMaxBand + 2) * 8 + 1024 * 16;

// p.fast's tables (made by the record pass) at `tables`, the axis test in the
// status block.
inline void fast_tables_bind(FarMixedParams &p, uint32_t n_bands, uint32_t nb, uint32_t M,
                             unsigned char *tables, unsigned char *status) {
  p.fast.uneven = (unsigned int *)(status + 64);
  p.fast.deconv = (double *)tables;
  p.fast.twiddle = (float4 *)(tables + (kFastMaxBand + 2) * 8);
  p.fast.n_bands = n_bands;
  p.fast.nb = nb;
  p.fast.M = M;
}

template <bool NEAR, int R1>
int launch_fast_r(const FarMixedParams &p, const FastLayout &l, cudaStream_t s) {
  constexpr int smem = (int)sizeof(FastSmem) * kFastWarps;
  const unsigned threads = kFastWarps * 32;
  cudaError_t e = cudaSuccess;
  auto launch = [&](auto *kernel, uint32_t blocks) {
    if (e == cudaSuccess) e = allow_smem((const void *)kernel, smem);
    if (e == cudaSuccess) kernel<<<blocks, threads, smem, s>>>(p);
  };
  // whether a track can have more steps than a circle takes
  const bool longer = p.total_steps > (int64_t)fold_steps(l.M);
  if (!l.split) {
    launch(fast_tracks_kernel<NEAR, R1, false>, l.slices / kFastWarps);
    if (longer) launch(fast_tracks_kernel<NEAR, R1, true>, l.slices / kFastWarps);
  } else {
    launch(fast_spread_kernel<NEAR, R1, false>, l.slices / kFastWarps);
    if (longer && (l.seg_steps == 0 || l.seg_steps > fold_steps(l.M)))
      launch(fast_spread_kernel<NEAR, R1, true>, l.slices / kFastWarps);
    if (e == cudaSuccess) fast_lists_kernel<NEAR, R1><<<4 * l.n_sm, threads, 0, s>>>(p);
    const uint32_t items = l.n_dwb * (32u / l.dirs_per_warp) * l.n_sub * p.n_snaps;
    const uint32_t blocks = (items + kFastWarps - 1) / kFastWarps;
    launch(fast_transform_kernel<NEAR, R1, false>, blocks);
    if (longer && l.seg_steps) launch(fast_transform_kernel<NEAR, R1, true>, blocks);
  }
  if (e != cudaSuccess) return cuda_fail(e, "fast sum smem attribute");
  return cuda_fail(cudaGetLastError(), "fast sum launch");
}

template <bool NEAR, int K>
int launch_uneven_k(const FarMixedParams &p, int n_sm, cudaStream_t s) {
  constexpr int smem = (int)sizeof(FastSmem) * kFastWarps;
  const cudaError_t e = allow_smem((const void *)uneven_axis_kernel<NEAR, K>, smem);
  if (e != cudaSuccess) return cuda_fail(e, "uneven axis smem attribute");
  uneven_axis_kernel<NEAR, K><<<(unsigned)n_sm * 3, kFastWarps * 32, smem, s>>>(p);
  return cuda_fail(cudaGetLastError(), "uneven axis launch");
}

// The fewest tiles of at most 8 (near: 3) x 32 frequencies, and the fewest
// frequencies per lane that fill them.
template <bool NEAR>
int launch_uneven(const FarMixedParams &p, int n_sm, cudaStream_t s) {
  constexpr uint32_t most = NEAR ? 3 : 8;
  const uint32_t tiles = (p.n_omega + 32 * most - 1) / (32 * most);
  const uint32_t K = (p.n_omega + 32 * tiles - 1) / (32 * tiles);
  switch (K) {
    case 1: return launch_uneven_k<NEAR, 1>(p, n_sm, s);
    case 2: return launch_uneven_k<NEAR, 2>(p, n_sm, s);
    case 3: return launch_uneven_k<NEAR, 3>(p, n_sm, s);
  }
  if constexpr (!NEAR) {
    switch (K) {
      case 4: return launch_uneven_k<NEAR, 4>(p, n_sm, s);
      case 5: return launch_uneven_k<NEAR, 5>(p, n_sm, s);
      case 6: return launch_uneven_k<NEAR, 6>(p, n_sm, s);
      case 7: return launch_uneven_k<NEAR, 7>(p, n_sm, s);
      case 8: return launch_uneven_k<NEAR, 8>(p, n_sm, s);
    }
  }
  return fail(SR_ERR_INVALID, "%u frequencies per lane", K);
}

template <bool NEAR>
int launch_fast(const FarMixedParams &p, const FastLayout &l, cudaStream_t s) {
  switch (l.M) {
    case 128: return launch_fast_r<NEAR, 4>(p, l, s);
    case 256: return launch_fast_r<NEAR, 8>(p, l, s);
    case 512: return launch_fast_r<NEAR, 16>(p, l, s);
    default: return launch_fast_r<NEAR, 32>(p, l, s);
  }
}

}  // namespace
}  // namespace sr
