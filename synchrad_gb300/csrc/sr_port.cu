// The reference kernels' arithmetic in FP64 or FP32, every track of the batch in
// sequence.
//
// This translation unit is compiled with --fmad=false so that, like the
// reference built without contraction, the products and sums of phases and
// amplitudes are rounded on their own (the phase and 1 - n.beta cancel: their
// rounding shows at 1e-11 of the spectrum); the FP64 results then differ from
// the CPU oracle only through the last bits of sin/cos and of the sums.  These kernels are the SR_PREC_DOUBLE path (the "plain FP64"
// baseline), and SR_PREC_FLOAT / SR_PREC_FLOAT_NATIVE (dtype='float').
#include <algorithm>
#include <cmath>

#include "sr_common.cuh"
#include "sr_internal.h"

namespace sr {
namespace {

template <typename T, bool NATIVE>
struct Math;
template <bool NATIVE>
struct Math<double, NATIVE> {
  static __device__ __forceinline__ double rsq(double v) { return 1.0 / sqrt(v); }
  static __device__ __forceinline__ double sqr(double v) { return sqrt(v); }
  static __device__ __forceinline__ double sn(double v) { return sin(v); }
  static __device__ __forceinline__ double cs(double v) { return cos(v); }
};
template <>
struct Math<float, false> {
  static __device__ __forceinline__ float rsq(float v) { return 1.0f / sqrtf(v); }
  static __device__ __forceinline__ float sqr(float v) { return sqrtf(v); }
  static __device__ __forceinline__ float sn(float v) { return sinf(v); }
  static __device__ __forceinline__ float cs(float v) { return cosf(v); }
};
template <>
struct Math<float, true> {  // OpenCL native_* counterparts
  static __device__ __forceinline__ float rsq(float v) { return rsqrtf(v); }
  static __device__ __forceinline__ float sqr(float v) { return sqrtf(v); }
  static __device__ __forceinline__ float sn(float v) { return __sinf(v); }
  static __device__ __forceinline__ float cs(float v) { return __cosf(v); }
};

struct TrackView {
  uint64_t base;
  uint32_t n_steps, it_start, it_end;
  double wp;
  const uint32_t *snaps;
};

__device__ __forceinline__ TrackView track_view(const PortParams &p, uint32_t t) {
  TrackView v;
  if (p.offsets == nullptr) {
    v.base = 0;
    v.n_steps = p.n_steps1;
    v.it_start = p.it_start1;
    v.it_end = p.it_end1;
    v.wp = p.wp1;
    v.snaps = p.snap_its;
  } else {
    v.base = (uint64_t)p.offsets[t];
    v.n_steps = (uint32_t)(p.offsets[t + 1] - p.offsets[t]);
    v.it_start = p.it_start[t];
    v.it_end = p.it_end[t];
    v.wp = p.weight[t];
    v.snaps = p.snap_its + (size_t)t * p.snap_stride;
  }
  return v;
}

// sin and cos of an FP32 phase: the phase in revolutions as a double-float
// (1/(2 pi) to 48 bits, whole turns dropped exactly), then the library's
// sin(pi x), cos(pi x).  Good to an ulp or two like sinf, without its slow
// reduction of large arguments; beyond 2^21 rad the 48 bits run out and sincosf
// takes over.
__device__ __forceinline__ void sincos_of(float v, float &sn, float &cs) {
  if (fabsf(v) < 2097152.f) {
    constexpr float ih = 0.15915494f, il = 6.4206382e-9f;  // 1/(2 pi)
    const float h = v * ih;
    const float l = __fmaf_rn(v, il, __fmaf_rn(v, ih, -h));
    const float f = (h - rintf(h)) + l;
    sincospif(f + f, &sn, &cs);
  } else {
    sincosf(v, &sn, &cs);
  }
}

// Which values a (direction, step) leaves in shared memory.
//   V_TAU: time - n.x (far), time + r (near): the phase is omega times it
//   V_RC, V_RS (FP64, several points a lane): exp(i d_omega tau); FP32 near: 1/r
//   V_A0..: far: the step's amplitude, near: (beta - n)/r and n/r^2
enum { V_TAU = 0, V_RC = 1, V_RS = 2 };
template <bool F64, bool NEAR, int K>
constexpr int first_amplitude() {
  return F64 ? (K > 1 ? 3 : 1) : (NEAR ? 2 : 1);
}
template <bool F64, bool NEAR, int K>
constexpr int shared_values() {
  return first_amplitude<F64, NEAR, K>() + (NEAR ? 6 : 3);
}

// One warp's 32 / L directions, K consecutive omega points per lane.
//
// The reference's kernels compute everything per point; of the ~160 FP64
// operations of a point and step only the phase, its sine and cosine and the
// sums depend on omega (FP64 runs at 1/64 of the FP32 rate here and is the
// bound).  So the lanes of a warp first compute, one step each, what depends on
// (direction, step) alone, with the reference's operations in its order, into
// shared memory; then each lane sums its K points over the 32 steps.
//
// FP64 on an even omega axis: the reference evaluates sin and cos at the
// rounded product p = fl(omega_m tau).  With omega_m = omega_0 + m d_omega +
// eps_m (eps_m: the axis' own rounding) and e_m = omega_m tau - p (exact, by
// FMA), exp(i p) = exp(i omega_0 tau) R^m exp(i delta_m), R = exp(i d_omega
// tau), delta_m = eps_m tau - e_m: a rotation per point and a first- or
// second-order factor for delta (~1e-16 of the phase) instead of a sine and a
// cosine.  Steps where |delta| could pass 1e-5, and uneven axes, call sincos
// per point.
//
// The |dphase| < pi rule is decided from |omega| |dtau| in FP32 with a guard
// band; inside it (and where the phases are so large that their rounding
// matters) the reference's FP64 expression decides.
template <typename T, int COMP, bool NEAR, bool NATIVE, int K>
__global__ void __launch_bounds__(128) port_kernel(PortParams p, int L) {
  using M = Math<T, NATIVE>;
  constexpr bool F64 = sizeof(T) == 8;
  constexpr bool ROT = F64 && K > 1;  // phasors by rotation from the first point's
  constexpr int V_A0 = first_amplitude<F64, NEAR, K>(), V_MAX = shared_values<F64, NEAR, K>();
  // total needs the two transverse components only (n.A is rounding noise,
  // ~1e-11 of A: 1e-22 of |A|^2)
  constexpr int NC = (!NEAR && COMP == 0 && F64) ? 2 : 3;
  extern __shared__ __align__(16) unsigned char port_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dpw = 32 / L, dsub = lane / L, ll = lane % L;
  T *val = (T *)port_smem + (size_t)warp * dpw * (V_MAX * 32 + 1);  // [dpw][V_MAX][32], padded
  const uint32_t nO = p.n_omega, n1 = p.n_1, n_dirs = p.n_1 * p.n_phi;
  const uint64_t nTotal = (uint64_t)nO * n_dirs;
  const uint32_t n_tiles = (nO + (uint32_t)(L * K) - 1) / (uint32_t)(L * K);
  const uint64_t task = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  const uint64_t n_groups = ((uint64_t)n_dirs + dpw - 1) / dpw;
  if (task >= n_groups * n_tiles) return;  // whole warps
  const uint32_t tile = (uint32_t)(task % n_tiles);
  const uint32_t dir0 = (uint32_t)(task / n_tiles) * dpw;
  const T *om = (const T *)p.omega, *ax1 = (const T *)p.axis1, *ax2 = (const T *)p.axis2,
          *sP = (const T *)p.sin_phi, *cP = (const T *)p.cos_phi;
  const T *X = (const T *)p.x, *Y = (const T *)p.y, *Z = (const T *)p.z;
  const T *UX = (const T *)p.ux, *UY = (const T *)p.uy, *UZ = (const T *)p.uz;
  const T dt = (T)p.dt;
  const T dtInv = (T)1. / dt;
  const T Ls = (T)p.L;
  const uint32_t n_tr = p.offsets ? p.n_tracks : 1u;

  // the lane's points
  const uint32_t dir = min(dir0 + dsub, n_dirs - 1);
  const uint32_t j0 = tile * (uint32_t)(L * K) + ll * K;
  const int nv = dir0 + dsub < n_dirs ? max(0, min(K, (int)nO - (int)j0)) : 0;
  T w[K], eps[K];
  float wmax = 0.f, epsmax = 0.f;
  const T dw = nO > 1 ? (om[nO - 1] - om[0]) / (T)(nO - 1) : (T)0.;
#pragma unroll
  for (int m = 0; m < K; ++m) {
    w[m] = nv > 0 ? om[j0 + min(m, nv - 1)] : (T)0.;
    // a NaN frequency fails the rule below like the reference's comparison
    wmax = w[m] == w[m] ? fmaxf(wmax, fabsf((float)w[m])) : INFINITY;
    eps[m] = (T)0.;
    if (F64 && m < nv) {  // (omega_m - omega_0) - m d_omega, the difference exact as a pair
      const T d = w[m] - w[0], v = d - w[m];
      const T err = (w[m] - (d - v)) - (w[0] + v);
      eps[m] = fma((T)(-m), dw, d) + err;
      epsmax = fmaxf(epsmax, fabsf((float)eps[m]));
    }
  }
  // |delta| <= dcoef |tau|: a NaN or large eps sends every step to sincos
  const float dcoef = epsmax * 1.0001f + wmax * 1.2e-16f;

  for (uint32_t tr = 0; tr < n_tr; ++tr) {
    const TrackView tv = track_view(p, tr);
    if (tv.it_end == 0 || tv.n_steps == 0) continue;  // rejected on the host
    const T wp = (T)tv.wp;
    const T wpdt2 = wp * dt * dt;
    const T wpdt = M::sqr(wp) * dt;
    T re[NC][K], im[NC][K];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int m = 0; m < K; ++m) re[c][m] = im[c][m] = (T)0.;
    SnapState snap;
    snap.init(tv.it_start, tv.it_end, tv.snaps, p.n_snaps);
    const uint32_t n_body = min(tv.it_end - 1u, tv.n_steps - 1u);

    auto flush = [&](uint32_t k) {
      const uint64_t o0 = (uint64_t)j0 + (uint64_t)nO * dir + nTotal * k;
      T *const *out = (T *const *)p.out;
      const T *ffa = (const T *)p.form_factor;
#pragma unroll
      for (int m = 0; m < K; ++m) {
        if (m >= nv) break;
        const uint64_t o = o0 + m;
        if (COMP == 0) {
          T a = re[0][m] * re[0][m] + re[1][m] * re[1][m];
          T b = im[0][m] * im[0][m] + im[1][m] * im[1][m];
          if constexpr (NC == 3) {
            a = a + re[2][m] * re[2][m];
            b = b + im[2][m] * im[2][m];
          }
          out[0][o] += wpdt2 * (a + b);
        } else if (COMP == 1 || COMP == 3) {
#pragma unroll
          for (int c = 0; c < NC; ++c)
            out[c][o] += wpdt2 * (re[c][m] * re[c][m] + im[c][m] * im[c][m]);
        } else {
          // FormFactor: cartesian_complex of the far field only, there a factor
          // of every term (synchrad/kernel_farfield.cl:364-370)
          const T f = (COMP == 2 && !NEAR) ? ffa[j0 + m] : (T)1.0;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            out[2 * c][o] += wpdt * (re[c][m] * f);
            out[2 * c + 1][o] += wpdt * (im[c][m] * f);
          }
        }
      }
    };

    // the last tau of the chunk before (0: the first step's phase is compared
    // with zero, synchrad/kernel_farfield.cl:49)
    T tau_before = (T)0.;
    const T *x = X + tv.base, *y = Y + tv.base, *z = Z + tv.base;
    const T *ux = UX + tv.base, *uy = UY + tv.base, *uz = UZ + tv.base;
    // nothing after the last snapshot write is seen
    for (uint32_t s0 = 0; s0 < n_body && snap.fire_it != SnapState::NEVER; s0 += 32) {
      const uint32_t cnt = min(32u, n_body - s0);
      __syncwarp();
      {  // ---- what depends on (direction, step): lane l -> step s0 + l ----
        const uint32_t it = s0 + min((uint32_t)lane, cnt - 1);
        const T time = (T)(tv.it_start + it) * dt;
        const T xx = x[it], yy = y[it], zz = z[it];
        T g = M::rsq((T)1. + (ux[it] * ux[it] + uy[it] * uy[it] + uz[it] * uz[it]));
        const T b0 = ux[it] * g, b1 = uy[it] * g, b2 = uz[it] * g;
        T a0, a1, a2, m0, m1, m2;
        if constexpr (!NEAR) {
          g = M::rsq((T)1. + (ux[it + 1] * ux[it + 1] + uy[it + 1] * uy[it + 1] +
                              uz[it + 1] * uz[it + 1]));
          const T bn0 = ux[it + 1] * g, bn1 = uy[it + 1] * g, bn2 = uz[it + 1] * g;
          a0 = (bn0 - b0) * dtInv; a1 = (bn1 - b1) * dtInv; a2 = (bn2 - b2) * dtInv;
          m0 = (T)0.5 * (bn0 + b0); m1 = (T)0.5 * (bn1 + b1); m2 = (T)0.5 * (bn2 + b2);
        }
#pragma unroll 1
        for (int dd = 0; dd < dpw; ++dd) {
          const uint32_t dk = min(dir0 + dd, n_dirs - 1);
          const uint32_t i1 = dk % n1, iP = dk / n1;
          T *v = val + (size_t)dd * (V_MAX * 32 + 1) + lane;
          T tau;
          if constexpr (!NEAR) {
            const T sT = ax1[i1], cT = ax2[i1];
            const T e0 = sT * cP[iP], e1 = sT * sP[iP], e2 = cT;
            tau = time - (xx * e0 + yy * e1 + zz * e2);
            T c1 = a0 * e0 + a1 * e1 + a2 * e2;
            T c2 = (T)1. - (m0 * e0 + m1 * e1 + m2 * e2);
            c2 = (T)1. / c2;
            c1 = c1 * c2 * c2;
            T A0 = c1 * (e0 - m0) - c2 * a0;
            T A1 = c1 * (e1 - m1) - c2 * a1;
            T A2 = c1 * (e2 - m2) - c2 * a2;
            if (COMP == 3 || COMP == 4 || NC == 2) {
              const T t0 = cT * cP[iP], t1 = cT * sP[iP], t2 = -sT;
              const T p0 = -sP[iP], p1 = cP[iP], p2 = (T)0.0;
              const T r = e0 * A0 + e1 * A1 + e2 * A2;
              const T th = t0 * A0 + t1 * A1 + t2 * A2;
              const T ph = p0 * A0 + p1 * A1 + p2 * A2;
              if constexpr (NC == 2) {
                A0 = th; A1 = ph;
              } else {
                A0 = r; A1 = th; A2 = ph;
              }
            }
            v[(V_A0 + 0) * 32] = A0;
            v[(V_A0 + 1) * 32] = A1;
            if constexpr (NC == 3) v[(V_A0 + 2) * 32] = A2;
          } else {
            const T R = ax1[i1];
            const T P0 = R * cP[iP], P1 = R * sP[iP], P2 = Ls;
            const T d0 = P0 - xx, d1 = P1 - yy, d2 = P2 - zz;
            const T r = M::sqr(d0 * d0 + d1 * d1 + d2 * d2);
            tau = time + r;
            const T rInv = (T)1. / r;
            const T e0 = rInv * d0, e1 = rInv * d1, e2 = rInv * d2;
            const T rr = rInv * rInv;
            if constexpr (F64) {
              v[(V_A0 + 0) * 32] = rInv * (b0 - e0);
              v[(V_A0 + 1) * 32] = rInv * (b1 - e1);
              v[(V_A0 + 2) * 32] = rInv * (b2 - e2);
            } else {  // the FP32 kernel's order: (omega / r) (beta - n)
              v[(V_A0 + 0) * 32] = b0 - e0;
              v[(V_A0 + 1) * 32] = b1 - e1;
              v[(V_A0 + 2) * 32] = b2 - e2;
              v[V_RC * 32] = rInv;
            }
            v[(V_A0 + 3) * 32] = rr * e0;
            v[(V_A0 + 4) * 32] = rr * e1;
            v[(V_A0 + 5) * 32] = rr * e2;
          }
          v[V_TAU * 32] = tau;
          if constexpr (ROT) {
            const T pr = dw * tau;
            const T e = fma(dw, tau, -pr);
            T sn, cs;
            sincos(pr, &sn, &cs);
            v[V_RC * 32] = fma(-e, sn, cs);
            v[V_RS * 32] = fma(e, cs, sn);
          }
        }
      }
      __syncwarp();
      // ---- the lane's points over the chunk's steps ----
      const T *v = val + (size_t)dsub * (V_MAX * 32 + 1);
#pragma unroll 1
      for (uint32_t i = 0; i < cnt; ++i) {
        const uint32_t s = s0 + i;
        const T tau = v[V_TAU * 32 + i];
        const T tprev = i ? v[V_TAU * 32 + i - 1] : tau_before;
        // one bit per included point
        uint32_t inc = 0u;
        const float adt = fabsf((float)(tau - tprev)), tf = fabsf((float)tau);
        if (F64 && wmax * adt < 3.14158f && wmax * tf < 1e10f) {
          inc = (1u << K) - 1u;
        } else {
#pragma unroll
          for (int m = 0; m < K; ++m) {
            const float ph = fabsf((float)w[m]) * adt;
            bool in;
            if (F64 && ph < 3.14158f && wmax * tf < 1e10f) in = true;
            else if (F64 && ph > 3.1416f && wmax * tf < 1e10f) in = false;
            else in = fabs(w[m] * tau - w[m] * tprev) < (T)M_PI;
            inc |= (uint32_t)in << m;
          }
        }
        if (__any_sync(0xffffffffu, inc != 0u)) {
          const T A0 = v[(V_A0 + 0) * 32 + i], A1 = v[(V_A0 + 1) * 32 + i];
          T A2 = (T)0., B0 = (T)0., B1 = (T)0., B2 = (T)0.;
          if constexpr (NC == 3) A2 = v[(V_A0 + 2) * 32 + i];
          if constexpr (NEAR) {
            B0 = v[(V_A0 + 3) * 32 + i];
            B1 = v[(V_A0 + 4) * 32 + i];
            B2 = v[(V_A0 + 5) * 32 + i];
          }
          auto add = [&](int m, T cs, T sn) {
            if constexpr (NEAR) {
              if constexpr (F64) {
                const T c0 = w[m] * A0, c1 = w[m] * A1, c2 = w[m] * A2;
                re[0][m] = fma(-c0, sn, fma(B0, cs, re[0][m]));
                im[0][m] = fma(c0, cs, fma(B0, sn, im[0][m]));
                re[1][m] = fma(-c1, sn, fma(B1, cs, re[1][m]));
                im[1][m] = fma(c1, cs, fma(B1, sn, im[1][m]));
                re[2][m] = fma(-c2, sn, fma(B2, cs, re[2][m]));
                im[2][m] = fma(c2, cs, fma(B2, sn, im[2][m]));
              } else {
                const T wr = w[m] * v[V_RC * 32 + i];
                const T c0 = wr * A0, c1 = wr * A1, c2 = wr * A2;
                re[0][m] += -c0 * sn + B0 * cs; im[0][m] += c0 * cs + B0 * sn;
                re[1][m] += -c1 * sn + B1 * cs; im[1][m] += c1 * cs + B1 * sn;
                re[2][m] += -c2 * sn + B2 * cs; im[2][m] += c2 * cs + B2 * sn;
              }
            } else if constexpr (F64) {
              re[0][m] = fma(A0, cs, re[0][m]); im[0][m] = fma(A0, sn, im[0][m]);
              re[1][m] = fma(A1, cs, re[1][m]); im[1][m] = fma(A1, sn, im[1][m]);
              if constexpr (NC == 3) {
                re[2][m] = fma(A2, cs, re[2][m]); im[2][m] = fma(A2, sn, im[2][m]);
              }
            } else {
              re[0][m] += A0 * cs; im[0][m] += A0 * sn;
              re[1][m] += A1 * cs; im[1][m] += A1 * sn;
              re[2][m] += A2 * cs; im[2][m] += A2 * sn;
            }
          };
          if constexpr (ROT) {
            const float dmax = dcoef * tf;  // bound of |delta|
            if (__all_sync(0xffffffffu, dmax < 1e-5f)) {
              // exp(i omega_0 tau) of the exact product, then rotations
              const T pr = w[0] * tau;
              const T e = fma(w[0], tau, -pr);
              T s1, c1;
              sincos(pr, &s1, &c1);
              T zc = fma(-e, s1, c1), zs = fma(e, c1, s1);
              const T Rc = v[V_RC * 32 + i], Rs = v[V_RS * 32 + i];
              const bool small = __all_sync(0xffffffffu, dmax < 1e-8f);
#pragma unroll
              for (int m = 0; m < K; ++m) {
                const T pm = w[m] * tau;
                const T d = fma(eps[m], tau, -fma(w[m], tau, -pm));
                T cs, sn;
                if (small) {
                  cs = fma(-d, zs, zc);
                  sn = fma(d, zc, zs);
                } else {  // 1 + i d - d^2/2
                  const T h = (T)0.5 * d;
                  cs = fma(-d, fma(h, zc, zs), zc);
                  sn = fma(d, fma(-h, zs, zc), zs);
                }
                if ((inc >> m) & 1u) add(m, cs, sn);
                if (m + 1 < K) {
                  const T u = zc * Rc, q = zc * Rs;
                  zc = fma(-zs, Rs, u);
                  zs = fma(zs, Rc, q);
                }
              }
            } else {
#pragma unroll
              for (int m = 0; m < K; ++m) {
                T sn, cs;
                sincos(w[m] * tau, &sn, &cs);
                if ((inc >> m) & 1u) add(m, cs, sn);
              }
            }
          } else {
#pragma unroll
            for (int m = 0; m < K; ++m) {
              const T phase = w[m] * tau;
              T sn, cs;
              if constexpr (NATIVE) {
                sn = M::sn(phase);
                cs = M::cs(phase);
              } else if constexpr (F64) {
                sincos(phase, &sn, &cs);
              } else {
                sincos_of(phase, sn, cs);
              }
              if ((inc >> m) & 1u) add(m, cs, sn);
            }
          }
        }
        if ((int64_t)s == snap.fire_it) {  // uniform over the warp
          flush(snap.k);
          snap.advance(tv.it_start, tv.it_end, tv.snaps, p.n_snaps);
        }
      }
      tau_before = v[V_TAU * 32 + cnt - 1];
    }
    // snapshot writes due after the last body step (the reference keeps
    // iterating up to itEnd - 2 without changing A)
    while (snap.fire_it != SnapState::NEVER) {
      flush(snap.k);
      snap.advance(tv.it_start, tv.it_end, tv.snaps, p.n_snaps);
    }
  }
}

template <typename T, int COMP, bool NEAR, bool NATIVE, int K>
int launch_shape(const PortParams &p, int L, cudaStream_t s) {
  const int dpw = 32 / L;
  const uint64_t tiles = ((uint64_t)p.n_omega + (uint64_t)L * K - 1) / ((uint64_t)L * K);
  const uint64_t tasks = (((uint64_t)p.n_1 * p.n_phi + dpw - 1) / dpw) * tiles;
  // few tasks: one warp per CTA, so that they spread over the SMs
  const int w = tasks >= 16ull * device_sm_count() && dpw <= 4 ? 4 : 1;
  const size_t smem =
      (size_t)w * dpw * (shared_values<sizeof(T) == 8, NEAR, K>() * 32 + 1) * sizeof(T);
  const uint64_t blocks = (tasks + w - 1) / w;
  if (blocks > 0x7fffffffull)
    return fail(SR_ERR_INVALID, "grid needs %llu blocks", (unsigned long long)blocks);
  if (smem > 48u << 10) {
    const cudaError_t e =
        allow_smem((const void *)port_kernel<T, COMP, NEAR, NATIVE, K>, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "port smem attribute");
  }
  port_kernel<T, COMP, NEAR, NATIVE, K><<<(unsigned)blocks, w * 32, smem, s>>>(p, L);
  return cuda_fail(cudaGetLastError(), "port kernel launch");
}

// Points per lane K and lanes per direction L by the cost of a warp's step:
// K points of `c` operations each, `seed` for what the lane shares (FP64: a
// sine and cosine, ~45 operations against 13 to 20 per point) and 4 per
// direction for the shared values, times the cycles an operation takes on the
// fullest SM: 16 per resident warp in FP64, at least the ~64 of a dependent
// chain (FP32: 1/4 per warp, at least 6).  Measured, 64 omega points on 480
// screen points: K = 2 with four warps per SM 23.8 ms, K = 4 with two 35.6 ms.
// FP64 at one point per lane takes down to one lane per direction: 1 omega point on
// 16384 directions, 1000 steps, far 14.2 ms with 8 lanes (one at work), 3.3 now;
// near 16.0, 3.9 (a thread per point, without shared values: 10.4, 8.8).
template <typename T, int COMP, bool NEAR, bool NATIVE>
int launch_comp(const PortParams &p, cudaStream_t s) {
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int KM = (F64 && !NEAR && COMP == 0) ? 8 : 4;
  const double c = F64 ? (NEAR ? 20 : 13) : 45, seed = F64 ? 45 : 25;
  const uint64_t dirs = (uint64_t)p.n_1 * p.n_phi;
  const uint64_t n_sm = (uint64_t)device_sm_count();
  int bK = 1, bL = 32;
  double best = 1e300;
  for (int K = KM; K >= 1; K /= 2)
    for (int L = 32; L >= (F64 && K == 1 ? 1 : 8); L /= 2) {
      const int dpw = 32 / L;
      const uint64_t tiles = ((uint64_t)p.n_omega + (uint64_t)L * K - 1) / ((uint64_t)L * K);
      const uint64_t tasks = ((dirs + dpw - 1) / dpw) * tiles;
      const double warps = (double)((tasks + n_sm - 1) / n_sm);
      // FP64 warps an SM holds, by their shared values
      const double held = std::min(warps, 232448.0 / (dpw * (NEAR ? 9 : 6) * 32.0 * 8.0));
      const double cycles =
          F64 ? warps * std::max(16.0, 64.0 / held) : std::max(0.25 * warps, 6.0);
      const double shared = F64 && K == 1 ? 3.0 : 4.0;
      const double cost = cycles * (K * c + seed + shared * dpw);
      if (cost < best) {
        best = cost;
        bK = K;
        bL = L;
      }
    }
  switch (bK) {
    case 8:
      if constexpr (KM == 8) return launch_shape<T, COMP, NEAR, NATIVE, 8>(p, bL, s);
      return SR_OK;
    case 4: return launch_shape<T, COMP, NEAR, NATIVE, 4>(p, bL, s);
    case 2: return launch_shape<T, COMP, NEAR, NATIVE, 2>(p, bL, s);
    default: return launch_shape<T, COMP, NEAR, NATIVE, 1>(p, bL, s);
  }
}

template <typename T, bool NATIVE>
int launch_typed(const PortParams &p, int mode, int comp, cudaStream_t s) {
  if (mode == 0) {
    switch (comp) {
      case 0: return launch_comp<T, 0, false, NATIVE>(p, s);
      case 1: return launch_comp<T, 1, false, NATIVE>(p, s);
      case 2: return launch_comp<T, 2, false, NATIVE>(p, s);
      case 3: return launch_comp<T, 3, false, NATIVE>(p, s);
      case 4: return launch_comp<T, 4, false, NATIVE>(p, s);
      default: return fail(SR_ERR_INVALID, "unknown comp %d", comp);
    }
  }
  switch (comp) {
    case 0: return launch_comp<T, 0, true, NATIVE>(p, s);
    case 1: return launch_comp<T, 1, true, NATIVE>(p, s);
    case 2: return launch_comp<T, 2, true, NATIVE>(p, s);
    default: return fail(SR_ERR_UNSUPPORTED, "near field has no comp %d", comp);
  }
}

}  // namespace

int launch_port(const PortParams &p, int mode, int comp, int dtype, bool native,
                cudaStream_t stream) {
  if ((uint64_t)p.n_omega * p.n_1 * p.n_phi == 0) return SR_OK;
  void *tok = nullptr;
  timing_record(stream, true, &tok);
  int rc;
  if (dtype == SR_DTYPE_F64)
    rc = launch_typed<double, false>(p, mode, comp, stream);
  else if (native)
    rc = launch_typed<float, true>(p, mode, comp, stream);
  else
    rc = launch_typed<float, false>(p, mode, comp, stream);
  timing_record(stream, false, &tok);
  return rc;
}

}  // namespace sr
