// Adjoint of the mixed-precision far field (every comp, one snapshot).
//
// Forward (sr_far_mixed.cu):  S(p) = sum_t w_t dt^2 |A_t(p)|^2,
//   A_t(p) = sum_s m_s(p) amp_s(p) exp(i omega tau_s(p)),  carried on
//   theta-hat and phi-hat, amp = -(c1 (e.bbar) + c2 (e.a)) for e in {th, ph},
//   c2 = 1/(1 - n.bbar), c1 = (a.n) c2^2, tau_s = t_s - n.x_s.
// Given g(p) = dL/dS(p), with U_c = 2 g w dt^2 conj(A_c) and W_c = omega U_c:
//   dL/dw_t       = sum_p g dt^2 |A_t|^2
//   dL/damp_c,s   = E_c(d,s) = sum_omega Re(U_c z_s)
//   dL/dx_s       = sum_d n (amp_th F_th + amp_ph F_ph),  F_c = sum_omega Im(W_c z_s)
//   dL/dbbar_s, dL/da_s from amp(bbar, a), then bbar_s = (beta_s + beta_{s+1})/2,
//   a_s = (beta_{s+1} - beta_s)/dt, beta = u/gamma.
// The |dphase| < pi mask is held fixed (its decisions are the forward's).
// The comps differ only in how the loss sees A (point sensitivity, below):
//   quadratic comps (total, cartesian, spheric: outputs w dt^2 |b_k . A|^2
//   with b_k the output's unit vector on (theta-hat, phi-hat)):
//     U = w M A,  M = 2 dt^2 sum_k g_k b_k b_k^T (2 x 2, real);
//   linear comps (cartesian_complex, spheric_complex: outputs sqrt(w) dt
//   f(omega) Re/Im (b_k . A), f the FormFactor or 1):
//     U = sqrt(w) V,  V = dt f sum_k (g_k,re + i g_k,im) b_k;
// so that dL = Re(conj(U) . dA), and dL/dw_t = sum_p Re(conj(U) . A_t) / (2 w_t).
//
// Layout: E and F are sums over omega for each (direction, step), so a lane
// owns one step and walks the omega axis of a direction with the rotation
// recurrence z <- z exp(i domega tau) (reseeded from the double-float phase
// every 8 points); U and W of a block of (direction, omega) points are built
// in shared memory from the saved amplitudes and read by every lane
// (broadcast).  A CTA owns 256 consecutive steps of one track and loops over
// every direction, so each step's gradient is summed in registers and written
// once: no atomics, no cross-lane reductions, a deterministic result.
// Phases are recomputed, not stored.
//
// On even omega axes the sums over omega come from transforms instead
// (adj_fields_kernel, adj_interp_kernel below); the walk keeps uneven axes,
// fewer than 8 frequencies and snapshots a few steps apart.
#include <algorithm>
#include <cmath>

#include "sr_common.cuh"
#include "sr_internal.h"
#include "sr_fast_sum.cuh"
#include "sr_mixed_common.cuh"
#include "sr_adjoint_common.cuh"

namespace sr {
namespace {

constexpr int kAW = 8;                // warps per CTA
constexpr int kASteps = kAW * 32;     // steps per work item (one per lane)
constexpr int kAStage = 1024;         // (direction, omega) points per constants stage
constexpr int kARS = 8;               // omega points per phasor reseed
constexpr int kAG = 9;                // per-step gradient components: x (3), bbar (3), a (3)

struct AdjParams {
  FarMixedParams f;            // tracks, grid, records, status
  const double *grad_out[6];   // [P] dL/dS_k per output of the comp, device layout
  int linear;                  // comp is linear in A (the *_complex comps)
  const float4 *save_A;        // [n_tracks][P] (A_th re, im, A_ph re, im)
  float4 *gcst;                // [P] point sensitivity in FP32: M (xx, xy, yy, 0) or V
  float4 *wtab;                // [nO] (omega/2pi hi, lo, omega, |omega|) in FP32
  float4 *dirtab;              // [n_dirs][4] direction constants
  AdjGlobals *glob;
  int64_t *item_off;           // [n_tracks + 1] first work item of each track
  double *gstep;               // [n_split][total_steps][kAG] per-step gradients (bbar, a form)
  uint32_t n_split;            // runs of directions summed apart
  float4 *bandtab;             // [n_bands] centre frequency / 2 pi
  float2 *fields;              // transforms' cells of a batch of tracks (see below)
  uint32_t t_lo, t_hi;         // the batch
  unsigned int *many_cut;      // whether the phase limit cuts many steps
  double *grad[6];             // x, y, z, ux, uy, uz  [total_steps]
  double *grad_w;              // [n_tracks]
  double *wpart;               // [n_tracks][w_chunks] partial weight gradients
  uint32_t w_chunks;
};

// Point sensitivity of the loss to (A_theta, A_phi) for output gradients g_k
// at point gi: M = (xx, xy, yy) of the quadratic comps (2 dt^2 included) or V
// = (th re, th im, ph re, ph im) of the linear ones (dt and FormFactor
// included), in FP64.
__device__ __forceinline__ void point_sens(const AdjParams &a, uint32_t ksnap, uint64_t gi,
                                           double out[4]) {
  const FarMixedParams &p = a.f;
  const uint32_t nO = p.n_omega, nT = p.n_theta;
  const uint64_t gk = (uint64_t)ksnap * nO * nT * p.n_phi + gi;  // snapshot ksnap's slot
  const uint64_t d = gi / nO;
  const uint32_t m = (uint32_t)(gi - d * nO);
  const uint32_t iT = (uint32_t)(d % nT), iP = (uint32_t)(d / nT);
  const double sT = p.sin_theta[iT], cT = p.cos_theta[iT];
  const double sP = p.sin_phi[iP], cP = p.cos_phi[iP];
  // output unit vectors x, y, z on (theta-hat, phi-hat)
  const double bt[3] = {cT * cP, cT * sP, -sT}, bp[3] = {-sP, cP, 0.0};
  const double s2 = 2.0 * p.dt * p.dt;
  auto g = [&](int k) { return a.grad_out[k][gk]; };
  out[0] = out[1] = out[2] = out[3] = 0.0;
  switch (p.comp) {
    case SR_COMP_TOTAL:
      out[0] = out[2] = s2 * g(0);
      break;
    case SR_COMP_CARTESIAN:
      for (int k = 0; k < 3; ++k) {
        const double gk = s2 * g(k);
        out[0] += gk * bt[k] * bt[k];
        out[1] += gk * bt[k] * bp[k];
        out[2] += gk * bp[k] * bp[k];
      }
      break;
    case SR_COMP_SPHERIC:  // outputs r (identically 0), theta, phi
      out[0] = s2 * g(1);
      out[2] = s2 * g(2);
      break;
    case SR_COMP_CARTESIAN_COMPLEX: {
      const double f = p.dt * p.form_factor[m];
      for (int k = 0; k < 3; ++k) {
        const double gr = f * g(2 * k), gim = f * g(2 * k + 1);
        out[0] += gr * bt[k];
        out[1] += gim * bt[k];
        out[2] += gr * bp[k];
        out[3] += gim * bp[k];
      }
      break;
    }
    default:  // SR_COMP_SPHERIC_COMPLEX: rre, rim (identically 0), theta, phi re/im
      out[0] = p.dt * g(2);
      out[1] = p.dt * g(3);
      out[2] = p.dt * g(4);
      out[3] = p.dt * g(5);
      break;
  }
}

// Point sensitivities in FP32, and the direction table:
//   [0] (1 - cos theta hi, lo, n_x hi, lo)   [1] (n_y hi, lo, 1 - cos theta, n_x)
//   [2] (n_y, n_z, theta-hat x, y)           [3] (theta-hat z, phi-hat x, y, 0)
__global__ void adj_prep_kernel(AdjParams a) {
  const FarMixedParams &p = a.f;
  const uint32_t nT = p.n_theta;
  const uint64_t n_dirs = (uint64_t)nT * p.n_phi;
  const uint64_t P = n_dirs * p.n_omega;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P * p.n_snaps;
       i += stride) {
    double v[4];
    point_sens(a, (uint32_t)(i / P), i % P, v);
    a.gcst[i] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  }
  for (uint64_t d = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; d < n_dirs; d += stride) {
    const uint32_t iT = (uint32_t)(d % nT), iP = (uint32_t)(d / nT);
    const double sT = p.sin_theta[iT], cT = p.cos_theta[iT];
    const double sPh = p.sin_phi[iP], cPh = p.cos_phi[iP];
    const double n0 = sT * cPh, n1 = sT * sPh;
    const df c = df_from_double(1.0 - cT), sx = df_from_double(n0), sy = df_from_double(n1);
    float4 *o = a.dirtab + 4 * d;
    o[0] = make_float4(c.hi, c.lo, sx.hi, sx.lo);
    o[1] = make_float4(sy.hi, sy.lo, (float)(1.0 - cT), (float)n0);
    o[2] = make_float4((float)n1, (float)cT, (float)(cT * cPh), (float)(cT * sPh));
    o[3] = make_float4((float)(-sT), (float)(-sPh), (float)cPh, 0.f);
  }
  if (p.fast.M != 0u) {
    // behind it, per theta: (1 - cos hi, lo, sin hi, lo) (1 - cos, sin, cos, 0);
    // per omega band: its centre frequency / 2 pi as a double-float
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nT; i += stride) {
      const double sT = p.sin_theta[i], cT = p.cos_theta[i];
      const df c = df_from_double(1.0 - cT), s = df_from_double(sT);
      float4 *o = a.dirtab + 4 * n_dirs + 2 * i;
      o[0] = make_float4(c.hi, c.lo, s.hi, s.lo);
      o[1] = make_float4((float)(1.0 - cT), (float)sT, (float)cT, 0.f);
    }
    const double w0 = p.omega[0];
    const double dw = (p.omega[p.n_omega - 1] - w0) / (double)(p.n_omega - 1);
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < p.fast.n_bands;
         b += stride) {
      const uint32_t j0 = (uint32_t)b * p.fast.nb, n = min(p.fast.nb, p.n_omega - j0);
      const df c = df_from_double((w0 + (double)(j0 + n / 2) * dw) * 0.15915494309189533577);
      a.bandtab[b] = make_float4(c.hi, c.lo, 0.f, 0.f);
    }
  }
}


// dL/dw_t = sum_p Re(conj(U) . A_t) / (2 w_t) in two fixed-order stages:
// block (t, b) sums chunk b of track t's points into wpart[t][b] (FP64, from
// the FP64 point sensitivities), then one thread per track adds its chunks.
__global__ void adj_weight_partial_far_kernel(AdjParams a, uint64_t P, uint32_t n_chunks,
                                              double *wpart) {
  const uint32_t t = blockIdx.x / n_chunks, b = blockIdx.x % n_chunks;
  const uint64_t chunk = (P + n_chunks - 1) / n_chunks;
  const uint64_t g0 = (uint64_t)b * chunk, g1 = min(P, g0 + chunk);
  double acc = 0.0;
  for (uint64_t g = g0 + threadIdx.x; g < g1; g += blockDim.x) {
    for (uint32_t k = 0; k < a.f.n_snaps; ++k) {  // a snapshot that never fired has A = 0
      double v[4];
      point_sens(a, k, g, v);
      const float4 A = a.save_A[((uint64_t)t * a.f.n_snaps + k) * P + g];
      const double ar = A.x, ai = A.y, br = A.z, bi = A.w;
      if (a.linear)  // Re(conj(V) . A)
        acc += v[0] * ar + v[1] * ai + v[2] * br + v[3] * bi;
      else           // A^H M A
        acc += v[0] * (ar * ar + ai * ai) + 2.0 * v[1] * (ar * br + ai * bi) +
               v[2] * (br * br + bi * bi);
    }
  }
  __shared__ double red[kWeightThreads];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) wpart[blockIdx.x] = red[0];
}

// quadratic comps: dL/dw = (A^H M A) / 2 (M holds 2 dt^2); linear comps:
// dL/dw = Re(conj(V) . A) / (2 sqrt(w)).

// Per-step gradients: map dL/dbbar and dL/da of steps s-1 and s to dL/dbeta_s
// and dL/du_s.
template <typename TT>
__global__ void adj_final_kernel(AdjParams a) {
  const FarMixedParams &p = a.f;
  const TT *UX = (const TT *)p.ux, *UY = (const TT *)p.uy, *UZ = (const TT *)p.uz;
  const double dtInv = 1.0 / p.dt;
  adj_weight_final(p, a.wpart, a.w_chunks, a.linear, a.grad_w);
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < p.total_steps;
       g += (int64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = p.n_tracks;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (p.offsets[mid] <= g) lo = mid; else hi = mid;
    }
    const uint32_t t = lo;
    const int64_t s = g - p.offsets[t];
    const int64_t n_body = (int64_t)track_body(p, t);
    double cur[kAG] = {0}, prev[kAG] = {0};
    for (uint32_t k = 0; k < a.n_split; ++k) {
      const double *gs = a.gstep + (int64_t)k * p.total_steps * kAG;
      if (s < n_body)
        for (int c = 0; c < kAG; ++c) cur[c] += gs[g * kAG + c];
      if (s >= 1 && s - 1 < n_body)
        for (int c = 3; c < kAG; ++c) prev[c] += gs[(g - 1) * kAG + c];
    }
    a.grad[0][g] = cur[0];
    a.grad[1][g] = cur[1];
    a.grad[2][g] = cur[2];
    // dL/dbeta_s = (gb_s + gb_{s-1})/2 + (ga_{s-1} - ga_s)/dt
    double gb[3];
    for (int c = 0; c < 3; ++c)
      gb[c] = 0.5 * (cur[3 + c] + prev[3 + c]) + (prev[6 + c] - cur[6 + c]) * dtInv;
    const double ux = (double)UX[g], uy = (double)UY[g], uz = (double)UZ[g];
    const double gam = sqrt(1.0 + (ux * ux + uy * uy + uz * uz));
    const double ug = (ux * gb[0] + uy * gb[1] + uz * gb[2]) / (gam * gam * gam);
    a.grad[3][g] = gb[0] / gam - ux * ug;
    a.grad[4][g] = gb[1] / gam - uy * ug;
    a.grad[5][g] = gb[2] / gam - uz * ug;
  }
}

// Shared memory of one CTA.  Constants are stored per pair of omega slots
// (m, m+1) of a direction whose omega axis is padded to a multiple of kARS
// slots (padding slots carry zero constants):
//   [0] (U_th re m, m+1, -Im U_th m, m+1)   [1] the same for U_ph
//   [2] (Re W_th m, m+1, Im W_th m, m+1)    [3] the same for W_ph
//   [4] (omega/2pi hi, lo of m, of m+1)     [5] (|omega| of m, m+1, 0, 0)
constexpr int kARecS = kRecF4;  // record stride in shared memory (80 bytes, as in HBM)

struct AdjSmem {
  float4 rec[kASteps + 1][kARecS];  // step records r0 - 1 .. r0 + 255
  float4 cst[kAStage / 2][6];
  uint64_t bar;
  uint64_t pad_;
};

__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }

// E += Re(U z), F += Im(W z) on theta-hat and phi-hat for a pair of points.
struct EF2 {
  float2 et, ep, ft, fp;
  __device__ __forceinline__ void add(const float4 *c, float2 zr, float2 zi) {
    const float4 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
    et = __ffma2_rn(lo2(c0), zr, et);
    et = __ffma2_rn(hi2(c0), zi, et);
    ep = __ffma2_rn(lo2(c1), zr, ep);
    ep = __ffma2_rn(hi2(c1), zi, ep);
    ft = __ffma2_rn(lo2(c2), zi, ft);
    ft = __ffma2_rn(hi2(c2), zr, ft);
    fp = __ffma2_rn(lo2(c3), zi, fp);
    fp = __ffma2_rn(hi2(c3), zr, fp);
  }
};

// tau = q + (1 - cos theta) z - n_x x - n_y y of one step record, double-float.
__device__ __forceinline__ df record_tau(const float4 *r, const float4 &d0, const float4 &d1) {
  const float4 r0 = r[0], r1 = r[1];
  df tau = df{r0.x, r0.y};
  tau = df_add(tau, df_mul(df{d0.x, d0.y}, df{r1.z, r1.w}));
  const df nx = df_mul(df{d0.z, d0.w}, df{r0.z, r0.w});
  const df ny = df_mul(df{d1.x, d1.y}, df{r1.x, r1.y});
  tau = df_add(tau, df{-nx.hi, -nx.lo});
  return df_add(tau, df{-ny.hi, -ny.lo});
}

template <int W>
__global__ void __launch_bounds__(W * 32, 2) adj_far_kernel(AdjParams a) {
  const FarMixedParams &p = a.f;
  if (by_transform(p)) return;  // adj_interp_kernel's
  extern __shared__ __align__(128) unsigned char smem_raw[];
  AdjSmem &sm = *reinterpret_cast<AdjSmem *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ls = (uint32_t)(warp * 32 + lane);  // this lane's step within the item
  if (threadIdx.x == 0) {
    mbar_init(&sm.bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  const AdjGlobals G = *a.glob;
  const uint32_t nO = p.n_omega, nT = p.n_theta;
  const uint32_t nOp = (nO + kARS - 1) / kARS * kARS;  // padded omega slots per direction
  const uint64_t P = (uint64_t)nO * nT * p.n_phi;
  const uint64_t Pp = (uint64_t)nOp * nT * p.n_phi;
  const int64_t n_items = a.item_off[p.n_tracks];
  const df d_dw = df{G.dw_h, G.dw_l};
  uint32_t it_no = 0;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x, ++it_no) {
    uint32_t lo = 0, hi = p.n_tracks;  // last track with item_off[t] <= item
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (a.item_off[mid] <= item) lo = mid; else hi = mid;
    }
    const uint32_t t = lo;
    const int64_t base = p.offsets[t];
    const uint32_t n_body = track_body(p, t);
    SnapSegment seg{0, 0, 0, 0};
    track_segments(p, t, (uint32_t)kASteps, (uint32_t)(item - a.item_off[t]), &seg);
    const uint32_t r0 = seg.r0, r1 = seg.r1;  // the steps enter snapshots seg.k0 .. seg.k1
    const uint32_t has_prev = r0 > 0 ? 1u : 0u;
    const uint32_t n_rec = r1 - r0 + has_prev;
    if (threadIdx.x == 0) {  // the item's records in one bulk copy
      fence_proxy_async();
      mbar_arrive_expect_tx(&sm.bar, n_rec * kRecBytes);
      bulk_g2s(sm.rec[0], p.records + (base + r0 - has_prev) * kRecF4, n_rec * kRecBytes,
               &sm.bar);
    }
    const bool ok = mbar_wait_bounded(&sm.bar, it_no & 1u, kWaitLimitNs);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        atomicExch(p.status, STATUS_WAIT_TIMEOUT);
        mbar_wait_bounded(&sm.bar, it_no & 1u, kWaitLimitNs);
      }
      __syncthreads();
      return;
    }

    const uint32_t s = r0 + ls;
    const bool valid = s < r1;
    const uint32_t si = min(has_prev + ls, n_rec - 1);  // record index of step s
    // record 0 is step 0 of the track (no previous phase) or, for lanes past
    // the end of a one-step item, the only record loaded
    const bool first = (si == 0);
    const float wt = (float)p.weight[t];
    const float swt = (float)sqrt(p.weight[t]);
    const uint32_t it_start = p.it_start[t];
    double gD[kAG];
#pragma unroll
    for (int c = 0; c < kAG; ++c) gD[c] = 0.0;

    // per (direction, step) state, kept across constants stages
    float th = 0.f, tl = 0.f, rc = 1.f, rs = 0.f, adt = 0.f;
    float2 r2c = make_float2(1.f, 1.f), r2s = make_float2(0.f, 0.f), nr2s = r2s;
    int mode = 1;  // 0: every omega included, 1: none, 2: per point
    EF2 ef;
    ef.et = ef.ep = ef.ft = ef.fp = make_float2(0.f, 0.f);

    for (uint64_t f0 = 0; f0 < Pp; f0 += kAStage) {
      const uint32_t nf = (Pp - f0 < (uint64_t)kAStage) ? (uint32_t)(Pp - f0) : (uint32_t)kAStage;
      __syncthreads();  // the previous stage's constants are no longer read
      for (uint32_t j = threadIdx.x; j < nf / 2; j += blockDim.x) {
        const uint64_t f = f0 + 2 * j;
        const uint64_t dj = f / nOp;
        const uint32_t m = (uint32_t)(f - dj * nOp);
        float4 u[2], w[2], wv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (m + e < nO) {
            const uint64_t gi = dj * nO + m + e;
            wv[e] = a.wtab[m + e];
            // U summed over the snapshots these steps enter
            u[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t k = seg.k0; k <= seg.k1; ++k) {
              const float4 C = a.gcst[(uint64_t)k * P + gi];
              if (a.linear) {
                u[e].x += swt * C.x; u[e].y += swt * C.y;
                u[e].z += swt * C.z; u[e].w += swt * C.w;
              } else {
                const float4 A = a.save_A[((uint64_t)t * p.n_snaps + k) * P + gi];
                u[e].x += wt * (C.x * A.x + C.y * A.z);
                u[e].y += wt * (C.x * A.y + C.y * A.w);
                u[e].z += wt * (C.y * A.x + C.z * A.z);
                u[e].w += wt * (C.y * A.y + C.z * A.w);
              }
            }
            w[e] = make_float4(wv[e].z * u[e].x, -wv[e].z * u[e].y, wv[e].z * u[e].z,
                               -wv[e].z * u[e].w);
          } else {
            u[e] = w[e] = wv[e] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        float4 *o = sm.cst[j];
        o[0] = make_float4(u[0].x, u[1].x, u[0].y, u[1].y);
        o[1] = make_float4(u[0].z, u[1].z, u[0].w, u[1].w);
        o[2] = make_float4(w[0].x, w[1].x, w[0].y, w[1].y);
        o[3] = make_float4(w[0].z, w[1].z, w[0].w, w[1].w);
        o[4] = make_float4(wv[0].x, wv[0].y, wv[1].x, wv[1].y);
        o[5] = make_float4(wv[0].w, wv[1].w, 0.f, 0.f);
      }
      __syncthreads();
      float gF[kAG];
#pragma unroll
      for (int c = 0; c < kAG; ++c) gF[c] = 0.f;

      uint32_t d = (uint32_t)(f0 / nOp);
      for (uint64_t fd = (uint64_t)d * nOp; fd < f0 + nf; fd += nOp, ++d) {
        const uint32_t m_lo = (uint32_t)(max(fd, f0) - fd);
        const uint32_t m_hi = (uint32_t)(min(fd + nOp, f0 + nf) - fd);
        // slot m of direction d sits at stage index fd + m - f0 >= 0 for m >= m_lo
        const int64_t seg = (int64_t)fd - (int64_t)f0;
        if (m_lo == 0) {  // a new direction: phase, rotation and mask of step s
          const float4 d0 = a.dirtab[4 * (uint64_t)d], d1 = a.dirtab[4 * (uint64_t)d + 1];
          const df tau = record_tau(sm.rec[si], d0, d1);
          float dtau = tau.hi + tau.lo;
          if (!first) {
            const df tp = record_tau(sm.rec[si - 1], d0, d1);
            dtau = (tau.hi - tp.hi) + (tau.lo - tp.lo);
          }
          th = tau.hi;
          tl = tau.lo;
          adt = fabsf(dtau);
          mode = (!valid || G.wabs_min * adt > kPiHi) ? 1 : (G.wabs_max * adt < kPiLo ? 0 : 2);
          const df rp = df_mul_raw(d_dw, tau);
          sincosf(reduce_2pi(rp.hi, rp.lo), &rs, &rc);
          float c2r, s2r;
          cmul(rc, rs, rc, rs, c2r, s2r);
          r2c = make_float2(c2r, c2r);
          r2s = make_float2(s2r, s2r);
          nr2s = make_float2(-s2r, -s2r);
          ef.et = ef.ep = ef.ft = ef.fp = make_float2(0.f, 0.f);
        }
        if (!__all_sync(0xffffffffu, mode == 1)) {
          if (G.uniform && __all_sync(0xffffffffu, mode != 2)) {
            // every point of the segment included (lanes with mode 1 are
            // discarded below): per block of kARS slots one reseed, then
            // pairs rotated by R^2
#pragma unroll 1
            for (uint32_t m = m_lo; m < m_hi; m += kARS) {
              const float4 *cp = sm.cst[(seg + (int64_t)m) >> 1];
              float zs, zc;
              phasor_rev(cp[4].x, cp[4].y, th, tl, zs, zc);
              float2 zr = make_float2(zc, zc * rc - zs * rs);
              float2 zi = make_float2(zs, zc * rs + zs * rc);
#pragma unroll
              for (int q = 0; q < kARS / 2; ++q) {
                ef.add(cp + 6 * q, zr, zi);
                if (q + 1 < kARS / 2) rot2p(zr, zi, r2c, r2s, nr2s, zr, zi);
              }
            }
          } else {
            // per-point mask (and one reseed per point on a non-uniform axis)
            double n0 = 0.0, n1 = 0.0, cT = 0.0;
            bool have_n = false;
#pragma unroll 1
            for (uint32_t m = m_lo; m < m_hi; m += kARS) {
              const float4 *cp = sm.cst[(seg + (int64_t)m) >> 1];
              float2 zr, zi;
              {
                float zs, zc;
                phasor_rev(cp[4].x, cp[4].y, th, tl, zs, zc);
                zr = make_float2(zc, zc * rc - zs * rs);
                zi = make_float2(zs, zc * rs + zs * rc);
              }
#pragma unroll 1
              for (int q = 0; q < kARS / 2; ++q) {
                const float4 *c = cp + 6 * q;
                if (!G.uniform) {
                  float zs, zc;
                  phasor_rev(c[4].x, c[4].y, th, tl, zs, zc);
                  zr.x = zc;
                  zi.x = zs;
                  phasor_rev(c[4].z, c[4].w, th, tl, zs, zc);
                  zr.y = zc;
                  zi.y = zs;
                }
                const float4 aw = c[5];
                bool inc[2] = {aw.x * adt < kPiLo, aw.y * adt < kPiLo};
                if (mode == 2) {
#pragma unroll
                  for (int e = 0; e < 2; ++e) {
                    const float ph = (e ? aw.y : aw.x) * adt;
                    const uint32_t mm = m + 2 * q + e;
                    if (!inc[e] && !(ph > kPiHi) && mm < nO) {
                      if (!have_n) {
                        const uint32_t iT = d % nT, iP = d / nT;
                        n0 = p.sin_theta[iT] * p.cos_phi[iP];
                        n1 = p.sin_theta[iT] * p.sin_phi[iP];
                        cT = p.cos_theta[iT];
                        have_n = true;
                      }
                      inc[e] = exact_mask(p, base, s, it_start, p.omega[mm], n0, n1, cT);
                    }
                  }
                }
                const float2 g = make_float2(inc[0] ? 1.f : 0.f, inc[1] ? 1.f : 0.f);
                ef.add(c, __fmul2_rn(zr, g), __fmul2_rn(zi, g));
                if (G.uniform) rot2p(zr, zi, r2c, r2s, nr2s, zr, zi);
              }
            }
          }
        }
        if (m_hi == nOp && mode != 1) {  // the direction is complete: chain rule
          const float et = ef.et.x + ef.et.y, ep = ef.ep.x + ef.ep.y;
          const float ft = ef.ft.x + ef.ft.y, fp = ef.fp.x + ef.fp.y;
          const float4 d1 = a.dirtab[4 * (uint64_t)d + 1], d2 = a.dirtab[4 * (uint64_t)d + 2],
                       d3 = a.dirtab[4 * (uint64_t)d + 3];
          const float4 q2 = sm.rec[si][2], q3 = sm.rec[si][3];
          const float f_c = d1.z, f_sx = d1.w, f_sy = d2.x, f_cz = d2.y;
          const float thx = d2.z, thy = d2.w, thz = d3.x, phx = d3.y, phy = d3.z;
          const float D = q2.w + f_c * q2.z - f_sx * q2.x - f_sy * q2.y;
          const float c2 = __frcp_rn(D);
          const float an = f_sx * q3.x + f_sy * q3.y + f_cz * q3.z;
          const float c22 = c2 * c2;
          const float c1 = an * c22;
          const float tb = thx * q2.x + thy * q2.y + thz * q2.z;
          const float ta = thx * q3.x + thy * q3.y + thz * q3.z;
          const float pb = phx * q2.x + phy * q2.y;
          const float pa = phx * q3.x + phy * q3.y;
          const float amp_t = -(c1 * tb + c2 * ta);
          const float amp_p = -(c1 * pb + c2 * pa);
          // x: n (amp_t F_t + amp_p F_p)
          const float fx = amp_t * ft + amp_p * fp;
          // bbar: -(2 an c2^3 e.b + c2^2 e.a) n E - c1 e E;  a: -(c2^2 e.b) n E - c2 e E
          const float kb = -(et * (2.f * an * c22 * c2 * tb + c22 * ta) +
                             ep * (2.f * an * c22 * c2 * pb + c22 * pa));
          const float ka = -(et * c22 * tb + ep * c22 * pb);
          const float nv3[3] = {f_sx, f_sy, f_cz};
          const float ev3[3] = {et * thx + ep * phx, et * thy + ep * phy, et * thz};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            gF[c] += nv3[c] * fx;
            gF[3 + c] += kb * nv3[c] - c1 * ev3[c];
            gF[6 + c] += ka * nv3[c] - c2 * ev3[c];
          }
        }
      }
#pragma unroll
      for (int c = 0; c < kAG; ++c) gD[c] += (double)gF[c];
    }
    if (valid) {
#pragma unroll
      for (int c = 0; c < kAG; ++c) a.gstep[(uint64_t)(base + s) * kAG + c] = gD[c];
    }
    __syncthreads();  // records of this item no longer read
  }
}

// ------------------------------------------------------------------------
// Even omega axes: the sums over omega by transforms (the transpose of the
// forward's, sr_fast_sum.cuh).  For a (track, direction) the sums
//   H_c(tau) = sum_j conj(U_cj) exp(i omega_j tau),  K_c the same with omega_j U
// are band-limited functions of tau: one FFT each of conj(U) divided by the
// spreading kernel's transform gives cells on the circle of d_omega tau, and
// every step takes 8 of them with the kernel's weights, whatever the number of
// frequencies.  E_c = Re H_c, F_c = Im K_c.
//
// adj_fields_kernel: a warp per (track, snapshot segment, direction, band)
// writes the cells of the four fields, [cell][H_th, H_ph, K_th, K_ph], the
// circle's first 8 cells again behind its last.
// adj_interp_kernel: as below a CTA owns 256 steps of a track, a lane one step,
// and loops over its directions; the records are turned into the plane of phi
// once per phi.  Bound by instructions (57 % of the issue slots at 16 warps an
// SM, 128 registers) with the 16 cell loads of a (direction, step), 64 cycles
// per warp and SM, beside them.  128 tracks of 2000 steps, 128 x 32 x 32 points:
// 33.9 ms walking, 5.2 with the transforms (0.4 for the fields).
// ------------------------------------------------------------------------

// U of one point: summed over the snapshots k0..k1 that the steps enter.
__device__ __forceinline__ float4 point_u(const AdjParams &a, uint32_t t, uint32_t k0, uint32_t k1,
                                          uint64_t P, uint64_t gi, float wt, float swt) {
  float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t k = k0; k <= k1; ++k) {
    const float4 C = a.gcst[(uint64_t)k * P + gi];
    if (a.linear) {
      u.x += swt * C.x; u.y += swt * C.y;
      u.z += swt * C.z; u.w += swt * C.w;
    } else {
      const float4 A = a.save_A[((uint64_t)t * a.f.n_snaps + k) * P + gi];
      u.x += wt * (C.x * A.x + C.y * A.z);
      u.y += wt * (C.x * A.y + C.y * A.w);
      u.z += wt * (C.y * A.x + C.z * A.z);
      u.w += wt * (C.y * A.y + C.z * A.w);
    }
  }
  return u;
}

template <int R1>
__global__ void __launch_bounds__(kFastWarps * 32, 3) adj_fields_kernel(
    const __grid_constant__ AdjParams a) {
  const FarMixedParams &p = a.f;
  if (!by_transform(p)) return;
  constexpr int NF = 32 / R1, M = 32 * R1;
  constexpr int DP = NF > 4 ? NF / 4 : 1;     // directions per pass
  constexpr int NPASS = 4 * DP / NF;
  __shared__ float2 tr_all[kFastWarps][32 * 33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2 *tr = tr_all[warp];
  const FastParams &f = p.fast;
  const uint32_t n_dirs = p.n_theta * p.n_phi;
  const uint64_t P = (uint64_t)p.n_omega * n_dirs;
  const uint32_t dgroups = (n_dirs + DP - 1) / DP;
  uint64_t task = (uint64_t)blockIdx.x * kFastWarps + warp;
  const uint32_t band = (uint32_t)(task % f.n_bands);
  task /= f.n_bands;
  const uint32_t d0 = (uint32_t)(task % dgroups) * DP;
  task /= dgroups;
  const uint32_t k0 = (uint32_t)(task % p.n_snaps), t = a.t_lo + (uint32_t)(task / p.n_snaps);
  if (t >= a.t_hi) return;
  const uint32_t k1 = last_fired(p, t);
  if (k1 == 0xffffffffu || k0 > k1) return;
  const uint32_t j0 = band * f.nb;
  const int nb = (int)min(f.nb, p.n_omega - j0);
  const float wt = (float)p.weight[t], swt = (float)sqrt(p.weight[t]);
#pragma unroll 1
  for (int ps = 0; ps < NPASS; ++ps) {
    float2 x[NF][R1], y[32];
#pragma unroll
    for (int dd = 0; dd < DP; ++dd) {
      const uint32_t d = min(d0 + dd, n_dirs - 1);
#pragma unroll
      for (int i = 0; i < R1; ++i) {
        const int n = 32 * i + lane;                        // frequency index mod M
        const int j = (n < M / 2 ? n : n - M) + nb / 2;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        float dv = 0.f, w = 0.f;
        if (j >= 0 && j < nb) {
          u = point_u(a, t, k0, k1, P, (uint64_t)d * p.n_omega + j0 + j, wt, swt);
          dv = (float)f.deconv[j - nb / 2 + kFastMaxBand / 2];
          w = a.wtab[j0 + j].z;
        }
        const float2 th = make_float2(u.x * dv, -u.y * dv), ph = make_float2(u.z * dv, -u.w * dv);
        auto field = [&](int q) {
          const float2 b = (q & 1) ? ph : th;
          return (q & 2) ? make_float2(b.x * w, b.y * w) : b;
        };
        if constexpr (NF >= 4) {
#pragma unroll
          for (int q = 0; q < 4; ++q) x[4 * dd + q][i] = field(q);
        } else {
#pragma unroll
          for (int q = 0; q < NF; ++q) x[q][i] = field(ps * NF + q);
        }
      }
    }
    fft_fields<R1, NF>(x, y, tr, f.twiddle, lane);
    const int q = lane / R1, al = lane % R1;
    const int fq = ps * NF + q;                             // field of the pass's directions
    const uint32_t d = d0 + fq / 4;
    if (d < n_dirs) {
      float2 *o = a.fields +
                  ((((uint64_t)(t - a.t_lo) * p.n_snaps + k0) * n_dirs + d) * f.n_bands + band) *
                      (4ull * (M + kTaps)) + (fq & 3);
#pragma unroll
      for (int b = 0; b < 32; ++b) o[4 * (al + R1 * b)] = y[bitrev<32>(b)];
      // the circle's first cells once more behind its last
#pragma unroll
      for (int b = 0; b * R1 < kTaps; ++b)
        if (al + R1 * b < kTaps) o[4 * (M + al + R1 * b)] = y[bitrev<32>(b)];
    }
    __syncwarp();
  }
}

// WALK: with the walk of warps with many cut steps, taken where a sample of steps
// says that there are some (beside it the loop of other steps loses 5 % to the
// registers and the L1 cache that it takes).
template <bool WALK>
__global__ void __launch_bounds__(kASteps, 2) adj_interp_kernel(
    const __grid_constant__ AdjParams a) {
  const FarMixedParams &p = a.f;
  if (!by_transform(p) || (*a.many_cut != 0u) != WALK) return;
  const FastParams &f = p.fast;
  __shared__ float sum[kAG][2][kASteps];
  __shared__ float4 cut_u[WALK ? kAW : 1][32][2];  // U, omega U of 32 frequencies, for cut steps
  const int lane = threadIdx.x & 31;
  const uint32_t nT = p.n_theta, n_dirs = nT * p.n_phi;
  const uint64_t P = (uint64_t)p.n_omega * n_dirs;
  const AdjGlobals G = *a.glob;
  const int M = (int)f.M;
  const float Mf = (float)M;
  const double inv2pi = 0.15915494309189533577;
  const double w0 = p.omega[0];
  const double dw = (p.omega[p.n_omega - 1] - w0) / (double)(p.n_omega - 1);
  const df f_d = df_from_double(dw * inv2pi);
  const int64_t i_lo = a.item_off[a.t_lo], i_hi = a.item_off[a.t_hi];
  const int64_t n_items = (i_hi - i_lo) * a.n_split;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int64_t it = i_lo + item / a.n_split;
    const uint32_t split = (uint32_t)(item % a.n_split);
    const uint32_t dA = (uint32_t)((uint64_t)n_dirs * split / a.n_split);
    const uint32_t dB = (uint32_t)((uint64_t)n_dirs * (split + 1) / a.n_split);
    uint32_t lo = a.t_lo, hi = a.t_hi;  // last track with item_off[t] <= it
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (a.item_off[mid] <= it) lo = mid; else hi = mid;
    }
    const uint32_t t = lo;
    const int64_t base = p.offsets[t];
    SnapSegment seg{0, 0, 0, 0};
    track_segments(p, t, (uint32_t)kASteps, (uint32_t)(it - a.item_off[t]), &seg);
    const uint32_t s = seg.r0 + threadIdx.x;
    const bool valid = s < seg.r1;
    if (!__any_sync(0xffffffffu, valid)) continue;  // whole warps
    const uint32_t sc = valid ? s : seg.r1 - 1;
    const uint32_t it_start = p.it_start[t];
    const float wt = (float)p.weight[t], swt = (float)sqrt(p.weight[t]);
    const float4 *rp = p.records + (base + sc) * kRecF4;
    const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1), r2 = __ldg(rp + 2), r3 = __ldg(rp + 3);
    // differences to the step before, for the quick test of the mask (the
    // track's first step compares its whole phase with zero)
    float dq = r0.x + r0.y, dz = r1.z + r1.w, dx = r0.z + r0.w, dy = r1.x + r1.y;
    if (sc > 0) {
      const float4 e0 = __ldg(rp - kRecF4), e1 = __ldg(rp - kRecF4 + 1);
      dq = (r0.x - e0.x) + (r0.y - e0.y);
      dx = (r0.z - e0.z) + (r0.w - e0.w);
      dy = (r1.x - e1.x) + (r1.y - e1.y);
      dz = (r1.z - e1.z) + (r1.w - e1.w);
    }
    // below it the FP32 difference is certainly inside the limit for every
    // frequency, with a 1e-3 margin, whatever its rounding
    const float sure = 0.999f * kPiLo / G.wabs_max -
                       kQuickErr * (fabsf(dq) + G.omc_max * fabsf(dz) +
                                    G.sin_max * (fabsf(dx) + fabsf(dy)));
    // x, bbar, a: FP32 over up to 8 directions of a phi (rho, phi, z of each),
    // turned back and added as double-floats
#pragma unroll
    for (int c = 0; c < kAG; ++c) sum[c][0][threadIdx.x] = sum[c][1][threadIdx.x] = 0.f;
    const float2 *fld = a.fields +
                        (((uint64_t)(t - a.t_lo) * p.n_snaps + seg.k0) * n_dirs) * f.n_bands *
                            (4ull * (M + kTaps));
    uint32_t d = dA;
    while (d < dB) {
      const uint32_t iP = d / nT, dE = min(dB, (iP + 1) * nT);
      // the record in the plane of phi
      const float4 ph = phi_pairs(p, iP);
      const df rho = df_add(df_mul(df{ph.x, ph.y}, df{r0.z, r0.w}),
                            df_mul(df{ph.z, ph.w}, df{r1.x, r1.y}));
      const float b_r = ph.x * r2.x + ph.z * r2.y, b_p = ph.x * r2.y - ph.z * r2.x;
      const float a_r = ph.x * r3.x + ph.z * r3.y, a_p = ph.x * r3.y - ph.z * r3.x;
      const float drho = ph.x * dx + ph.z * dy;
      float g_xr = 0.f, g_xz = 0.f, g_br = 0.f, g_bp = 0.f, g_bz = 0.f, g_ar = 0.f, g_ap = 0.f,
            g_az = 0.f;
#pragma unroll 1
      for (; d < dE; ++d) {
        // 1 - cos, sin, cos of theta: (dc hi, lo, sin hi, lo), (dc, sin, cos)
        const float4 c0 = __ldg(a.dirtab + 4 * (uint64_t)nT * p.n_phi + 2 * (d - iP * nT));
        const float4 c1v = __ldg(a.dirtab + 4 * (uint64_t)nT * p.n_phi + 2 * (d - iP * nT) + 1);
        const df p1 = df_mul_raw(df{c0.x, c0.y}, df{r1.z, r1.w});
        const df p2 = df_mul_raw(df{c0.z, c0.w}, rho);
        const df s1 = two_sum(r0.x, p1.hi);
        const df s2 = two_sum(s1.hi, -p2.hi);
        const df tau = fast_two_sum(s2.hi, ((r0.y + p1.lo) - p2.lo) + (s1.lo + s2.lo));
        // mask: certain where the FP32 difference is small enough, else from the
        // double-float tau of both steps
        int mode = valid ? 0 : 1;  // 0: every frequency enters, 1: none, 2: some
        float et = 0.f, ep = 0.f, ft = 0.f, fp = 0.f;
        const float quick = fabsf(dq + c1v.x * dz - c1v.y * drho);
        if (__any_sync(0xffffffffu, valid && !(quick < sure))) {
          float dt0 = tau.hi + tau.lo;
          if (sc > 0) {
            const float4 e0 = __ldg(rp - kRecF4), e1 = __ldg(rp - kRecF4 + 1);
            const df rb = df_add(df_mul(df{ph.x, ph.y}, df{e0.z, e0.w}),
                                 df_mul(df{ph.z, ph.w}, df{e1.x, e1.y}));
            const df q1 = df_mul_raw(df{c0.x, c0.y}, df{e1.z, e1.w});
            const df q2 = df_mul_raw(df{c0.z, c0.w}, rb);
            const df v1 = two_sum(e0.x, q1.hi);
            const df v2 = two_sum(v1.hi, -q2.hi);
            const df tb = fast_two_sum(v2.hi, ((e0.y + q1.lo) - q2.lo) + (v1.lo + v2.lo));
            dt0 = (tau.hi - tb.hi) + (tau.lo - tb.lo);
          }
          const float adt = fabsf(dt0);
          if (valid)
            mode = G.wabs_max * adt < kPiLo ? 0 : (G.wabs_min * adt > kPiHi ? 1 : 2);
          // cut steps: each lane finds its included frequencies; where many of the
          // warp's steps are cut, each lane walks its own by rotations, reseeded
          // every 8 frequencies; where few are, the warp sums four steps' at a
          // time term by term, lane + 32 k (20 tracks of 1500 steps, 88 % cut, 16 x 16
          // directions, 16 / 64 / 128 frequencies: walked 0.49 / 0.72 / 1.07 ms, four
          // at a time 1.95 / 2.61 / 3.85; without the transforms 0.76 / 1.73 / 3.07)
          const uint32_t mine =
              mode == 2 ? cut_interval<false>(p, 0, (int)p.n_omega, G.w0f, G.dwf, d, base, s,
                                              it_start, adt)
                        : 1u;
          uint32_t cut = __ballot_sync(0xffffffffu, mode == 2);
          if (WALK && walk_cut(cut, p.n_omega, 45u, 23u)) {
            cut = 0u;
            const int jf = (int)(mine & 0xffffu), jl = (int)(mine >> 16);
            int first, last;
            cut_span(mode == 2, mine, first, last);
            float4 (*su)[2] = cut_u[threadIdx.x >> 5];
            float rs, rc, w_et = 0.f, w_ep = 0.f, w_ft = 0.f, w_fp = 0.f;
            phasor_rev(f_d.hi, f_d.lo, tau.hi, tau.lo, rs, rc);
#pragma unroll 1
            for (int j0 = first & ~31; j0 <= last; j0 += 32) {
              float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
              float w = 0.f;
              if (j0 + lane <= last) {
                u = point_u(a, t, seg.k0, seg.k1, P, (uint64_t)d * p.n_omega + j0 + lane, wt, swt);
                w = a.wtab[j0 + lane].z;
              }
              __syncwarp();
              su[lane][0] = u;
              su[lane][1] = make_float4(w * u.x, w * u.y, w * u.z, w * u.w);
              __syncwarp();
#pragma unroll 1
              for (int j8 = j0; j8 < j0 + 32 && j8 <= last; j8 += 8) {
                const float4 w8 = __ldg(a.wtab + j8);
                float zs, zc;
                phasor_rev(w8.x, w8.y, tau.hi, tau.lo, zs, zc);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float4 v = su[j8 - j0 + i][0], wv = su[j8 - j0 + i][1];
                  const bool in = j8 + i >= jf && j8 + i <= jl;
                  const float c = in ? zc : 0.f, s1 = in ? zs : 0.f;
                  w_et = __fmaf_rn(v.x, c, __fmaf_rn(v.y, s1, w_et));
                  w_ep = __fmaf_rn(v.z, c, __fmaf_rn(v.w, s1, w_ep));
                  w_ft = __fmaf_rn(wv.x, s1, __fmaf_rn(-wv.y, c, w_ft));
                  w_fp = __fmaf_rn(wv.z, s1, __fmaf_rn(-wv.w, c, w_fp));
                  const float q = zc * rc - zs * rs;
                  zs = zc * rs + zs * rc;
                  zc = q;
                }
              }
            }
            if (mode == 2) { et = w_et; ep = w_ep; ft = w_ft; fp = w_fp; }
          }
          while (cut) {
            float v[16];
            uint32_t batch = 0u;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              v[4 * e] = v[4 * e + 1] = v[4 * e + 2] = v[4 * e + 3] = 0.f;
              if (cut) {
                const int b = __ffs(cut) - 1;
                cut &= cut - 1;
                batch |= 1u << b;
                const uint32_t r = __shfl_sync(0xffffffffu, mine, b);
                const float th = __shfl_sync(0xffffffffu, tau.hi, b);
                const float tl = __shfl_sync(0xffffffffu, tau.lo, b);
                const int jl = (int)(r >> 16);
                for (int j = (int)(r & 0xffffu) + lane; j <= jl; j += 32) {
                  const float4 u =
                      point_u(a, t, seg.k0, seg.k1, P, (uint64_t)d * p.n_omega + j, wt, swt);
                  const float4 w = __ldg(a.wtab + j);
                  float zs, zc;
                  phasor_rev(w.x, w.y, th, tl, zs, zc);
                  v[4 * e] += u.x * zc + u.y * zs;
                  v[4 * e + 1] += u.z * zc + u.w * zs;
                  v[4 * e + 2] += w.z * (u.x * zs - u.y * zc);
                  v[4 * e + 3] += w.z * (u.z * zs - u.w * zc);
                }
              }
            }
            // lane i ends with the warp's sum of value i / 2
#pragma unroll
            for (int n = 8; n > 0; n >>= 1) {
              const int o = 2 * n;
              const bool up = (lane & o) != 0;
#pragma unroll
              for (int i = 0; i < n; ++i) {
                const float keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
              }
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            const int e = __popc(batch & ((1u << lane) - 1u)) & 3;
            const float s0 = __shfl_sync(0xffffffffu, v[0], 8 * e);
            const float s1 = __shfl_sync(0xffffffffu, v[0], 8 * e + 2);
            const float s2 = __shfl_sync(0xffffffffu, v[0], 8 * e + 4);
            const float s3 = __shfl_sync(0xffffffffu, v[0], 8 * e + 6);
            if ((batch >> lane) & 1u) { et = s0; ep = s1; ft = s2; fp = s3; }
          }
        }
        if (mode == 0) {
          const float pr = f_d.hi * tau.hi;
          float e = __fmaf_rn(f_d.hi, tau.hi, -pr);
          e = __fmaf_rn(f_d.hi, tau.lo, e);
          e = __fmaf_rn(f_d.lo, tau.hi, e);
          const float uh = (pr - rintf(pr)) * Mf, ul = e * Mf;
          const float rm = rintf((uh - 0.5f) + ul);
          float wk[kTaps];
          kb_taps(((uh - rm) - 0.5f) + ul, wk);
          const int m = ((int)rm - 3) & (M - 1);
          for (uint32_t band = 0; band < f.n_bands; ++band) {
            const float4 *cell = reinterpret_cast<const float4 *>(
                fld + ((uint64_t)d * f.n_bands + band) * (4ull * (M + kTaps)) + 4 * m);
            float2 ht = make_float2(0.f, 0.f), hp = ht, kt = ht, kp = ht;
#pragma unroll
            for (int l = 0; l < kTaps; ++l) {
              const float4 h = __ldg(cell + 2 * l), k = __ldg(cell + 2 * l + 1);
              const float2 ww = make_float2(wk[l], wk[l]);
              ht = __ffma2_rn(ww, make_float2(h.x, h.y), ht);
              hp = __ffma2_rn(ww, make_float2(h.z, h.w), hp);
              kt = __ffma2_rn(ww, make_float2(k.x, k.y), kt);
              kp = __ffma2_rn(ww, make_float2(k.z, k.w), kp);
            }
            const float4 fc = __ldg(a.bandtab + band);  // its centre frequency / 2 pi
            float zs, zc;
            phasor_exact(fc.x, fc.y, tau.hi, tau.lo, zs, zc);
            et += ht.x * zc - ht.y * zs;
            ep += hp.x * zc - hp.y * zs;
            ft += kt.x * zs + kt.y * zc;
            fp += kp.x * zs + kp.y * zc;
          }
        }
        if (mode != 1) {  // the chain rule, in the plane of phi
          const float st = c1v.y, ct = c1v.z;
          const float D = r2.w + c1v.x * r2.z - st * b_r;
          const float c2 = rcp_newton(D);
          const float an = st * a_r + ct * r3.z;
          const float c22 = c2 * c2;
          const float c1 = an * c22;
          const float tb = ct * b_r - st * r2.z, ta = ct * a_r - st * r3.z;
          const float amp_t = -(c1 * tb + c2 * ta), amp_p = -(c1 * b_p + c2 * a_p);
          // x: n (amp_t F_t + amp_p F_p)
          const float fx = amp_t * ft + amp_p * fp;
          // bbar: -(2 an c2^3 e.b + c2^2 e.a) n E - c1 e E;  a: -(c2^2 e.b) n E - c2 e E
          const float m3 = 2.f * c1 * c2;
          const float kb = -(et * (m3 * tb + c22 * ta) + ep * (m3 * b_p + c22 * a_p));
          const float ka = -c22 * (et * tb + ep * b_p);
          const float er = et * ct, ez = -et * st;  // theta-hat = (cos, -sin) in (rho, z)
          g_xr += st * fx;
          g_xz += ct * fx;
          g_br += kb * st - c1 * er;
          g_bp -= c1 * ep;
          g_bz += kb * ct - c1 * ez;
          g_ar += ka * st - c2 * er;
          g_ap -= c2 * ep;
          g_az += ka * ct - c2 * ez;
        }
        if (((d - dA) & 7u) == 7u || d + 1u == dE) {
          const float gF[kAG] = {ph.x * g_xr,
                                 ph.z * g_xr,
                                 g_xz,
                                 ph.x * g_br - ph.z * g_bp,
                                 ph.z * g_br + ph.x * g_bp,
                                 g_bz,
                                 ph.x * g_ar - ph.z * g_ap,
                                 ph.z * g_ar + ph.x * g_ap,
                                 g_az};
#pragma unroll
          for (int c = 0; c < kAG; ++c) {
            const df v = two_sum(sum[c][0][threadIdx.x], gF[c]);
            sum[c][0][threadIdx.x] = v.hi;
            sum[c][1][threadIdx.x] += v.lo;
          }
          g_xr = g_xz = g_br = g_bp = g_bz = g_ar = g_ap = g_az = 0.f;
        }
      }
    }
    if (valid) {
#pragma unroll
      for (int c = 0; c < kAG; ++c)
        a.gstep[((uint64_t)split * p.total_steps + base + s) * kAG + c] =
            (double)sum[c][0][threadIdx.x] + (double)sum[c][1][threadIdx.x];
    }
  }
}

size_t adj_smem_bytes() { return sizeof(AdjSmem); }

void launch_adj_fields(const AdjParams &a, uint64_t n_dirs, cudaStream_t s) {
  const uint64_t dp = std::max(1u, 256u / a.f.fast.M);
  const uint64_t warps = (uint64_t)(a.t_hi - a.t_lo) * a.f.n_snaps * ((n_dirs + dp - 1) / dp) *
                         a.f.fast.n_bands;
  const unsigned blocks = (unsigned)((warps + kFastWarps - 1) / kFastWarps);
  switch (a.f.fast.M) {
    case 128: adj_fields_kernel<4><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    case 256: adj_fields_kernel<8><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    case 512: adj_fields_kernel<16><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    default: adj_fields_kernel<32><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
  }
}

struct AdjLayout {
  size_t records, gcst, wtab, dirtab, glob, item_off, gstep, wpart, tables, bandtab, fields, total;
  uint32_t w_chunks;
  AdjFields fl;
};

AdjLayout adj_layout(int64_t total_steps, uint64_t P, uint32_t n_omega, uint64_t n_dirs,
                     uint32_t n_tracks, uint32_t n_snaps, bool least) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  AdjLayout l;
  l.w_chunks = adj_weight_chunks(P, n_tracks, device_sm_count());
  l.fl = adj_fields_layout(total_steps, n_omega, n_dirs, n_tracks, n_snaps, 32, kASteps, least);
  l.gstep = 256;
  l.records = l.gstep + up((size_t)total_steps * kAG * 8 * l.fl.n_split);
  l.gcst = l.records + up((size_t)total_steps * kRecBytes);
  l.wtab = l.gcst + up((size_t)P * 16 * (n_snaps ? n_snaps : 1));
  l.dirtab = l.wtab + up((size_t)n_omega * 16);
  l.glob = l.dirtab + up((size_t)n_dirs * 96);
  l.item_off = l.glob + 256;
  l.wpart = l.item_off + up(((size_t)n_tracks + 1) * 8);
  l.tables = l.wpart + up((size_t)n_tracks * l.w_chunks * 8);
  l.bandtab = l.tables + up(kFastTables);
  l.fields = l.bandtab + up((size_t)l.fl.n_bands * 16);
  l.total = l.fields + l.fl.bytes;
  return l;
}

int check_adjoint_args(const sr_tracks *t, const sr_grid *g, void *const *out,
                       int comp = SR_COMP_TOTAL) {
  int rc = validate_spectrum_args(t, g, comp, SR_PREC_MIXED, out);
  if (rc) return rc;
  if (g->mode != SR_MODE_FAR) return fail(SR_ERR_UNSUPPORTED, "the adjoint is far field only");
  if (t->n_snaps < 1)
    return fail(SR_ERR_UNSUPPORTED, "the adjoint needs at least one snapshot (n_snaps >= 1)");
  return SR_OK;
}

}  // namespace
}  // namespace sr

using namespace sr;

extern "C" int sr_far_forward_saved(const sr_tracks *t, const sr_grid *g, int comp,
                                    int precision, void *const *out, float *saved_A,
                                    void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  int rc = check_adjoint_args(t, g, out, comp);
  if (rc) return rc;
  if (precision != SR_PREC_MIXED && precision != SR_PREC_DF)
    return fail(SR_ERR_INVALID, "precision %d (SR_PREC_MIXED or SR_PREC_DF)", precision);
  if (!saved_A) return fail(SR_ERR_INVALID, "saved_A is NULL");
  const uint64_t P = (uint64_t)g->n_omega * g->n_theta * g->n_phi;
  if (P == 0 || t->n_tracks == 0) return SR_OK;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(saved_A, 0, (size_t)t->n_tracks * t->n_snaps * P * 16, s);
  if (e != cudaSuccess) return cuda_fail(e, "saved_A reset");
  FarMixedParams p = make_far_mixed_params(t, g, comp, out);
  p.save_A = saved_A;
  if (precision == SR_PREC_DF) {
    const FarMixedConfig cfg =
        far_df_choose(g->n_omega, g->n_theta * g->n_phi, t->n_tracks, device_sm_count());
    return launch_far_df(p, cfg, workspace, workspace_bytes, s);
  }
  return launch_far_mixed(p, mixed_config(t, g, comp), workspace, workspace_bytes, s);
}

extern "C" int sr_far_total_forward_saved(const sr_tracks *t, const sr_grid *g, double *spectrum,
                                          float *saved_A, void *workspace,
                                          size_t workspace_bytes, void *stream) {
  void *out[6] = {spectrum};
  return sr_far_forward_saved(t, g, SR_COMP_TOTAL, SR_PREC_MIXED, out, saved_A, workspace,
                              workspace_bytes, stream);
}

extern "C" int sr_far_total_forward_saved_df(const sr_tracks *t, const sr_grid *g,
                                             double *spectrum, float *saved_A, void *workspace,
                                             size_t workspace_bytes, void *stream) {
  void *out[6] = {spectrum};
  return sr_far_forward_saved(t, g, SR_COMP_TOTAL, SR_PREC_DF, out, saved_A, workspace,
                              workspace_bytes, stream);
}

namespace {
int64_t backward_bytes(const sr_tracks *t, const sr_grid *g, bool least) {
  if (!t || !g) return -1;
  const uint64_t n_dirs = (uint64_t)g->n_theta * g->n_phi;
  return (int64_t)adj_layout(t->total_steps, n_dirs * g->n_omega, g->n_omega, n_dirs,
                             t->n_tracks, t->n_snaps, least)
      .total;
}
}  // namespace

extern "C" int64_t sr_far_backward_workspace_bytes(const sr_tracks *t, const sr_grid *g) {
  return backward_bytes(t, g, false);
}

extern "C" int64_t sr_far_backward_workspace_bytes_min(const sr_tracks *t, const sr_grid *g) {
  return backward_bytes(t, g, true);
}

extern "C" int64_t sr_far_total_backward_workspace_bytes(const sr_tracks *t, const sr_grid *g) {
  return sr_far_backward_workspace_bytes(t, g);
}

extern "C" int sr_far_total_backward(const sr_tracks *t, const sr_grid *g,
                                     const double *grad_spectrum, const float *saved_A,
                                     double *const *grad_track, double *grad_weight,
                                     void *workspace, size_t workspace_bytes, void *stream) {
  const double *grad_out[6] = {grad_spectrum};
  return sr_far_backward(t, g, SR_COMP_TOTAL, grad_out, saved_A, grad_track, grad_weight,
                         workspace, workspace_bytes, stream);
}

extern "C" int sr_far_backward(const sr_tracks *t, const sr_grid *g, int comp,
                               const double *const *grad_out, const float *saved_A,
                               double *const *grad_track, double *grad_weight, void *workspace,
                               size_t workspace_bytes, void *stream) {
  clear_error();
  if (!grad_out) return fail(SR_ERR_INVALID, "grad_out must not be NULL");
  int rc = check_adjoint_args(t, g, (void *const *)grad_out, comp);
  if (rc) return rc;
  if (!saved_A || !grad_track || !grad_weight)
    return fail(SR_ERR_INVALID, "saved_A, grad_track and grad_weight must not be NULL");
  for (int i = 0; i < 6; ++i)
    if (!grad_track[i]) return fail(SR_ERR_INVALID, "grad_track[%d] is NULL", i);
  if (t->n_tracks == 0) return SR_OK;
  const uint64_t n_dirs = (uint64_t)g->n_theta * g->n_phi;
  const uint64_t P = n_dirs * g->n_omega;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e;
  if (P == 0) {  // no spectrum: every gradient is zero
    for (int i = 0; i < 6; ++i) {
      e = cudaMemsetAsync(grad_track[i], 0, (size_t)t->total_steps * 8, s);
      if (e != cudaSuccess) return cuda_fail(e, "gradient reset");
    }
    e = cudaMemsetAsync(grad_weight, 0, (size_t)t->n_tracks * 8, s);
    return e == cudaSuccess ? SR_OK : cuda_fail(e, "gradient reset");
  }
  // the walk along the frequencies where the scratch does not hold the cells
  AdjLayout lay = adj_layout(t->total_steps, P, g->n_omega, n_dirs, t->n_tracks, t->n_snaps, false);
  if (workspace_bytes < lay.total)
    lay = adj_layout(t->total_steps, P, g->n_omega, n_dirs, t->n_tracks, t->n_snaps, true);
  if (!workspace || workspace_bytes < lay.total)
    return fail(SR_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", lay.total,
                workspace_bytes);
  if (((uintptr_t)workspace & 255u) != 0)
    return fail(SR_ERR_WORKSPACE, "workspace not 256-byte aligned");
  unsigned char *w = (unsigned char *)workspace;

  AdjParams a;
  memset(&a, 0, sizeof(a));
  a.f = make_far_mixed_params(t, g, comp, (void *const *)grad_out);
  a.f.status = (int *)w;
  a.f.records = (float4 *)(w + lay.records);
  for (int i = 0; i < n_outputs(comp); ++i) a.grad_out[i] = grad_out[i];
  a.linear = (comp == SR_COMP_CARTESIAN_COMPLEX || comp == SR_COMP_SPHERIC_COMPLEX) ? 1 : 0;
  a.save_A = (const float4 *)saved_A;
  a.gcst = (float4 *)(w + lay.gcst);
  a.wtab = (float4 *)(w + lay.wtab);
  a.dirtab = (float4 *)(w + lay.dirtab);
  a.glob = (AdjGlobals *)(w + lay.glob);
  a.item_off = (int64_t *)(w + lay.item_off);
  a.gstep = (double *)(w + lay.gstep);
  for (int i = 0; i < 6; ++i) a.grad[i] = grad_track[i];
  a.grad_w = grad_weight;
  a.n_split = lay.fl.n_split;
  a.many_cut = (unsigned int *)(w + 96);  // in the zeroed status block
  a.bandtab = (float4 *)(w + lay.bandtab);
  a.fields = (float2 *)(w + lay.fields);
  if (lay.fl.batch) fast_tables_bind(a.f, lay.fl.n_bands, lay.fl.nb, lay.fl.M, w + lay.tables, w);

  // the status block and, behind it, the per-step gradients: steps that enter
  // no snapshot (after the last one written) are not visited
  e = cudaMemsetAsync(w, 0, lay.records, s);
  if (e != cudaSuccess) return cuda_fail(e, "status reset");
  const int n_sm = device_sm_count();
  const int64_t step_blocks = std::max<int64_t>(
      16, std::min<int64_t>((t->total_steps + 255) / 256, (int64_t)n_sm * 128));
  if (t->total_steps > 0) launch_far_prepass(a.f, (int)step_blocks, s);
  adj_setup_kernel<false><<<3, 1024, 0, s>>>(a.f, a.wtab, a.glob, a.item_off, (uint32_t)kASteps,
                                       a.many_cut);
  {
    const uint64_t work = std::max<uint64_t>(P, n_dirs);
    const uint64_t nb = std::min<uint64_t>((work + 255) / 256, (uint64_t)n_sm * 64);
    adj_prep_kernel<<<(unsigned)nb, 256, 0, s>>>(a);
  }
  a.wpart = (double *)(w + lay.wpart);
  a.w_chunks = lay.w_chunks;
  adj_weight_partial_far_kernel<<<t->n_tracks * lay.w_chunks, kWeightThreads, 0, s>>>(
      a, P, lay.w_chunks, a.wpart);
  rc = cuda_fail(cudaGetLastError(), "adjoint prep launch");
  if (rc) return rc;
  const size_t smem = adj_smem_bytes();
  e = allow_smem((const void *)adj_far_kernel<kAW>, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "adjoint smem attribute");
  // upper bound of the work items (sum over tracks of ceil(n_body / 256))
  const int64_t items_max = t->total_steps / kASteps + (int64_t)t->n_tracks * t->n_snaps;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(items_max, 2 * (int64_t)n_sm));
  void *tok = nullptr;
  timing_record(s, true, &tok);
  for (uint32_t lo = 0; lay.fl.batch && lo < t->n_tracks; lo += lay.fl.batch) {
    a.t_lo = lo;
    a.t_hi = std::min(t->n_tracks, lo + lay.fl.batch);
    launch_adj_fields(a, n_dirs, s);
    const int64_t most = items_max * lay.fl.n_split;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(most, 2 * (int64_t)n_sm));
    adj_interp_kernel<false><<<blocks, kASteps, 0, s>>>(a);
    adj_interp_kernel<true><<<blocks, kASteps, 0, s>>>(a);
  }
  adj_far_kernel<kAW><<<grid, kAW * 32, smem, s>>>(a);
  timing_record(s, false, &tok);
  rc = cuda_fail(cudaGetLastError(), "adjoint kernel launch");
  if (rc) return rc;
  if (a.f.track_f32)
    adj_final_kernel<float><<<(int)step_blocks, 256, 0, s>>>(a);
  else
    adj_final_kernel<double><<<(int)step_blocks, 256, 0, s>>>(a);
  return cuda_fail(cudaGetLastError(), "adjoint final launch");
}
