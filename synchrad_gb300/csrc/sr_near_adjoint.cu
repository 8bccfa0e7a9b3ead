// Adjoint of the mixed-precision near field (every comp, one snapshot).
//
// Forward (sr_near_mixed.cu, the reference's synchrad/kernel_nearfield.cl:58-102):
//   S(p) = sum_t w_t dt^2 |A_t(p)|^2,   A = sum_s a_s e^{i phi_s},
//   a = n/r^2 + i omega (beta - n)/r,   phi = omega (t + r),
//   r = |P - x_s|, n = (P - x_s)/r, beta at step s.
// With g(p) = dL/dS(p), U = 2 g w dt^2 conj(A) and z = e^{i phi}:
//   dL/dw_t  = sum_p g dt^2 |A_t|^2,
//   dL/dbeta = -I1/r,
//   dL/dx    = (-R0 + 3 n (n.R0))/r^3 - (I1 + n ((beta-n).I1) - 2 n (n.I1))/r^2
//              + n ((beta-n).R2)/r,
// per step and screen point, with the omega sums (per component k)
//   R0_k = sum Re(U_k z),  I1_k = sum omega Im(U_k z),  R2_k = sum omega^2 Re(U_k z)
// (from d phi/dx = -omega n, dn/dx = -(I - n n^T)/r, dr/dx = -n), then
// dL/du = dL/dbeta / gamma - u (u . dL/dbeta) / gamma^3.  The comps differ in
// U_k only: total and cartesian (outputs w dt^2 |A_k|^2 summed or apart) give
// U_k = 2 g_k w dt^2 A_k (g_k = g for total); cartesian_complex (outputs sqrt(w)
// dt Re/Im(e^{i omega L} A_k)) gives U_k = sqrt(w) dt (g_k,re + i g_k,im)
// e^{-i omega L}; with dL = Re(conj(U) . dA), dL/dw = sum_p Re(conj(U) . A)/(2w).
// beta - n is formed
// as in the forward ((1 - n_z) - (1 - beta_z) along z).  The |dphase| < pi
// mask is held fixed (its decisions are the forward's).
//
// Layout as in the far-field adjoint (sr_far_adjoint.cu): a lane owns one
// step and walks a screen point's omega axis (rotation recurrence reseeded
// every 8 points, pairs of points in packed FP32), the U/W/Y constants of a
// block of (screen point, omega) slots are built in shared memory from the
// saved amplitudes, and a CTA owns 256 steps of one track and loops over
// every screen point, so each step's gradient is written once.  On even omega
// axes the sums over omega come from transforms (nadj_fields_kernel,
// nadj_interp_kernel below).
#include <algorithm>
#include <cmath>

#include "sr_common.cuh"
#include "sr_internal.h"
#include "sr_fast_sum.cuh"
#include "sr_mixed_common.cuh"
#include "sr_adjoint_common.cuh"

namespace sr {
namespace {

constexpr int kNAW = 8;               // warps per CTA
constexpr int kNASteps = kNAW * 32;   // steps per work item (one per lane)
constexpr int kNAStage = 512;         // (screen point, omega) slots per constants stage
constexpr int kNARS = 8;              // omega slots per phasor reseed
constexpr int kNAG = 6;               // per-step gradient components: x (3), beta (3)
constexpr int kNARecS = kRecF4;       // record stride in shared memory (80 bytes, as in HBM)
constexpr int kNAPair = 11;           // float4 per pair of slots in the constants

struct NearAdjParams {
  FarMixedParams f;            // tracks, grid (n_theta = radii), records, status
  const double *grad_out[6];   // [P] dL/dS_k per output of the comp, device layout
  int linear;                  // cartesian_complex: U does not depend on A
  const float4 *save_A;        // [n_tracks][P][2] (A_x re, im, A_y re, im), (A_z re, im, 0, 0)
  float4 *gcst;                // [P][2] point sensitivity in FP32: quadratic comps
                               // (2 dt^2 g_x, g_y, g_z, 0), 0; linear (V_x re, im,
                               // V_y re, im), (V_z re, im, 0, 0)
  float4 *wtab;                // [nO] (omega/2pi hi, lo, omega, |omega|) in FP32
  float4 *sctab;               // [n_screen] (X hi, lo, Y hi, lo) of the screen point
  AdjGlobals *glob;
  int64_t *item_off;           // [n_tracks + 1] first work item of each track
  double *gstep;               // [n_split][total_steps][kNAG] per-step gradients (x, beta)
  uint32_t n_split;            // runs of screen points summed apart
  float4 *bandtab;             // [n_bands] centre frequency / 2 pi
  float2 *fields;              // transforms' cells of a batch of tracks (see below)
  uint32_t t_lo, t_hi;         // the batch
  unsigned int *many_cut;      // whether the phase limit cuts many steps
  double *grad[6];             // x, y, z, ux, uy, uz  [total_steps]
  double *grad_w;              // [n_tracks]
  double *wpart;               // [n_tracks][w_chunks] partial weight gradients
  uint32_t w_chunks;
};

// Point sensitivity (FP64) of the loss to (A_x, A_y, A_z) at point gi for the
// output gradients g_k: quadratic comps 2 dt^2 (g_x, g_y, g_z) in v[0..2];
// cartesian_complex V_k = dt (g_k,re + i g_k,im) e^{-i omega L} in v[0..5].
__device__ __forceinline__ void near_point_sens(const NearAdjParams &a, uint32_t ksnap,
                                                uint64_t gi, double v[6]) {
  const FarMixedParams &p = a.f;
  const double s2 = 2.0 * p.dt * p.dt;
  const uint64_t gk = (uint64_t)ksnap * p.n_omega * p.n_theta * p.n_phi + gi;  // snapshot slot
  for (int k = 0; k < 6; ++k) v[k] = 0.0;
  if (p.comp == SR_COMP_TOTAL) {
    v[0] = v[1] = v[2] = s2 * a.grad_out[0][gk];
  } else if (p.comp == SR_COMP_CARTESIAN) {
    for (int k = 0; k < 3; ++k) v[k] = s2 * a.grad_out[k][gk];
  } else {  // cartesian_complex (FormFactor not applied, as the reference)
    const double w = p.omega[gi % p.n_omega];
    double sL, cL;
    sincos(w * p.L_screen, &sL, &cL);
    for (int k = 0; k < 3; ++k) {
      const double gr = a.grad_out[2 * k][gk], gim = a.grad_out[2 * k + 1][gk];
      v[2 * k] = p.dt * (gr * cL + gim * sL);
      v[2 * k + 1] = p.dt * (gim * cL - gr * sL);
    }
  }
}

// dL/dw_t = sum_p Re(conj(U) . A_t) / (2 w_t): chunk sums in FP64 from the
// FP64 point sensitivities, then one thread per track adds its chunks.
__global__ void nadj_weight_partial_kernel(NearAdjParams a, uint64_t P, uint32_t n_chunks,
                                           double *wpart) {
  const uint32_t t = blockIdx.x / n_chunks, b = blockIdx.x % n_chunks;
  const uint64_t chunk = (P + n_chunks - 1) / n_chunks;
  const uint64_t g0 = (uint64_t)b * chunk, g1 = min(P, g0 + chunk);
  double acc = 0.0;
  for (uint64_t g = g0 + threadIdx.x; g < g1; g += blockDim.x) {
    for (uint32_t ks = 0; ks < a.f.n_snaps; ++ks) {  // a snapshot that never fired has A = 0
      double v[6];
      near_point_sens(a, ks, g, v);
      const uint64_t ia = 2 * (((uint64_t)t * a.f.n_snaps + ks) * P + g);
      const float4 A0 = a.save_A[ia], A1 = a.save_A[ia + 1];
      const double re[3] = {A0.x, A0.z, A1.x}, im[3] = {A0.y, A0.w, A1.y};
      for (int k = 0; k < 3; ++k)
        acc += a.linear ? v[2 * k] * re[k] + v[2 * k + 1] * im[k]
                        : v[k] * (re[k] * re[k] + im[k] * im[k]);
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

// Point sensitivities in FP32 and the screen table.
__global__ void nadj_prep_kernel(NearAdjParams a) {
  const FarMixedParams &p = a.f;
  const uint32_t nR = p.n_theta;
  const uint64_t n_scr = (uint64_t)nR * p.n_phi;
  const uint64_t P = n_scr * p.n_omega;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P * p.n_snaps;
       i += stride) {
    double v[6];
    near_point_sens(a, (uint32_t)(i / P), i % P, v);
    a.gcst[2 * i] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
    a.gcst[2 * i + 1] = make_float4((float)v[4], (float)v[5], 0.f, 0.f);
  }
  for (uint64_t d = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; d < n_scr; d += stride) {
    const uint32_t iR = (uint32_t)(d % nR), iP = (uint32_t)(d / nR);
    const df X = df_from_double(p.sin_theta[iR] * p.cos_phi[iP]);  // radius * cos(phi)
    const df Y = df_from_double(p.sin_theta[iR] * p.sin_phi[iP]);  // radius * sin(phi)
    a.sctab[d] = make_float4(X.hi, X.lo, Y.hi, Y.lo);
  }
  if (p.fast.M != 0u) {
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

// dL/du_s from dL/dbeta_s (beta = u / gamma at the same step).
template <typename TT>
__global__ void nadj_final_kernel(NearAdjParams a) {
  const FarMixedParams &p = a.f;
  const TT *UX = (const TT *)p.ux, *UY = (const TT *)p.uy, *UZ = (const TT *)p.uz;
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
    double v[kNAG] = {0, 0, 0, 0, 0, 0};
    if (s < (int64_t)track_body(p, t))
      for (uint32_t k = 0; k < a.n_split; ++k)
        for (int c = 0; c < kNAG; ++c) v[c] += a.gstep[((int64_t)k * p.total_steps + g) * kNAG + c];
    a.grad[0][g] = v[0];
    a.grad[1][g] = v[1];
    a.grad[2][g] = v[2];
    const double ux = (double)UX[g], uy = (double)UY[g], uz = (double)UZ[g];
    const double gam = sqrt(1.0 + (ux * ux + uy * uy + uz * uz));
    const double ug = (ux * v[3] + uy * v[4] + uz * v[5]) / (gam * gam * gam);
    a.grad[3][g] = v[3] / gam - ux * ug;
    a.grad[4][g] = v[4] / gam - uy * ug;
    a.grad[5][g] = v[5] / gam - uz * ug;
  }
}

// Shared memory of one CTA.  Constants per pair of omega slots (m, m+1) of a
// screen point whose omega axis is padded to a multiple of kNARS slots:
//   [0..2] U_k (G Re A_k m, m+1, G Im A_k m, m+1)          k = x, y, z
//   [3..5] W_k (omega G Re A_k ..., -omega G Im A_k ...)
//   [6..8] Y_k (omega^2 G Re A_k ..., omega^2 G Im A_k ...)
//   [9]  (omega/2pi hi, lo of m, of m+1)    [10] (|omega| of m, m+1, 0, 0)
struct NearAdjSmem {
  float4 rec[kNASteps + 1][kNARecS];
  float4 cst[kNAStage / 2][kNAPair];
  uint64_t bar;
  uint64_t pad_;
};

__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }

// R0 += Re(U z), I1 += omega Im(U z), R2 += omega^2 Re(U z), per component,
// for a pair of points.
struct NearSums {
  float2 r0[3], i1[3], r2[3];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < 3; ++k) r0[k] = i1[k] = r2[k] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(const float4 *c, float2 zr, float2 zi) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 u = c[k], w = c[3 + k], y = c[6 + k];
      r0[k] = __ffma2_rn(lo2(u), zr, r0[k]);
      r0[k] = __ffma2_rn(hi2(u), zi, r0[k]);
      i1[k] = __ffma2_rn(lo2(w), zi, i1[k]);
      i1[k] = __ffma2_rn(hi2(w), zr, i1[k]);
      r2[k] = __ffma2_rn(lo2(y), zr, r2[k]);
      r2[k] = __ffma2_rn(hi2(y), zi, r2[k]);
    }
  }
};

// Geometry of one step and screen point from the step record: the retarded
// time tau' = t + r - L = (t - z) + rho^2/(r + L - z) (double-float), the
// distance r and n (FP32), and 1 - n_z.
struct NearGeo {
  df tau;
  float r, nx, ny, nz, omn;
};

__device__ __forceinline__ NearGeo near_geo(const float4 *rec, const float4 &sc, const df &dL) {
  const float4 r0 = rec[0], r1 = rec[1];
  const df ddx = df_sub(df{sc.x, sc.y}, df{r0.z, r0.w});
  const df ddy = df_sub(df{sc.z, sc.w}, df{r1.x, r1.y});
  const df D = df_sub(dL, df{r1.z, r1.w});
  const df rho2 = df_add(df_mul(ddx, ddx), df_mul(ddy, ddy));
  const df r = df_sqrt(df_add(rho2, df_mul(D, D)));
  const df F = (D.hi > 0.f) ? df_div(rho2, df_add(r, D)) : df_sub(r, D);
  NearGeo g;
  g.tau = df_add(df{r0.x, r0.y}, F);
  g.r = r.hi + r.lo;
  const float rinv = __frcp_rn(g.r);
  g.nx = (ddx.hi + ddx.lo) * rinv;
  g.ny = (ddy.hi + ddy.lo) * rinv;
  g.nz = (D.hi + D.lo) * rinv;
  g.omn = (F.hi + F.lo) * rinv;
  return g;
}

template <int W>
__global__ void __launch_bounds__(W * 32, 2) nadj_kernel(NearAdjParams a) {
  const FarMixedParams &p = a.f;
  if (by_transform(p)) return;  // nadj_interp_kernel's
  extern __shared__ __align__(128) unsigned char smem_raw[];
  NearAdjSmem &sm = *reinterpret_cast<NearAdjSmem *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ls = (uint32_t)(warp * 32 + lane);  // this lane's step within the item
  if (threadIdx.x == 0) {
    mbar_init(&sm.bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  const AdjGlobals G = *a.glob;
  const uint32_t nO = p.n_omega, nR = p.n_theta;
  const uint32_t nOp = (nO + kNARS - 1) / kNARS * kNARS;  // padded omega slots per point
  const uint64_t P = (uint64_t)nO * nR * p.n_phi;
  const uint64_t Pp = (uint64_t)nOp * nR * p.n_phi;
  const int64_t n_items = a.item_off[p.n_tracks];
  const df d_dw = df{G.dw_h, G.dw_l};
  const df dL = df_from_double(p.L_screen);
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
    track_segments(p, t, (uint32_t)kNASteps, (uint32_t)(item - a.item_off[t]), &seg);
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
    double gD[kNAG];
#pragma unroll
    for (int c = 0; c < kNAG; ++c) gD[c] = 0.0;

    // per (screen point, step) state, kept across constants stages
    float th = 0.f, tl = 0.f, rc = 1.f, rs = 0.f, adt = 0.f;
    float gr = 1.f, gnx = 0.f, gny = 0.f, gnz = 1.f, gomn = 0.f;
    float2 r2c = make_float2(1.f, 1.f), r2s = make_float2(0.f, 0.f), nr2s = r2s;
    int mode = 1;  // 0: every omega included, 1: none, 2: per point
    NearSums ns;
    ns.zero();

    for (uint64_t f0 = 0; f0 < Pp; f0 += kNAStage) {
      const uint32_t nf =
          (Pp - f0 < (uint64_t)kNAStage) ? (uint32_t)(Pp - f0) : (uint32_t)kNAStage;
      __syncthreads();  // the previous stage's constants are no longer read
      for (uint32_t j = threadIdx.x; j < nf / 2; j += blockDim.x) {
        const uint64_t f = f0 + 2 * j;
        const uint64_t dj = f / nOp;
        const uint32_t m = (uint32_t)(f - dj * nOp);
        float ar[2][3], ai[2][3], om[2];
        float4 wv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (m + e < nO) {
            const uint64_t gi = dj * nO + m + e;
#pragma unroll
            for (int k = 0; k < 3; ++k) ar[e][k] = ai[e][k] = 0.f;
            // U summed over the snapshots these steps enter
            for (uint32_t ks = seg.k0; ks <= seg.k1; ++ks) {
              const uint64_t ic = 2 * ((uint64_t)ks * P + gi);
              const float4 C0 = a.gcst[ic], C1 = a.gcst[ic + 1];
              if (a.linear) {  // U_k = sqrt(w) V_k
                ar[e][0] += swt * C0.x; ai[e][0] += swt * C0.y;
                ar[e][1] += swt * C0.z; ai[e][1] += swt * C0.w;
                ar[e][2] += swt * C1.x; ai[e][2] += swt * C1.y;
              } else {         // U_k = w g'_k A_k
                const uint64_t ia = 2 * (((uint64_t)t * p.n_snaps + ks) * P + gi);
                const float4 A0 = a.save_A[ia], A1 = a.save_A[ia + 1];
                ar[e][0] += wt * C0.x * A0.x; ai[e][0] += wt * C0.x * A0.y;
                ar[e][1] += wt * C0.y * A0.z; ai[e][1] += wt * C0.y * A0.w;
                ar[e][2] += wt * C0.z * A1.x; ai[e][2] += wt * C0.z * A1.y;
              }
            }
            wv[e] = a.wtab[m + e];
          } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) ar[e][k] = ai[e][k] = 0.f;
            wv[e] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
          om[e] = wv[e].z;
        }
        float4 *o = sm.cst[j];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float u0r = ar[0][k], u1r = ar[1][k];
          const float u0i = ai[0][k], u1i = ai[1][k];
          o[k] = make_float4(u0r, u1r, u0i, u1i);
          o[3 + k] = make_float4(om[0] * u0r, om[1] * u1r, -om[0] * u0i, -om[1] * u1i);
          o[6 + k] = make_float4(om[0] * om[0] * u0r, om[1] * om[1] * u1r, om[0] * om[0] * u0i,
                                 om[1] * om[1] * u1i);
        }
        o[9] = make_float4(wv[0].x, wv[0].y, wv[1].x, wv[1].y);
        o[10] = make_float4(wv[0].w, wv[1].w, 0.f, 0.f);
      }
      __syncthreads();
      float gF[kNAG];
#pragma unroll
      for (int c = 0; c < kNAG; ++c) gF[c] = 0.f;

      uint32_t d = (uint32_t)(f0 / nOp);
      for (uint64_t fd = (uint64_t)d * nOp; fd < f0 + nf; fd += nOp, ++d) {
        const uint32_t m_lo = (uint32_t)(max(fd, f0) - fd);
        const uint32_t m_hi = (uint32_t)(min(fd + nOp, f0 + nf) - fd);
        // slot m of screen point d sits at stage index fd + m - f0 >= 0 for m >= m_lo
        const int64_t seg = (int64_t)fd - (int64_t)f0;
        if (m_lo == 0) {  // a new screen point: phase, rotation and mask of step s
          const float4 sc = a.sctab[d];
          const NearGeo gs = near_geo(sm.rec[si], sc, dL);
          // the track's first step compares the whole phase omega (t + r) with zero
          float dtau = (gs.tau.hi + gs.tau.lo) + (dL.hi + dL.lo);
          if (!first) {
            const NearGeo gp = near_geo(sm.rec[si - 1], sc, dL);
            dtau = (gs.tau.hi - gp.tau.hi) + (gs.tau.lo - gp.tau.lo);
          }
          th = gs.tau.hi;
          tl = gs.tau.lo;
          gr = gs.r;
          gnx = gs.nx;
          gny = gs.ny;
          gnz = gs.nz;
          gomn = gs.omn;
          adt = fabsf(dtau);
          mode = (!valid || G.wabs_min * adt > kPiHi) ? 1 : (G.wabs_max * adt < kPiLo ? 0 : 2);
          const df rp = df_mul_raw(d_dw, gs.tau);
          sincosf(reduce_2pi(rp.hi, rp.lo), &rs, &rc);
          float c2r, s2r;
          cmul(rc, rs, rc, rs, c2r, s2r);
          r2c = make_float2(c2r, c2r);
          r2s = make_float2(s2r, s2r);
          nr2s = make_float2(-s2r, -s2r);
          ns.zero();
        }
        if (!__all_sync(0xffffffffu, mode == 1)) {
          if (G.uniform && __all_sync(0xffffffffu, mode != 2)) {
            // every point included (lanes with mode 1 are discarded below)
#pragma unroll 1
            for (uint32_t m = m_lo; m < m_hi; m += kNARS) {
              const float4 *cp = sm.cst[(seg + (int64_t)m) >> 1];
              float zs, zc;
              phasor_rev(cp[9].x, cp[9].y, th, tl, zs, zc);
              float2 zr = make_float2(zc, zc * rc - zs * rs);
              float2 zi = make_float2(zs, zc * rs + zs * rc);
#pragma unroll
              for (int q = 0; q < kNARS / 2; ++q) {
                ns.add(cp + kNAPair * q, zr, zi);
                if (q + 1 < kNARS / 2) rot2p(zr, zi, r2c, r2s, nr2s, zr, zi);
              }
            }
          } else {
            // per-point mask (and one reseed per point on a non-uniform axis)
            double P0 = 0.0, P1 = 0.0;
            bool have_p = false;
#pragma unroll 1
            for (uint32_t m = m_lo; m < m_hi; m += kNARS) {
              const float4 *cp = sm.cst[(seg + (int64_t)m) >> 1];
              float2 zr, zi;
              {
                float zs, zc;
                phasor_rev(cp[9].x, cp[9].y, th, tl, zs, zc);
                zr = make_float2(zc, zc * rc - zs * rs);
                zi = make_float2(zs, zc * rs + zs * rc);
              }
#pragma unroll 1
              for (int q = 0; q < kNARS / 2; ++q) {
                const float4 *c = cp + kNAPair * q;
                if (!G.uniform) {
                  float zs, zc;
                  phasor_rev(c[9].x, c[9].y, th, tl, zs, zc);
                  zr.x = zc;
                  zi.x = zs;
                  phasor_rev(c[9].z, c[9].w, th, tl, zs, zc);
                  zr.y = zc;
                  zi.y = zs;
                }
                const float4 aw = c[10];
                bool inc[2] = {aw.x * adt < kPiLo, aw.y * adt < kPiLo};
                if (mode == 2) {
#pragma unroll
                  for (int e = 0; e < 2; ++e) {
                    const float ph = (e ? aw.y : aw.x) * adt;
                    const uint32_t mm = m + 2 * q + e;
                    if (!inc[e] && !(ph > kPiHi) && mm < nO) {
                      if (!have_p) {
                        const uint32_t iR = d % nR, iP = d / nR;
                        P0 = p.sin_theta[iR] * p.cos_phi[iP];
                        P1 = p.sin_theta[iR] * p.sin_phi[iP];
                        have_p = true;
                      }
                      inc[e] = exact_mask_near(p, base, s, it_start, p.omega[mm], P0, P1);
                    }
                  }
                }
                const float2 gm = make_float2(inc[0] ? 1.f : 0.f, inc[1] ? 1.f : 0.f);
                ns.add(c, __fmul2_rn(zr, gm), __fmul2_rn(zi, gm));
                if (G.uniform) rot2p(zr, zi, r2c, r2s, nr2s, zr, zi);
              }
            }
          }
        }
        if (m_hi == nOp && mode != 1) {  // the screen point is complete: chain rule
          const float4 q2 = sm.rec[si][2];  // (beta_x, beta_y, beta_z, 1 - beta_z)
          float R0[3], I1[3], R2[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            R0[k] = ns.r0[k].x + ns.r0[k].y;
            I1[k] = ns.i1[k].x + ns.i1[k].y;
            R2[k] = ns.r2[k].x + ns.r2[k].y;
          }
          const float n[3] = {gnx, gny, gnz};
          const float bmn[3] = {q2.x - gnx, q2.y - gny, gomn - q2.w};  // beta - n
          const float ir = __frcp_rn(gr);
          const float ir2 = ir * ir, ir3 = ir2 * ir;
          const float nR0 = n[0] * R0[0] + n[1] * R0[1] + n[2] * R0[2];
          const float nI1 = n[0] * I1[0] + n[1] * I1[1] + n[2] * I1[2];
          const float bI1 = bmn[0] * I1[0] + bmn[1] * I1[1] + bmn[2] * I1[2];
          const float bR2 = bmn[0] * R2[0] + bmn[1] * R2[1] + bmn[2] * R2[2];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            gF[k] += (3.f * n[k] * nR0 - R0[k]) * ir3 -
                     (I1[k] + n[k] * bI1 - 2.f * n[k] * nI1) * ir2 + n[k] * bR2 * ir;
            gF[3 + k] -= I1[k] * ir;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < kNAG; ++c) gD[c] += (double)gF[c];
    }
    if (valid) {
#pragma unroll
      for (int c = 0; c < kNAG; ++c) a.gstep[(uint64_t)(base + s) * kNAG + c] = gD[c];
    }
    __syncthreads();  // records of this item no longer read
  }
}

// ------------------------------------------------------------------------
// Even omega axes: the sums over omega by transforms, as in the far-field
// adjoint (sr_far_adjoint.cu).  Nine fields per (track, screen point): conj(U_k),
// omega conj(U_k) and omega^2 conj(U_k), k = x, y, z; a cell holds the nine
// complex values and one of padding (80 bytes, five 16-byte loads), and a
// (screen point, step) takes 8 cells: bound by the 40 loads, 160 cycles per
// warp and SM.  24 tracks of 2500 to 3000 steps, 128 x 24 x 24 points, forward and
// backward: 10.6 ms walking, 3.3 with the transforms.
// ------------------------------------------------------------------------
constexpr int kNAFields = 9, kNACell = 10;  // fields; float2 per cell

__device__ __forceinline__ void near_point_u(const NearAdjParams &a, uint32_t t, uint32_t k0,
                                             uint32_t k1, uint64_t P, uint64_t gi, float wt,
                                             float swt, float (&ur)[3], float (&ui)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) ur[k] = ui[k] = 0.f;
  for (uint32_t ks = k0; ks <= k1; ++ks) {
    const uint64_t ic = 2 * ((uint64_t)ks * P + gi);
    const float4 C0 = a.gcst[ic], C1 = a.gcst[ic + 1];
    if (a.linear) {  // U_k = sqrt(w) V_k
      ur[0] += swt * C0.x; ui[0] += swt * C0.y;
      ur[1] += swt * C0.z; ui[1] += swt * C0.w;
      ur[2] += swt * C1.x; ui[2] += swt * C1.y;
    } else {         // U_k = w g'_k A_k
      const uint64_t ia = 2 * (((uint64_t)t * a.f.n_snaps + ks) * P + gi);
      const float4 A0 = a.save_A[ia], A1 = a.save_A[ia + 1];
      ur[0] += wt * C0.x * A0.x; ui[0] += wt * C0.x * A0.y;
      ur[1] += wt * C0.y * A0.z; ui[1] += wt * C0.y * A0.w;
      ur[2] += wt * C0.z * A1.x; ui[2] += wt * C0.z * A1.y;
    }
  }
}

template <int R1>
__global__ void __launch_bounds__(kFastWarps * 32, 3) nadj_fields_kernel(
    const __grid_constant__ NearAdjParams a) {
  const FarMixedParams &p = a.f;
  if (!by_transform(p)) return;
  constexpr int NF = 32 / R1, M = 32 * R1;
  __shared__ float2 tr_all[kFastWarps][32 * 33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2 *tr = tr_all[warp];
  const FastParams &f = p.fast;
  const uint32_t n_scr = p.n_theta * p.n_phi;
  const uint64_t P = (uint64_t)p.n_omega * n_scr;
  uint64_t task = (uint64_t)blockIdx.x * kFastWarps + warp;
  const uint32_t band = (uint32_t)(task % f.n_bands);
  task /= f.n_bands;
  const uint32_t d = (uint32_t)(task % n_scr);
  task /= n_scr;
  const uint32_t k0 = (uint32_t)(task % p.n_snaps), t = a.t_lo + (uint32_t)(task / p.n_snaps);
  if (t >= a.t_hi) return;
  const uint32_t k1 = last_fired(p, t);
  if (k1 == 0xffffffffu || k0 > k1) return;
  const uint32_t j0 = band * f.nb;
  const int nb = (int)min(f.nb, p.n_omega - j0);
  const float wt = (float)p.weight[t], swt = (float)sqrt(p.weight[t]);
#pragma unroll 1
  for (int f0 = 0; f0 < kNAFields; f0 += NF) {
    float2 x[NF][R1], y[32];
#pragma unroll
    for (int i = 0; i < R1; ++i) {
      const int n = 32 * i + lane;                        // frequency index mod M
      const int j = (n < M / 2 ? n : n - M) + nb / 2;
      float ur[3] = {0.f, 0.f, 0.f}, ui[3] = {0.f, 0.f, 0.f}, dv = 0.f, w = 0.f;
      if (j >= 0 && j < nb) {
        near_point_u(a, t, k0, k1, P, (uint64_t)d * p.n_omega + j0 + j, wt, swt, ur, ui);
        dv = (float)f.deconv[j - nb / 2 + kFastMaxBand / 2];
        w = a.wtab[j0 + j].z;
      }
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        const int fq = f0 + q, c = fq % 3, e = fq / 3;    // component, power of omega
        const float g = dv * (e == 0 ? 1.f : e == 1 ? w : w * w);
        const float re = c == 0 ? ur[0] : c == 1 ? ur[1] : ur[2];
        const float im = c == 0 ? ui[0] : c == 1 ? ui[1] : ui[2];
        x[q][i] = make_float2(re * g, -im * g);
      }
    }
    fft_fields<R1, NF>(x, y, tr, f.twiddle, lane);
    const int q = lane / R1, al = lane % R1, fq = f0 + q;
    if (fq < kNAFields) {
      float2 *o = a.fields +
                  ((((uint64_t)(t - a.t_lo) * p.n_snaps + k0) * n_scr + d) * f.n_bands + band) *
                      ((uint64_t)kNACell * (M + kTaps)) + fq;
#pragma unroll
      for (int b = 0; b < 32; ++b) o[kNACell * (al + R1 * b)] = y[bitrev<32>(b)];
      // the circle's first cells once more behind its last
#pragma unroll
      for (int b = 0; b * R1 < kTaps; ++b)
        if (al + R1 * b < kTaps) o[kNACell * (M + al + R1 * b)] = y[bitrev<32>(b)];
    }
    __syncwarp();
  }
}

// WALK: as in the far field.
template <bool WALK>
__global__ void __launch_bounds__(kNASteps, 2) nadj_interp_kernel(
    const __grid_constant__ NearAdjParams a) {
  const FarMixedParams &p = a.f;
  if (!by_transform(p) || (*a.many_cut != 0u) != WALK) return;
  const FastParams &f = p.fast;
  __shared__ float4 cut_u[WALK ? kNAW : 1][32][2];  // U and omega of 32 frequencies, for cut steps
  const int lane = threadIdx.x & 31;
  const uint32_t nR = p.n_theta, n_scr = nR * p.n_phi;
  const uint64_t P = (uint64_t)p.n_omega * n_scr;
  const AdjGlobals G = *a.glob;
  const df dL = df_from_double(p.L_screen);
  const int M = (int)f.M;
  const float Mf = (float)M;
  const double dw = (p.omega[p.n_omega - 1] - p.omega[0]) / (double)(p.n_omega - 1);
  const df f_d = df_from_double(dw * 0.15915494309189533577);
  const int64_t i_lo = a.item_off[a.t_lo], i_hi = a.item_off[a.t_hi];
  const int64_t n_items = (i_hi - i_lo) * a.n_split;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int64_t it = i_lo + item / a.n_split;
    const uint32_t split = (uint32_t)(item % a.n_split);
    const uint32_t dA = (uint32_t)((uint64_t)n_scr * split / a.n_split);
    const uint32_t dB = (uint32_t)((uint64_t)n_scr * (split + 1) / a.n_split);
    uint32_t lo = a.t_lo, hi = a.t_hi;  // last track with item_off[t] <= it
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (a.item_off[mid] <= it) lo = mid; else hi = mid;
    }
    const uint32_t t = lo;
    const int64_t base = p.offsets[t];
    SnapSegment seg{0, 0, 0, 0};
    track_segments(p, t, (uint32_t)kNASteps, (uint32_t)(it - a.item_off[t]), &seg);
    const uint32_t s = seg.r0 + threadIdx.x;
    const bool valid = s < seg.r1;
    if (!__any_sync(0xffffffffu, valid)) continue;  // whole warps
    const uint32_t sc = valid ? s : seg.r1 - 1;
    const uint32_t it_start = p.it_start[t];
    const float wt = (float)p.weight[t], swt = (float)sqrt(p.weight[t]);
    const float4 *rp = p.records + (base + sc) * kRecF4;
    const float4 rec[3] = {__ldg(rp), __ldg(rp + 1), __ldg(rp + 2)};
    // differences to the step before, for the quick test of the mask
    float dq = 0.f, dz = 0.f, dx = 0.f, dy = 0.f, d2 = 0.f;
    if (sc > 0) {
      const float4 e0 = __ldg(rp - kRecF4), e1 = __ldg(rp - kRecF4 + 1);
      dq = (rec[0].x - e0.x) + (rec[0].y - e0.y);
      dx = (rec[0].z - e0.z) + (rec[0].w - e0.w);
      dy = (rec[1].x - e1.x) + (rec[1].y - e1.y);
      dz = (rec[1].z - e1.z) + (rec[1].w - e1.w);
      d2 = dx * dx + dy * dy + dz * dz;
    }
    double gD[kNAG];
    float gF[kNAG];
#pragma unroll
    for (int c = 0; c < kNAG; ++c) {
      gD[c] = 0.0;
      gF[c] = 0.f;
    }
    const float2 *fld = a.fields + (((uint64_t)(t - a.t_lo) * p.n_snaps + seg.k0) * n_scr) *
                                       f.n_bands * ((uint64_t)kNACell * (M + kTaps));
#pragma unroll 1
    for (uint32_t d = dA; d < dB; ++d) {
      const float4 scr = __ldg(a.sctab + d);
      const NearGeo g = near_geo(rec, scr, dL);
      const float ir = __frcp_rn(g.r);
      int mode = valid ? 0 : 1;  // 0: every frequency enters, 1: none, 2: some
      float R0[3] = {0.f, 0.f, 0.f}, I1[3] = {0.f, 0.f, 0.f}, R2[3] = {0.f, 0.f, 0.f};
      // mask: certain where the FP32 difference (first order in the step, with
      // the second as a bound) leaves a 1e-3 margin, else from the double-float
      // times of both steps
      const float quick =
          sc > 0 ? fabsf(dq + g.omn * dz - g.nx * dx - g.ny * dy) + d2 * ir : INFINITY;
      if (__any_sync(0xffffffffu, valid && !(G.wabs_max * quick < 0.999f * kPiLo))) {
        // the track's first step compares the whole phase omega (t + r) with zero
        float dt0 = (g.tau.hi + g.tau.lo) + (dL.hi + dL.lo);
        if (sc > 0) {
          const float4 prev[3] = {__ldg(rp - kRecF4), __ldg(rp - kRecF4 + 1),
                                  __ldg(rp - kRecF4 + 2)};
          const NearGeo gp = near_geo(prev, scr, dL);
          dt0 = (g.tau.hi - gp.tau.hi) + (g.tau.lo - gp.tau.lo);
        }
        const float adt = fabsf(dt0);
        if (valid) mode = G.wabs_max * adt < kPiLo ? 0 : (G.wabs_min * adt > kPiHi ? 1 : 2);
        // cut steps: many of them by a walk of each lane along its own included
        // frequencies, few one after the other, the warp's lanes along them (20 tracks
        // of 1500 steps, 5 a period, 16 x 16 points, 16 / 64 / 128 frequencies: walked
        // 0.71 / 1.07 / 1.54 ms, one after the other 1.40 / 1.64 / 2.23; without the
        // transforms 0.86 / 2.12 / 3.79)
        const uint32_t mine =
            mode == 2 ? cut_interval<true>(p, 0, (int)p.n_omega, G.w0f, G.dwf, d, base, s,
                                           it_start, adt)
                      : 1u;
        uint32_t cut = __ballot_sync(0xffffffffu, mode == 2);
        if (WALK && walk_cut(cut, p.n_omega, 70u, 38u)) {
          cut = 0u;
          const int jf = (int)(mine & 0xffffu), jl = (int)(mine >> 16);
          int first, last;
          cut_span(mode == 2, mine, first, last);
          float4 (*su)[2] = cut_u[threadIdx.x >> 5];
          float rs, rc, v0[3] = {0.f, 0.f, 0.f}, v1[3] = {0.f, 0.f, 0.f}, v2[3] = {0.f, 0.f, 0.f};
          phasor_rev(f_d.hi, f_d.lo, g.tau.hi, g.tau.lo, rs, rc);
#pragma unroll 1
          for (int j0 = first & ~31; j0 <= last; j0 += 32) {
            float ur[3] = {0.f, 0.f, 0.f}, ui[3] = {0.f, 0.f, 0.f}, w = 0.f;
            if (j0 + lane <= last) {
              near_point_u(a, t, seg.k0, seg.k1, P, (uint64_t)d * p.n_omega + j0 + lane, wt, swt,
                           ur, ui);
              w = a.wtab[j0 + lane].z;
            }
            __syncwarp();
            su[lane][0] = make_float4(ur[0], ui[0], ur[1], ui[1]);
            su[lane][1] = make_float4(ur[2], ui[2], w, w * w);
            __syncwarp();
#pragma unroll 1
            for (int j8 = j0; j8 < j0 + 32 && j8 <= last; j8 += 8) {
              const float4 w8 = __ldg(a.wtab + j8);
              float zs, zc;
              phasor_rev(w8.x, w8.y, g.tau.hi, g.tau.lo, zs, zc);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 q0 = su[j8 - j0 + i][0];
                const float4 q1 = su[j8 - j0 + i][1];
                const bool in = j8 + i >= jf && j8 + i <= jl;
                const float c = in ? zc : 0.f, s1 = in ? zs : 0.f;
                const float wc = q1.z * c, ws = q1.z * s1;
                const float ar[3] = {q0.x, q0.z, q1.x}, ai[3] = {q0.y, q0.w, q1.y};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                  const float re = ar[k] * c + ai[k] * s1;
                  v0[k] += re;
                  v1[k] = __fmaf_rn(ar[k], ws, __fmaf_rn(-ai[k], wc, v1[k]));
                  v2[k] = __fmaf_rn(q1.w, re, v2[k]);
                }
                const float q = zc * rc - zs * rs;
                zs = zc * rs + zs * rc;
                zc = q;
              }
            }
          }
          if (mode == 2) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              R0[k] = v0[k];
              I1[k] = v1[k];
              R2[k] = v2[k];
            }
          }
        }
        for (; cut; cut &= cut - 1) {
          const int b = __ffs(cut) - 1;
          const uint32_t r = __shfl_sync(0xffffffffu, mine, b);
          const float th = __shfl_sync(0xffffffffu, g.tau.hi, b);
          const float tl = __shfl_sync(0xffffffffu, g.tau.lo, b);
          const int jf = (int)(r & 0xffffu), jl = (int)(r >> 16);
          float v[9];
#pragma unroll
          for (int k = 0; k < 9; ++k) v[k] = 0.f;
          for (int j = jf + lane; j <= jl; j += 32) {
            float ur[3], ui[3];
            near_point_u(a, t, seg.k0, seg.k1, P, (uint64_t)d * p.n_omega + j, wt, swt, ur, ui);
            const float4 w = a.wtab[j];
            float zs, zc;
            phasor_rev(w.x, w.y, th, tl, zs, zc);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const float re = ur[k] * zc + ui[k] * zs;
              v[k] += re;
              v[3 + k] += w.z * (ur[k] * zs - ui[k] * zc);
              v[6 + k] += w.z * w.z * re;
            }
          }
#pragma unroll
          for (int k = 0; k < 9; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
          }
          if (lane == b) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              R0[k] = v[k];
              I1[k] = v[3 + k];
              R2[k] = v[6 + k];
            }
          }
        }
      }
      if (mode == 0) {
        const float pr = f_d.hi * g.tau.hi;
        float e = __fmaf_rn(f_d.hi, g.tau.hi, -pr);
        e = __fmaf_rn(f_d.hi, g.tau.lo, e);
        e = __fmaf_rn(f_d.lo, g.tau.hi, e);
        const float uh = (pr - rintf(pr)) * Mf, ul = e * Mf;
        const float rm = rintf((uh - 0.5f) + ul);
        float wk[kTaps];
        kb_taps(((uh - rm) - 0.5f) + ul, wk);
        const int m = ((int)rm - 3) & (M - 1);
        for (uint32_t band = 0; band < f.n_bands; ++band) {
          const float4 *cell = reinterpret_cast<const float4 *>(
              fld + ((uint64_t)d * f.n_bands + band) * ((uint64_t)kNACell * (M + kTaps)) +
              kNACell * m);
          float2 h[kNACell];
#pragma unroll
          for (int k = 0; k < kNACell; ++k) h[k] = make_float2(0.f, 0.f);
#pragma unroll
          for (int l = 0; l < kTaps; ++l) {
            const float2 ww = make_float2(wk[l], wk[l]);
#pragma unroll
            for (int k = 0; k < kNACell / 2; ++k) {
              const float4 v = __ldg(cell + (kNACell / 2) * l + k);
              h[2 * k] = __ffma2_rn(ww, make_float2(v.x, v.y), h[2 * k]);
              if (2 * k + 1 < kNAFields)
                h[2 * k + 1] = __ffma2_rn(ww, make_float2(v.z, v.w), h[2 * k + 1]);
            }
          }
          const float4 fc = __ldg(a.bandtab + band);  // its centre frequency / 2 pi
          float zs, zc;
          phasor_exact(fc.x, fc.y, g.tau.hi, g.tau.lo, zs, zc);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            R0[k] += h[k].x * zc - h[k].y * zs;
            I1[k] += h[3 + k].x * zs + h[3 + k].y * zc;
            R2[k] += h[6 + k].x * zc - h[6 + k].y * zs;
          }
        }
      }
      if (mode != 1) {  // the chain rule
        const float n[3] = {g.nx, g.ny, g.nz};
        const float bmn[3] = {rec[2].x - g.nx, rec[2].y - g.ny, g.omn - rec[2].w};  // beta - n
        const float ir2 = ir * ir, ir3 = ir2 * ir;
        const float nR0 = n[0] * R0[0] + n[1] * R0[1] + n[2] * R0[2];
        const float nI1 = n[0] * I1[0] + n[1] * I1[1] + n[2] * I1[2];
        const float bI1 = bmn[0] * I1[0] + bmn[1] * I1[1] + bmn[2] * I1[2];
        const float bR2 = bmn[0] * R2[0] + bmn[1] * R2[1] + bmn[2] * R2[2];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          gF[k] += (3.f * n[k] * nR0 - R0[k]) * ir3 -
                   (I1[k] + n[k] * bI1 - 2.f * n[k] * nI1) * ir2 + n[k] * bR2 * ir;
          gF[3 + k] -= I1[k] * ir;
        }
      }
      if (((d - dA) & 31u) == 31u || d + 1 == dB) {  // FP32 over 32 points, then FP64
#pragma unroll
        for (int c = 0; c < kNAG; ++c) {
          gD[c] += (double)gF[c];
          gF[c] = 0.f;
        }
      }
    }
    if (valid) {
#pragma unroll
      for (int c = 0; c < kNAG; ++c)
        a.gstep[((uint64_t)split * p.total_steps + base + s) * kNAG + c] = gD[c];
    }
  }
}

void launch_nadj_fields(const NearAdjParams &a, uint64_t n_scr, cudaStream_t s) {
  const uint64_t warps =
      (uint64_t)(a.t_hi - a.t_lo) * a.f.n_snaps * n_scr * a.f.fast.n_bands;
  const unsigned blocks = (unsigned)((warps + kFastWarps - 1) / kFastWarps);
  switch (a.f.fast.M) {
    case 128: nadj_fields_kernel<4><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    case 256: nadj_fields_kernel<8><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    case 512: nadj_fields_kernel<16><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
    default: nadj_fields_kernel<32><<<blocks, kFastWarps * 32, 0, s>>>(a); break;
  }
}

size_t nadj_smem_bytes() { return sizeof(NearAdjSmem); }

struct NearAdjLayout {
  size_t records, gcst, wtab, sctab, glob, item_off, gstep, wpart, tables, bandtab, fields, total;
  uint32_t w_chunks;
  AdjFields fl;
};

NearAdjLayout nadj_layout(int64_t total_steps, uint64_t P, uint32_t n_omega, uint64_t n_scr,
                          uint32_t n_tracks, uint32_t n_snaps, bool least) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  NearAdjLayout l;
  l.w_chunks = adj_weight_chunks(P, n_tracks, device_sm_count());
  l.fl = adj_fields_layout(total_steps, n_omega, n_scr, n_tracks, n_snaps, kNACell * 8, kNASteps,
                           least);
  l.gstep = 256;
  l.records = l.gstep + up((size_t)total_steps * kNAG * 8 * l.fl.n_split);
  l.gcst = l.records + up((size_t)total_steps * kRecBytes);
  l.wtab = l.gcst + up((size_t)P * 32 * (n_snaps ? n_snaps : 1));
  l.sctab = l.wtab + up((size_t)n_omega * 16);
  l.glob = l.sctab + up((size_t)n_scr * 16);
  l.item_off = l.glob + 256;
  l.wpart = l.item_off + up(((size_t)n_tracks + 1) * 8);
  l.tables = l.wpart + up((size_t)n_tracks * l.w_chunks * 8);
  l.bandtab = l.tables + up(kFastTables);
  l.fields = l.bandtab + up((size_t)l.fl.n_bands * 16);
  l.total = l.fields + l.fl.bytes;
  return l;
}

int check_near_adjoint_args(const sr_tracks *t, const sr_grid *g, void *const *out,
                            int comp = SR_COMP_TOTAL) {
  int rc = validate_spectrum_args(t, g, comp, SR_PREC_MIXED, out);
  if (rc) return rc;
  if (g->mode != SR_MODE_NEAR) return fail(SR_ERR_UNSUPPORTED, "near-field adjoint: mode near");
  if (t->n_snaps < 1)
    return fail(SR_ERR_UNSUPPORTED, "the adjoint needs at least one snapshot (n_snaps >= 1)");
  return SR_OK;
}

}  // namespace
}  // namespace sr

using namespace sr;

extern "C" int sr_near_forward_saved(const sr_tracks *t, const sr_grid *g, int comp,
                                     void *const *out, float *saved_A, void *workspace,
                                     size_t workspace_bytes, void *stream) {
  clear_error();
  int rc = check_near_adjoint_args(t, g, out, comp);
  if (rc) return rc;
  if (!saved_A) return fail(SR_ERR_INVALID, "saved_A is NULL");
  const uint64_t P = (uint64_t)g->n_omega * g->n_theta * g->n_phi;
  if (P == 0 || t->n_tracks == 0) return SR_OK;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(saved_A, 0, (size_t)t->n_tracks * t->n_snaps * P * 32, s);
  if (e != cudaSuccess) return cuda_fail(e, "saved_A reset");
  FarMixedParams p = make_far_mixed_params(t, g, comp, out);
  p.save_A = saved_A;
  return launch_near_mixed(p, mixed_config(t, g, comp), workspace, workspace_bytes, s);
}

extern "C" int sr_near_total_forward_saved(const sr_tracks *t, const sr_grid *g, double *spectrum,
                                           float *saved_A, void *workspace,
                                           size_t workspace_bytes, void *stream) {
  void *out[6] = {spectrum};
  return sr_near_forward_saved(t, g, SR_COMP_TOTAL, out, saved_A, workspace, workspace_bytes,
                               stream);
}

extern "C" int64_t sr_near_total_backward_workspace_bytes(const sr_tracks *t, const sr_grid *g) {
  return sr_near_backward_workspace_bytes(t, g);
}

namespace {
int64_t backward_bytes(const sr_tracks *t, const sr_grid *g, bool least) {
  if (!t || !g) return -1;
  const uint64_t n_scr = (uint64_t)g->n_theta * g->n_phi;
  return (int64_t)nadj_layout(t->total_steps, n_scr * g->n_omega, g->n_omega, n_scr,
                              t->n_tracks, t->n_snaps, least)
      .total;
}
}  // namespace

extern "C" int64_t sr_near_backward_workspace_bytes(const sr_tracks *t, const sr_grid *g) {
  return backward_bytes(t, g, false);
}

extern "C" int64_t sr_near_backward_workspace_bytes_min(const sr_tracks *t, const sr_grid *g) {
  return backward_bytes(t, g, true);
}

extern "C" int sr_near_total_backward(const sr_tracks *t, const sr_grid *g,
                                      const double *grad_spectrum, const float *saved_A,
                                      double *const *grad_track, double *grad_weight,
                                      void *workspace, size_t workspace_bytes, void *stream) {
  const double *grad_out[6] = {grad_spectrum};
  return sr_near_backward(t, g, SR_COMP_TOTAL, grad_out, saved_A, grad_track, grad_weight,
                          workspace, workspace_bytes, stream);
}

extern "C" int sr_near_backward(const sr_tracks *t, const sr_grid *g, int comp,
                                const double *const *grad_out, const float *saved_A,
                                double *const *grad_track, double *grad_weight, void *workspace,
                                size_t workspace_bytes, void *stream) {
  clear_error();
  if (!grad_out) return fail(SR_ERR_INVALID, "grad_out must not be NULL");
  int rc = check_near_adjoint_args(t, g, (void *const *)grad_out, comp);
  if (rc) return rc;
  if (!saved_A || !grad_track || !grad_weight)
    return fail(SR_ERR_INVALID, "saved_A, grad_track and grad_weight must not be NULL");
  for (int i = 0; i < 6; ++i)
    if (!grad_track[i]) return fail(SR_ERR_INVALID, "grad_track[%d] is NULL", i);
  if (t->n_tracks == 0) return SR_OK;
  const uint64_t n_scr = (uint64_t)g->n_theta * g->n_phi;
  const uint64_t P = n_scr * g->n_omega;
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
  NearAdjLayout lay = nadj_layout(t->total_steps, P, g->n_omega, n_scr, t->n_tracks, t->n_snaps, false);
  if (workspace_bytes < lay.total)
    lay = nadj_layout(t->total_steps, P, g->n_omega, n_scr, t->n_tracks, t->n_snaps, true);
  if (!workspace || workspace_bytes < lay.total)
    return fail(SR_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", lay.total,
                workspace_bytes);
  if (((uintptr_t)workspace & 255u) != 0)
    return fail(SR_ERR_WORKSPACE, "workspace not 256-byte aligned");
  unsigned char *w = (unsigned char *)workspace;

  NearAdjParams a;
  memset(&a, 0, sizeof(a));
  a.f = make_far_mixed_params(t, g, comp, (void *const *)grad_out);
  a.f.status = (int *)w;
  a.f.records = (float4 *)(w + lay.records);
  for (int i = 0; i < n_outputs(comp); ++i) a.grad_out[i] = grad_out[i];
  a.linear = comp == SR_COMP_CARTESIAN_COMPLEX ? 1 : 0;
  a.save_A = (const float4 *)saved_A;
  a.gcst = (float4 *)(w + lay.gcst);
  a.wtab = (float4 *)(w + lay.wtab);
  a.sctab = (float4 *)(w + lay.sctab);
  a.glob = (AdjGlobals *)(w + lay.glob);
  a.item_off = (int64_t *)(w + lay.item_off);
  a.gstep = (double *)(w + lay.gstep);
  for (int i = 0; i < 6; ++i) a.grad[i] = grad_track[i];
  a.grad_w = grad_weight;
  a.n_split = lay.fl.n_split;
  a.many_cut = (unsigned int *)(w + 96);  // in the zeroed status block
  a.bandtab = (float4 *)(w + lay.bandtab);
  a.fields = (float2 *)(w + lay.fields);
  if (lay.fl.batch)
    fast_tables_bind(a.f, lay.fl.n_bands, lay.fl.nb, lay.fl.M, w + lay.tables, w);

  // the status block and, behind it, the per-step gradients: steps that enter
  // no snapshot (after the last one written) are not visited
  e = cudaMemsetAsync(w, 0, lay.records, s);
  if (e != cudaSuccess) return cuda_fail(e, "status reset");
  const int n_sm = device_sm_count();
  const int64_t step_blocks = std::max<int64_t>(
      16, std::min<int64_t>((t->total_steps + 255) / 256, (int64_t)n_sm * 128));
  if (t->total_steps > 0) launch_near_prepass(a.f, (int)step_blocks, s);
  adj_setup_kernel<true><<<3, 1024, 0, s>>>(a.f, a.wtab, a.glob, a.item_off, (uint32_t)kNASteps,
                                       a.many_cut);
  {
    const uint64_t work = std::max<uint64_t>(P, n_scr);
    const uint64_t nb = std::min<uint64_t>((work + 255) / 256, (uint64_t)n_sm * 64);
    nadj_prep_kernel<<<(unsigned)nb, 256, 0, s>>>(a);
  }
  a.wpart = (double *)(w + lay.wpart);
  a.w_chunks = lay.w_chunks;
  nadj_weight_partial_kernel<<<t->n_tracks * lay.w_chunks, kWeightThreads, 0, s>>>(
      a, P, lay.w_chunks, a.wpart);
  rc = cuda_fail(cudaGetLastError(), "near adjoint prep launch");
  if (rc) return rc;
  const size_t smem = nadj_smem_bytes();
  e = allow_smem((const void *)nadj_kernel<kNAW>, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "near adjoint smem attribute");
  const int64_t items_max = t->total_steps / kNASteps + (int64_t)t->n_tracks * t->n_snaps;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(items_max, 2 * (int64_t)n_sm));
  void *tok = nullptr;
  timing_record(s, true, &tok);
  for (uint32_t lo = 0; lay.fl.batch && lo < t->n_tracks; lo += lay.fl.batch) {
    a.t_lo = lo;
    a.t_hi = std::min(t->n_tracks, lo + lay.fl.batch);
    launch_nadj_fields(a, n_scr, s);
    const int64_t most = items_max * lay.fl.n_split;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(most, 2 * (int64_t)n_sm));
    nadj_interp_kernel<false><<<blocks, kNASteps, 0, s>>>(a);
    nadj_interp_kernel<true><<<blocks, kNASteps, 0, s>>>(a);
  }
  nadj_kernel<kNAW><<<grid, kNAW * 32, smem, s>>>(a);
  timing_record(s, false, &tok);
  rc = cuda_fail(cudaGetLastError(), "near adjoint kernel launch");
  if (rc) return rc;
  if (a.f.track_f32)
    nadj_final_kernel<float><<<(int)step_blocks, 256, 0, s>>>(a);
  else
    nadj_final_kernel<double><<<(int)step_blocks, 256, 0, s>>>(a);
  return cuda_fail(cudaGetLastError(), "near adjoint final launch");
}
