// Pieces shared by the far- and near-field adjoint kernels.
#pragma once

#include <algorithm>

#include "sr_common.cuh"
#include "sr_internal.h"
#include "sr_fast_sum.cuh"
#include "sr_mixed_common.cuh"

namespace sr {
namespace {

struct AdjGlobals {
  float dw_h, dw_l;        // omega spacing (rad per unit time) as a double-float
  float w0f, dwf;          // first omega and spacing in FP32
  float wabs_min, wabs_max;
  int uniform;             // omega axis uniform to 1e-12
  float sin_max, omc_max;  // far field: largest |sin(theta)|, 1 - cos(theta)
};

// Omega table, axis uniformity and |omega| range (one block).
__device__ __forceinline__ void adj_globals(const FarMixedParams &p, float4 *wtab,
                                            AdjGlobals *glob) {
  const uint32_t nO = p.n_omega;
  const double w0 = p.omega[0];
  const double dw = (nO > 1) ? (p.omega[nO - 1] - w0) / (double)(nO - 1) : 0.0;
  bool uni = true;
  float amin = 3.0e38f, amax = 0.f;
  for (uint32_t m = threadIdx.x; m < nO; m += blockDim.x) {
    const double wm = p.omega[m];
    if (fabs(wm - (w0 + (double)m * dw)) > 1e-12 * fabs(wm) + 1e-300) uni = false;
    const df r = df_from_double(wm * 0.15915494309189533577);
    const float aw = (float)fabs(wm);
    wtab[m] = make_float4(r.hi, r.lo, (float)wm, aw);
    amin = fminf(amin, aw);
    amax = fmaxf(amax, aw);
  }
  __shared__ float smin[1024], smax[1024];
  __shared__ unsigned int angle[2];
  if (threadIdx.x < 2u) angle[threadIdx.x] = 0u;
  smin[threadIdx.x] = amin;
  smax[threadIdx.x] = amax;
  const int all_uni = __syncthreads_and(uni ? 1 : 0);
  if (p.cos_theta != nullptr)  // not negative: ordered as integers, a NaN largest
    for (uint32_t i = threadIdx.x; i < p.n_theta; i += blockDim.x) {
      atomicMax(&angle[0], __float_as_uint(fabsf((float)p.sin_theta[i])));
      atomicMax(&angle[1], __float_as_uint(fabsf((float)(1.0 - p.cos_theta[i]))));
    }
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      smin[threadIdx.x] = fminf(smin[threadIdx.x], smin[threadIdx.x + o]);
      smax[threadIdx.x] = fmaxf(smax[threadIdx.x], smax[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    AdjGlobals g;
    const df d = df_from_double(dw);
    g.dw_h = d.hi;
    g.dw_l = d.lo;
    g.w0f = (float)w0;
    g.dwf = (float)dw;
    g.wabs_min = smin[0];
    g.wabs_max = smax[0];
    g.uniform = all_uni;
    g.sin_max = __uint_as_float(angle[0]);
    g.omc_max = __uint_as_float(angle[1]);
    *glob = g;
  }
}

// Snapshot segments of a track.  The forward writes snapshot k after step
// f_k (the reference's state machine, SnapState); the snapshots that fire form
// a run k_first .. k_last with increasing f_k, a step s enters every fired
// snapshot with f_k >= s, and steps after the last fired one enter none.  So
// the body steps fall into segments, segment i holding the steps after
// f_{k_first + i - 1} up to f_{k_first + i}, each entering snapshots
// k_first + i .. k_last.  Work items never cross a segment; a segment of n
// steps makes ceil(n / per_item) items.
struct SnapSegment {
  uint32_t r0, r1;  // steps [r0, r1) of the item
  uint32_t k0, k1;  // snapshots k0 .. k1 (inclusive) receive them
};

__device__ __forceinline__ uint32_t last_fired(const FarMixedParams &p, uint32_t t) {
  SnapState st;
  const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
  st.init(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  uint32_t last = 0xffffffffu;
  while (st.fire_it != SnapState::NEVER) {
    last = st.k;
    st.advance(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  }
  return last;
}

// Items of track t (count == nullptr) or the j-th of them (into *seg).
__device__ __forceinline__ uint32_t track_segments(const FarMixedParams &p, uint32_t t,
                                                   uint32_t per_item, uint32_t j,
                                                   SnapSegment *seg) {
  const uint32_t n_body = track_body(p, t);
  if (n_body == 0) return 0;
  const uint32_t k_last = last_fired(p, t);
  if (k_last == 0xffffffffu) return 0;  // no snapshot fires: nothing to differentiate
  SnapState st;
  const uint32_t *snaps = p.snap_its + (size_t)t * p.snap_stride;
  st.init(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  uint32_t lo = 0, items = 0;
  while (st.fire_it != SnapState::NEVER && lo < n_body) {
    const int64_t last_body = (int64_t)n_body - 1;
    const uint32_t hi = (uint32_t)(st.fire_it < last_body ? st.fire_it : last_body);  // inclusive
    if (hi >= lo) {
      const uint32_t n = (hi - lo + per_item) / per_item;
      if (seg != nullptr && j < items + n) {
        seg->r0 = lo + (j - items) * per_item;
        seg->r1 = min(hi + 1, seg->r0 + per_item);
        seg->k0 = st.k;
        seg->k1 = k_last;
        return items + n;
      }
      items += n;
      lo = hi + 1;
    }
    st.advance(p.it_start[t], p.it_end[t], snaps, p.n_snaps);
  }
  return items;
}

// Work items per track (snapshot segments cut into runs of steps_per_item),
// as an exclusive prefix (one block of 1024 threads, each scanning a
// contiguous run of tracks).
__device__ __forceinline__ void adj_items(const FarMixedParams &p, int64_t *item_off,
                                          uint32_t steps_per_item) {
  const uint32_t n = p.n_tracks;
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t t0 = min(n, threadIdx.x * per), t1 = min(n, t0 + per);
  int64_t local = 0;
  for (uint32_t t = t0; t < t1; ++t) local += track_segments(p, t, steps_per_item, 0, nullptr);
  __shared__ int64_t sums[1024];
  sums[threadIdx.x] = local;
  __syncthreads();
  for (uint32_t off = 1; off < blockDim.x; off <<= 1) {
    const int64_t v = threadIdx.x >= off ? sums[threadIdx.x - off] : 0;
    __syncthreads();
    sums[threadIdx.x] += v;
    __syncthreads();
  }
  int64_t run = threadIdx.x ? sums[threadIdx.x - 1] : 0;
  for (uint32_t t = t0; t < t1; ++t) {
    item_off[t] = run;
    run += track_segments(p, t, steps_per_item, 0, nullptr);
  }
  if (threadIdx.x == blockDim.x - 1) item_off[n] = sums[blockDim.x - 1];
}

// Whether the phase limit cuts the axis inside at the i-th of kCutSamples
// (direction, step) pairs, spread over the tracks (to FP32: for the choice of a
// kernel only).
constexpr uint32_t kCutSamples = 128;
template <bool NEAR>
__device__ __forceinline__ bool sampled_cut(const FarMixedParams &p, uint32_t i) {
  if (i >= kCutSamples) return false;
  const uint32_t t = (uint32_t)((uint64_t)i * p.n_tracks / kCutSamples), nT = p.n_theta;
  const uint32_t n = track_body(p, t);
  if (n < 2u) return false;
  const uint32_t s = 1u + (i * 2654435761u >> 8) % (n - 1u), d = (i * 40503u) % (nT * p.n_phi);
  const uint32_t iT = d % nT, iP = d / nT;
  const float c0 = (float)(p.sin_theta[iT] * p.cos_phi[iP]);
  const float c1 = (float)(p.sin_theta[iT] * p.sin_phi[iP]);
  const int64_t g = p.offsets[t] + s;
  auto ld = [&](const void *a, int64_t k) {
    return p.track_f32 ? (double)((const float *)a)[k] : ((const double *)a)[k];
  };
  const double z = ld(p.z, g), dzd = z - ld(p.z, g - 1);
  const float x = (float)ld(p.x, g), y = (float)ld(p.y, g), dz = (float)dzd;
  const float dx = x - (float)ld(p.x, g - 1), dy = y - (float)ld(p.y, g - 1);
  float nx = c0, ny = c1, omn;  // direction to the observer, 1 - n_z
  if (NEAR) {
    const float rx = c0 - x, ry = c1 - y, D = (float)(p.L_screen - z);
    const float rho2 = rx * rx + ry * ry, r = sqrtf(rho2 + D * D);
    nx = rx / r;
    ny = ry / r;
    omn = rho2 / (r * (r + D));
  } else {
    omn = (float)(1.0 - p.cos_theta[iT]);
  }
  const float adt = fabsf((float)(p.dt - dzd) + omn * dz - nx * dx - ny * dy);
  const double wa = p.omega[0], wb = p.omega[p.n_omega - 1u];
  const float wmin = (wa <= 0.0) != (wb <= 0.0) ? 0.f : (float)fmin(fabs(wa), fabs(wb));
  return !((float)fmax(fabs(wa), fabs(wb)) * adt < kPiLo) && !(wmin * adt > kPiHi);
}

// Sets *many where the phase limit cuts more than 1/32 of 128 sampled
// (direction, step) pairs.
template <bool NEAR>
__device__ __forceinline__ void adj_cut_share(const FarMixedParams &p, unsigned int *many) {
  const int cut = __syncthreads_count(sampled_cut<NEAR>(p, threadIdx.x));
  if (32 * cut > (int)kCutSamples && threadIdx.x == 0) *many = 1u;
}

// The one-block preparations in one launch (three blocks of 1024 threads).
template <bool NEAR>
__global__ void adj_setup_kernel(FarMixedParams p, float4 *wtab, AdjGlobals *glob,
                                 int64_t *item_off, uint32_t steps_per_item, unsigned int *many) {
  if (blockIdx.x == 0)
    adj_globals(p, wtab, glob);
  else if (blockIdx.x == 1)
    adj_items(p, item_off, steps_per_item);
  else if (p.fast.M != 0u)
    adj_cut_share<NEAR>(p, many);
}

// Weight gradients are summed in two fixed-order stages: block (t, b) sums
// chunk b of track t's points into wpart[t][b] by a fixed tree, then one
// thread of the last launch per track adds its chunks in order
// (sr_far_adjoint.cu, sr_near_adjoint.cu).
constexpr int kWeightThreads = 256;

inline uint32_t adj_weight_chunks(uint64_t P, uint32_t n_tracks, int n_sm) {
  uint64_t c = (4ull * (uint64_t)n_sm + n_tracks - 1) / (n_tracks ? n_tracks : 1);
  const uint64_t cmax = (P + kWeightThreads - 1) / kWeightThreads;
  if (c > cmax) c = cmax;
  if (c > 256) c = 256;
  return (uint32_t)(c < 1 ? 1 : c);
}

__device__ __forceinline__ void adj_weight_final(const FarMixedParams &p, const double *wpart,
                                                 uint32_t n_chunks, int linear, double *grad_w) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < p.n_tracks;
       t += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (uint32_t b = 0; b < n_chunks; ++b) s += wpart[(uint64_t)t * n_chunks + b];
    const double w = p.weight[t];
    grad_w[t] = linear ? (w > 0.0 ? s / (2.0 * sqrt(w)) : 0.0) : 0.5 * s;
  }
}

// Rounding of a step's retarded time difference formed in FP32, as a fraction of
// the sum of its terms' sizes (which cancel by (gamma theta)^2 along the
// motion): constants, differences, products and sums, 8 x 2^-24 at most, doubled.
constexpr float kQuickErr = 1e-6f;

// Cut steps of a warp (steps of which the phase limit takes a part of the axis):
// a few are summed one after the other, 32 frequencies at a time over the lanes
// (`each` instructions per step and 32 frequencies, 35 for the sums over the
// lanes); many are walked side by side, a lane its own step (`walk` instructions
// per frequency).  The counts are the loops' instructions; the measured times
// cross where they do.
__device__ __forceinline__ bool walk_cut(uint32_t cut, uint32_t n_omega, uint32_t each,
                                         uint32_t walk) {
  return (uint32_t)__popc(cut) * (35u + each * ((n_omega + 31u) / 32u)) > 60u + walk * n_omega;
}

// First and last frequency that any of the warp's cut steps includes (of none:
// first > last).
__device__ __forceinline__ void cut_span(bool is_cut, uint32_t range, int &first, int &last) {
  const int jf = (int)(range & 0xffffu), jl = (int)(range >> 16);
  const bool some = is_cut && jf <= jl;
  first = __reduce_min_sync(0xffffffffu, some ? jf : 0x7fffffff);
  last = __reduce_max_sync(0xffffffffu, some ? jl : -1);
}

// The transforms' cells (`cell` bytes each) of every (track, snapshot,
// direction, omega band), of as many tracks at a time as 2 GiB hold; none
// (batch 0) where one track's do not fit, the axis is too short to gain or the
// least scratch is asked for.
struct AdjFields {
  uint32_t n_split;  // runs of directions whose gradients are summed apart
  uint32_t batch;    // tracks at a time
  uint32_t n_bands, nb, M;
  size_t bytes;
};

inline AdjFields adj_fields_layout(int64_t total_steps, uint32_t n_omega, uint64_t n_dirs,
                                   uint32_t n_tracks, uint32_t n_snaps, size_t cell,
                                   int steps_per_item, bool least) {
  AdjFields l{1, 0, 0, 0, 0, 0};
  if (least || n_omega < 8 || n_omega >= 65536u || n_tracks == 0 || n_snaps == 0 || total_steps <= 0)
    return l;
  l.n_bands = (n_omega + kFastMaxBand - 1) / kFastMaxBand;
  l.nb = (n_omega + l.n_bands - 1) / l.n_bands;
  l.M = fast_cells(l.nb);
  // A snapshot's transforms cost as much as walking the frequencies of about
  // 60 M / nb steps; with several snapshots the steps between two must be more
  // (400 frequencies, 45 steps a snapshot: far 11.3 / 9.3 ms, near 30.6 / 13.9 ms
  // transforms / walking; 64 frequencies, 150 steps: 0.49 / 1.13, 0.56 / 1.81).
  if (n_snaps > 1 && (uint64_t)total_steps * n_omega <
                         60ull * l.M * l.n_bands * n_snaps * n_tracks)
    return l;
  const uint64_t per = (uint64_t)n_snaps * n_dirs * l.n_bands * (l.M + kTaps) * cell;
  l.batch = (uint32_t)std::min<uint64_t>(n_tracks, (2ull << 30) / per);
  if (l.batch == 0) return l;
  l.bytes = (size_t)(l.batch * per);
  // few items: runs of at least 16 directions apart, so that the SMs fill
  const uint64_t slots = 2ull * device_sm_count();
  const uint64_t items = l.batch * ((uint64_t)total_steps / n_tracks / steps_per_item + 1);
  l.n_split = (uint32_t)std::max<uint64_t>(
      1, std::min<uint64_t>({(2 * slots + items - 1) / items, n_dirs / 16, 16}));
  return l;
}

}  // namespace
}  // namespace sr
