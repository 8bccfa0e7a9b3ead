// Far-field instances of the summation by transforms, and its work split.
#include <algorithm>
#include <cmath>

#include "sr_fast_sum.cuh"

namespace sr {

namespace {
size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// Mean steps of a track from which the transforms are ahead of the term-by-term
// kernel.  That one walks a track's steps one after the other at a cost that
// falls with the number of (track, 32 directions) units once they fill the SMs;
// the transforms pay for circles of M cells per unit, whatever its steps, and for
// whole warps where there are fewer than 32 directions (`part`).  Term by term /
// transforms, times of undulator batches of 20 to 1280 steps (each line: sizes,
// ratio below and above its entry):
//   far, 512 frequencies, 1024 directions, 64 tracks: 40 steps 0.72, 80 1.4
//     64 directions, 500 tracks: 0.70 at 40, 1.03 at 80, 1000 units
//     256 directions, 64 tracks: 0.80 at 80, 1.28 at 160, 512 units
//     64 directions, 64 tracks: 0.91 at 160, 1.28 at 320, 128 units
//     8 directions, 64 tracks: 0.69 at 320, 1.1 at 640
//   far, 64 frequencies, same: 0.89 / 1.58 at 40 / 80, 0.97 / 1.54 at 80 / 160,
//     0.93 / 1.34 at 80 / 160, 0.90 / 1.07 at 160 / 320, 0.87 / 1.08 at 160 / 320
//   near, 16 frequencies: 1.37 at 40, 1.19 at 80, 0.86 / 1.06 at 80 / 160,
//     0.64 at 320 and 0.99 at 1280, 0.71 / 1.24 at 640 / 1280
//   near, 300 frequencies: 0.98 / 1.6 at 20 / 40, 0.72 / 1.29 at 20 / 40, 0.62 / 1.03
//     at 20 / 40, 0.93 / 1.02 at 40 / 80, 0.68 / 0.90 at 640 / 1280
uint64_t least_steps(bool near, uint32_t M, uint64_t units, bool part) {
  if (!near) {
    if (units >= 1824) return 64;
    if (units >= 768) return M <= 512 ? 96 : 128;
    if (units >= 140) {
      if (part) return M > 512 ? 320 : units >= 400 ? 24 : 80;
      return M <= 512 ? 112 : 128;
    }
    if (units >= 56) return M <= 512 ? 320 : part ? 800 : 256;
    if (M <= 512) return M <= 256 ? 320 : part ? 200 : 160;
    return part ? 640 : units >= 24 ? 400 : 320;
  }
  if (units >= 1216) return 32;
  if (units >= 768) return M == 128 ? 128 : 64;
  if (units >= 140) {
    if (part) return M <= 256 ? 40 : M == 512 ? 200 : 400;
    return M == 128 ? 280 : M <= 512 ? 64 : 96;
  }
  if (units >= 56) return M == 128 ? 1280 : M == 256 ? 400 : part ? 2 * (uint64_t)M : 200;
  return M <= 512 ? 512 : 800;
}
}  // namespace

FastLayout fast_layout(const FarMixedConfig &c, bool near, int64_t total_steps, int n_out,
                       uint32_t n_snaps) {
  FastLayout l{};
  if (c.direct || c.n_omega < 4 || c.n_dirs == 0 || c.n_tracks == 0 || n_snaps == 0 ||
      total_steps <= 0)
    return l;
  const uint64_t mean = (uint64_t)total_steps / c.n_tracks;
  l.on = true;
  l.n_sm = (uint32_t)c.n_sm;
  const int np = near ? 3 : 1;
  l.n_bands = (c.n_omega + kFastMaxBand - 1) / kFastMaxBand;
  l.nb = (c.n_omega + l.n_bands - 1) / l.n_bands;
  l.M = fast_cells(l.nb);
  l.n_dwb = (c.n_dirs + 31) / 32 * l.n_bands;
  // A list holds what a segment of a block can add and a chunk more (it is
  // summed when a further chunk might not fit), longer walks get longer ones:
  // each emptying reads and writes the warp's direct sums (half of the steps
  // listed, 256 frequencies: 48.9 ms with 96 entries, 38.5 with 512).
  auto use_list = [&](uint32_t entries) {
    l.list = entries;
    l.slice_bytes = up256((size_t)32 * (np * (size_t)(l.M + 2 * l.nb) * 16 +
                                        entries * (16 + 8 * (size_t)np)));
  };
  // Steps between two writes of the whole window: 128, fewer where they could
  // lap the circle (a step moves by up to M / (2 nb) cells).
  l.block = 128;
  while (l.block > 32 && (uint64_t)l.block * l.M + 16ull * l.nb > 2ull * l.nb * l.M) l.block /= 2;
  use_list(l.block + 32);
  const uint64_t resident = (uint64_t)c.n_sm * (near ? 2 : 3) * kFastWarps;
  const uint64_t units = (uint64_t)c.n_tracks * l.n_dwb;
  const uint64_t least = least_steps(near, l.M, units, c.n_dirs < 32);
  // few tracks: the rule of before the measurements by units, no lower
  const uint64_t few = near ? 512 : c.n_omega > 128 && c.n_omega <= 256 ? 160 : 320;
  if (mean < (c.n_tracks < 64 ? std::max(least, few) : least)) return FastLayout{};
  l.dirs_per_warp = std::max(1u, 512u / l.M);
  const uint64_t P = (uint64_t)c.n_omega * c.n_dirs;
  // Few (track, 32 directions) units: their steps are split in segments of a
  // block, after which a whole track's window is written out too, so that far-field
  // sums of up to 128 frequencies come out the same either way where no step is cut
  // (other sizes, and chunks of a batch that take another path than the whole,
  // agree to the precision's tolerance only).  Larger circles and the near field's
  // three take longer segments: each one is cleared and read once per segment
  // (~4 TB/s) while a step takes ~0.4 us, shortest together at
  // sqrt(steps x bytes / (4e12 x 0.4e-6))
  // (near, 8 tracks of 1280 steps, 1024 directions, 16 frequencies: 0.63 of the
  // term-by-term kernel's speed with segments of a block, 1.5 times it now).  Where that
  // leaves more than four units per resident warp or 4 GiB, segments grow for
  // the few long tracks that would not fill the SMs, else tracks stay whole.
  if (n_snaps == 1 && units <= resident) {
    const uint64_t all = (uint64_t)total_steps * l.n_dwb;
    uint64_t seg = l.block;
    const bool larger = near || l.M >= 512;
    if (larger) use_list(kFastList);
    const uint64_t room = (4ull << 30) / l.slice_bytes;
    if (larger)
      seg = std::max<uint64_t>(
          seg, (uint64_t)(std::sqrt((double)all * (2.0 * np * l.M * 512.0) / 1.6e6) / 128.0) * 128);
    bool split = true;
    if (all / seg + units > room) {
      split = 2 * units < resident || l.M >= 512;
      const uint64_t most =
          std::max<uint64_t>(2 * resident, std::min<uint64_t>(4 * resident, room));
      seg = std::max<uint64_t>(seg, (all / (most - units) / 128 + 1) * 128);
      use_list(kFastList);
    }
    if (split && (uint64_t)total_steps > seg) {
      l.split = true;
      l.seg_steps = (uint32_t)std::min<uint64_t>(seg, 0xffffff00u);
      l.n_segs = (uint32_t)((uint64_t)total_steps / seg + c.n_tracks);
      // lists that hold a whole segment, where they fit 4 GiB: one that fills up
      // is emptied by its warp, which the others then wait for (near, 87 tracks of
      // 600 steps, 5 a period, 140 directions, 512 frequencies: 14.5 ms, now 4.7)
      const uint32_t fixed = l.list;
      use_list((uint32_t)std::max<uint64_t>(fixed, std::min<uint64_t>(seg, 1u << 20) + 32));
      if ((uint64_t)l.n_segs * l.n_dwb * l.slice_bytes > (4ull << 30)) use_list(fixed);
    }
  }
  if (n_snaps > 1) {
    // A snapshot costs transforms that grow with the circle and, of several
    // units' circles, leave the L2: with few steps between two, the term-by-term
    // kernel, which only reads its sums out, is ahead (ms, transforms / term by
    // term, 40 tracks, 24 x 24 directions, steps x frequencies / cells in
    // brackets: far 64 frequencies 4.6 / 5.4 [7], 256: 4.4 / 9.2 [22] and
    // 26 / 24 [7], 400: 11.1 / 14.9 [22] and 76 / 46 [5]; near 400: 34.9 / 35.0
    // [22], 298 / 120 [5]).
    if (mean * c.n_omega * 128 < 3ull * l.M * l.M * l.n_bands * n_snaps) return FastLayout{};
    // A unit per interval between them; a snapshot's transform adds up the
    // circles of the intervals before it.  More than 16 or 4 GiB: whole tracks,
    // which takes some hundred of them (32 directions, 900 steps, 20 snapshots,
    // 256 frequencies: 40 tracks far 2.84 / 1.81 ms, near 10.5 / 2.3; 300 tracks
    // 3.4 / 8.9 and 11.4 / 11.3).
    use_list(kFastList);
    if (n_snaps <= 16 && units <= resident &&
        units * n_snaps * l.slice_bytes <= (4ull << 30)) {
      l.split = true;
      l.seg_steps = 0;
      l.n_segs = c.n_tracks * n_snaps;
    } else if (8 * units < resident) {
      return FastLayout{};
    }
  }
  if (!l.split) use_list(kFastList);
  uint64_t subs;
  if (l.split) {
    const uint64_t groups = (uint64_t)l.n_dwb * (32u / l.dirs_per_warp) * n_snaps;
    subs = (resident + groups - 1) / groups;
  } else {
    subs = (8 * resident + l.n_dwb - 1) / l.n_dwb;
  }
  // partial spectra of at most 1 GiB, or one
  const uint64_t room = (1ull << 30) / std::max<uint64_t>(1, P * n_out * n_snaps * 8);
  subs = std::max<uint64_t>(1, std::min({subs, room, (uint64_t)c.n_tracks}));
  l.n_sub = (uint32_t)subs;
  const uint64_t warps = l.split ? (uint64_t)l.n_segs * l.n_dwb : std::min(resident, l.n_dwb * subs);
  l.slices = (uint32_t)((warps + kFastWarps - 1) / kFastWarps * kFastWarps);
  return l;
}

size_t fast_workspace(const FastLayout &l) {
  if (!l.on) return 0;
  return up256(kFastTables) + up256((size_t)l.slices * 4) +
         (l.split ? up256((size_t)l.slices * 32 * sizeof(uint2)) : 0) +
         (size_t)l.slices * l.slice_bytes;
}

void fast_bind(FarMixedParams &p, const FastLayout &l, bool near, unsigned char *base,
               unsigned char *status) {
  FastParams &f = p.fast;
  f.uneven = (unsigned int *)(status + 64);
  f.M = 0;
  if (!l.on) return;
  f.queue = (unsigned int *)(status + 192);
  fast_tables_bind(p, l.n_bands, l.nb, l.M, base, status);
  base += up256(kFastTables);
  f.dirty = (unsigned int *)base;
  base += up256((size_t)l.slices * 4);
  f.work = (uint2 *)base;
  f.n_work = (unsigned int *)(status + 200);
  if (l.split) base += up256((size_t)l.slices * 32 * sizeof(uint2));
  f.scratch = base;
  f.slice_bytes = l.slice_bytes;
  f.n_dwb = l.n_dwb;
  f.n_sub = l.n_sub;
  f.n_segs = l.n_segs;
  f.seg_steps = l.seg_steps;
  f.block = l.block;
  f.list = l.list;
  f.dirs_per_warp = l.dirs_per_warp;
  // phi nodes spanned by 32 consecutive directions, and the steps whose turned
  // records of all of them fit the staging buffer (128 records)
  f.n_phik = near ? 1u : std::min(p.n_phi, (p.n_theta + 30u) / p.n_theta + 1u);
  f.chunk = 32u;
  while (!near && f.chunk * f.n_phik > 128u) f.chunk /= 2u;
}

int launch_uneven_far(const FarMixedParams &p, int n_sm, cudaStream_t s) {
  return launch_uneven<false>(p, n_sm, s);
}

int launch_fast_far(const FarMixedParams &p, const FastLayout &l, cudaStream_t s) {
  return launch_fast<false>(p, l, s);
}

}  // namespace sr
