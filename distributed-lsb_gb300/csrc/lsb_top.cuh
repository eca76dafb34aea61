// lsb_top.cuh -- device code shared by the kernels that sort by top digits
// (lsb_top.cu, lsb_mid.cu): the sample that chooses the digits, runs of keys
// that agree in them, and the barrier of a co-resident grid.
#pragma once

#include "lsb_internal.h"
#include "lsb_tile.cuh"

namespace lsb {

// The pass plan lsb_query reports, from the bits in which the keys differ: a
// digit in which no key differs counts as skipped (thread 0 of one CTA).
__device__ __forceinline__ void write_plan(Ctrl* ctrl, uint64_t diff, uint32_t n, int bits, int num_digits,
                                           int api_bits, int sub) {
  uint32_t lo = 0, hi = 0, runs = 0;
  const uint64_t mask = (1ull << bits) - 1ull;
  for (int p = 0; p < num_digits; p++) {
    if ((diff >> (bits * p)) & mask) runs++;
    else if (p < 32) lo |= 1u << p;
    else hi |= 1u << (p - 32);
  }
  ctrl->skip_mask_lo = lo;
  ctrl->skip_mask_hi = hi;
  ctrl->passes_run = runs;
  ctrl->final_copy = runs & 1u;
  ctrl->num_passes = (uint32_t)num_digits;
  ctrl->api_bits = (uint32_t)api_bits;
  ctrl->sub = (uint32_t)sub;
  ctrl->n = n;
}

// ---------------------------------------------------------------------------
// the sample

constexpr int kSampleThreads = 1024;
// S keys per thread: 1024 S sample keys.
template <int S>
using SampleTile = TileSort<kSampleThreads, S>;
template <int S>
constexpr size_t kSampleSmem = SampleTile<S>::kSmem + (size_t)SampleTile<S>::kCap * 8u;

// What the sample's statistics are held against (from n and the tile alone).
struct SampleRule {
  uint32_t tmin, tmax;  // fewest passes that shorten even runs to a tile, most passes there can be
  uint32_t heavy;       // a key this often in the sample is heavy
  uint32_t tall;        // passes that leave a heavy key alone in its run
  uint32_t far;         // this many sample keys apart in one window: a run longer than a tile
  uint32_t near_limit;  // neighbours that may share a window before the mean run is too long
  uint32_t dups;        // equal neighbours from which most keys occur eight times or more
  uint32_t far_limit;   // keys in runs longer than a tile that are put up with
  uint32_t big_tmin, big_near;  // tmin and near_limit for the big tile; tmax and more: it is not to be had
};
// mean_run: the mean run length up to which a pass is saved. Keys that occur
// more than `often` times are heavy, and the passes then have `spread` windows
// or more per element. sample: keys in the sample.
__host__ __device__ inline uint32_t passes_for(float n, float per_run) {
  uint32_t t = 1;
  for (float most = per_run * 256.0f; t < 8u && n > most; most *= 256.0f) t++;
  return t;
}
__host__ __device__ inline SampleRule sample_rule(uint32_t n, uint32_t sample, uint32_t mean_run, uint32_t often,
                                                  float spread) {
  SampleRule r;
  const float per = (float)sample / (float)n;
  r.tmin = passes_for((float)n, (float)mean_run);
  r.tmax = 8u;
  r.big_tmin = 9u;
  r.big_near = 0u;
  r.tall = passes_for((float)n, 1.0f / spread);
  const float lam = (float)mean_run * per, lom = (float)often * per;
  r.far = (uint32_t)(lam + 4.0f * sqrtf(lam) + 4.0f);
  r.heavy = (uint32_t)(lom + 4.0f * sqrtf(lom) + 4.0f);
  const float l = 1.25f * lam, f = 1.0f - (1.0f - expf(-l)) / l;
  r.near_limit = (uint32_t)((float)sample * f + 3.0f * sqrtf((float)sample * f)) + 1u;
  r.far_limit = sample / 64u;
  // sampled twice by chance: sample^2 / (2 n) pairs; every key k times in the array: k times that
  const float pairs = 4.0f * (float)sample * per;
  r.dups = pairs > 3.0f ? (uint32_t)pairs : 3u;
  return r;
}

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  return x ^ x >> 16;
}

// Sorts a sample of the keys of data[0, n) into shared memory (smem,
// kSampleSmem<S> bytes; all kSampleThreads threads call, with smem not in use) and
// returns it. The places are drawn independently of each other, not one per
// stretch: of an array nearly in order that would be the most even sample there is.
template <int S>
__device__ __forceinline__ const uint64_t* sample_keys(const Elem* data, uint32_t n, unsigned char* smem,
                                                       typename SampleTile<S>::Shared& sh) {
  using Sample = SampleTile<S>;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Sample::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Sample::kElemBytes + Sample::kSlotBytes);
  uint64_t* s = reinterpret_cast<uint64_t*>(smem + Sample::kSmem);
  uint64_t key[S];
#pragma unroll
  for (int k = 0; k < S; k++) {
    const uint32_t i = threadIdx.x + (uint32_t)k * kSampleThreads;
    key[k] = ld_relaxed_u64(&data[((uint64_t)mix32(i + 1u) * n) >> 32].key);
  }
#pragma unroll
  for (int k = 0; k < S; k++) in[threadIdx.x + (uint32_t)k * kSampleThreads] = Elem{key[k], 0};
  __syncthreads();
  Sample::sort(in, 0, Sample::kCap, 0, 0, slot, bins, sh, false, [&](bool on, uint32_t r, const Elem& e) {
    if (on) s[r] = e.key;
  });
  __syncthreads();
  return s;
}

// Passes over the highest bytes below bit hb1 after which the sample s lets
// expect runs of at most a tile, the same answer in every thread. near, far: 8
// and 9 shared words, 11 with `big`, zeroed before the sample was sorted. *skewed:
// a key is heavy. *big: the runs are for the big tile (null: not to be had).
template <int S>
__device__ __forceinline__ uint32_t sample_passes(const uint64_t* s, uint32_t hb1, const SampleRule& rule,
                                                  uint32_t* s_near, uint32_t* s_far, bool* skewed,
                                                  bool* big = nullptr) {
  // nibble T-1 of near / far: this thread's keys that share T windows (but
  // not all 64 bits) with the next key / with the key `far` places on
  constexpr uint32_t kSample = SampleTile<S>::kCap;
  uint32_t near = 0, farm = 0, equal = 0;
  uint64_t diff = 0;
  bool heavy = false;
#pragma unroll
  for (int k = 0; k < S; k++) {
    const uint32_t i = threadIdx.x + (uint32_t)k * kSampleThreads;
    const uint64_t ki = s[i];
    diff |= ki ^ s[0];
    auto shared_windows = [&](uint32_t j) {
      const uint32_t bits = hb1 - min(hb1, 64u - (uint32_t)__clzll((long long)(ki ^ s[j])));
      return 0x11111111u & ((1u << (4u * (bits >> 3))) - 1u);  // bits < 64: the keys differ
    };
    if (i + 1u < kSample) {
      if (s[i + 1u] != ki) near += shared_windows(i + 1u);
      else equal++;
    }
    if (i + rule.far - 1u < kSample && s[i + rule.far - 1u] != ki) farm += shared_windows(i + rule.far - 1u);
    heavy |= i + rule.heavy - 1u < kSample && s[i + rule.heavy - 1u] == ki;
  }
  {
    const uint32_t n0 = __reduce_add_sync(0xffffffffu, near & 0x0F0F0F0Fu);
    const uint32_t n1 = __reduce_add_sync(0xffffffffu, (near >> 4) & 0x0F0F0F0Fu);
    const uint32_t f0 = __reduce_add_sync(0xffffffffu, farm & 0x0F0F0F0Fu);
    const uint32_t f1 = __reduce_add_sync(0xffffffffu, (farm >> 4) & 0x0F0F0F0Fu);
    const uint32_t l = lane_id();
    if (l < 8) {
      atomicAdd(&s_near[l], ((l & 1u ? n1 : n0) >> (8u * (l >> 1))) & 0xFFu);
      atomicAdd(&s_far[l], ((l & 1u ? f1 : f0) >> (8u * (l >> 1))) & 0xFFu);
    }
  }
  if (big) {  // bits in which keys differ
    const uint32_t d0 = __reduce_or_sync(0xffffffffu, (uint32_t)diff), d1 = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    if (lane_id() == 0) {
      atomicOr(&s_far[9], d0);
      atomicOr(&s_far[10], d1);
    }
  }
  equal = __reduce_add_sync(0xffffffffu, equal);
  if (lane_id() == 0 && equal) atomicAdd(&s_far[8], equal);
  heavy = __syncthreads_or(heavy);
  *skewed = heavy;
  auto enough = [&](uint32_t t, uint32_t near_limit) {
    return s_near[t - 1u] <= near_limit && s_far[t - 1u] <= rule.far_limit && (!heavy || t >= rule.tall);
  };
  const uint32_t full = (hb1 + 7u) / 8u, most = min(rule.tmax, full);
  uint32_t t = min(rule.tmin, full);
  while (t < most && !enough(t, rule.near_limit)) t++;
  if (big) {  // a pass less, if the big tile's bins will be even: no bit of the keys constant
    const uint64_t varies = (uint64_t)s_far[10] << 32 | s_far[9];
    *big = t > 1u && t - 1u >= rule.big_tmin && t < full && enough(t - 1u, rule.big_near) && s_far[8] < rule.dups &&
           varies == ~0ull >> (64u - hb1);
    if (*big) return t - 1u;
  }
  // one pass more that leaves nothing to sort costs less than sorting runs of duplicates
  return t + 1u == full && t < rule.tmax && s_far[8] >= rule.dups ? full : t;
}

// ---------------------------------------------------------------------------
// runs of keys that agree in the passes' digits

// The window a key falls in: equal for the keys of one run.
struct RunKey {
  uint64_t lo, hi;  // smallest and largest key of the block
  uint32_t shift;
};
__device__ __forceinline__ uint64_t run_of(const RunKey& w, uint64_t key) {
  const uint64_t k = key < w.lo ? w.lo : key > w.hi ? w.hi : key;
  return k >> w.shift;
}
template <class Plan>
__device__ __forceinline__ RunKey run_key(const Plan& p) {
  RunKey w;
  w.lo = p.clamp ? p.lo : 0ull;
  w.hi = p.clamp ? p.hi : ~0ull;
  w.shift = p.hb1 > 8u * p.passes ? p.hb1 - 8u * p.passes : 0u;
  return w;
}

// One warp: first index in [from, to) whose key is in another run than r
// (every key before it in r), else `to`. In global memory by relaxed loads: a
// neighbouring CTA may be sorting the run, which keeps its keys inside it.
template <bool GLOBAL>
__device__ __forceinline__ uint32_t run_end(const Elem* a, const RunKey& w, uint64_t r, uint32_t from, uint32_t to) {
  uint32_t lo = from, hi = to;
  while (lo < hi) {
    const uint32_t step = (hi - lo - 1u) / 32u + 1u;
    const uint64_t i = (uint64_t)lo + (uint64_t)lane_id() * step;
    const bool same = i < hi && run_of(w, GLOBAL ? ld_relaxed_u64(&a[i].key) : a[i].key) == r;
    const uint32_t t = (uint32_t)__popc(__ballot_sync(0xffffffffu, same));
    if (t == 0) return lo;
    const uint64_t nhi = (uint64_t)lo + (uint64_t)t * step;
    hi = nhi < hi ? (uint32_t)nhi : hi;
    lo += (t - 1u) * step + 1u;
  }
  return lo;
}

// One warp: first index in [0, to] of the run r that a[to] (shared memory) is in.
__device__ __forceinline__ uint32_t run_start(const Elem* a, const RunKey& w, uint64_t r, uint32_t to) {
  uint32_t lo = 0, hi = to;  // a[i] for i < lo is in earlier runs, a[hi] in r
  while (lo < hi) {
    const uint32_t step = (hi - lo - 1u) / 32u + 1u;
    const uint32_t i = lo + lane_id() * step;
    const bool earlier = i < hi && run_of(w, a[i].key) != r;
    const uint32_t t = (uint32_t)__popc(__ballot_sync(0xffffffffu, earlier));
    if (t == 0) return lo;
    hi = min(hi, lo + t * step);
    lo += (t - 1u) * step + 1u;
  }
  return lo;
}

__device__ __forceinline__ Elem load_elem_l2(const Elem* p) {
  Elem e;  // L2 only: another CTA has written it since this kernel began
  asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(e.key), "=l"(e.val) : "l"(p) : "memory");
  return e;
}

// Sorts the runs that start in [g, limit) of src[0, n) into X (src = X: in
// place), as many whole runs at a time as fit in a tile: a tile's worth comes
// in from where the CTA stands (the piece of a run at its end comes again with
// the next tile), the last run start in it is found, and the runs up to there
// are sorted. known: g is a run's start. load(from, count) brings src[from,
// from + count) into in[], a barrier before it and one after, and returns false
// for the whole CTA on an error; long_run(b, e), called by warp 0, takes a run of at
// least a tile. False after a failed load.
// skewed: heavy keys are about, and tiles are mostly in order, but for a run
// here and there that holds two keys: one or two such runs are sorted by
// themselves, where the whole tile's bins would be uneven.
// In place, the CTA may see elements of a run that another one is rewriting,
// but only to tell which run they are in, which does not change.
struct RunMarks {
  uint32_t first, beyond, last, end, inversion;
};
template <class TS, class Load, class Long>
__device__ __forceinline__ bool sort_runs(const Elem* src, Elem* X, uint32_t n, uint32_t g, uint32_t limit, bool known,
                                          const RunKey& w, bool clamped, bool skewed, uint32_t shift, const Elem* in, uint32_t* slot,
                                          uint32_t* bins, typename TS::Shared& sh, RunMarks& marks, Load load,
                                          Long long_run) {
  constexpr uint32_t kNone = 0xffffffffu;
  constexpr int kMaxMixed = 2;                     // runs fixed one by one
  constexpr int kFewThreads = 4, kManyThreads = 64;  // threads that see an inversion: small runs, or one long one
  const uint32_t warp = threadIdx.x >> 5;
  const bool in_place = src == X;
  while (g < limit) {
    const uint32_t w0 = known ? g : g - 1u;
    const uint32_t cnt = min(TS::kCap, n - w0);
    if (!load(w0, cnt)) return false;
    // first run start, first one at or after `limit`, last one (tile
    // positions; kNone, cnt and 0 when there is none), by one warp each
    if (warp == 0) {
      const uint32_t e = run_start(in, w, run_of(w, in[cnt - 1u].key), cnt - 1u);
      if (lane_id() == 0) marks.last = e;
    } else if (warp == 1) {
      const uint32_t l = limit - w0;
      const uint32_t e = l < cnt ? run_end<false>(in, w, run_of(w, in[l - 1u].key), l, cnt) : cnt;
      if (lane_id() == 0) marks.beyond = e;
    } else if (warp == 2) {
      const uint32_t e = known ? 0u : run_end<false>(in, w, run_of(w, in[0].key), 1u, cnt);
      if (lane_id() == 0) marks.first = e < cnt ? e : kNone;
    }
    __syncthreads();
    const uint32_t first = marks.first, beyond = marks.beyond, last = marks.last;
    const bool at_end = w0 + cnt == n;
    if (first == kNone) {  // inside a run that an earlier part has
      if (at_end || w0 + cnt >= limit) break;
      if (warp == 0) {
        const uint32_t e = run_end<true>(src, w, run_of(w, in[0].key), w0 + cnt, limit);
        if (lane_id() == 0) marks.end = e;
      }
      __syncthreads();
      g = marks.end;
      known = true;
      continue;
    }
    if (w0 + first >= limit) break;
    const uint32_t end = beyond < cnt ? beyond : at_end ? cnt : last;
    known = true;
    if (end > first) {
      g = w0 + end;
      if (end - first == 1u && in_place) continue;
      uint32_t from = first;
      if (skewed) {
        for (int i = 0; i < kMaxMixed && from < end; i++) {
          // the first element above the next one, and its run
          if (threadIdx.x == 0) marks.inversion = kNone;
          __syncthreads();
          uint32_t p = kNone;
          for (uint32_t q = from + threadIdx.x; q + 1u < end && p == kNone; q += TS::kThreads)
            if (in[q].key > in[q + 1u].key) p = q;
          const bool seen = p != kNone;
          p = __reduce_min_sync(0xffffffffu, p);
          if (lane_id() == 0 && p != kNone) atomicMin(&marks.inversion, p);
          const int threads = __syncthreads_count(seen);
          if (threads > kFewThreads && threads < kManyThreads) break;
          p = marks.inversion;
          if (p != kNone) {
            if (warp == 0) {
              const uint32_t e = run_start(in, w, run_of(w, in[p].key), p);
              if (lane_id() == 0) marks.last = e;
            } else if (warp == 1) {
              const uint32_t e = run_end<false>(in, w, run_of(w, in[p].key), p + 1u, end);
              if (lane_id() == 0) marks.beyond = e;
            }
          }
          __syncthreads();
          const uint32_t a = p != kNone ? marks.last : end, b = p != kNone ? marks.beyond : end;
          if (!in_place)
            for (uint32_t q = from + threadIdx.x; q < a; q += TS::kThreads) store_elem(X + w0 + q, in[q]);
          if (a < b) {
            Elem* out = X + w0 + a;
            TS::sort_any(in, a, b, slot, bins, sh, true, in_place,
                         [=](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); });
          }
          from = b;
          __syncthreads();
        }
        if (from >= end) continue;
      }
      // whole runs: bins over their range of keys; keys outside the block are in
      // its first and last run, which take the tile's own range
      uint64_t base = 0, range = 0;
      const uint64_t r0 = run_of(w, in[from].key), r1 = run_of(w, in[end - 1u].key);
      if (!clamped || (r0 != w.lo >> shift && r1 != w.hi >> shift)) {
        base = r0 << shift;
        range = (r1 << shift | ((1ull << shift) - 1ull)) - base;
      }
      Elem* out = X + w0 + from;
      TS::sort(in, from, end, base, range, slot, bins, sh, in_place,
               [=](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); });
    } else if (first > 0u) {  // one run from `first`, not whole in the tile yet
      g = w0 + first;
    } else {  // a run of at least a tile
      if (warp == 0) {
        const uint32_t e = run_end<true>(src, w, run_of(w, in[0].key), w0 + cnt, n);
        long_run(w0, e);
        if (lane_id() == 0) marks.end = e;
      }
      __syncthreads();
      g = marks.end;
    }
  }
  return true;
}

// ---------------------------------------------------------------------------
// tiles of runs and runs longer than a tile

using Tile = TileSort<512, 9>;  // 106 KB: two CTAs per SM, one's loads and stores beside the other's sort
constexpr uint32_t kCap = Tile::kCap;
using SmallTile = TileSort<256, 9>;  // 54 KB: four CTAs per SM
using BigTile = TileSort<1024, 9>;   // 212 KB: one CTA per SM
// Mean run length up to which a pass is saved: six standard deviations below a tile.
constexpr uint32_t kMeanRun = 4220;
// A chunk of a run too long for a tile: elements [b + k kCap, ...) of the run [b, e).
struct RunChunk {
  uint32_t b, e, k, run : 31, par : 1;  // par: the run lies in Y
};
__host__ __device__ __forceinline__ uint32_t max_chunks(uint32_t n) { return 3u * (n / kCap) + 2u; }

// One warp: the run [b, e) goes to the merge kernel's list (in the ring, which
// the passes are done with): runs of at least kCap / 2 elements, so at most
// 2 n / kCap of them.
__device__ __forceinline__ void push_run(Ctrl* ctrl, RunChunk* chunks, uint32_t* unsorted, uint32_t n, uint32_t b,
                                         uint32_t e, uint32_t par) {
  const uint32_t lane = lane_id();
  const uint32_t m = (e - b - 1u) / kCap + 1u;
  uint32_t at = 0, run = 0;
  if (lane == 0) {
    at = atomicAdd(&ctrl->top.num_chunks, m);
    run = atomicAdd(&ctrl->top.num_runs, 1u);
    atomicMax(&ctrl->top.max_rounds, 32u - (uint32_t)__clz((int)(m - 1u)));
  }
  at = __shfl_sync(0xffffffffu, at, 0);
  run = __shfl_sync(0xffffffffu, run, 0);
  if ((uint64_t)at + m > max_chunks(n)) {  // the keys changed while they were sorted
    if (lane == 0) record_error(ctrl, kStatusInconsistent, kWhereScatter);
    return;
  }
  if (lane == 0) unsorted[run] = 0u;
  for (uint32_t k = lane; k < m; k += 32u) chunks[at + k] = RunChunk{b, e, k, run, par};
}

// src[0, cnt) into in[] by bulk copies that complete on the barrier `bar` (of one
// arrival), for the whole CTA; false when the wait ran out.
__device__ __forceinline__ bool load_tile_bulk(Elem* in, const Elem* src, uint32_t cnt, uint32_t bar, uint32_t* phase,
                                               Ctrl* ctrl) {
  __syncthreads();  // in[] is no longer read
  if (threadIdx.x == 0) {
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(bar, cnt * (uint32_t)sizeof(Elem));
    for (uint32_t o = 0; o < cnt; o += 2048u)
      bulk_g2s(smem_u32(in + o), src + o, min(2048u, cnt - o) * (uint32_t)sizeof(Elem), bar);
  }
  const bool ok = wait_copies(bar, *phase, ctrl);
  *phase ^= 1u;
  return !__syncthreads_or(!ok);
}

// ---------------------------------------------------------------------------
// a co-resident grid's barrier

// Every CTA of the (co-resident) grid arrives; false when the wait ran out or
// an error was raised.
__device__ __forceinline__ bool grid_barrier(Ctrl* ctrl, uint32_t* round) {
  __shared__ bool s_ok;
  *round += 1u;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&ctrl->top.barrier, 1u);
    s_ok = wait_arrivals(&ctrl->top.barrier, *round * gridDim.x, ctrl);
    __threadfence();
  }
  __syncthreads();
  return s_ok;
}

// The same of one cluster of CTAs, in hardware; global memory is ordered by it too.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

}  // namespace lsb
