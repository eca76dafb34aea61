// lsb_top.cu -- the "top" kernel family: whole sorts that do not go through
// every digit of the key.
//
// mySort (mpi/mpi_lsbsort.cpp:592-597) sorts by all 64/RADIX digits, lowest
// first, each digit one pass over memory. Its result is the stable order of
// the keys, and that is what the kernels here produce with fewer passes: an
// array that fits in one CTA's shared memory is sorted there, in one launch; a
// larger one is passed over by its top digits only, and the runs of keys that
// agree in them are sorted in shared memory.
#include <algorithm>
#include <cmath>

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
// one CTA, one launch

// Bound by latency: one read of the tile, seven barriers, one write. Twelve
// launches (clears, the histogram, the plan, eight passes and the copy back)
// took 112 us for 1000 elements with the array's own copy; this takes 20.5 us.
template <int THREADS, int K>
__global__ void __launch_bounds__(THREADS, 1)
    k_small_sort(Elem* __restrict__ a, uint32_t n, int bits, int num_digits, int api_bits, int sub, Ctrl* ctrl) {
  using TS = TileSort<THREADS, K>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename TS::Shared sh;
  __shared__ uint32_t s_diff[2];
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes + TS::kSlotBytes);
  for (uint32_t i = threadIdx.x; i < kCtrlBytes / 4u; i += THREADS) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
  uint64_t key[K];
  {
    Elem v[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = threadIdx.x + (uint32_t)k * THREADS;
      if (p < n) v[k] = a[p];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = threadIdx.x + (uint32_t)k * THREADS;
      if (p < n) in[p] = v[k];
      key[k] = p < n ? v[k].key : 0ull;
    }
  }
  if (threadIdx.x < 2) s_diff[threadIdx.x] = 0u;
  __syncthreads();
  {
    uint64_t diff = 0;
    const uint64_t first = in[0].key;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (threadIdx.x + (uint32_t)k * THREADS < n) diff |= key[k] ^ first;
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    if (lane_id() == 0) {
      atomicOr(&s_diff[0], lo);
      atomicOr(&s_diff[1], hi);
    }
  }
  TS::sort(in, 0, n, 0, 0, slot, bins, sh, true, [&](bool on, uint32_t r, const Elem& e) { store_elem_if(on, a + r, e); });
  // s_diff: the sort's barriers lie between
  if (threadIdx.x == 0)
    write_plan(ctrl, (uint64_t)s_diff[1] << 32 | s_diff[0], n, bits, num_digits, api_bits, sub);
}

// 1024 threads hold up to 9216 elements (212 KB of shared memory); up to half
// that 512 threads do, whose barriers cost less.
using SmallHalf = TileSort<512, 9>;
using SmallFull = TileSort<1024, 9>;

// Between the two the launches and their latency set the time, and eight passes
// of one tile per SM were no worse than one or two with a sample before them
// when keys are skewed (10^6 Zipf keys: 153 us against 234; uniform 153 against 62).
constexpr uint32_t kTopFrom = 5u << 18;
bool top_serves(uint32_t n) { return n <= SmallFull::kCap || n >= kTopFrom; }

template <int THREADS>
static int small_sort(Elem* X, const Layout& L, Ctrl* ctrl, cudaStream_t st) {
  auto kern = k_small_sort<THREADS, 9>;
  const size_t smem = TileSort<THREADS, 9>::kSmem;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 5;
  ProfScope prof("small_sort", st);
  kern<<<1, THREADS, smem, st>>>(X, L.n, L.stat_bits, L.stat_digits, L.api_bits, L.sub, ctrl);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 5;
}

// ---------------------------------------------------------------------------
// larger arrays: passes over the top digits, then runs sorted on chip
//
//   k_top_sample  one CTA: a sorted sample of the keys chooses the digits
//   k_top_hist    one read of the keys: counts of those digits; its last CTA
//                 writes the pass plan
//   k_onesweep    one stable pass per digit, lowest first
//   k_top_finish  the array is now in the order of the digits' windows; each
//                 CTA takes whole runs of equal windows, up to a tile of them
//                 at a time, and sorts them by the whole key
//   k_top_merge   runs longer than a tile (the sample missed them): checked,
//                 and sorted by chunks and merges unless they are in order
// The result does not depend on the sample: it only decides how short the
// runs are, and so the time. Measured (GB300, sort alone): 2^24 uniform 1.10 ->
// 0.48 ms, 2^28 15.0 -> 6.4 ms, 2^30 58.6 -> 30.8 ms (three passes), 2^28 Zipf
// 16.0 -> 9.8 ms (four passes; heavy keys stay in order), against eight passes.

using Tile = TileSort<512, 9>;  // 106 KB: two CTAs per SM, one's loads and stores beside the other's sort
constexpr uint32_t kCap = Tile::kCap;
// Mean run length up to which a pass is saved: six standard deviations below a tile.
constexpr uint32_t kMeanRun = 4220;
constexpr int kSampleThreads = 1024;
using SampleTile = TileSort<kSampleThreads, 4>;
constexpr uint32_t kSample = SampleTile::kCap;
constexpr size_t kSampleSmem = SampleTile::kSmem + (size_t)kSample * 8u;
constexpr int kTopHistThreads = 512;
constexpr int kTopHistUnroll = 4;

// What the sample's statistics are held against (host-side, from n alone).
struct SampleRule {
  uint32_t tmin, tmax;  // fewest passes that shorten even runs to a tile, most passes launched
  uint32_t tall;        // passes that leave a heavy key alone in its run
  uint32_t far;         // this many sample keys apart in one window: a run longer than a tile
  uint32_t near_limit;  // neighbours that may share a window before the mean run is too long
  uint32_t far_limit;   // keys in runs longer than a tile that are left to the merges
};

static SampleRule sample_rule(uint32_t n) {
  SampleRule r;
  auto passes_for = [&](double per_run) {
    uint32_t t = 1;
    while (t < 8 && (double)n > per_run * std::pow(256.0, (double)t)) t++;
    return t;
  };
  r.tmin = passes_for(kMeanRun);
  // Unused launches cost about 2 us each: below 2^26 elements only two passes
  // more than even keys need are kept ready, and the merges, whose rounds then
  // stay nearly in L2, take what those leave.
  r.tmax = n >= (1u << 26) ? 8u : std::min(8u, r.tmin + 2u);
  r.tall = passes_for(1.0 / 16.0);
  const double lam = (double)kMeanRun * kSample / n;
  r.far = (uint32_t)(lam + 4.0 * std::sqrt(lam) + 4.0);
  const double l = 1.25 * lam, f = 1.0 - (1.0 - std::exp(-l)) / l;
  r.near_limit = (uint32_t)(kSample * f + 3.0 * std::sqrt(kSample * f)) + 1u;
  r.far_limit = kSample / 64u;
  return r;
}

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  return x ^ x >> 16;
}

// Bound by latency (one CTA: 4096 scattered reads, a tile sort, two counts);
// it also clears what the later kernels count in, in place of three memsets.
__global__ void __launch_bounds__(kSampleThreads, 1)
    k_top_sample(const Elem* __restrict__ data, uint32_t n, SampleRule rule, uint32_t* __restrict__ hist, Ctrl* ctrl) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename SampleTile::Shared sh;
  __shared__ uint32_t s_near[8], s_far[8];
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + SampleTile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + SampleTile::kElemBytes + SampleTile::kSlotBytes);
  uint64_t* s = reinterpret_cast<uint64_t*>(smem + SampleTile::kSmem);
  const uint32_t tid = threadIdx.x;
  uint64_t key[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t i = tid + (uint32_t)k * kSampleThreads;
    // places drawn independently of each other (not one per stretch: of an
    // array nearly in order that would be the most even sample there is)
    key[k] = data[((uint64_t)mix32(i + 1u) * n) >> 32].key;
  }
  for (uint32_t i = tid; i < kCtrlBytes / 4u; i += kSampleThreads) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
  for (uint32_t i = tid; i < 8u * 256u; i += kSampleThreads) hist[i] = 0u;
  if (tid < 8) s_near[tid] = s_far[tid] = 0u;
#pragma unroll
  for (int k = 0; k < 4; k++) in[tid + (uint32_t)k * kSampleThreads] = Elem{key[k], 0};
  __syncthreads();
  SampleTile::sort(in, 0, kSample, 0, 0, slot, bins, sh, false, [&](bool on, uint32_t r, const Elem& e) {
    if (on) s[r] = e.key;
  });
  __syncthreads();
  const uint64_t first = s[0], span = first ^ s[kSample - 1u];
  const uint32_t hb1 = span ? 64u - (uint32_t)__clzll((long long)span) : 64u;
  // nibble T-1 of near / far: this thread's keys that share T windows (but
  // not all 64 bits) with the next key / with the key `far` places on
  uint32_t near = 0, farm = 0;
  bool heavy = false;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t i = tid + (uint32_t)k * kSampleThreads;
    const uint64_t ki = s[i];
    auto shared_windows = [&](uint32_t j) {
      const uint32_t bits = hb1 - min(hb1, 64u - (uint32_t)__clzll((long long)(ki ^ s[j])));
      return 0x11111111u & ((1u << (4u * (bits >> 3))) - 1u);  // bits < 64: the keys differ
    };
    if (i + 1u < kSample && s[i + 1u] != ki) near += shared_windows(i + 1u);
    if (i + rule.far - 1u < kSample) {
      if (s[i + rule.far - 1u] == ki) heavy = true;
      else farm += shared_windows(i + rule.far - 1u);
    }
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
  heavy = __syncthreads_or(heavy);
  if (tid == 0) {
    TopPlan& p = ctrl->top;
    const uint32_t full = (hb1 + 7u) / 8u, most = min(rule.tmax, full);
    uint32_t t = min(rule.tmin, full);
    while (t < most && !(s_near[t - 1u] <= rule.near_limit && s_far[t - 1u] <= rule.far_limit &&
                         (!heavy || t >= rule.tall)))
      t++;
    // one pass more that leaves nothing to sort costs no more than sorting the runs
    if (t + 1u == full && t < rule.tmax) t = full;
    p.passes = t;
    p.hb1 = hb1;
    p.lo = hb1 < 64u ? first >> hb1 << hb1 : 0ull;
    p.hi = hb1 < 64u ? p.lo | ((1ull << hb1) - 1ull) : ~0ull;
  }
}

// One read of the keys: counts of the plan's T digits in shared memory, the
// bits that differ, and the cleared look-back ring (2 KiB per 8192 elements,
// instead of a memset of its own). T <= 4: the digits are bytes of one word.
// A digit that is the same in the whole warp takes one shared atomic of 32
// instead of 32 conflicting ones (skewed keys).
template <int T, bool CLAMP>
__device__ __forceinline__ void count_windows(const Elem* __restrict__ data, uint32_t n, const TopPlan& p,
                                              uint32_t* h, uint64_t first, uint64_t* diff) {
  const uint32_t lane = lane_id();
  const uint64_t warps_total = (uint64_t)gridDim.x * (kTopHistThreads / 32);
  const uint64_t gw = (uint64_t)blockIdx.x * (kTopHistThreads / 32) + (threadIdx.x >> 5);
  constexpr uint32_t chunk = 32u * kTopHistUnroll;
  const uint64_t block_lo = p.lo, block_hi = p.hi;
  const uint32_t left = 64u - p.hb1;
  uint64_t acc = 0;
  auto word_of = [&](uint64_t key) {
    const uint32_t w = (uint32_t)((key << left) >> 32);
    return CLAMP ? (key < block_lo ? 0u : key > block_hi ? 0xffffffffu : w) : w;
  };
  const uint64_t full_end = (uint64_t)n / chunk * chunk;
  for (uint64_t base = gw * chunk; base < full_end; base += warps_total * chunk) {
    uint64_t key[kTopHistUnroll];
#pragma unroll
    for (int u = 0; u < kTopHistUnroll; u++) key[u] = load_elem_stream(data + base + (uint64_t)u * 32u + lane).key;
#pragma unroll
    for (int u = 0; u < kTopHistUnroll; u++) {
      acc |= key[u] ^ first;
      const uint32_t w = word_of(key[u]);
      const uint32_t x = __reduce_or_sync(0xffffffffu, w ^ __shfl_sync(0xffffffffu, w, 0));
#pragma unroll
      for (int t = 0; t < T; t++) {  // digit t: byte 4 - T + t
        uint32_t* c = &h[t * 256 + ((w >> (8 * (4 - T + t))) & 255u)];
        if ((x >> (8 * (4 - T + t))) & 255u) atomicAdd(c, 1u);
        else if (lane == 0) atomicAdd(c, 32u);
      }
    }
  }
  for (uint64_t i = full_end + (uint64_t)blockIdx.x * kTopHistThreads + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * kTopHistThreads) {
    const uint64_t key = load_elem_stream(data + i).key;
    acc |= key ^ first;
    const uint32_t w = word_of(key);
#pragma unroll
    for (int t = 0; t < T; t++) atomicAdd(&h[t * 256 + ((w >> (8 * (4 - T + t))) & 255u)], 1u);
  }
  *diff = acc;
}

// The same for five to eight digits, which only unusual keys need.
__device__ __noinline__ void count_many_windows(const Elem* __restrict__ data, uint32_t n, const TopPlan& p,
                                                uint32_t* h, uint64_t first, uint64_t* diff) {
  const uint64_t warps_total = (uint64_t)gridDim.x * (kTopHistThreads / 32);
  const uint64_t gw = (uint64_t)blockIdx.x * (kTopHistThreads / 32) + (threadIdx.x >> 5);
  const int T = (int)p.passes;
  uint64_t acc = 0;
  for (uint64_t base = gw * 32u; base < n; base += warps_total * 32u) {
    const bool valid = base + lane_id() < n;
    const uint64_t key = valid ? load_elem_stream(data + base + lane_id()).key : first;
    acc |= key ^ first;
    const bool whole = base + 32u <= n;
    for (int t = 0; t < T; t++) {
      const TopWindow w = top_window(p, t);
      const uint32_t d = w.clamp ? top_digit_clamped(w, key) : top_digit(w, key);
      if (whole && __all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {
        if (lane_id() == 0) atomicAdd(&h[t * 256 + d], 32u);
      } else if (valid) {
        atomicAdd(&h[t * 256 + d], 1u);
      }
    }
  }
  *diff = acc;
}

__global__ void __launch_bounds__(kTopHistThreads, 4)
    k_top_hist(const Elem* __restrict__ data, uint32_t n, uint32_t* __restrict__ hist, uint32_t* __restrict__ gstart,
               uint4* __restrict__ ring, uint64_t ring_words, int bits, int num_digits, int api_bits, int sub,
               Ctrl* ctrl) {
  __shared__ uint32_t h[8 * 256];
  __shared__ uint32_t s_diff[2];
  __shared__ uint32_t s_const;
  __shared__ bool s_last;
  const TopPlan& p = ctrl->top;
  const uint32_t T = p.passes;
  for (uint32_t i = threadIdx.x; i < T * 256u; i += kTopHistThreads) h[i] = 0u;
  if (threadIdx.x < 2) s_diff[threadIdx.x] = 0u;
  if (threadIdx.x == 0) s_const = 0u;
  for (uint64_t i = (uint64_t)blockIdx.x * kTopHistThreads + threadIdx.x; i < ring_words;
       i += (uint64_t)gridDim.x * kTopHistThreads)
    ring[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  const uint64_t first = data[0].key;
  uint64_t diff = 0;
  if (p.hb1 < 64u) {
    switch (T) {
      case 1: count_windows<1, true>(data, n, p, h, first, &diff); break;
      case 2: count_windows<2, true>(data, n, p, h, first, &diff); break;
      case 3: count_windows<3, true>(data, n, p, h, first, &diff); break;
      case 4: count_windows<4, true>(data, n, p, h, first, &diff); break;
      default: count_many_windows(data, n, p, h, first, &diff); break;
    }
  } else {
    switch (T) {
      case 1: count_windows<1, false>(data, n, p, h, first, &diff); break;
      case 2: count_windows<2, false>(data, n, p, h, first, &diff); break;
      case 3: count_windows<3, false>(data, n, p, h, first, &diff); break;
      case 4: count_windows<4, false>(data, n, p, h, first, &diff); break;
      default: count_many_windows(data, n, p, h, first, &diff); break;
    }
  }
  {
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    if (lane_id() == 0) {
      if (lo) atomicOr(&s_diff[0], lo);
      if (hi) atomicOr(&s_diff[1], hi);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < T * 256u; i += kTopHistThreads) {
    const uint32_t v = h[i];
    if (v) atomicAdd(&hist[i], v);
  }
  if (threadIdx.x < 2 && s_diff[threadIdx.x]) atomicOr(&ctrl->top.diff[threadIdx.x], s_diff[threadIdx.x]);
  // the last CTA to get here writes the plan
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ctrl->top.hist_done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  if (warp < T) {  // warp t scans digit t: exclusive starts, and whether one value holds every key
    uint32_t c[8], sum = 0;
    bool one = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      c[i] = __ldcg(&hist[warp * 256u + lane * 8u + i]);
      one |= c[i] == n;
      sum += c[i];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
    uint32_t off = inc - sum;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      gstart[warp * 256u + lane * 8u + i] = off;
      off += c[i];
    }
    if (__any_sync(0xffffffffu, one) && lane == 0) atomicOr(&s_const, 1u << warp);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    TopPlan& q = ctrl->top;
    const uint64_t d = (uint64_t)__ldcg(&q.diff[1]) << 32 | __ldcg(&q.diff[0]);
    uint32_t par = 0, pars = 0, run = 0;
    for (uint32_t t = 0; t < T; t++) {
      pars |= par << t;
      if (!((s_const >> t) & 1u)) {
        run |= 1u << t;
        par ^= 1u;
      }
    }
    q.run_mask = run;
    q.par_mask = pars;
    q.src_parity = par;
    const bool inside = q.hb1 >= 64u || ((d | (first ^ q.lo)) >> q.hb1) == 0;
    q.complete = (d == 0 || (q.hb1 <= 8u * T && inside)) ? 1u : 0u;
    write_plan(ctrl, d, n, bits, num_digits, api_bits, sub);
  }
}

// ---------------------------------------------------------------------------
// runs of equal windows

// The window a key falls in: equal for the keys of one run.
struct RunKey {
  uint64_t lo, hi;  // smallest and largest key of the block
  uint32_t shift;
};
__device__ __forceinline__ uint64_t run_of(const RunKey& w, uint64_t key) {
  const uint64_t k = key < w.lo ? w.lo : key > w.hi ? w.hi : key;
  return k >> w.shift;
}
__device__ __forceinline__ RunKey run_key(const TopPlan& p) {
  RunKey w;
  w.lo = p.lo;
  w.hi = p.hi;
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

// A chunk of a run too long for a tile: elements [b + k kCap, ...) of the run [b, e).
struct RunChunk {
  uint32_t b, e, k, run;
};
__host__ __device__ __forceinline__ uint32_t max_chunks(uint32_t n) { return 2u * (n / kCap) + 2u; }

// One warp: the run [b, e) goes to the merge kernel's list (in the ring, which
// the passes are done with): at most n / kCap runs of at least kCap elements.
__device__ __forceinline__ void push_run(Ctrl* ctrl, RunChunk* chunks, uint32_t* unsorted, uint32_t n, uint32_t b,
                                         uint32_t e) {
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
  for (uint32_t k = lane; k < m; k += 32u) chunks[at + k] = RunChunk{b, e, k, run};
}

// Sorts the runs in place (data in X) or from Y into X. The array is cut every
// `stride` elements; a CTA takes the runs that start in its part, as many whole
// runs at a time as fit in a tile: it brings in a tile's worth from where it
// stands (one bulk copy; the piece of a run at the end comes again with the
// next tile), finds the last run start in it and sorts up to there.
// In place a CTA may read elements of a run that its neighbour is rewriting,
// but only to see which run they are in, which does not change.
// 2^30 elements after three passes: 7.4 ms, 4.6 TB/s of the 32 bytes per
// element, bound by the sort's instructions (about 150 per 32 elements) and
// shared-memory accesses (45 wavefronts per 32) at 32 resident warps per SM.
__global__ void __launch_bounds__(Tile::kThreads, 2)
    k_top_finish(Elem* __restrict__ X, Elem* __restrict__ Y, uint32_t n, uint32_t stride,
                 RunChunk* __restrict__ chunks, uint32_t* __restrict__ unsorted, Ctrl* ctrl) {
  constexpr int THREADS = Tile::kThreads;
  constexpr uint32_t kNone = 0xffffffffu;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename Tile::Shared sh;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_first, s_beyond, s_last, s_end;
  __shared__ RunKey s_w;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes + Tile::kSlotBytes);
  const TopPlan& plan = ctrl->top;
  const uint32_t par = plan.src_parity;
  const Elem* src = par ? Y : X;
  const bool in_place = par == 0;
  if (plan.complete) {  // in order: at most to be copied
    if (!in_place)
      for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * THREADS)
        store_elem(X + i, load_elem_stream(Y + i));
    return;
  }
  if (error_raised(ctrl)) return;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t bar = smem_u32(&s_bar);
  if (tid == 0) {
    s_w = run_key(plan);
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  const bool clamped = plan.hb1 < 64u;
  const uint32_t shift = run_key(plan).shift;
  const uint32_t parts = (uint32_t)(((uint64_t)n + stride - 1u) / stride);
  uint32_t phase = 0;
  for (uint32_t part = blockIdx.x; part < parts; part += gridDim.x) {
    uint32_t g = (uint32_t)((uint64_t)part * stride);
    const uint32_t limit = (uint32_t)min((uint64_t)g + stride, (uint64_t)n);
    bool known = part == 0;  // g is known to be a run's start
    while (g < limit) {
      const uint32_t w0 = known ? g : g - 1u;
      const uint32_t cnt = min(kCap, n - w0);
      // src[w0, w0 + cnt) into in[]
      __syncthreads();  // in[] is no longer read
      if (tid == 0) {
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(bar, cnt * (uint32_t)sizeof(Elem));
        for (uint32_t o = 0; o < cnt; o += 2048u)
          bulk_g2s(smem_u32(in + o), src + w0 + o, min(2048u, cnt - o) * (uint32_t)sizeof(Elem), bar);
      }
      const bool ok = mbar_wait_bounded(bar, phase);
      phase ^= 1u;
      if (!ok) record_error(ctrl, kStatusTimeout, kWhereBulkCopy);
      if (__syncthreads_or(!ok)) return;
      // first run start, first one at or after `limit`, last one (tile
      // positions; kNone, cnt and 0 when there is none), by one warp each
      if (warp == 0) {
        const uint32_t e = run_start(in, s_w, run_of(s_w, in[cnt - 1u].key), cnt - 1u);
        if (lane_id() == 0) s_last = e;
      } else if (warp == 1) {
        const uint32_t l = limit - w0;
        const uint32_t e = l < cnt ? run_end<false>(in, s_w, run_of(s_w, in[l - 1u].key), l, cnt) : cnt;
        if (lane_id() == 0) s_beyond = e;
      } else if (warp == 2) {
        const uint32_t e = known ? 0u : run_end<false>(in, s_w, run_of(s_w, in[0].key), 1u, cnt);
        if (lane_id() == 0) s_first = e < cnt ? e : kNone;
      }
      __syncthreads();
      const uint32_t first = s_first, beyond = s_beyond, last = s_last;
      const bool at_end = w0 + cnt == n;
      if (first == kNone) {  // inside a run that an earlier part has
        if (at_end || w0 + cnt >= limit) break;
        if (warp == 0) {
          const uint32_t e = run_end<true>(src, s_w, run_of(s_w, in[0].key), w0 + cnt, limit);
          if (lane_id() == 0) s_end = e;
        }
        __syncthreads();
        g = s_end;
        known = true;
        continue;
      }
      if (w0 + first >= limit) break;
      const uint32_t end = beyond < cnt ? beyond : at_end ? cnt : last;
      known = true;
      if (end > first) {
        g = w0 + end;
        if (end - first == 1u && in_place) continue;
        // whole runs: bins over their range of keys (clamped keys can lie
        // outside it: then over the tile's own range)
        uint64_t base = 0, range = 0;
        if (!clamped) {
          base = in[first].key >> shift << shift;
          range = (in[end - 1u].key | ((1ull << shift) - 1ull)) - base;
        }
        Elem* out = X + w0 + first;
        Tile::sort(in, first, end, base, range, slot, bins, sh, in_place,
                   [&](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); });
      } else if (first > 0u) {  // one run from `first`, not whole in the tile yet
        g = w0 + first;
      } else {  // a run longer than a tile
        if (warp == 0) {
          const uint32_t e = run_end<true>(src, s_w, run_of(s_w, in[0].key), w0 + cnt, n);
          push_run(ctrl, chunks, unsorted, n, w0, e);
          if (lane_id() == 0) s_end = e;
        }
        __syncthreads();
        g = s_end;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// runs longer than a tile

// Every CTA of the (co-resident) grid arrives; false when the wait ran out or
// an error was raised.
__device__ __forceinline__ bool grid_barrier(Ctrl* ctrl, uint32_t* round) {
  __shared__ bool s_ok;
  *round += 1u;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&ctrl->top.barrier, 1u);
    const uint32_t want = *round * gridDim.x;
    uint32_t it = 0, ns = 32;
    bool ok = true;
    while (ld_acquire_u32(&ctrl->top.barrier) < want) {
      if (++it >= kSpinLimit || ((it & 63u) == 0u && error_raised(ctrl))) {
        record_error(ctrl, kStatusTimeout, kWhereGridBarrier);
        ok = false;
        break;
      }
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok;
}

__device__ __forceinline__ Elem load_elem_l2(const Elem* p) {
  Elem e;  // L2 only: another CTA has written it since this kernel began
  asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(e.key), "=l"(e.val) : "l"(p) : "memory");
  return e;
}

// One warp: elements of a among the first d of the stable merge of a and b.
__device__ __forceinline__ uint32_t merge_split(const Elem* a, uint32_t la, const Elem* b, uint32_t lb, uint32_t d) {
  uint32_t lo = d > lb ? d - lb : 0u, hi = min(d, la);
  while (lo < hi) {
    const uint32_t step = (hi - lo - 1u) / 32u + 1u;
    const uint64_t i = (uint64_t)lo + (uint64_t)lane_id() * step;
    const bool before = i < hi && ld_relaxed_u64(&a[i].key) <= ld_relaxed_u64(&b[d - 1u - (uint32_t)i].key);
    const uint32_t t = (uint32_t)__popc(__ballot_sync(0xffffffffu, before));
    if (t == 0) return lo;
    const uint64_t nhi = (uint64_t)lo + (uint64_t)t * step;
    hi = nhi < hi ? (uint32_t)nhi : hi;
    lo += (t - 1u) * step + 1u;
  }
  return lo;
}

// Runs that do not fit in a tile. Usual keys leave none and the kernel returns
// at once. Heavy keys do: one key fills the run, it is in order and only read
// (or copied into X). The rest is sorted by chunks of a tile and pairwise
// stable merges, all CTAs on one round at a time. A cooperative launch: the
// grid barrier needs every CTA resident.
__global__ void __launch_bounds__(Tile::kThreads, 2)
    k_top_merge(Elem* X, Elem* Y, uint32_t n, const RunChunk* __restrict__ chunks, uint32_t* unsorted, Ctrl* ctrl) {
  constexpr int K = Tile::kItems, THREADS = Tile::kThreads;
  const uint32_t total = ctrl->top.num_chunks;
  if (total == 0u || error_raised(ctrl)) return;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename Tile::Shared sh;
  __shared__ uint32_t s_split[2];
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes + Tile::kSlotBytes);
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t par = ctrl->top.src_parity;
  const Elem* src = par ? Y : X;
  const uint32_t rounds = ctrl->top.max_rounds;
  uint32_t barriers = 0;
  // runs in order stay (or are copied); the others are marked. Each warp reads
  // its part of a chunk and the element after it, nine loads at a time.
  for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
    const RunChunk t = chunks[c];
    const Elem* run = src + t.b;
    const uint32_t len = t.e - t.b, at = t.k * kCap + warp * 32u * K;
    const uint32_t m = min(len - t.k * kCap, kCap);  // the chunk's
    Elem e[K];
#pragma unroll
    for (int k = 0; k < K; k++) e[k] = load_elem_stream(run + min(at + (uint32_t)k * 32u + lane_id(), len - 1u));
    const uint64_t after = at + 32u * K < len ? run[at + 32u * K].key : ~0ull;
    bool inversion = false;
#pragma unroll
    for (int k = 0; k < K; k++) {
      uint64_t next = __shfl_down_sync(0xffffffffu, e[k].key, 1);
      const uint64_t head = k + 1 < K ? __shfl_sync(0xffffffffu, e[k + 1 < K ? k + 1 : k].key, 0) : after;
      if (lane_id() == 31) next = head;
      inversion |= e[k].key > next;
      const uint32_t i = warp * 32u * K + (uint32_t)k * 32u + lane_id();
      if (par && i < m) store_elem(X + t.b + t.k * kCap + i, e[k]);
    }
    if (__any_sync(0xffffffffu, inversion) && lane_id() == 0) unsorted[t.run] = 1u;
  }
  if (!grid_barrier(ctrl, &barriers)) return;
  auto rounds_of = [](const RunChunk& t) { return 32u - (uint32_t)__clz((int)((t.e - t.b - 1u) / kCap)); };
  // chunks, each into the buffer from which the merges end in X
  bool any = false;
  for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
    const RunChunk t = chunks[c];
    if (!ld_relaxed_u32(unsorted + t.run)) continue;
    any = true;
    const uint32_t lo = t.b + t.k * kCap, m = min(t.e - lo, kCap);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t i = tid + (uint32_t)k * THREADS;
      if (i < m) in[i] = load_elem_l2(src + lo + i);
    }
    __syncthreads();
    Elem* out = ((rounds_of(t) & 1u) ? Y : X) + lo;
    Tile::sort(in, 0, m, 0, 0, slot, bins, sh, out == src + lo,
               [&](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); });
  }
  // no run to merge anywhere: the marks are the same for every CTA
  if (!any) {
    for (uint32_t c = tid; c < total; c += THREADS) any |= ld_relaxed_u32(unsorted + chunks[c].run) != 0u;
  }
  if (!__syncthreads_or(any)) return;
  if (!grid_barrier(ctrl, &barriers)) return;
  for (uint32_t r = 0; r < rounds; r++) {
    for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
      const RunChunk t = chunks[c];
      const uint32_t mine = rounds_of(t);
      if (r >= mine || !ld_relaxed_u32(unsorted + t.run)) continue;
      const Elem* from = (((mine - r) & 1u) ? Y : X) + t.b;
      Elem* to = (((mine - r) & 1u) ? X : Y) + t.b;
      const uint32_t len = t.e - t.b, pos = t.k * kCap, cnt = min(kCap, len - pos);
      const uint64_t half = (uint64_t)kCap << r;
      const uint32_t base = (uint32_t)(pos / (2u * half) * (2u * half));
      const uint32_t la = (uint32_t)min(half, (uint64_t)(len - base));
      const uint32_t lb = (uint32_t)min(half, (uint64_t)(len - base - la));
      const Elem* a = from + base;
      const Elem* b = a + la;
      const uint32_t d0 = pos - base, d1 = d0 + cnt;
      __syncthreads();
      if (warp < 2) {
        const uint32_t i = merge_split(a, la, b, lb, warp ? d1 : d0);
        if (lane_id() == 0) s_split[warp] = i;
      }
      __syncthreads();
      const uint32_t i0 = s_split[0], na = s_split[1] - i0, j0 = d0 - i0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t i = tid + (uint32_t)k * THREADS;
        if (i < cnt) in[i] = load_elem_l2(i < na ? a + i0 + i : b + j0 + (i - na));
      }
      uint16_t* id = reinterpret_cast<uint16_t*>(slot);
      uint16_t* order = id + kCap;
      for (uint32_t i = tid; i < cnt; i += THREADS) id[i] = (uint16_t)i;
      __syncthreads();
      Tile::merge_parts(in, id, order, na, cnt - na);
      __syncthreads();
      for (uint32_t i = tid; i < cnt; i += THREADS) store_elem(to + pos + i, in[order[i]]);
    }
    if (!grid_barrier(ctrl, &barriers)) return;
  }
}

// ---------------------------------------------------------------------------
// driver

int top_run(Elem* X, Elem* Y, unsigned char* ws, const Layout& L, cudaStream_t st) {
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(ws);
  const uint32_t n = L.n;
  if (n <= SmallHalf::kCap) return small_sort<512>(X, L, ctrl, st);
  if (n <= SmallFull::kCap) return small_sort<1024>(X, L, ctrl, st);
  DeviceInfo dev;
  if (int rc = current_device_info(&dev)) return rc;
  uint32_t* hist = reinterpret_cast<uint32_t*>(ws + L.off_hist);
  uint32_t* gstart = reinterpret_cast<uint32_t*>(ws + L.off_gstart);
  uint64_t* ring = reinterpret_cast<uint64_t*>(ws + L.off_ring);
  const SampleRule rule = sample_rule(n);
  if (cudaFuncSetAttribute(k_top_sample, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSampleSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_top_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile::kSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_top_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile::kSmem) != cudaSuccess)
    return 5;
  {
    ProfScope prof("top_sample", st);
    k_top_sample<<<1, kSampleThreads, kSampleSmem, st>>>(X, n, rule, hist, ctrl);
  }
  {
    // four CTAs per SM, fewer when they would have under four rounds of reads each
    const uint32_t per_cta = (uint32_t)kTopHistThreads * kTopHistUnroll * 4u;
    const uint32_t grid = std::max<uint32_t>(1u, std::min<uint32_t>((n - 1u) / per_cta + 1u, (uint32_t)dev.sm_count * 4u));
    ProfScope prof("top_hist", st);
    k_top_hist<<<grid, kTopHistThreads, 0, st>>>(X, n, hist, gstart, reinterpret_cast<uint4*>(ring),
                                                 (uint64_t)L.ring_tiles * 256u * 8u / 16u, L.stat_bits, L.stat_digits,
                                                 L.api_bits, L.sub, ctrl);
  }
  if (cudaPeekAtLastError() != cudaSuccess) return 5;
  for (uint32_t p = 0; p < rule.tmax; p++)
    if (int rc = onesweep_top_pass(X, Y, n, (int)p, gstart + p * 256u, ring, L.ring_tiles, ctrl, dev, st)) return rc;
  RunChunk* chunks = reinterpret_cast<RunChunk*>(ring);
  uint32_t* unsorted = reinterpret_cast<uint32_t*>(chunks + max_chunks(n));
  {
    // A tile is left a run short on average (its last run is not whole), so a
    // part of `per` tiles is as long as its runs fill `per` tiles, or, with runs
    // that fill a tile by themselves, as `per` runs. Parts of 1 to 16 tiles:
    // enough of them for six rounds of two CTAs per SM, and else few, since the
    // run across a part's start is read twice.
    const uint32_t run = (uint32_t)((double)n / std::pow(256.0, (double)rule.tmin));
    const uint32_t fill = std::max(run, kCap - std::min(kCap, run + run / 2u));
    const uint32_t per = std::max<uint32_t>(1u, std::min<uint32_t>(16u, n / fill / ((uint32_t)dev.sm_count * 12u)));
    const uint32_t stride = per * fill;
    const uint32_t grid = (uint32_t)(((uint64_t)n + stride - 1u) / stride);
    ProfScope prof("top_finish", st);
    k_top_finish<<<grid, Tile::kThreads, Tile::kSmem, st>>>(X, Y, n, stride, chunks, unsorted, ctrl);
  }
  if (cudaPeekAtLastError() != cudaSuccess) return 5;
  {
    uint32_t nn = n;
    const RunChunk* cc = chunks;
    void* args[] = {&X, &Y, &nn, &cc, &unsorted, &ctrl};
    ProfScope prof("top_merge", st);
    if (cudaLaunchCooperativeKernel((const void*)k_top_merge, dim3((uint32_t)dev.sm_count * 2u), dim3(Tile::kThreads), args,
                                    Tile::kSmem, st) != cudaSuccess)
      return 5;
  }
  return 0;
}

}  // namespace lsb
