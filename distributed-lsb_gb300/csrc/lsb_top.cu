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

#include "lsb_top.cuh"

namespace lsb {

// ---------------------------------------------------------------------------
// one CTA, one launch

// Bound by latency: one read of the tile, nine barriers, one write. Twelve
// launches (clears, the histogram, the plan, eight passes and the copy back)
// took 112 us for 1000 elements with the array's own copy; this takes 11.3 us.
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
  TS::sort(in, 0, n, 0, 0, slot, bins, sh, true, Uneven::kBits, [&](bool on, uint32_t r, const Elem& e) { store_elem_if(on, a + r, e); });
  // s_diff: the sort's barriers lie between
  if (threadIdx.x == 0)
    write_plan(ctrl, (uint64_t)s_diff[1] << 32 | s_diff[0], n, bits, num_digits, api_bits, sub);
}

// 1024 threads hold up to 9216 elements (212 KB of shared memory); up to half
// that 512 threads do, whose barriers cost less.
using SmallHalf = TileSort<512, 9>;
using SmallFull = TileSort<1024, 9>;

template <int THREADS>
static int small_sort(Elem* X, const Layout& L, Ctrl* ctrl, cudaStream_t st) {
  auto kern = k_small_sort<THREADS, 9>;
  const size_t smem = TileSort<THREADS, 9>::kSmem;
  static std::atomic<uint64_t> allowed;  // of this instance
  if (!allow_smem((const void*)kern, smem, &allowed)) return 5;
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
//   k_onesweep    one stable pass per digit, lowest first, as many as even keys need,
//   k_onesweep_rest  and any further ones in one launch
//   k_top_finish  the array is now in the order of the digits' windows; each
//                 CTA takes whole runs of equal windows, up to a tile of them
//                 at a time, and sorts them by the whole key
//   k_top_merge   runs longer than a tile (the sample missed them): checked,
//                 and sorted by chunks and merges unless they are in order
// Keys of which so many digits would be needed, or that the last step would take
// long for, are passed over by every byte in which they differ (choose_passes).
// The result does not depend on the sample: it only decides how short the
// runs are, and so the time. Measured (GB300, sort alone): 2^24 uniform 1.10 ->
// 0.47 ms, 2^28 15.0 -> 6.5 ms, 2^29 29.4 -> 13.7 ms (two passes), 2^30 58.6 ->
// 30.9 ms (three), 2^28 Zipf 16.0 -> 9.4 ms (four; heavy keys stay in order),
// against eight passes.

// Longest even runs for the small tile (one and a half of them fit) and for the
// big one (six standard deviations below it); for the usual one: kMeanRun.
constexpr uint32_t kSmallRun = 1700, kBigRun = 8640;
constexpr int kTopSample = 4;  // keys per thread of the sample: 4096
constexpr int kTopHistThreads = 512;
constexpr int kTopHistUnroll = 4;

// Bound by latency (one CTA: scattered reads, a sort of the keys, two counts: with
// 1024 keys 13 us under events, whatever the keys are, with 4096 up to 55); it also clears what the later kernels count in,
// in place of three memsets.
template <int S>
__global__ void __launch_bounds__(kSampleThreads, 1)
    k_top_sample(const Elem* __restrict__ data, uint32_t n, SampleRule rule, uint32_t* __restrict__ hist, Ctrl* ctrl) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename SampleTile<S>::Shared sh;
  __shared__ SampleStats s_stats;
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < kCtrlBytes / 4u; i += kSampleThreads) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
  for (uint32_t i = tid; i < 8u * 256u; i += kSampleThreads) hist[i] = 0u;
  clear_stats(s_stats);
  const uint64_t* s = sample_keys<S>(data, n, smem, sh);
  const uint64_t first = s[0], span = first ^ s[S * kSampleThreads - 1];
  const uint32_t hb1 = span ? 64u - (uint32_t)__clzll((long long)span) : 64u;
  const SampleChoice c = choose_passes<S, true>(s, hb1, rule, 0u, s_stats, 0ull, [=](uint32_t t) { return hb1 > 8u * t ? hb1 - 8u * t : 0u; });
  if (tid == 0) {
    TopPlan& p = ctrl->top;
    const bool block = hb1 < 64u && !c.plain;
    p.passes = c.plain ? 8u : c.passes;
    p.skewed = (c.skewed ? 1u : 0u) | (c.dups ? 2u : 0u);
    p.big = c.big ? 1u : 0u;
    p.hb1 = c.plain ? 64u : hb1;
    p.clamp = block ? 1u : 0u;
    p.lo = block ? first >> hb1 << hb1 : 0ull;
    p.hi = block ? p.lo | ((1ull << hb1) - 1ull) : ~0ull;
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

// The same for five to eight digits: bytes of two words. (2^26 keys, five digits:
// 590 us a key and a digit at a time, 178 so.)
template <bool CLAMP>
__device__ __noinline__ void count_many_windows(const Elem* __restrict__ data, uint32_t n, const TopPlan& p,
                                                uint32_t* h, uint64_t first, uint64_t* diff) {
  const uint32_t lane = lane_id();
  const uint64_t warps_total = (uint64_t)gridDim.x * (kTopHistThreads / 32);
  const uint64_t gw = (uint64_t)blockIdx.x * (kTopHistThreads / 32) + (threadIdx.x >> 5);
  constexpr uint32_t chunk = 32u * kTopHistUnroll;
  const uint64_t block_lo = p.lo, block_hi = p.hi;
  const uint32_t left = 64u - p.hb1;
  const int low = 8 - (int)p.passes;  // lowest byte that is a digit
  uint64_t acc = 0;
  auto digits_of = [&](uint64_t key) {
    return CLAMP ? (key < block_lo ? 0ull : key > block_hi ? ~0ull : key << left) : key << left;
  };
  const uint64_t full_end = (uint64_t)n / chunk * chunk;
  for (uint64_t base = gw * chunk; base < full_end; base += warps_total * chunk) {
    uint64_t key[kTopHistUnroll];
#pragma unroll
    for (int u = 0; u < kTopHistUnroll; u++) key[u] = load_elem_stream(data + base + (uint64_t)u * 32u + lane).key;
#pragma unroll
    for (int u = 0; u < kTopHistUnroll; u++) {
      acc |= key[u] ^ first;
      const uint64_t d = digits_of(key[u]);
#pragma unroll
      for (int half = 1; half >= 0; half--) {
        const uint32_t w = (uint32_t)(d >> (32 * half));
        const uint32_t x = __reduce_or_sync(0xffffffffu, w ^ __shfl_sync(0xffffffffu, w, 0));
#pragma unroll
        for (int t = 3; t >= 0; t--) {
          if (half == 0 && t < low) break;
          uint32_t* c = &h[(4 * half + t - low) * 256 + ((w >> (8 * t)) & 255u)];
          if ((x >> (8 * t)) & 255u) atomicAdd(c, 1u);
          else if (lane == 0) atomicAdd(c, 32u);
        }
      }
    }
  }
  for (uint64_t i = full_end + (uint64_t)blockIdx.x * kTopHistThreads + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * kTopHistThreads) {
    const uint64_t key = load_elem_stream(data + i).key;
    acc |= key ^ first;
    const uint64_t d = digits_of(key);
    for (int t = low; t < 8; t++) atomicAdd(&h[(t - low) * 256 + ((d >> (8 * t)) & 255u)], 1u);
  }
  *diff = acc;
}

__global__ void __launch_bounds__(kTopHistThreads, 4)
    k_top_hist(const Elem* __restrict__ data, uint32_t n, uint32_t* __restrict__ hist, uint32_t* __restrict__ gstart,
               uint4* __restrict__ ring, uint64_t ring_words, int bits, int num_digits, int api_bits, int sub,
               uint32_t single, Ctrl* ctrl) {
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
  if (p.clamp) {
    switch (T) {
      case 1: count_windows<1, true>(data, n, p, h, first, &diff); break;
      case 2: count_windows<2, true>(data, n, p, h, first, &diff); break;
      case 3: count_windows<3, true>(data, n, p, h, first, &diff); break;
      case 4: count_windows<4, true>(data, n, p, h, first, &diff); break;
      default: count_many_windows<true>(data, n, p, h, first, &diff); break;
    }
  } else {
    switch (T) {
      case 1: count_windows<1, false>(data, n, p, h, first, &diff); break;
      case 2: count_windows<2, false>(data, n, p, h, first, &diff); break;
      case 3: count_windows<3, false>(data, n, p, h, first, &diff); break;
      case 4: count_windows<4, false>(data, n, p, h, first, &diff); break;
      default: count_many_windows<false>(data, n, p, h, first, &diff); break;
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
  scan_digits(hist, gstart, n, T, &s_const);
  __syncthreads();
  if (threadIdx.x == 0) {
    TopPlan& q = ctrl->top;
    const uint64_t d = (uint64_t)__ldcg(&q.diff[1]) << 32 | __ldcg(&q.diff[0]);
    if (single) {  // every pass runs, so that the result lands in its place whatever the digits
      const uint32_t constant = single == 1u ? s_const & 1u : 0u;
      q.copy = constant;
      q.run_mask = (1u << T) - 1u;
      q.par_mask = 2u;
      ctrl->skip_mask_lo = constant;
      ctrl->passes_run = single - constant;
      ctrl->final_copy = constant;
      ctrl->num_passes = single;
      ctrl->api_bits = (uint32_t)api_bits;
      ctrl->sub = (uint32_t)sub;
      ctrl->n = n;
      return;
    }
    chain_passes(q, T, s_const);
    // keys in the block, as usual: no pass need look
    const bool inside = q.hb1 >= 64u || ((d | (first ^ q.lo)) >> q.hb1) == 0;
    q.clamp = inside ? 0u : 1u;
    q.complete = (d == 0 || (q.hb1 <= 8u * T && inside)) ? 1u : 0u;
    write_plan(ctrl, d, n, bits, num_digits, api_bits, sub);
  }
}

// ---------------------------------------------------------------------------
// the runs

// Sorts the runs in place (data in X) or from Y into X. The array is cut every
// `stride` elements; a CTA takes the runs that start in its part, as many whole
// runs at a time as fit in a tile: it brings in a tile's worth from where it
// stands by one bulk copy, and sorts the whole runs in it (sort_runs).
// 2^30 elements after three passes (runs of 64): 7.7 ms with tiles of 4608 in
// two CTAs per SM, 7.1 ms (4.8 TB/s of the 32 bytes per element) with 2304 in
// four, whose phases overlap better; three of 3072 take 7.4, one of 9216 9.2.
// Bound by the shared-memory pipe (70 % busy: 50 wavefronts and 180
// instructions per 32 elements) at 32 resident warps per SM. (Digits of 7 bits
// make a pass 4 % faster and the runs eight times as long, which costs the
// small tiles as much: 27.7 ms for passes and runs either way.)
template <class TS, int CTAS>
__global__ void __launch_bounds__(TS::kThreads, CTAS)
    k_top_finish(Elem* __restrict__ X, Elem* __restrict__ Y, uint32_t n, uint32_t stride,
                 RunChunk* __restrict__ chunks, uint32_t* __restrict__ unsorted, uint32_t big, Ctrl* ctrl) {
  constexpr int THREADS = TS::kThreads;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename TS::Shared sh;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ RunMarks s_marks;
  __shared__ RunKey s_w;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes + TS::kSlotBytes);
  const TopPlan& plan = ctrl->top;
  if (plan.big != big) return;
  const uint32_t par = plan.src_parity;
  const Elem* src = par ? Y : X;
  if (plan.complete) {  // in order: at most to be copied
    if (par)
      for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * THREADS)
        store_elem(X + i, load_elem_stream(Y + i));
    return;
  }
  if (error_raised(ctrl)) return;
  const uint32_t bar = smem_u32(&s_bar);
  if (threadIdx.x == 0) {
    s_w = run_key(plan);
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  const bool clamped = plan.clamp != 0u, skewed = (plan.skewed & 1u) != 0u, dups = (plan.skewed & 2u) != 0u;
  const uint32_t shift = run_key(plan).shift;
  const uint32_t parts = (uint32_t)(((uint64_t)n + stride - 1u) / stride);
  uint32_t phase = 0;
  auto load = [&](uint32_t from, uint32_t cnt) { return load_tile_bulk(in, src + from, cnt, bar, &phase, ctrl); };
  auto long_run = [&](uint32_t b, uint32_t e) { push_run(ctrl, chunks, unsorted, n, b, e, par); };
  for (uint32_t part = blockIdx.x; part < parts; part += gridDim.x) {
    const uint32_t g = (uint32_t)((uint64_t)part * stride);
    const uint32_t limit = (uint32_t)min((uint64_t)g + stride, (uint64_t)n);
    if (!sort_runs<TS>(src, X, n, g, limit, part == 0, s_w, clamped, skewed, dups, shift, in, slot, bins, sh, s_marks, load,
                         long_run))
      return;
  }
}

// ---------------------------------------------------------------------------
// runs longer than a tile

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
// stable merges. Step 0 checks, step 1 sorts the chunks, step 2 + r is round r of
// the merges; an item of work is a few chunks' share of a step, and the items of all
// steps are handed out in order by one ticket. An item waits until the steps before its own
// are finished. Whoever has those items is running and waits for earlier ones
// only, so no CTA needs another one to be resident, and the stream may own fewer
// SMs than the device has.
__global__ void __launch_bounds__(Tile::kThreads, 2)
    k_top_merge(Elem* X, Elem* Y, uint32_t n, const RunChunk* __restrict__ chunks, uint32_t* unsorted, Ctrl* ctrl) {
  constexpr int K = Tile::kItems, THREADS = Tile::kThreads;
  const uint32_t total = ctrl->top.num_chunks;
  if (total == 0u || error_raised(ctrl)) return;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename Tile::Shared sh;
  __shared__ uint32_t s_split[2], s_item;
  __shared__ bool s_go;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes + Tile::kSlotBytes);
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t steps = 2u + ctrl->top.max_rounds;
  // sixteen items for each CTA: an item costs a trip to the ticket and two barriers, and
  // few of them leave CTAs idle at a step's end (2^28 Zipf keys, 58000 chunks in order:
  // 11.2 ms the sort with an item per chunk, 10.2 so, 10.1 with eight for each; keys
  // that occur a thousand times: 16.1 with one for each, 15.4 with eight, 15.05 so)
  const uint32_t items = min(total, gridDim.x * 16u);
  auto rounds_of = [](const RunChunk& t) { return 32u - (uint32_t)__clz((int)((t.e - t.b - 1u) / kCap)); };
  uint32_t step_now = 0;
  if (tid == 0) s_item = atomicAdd(&ctrl->top.merge_ticket, 1u);
  __syncthreads();
  for (;;) {
    const uint32_t item = s_item, step = item / items;
    if (step >= steps) return;
    if (step != step_now) {
      if (tid == 0) {
        // when the check has found nothing to merge, every later step is left out
        bool go = step_now != 0u || (wait_arrivals(&ctrl->top.merge_done, items, ctrl) &&
                                     ld_relaxed_u32(&ctrl->top.merge_any) != 0u);
        go = go && wait_arrivals(&ctrl->top.merge_done, step * items, ctrl);
        __threadfence();
        s_go = go;
      }
      __syncthreads();
      if (!s_go) return;
      step_now = step;
    }
    for (uint32_t c = item % items; c < total; c += items) {  // (neighbours are chunks of one run: all to be merged, or none)
      const RunChunk t = chunks[c];
      const uint32_t len = t.e - t.b, pos = t.k * kCap, cnt = min(kCap, len - pos);
      if (step == 0u) {
        // runs in order stay (or are copied); the others are marked. Each warp reads
        // its part of a chunk and the element after it, nine loads at a time.
        const Elem* run = (t.par ? Y : X) + t.b;
        const uint32_t at = pos + warp * 32u * K;
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
          if (t.par && i < cnt) store_elem(X + t.b + pos + i, e[k]);
        }
        if (__any_sync(0xffffffffu, inversion) && lane_id() == 0) {
          unsorted[t.run] = 1u;
          ctrl->top.merge_any = 1u;
        }
      } else if (ld_relaxed_u32(unsorted + t.run)) {
        if (step == 1u) {  // a chunk, into the buffer from which the merges end in X
          const Elem* src = (t.par ? Y : X) + t.b + pos;
          __syncthreads();
#pragma unroll
          for (int k = 0; k < K; k++) {
            const uint32_t i = tid + (uint32_t)k * THREADS;
            if (i < cnt) in[i] = load_elem_l2(src + i);
          }
          __syncthreads();
          Elem* out = ((rounds_of(t) & 1u) ? Y : X) + t.b + pos;
          Tile::sort(in, 0, cnt, 0, 0, slot, bins, sh, out == src, Uneven::kSpread,
                     [&](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); });
        } else if (const uint32_t r = step - 2u, mine = rounds_of(t); r < mine) {
          const Elem* from = (((mine - r) & 1u) ? Y : X) + t.b;
          Elem* to = (((mine - r) & 1u) ? X : Y) + t.b;
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
      }
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(&ctrl->top.merge_done, 1u);
      // not sooner: a CTA would hold two items of a step while others have none
      s_item = atomicAdd(&ctrl->top.merge_ticket, 1u);
    }
    __syncthreads();
  }
}

size_t top_list_bytes(uint32_t n) { return (size_t)max_chunks(n) * (sizeof(RunChunk) + 4u); }

int top_merge(Elem* X, Elem* Y, uint32_t n, RunChunk* chunks, uint32_t* unsorted, Ctrl* ctrl, const DeviceInfo& dev,
              cudaStream_t st) {
  static std::atomic<uint64_t> allowed;
  if (!allow_smem((const void*)k_top_merge, Tile::kSmem, &allowed)) return 5;
  ProfScope prof("top_merge", st);
  k_top_merge<<<(uint32_t)dev.sm_count * 2u, Tile::kThreads, Tile::kSmem, st>>>(X, Y, n, chunks, unsorted, ctrl);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 5;
}

// ---------------------------------------------------------------------------
// one digit

// Plan of a single pass over the `passes` bytes below bit hb1; it also clears
// what the later kernels count in.
__global__ void __launch_bounds__(kSampleThreads) k_pass_plan(uint32_t* __restrict__ hist, uint32_t hb1, uint32_t passes, Ctrl* ctrl) {
  for (uint32_t i = threadIdx.x; i < kCtrlBytes / 4u; i += kSampleThreads) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
  for (uint32_t i = threadIdx.x; i < passes * 256u; i += kSampleThreads) hist[i] = 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->top.passes = passes;
    ctrl->top.hb1 = hb1;
  }
}

static int top_hist(const Elem* X, unsigned char* ws, const Layout& L, uint32_t single, const DeviceInfo& dev, cudaStream_t st) {
  // four CTAs per SM, fewer when they would have under four rounds of reads each
  const uint32_t per_cta = (uint32_t)kTopHistThreads * kTopHistUnroll * 4u;
  const uint32_t grid = std::max<uint32_t>(1u, std::min<uint32_t>((L.n - 1u) / per_cta + 1u, (uint32_t)dev.sm_count * 4u));
  ProfScope prof("top_hist", st);
  k_top_hist<<<grid, kTopHistThreads, 0, st>>>(
      X, L.n, reinterpret_cast<uint32_t*>(ws + L.off_hist), reinterpret_cast<uint32_t*>(ws + L.off_gstart),
      reinterpret_cast<uint4*>(ws + L.off_ring), ((uint64_t)(L.n - 1u) / onesweep_top_tile(0) + 1u) * 256u * 8u / 16u, L.stat_bits, L.stat_digits,
      L.api_bits, L.sub, single, reinterpret_cast<Ctrl*>(ws));
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 5;
}

// globalShuffle of an 8-bit digit (mpi/mpi_lsbsort.cpp:493-589), or of two in
// turn through mid. Clears, histogram and plan take two launches, not seven: with
// the count of its digits, a 16-bit digit of 65537 elements 122 -> 75 us, of 2^26
// 1409 -> 1352.
bool top_pass_fits(const Layout& L) {
  return L.bits == 8 && L.tile_elems == onesweep_top_tile(0) && L.ring_tiles >= (L.n - 1u) / L.tile_elems + 1u;
}
int top_pass_run(const Elem* src, Elem* mid, Elem* dst, int first_digit, unsigned char* ws, const Layout& L, cudaStream_t st) {
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(ws);
  DeviceInfo dev;
  if (int rc = current_device_info(&dev)) return rc;
  const uint32_t passes = (uint32_t)L.num_digits;
  const uint32_t* gstart = reinterpret_cast<const uint32_t*>(ws + L.off_gstart);
  uint64_t* ring = reinterpret_cast<uint64_t*>(ws + L.off_ring);
  {
    ProfScope prof("plan", st);
    k_pass_plan<<<1, kSampleThreads, 0, st>>>(reinterpret_cast<uint32_t*>(ws + L.off_hist),
                                              8u * ((uint32_t)first_digit + passes), passes, ctrl);
  }
  if (int rc = top_hist(src, ws, L, passes, dev, st)) return rc;
  Elem* in = const_cast<Elem*>(src);  // read only: pass 0 reads X
  if (int rc = onesweep_top_pass(in, passes == 1u ? dst : mid, L.n, 0, gstart, ring, L.ring_tiles, ctrl, SegDesc{}, 0, 0u, dev, st))
    return rc;
  if (passes == 1u) return 0;
  return onesweep_top_pass(dst, mid, L.n, 1, gstart + 256u, ring, L.ring_tiles, ctrl, SegDesc{}, 0, 0u, dev, st);
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
  if (n <= mid_limit(dev)) {
    const int rc = mid_run(X, Y, ws, L, dev, st);
    if (rc != kMidRefused) return rc;
  }
  uint32_t* hist = reinterpret_cast<uint32_t*>(ws + L.off_hist);
  uint32_t* gstart = reinterpret_cast<uint32_t*>(ws + L.off_gstart);
  uint64_t* ring = reinterpret_cast<uint64_t*>(ws + L.off_ring);
  // The tile of the last step. The big one is slower (one CTA per SM) but holds
  // runs twice as long. Where it can save the second or third pass, it is launched
  // beside the other one and the sample decides, which may find keys denser than
  // even ones: 2^29 uniform keys 15.5 -> 13.7 ms, 2^28 of a 29-bit range 8.2 -> 6.7
  // ms, 1.5 10^6 neighbours 101 -> 86 us (uniform keys 96 -> 95; as the only tile there it
  // took 221 instead of 111 us for keys that occur a thousand times). Up to 7600 elements in a
  // run of one pass: 2.05 10^6 uniform keys 103 -> 93 us, but with a thousandth of
  // sentinels 132 -> 179. (After the one or two top windows only: behind more of them are clusters,
  // whose runs it cannot tell from longer ones.) Else even runs up to kSmallRun leave the small one half full or better,
  // with six standard deviations of room.
  const uint32_t least = passes_for((float)n, (float)kMeanRun);
  const uint32_t big_passes = least == 2u && n <= 256u * 7600u ? 1u : n > (1u << 27) && n <= 65536u * kBigRun ? 2u : 0u;
  const double even_run = (double)n / std::pow(256.0, (double)least);
  const bool small_tile = even_run <= (double)kSmallRun;
  // Windows per element after which a heavy key is alone in its run: 16 ask for three
  // passes up to 2^20 elements and for four up to 2^28, and 4 for four up to 2^30. With 2,
  // a pass less, 2 to 5 10^6 Zipf keys take 234 and 350 us, not 150 and 266; with 16 above 2^28,
  // a pass more, 3 10^8 of them 13.6 ms, not 11.7. (Half zeros and half even keys take
  // less with 2: 151 -> 125, 268 -> 258 us.)
  // a smaller sample decides as well for fewer elements, and 5 us sooner
  const bool short_sample = n < (1u << 26);
  const uint32_t mean_run = small_tile ? kSmallRun : kMeanRun;
  const uint32_t tile = small_tile ? SmallTile::kCap : Tile::kCap;
  SampleRule rule = sample_rule(n, kSampleThreads * (short_sample ? 1u : (uint32_t)kTopSample), tile, mean_run, mean_run,
                                n <= (1u << 28) ? 16.0f : 4.0f);
  if (big_passes) {
    const SampleRule wide = sample_rule(n, kSampleThreads * (short_sample ? 1u : (uint32_t)kTopSample), BigTile::kCap, kBigRun, kBigRun, 16.0f);
    rule.big_passes = big_passes;
    rule.big_near = wide.near_limit;
    rule.big_far = big_passes == 1u ? wide.far : rule.far;
  }
  // passes with a launch each; of large arrays as many as heavy keys take, which are 4 %
  // faster so (2^28 Zipf keys 10.15 -> 10.07 ms), for a launch or two that find nothing to do
  const uint32_t lead = big_passes == 1u ? 1u : n > (1u << 27) ? std::max(rule.tmin, 4u) : rule.tmin;
  static std::atomic<uint64_t> allowed[5];
  const auto sample = short_sample ? k_top_sample<1> : k_top_sample<kTopSample>;
  const size_t sample_smem = short_sample ? kSampleSmem<1> : kSampleSmem<kTopSample>;
  if (!allow_smem((const void*)sample, sample_smem, &allowed[short_sample ? 3 : 4])) return 5;
  {
    ProfScope prof("top_sample", st);
    sample<<<1, kSampleThreads, sample_smem, st>>>(X, n, rule, hist, ctrl);
  }
  if (int rc = top_hist(X, ws, L, 0u, dev, st)) return rc;
  for (uint32_t p = 0; p < lead; p++)  // (one may not be in the plan: the big tile's)
    if (int rc = onesweep_top_pass(X, Y, n, (int)p, gstart + p * 256u, ring, L.ring_tiles, ctrl, SegDesc{}, 0, 0u, dev, st, p >= rule.tmin))
      return rc;
  if (int rc = onesweep_top_rest(X, Y, n, (int)lead, gstart, ring, L.ring_tiles, ctrl, SegDesc{}, 0, 0u, dev, st))
    return rc;
  RunChunk* chunks = reinterpret_cast<RunChunk*>(ring);
  uint32_t* unsorted = reinterpret_cast<uint32_t*>(chunks + max_chunks(n));
  // A tile is left a run short on average (its last run is not whole), so a
  // part of `per` tiles is as long as its runs fill `per` tiles, or, with runs
  // that fill a tile by themselves, as `per` runs. Parts of 1 to 16 tiles:
  // enough of them for six rounds of every resident CTA, and else few, since
  // the run across a part's start is read twice.
  auto finish = [&](auto kernel, auto tile, uint32_t ctas, double run_length, uint32_t big, std::atomic<uint64_t>* ok) {
    using TS = decltype(tile);
    if (!allow_smem((const void*)kernel, TS::kSmem, ok)) return false;
    const uint32_t run = (uint32_t)run_length;
    const uint32_t fill = std::max(run, TS::kCap - std::min(TS::kCap, run + run / 2u));
    const uint32_t resident = (uint32_t)dev.sm_count * ctas;
    const uint32_t per = std::max<uint32_t>(1u, std::min<uint32_t>(16u, n / fill / (resident * 6u)));
    const uint32_t stride = per * fill;
    const uint32_t grid = (uint32_t)(((uint64_t)n + stride - 1u) / stride);
    ProfScope prof("top_finish", st);
    kernel<<<grid, TS::kThreads, TS::kSmem, st>>>(X, Y, n, stride, chunks, unsorted, big, ctrl);
    return cudaPeekAtLastError() == cudaSuccess;
  };
  if (!(small_tile ? finish(k_top_finish<SmallTile, 4>, SmallTile{}, 4u, even_run, 0u, &allowed[1])
                   : finish(k_top_finish<Tile, 2>, Tile{}, 2u, even_run, 0u, &allowed[0])) ||
      (big_passes && !finish(k_top_finish<BigTile, 1>, BigTile{}, 1u, (double)n / (big_passes == 1u ? 256.0 : 65536.0), 1u, &allowed[2])))
    return 5;
  if (cudaPeekAtLastError() != cudaSuccess) return 5;
  return top_merge(X, Y, n, chunks, unsorted, ctrl, dev, st);
}

}  // namespace lsb
