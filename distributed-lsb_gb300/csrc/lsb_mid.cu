// lsb_mid.cu -- whole sorts of arrays too large for one CTA but small enough
// for every CTA to hold a tile of them: one launch, cooperative or of one cluster.
//
// At these sizes (9217 elements to 8192 per SM) memory traffic is nothing and
// launches are everything: the histogram, the plan and each pass cost a launch
// and a start-up. Here one CTA per tile stays for the whole sort and a grid
// barrier takes a launch's place:
//   1. every CTA brings its tile into shared memory; the bits in which keys
//      differ are gathered: the highest says where the top digit lies;
//   2. each tile counts the digit (ranks by ballots and per-warp counters);
//      all counts are exchanged through a table of [tile][digit] counts, the
//      reference's GlobalCounts (mpi/mpi_lsbsort.cpp:339-395), whose columns
//      every CTA adds up for itself: digit totals, and its own tile's starts;
//   3. the totals are the exact lengths of the runs that one pass over the top
//      digit leaves. If all fit in a tile, that one pass is made and the runs
//      are sorted on chip. Otherwise a sample (the same in every CTA) says
//      which digits to pass over, lowest first: digits of bits that vary, and not
//      those that the top digit tells (of signs, tags, sentinels), which is checked
//      against every key (signed 8-bit numbers, 1.1 10^6: 152 us in eight passes,
//      73 in two);
//   4. runs longer than a tile that are not in order after that (the sample
//      missed them) have the array passed over by every digit that differs.
// Bound by latency: about four grid barriers and as many trips to L2. Measured
// (GB300, sort alone, eight launched passes -> this): 2 10^4 uniform keys 135 ->
// 23 us, 2 10^5 152 -> 30, 1.1 10^6 157 -> 44; Zipf keys (four digits) 2 10^5 153 -> 82,
// 1.1 10^6 155 -> 137. Above 622592 elements (152 SMs) a pass takes 18 us, and keys that
// need seven or eight (exponents, many clusters) 170 in all where eight launched
// passes took 154. The tile
// stays in shared memory, not in registers: with 1024 threads its elements
// spill, and beside 217 KB of shared memory there is no L1 to spill to (a
// digit's count took 6.4 us).
#include <algorithm>
#include <cmath>

#include "lsb_top.cuh"

namespace lsb {

using MidTile = TileSort<1024, 9>;
// Passes that leave nothing to sort: no sample is worth its time. (With one, all is
// within 2 %; with eight, 2 10^5 exponents take 91 us, not 100, but signed 20-bit keys 89,
// not 69, and 1.1 10^6 of those 159, not 106.)
constexpr uint32_t kMidFewPasses = 3;
constexpr int kMidThreads = MidTile::kThreads;
constexpr int kMidWarps = kMidThreads / 32;
constexpr int kMidRow = kMidWarps + 1;  // padded row of a digit's per-warp counters
constexpr size_t kMidStageBytes = (size_t)kMidThreads * 8u * sizeof(Elem);
constexpr size_t kMidSmem = MidTile::kSmem;
constexpr size_t kMidSampleAt = kMidStageBytes + 256u * kMidRow * 2u + kMidThreads * 16u;  // beside the tile
static_assert(kMidSampleAt + kSampleSmem<1> + 256u * 8u <= kMidSmem && kMidSampleAt % 16u == 0u, "shared memory is reused");
static_assert(kSampleThreads == kMidThreads, "the sample is taken by the whole CTA");

struct MidRun {
  uint32_t b, e;
};

// A digit here is eight bits of the key that vary, wherever they are, and the
// windows are counted from the top: bits that are the same in all keys take no pass.
// (All bits are known exactly by then. 1.1 10^6 keys of 16 bits spread over 64: two
// passes, not eight.) Digits keep the order of keys that differ in those bits only.
struct MidDigit {  // its runs of neighbouring bits: ((key >> shift) & mask) << up
  uint32_t runs, shift[8], mask[8], up[8];
};
__device__ __forceinline__ void set_digit(MidDigit& g, uint64_t bits) {  // one thread
  uint32_t n = 0, up = 0;
  while (bits) {
    const uint32_t at = (uint32_t)__ffsll((long long)bits) - 1u;
    const uint64_t rest = ~(bits >> at);
    const uint32_t len = rest ? (uint32_t)__ffsll((long long)rest) - 1u : 64u;
    g.shift[n] = at;
    g.mask[n] = (1u << len) - 1u;
    g.up[n++] = up;
    up += len;
    bits &= ~(((1ull << len) - 1ull) << at);
  }
  g.runs = n;
}
// The keys' block, as in TopPlan: keys outside it count as its ends.
struct MidBlock {
  uint64_t lo, hi;
  bool clamp;
};
// The digits of K keys (every thread the same g and w).
template <int K>
__device__ __forceinline__ void mid_digits(const MidDigit& g, const MidBlock& w, const uint64_t (&key)[K], uint32_t (&d)[K]) {
  const uint32_t runs = g.runs, shift = g.shift[0], mask = g.mask[0];
#pragma unroll
  for (int k = 0; k < K; k++) d[k] = (uint32_t)(key[k] >> shift) & mask;
  for (uint32_t r = 1; r < runs; r++) {
    const uint32_t s = g.shift[r], m = g.mask[r], up = g.up[r];
#pragma unroll
    for (int k = 0; k < K; k++) d[k] |= ((uint32_t)(key[k] >> s) & m) << up;
  }
  if (w.clamp) {
#pragma unroll
    for (int k = 0; k < K; k++) d[k] = key[k] < w.lo ? 0u : key[k] > w.hi ? 255u : d[k];
  }
}
// The bits of `key` where `bits` has ones, next to each other.
__device__ __forceinline__ uint64_t gather_bits(uint64_t key, uint64_t bits) {
  uint64_t out = 0;
  uint32_t up = 0;
  while (bits) {
    const uint32_t at = (uint32_t)__ffsll((long long)bits) - 1u;
    const uint64_t rest = ~(bits >> at);
    const uint32_t len = rest ? (uint32_t)__ffsll((long long)rest) - 1u : 64u;
    const uint64_t ones = len < 64u ? (1ull << len) - 1ull : ~0ull;
    out |= ((key >> at) & ones) << up;
    up += len;
    bits &= ~(ones << at);
  }
  return out;
}

// The runs that start in [g, limit) of src[0, n), into X.
__device__ __forceinline__ void mid_finish(const Elem* src, Elem* X, uint32_t n, uint32_t g, uint32_t limit, bool known, const RunKey& w, const bool& clamped,
                                           const bool& skewed, const bool& dups, uint32_t shift, unsigned char* smem, MidTile::Shared& sh, RunMarks& marks, MidRun* runs,
                                        uint32_t max_runs, Ctrl* ctrl) {
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + MidTile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + MidTile::kElemBytes + MidTile::kSlotBytes);
  auto load = [&](uint32_t from, uint32_t count) {
    __syncthreads();  // in[] is no longer read
    Elem e[MidTile::kItems];
#pragma unroll
    for (int k = 0; k < MidTile::kItems; k++) {
      const uint32_t p = threadIdx.x + (uint32_t)k * kMidThreads;
      if (p < count) e[k] = load_elem_l2(src + from + p);
    }
#pragma unroll
    for (int k = 0; k < MidTile::kItems; k++) {
      const uint32_t p = threadIdx.x + (uint32_t)k * kMidThreads;
      if (p < count) in[p] = e[k];
    }
    __syncthreads();
    return true;
  };
  auto long_run = [&](uint32_t b, uint32_t e) {
    if (lane_id() == 0) {
      const uint32_t i = atomicAdd(&ctrl->top.num_runs, 1u);
      if (i < max_runs) runs[i] = MidRun{b, e};
      else record_error(ctrl, kStatusInconsistent, kWhereScatter);
    }
  };
  sort_runs<MidTile>(src, X, n, g, limit, known, w, clamped, skewed, dups, shift, in, slot, bins, sh, marks, load, long_run);
}

// K elements per thread: tiles of 1024 K. CLUSTER: the grid is one cluster, whose
// barriers are in hardware, and clears the control block itself.
template <int K, bool CLUSTER>
__global__ void __launch_bounds__(kMidThreads, 1)
    k_mid_sort(Elem* X, Elem* Y, uint32_t n, SampleRule rule, uint16_t* table, MidRun* runs, uint32_t max_runs, uint64_t* keys_of,
               int bits, int num_digits, int api_bits, int sub, Ctrl* ctrl) {
  constexpr uint32_t E = (uint32_t)kMidThreads * K;
  constexpr int R = K < 4 ? K : 4;  // rows at a time, where a thread would keep too much of all
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename MidTile::Shared sh;
  __shared__ SampleStats s_stats;
  __shared__ uint32_t s_tot[256], s_pre[256];      // digit d at [(d & 7) 32 + (d >> 3)]
  __shared__ uint32_t s_start[256], s_delta[256], s_tstart[256];
  __shared__ uint32_t s_scan[8], s_diff[2], s_max, s_one, s_part[2];
  __shared__ unsigned long long s_bits[8];  // the windows' bits, the highest first
  __shared__ MidDigit s_digit[8];           // and how they are taken from a key
  __shared__ uint32_t s_window;             // of the pass
  __shared__ bool s_go;
  // What is decided once, written by one thread with barriers around: with 1024
  // threads a register kept for it is one that a pass has to take from local memory.
  __shared__ struct {
    uint64_t diff;         // bits in which keys differ
    uint32_t all;          // passes over all of those, which leave nothing to sort
    uint32_t passes, full;  // windows passed over, and those that there are
    bool skewed, dups;
  } s_plan;
  __shared__ RunMarks s_marks;
  __shared__ RunKey s_w;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint16_t* cnt = reinterpret_cast<uint16_t*>(smem + kMidStageBytes);  // [256][kMidRow]
  uint16_t* order = cnt + 256u * kMidRow;                              // [E] tile positions in digit order
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = lane_id(), lt = lanemask_lt();
  const uint32_t tiles = (n - 1u) / E + 1u, t = blockIdx.x;
  // The tile's place and length, reckoned anew at each use: kept, they are two more
  // values that a pass has to fetch from local memory.
  auto tile_begin = []() {
    uint32_t cta;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
    return cta * E;
  };
  auto tile_len = [&](uint32_t begin) { return begin < n ? min(E, n - begin) : 0u; };  // a CTA without a tile helps with the runs
  uint32_t barriers = 0, buf = 0;
  __shared__ MidBlock win;  // written by one thread, with barriers around

  auto all_arrived = [&]() {
    if (!CLUSTER) return grid_barrier(ctrl, &barriers);
    cluster_arrive();
    cluster_wait();
    return true;
  };
  auto load_tile = [&](const Elem* src) {
    __syncthreads();
    const uint32_t begin = tile_begin(), m = tile_len(begin);
    Elem v[K];
#pragma unroll
    for (int k = 0; k < K; k++)
      if (tid + (uint32_t)k * kMidThreads < m) v[k] = load_elem_l2(src + begin + tid + (uint32_t)k * kMidThreads);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (tid + (uint32_t)k * kMidThreads < m) in[tid + (uint32_t)k * kMidThreads] = v[k];
    __syncthreads();
  };
  // ranks and counts of the digit in the tile: order[], and the counts to the table
  auto count_tile = [&]() {
    const uint32_t m = tile_len(tile_begin());
    const uint32_t p0 = warp * 32u * K + lane;  // this thread ranks positions p0 + 32 k
    for (uint32_t i = tid; i < 256u * kMidRow / 2u; i += kMidThreads) reinterpret_cast<uint32_t*>(cnt)[i] = 0u;
    if (tid < 256) s_tot[tid] = s_pre[tid] = 0u;
    if (tid == 0) s_max = s_one = 0u;
    __syncthreads();
    uint32_t rd[K];  // rank in the warp | digit << 16
#pragma unroll
    for (int k = 0; k < K; k += R) {
      uint64_t key[R];
      uint32_t d[R];
#pragma unroll
      for (int i = 0; i < R; i++) key[i] = in[min(p0 + 32u * (uint32_t)(k + i), E - 1u)].key;
      mid_digits<R>(s_digit[s_window], win, key, d);
#pragma unroll
      for (int i = 0; i < R; i++) rd[k + i] = d[i] << 16;
    }
    if (m == E) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t d = rd[k] >> 16;
        const uint32_t peers = warp_peers_fixed<8>(d);
        uint16_t* c = &cnt[d * kMidRow + warp];
        const uint32_t before = *c;
        rd[k] |= before + __popc(peers & lt);
        __syncwarp();
        *c = (uint16_t)(before + __popc(peers));
        __syncwarp();
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const bool valid = p0 + 32u * (uint32_t)k < m;
        const uint32_t d = rd[k] >> 16;
        const uint32_t peers = warp_peers(d, 8, valid);
        uint16_t* c = &cnt[d * kMidRow + warp];
        const uint32_t before = *c;
        rd[k] |= before + __popc(peers & lt);
        __syncwarp();
        if (valid) *c = (uint16_t)(before + __popc(peers));
        __syncwarp();
      }
    }
    __syncthreads();
    // exclusive scan in [digit][warp] order: thread 4 d + q has warps [8 q, 8 q + 8) of digit d
    uint16_t* c = &cnt[tid / 4u * kMidRow + tid % 4u * 8u];
    uint32_t p8[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      p8[j] = sum;
      sum += c[j];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
    uint32_t of_digit = sum + __shfl_xor_sync(0xffffffffu, sum, 1);
    of_digit += __shfl_xor_sync(0xffffffffu, of_digit, 2);
    if (lane == 31) sh.wtot[warp] = inc;
    __syncthreads();
    const uint32_t off = inc - sum + __reduce_add_sync(0xffffffffu, lane < warp ? sh.wtot[lane] : 0u);
#pragma unroll
    for (int j = 0; j < 8; j++) c[j] = (uint16_t)(off + p8[j]);
    if (tid % 4u == 0u) {
      s_tstart[tid / 4u] = off;
      if (t < tiles) table[((size_t)buf * tiles + t) * 256u + tid / 4u] = (uint16_t)of_digit;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = p0 + 32u * (uint32_t)k;
      if (p < m) order[(rd[k] & 0xffffu) + cnt[(rd[k] >> 16) * kMidRow + warp]] = (uint16_t)p;
    }
  };
  // after the grid barrier: totals of every digit, where this tile's elements of each go
  auto add_up = [&]() {
    uint32_t tot[8] = {}, pre[8] = {};
    for (uint32_t o = warp; o < tiles; o += kMidWarps) {
      const uint4 q = __ldcg(reinterpret_cast<const uint4*>(table + ((size_t)buf * tiles + o) * 256u) + lane);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t c = (w[i >> 1] >> (16 * (i & 1))) & 0xffffu;
        tot[i] += c;
        pre[i] += o < t ? c : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      atomicAdd(&s_tot[i * 32 + lane], tot[i]);
      atomicAdd(&s_pre[i * 32 + lane], pre[i]);
    }
    __syncthreads();
    uint32_t total = 0, inc = 0;
    const uint32_t at = (tid & 7u) * 32u + (tid >> 3);
    if (tid < 256) {
      inc = total = s_tot[at];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      if (lane == 31) s_scan[warp] = inc;
      const uint32_t mx = __reduce_max_sync(0xffffffffu, total);
      if (lane == 0) atomicMax(&s_max, mx);
      if (total == n) s_one = 1u;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t off = inc - total;
#pragma unroll
      for (int w = 0; w < 8; w++) off += (uint32_t)w < warp ? s_scan[w] : 0u;
      s_start[tid] = off;
      s_delta[tid] = off + s_pre[at] - s_tstart[tid];
    }
    __syncthreads();
  };
  auto scatter = [&](Elem* dst) {
    const uint32_t m = tile_len(tile_begin());
    const MidDigit& g = s_digit[s_window];
    if (g.runs == 1u && !win.clamp) {  // as most digits are
      const uint32_t shift = g.shift[0], mask = g.mask[0];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t p = tid + (uint32_t)k * kMidThreads;
        if (p < m) {
          const Elem e = in[order[p]];
          const uint32_t o = s_delta[(uint32_t)(e.key >> shift) & mask] + p;
          if (o < n) store_elem(dst + o, e);
        }
      }
      return;
    }
#pragma unroll 1
    for (uint32_t row = tid; row < E; row += (uint32_t)(R * kMidThreads)) {
      uint64_t key[R], val[R];
      uint32_t d[R];
#pragma unroll
      for (int k = 0; k < R; k++) {
        const uint32_t p = row + (uint32_t)k * kMidThreads;
        const Elem e = in[p < m ? order[p] : 0u];
        key[k] = e.key;
        val[k] = e.val;
      }
      mid_digits<R>(g, win, key, d);
#pragma unroll
      for (int k = 0; k < R; k++) {
        const uint32_t p = row + (uint32_t)k * kMidThreads;
        const uint32_t o = s_delta[d[k]] + p;
        if (p < m && o < n) store_elem(dst + o, Elem{key[k], val[k]});
      }
    }
  };

  // 1. the tile, and the bits in which keys differ
  if (tid < 2) s_diff[tid] = 0u;
  clear_stats(s_stats);
  const uint64_t first_key = ld_relaxed_u64(&X[0].key);
  if (CLUSTER) {
    if (t == 0)
      for (uint32_t i = tid; i < kCtrlBytes / 4u; i += kMidThreads) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
    cluster_arrive();
  }
  load_tile(X);
  {
    const uint32_t m = tile_len(tile_begin());
    uint64_t x = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * kMidThreads;
      x |= p < m ? in[p].key ^ first_key : 0ull;
    }
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)x);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(x >> 32));
    if (lane == 0) {
      if (lo) atomicOr(&s_diff[0], lo);
      if (hi) atomicOr(&s_diff[1], hi);
    }
  }
  __syncthreads();
  if (CLUSTER) cluster_wait();
  if (tid < 2 && s_diff[tid]) atomicOr(&ctrl->top.diff[tid], s_diff[tid]);
  if (!all_arrived()) return;
  const uint64_t diff = (uint64_t)__ldcg(&ctrl->top.diff[1]) << 32 | __ldcg(&ctrl->top.diff[0]);
  if (t == 0 && tid == 0) write_plan(ctrl, diff, n, bits, num_digits, api_bits, sub);
  if (diff == 0) return;
  // the windows of eight of the bits `of`, into s_bits and s_digit; a barrier behind it
  auto set_windows = [&](uint64_t of) {
    if (tid < 8) s_bits[tid] = 0ull;
    __syncthreads();
    if (tid < 64 && (of >> tid & 1ull)) atomicOr(&s_bits[(__popcll(of >> tid) - 1) >> 3], 1ull << tid);
    __syncthreads();
    if (lane == 0 && warp < 8u && s_bits[warp]) set_digit(s_digit[warp], s_bits[warp]);
    __syncthreads();
  };
  auto passes_over = [](uint64_t of) { return ((uint32_t)__popcll(of) + 7u) / 8u; };
  const uint32_t all = passes_over(diff);  // passes that leave nothing to sort
  // v of all threads of the CTA, or'ed together
  auto or_all = [&](uint64_t v) {
    __syncthreads();
    if (tid < 2) s_diff[tid] = 0u;
    __syncthreads();
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
    if (lane == 0) {
      if (lo) atomicOr(&s_diff[0], lo);
      if (hi) atomicOr(&s_diff[1], hi);
    }
    __syncthreads();
    return (uint64_t)s_diff[1] << 32 | s_diff[0];
  };
  // The bits in which keys with the same digit in the top window differ: exactly,
  // against one key of each digit that all CTAs agree on. s_go: no wait ran out.
  auto told_apart = [&]() -> uint64_t {
    uint64_t* one = reinterpret_cast<uint64_t*>(smem + kMidSampleAt + kSampleSmem<1>);
    const uint32_t m = tile_len(tile_begin());
    auto with_digit = [&](auto f) {
#pragma unroll 1
      for (uint32_t p = tid; p < m; p += (uint32_t)kMidThreads) {
        const uint64_t key[1] = {in[p].key};
        uint32_t d[1];
        mid_digits<1>(s_digit[0], win, key, d);
        f(key[0], d[0]);
      }
    };
    __syncthreads();
    with_digit([&](uint64_t key, uint32_t d) { one[d] = key; });  // any one of the tile's
    __syncthreads();
    if (tid < 256u && t < tiles && (tid < 255u ? s_tstart[tid + 1u] : m) > s_tstart[tid]) keys_of[tid] = one[tid];
    bool go = all_arrived();
    if (tid < 256u) one[tid] = __ldcg(&keys_of[tid]);
    __syncthreads();
    uint64_t x = 0;
    with_digit([&](uint64_t key, uint32_t d) { x |= key ^ one[d]; });
    x = or_all(x);
    if (tid == 0) {
      if ((uint32_t)x) atomicOr(&ctrl->top.apart[0], (uint32_t)x);
      if (x >> 32) atomicOr(&ctrl->top.apart[1], (uint32_t)(x >> 32));
    }
    go = go && all_arrived();
    if (tid == 0) s_go = go;
    __syncthreads();
    return (uint64_t)__ldcg(&ctrl->top.apart[1]) << 32 | __ldcg(&ctrl->top.apart[0]);
  };

  // 2. the top digit alone, 3. or the digits that the sample says
  if (tid == 0) win.clamp = false;
  if (tid == 0) s_plan = {diff, all, 1u, all, false, false};
  auto low_bit = [&](uint32_t windows) { return (uint32_t)__ffsll((long long)s_bits[windows - 1u]) - 1u; };
  if (tid == 0) {  // the first window: the eight highest bits that vary, mostly neighbours
    const uint32_t hb1 = 64u - (uint32_t)__clzll((long long)diff);
    s_window = 0u;
    if (hb1 >= 8u && diff >> (hb1 - 8u) == 255u) {
      s_digit[0].runs = 1u;
      s_digit[0].shift[0] = hb1 - 8u;
      s_digit[0].mask[0] = 255u;
      s_bits[0] = 255ull << (hb1 - 8u);
    } else {
      uint64_t top = 0;
      for (uint64_t rest = diff; rest && __popcll(top) < 8; rest = diff & ~top) top |= 1ull << (63u - (uint32_t)__clzll((long long)rest));
      s_bits[0] = top;
      set_digit(s_digit[0], top);
    }
  }
  count_tile();
  // a tile or two for each CTA: the ways of duplicates are the ones to try first
  // unless there are bits that would make other keys uneven
  if (tid == 32u) s_plan.dups = !ragged(low_bit(1u), 13u, 5u, diff);
  if (!all_arrived()) return;
  add_up();
  const bool exact = all == 1u || s_max <= MidTile::kCap;
  if (!exact) {
    const uint64_t top_bits = s_bits[0];
    if (tid == 0) s_plan.passes = all;
    __syncthreads();
    set_windows(diff);
    if (all > kMidFewPasses) {
      uint64_t* buf = reinterpret_cast<uint64_t*>(smem + kMidSampleAt);
      const uint64_t* s = sort_sample(sample_key(X, n, tid), buf);
      const uint64_t lowest = s[0], span = lowest ^ s[kSampleThreads - 1];
      uint64_t bits = diff;
      MidBlock block{0ull, ~0ull, false};
      if (span && (diff >> (63u - (uint32_t)__clzll((long long)span))) >> 1) {
        // the few keys outside the sample's block are clamped to it
        const uint32_t hb = 64u - (uint32_t)__clzll((long long)span);
        bits &= (1ull << hb) - 1ull;
        block.lo = lowest >> hb << hb;
        block.hi = block.lo | ((1ull << hb) - 1ull);
        block.clamp = true;
      } else {
        rule.tmin = 2u;  // one pass over these bits has been ruled out
        // bits that the top window tells (of a sign, a tag, a sentinel) need no pass
        const uint64_t step = tid + 1u < kSampleThreads ? s[tid] ^ s[tid + 1u] : 0ull;
        if (passes_over(top_bits | or_all((step & top_bits) ? 0ull : step)) + 2u <= all) {
          const uint64_t apart = told_apart();
          if (!s_go) return;
          bits = top_bits | apart;
        }
      }
      const uint32_t count = (uint32_t)__popcll(bits);
      const uint64_t mine = gather_bits(s[tid], bits);
      set_windows(bits);
      buf[tid] = mine;  // either half: every thread has read its key before the barrier
      __syncthreads();
      const uint32_t full = passes_over(bits);
      const SampleChoice c = choose_passes<1>(buf, count, rule, block.clamp ? all : full, s_stats, bits, low_bit);
      if (c.plain && block.clamp) {
        __syncthreads();
        set_windows(diff);
      } else if (tid == 0) {
        win = block;
        s_plan.passes = c.plain ? full : c.passes;
        s_plan.full = full;
        s_plan.skewed = c.skewed;
        s_plan.dups = c.dups || !ragged(low_bit(s_plan.passes), 13u, 5u, bits);
      }
      __syncthreads();
    }
  }
  for (bool first = true;; first = false) {
    uint32_t par = 0;
    for (uint32_t p = 0; p < s_plan.passes; p++) {
      if (p || !first || !exact) {
        if (p || !first) load_tile(par ? Y : X);  // else it is still there
        if (tid == 0) s_window = s_plan.passes - 1u - p;
        buf ^= 1u;
        count_tile();
        if (!all_arrived()) return;
        add_up();
      }
      if (s_one) continue;  // the digit is the same everywhere
      scatter(par ? X : Y);
      par ^= 1u;
      if (!all_arrived()) return;
    }
    const Elem* src = par ? Y : X;
    if (s_plan.passes == s_plan.full && !win.clamp) {  // in order
      const uint32_t begin = tile_begin(), m = tile_len(begin);
      if (par)
        for (uint32_t i = tid; i < m; i += kMidThreads) store_elem(X + begin + i, load_elem_l2(Y + begin + i));
      return;
    }
    // the runs that start in this CTA's part of the array
    const uint32_t shift = low_bit(s_plan.passes);
    uint32_t g = (uint32_t)((uint64_t)n * blockIdx.x / gridDim.x);
    uint32_t limit = (uint32_t)((uint64_t)n * (blockIdx.x + 1u) / gridDim.x);
    bool known = blockIdx.x == 0;
    __syncthreads();
    if (tid == 0) s_w = RunKey{win.clamp ? win.lo : 0ull, win.clamp ? win.hi : ~0ull, shift};
    if (exact && first) {  // after one pass the runs are the digit's buckets
      if (tid < 2) s_part[tid] = n;
      __syncthreads();
      if (tid < 256) {
        if (s_start[tid] >= g) atomicMin(&s_part[0], s_start[tid]);
        if (s_start[tid] >= limit) atomicMin(&s_part[1], s_start[tid]);
      }
      __syncthreads();
      g = s_part[0];
      limit = s_part[1];
      known = true;
    }
    mid_finish(src, X, exact ? limit : n, g, limit, known, s_w, win.clamp, s_plan.skewed, s_plan.dups, shift, smem, sh, s_marks, runs, max_runs, ctrl);
    if (exact) return;
    // 4. runs longer than a tile: copied into X, and whether they are in order
    if (!all_arrived()) return;
    const uint32_t count = min(ld_relaxed_u32(&ctrl->top.num_runs), max_runs);
    if (count == 0) return;
    MidRun* list = reinterpret_cast<MidRun*>(smem);
    for (uint32_t i = tid; i < count; i += kMidThreads)
      list[i] = MidRun{ld_relaxed_u32(&runs[i].b), ld_relaxed_u32(&runs[i].e)};
    __syncthreads();
    const uint32_t begin = tile_begin(), m = tile_len(begin);
    bool inversion = false;
    for (uint32_t i = 0; i < count; i++) {
      const uint32_t b = list[i].b, e = list[i].e;
      for (uint32_t j = max(b, begin) + tid; j < min(e, begin + m); j += kMidThreads) {
        const Elem x = load_elem_l2(src + j);
        if (j + 1u < e) inversion |= x.key > ld_relaxed_u64(&src[j + 1u].key);
        if (par) store_elem(X + j, x);
      }
    }
    if (__any_sync(0xffffffffu, inversion) && lane == 0) atomicOr(&ctrl->top.num_chunks, 1u);
    if (!all_arrived()) return;
    if (ld_relaxed_u32(&ctrl->top.num_chunks) == 0u) return;
    if (tid == 0) win.clamp = false, s_plan.passes = s_plan.full = s_plan.all;
    set_windows(s_plan.diff);
    __syncthreads();
  }
}

// A tile per CTA and one CTA per SM: 1024, 2048 ... 8192 elements per tile, the
// smallest that the SMs hold (small tiles rank and place in fewer rounds).
constexpr uint32_t kMidLargestTile = (uint32_t)kMidThreads * 8u;
uint32_t mid_limit(const DeviceInfo& dev) { return (uint32_t)dev.sm_count * kMidLargestTile; }

static uint32_t mid_items(uint32_t n, const DeviceInfo& dev) {
  uint32_t k = 2;
  while (k < 8u && (uint64_t)k * kMidThreads * (uint32_t)dev.sm_count < n) k *= 2u;
  return k;
}
static uint32_t mid_tiles(uint32_t n, uint32_t items) { return (n - 1u) / (items * (uint32_t)kMidThreads) + 1u; }
static uint32_t mid_max_runs(uint32_t n) { return n / MidTile::kCap + 1u; }

// Two count tables, the list of long runs and a key for each digit, after the control block: what any
// size up to n needs, so that a workspace of the largest array serves the smaller
// ones (the tiles double where they outnumber the SMs, and are then half as many).
size_t mid_workspace_bytes(uint32_t n, const DeviceInfo& dev) {
  n = std::min(n, mid_limit(dev));
  const uint32_t tiles = std::min(mid_tiles(n, 2u), (uint32_t)dev.sm_count);
  return kCtrlBytes + (size_t)tiles * 256u * 2u * 2u + (size_t)mid_max_runs(n) * sizeof(MidRun) + 256u * 8u;
}

// Up to 16 tiles of 2048 elements the grid is one cluster of 16 CTAs: no clear
// before it, no cooperative launch, barriers in hardware. 32768 uniform elements
// 26 -> 23 us, Zipf keys 49 -> 45. Larger tiles in the cluster lose that again
// against more CTAs (50000: 27 us either way, 65537: 31 against 26).
constexpr uint32_t kMidCluster = 16, kMidClusterItems = 2;

static cudaLaunchConfig_t mid_cluster_config(cudaLaunchAttribute* attr, cudaStream_t st) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = kMidCluster;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(kMidCluster);
  c.blockDim = dim3(kMidThreads);
  c.dynamicSmemBytes = kMidSmem;
  c.stream = st;
  c.attrs = attr;
  c.numAttrs = 1;
  return c;
}

// Whether the current device has room for such a cluster; asked once per device.
static bool mid_cluster_fits(const void* kern) {
  static std::atomic<uint64_t> yes, no;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  const uint64_t bit = 1ull << dev;
  if (yes.load(std::memory_order_acquire) & bit) return true;
  if (no.load(std::memory_order_acquire) & bit) return false;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t config = mid_cluster_config(&attr, nullptr);
  int clusters = 0;
  const bool fits = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmem) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern, &config) == cudaSuccess && clusters > 0;
  if (!fits) cudaGetLastError();
  (fits ? yes : no).fetch_or(bit, std::memory_order_release);
  return fits;
}

int mid_run(Elem* X, Elem* Y, unsigned char* ws, const Layout& L, const DeviceInfo& dev, cudaStream_t st) {
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(ws);
  uint32_t n = L.n;
  const uint32_t items = mid_items(n, dev), tiles = mid_tiles(n, items);
  uint16_t* table = reinterpret_cast<uint16_t*>(ws + kCtrlBytes);
  MidRun* runs = reinterpret_cast<MidRun*>(ws + kCtrlBytes + (size_t)tiles * 256u * 2u * 2u);
  uint32_t max_runs = mid_max_runs(n);
  // A key that overfills its bins makes a tile uneven, unless the tile is in
  // order: 2048 windows per element leave a tile without a mixed run (1.1 10^6 Zipf
  // keys 136 us; with 16384, a pass more, 153; 128 asks for as many passes as 2048 here).
  SampleRule rule = sample_rule(n, kSampleThreads, MidTile::kCap, MidTile::kCap - 576u, MidTile::kMaxBin, 2048.0f);
  rule.finish = 8u;
  rule.copy = 2u;
  rule.straddle = 25u;
  // A run longer than a tile has the array passed over by every digit once more: a
  // window with a tile's share of the sample, less half a deviation, is taken
  // for one.
  const float share = (float)MidTile::kCap * (float)kSampleThreads / (float)n;
  rule.far = (uint32_t)std::max(4.0f, share - 0.5f * std::sqrt(share));
  rule.far_limit = 2u;
  int bits = L.stat_bits, digits = L.stat_digits, api_bits = L.api_bits, sub = L.sub;
  uint64_t* keys_of = reinterpret_cast<uint64_t*>(runs + max_runs);
  void* args[] = {&X, &Y, &n, &rule, &table, &runs, &max_runs, &keys_of, &bits, &digits, &api_bits, &sub, &ctrl};
  const uint32_t sms = stream_sms(st, dev);
  if (tiles > sms) return kMidRefused;
  if (n <= kMidCluster * kMidClusterItems * (uint32_t)kMidThreads && sms == (uint32_t)dev.sm_count) {
    const void* kern = (const void*)k_mid_sort<(int)kMidClusterItems, true>;
    if (mid_cluster_fits(kern)) {
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t config = mid_cluster_config(&attr, st);
      ProfScope prof("mid_sort", st);
      if (cudaLaunchKernelExC(&config, kern, args) == cudaSuccess) return 0;
      cudaGetLastError();
    }
  }
  const void* kern = items == 2u   ? (const void*)k_mid_sort<2, false>
                     : items == 4u ? (const void*)k_mid_sort<4, false>
                                   : (const void*)k_mid_sort<8, false>;
  static std::atomic<uint64_t> allowed[3];
  if (!allow_smem(kern, kMidSmem, &allowed[items >> 2]) || cudaMemsetAsync(ws, 0, kCtrlBytes, st) != cudaSuccess)
    return 5;
  // CTAs beyond the tiles take a share of the runs
  const uint32_t grid = std::min<uint32_t>(sms, std::max(tiles, (n - 1u) / 2048u + 1u));
  ProfScope prof("mid_sort", st);
  if (cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kMidThreads), args, kMidSmem, st) == cudaSuccess) return 0;
  cudaGetLastError();
  return kMidRefused;
}

}  // namespace lsb
