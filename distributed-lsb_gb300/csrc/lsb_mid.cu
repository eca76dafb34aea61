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
//      which digits to pass over, lowest first;
//   4. runs longer than a tile that are not in order after that (the sample
//      missed them) have the array passed over by every digit that differs.
// Bound by latency: about four grid barriers and as many trips to L2. Measured
// (GB300, sort alone, eight launched passes -> this): 10^4 uniform keys 131 ->
// 25 us, 10^5 153 -> 28, 10^6 153 -> 42; Zipf keys (four digits) 10^5 153 -> 79,
// 10^6 155 -> 139. The tile
// stays in shared memory, not in registers: with 1024 threads its elements
// spill, and beside 217 KB of shared memory there is no L1 to spill to (a
// digit's count took 6.4 us).
#include <algorithm>

#include "lsb_top.cuh"

namespace lsb {

using MidTile = TileSort<1024, 9>;
constexpr int kMidSample = 1;  // keys per thread of the sample, which only skewed keys need: 1024
constexpr int kMidThreads = MidTile::kThreads;
constexpr int kMidWarps = kMidThreads / 32;
constexpr int kMidRow = kMidWarps + 1;  // padded row of a digit's per-warp counters
constexpr size_t kMidStageBytes = (size_t)kMidThreads * 8u * sizeof(Elem);
constexpr size_t kMidSmem = MidTile::kSmem;
static_assert(kMidStageBytes + 256u * kMidRow * 2u + kMidThreads * 16u <= kMidSmem && kSampleSmem<kMidSample> <= kMidSmem, "shared memory is reused");
static_assert(kSampleThreads == kMidThreads, "the sample is taken by the whole CTA");

struct MidRun {
  uint32_t b, e;
};

// The keys' block, as in TopPlan, and the digit of the current pass.
struct MidWindow {
  uint64_t lo, hi;
  uint32_t hb1, passes, right, left;
  bool clamp;
  __device__ __forceinline__ uint32_t digit(uint64_t key) const {
    const uint32_t d = ((uint32_t)(key >> right) << left) & 255u;
    return clamp ? (key < lo ? 0u : key > hi ? 255u : d) : d;
  }
  __device__ __forceinline__ void set_pass(uint32_t p) {
    const uint32_t up = 8u * (passes - p);
    right = hb1 > up ? hb1 - up : 0u;
    left = hb1 < up ? up - hb1 : 0u;
  }
};

// K elements per thread: tiles of 1024 K. CLUSTER: the grid is one cluster, whose
// barriers are in hardware, and clears the control block itself.
template <int K, bool CLUSTER>
__global__ void __launch_bounds__(kMidThreads, 1)
    k_mid_sort(Elem* X, Elem* Y, uint32_t n, SampleRule rule, uint16_t* table, MidRun* runs, uint32_t max_runs,
               int bits, int num_digits, int api_bits, int sub, Ctrl* ctrl) {
  constexpr uint32_t E = (uint32_t)kMidThreads * K;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ union {
    typename MidTile::Shared tile;
    SampleTile<kMidSample>::Shared sample;
  } sh;
  __shared__ uint32_t s_tot[256], s_pre[256];      // digit d at [(d & 7) 32 + (d >> 3)]
  __shared__ uint32_t s_start[256], s_delta[256], s_tstart[256];
  __shared__ uint32_t s_near[8], s_far[9], s_scan[8], s_diff[2], s_max, s_one, s_part[2];
  __shared__ RunMarks s_marks;
  __shared__ RunKey s_w;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + MidTile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + MidTile::kElemBytes + MidTile::kSlotBytes);
  uint16_t* cnt = reinterpret_cast<uint16_t*>(smem + kMidStageBytes);  // [256][kMidRow]
  uint16_t* order = cnt + 256u * kMidRow;                              // [E] tile positions in digit order
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = lane_id(), lt = lanemask_lt();
  const uint32_t tiles = (n - 1u) / E + 1u, t = blockIdx.x;
  const uint32_t begin = t * E;
  const uint32_t m = t < tiles ? min(E, n - begin) : 0u;  // a CTA without a tile helps with the runs
  const uint32_t p0 = warp * 32u * K + lane;              // this thread ranks positions p0 + 32 k
  uint32_t barriers = 0, buf = 0;
  MidWindow win;

  auto all_arrived = [&]() {
    if (!CLUSTER) return grid_barrier(ctrl, &barriers);
    cluster_arrive();
    cluster_wait();
    return true;
  };
  auto load_tile = [&](const Elem* src) {
    __syncthreads();
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
    for (uint32_t i = tid; i < 256u * kMidRow / 2u; i += kMidThreads) reinterpret_cast<uint32_t*>(cnt)[i] = 0u;
    if (tid < 256) s_tot[tid] = s_pre[tid] = 0u;
    if (tid == 0) s_max = s_one = 0u;
    __syncthreads();
    uint32_t rd[K];  // rank in the warp | digit << 16
#pragma unroll
    for (int k = 0; k < K; k++) rd[k] = win.digit(in[min(p0 + 32u * (uint32_t)k, E - 1u)].key) << 16;
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
    if (lane == 31) sh.tile.wtot[warp] = inc;
    __syncthreads();
    const uint32_t off = inc - sum + __reduce_add_sync(0xffffffffu, lane < warp ? sh.tile.wtot[lane] : 0u);
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
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * kMidThreads;
      if (p < m) {
        const Elem e = in[order[p]];
        const uint32_t o = s_delta[win.digit(e.key)] + p;
        if (o < n) store_elem(dst + o, e);
      }
    }
  };

  // 1. the tile, and the bits in which keys differ
  if (tid < 2) s_diff[tid] = 0u;
  if (tid < 8) s_near[tid] = 0u;
  if (tid < 9) s_far[tid] = 0u;
  const uint64_t first_key = ld_relaxed_u64(&X[0].key);
  if (CLUSTER) {
    if (t == 0)
      for (uint32_t i = tid; i < kCtrlBytes / 4u; i += kMidThreads) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
    cluster_arrive();
  }
  load_tile(X);
  {
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
  const uint32_t hb1 = 64u - (uint32_t)__clzll((long long)diff), full = (hb1 + 7u) / 8u;

  // 2. the top digit alone, 3. or the digits that the sample says
  win.lo = 0ull, win.hi = ~0ull, win.clamp = false;
  win.hb1 = hb1, win.passes = 1u;
  win.set_pass(0);
  count_tile();
  if (!all_arrived()) return;
  add_up();
  const bool exact = full == 1u || s_max <= MidTile::kCap;
  bool skewed = false;
  if (!exact) {
    __syncthreads();
    const uint64_t* s = sample_keys<kMidSample>(X, n, smem, sh.sample);
    const uint64_t span = s[0] ^ s[SampleTile<kMidSample>::kCap - 1u];
    if (span) win.hb1 = 64u - (uint32_t)__clzll((long long)span);
    if (win.hb1 < hb1) {  // the few keys outside the sample's block are clamped to it
      win.lo = s[0] >> win.hb1 << win.hb1;
      win.hi = win.lo | ((1ull << win.hb1) - 1ull);
      win.clamp = true;
    } else {
      rule.tmin = 2u;  // one pass over these bits has been ruled out
    }
    win.passes = sample_passes<kMidSample>(s, win.hb1, rule, s_near, s_far, &skewed);
  }
  for (bool first = true;; first = false) {
    uint32_t par = 0;
    for (uint32_t p = 0; p < win.passes; p++) {
      win.set_pass(p);
      if (p || !first || !exact) {
        load_tile(par ? Y : X);
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
    if (win.passes == full && !win.clamp) {  // in order
      if (par)
        for (uint32_t i = tid; i < m; i += kMidThreads) store_elem(X + begin + i, load_elem_l2(Y + begin + i));
      return;
    }
    // the runs that start in this CTA's part of the array
    const uint32_t shift = win.hb1 > 8u * win.passes ? win.hb1 - 8u * win.passes : 0u;
    uint32_t g = (uint32_t)((uint64_t)n * blockIdx.x / gridDim.x);
    uint32_t limit = (uint32_t)((uint64_t)n * (blockIdx.x + 1u) / gridDim.x);
    bool known = blockIdx.x == 0;
    __syncthreads();
    if (tid == 0) s_w = RunKey{win.lo, win.hi, shift};
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
    auto load = [&](uint32_t from, uint32_t count) {
      __syncthreads();  // in[] is no longer read
      Elem e[MidTile::kItems];
#pragma unroll
      for (int k = 0; k < MidTile::kItems; k++) {
        const uint32_t p = tid + (uint32_t)k * kMidThreads;
        if (p < count) e[k] = load_elem_l2(src + from + p);
      }
#pragma unroll
      for (int k = 0; k < MidTile::kItems; k++) {
        const uint32_t p = tid + (uint32_t)k * kMidThreads;
        if (p < count) in[p] = e[k];
      }
      __syncthreads();
      return true;
    };
    auto long_run = [&](uint32_t b, uint32_t e) {
      if (lane == 0) {
        const uint32_t i = atomicAdd(&ctrl->top.num_runs, 1u);
        if (i < max_runs) runs[i] = MidRun{b, e};
        else record_error(ctrl, kStatusInconsistent, kWhereScatter);
      }
    };
    sort_runs<MidTile>(src, X, exact ? limit : n, g, limit, known, s_w, win.clamp, skewed, shift, in, slot, bins, sh.tile, s_marks,
                       load, long_run);
    if (exact) return;
    // 4. runs longer than a tile: copied into X, and whether they are in order
    if (!all_arrived()) return;
    const uint32_t count = min(ld_relaxed_u32(&ctrl->top.num_runs), max_runs);
    if (count == 0) return;
    MidRun* list = reinterpret_cast<MidRun*>(smem);
    for (uint32_t i = tid; i < count; i += kMidThreads)
      list[i] = MidRun{ld_relaxed_u32(&runs[i].b), ld_relaxed_u32(&runs[i].e)};
    __syncthreads();
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
    win.lo = 0ull, win.hi = ~0ull, win.clamp = false;
    win.hb1 = hb1, win.passes = full;
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

// Two count tables and the list of long runs, after the control block: what any
// size up to n needs, so that a workspace of the largest array serves the smaller
// ones (the tiles double where they outnumber the SMs, and are then half as many).
size_t mid_workspace_bytes(uint32_t n, const DeviceInfo& dev) {
  n = std::min(n, mid_limit(dev));
  const uint32_t tiles = std::min(mid_tiles(n, 2u), (uint32_t)dev.sm_count);
  return kCtrlBytes + (size_t)tiles * 256u * 2u * 2u + (size_t)mid_max_runs(n) * sizeof(MidRun);
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
  // order: 2048 windows per element leave a tile without a mixed run.
  SampleRule rule = sample_rule(n, SampleTile<kMidSample>::kCap, MidTile::kCap - 576u, MidTile::kMaxBin, 2048.0f);
  int bits = L.stat_bits, digits = L.stat_digits, api_bits = L.api_bits, sub = L.sub;
  void* args[] = {&X, &Y, &n, &rule, &table, &runs, &max_runs, &bits, &digits, &api_bits, &sub, &ctrl};
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
