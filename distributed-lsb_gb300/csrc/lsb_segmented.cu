// lsb_segmented.cu -- batched segmented sort: many independent arrays of
// uneven sizes, stored back to back in one buffer, sorted by the same
// persistent onesweep launches (one per pass), plus the project's autotuner
// and CUDA-graph capture of the whole batch.
//
// The reference sorts one distributed array per program run (mySort,
// mpi/mpi_lsbsort.cpp:592-597); sorting many arrays means running it once per
// array. Here a batch is one sort, by the steps of lsb_top.cu for every array
// at once: arrays that fit in a tile are only sorted there; for the others a
// sample each says how many top digits to pass over. The passes go over the
// flattened list of (segment, tile) pairs, arrays with more passes first, and
// every segment's first tile publishes its digit counts as an inclusive prefix
// at once (so no look-back crosses a segment boundary). Small and large arrays
// share the same launches, so every SM stays busy however uneven the sizes are.
// Measured (GB300, against eight passes over every array): 512 arrays of
// 2^U(10,22) elements 13.5 -> 5.6 ms, 64 of 2^U(10,16) 160 -> 92 us, Zipf keys
// 14.1 -> 8.8 ms and 158 -> 139 us.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "../../include/lsb.h"
#include "lsb_top.cuh"

namespace lsb {

// ---------------------------------------------------------------------------
// plans: which digits each array is passed over by

constexpr int kSegSample = 1;  // keys per thread of an array's sample: 1024

// Plan of every array, one CTA per array in turn: none for arrays that fit in
// a tile, else from a sample, as for one array (lsb_top.cu). Two CTAs per SM,
// about 6 us per sampled array.
__global__ void __launch_bounds__(kSampleThreads, 2)
    k_seg_sample(const Elem* __restrict__ data, const int64_t* __restrict__ seg_off, uint32_t nseg, uint32_t straddle,
                 SegPlan* __restrict__ plans) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename SampleTile<kSegSample>::Shared sh;
  __shared__ SampleStats s_stats;
  for (uint32_t s = blockIdx.x; s < nseg; s += gridDim.x) {
    const uint32_t len = (uint32_t)(seg_off[s + 1] - seg_off[s]);
    SegPlan p{};
    p.hb1 = 64u;
    p.hi = ~0ull;
    if (len > kCap) {
      __syncthreads();
      clear_stats(s_stats);
      const uint64_t* k = sample_keys<kSegSample>(data + seg_off[s], len, smem, sh);
      const uint64_t first = k[0], span = first ^ k[kSegSample * kSampleThreads - 1];
      if (span) p.hb1 = 64u - (uint32_t)__clzll((long long)span);
      // a key that overfills its bins is heavy (lsb_mid.cu); four passes leave
      // its runs pure up to 2^28 elements. Zipf keys in arrays of 2^10 to 2^20 take
      // 2690 us in all; with 16 windows per element for all lengths 3658. Of 2^20 to 2^23:
      // 2031; with 2048 for all 2433.
      const float spread = fminf(2048.0f, fmaxf(16.0f, 4294967296.0f / (float)len));
      SampleRule rule = sample_rule(len, kSegSample * kSampleThreads, Tile::kCap, kMeanRun, Tile::kMaxBin, spread);
      rule.skips = false;
      rule.straddle = straddle;
      const SampleChoice c = choose_passes<kSegSample>(k, p.hb1, rule, 8u, s_stats, 0ull,
                                                          [&](uint32_t t) { return p.hb1 > 8u * t ? p.hb1 - 8u * t : 0u; });
      p.passes = c.passes;
      p.skewed = (c.skewed ? 1u : 0u) | (c.dups ? 2u : 0u);
      if (p.hb1 < 64u) {
        p.clamp = 1u;
        p.lo = first >> p.hb1 << p.hb1;
        p.hi = p.lo | ((1ull << p.hb1) - 1ull);
      }
    }
    if (threadIdx.x == 0) plans[s] = p;
  }
}

// ---------------------------------------------------------------------------
// tile map

constexpr int kSegScanThreads = 1024;

// First pass tile and first part of each array, arrays with more passes first;
// tiles of every pass (num_tiles[0..7]) and parts (num_tiles[8]).
__global__ void __launch_bounds__(kSegScanThreads)
    k_seg_tiles(const int64_t* __restrict__ seg_off, uint32_t nseg, uint32_t tile, uint32_t stride, const SegPlan* __restrict__ plans,
                uint32_t* __restrict__ seg_tile0, uint32_t* __restrict__ seg_part0, uint32_t* __restrict__ num_tiles) {
  __shared__ uint32_t wt[33];
  const uint32_t per = (nseg + blockDim.x - 1) / blockDim.x;
  const uint32_t lo = min(threadIdx.x * per, nseg), hi = min(lo + per, nseg);
  uint32_t tiles[9] = {}, parts = 0;
  for (uint32_t s = lo; s < hi; s++) {
    const uint64_t len = (uint64_t)(seg_off[s + 1] - seg_off[s]);
    const uint32_t passes = plans[s].passes, n = (uint32_t)((len + tile - 1) / tile);
#pragma unroll
    for (uint32_t c = 1; c <= 8u; c++) tiles[c] += passes == c ? n : 0u;
    parts += passes ? (uint32_t)((len + stride - 1) / stride) : len ? 1u : 0u;
  }
  uint32_t tot, base = 0;
#pragma unroll
  for (int c = 8; c >= 1; c--) {
    if (__syncthreads_or(tiles[c])) {
      const uint32_t ex = block_exclusive_scan(tiles[c], wt, &tot);
      tiles[c] = base + ex;
      base += tot;
    }
    if (threadIdx.x == 0) num_tiles[c - 1] = base;  // arrays with more than c - 1 passes
  }
  uint32_t part = block_exclusive_scan(parts, wt, &tot);
  if (threadIdx.x == 0) num_tiles[8] = tot;
  for (uint32_t s = lo; s < hi; s++) {
    const uint64_t len = (uint64_t)(seg_off[s + 1] - seg_off[s]);
    const uint32_t passes = plans[s].passes, n = (uint32_t)((len + tile - 1) / tile);
    uint32_t at = 0;
#pragma unroll
    for (uint32_t c = 1; c <= 8u; c++)
      if (passes == c) {
        at = tiles[c];
        tiles[c] += n;
      }
    seg_tile0[s] = at;
    seg_part0[s] = part;
    part += passes ? (uint32_t)((len + stride - 1) / stride) : len ? 1u : 0u;
  }
}

// tile_seg[t], part_seg[p] = the segment tile t or part p belongs to (one warp per segment)
__global__ void k_seg_fill(const int64_t* __restrict__ seg_off, uint32_t nseg, uint32_t tile, uint32_t stride,
                           const SegPlan* __restrict__ plans, const uint32_t* __restrict__ seg_tile0,
                           const uint32_t* __restrict__ seg_part0, uint32_t* __restrict__ tile_seg,
                           uint32_t* __restrict__ part_seg) {
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nseg; s += warps) {
    const uint64_t len = (uint64_t)(seg_off[s + 1] - seg_off[s]);
    if (plans[s].passes) {
      const uint32_t tiles = (uint32_t)((len + tile - 1) / tile);
      const uint32_t parts = (uint32_t)((len + stride - 1) / stride);
      for (uint32_t j = lane_id(); j < tiles; j += 32) tile_seg[seg_tile0[s] + j] = s;
      for (uint32_t j = lane_id(); j < parts; j += 32) part_seg[seg_part0[s] + j] = s;
    } else if (len && lane_id() == 0) {
      part_seg[seg_part0[s]] = s;
    }
  }
}

// ---------------------------------------------------------------------------
// segmented histogram of the passes' digits: counts[seg][pass][digit]

constexpr int kSegHistThreads = 512;
constexpr uint32_t kSegHistUnroll = 4;

__global__ void __launch_bounds__(kSegHistThreads, 4)
    k_seg_hist(const Elem* __restrict__ data, const int64_t* __restrict__ seg_off,
               const uint32_t* __restrict__ seg_tile0, const uint32_t* __restrict__ tile_seg,
               const uint32_t* __restrict__ num_tiles, uint32_t tile, SegPlan* __restrict__ plans,
               uint32_t* __restrict__ counts) {
  __shared__ uint32_t h[8 * 256];
  __shared__ uint32_t s_diff[2];
  __shared__ TopWindow s_win[8];
  const uint32_t T = num_tiles[0];
  // a contiguous range of tiles per CTA: segment changes are rare
  const uint32_t t_lo = (uint32_t)((uint64_t)T * blockIdx.x / gridDim.x);
  const uint32_t t_hi = (uint32_t)((uint64_t)T * (blockIdx.x + 1) / gridDim.x);
  for (uint32_t i = threadIdx.x; i < 8u * 256u; i += kSegHistThreads) h[i] = 0u;
  if (threadIdx.x < 2) s_diff[threadIdx.x] = 0u;
  uint32_t cur = 0xffffffffu, passes = 0;
  uint64_t first = 0, diff = 0;
  auto flush = [&]() {  // the segment's counts so far, with barriers around
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    if (lane_id() == 0) {
      if (lo) atomicOr(&s_diff[0], lo);
      if (hi) atomicOr(&s_diff[1], hi);
    }
    __syncthreads();
    uint32_t* dst = counts + (size_t)cur * 8u * 256u;
    for (uint32_t i = threadIdx.x; i < passes * 256u; i += kSegHistThreads) {
      const uint32_t v = h[i];
      if (v) atomicAdd(dst + i, v);
      h[i] = 0u;
    }
    if (threadIdx.x < 2) {
      if (s_diff[threadIdx.x]) atomicOr(&plans[cur].diff[threadIdx.x], s_diff[threadIdx.x]);
      s_diff[threadIdx.x] = 0u;
    }
    __syncthreads();
    diff = 0;
  };
  for (uint32_t t = t_lo; t < t_hi; t++) {
    const uint32_t sg = tile_seg[t];
    if (sg != cur) {  // uniform: every thread reads the same word
      __syncthreads();
      if (cur != 0xffffffffu) flush();
      cur = sg;
      passes = plans[sg].passes;
      first = data[seg_off[sg]].key;
      if (threadIdx.x < passes) s_win[threadIdx.x] = top_window(plans[sg], (int)threadIdx.x);
      __syncthreads();
    }
    const uint64_t sb = (uint64_t)seg_off[sg], se = (uint64_t)seg_off[sg + 1];
    const uint64_t b0 = sb + (uint64_t)(t - seg_tile0[sg]) * tile;
    const uint64_t b1 = min(se, b0 + tile);
    for (uint64_t i = b0 + threadIdx.x; i < b1; i += kSegHistThreads * kSegHistUnroll) {
      uint64_t key[kSegHistUnroll];
#pragma unroll
      for (uint32_t u = 0; u < kSegHistUnroll; u++)
        key[u] = i + u * kSegHistThreads < b1 ? load_elem_stream(data + i + u * kSegHistThreads).key : first;
#pragma unroll
      for (uint32_t u = 0; u < kSegHistUnroll; u++) diff |= key[u] ^ first;
      for (uint32_t p = 0; p < passes; p++) {
        const TopWindow w = s_win[p];
#pragma unroll
        for (uint32_t u = 0; u < kSegHistUnroll; u++)
          if (i + u * kSegHistThreads < b1)
            atomicAdd(&h[p * 256u + (w.clamp ? top_digit_clamped(w, key[u]) : top_digit(w, key[u]))], 1u);
      }
    }
  }
  __syncthreads();
  if (t_lo < t_hi) flush();
}

// per (segment, pass): exclusive scan of the digit counts, in place; whether
// the digits are all there is; block 0 also writes what lsb_query reports (every
// pass runs, no digit is skipped per batch)
__global__ void __launch_bounds__(256)
    k_seg_plan(const Elem* __restrict__ data, const int64_t* __restrict__ seg_off, SegPlan* __restrict__ plans,
               uint32_t* __restrict__ counts, uint32_t nseg, int num_digits, uint32_t n, int api_bits, int sub,
               Ctrl* ctrl) {
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  for (uint32_t sg = blockIdx.x; sg < nseg; sg += gridDim.x) {
    const uint32_t passes = plans[sg].passes;
    if (warp < passes) {  // warp p scans digit p
      uint32_t* c = counts + ((size_t)sg * 8u + warp) * 256u + lane * 8u;
      uint32_t v[8], sum = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        v[i] = sum;
        sum += c[i];
      }
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) c[i] = inc - sum + v[i];
    }
    if (passes && threadIdx.x == 0) {
      SegPlan& p = plans[sg];
      const uint64_t d = (uint64_t)p.diff[1] << 32 | p.diff[0];
      const bool inside = p.hb1 >= 64u || ((d | (data[seg_off[sg]].key ^ p.lo)) >> p.hb1) == 0;
      p.clamp = inside ? 0u : 1u;
      p.complete = (d == 0 || (p.hb1 <= 8u * passes && inside)) ? 1u : 0u;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl->skip_mask_lo = 0;
    ctrl->skip_mask_hi = 0;
    ctrl->passes_run = (uint32_t)num_digits;
    ctrl->num_passes = (uint32_t)num_digits;
    ctrl->final_copy = (uint32_t)num_digits & 1u;
    ctrl->api_bits = (uint32_t)api_bits;
    ctrl->sub = (uint32_t)sub;
    ctrl->n = n;
  }
}

// ---------------------------------------------------------------------------
// the arrays' runs, as k_top_finish for one array; arrays of a tile whole

__global__ void __launch_bounds__(Tile::kThreads, 2)
    k_seg_finish(Elem* __restrict__ X, Elem* __restrict__ Y, uint32_t n, uint32_t stride,
                 const int64_t* __restrict__ seg_off,
                 const SegPlan* __restrict__ plans, const uint32_t* __restrict__ seg_part0,
                 const uint32_t* __restrict__ part_seg, const uint32_t* __restrict__ num_parts,
                 RunChunk* __restrict__ chunks, uint32_t* __restrict__ unsorted, Ctrl* ctrl) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ typename Tile::Shared sh;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ RunMarks s_marks;
  __shared__ RunKey s_w;
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Tile::kElemBytes + Tile::kSlotBytes);
  if (error_raised(ctrl)) return;
  const uint32_t bar = smem_u32(&s_bar);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  uint32_t phase = 0;
  const uint32_t parts = *num_parts;
  for (uint32_t part = blockIdx.x; part < parts; part += gridDim.x) {
    const uint32_t s = part_seg[part];
    const SegPlan& plan = plans[s];
    const uint32_t at = (uint32_t)seg_off[s], len = (uint32_t)(seg_off[s + 1] - seg_off[s]);
    const uint32_t passes = plan.passes, par = passes & 1u;
    const uint32_t g = (part - seg_part0[s]) * stride;
    const uint32_t limit = (uint32_t)min((uint64_t)g + stride, (uint64_t)len);
    const Elem* src = (par ? Y : X) + at;
    Elem* dst = X + at;
    if (passes && plan.complete) {  // in order: at most to be copied
      if (par)
        for (uint32_t i = g + threadIdx.x; i < limit; i += Tile::kThreads) store_elem(dst + i, load_elem_stream(src + i));
      continue;
    }
    auto load = [&](uint32_t from, uint32_t cnt) { return load_tile_bulk(in, src + from, cnt, bar, &phase, ctrl); };
    if (passes == 0u) {
      if (len < 2u) continue;
      if (!load(0u, len)) return;
      Tile::sort(in, 0u, len, 0ull, 0ull, slot, bins, sh, true, Uneven::kDups,
                 [=](bool on, uint32_t r, const Elem& e) { store_elem_if(on, dst + r, e); });
      continue;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_w = run_key(plan);
    auto long_run = [&](uint32_t b, uint32_t e) { push_run(ctrl, chunks, unsorted, n, at + b, at + e, par); };
    if (!sort_runs<Tile>(src, dst, len, g, limit, g == 0, s_w, plan.clamp != 0u, (plan.skewed & 1u) != 0u, (plan.skewed & 2u) != 0u,
                         run_key(plan).shift, in, slot, bins, sh, s_marks, load, long_run))
      return;
  }
}

// ---------------------------------------------------------------------------
// layout and driver

struct SegLayout {
  int api_bits = 0, sub = 1, num_digits = 0, variant = 0;
  uint32_t n = 0, nseg = 0, tile = 0, stride = 0, max_tiles = 0, max_parts = 0, ctas = 0;
  size_t off_plans = 0, off_tile0 = 0, off_part0 = 0, off_ntiles = 0, off_tile_seg = 0, off_part_seg = 0,
         off_counts = 0, off_ring = 0, total = 0;
};

// ctas: persistent CTAs of the scatter passes (0 = every resident slot: SMs x
// CTAs per SM); fewer CTAs keep fewer tiles in flight at once.
static int seg_plan_layout(int64_t n, int64_t nseg, int digit_bits, int variant, SegLayout* L,
                           int ctas = 0) {
  DeviceInfo dev;
  if (int rc = current_device_info(&dev)) return rc;
  *L = SegLayout();
  int sub = 1, P = lsb_num_passes(digit_bits);
  if (digit_bits > 11) {
    if (digit_bits % 2 || digit_bits > 16) return LSB_ERR_INVALID_ARG;  // odd wide widths: no segmented form
    const int bits = digit_bits / 2;
    sub = 2;
    P = std::min(2 * P, (64 + bits - 1) / bits);
  }
  L->api_bits = digit_bits;
  L->sub = sub;
  L->num_digits = P;  // as lsb_query reports them; the kernels choose their own digits
  L->variant = variant;
  L->n = (uint32_t)n;
  L->nseg = (uint32_t)nseg;
  L->ctas = ctas > 0 ? (uint32_t)ctas : 0u;
  L->tile = onesweep_top_tile(variant);
  L->max_tiles = (uint32_t)((uint64_t)n / L->tile + (uint64_t)nseg + 1u);
  // a CTA's part of an array in the last step: up to four tiles, less when the
  // batch would not give every resident CTA four parts
  L->stride = (uint32_t)std::min<uint64_t>(4u * kCap, std::max<uint64_t>(2048u, (uint64_t)n / ((uint64_t)dev.sm_count * 8u)));
  L->max_parts = (uint32_t)((uint64_t)n / L->stride + (uint64_t)nseg + 1u);
  size_t off = kCtrlBytes;
  L->off_plans = off;
  off = align_up(off + (size_t)nseg * sizeof(SegPlan), 256);
  L->off_tile0 = off;
  off = align_up(off + (size_t)nseg * 4u, 256);
  L->off_part0 = off;
  off = align_up(off + (size_t)nseg * 4u, 256);
  L->off_ntiles = off;
  off = align_up(off + 9u * 4u, 256);
  L->off_tile_seg = off;
  off = align_up(off + (size_t)L->max_tiles * 4u, 256);
  L->off_part_seg = off;
  off = align_up(off + (size_t)L->max_parts * 4u, 256);
  L->off_counts = off;
  off = align_up(off + (size_t)nseg * 8u * 256u * 4u, 256);
  // the ring: a slot for each tile of an array above a tile's size (fewer than
  // n / tile plus one for each such array), later the list of long runs
  const uint64_t ring_tiles = (uint64_t)n / L->tile + std::min<uint64_t>((uint64_t)nseg, (uint64_t)n / kCap) + 1u;
  L->off_ring = off;
  off = align_up(off + std::max<size_t>((size_t)ring_tiles * 256u * 8u, top_list_bytes((uint32_t)n)), 256);
  L->total = off;
  return LSB_OK;
}

static int seg_run(Elem* A, Elem* B, const int64_t* seg_off, void* ws, const SegLayout& L,
                   cudaStream_t st) {
  unsigned char* w = static_cast<unsigned char*>(ws);
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(w);
  SegPlan* plans = reinterpret_cast<SegPlan*>(w + L.off_plans);
  uint32_t* seg_tile0 = reinterpret_cast<uint32_t*>(w + L.off_tile0);
  uint32_t* seg_part0 = reinterpret_cast<uint32_t*>(w + L.off_part0);
  uint32_t* ntiles = reinterpret_cast<uint32_t*>(w + L.off_ntiles);
  uint32_t* tile_seg = reinterpret_cast<uint32_t*>(w + L.off_tile_seg);
  uint32_t* part_seg = reinterpret_cast<uint32_t*>(w + L.off_part_seg);
  uint32_t* counts = reinterpret_cast<uint32_t*>(w + L.off_counts);
  uint64_t* ring = reinterpret_cast<uint64_t*>(w + L.off_ring);
  if (cudaMemsetAsync(w, 0, kCtrlBytes, st) != cudaSuccess ||
      cudaMemsetAsync(counts, 0, L.total - L.off_counts, st) != cudaSuccess)
    return LSB_ERR_CUDA;
  DeviceInfo dev;
  if (int rc = current_device_info(&dev)) return rc;
  const size_t sample_smem = kSampleSmem<kSegSample>;
  static std::atomic<uint64_t> allowed[2];
  if (!allow_smem((const void*)k_seg_sample, sample_smem, &allowed[0]) ||
      !allow_smem((const void*)k_seg_finish, Tile::kSmem, &allowed[1]))
    return LSB_ERR_CUDA;
  {
    ProfScope prof("seg_sample", st);
    k_seg_sample<<<std::min<uint32_t>(L.nseg, (uint32_t)dev.sm_count * 2u), kSampleThreads, sample_smem, st>>>(
        A, seg_off, L.nseg, straddle_time(L.n), plans);
  }
  {
    ProfScope prof("seg_tiles", st);
    k_seg_tiles<<<1, kSegScanThreads, 0, st>>>(seg_off, L.nseg, L.tile, L.stride, plans, seg_tile0, seg_part0, ntiles);
    k_seg_fill<<<std::max<uint32_t>(1, std::min<uint32_t>((L.nseg + 7) / 8, 4096)), 256, 0, st>>>(
        seg_off, L.nseg, L.tile, L.stride, plans, seg_tile0, seg_part0, tile_seg, part_seg);
  }
  {
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(L.max_tiles, dev.sm_count * 4u));
    ProfScope prof("seg_hist", st);
    k_seg_hist<<<grid, kSegHistThreads, 0, st>>>(A, seg_off, seg_tile0, tile_seg, ntiles, L.tile, plans, counts);
  }
  {
    ProfScope prof("seg_plan", st);
    k_seg_plan<<<std::max<uint32_t>(1, std::min<uint32_t>(L.nseg, 4096)), 256, 0, st>>>(
        A, seg_off, plans, counts, L.nseg, L.num_digits, L.n, L.api_bits, L.sub, ctrl);
  }
  if (cudaPeekAtLastError() != cudaSuccess) return LSB_ERR_CUDA;
  SegDesc seg;
  seg.tile_seg = tile_seg;
  seg.seg_tile0 = seg_tile0;
  seg.seg_off = seg_off;
  seg.seg_gstart = counts;
  seg.num_tiles = ntiles;
  seg.plan = plans;
  // a launch for each pass that an array of all the elements needs when its keys
  // are even, and one for whatever passes follow
  const uint32_t passes = passes_for((float)L.n, (float)kMeanRun);
  for (uint32_t p = 0; p < passes; p++)
    if (onesweep_top_pass(A, B, L.n, (int)p, nullptr, ring, L.max_tiles, ctrl, seg, L.variant, L.ctas, dev, st))
      return LSB_ERR_CUDA;
  if (onesweep_top_rest(A, B, L.n, (int)passes, nullptr, ring, L.max_tiles, ctrl, seg, L.variant, L.ctas, dev, st))
    return LSB_ERR_CUDA;
  RunChunk* chunks = reinterpret_cast<RunChunk*>(ring);
  uint32_t* unsorted = reinterpret_cast<uint32_t*>(chunks + max_chunks(L.n));
  {
    // parts beyond the grid follow in turn; the grid is as long as most batches
    ProfScope prof("seg_finish", st);
    k_seg_finish<<<std::min<uint32_t>(L.max_parts, 1u << 20), Tile::kThreads, Tile::kSmem, st>>>(
        A, B, L.n, L.stride, seg_off, plans, seg_part0, part_seg, ntiles + 8, chunks, unsorted, ctrl);
  }
  if (cudaPeekAtLastError() != cudaSuccess) return LSB_ERR_CUDA;
  return top_merge(A, B, L.n, chunks, unsorted, ctrl, dev, st) ? LSB_ERR_CUDA : LSB_OK;
}

static int tuning_variant(const lsb_tuning_t* t) {
  return (t && (t->variant == 0 || t->variant == 2)) ? t->variant : 0;
}
static int tuning_bits(const lsb_tuning_t* t) {
  return (t && t->digit_bits >= 1 && t->digit_bits <= 16) ? t->digit_bits : 8;
}
static int tuning_ctas(const lsb_tuning_t* t) { return (t && t->ctas > 0) ? t->ctas : 0; }

static int seg_check(const lsb_elem_t* a, const lsb_elem_t* b, int64_t n, const int64_t* off,
                     int64_t nseg) {
  if (n < 0 || nseg < 0) return LSB_ERR_INVALID_ARG;
  if (n > LSB_MAX_ELEMENTS || nseg > LSB_MAX_ELEMENTS) return LSB_ERR_TOO_LARGE;
  if (nseg > 0 && !off) return LSB_ERR_INVALID_ARG;
  if (n > 0 && (!a || !b)) return LSB_ERR_INVALID_ARG;
  if ((((uintptr_t)a) | ((uintptr_t)b)) & 15u) return LSB_ERR_ALIGNMENT;
  if (((uintptr_t)off) & 7u) return LSB_ERR_ALIGNMENT;
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b, len = (uintptr_t)n * 16u;
  if (n > 0 && x < y + len && y < x + len) return LSB_ERR_OVERLAP;
  return LSB_OK;
}

// ---------------------------------------------------------------------------
// autotuner: times the candidate configurations on a sample batch with the
// caller's segment sizes (random keys) and keeps the fastest per size class

static std::mutex g_tune_mu;
static std::map<std::pair<int, int>, lsb_tuning_t> g_tune_cache;

}  // namespace lsb

using namespace lsb;

extern "C" {

int lsb_segmented_workspace_bytes(int64_t n_total, int64_t nseg, int digit_bits, size_t* bytes) {
  if (!bytes || n_total < 0 || nseg < 0 || digit_bits < 1 || digit_bits > 16)
    return LSB_ERR_INVALID_ARG;
  if (n_total > LSB_MAX_ELEMENTS || nseg > LSB_MAX_ELEMENTS) return LSB_ERR_TOO_LARGE;
  size_t best = 0;
  for (int v : {0, 2}) {
    SegLayout L;
    if (int rc = seg_plan_layout(n_total, nseg, digit_bits, v, &L)) return rc;
    best = std::max(best, L.total);
  }
  *bytes = best;
  return LSB_OK;
}

int lsb_sort_segmented(lsb_elem_t* d_a, lsb_elem_t* d_b, int64_t n_total,
                       const int64_t* d_seg_offsets, int64_t nseg, const lsb_tuning_t* opt_tuning,
                       void* d_workspace, size_t workspace_bytes, void* stream) {
  if (int rc = seg_check(d_a, d_b, n_total, d_seg_offsets, nseg)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_total <= 1 || nseg == 0) return LSB_OK;
  SegLayout L;
  if (int rc = seg_plan_layout(n_total, nseg, tuning_bits(opt_tuning), tuning_variant(opt_tuning),
                               &L, tuning_ctas(opt_tuning)))
    return rc;
  Elem* A = reinterpret_cast<Elem*>(d_a);
  Elem* B = reinterpret_cast<Elem*>(d_b);
  if (d_workspace) {
    if (((uintptr_t)d_workspace & 255u) || workspace_bytes < L.total) return LSB_ERR_WORKSPACE;
    return seg_run(A, B, d_seg_offsets, d_workspace, L, st);
  }
  if (workspace_bytes) return LSB_ERR_WORKSPACE;
  void* w = nullptr;
  if (cudaMallocAsync(&w, L.total, st) != cudaSuccess) {
    cudaGetLastError();
    return LSB_ERR_NO_MEMORY;
  }
  int rc = seg_run(A, B, d_seg_offsets, w, L, st);
  uint32_t dev_err = 0;
  if (rc == LSB_OK &&
      cudaMemcpyAsync(&dev_err, w, sizeof dev_err, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    rc = LSB_ERR_CUDA;
  cudaFreeAsync(w, st);
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == LSB_OK) rc = LSB_ERR_CUDA;
  return (rc == LSB_OK && dev_err) ? (int)dev_err : rc;
}

int lsb_tune_segmented(const int64_t* h_seg_offsets, int64_t nseg, lsb_tuning_t* out,
                       void* stream) {
  if (!out || nseg < 0 || (nseg > 0 && !h_seg_offsets)) return LSB_ERR_INVALID_ARG;
  std::memset(out, 0, sizeof *out);
  out->digit_bits = 8;
  out->variant = 0;
  if (nseg == 0) return LSB_OK;
  const int64_t n = h_seg_offsets[nseg] - h_seg_offsets[0];
  if (n <= 0) return LSB_OK;
  if (n > LSB_MAX_ELEMENTS) return LSB_ERR_TOO_LARGE;
  // size class: log2 of the total and of the mean segment size
  int lt = 0, lm = 0;
  while ((int64_t(1) << lt) < n) lt++;
  while ((int64_t(1) << lm) < n / nseg) lm++;
  const std::pair<int, int> key{lt, lm};
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      *out = it->second;
      return LSB_OK;
    }
  }
  // sample: every k-th segment, at most ~2^26 elements, same size mix
  const int64_t budget = int64_t(1) << 26;
  const int64_t stride = std::max<int64_t>(1, (n + budget - 1) / budget);
  std::vector<int64_t> off{0};
  for (int64_t s = 0; s < nseg; s += stride)
    off.push_back(off.back() + (h_seg_offsets[s + 1] - h_seg_offsets[s]));
  const int64_t sn = off.back();
  const int64_t sseg = (int64_t)off.size() - 1;
  if (sn <= 1) return LSB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int width = 8;  // the kernels choose their own digits: another width changes nothing
  const int cand_var[] = {0, 2};
  size_t wsb = 0;
  if (int rc = lsb_segmented_workspace_bytes(sn, sseg, width, &wsb)) return rc;
  DeviceInfo dev;
  if (int rc = current_device_info(&dev)) return rc;
  // CTA counts: every resident slot, or one CTA per SM with two-CTA shapes, or half the SMs
  const int cand_ctas[] = {0, dev.sm_count, std::max(1, dev.sm_count / 2)};
  void *in = nullptr, *a = nullptr, *b = nullptr, *ws = nullptr, *doff = nullptr;
  const size_t bytes = (size_t)sn * sizeof(Elem);
  int rc = LSB_OK;
  if (cudaMallocAsync(&in, bytes, st) != cudaSuccess || cudaMallocAsync(&a, bytes, st) != cudaSuccess ||
      cudaMallocAsync(&b, bytes, st) != cudaSuccess || cudaMallocAsync(&ws, wsb, st) != cudaSuccess ||
      cudaMallocAsync(&doff, off.size() * 8u, st) != cudaSuccess) {
    cudaGetLastError();
    rc = LSB_ERR_NO_MEMORY;
  }
  if (rc == LSB_OK &&
      (cudaMemcpyAsync(doff, off.data(), off.size() * 8u, cudaMemcpyHostToDevice, st) != cudaSuccess ||
       lsb_generate((lsb_elem_t*)in, sn, LSB_DIST_UNIFORM, 12345, stream) != LSB_OK))
    rc = LSB_ERR_CUDA;
  float best_ms = 1e30f;
  lsb_tuning_t best = *out;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (rc == LSB_OK && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess))
    rc = LSB_ERR_CUDA;
  for (int cv : cand_var) {
    for (int cc : cand_ctas) {
      if (rc != LSB_OK) break;
      if (cv == 0 && cc == dev.sm_count) continue;  // the variant-0 default is already one CTA per SM
      lsb_tuning_t t;
      std::memset(&t, 0, sizeof t);
      t.digit_bits = width;
      t.variant = cv;
      t.ctas = cc;
      float total = 0.f;
      for (int rep = 0; rep < 3 && rc == LSB_OK; rep++) {
        if (cudaMemcpyAsync(a, in, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess) rc = LSB_ERR_CUDA;
        cudaEventRecord(e0, st);
        if (rc == LSB_OK)
          rc = lsb_sort_segmented((lsb_elem_t*)a, (lsb_elem_t*)b, sn, (const int64_t*)doff, sseg, &t,
                                  ws, wsb, stream);
        cudaEventRecord(e1, st);
        if (cudaEventSynchronize(e1) != cudaSuccess) rc = LSB_ERR_CUDA;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0) total += ms;  // first run warms the configuration up
      }
      if (rc == LSB_OK && total < best_ms) {
        best_ms = total;
        best = t;
      }
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  for (void* p : {in, a, b, ws, doff})
    if (p) cudaFreeAsync(p, st);
  cudaStreamSynchronize(st);
  if (rc != LSB_OK) return rc;
  *out = best;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune_cache[key] = best;
  return LSB_OK;
}

struct lsb_graph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

int lsb_graph_capture_segmented(lsb_elem_t* d_a, lsb_elem_t* d_b, int64_t n_total,
                                const int64_t* d_seg_offsets, int64_t nseg,
                                const lsb_tuning_t* opt_tuning, void* d_workspace,
                                size_t workspace_bytes, lsb_graph_t** out) {
  if (!out || !d_workspace) return LSB_ERR_INVALID_ARG;
  *out = nullptr;
  if (int rc = seg_check(d_a, d_b, n_total, d_seg_offsets, nseg)) return rc;
  // resolve device properties and kernel attributes before capturing
  SegLayout L;
  if (int rc = seg_plan_layout(n_total, nseg, tuning_bits(opt_tuning), tuning_variant(opt_tuning),
                               &L, tuning_ctas(opt_tuning)))
    return rc;
  if (((uintptr_t)d_workspace & 255u) || workspace_bytes < L.total) return LSB_ERR_WORKSPACE;
  cudaStream_t cs = nullptr;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) return LSB_ERR_CUDA;
  lsb_graph* g = new lsb_graph();
  int rc = LSB_OK;
  if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = LSB_ERR_CUDA;
  if (rc == LSB_OK) {
    rc = lsb_sort_segmented(d_a, d_b, n_total, d_seg_offsets, nseg, opt_tuning, d_workspace,
                            workspace_bytes, cs);
    if (cudaStreamEndCapture(cs, &g->graph) != cudaSuccess && rc == LSB_OK) rc = LSB_ERR_CUDA;
  }
  if (rc == LSB_OK && cudaGraphInstantiate(&g->exec, g->graph, 0) != cudaSuccess) rc = LSB_ERR_CUDA;
  cudaStreamDestroy(cs);
  if (rc != LSB_OK) {
    cudaGetLastError();
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    delete g;
    return rc;
  }
  *out = g;
  return LSB_OK;
}

int lsb_graph_launch(lsb_graph_t* g, void* stream) {
  if (!g || !g->exec) return LSB_ERR_INVALID_ARG;
  return cudaGraphLaunch(g->exec, (cudaStream_t)stream) == cudaSuccess ? LSB_OK : LSB_ERR_CUDA;
}

int lsb_graph_destroy(lsb_graph_t* g) {
  if (!g) return LSB_OK;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  delete g;
  return LSB_OK;
}

}  // extern "C"
