// lsb_tile.cuh -- the stable sort of one tile that lies in shared memory, by
// its whole 64-bit keys, in one CTA.
//
// A tile of m elements is sorted through an array of 32-bit slots, so that
// the 16-byte elements themselves are read once, at the end, in sorted order:
//   1. smallest and largest key; a tile that is in order already is done;
//   2. each key's bin: the range [min, max] is cut into NB equal bins, 1.8
//      or more per element, and one shared atomic per element counts them and
//      gives the element a place among its bin's (in any order);
//   3. an exclusive scan of the bins' counts; each element's slot is written:
//      (the key's next 18 or 19 bits below the bin, the element's position in the tile);
//   4. an element's rank in its bin is the number of its bin's slots below
//      its own: positions break ties, which makes the sort stable although the
//      atomics are not. Slots that agree in the key bits compare whole keys.
// So a tile costs one atomic per element whatever the key width, where ranking
// by 8-bit digits (ballots and per-warp counters) costs one round per digit.
// Evenly spread keys put 0.56 elements in a bin at most on average. A tile
// with a bin above kMaxBin elements (duplicates, clusters) is sorted by merging
// instead: K consecutive elements per thread by a sorting network, then
// log2(threads) rounds of merge-path merges of position lists. That costs the
// same for any keys: about six times the even case.
#pragma once

#include "lsb_device.cuh"

namespace lsb {

template <int THREADS, int K>
struct TileSort {
  static constexpr int kThreads = THREADS;
  static constexpr int kItems = K;
  static constexpr int kWarps = THREADS / 32;
  static constexpr uint32_t kCap = (uint32_t)THREADS * K;     // largest tile
  static constexpr int kBinsPerThread = 16;
  static constexpr uint32_t kBins = (uint32_t)THREADS * kBinsPerThread;
  static constexpr uint32_t kPosBits = kCap <= 8192 ? 13 : 14;  // bits of a position in a slot
  static constexpr uint32_t kPosMask = (1u << kPosBits) - 1u;
  static constexpr uint32_t kMaxBin = 40;
  static_assert(kCap <= (1u << kPosBits) && K <= 16 && kWarps <= 32, "position bits, network, warp totals");

  // shared memory: elements, slots (or two position lists), bin counts (16 bits each)
  static constexpr size_t kElemBytes = (size_t)kCap * sizeof(Elem);
  static constexpr size_t kSlotBytes = (size_t)kCap * 4u;
  static constexpr size_t kBinBytes = (size_t)kBins * 2u;
  static constexpr size_t kSmem = kElemBytes + kSlotBytes + kBinBytes;

  struct Shared {
    uint64_t wmin[kWarps], wmax[kWarps];
    uint32_t wdiff[2][kWarps];
    uint32_t wtot[kWarps];
  };

  static __device__ __forceinline__ uint64_t warp_min(uint64_t v) {
    const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(v >> 32));
    const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0xffffffffu);
    return (uint64_t)hi << 32 | lo;
  }
  static __device__ __forceinline__ uint64_t warp_max(uint64_t v) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u);
    return (uint64_t)hi << 32 | lo;
  }

  // Bin and, below it, 32 bits of fraction of a key: monotone in the key.
  // x = (key - min) >> sh fits 32 bits; with f = 0 there are fewer distinct x
  // than bins (then sh is 0 and a bin holds one key value), else the bin is
  // floor(x * f / 2^32).
  struct Scale {
    uint64_t base;
    uint32_t sh, f;
  };
  static __device__ __forceinline__ Scale make_scale(uint64_t mn, uint64_t mx) {
    Scale s;
    const uint64_t range = mx - mn;
    s.base = mn;
    const int lz = __clzll((long long)range);
    s.sh = lz < 32 ? (uint32_t)(32 - lz) : 0u;
    const uint32_t xr = (uint32_t)(range >> s.sh);
    s.f = xr < kBins ? 0u : (uint32_t)(((uint64_t)kBins << 32) / ((uint64_t)xr + 1u));
    return s;
  }
  static __device__ __forceinline__ uint32_t bin_of(const Scale& s, uint64_t key, uint32_t* frac) {
    const uint32_t x = (uint32_t)((key - s.base) >> s.sh);
    const uint64_t p = (uint64_t)x * s.f;
    *frac = s.f ? (uint32_t)p : 0u;
    return s.f ? (uint32_t)(p >> 32) : x;
  }

  // Sorts the m <= kCap elements in[0..m) (shared memory, not changed) and
  // calls emit(rank, element) once for each from the thread that holds it;
  // neighbouring threads get neighbouring ranks but for a bin's few elements.
  // If the tile is in order already: nothing is emitted when `in_place`.
  // `slot` and `bins` are the tile's shared arrays; every thread of the CTA
  // calls this together, after a barrier that makes in[] visible. On return
  // threads may still be reading in[], slot[] and bins[]: a barrier is due
  // before they are written again. With diff_out, thread 0 gets there the bits
  // in which any two keys differ.
  template <typename Emit>
  static __device__ __forceinline__ void sort(const Elem* in, uint32_t m, uint32_t* slot, uint32_t* bins,
                                              Shared& sh, bool in_place, Emit emit,
                                              uint64_t* diff_out = nullptr) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    // 1. zero the bins; smallest and largest key, order
    {
      uint4* z = reinterpret_cast<uint4*>(bins) + tid * 2u;
      z[0] = make_uint4(0, 0, 0, 0);
      z[1] = make_uint4(0, 0, 0, 0);
    }
    uint64_t mn = ~0ull, mx = 0ull;
    bool inversion = false;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p < m) {
        const uint64_t key = in[p].key;
        mn = key < mn ? key : mn;
        mx = key > mx ? key : mx;
        if (p) inversion |= in[p - 1u].key > key;
      }
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane == 0) {
      sh.wmin[warp] = mn;
      sh.wmax[warp] = mx;
    }
    if (diff_out) {
      uint64_t x = 0;
      const uint64_t k0 = in[0].key;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t p = tid + (uint32_t)k * THREADS;
        if (p < m) x |= in[p].key ^ k0;
      }
      const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)x);
      const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(x >> 32));
      if (lane == 0) {
        sh.wdiff[0][warp] = lo;
        sh.wdiff[1][warp] = hi;
      }
    }
    const bool unsorted = __syncthreads_or(inversion);
    if (diff_out && tid == 0) {
      uint64_t x = 0;
      for (int w = 0; w < kWarps; w++) x |= (uint64_t)sh.wdiff[1][w] << 32 | sh.wdiff[0][w];
      *diff_out = x;
    }
    if (!unsorted) {
      if (!in_place) {
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t p = tid + (uint32_t)k * THREADS;
          if (p < m) emit(p, in[p]);
        }
      }
      return;
    }
    mn = warp_min(lane < (uint32_t)kWarps ? sh.wmin[lane] : ~0ull);
    mx = warp_max(lane < (uint32_t)kWarps ? sh.wmax[lane] : 0ull);
    const Scale sc = make_scale(mn, mx);

    // 2. count: bin, place among the bin's elements and fraction of each element
    uint32_t place[K], frac[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p < m) {
        const uint32_t b = bin_of(sc, in[p].key, &frac[k]);
        const uint32_t s16 = (b & 1u) << 4;
        const uint32_t old = atomicAdd(&bins[b >> 1], 1u << s16);
        place[k] = b << 16 | ((old >> s16) & 0xffffu);
      }
    }
    __syncthreads();
    // 3. exclusive scan of the counts; thread t owns bins [16 t, 16 t + 16)
    uint32_t w8[8], maxc = 0, sum = 0;
    {
      const uint4* q = reinterpret_cast<const uint4*>(bins) + tid * 2u;
      const uint4 a = q[0], b = q[1];
      w8[0] = a.x, w8[1] = a.y, w8[2] = a.z, w8[3] = a.w;
      w8[4] = b.x, w8[5] = b.y, w8[6] = b.z, w8[7] = b.w;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t lo = w8[i] & 0xffffu, hi = w8[i] >> 16;
      maxc = max(maxc, max(lo, hi));
      w8[i] = sum | (sum + lo) << 16;
      sum += lo + hi;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) sh.wtot[warp] = inc;
    const bool uneven = __syncthreads_or(maxc > kMaxBin);
    if (uneven) {
      merge_sorted(in, m, slot, emit);
      return;
    }
    {
      uint32_t off = inc - sum;
      const uint32_t wt = lane < (uint32_t)kWarps ? sh.wtot[lane] : 0u;
      off += __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
      const uint32_t both = off | off << 16;
      uint4* q = reinterpret_cast<uint4*>(bins) + tid * 2u;
      q[0] = make_uint4(w8[0] + both, w8[1] + both, w8[2] + both, w8[3] + both);
      q[1] = make_uint4(w8[4] + both, w8[5] + both, w8[6] + both, w8[7] + both);
    }
    __syncthreads();
    const uint16_t* start = reinterpret_cast<const uint16_t*>(bins);
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p < m) slot[start[place[k] >> 16] + (place[k] & 0xffffu)] = (frac[k] & ~kPosMask) | p;
    }
    __syncthreads();
    // 4. rank inside the bin, elements out
#pragma unroll 3
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p < m) {
        const uint32_t v = slot[p];
        const Elem e = in[v & kPosMask];
        uint32_t f;
        const uint32_t b = bin_of(sc, e.key, &f);
        const uint32_t s = start[b], t = b + 1u < kBins ? start[b + 1u] : m;
        uint32_t r = s, close = 0;
        for (uint32_t q = s; q < t; q++) {
          const uint32_t u = slot[q];
          r += u < v ? 1u : 0u;
          close += (u ^ v) <= kPosMask ? 1u : 0u;
        }
        if (close > 1u) {  // key bits of the slots agree: whole keys, then positions
          r = s;
          for (uint32_t q = s; q < t; q++) {
            const uint32_t j = slot[q] & kPosMask;
            const uint64_t kj = in[j].key;
            r += (kj < e.key || (kj == e.key && j < (v & kPosMask))) ? 1u : 0u;
          }
        }
        emit(r, e);
      }
    }
  }

  // One thread's K outputs of the stable merge of neighbouring sorted position
  // lists of length len (src, m positions in all) into dst.
  static __device__ __forceinline__ void merge_round(const Elem* in, const uint16_t* src, uint16_t* dst,
                                                     uint32_t m, uint32_t len) {
    const uint32_t d0 = threadIdx.x * (uint32_t)K;
    if (d0 >= m) return;
    const uint32_t base = d0 / (2u * len) * (2u * len);
    const uint32_t la = min(len, m - base), lb = min(len, m - base - la);
    const uint16_t* a = src + base;
    const uint16_t* b = a + la;
    const uint32_t d = d0 - base;
    uint32_t lo = d > lb ? d - lb : 0u, hi = min(d, la);
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (in[a[mid]].key <= in[b[d - 1u - mid]].key) lo = mid + 1u;
      else hi = mid;
    }
    uint32_t i = lo, j = d - lo;
    const uint32_t cnt = min((uint32_t)K, m - d0);
    uint32_t pa = i < la ? a[i] : 0u, pb = j < lb ? b[j] : 0u;
    uint64_t ka = in[pa].key, kb = in[pb].key;
    for (uint32_t q = 0; q < cnt; q++) {
      if (j >= lb || (i < la && ka <= kb)) {
        dst[d0 + q] = (uint16_t)pa;
        if (++i < la) ka = in[pa = a[i]].key;
      } else {
        dst[d0 + q] = (uint16_t)pb;
        if (++j < lb) kb = in[pb = b[j]].key;
      }
    }
  }

  // The same result for any keys, by merging (see the head of this file).
  template <typename Emit>
  static __device__ __noinline__ void merge_sorted(const Elem* in, uint32_t m, uint32_t* slot, Emit emit) {
    uint16_t* cur = reinterpret_cast<uint16_t*>(slot);
    uint16_t* nxt = cur + kCap;
    const uint32_t d0 = threadIdx.x * (uint32_t)K;
    {
      // K neighbours per thread: odd-even transposition, which keeps equal keys in place
      uint64_t key[K];
      uint32_t pos[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        pos[k] = d0 + (uint32_t)k;
        key[k] = pos[k] < m ? in[pos[k]].key : ~0ull;
      }
#pragma unroll
      for (int r = 0; r < K; r++) {
#pragma unroll
        for (int k = r & 1; k + 1 < K; k += 2) {
          if (key[k] > key[k + 1]) {
            const uint64_t t = key[k];
            key[k] = key[k + 1];
            key[k + 1] = t;
            const uint32_t u = pos[k];
            pos[k] = pos[k + 1];
            pos[k + 1] = u;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; k++)
        if (d0 + (uint32_t)k < m) cur[d0 + k] = (uint16_t)pos[k];
    }
    __syncthreads();
    for (uint32_t len = K; len < m; len *= 2u) {
      merge_round(in, cur, nxt, m, len);
      __syncthreads();
      uint16_t* t = cur;
      cur = nxt;
      nxt = t;
    }
    for (uint32_t p = threadIdx.x; p < m; p += THREADS) emit(p, in[cur[p]]);
  }
};

}  // namespace lsb
