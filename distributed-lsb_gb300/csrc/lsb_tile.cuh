// lsb_tile.cuh -- the stable sort of one tile that lies in shared memory, by
// its whole 64-bit keys, in one CTA.
//
// A tile of m elements is sorted through an array of 32-bit slots, so that
// the 16-byte elements themselves are read once, at the end, in sorted order:
//   1. each key's bin: a range that holds the tile's keys is cut into NB equal
//      bins, 1.8 or more per element, and one shared atomic per element counts
//      them and gives the element a place among its bin's (in any order);
//   2. an exclusive scan of the bins' counts; each element's slot is written:
//      (the key's next 18 to 22 bits below the bin, the element's position in the tile);
//   3. an element's rank in its bin is the number of its bin's slots below
//      its own: positions break ties, which makes the sort stable although the
//      atomics are not. Slots that agree in the key bits compare whole keys.
// So a tile costs one atomic per element whatever the key width, where ranking
// by 8-bit digits (ballots and per-warp counters) costs one round per digit.
// Evenly spread keys put 0.56 elements in a bin at most on average. When a bin
// has more than kMaxBin elements, the bins are laid over the range from the
// smallest to the largest key instead. What shares a bin then are mostly
// duplicates: bins of up to kSlotsBin elements are ranked by slots alone, which
// is checked before any element goes out (2^28 elements, every key thirty times:
// 12.1 ms; 14.7 ms when every pair's whole keys are compared); a warp takes a
// larger one key by key, and a bitmap of the key's positions gives the ranks
// (heavy_bins). A tile with many different keys in a large bin (clusters, signs,
// bits that never vary) gets bins that follow its keys (sort_spread); when that
// fails too it is sorted by the bits in which its keys differ, eight at a time from
// the lowest (stable ranks by ballots and per-warp counters; 10^4 Zipf keys took
// 52 us so, 37 with heavy_bins).
#pragma once

#include "lsb_device.cuh"

namespace lsb {

// Shared-memory accesses under a predicate: no branch around them, so that the
// K independent accesses of a thread are all in flight together.
__device__ __forceinline__ uint32_t atom_add_if(bool on, uint32_t* p, uint32_t v) {
  uint32_t old = 0;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p atom.shared.add.u32 %0, [%1], %2;\n}\n"
               : "+r"(old)
               : "r"(smem_u32(p)), "r"(v), "r"((uint32_t)on)
               : "memory");
  return old;
}
__device__ __forceinline__ void st_shared_if(bool on, uint32_t* p, uint32_t v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p st.shared.u32 [%0], %1;\n}\n" ::"r"(smem_u32(p)), "r"(v),
               "r"((uint32_t)on)
               : "memory");
}
__device__ __forceinline__ void store_elem_if(bool on, Elem* p, const Elem& e) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.global.v2.u64 [%0], {%1, %2};\n}\n" ::"l"(p), "l"(e.key),
               "l"(e.val), "r"((uint32_t)on)
               : "memory");
}

// What a tile whose keys are spread too unevenly for equal bins tries before it is
// sorted bit by bit: nothing (where a kernel sorts a tile or two, code that has to
// be fetched first costs as much as it saves), bins that follow the keys, or those
// only after the ways of duplicates.
enum class Uneven : uint32_t { kBits, kSpread, kDups };

template <int THREADS, int K>
struct TileSort {
  static constexpr int kThreads = THREADS;
  static constexpr int kItems = K;
  static constexpr int kWarps = THREADS / 32;
  static constexpr uint32_t kCap = (uint32_t)THREADS * K;     // largest tile
  static constexpr int kBinsPerThread = 16;
  static constexpr uint32_t kBins = (uint32_t)THREADS * kBinsPerThread;
  // bits of a position in a slot
  static constexpr uint32_t kPosBits = kCap <= 1024 ? 10 : kCap <= 2048 ? 11 : kCap <= 4096 ? 12 : kCap <= 8192 ? 13 : 14;
  static constexpr uint32_t kPosMask = (1u << kPosBits) - 1u;
  static constexpr uint32_t kMaxBin = 24;    // elements of a bin compared by whole keys
  static constexpr uint32_t kSlotsBin = 64;  // and, in a tile with bins above that, by slots
  static constexpr uint32_t kMaxHeavy = kCap / (kSlotsBin + 1u);  // bins above it
  static constexpr uint32_t kFewRounds = 4;  // of eight bits: no dearer than another try with bins
  static constexpr uint32_t kFewKeys = 12;   // of 32 in a heavy bin: taken key by key (6 and 24: within 1 %, whatever the keys)
  static_assert(kCap <= (1u << kPosBits) && K <= 16 && kWarps <= 32, "position bits, network, warp totals");

  // shared memory: elements, slots (or two position lists), bin counts (16 bits each)
  static constexpr size_t kElemBytes = (size_t)kCap * sizeof(Elem);
  static constexpr size_t kSlotBytes = (size_t)kCap * 4u + 16u;  // two position lists; what is read past the last slot
  static constexpr size_t kBinBytes = (size_t)kBins * 2u + 16u;  // and the end of the last bin
  static constexpr size_t kSmem = kElemBytes + kSlotBytes + kBinBytes;

  struct Shared {
    uint64_t wmin[kWarps], wmax[kWarps], wdiff[kWarps];
    uint32_t wtot[kWarps];
    uint32_t heavy_n, heavy[kMaxHeavy];  // first slot << 16 | elements
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

  // Bin and, below it, 32 bits of fraction of a key: monotone in the key. The
  // distance from base, shifted up until range's highest bit is the 64th, has
  // its upper 32 bits scaled to bins: floor(x * f / 2^32).
  struct Scale {
    uint64_t base;
    uint32_t up, f;
  };
  static __device__ __forceinline__ Scale make_scale(uint64_t base, uint64_t range) {  // range > 0
    Scale s;
    s.base = base;
    s.up = (uint32_t)__clzll((long long)range);
    const uint32_t xr = (uint32_t)((range << s.up) >> 32);
    // kBins 2^32 / (xr + 1), a little less: xr's bin must stay below kBins. In
    // 32-bit floats (relative errors below 2^-21 in all), taken down by 2^-19.
    s.f = (uint32_t)(__fdividef((float)kBins * 4294967296.0f, (float)xr + 1.0f) * (1.0f - 1.0f / 524288.0f));
    return s;
  }
  static __device__ __forceinline__ uint32_t bin_of(const Scale& s, uint64_t key, uint32_t* frac) {
    const uint64_t d = key - s.base;
    const uint32_t hi = s.up < 32u ? (uint32_t)(d >> 32) : (uint32_t)d, lo = s.up < 32u ? (uint32_t)d : 0u;
    const uint64_t p = (uint64_t)__funnelshift_l(lo, hi, s.up) * s.f;  // the shift counts modulo 32
    *frac = (uint32_t)p;
    return (uint32_t)(p >> 32);
  }

  // Sorts the elements in[lo, hi) (shared memory, not changed; hi <= kCap) and
  // calls emit(on, rank, element) for each, from the thread that holds it, and
  // possibly more often with on = false; neighbouring threads get neighbouring
  // ranks but for a bin's few elements. Every key is in [base, base + range];
  // with range = 0 that is not known yet. A tile that turns out to be in order
  // need not be emitted when `in_place`.
  // `slot` and `bins` are the tile's shared arrays; every thread of the CTA
  // calls this together, with in[] visible and bins[] not in use. On return
  // threads may still be reading in[], slot[] and bins[]: a barrier is due
  // before they are written again.
  template <typename Emit>
  static __device__ __forceinline__ void sort(const Elem* in, uint32_t lo, uint32_t hi, uint64_t base, uint64_t range,
                                              uint32_t* slot, uint32_t* bins, Shared& sh, bool in_place, Uneven uneven,
                                              Emit emit) {
    if (range == 0 || !sort_even<false>(in, lo, hi, make_scale(base, range), slot, bins, sh, emit))
      sort_any(in, lo, hi, slot, bins, sh, range == 0, in_place, uneven, emit);
  }

  // Bins over the tile's own range of keys (unless other bins were tried and a
  // few rounds of bits will do), bins that follow the keys; bit by bit when those
  // are uneven too.
  template <typename Emit>
  static __device__ __noinline__ void sort_any(const Elem* in, uint32_t lo, uint32_t hi, uint32_t* slot,
                                               uint32_t* bins, Shared& sh, bool first_try, bool in_place,
                                               Uneven uneven, Emit emit) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint64_t k0 = in[lo].key;
    uint64_t mn = ~0ull, mx = 0ull, diff = 0ull;
    bool inversion = false;
    for (uint32_t p = lo + threadIdx.x; p < hi; p += THREADS) {
      const uint64_t key = in[p].key;
      mn = key < mn ? key : mn;
      mx = key > mx ? key : mx;
      diff |= key ^ k0;
      if (p + 1u < hi) inversion |= key > in[p + 1u].key;
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    diff = (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32)) << 32 |
           __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    __syncthreads();  // sh and the arrays are no longer read
    if (lane == 0) {
      sh.wmin[warp] = mn;
      sh.wmax[warp] = mx;
      sh.wdiff[warp] = diff;
    }
    if (!__syncthreads_or(inversion)) {
      if (!in_place)
        for (uint32_t p = lo + threadIdx.x; p < hi; p += THREADS) emit(true, p - lo, in[p]);
      return;
    }
    mn = warp_min(lane < (uint32_t)kWarps ? sh.wmin[lane] : ~0ull);
    mx = warp_max(lane < (uint32_t)kWarps ? sh.wmax[lane] : 0ull);
    diff = lane < (uint32_t)kWarps ? sh.wdiff[lane] : 0ull;
    diff = (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32)) << 32 |
           __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    uint32_t rounds = 0;
    for (uint64_t d = diff; d; d &= ~(255ull << (__ffsll((long long)d) - 1))) rounds++;
    constexpr bool kSpreads = kCuts * 8u + (kCuts + 1u) * sizeof(Part) <= kSlotBytes;  // cuts and parts in the slots' place
    // bins that follow the keys at once, unless most of them are duplicates, which
    // the sort by even bins has its own ways with, if it can; then they are better than bits
    bool strict = kSpreads && uneven == Uneven::kSpread && !first_try && rounds > kFewRounds;
    if (strict) {  // of keys that occur five times and more in the tile, eight of the CTA's have an equal in their warp
      const uint64_t key = in[lo + threadIdx.x * (hi - lo) / (uint32_t)THREADS].key;
      const uint32_t same = __match_any_sync(0xffffffffu, (unsigned long long)key);
      strict = __syncthreads_count(__ffs((int)same) - 1 != (int)lane) < (int)(THREADS / 64);
    }
    for (bool even = true;; strict = false, even = false) {
      if constexpr (kSpreads)
        if ((strict || !even) && sort_spread(in, lo, hi, mn, mx, strict, slot, bins, sh, emit)) return;
      if (!even) break;
      if ((first_try || rounds > kFewRounds) &&
          sort_even<true>(in, lo, hi, make_scale(mn, mx - mn), slot, bins, sh, emit))
        return;
      if (!kSpreads || uneven == Uneven::kBits || rounds <= kFewRounds) break;
    }
    __syncthreads();
    sort_bits(in + lo, hi - lo, diff, slot, bins, sh, emit);
  }

  // The rank of (v, key) among the slots q[0, cnt): whole keys where key bits agree, then positions.
  static __device__ __forceinline__ uint32_t rank_exact(const Elem* in, const uint32_t* q, uint32_t cnt, uint32_t v,
                                                        uint64_t key) {
    uint32_t r = 0;
    for (uint32_t j = 0; j < cnt; j += 4u) {
      uint32_t u[4];
      uint64_t ku[4];
#pragma unroll
      for (uint32_t x = 0; x < 4u; x++) u[x] = q[min(j + x, cnt - 1u)];
#pragma unroll
      for (uint32_t x = 0; x < 4u; x++) ku[x] = in[u[x] & kPosMask].key;
#pragma unroll
      for (uint32_t x = 0; x < 4u; x++) {
        const bool tie = (u[x] ^ v) <= kPosMask && ku[x] != key;
        r += j + x < cnt && (tie ? ku[x] < key : u[x] < v) ? 1u : 0u;
      }
    }
    return r;
  }

  // The sort by bins that follow the keys: a key per thread, sorted, cut the tile's
  // range into parts of some nine elements each, and every part has the same
  // number of bins, equal cuts of its own range. Signs, clusters, exponents, text and
  // keys with bits that never vary are spread by it like even ones, for a search
  // among the cuts per element; false when a bin has too many elements, all the same
  // (few different keys), or, when `strict`, an eighth of the cuts are equal to another. Ranks are found where an element lies, and an order list
  // brings the elements out in theirs.
  static constexpr uint32_t kCuts = (uint32_t)THREADS, kPartBins = kBins / (kCuts + 1u);
  struct Part {
    uint64_t base;
    uint32_t up, f;
  };
  template <typename Emit>
  static __device__ __noinline__ bool sort_spread(const Elem* in, uint32_t lo, uint32_t hi, uint64_t mn, uint64_t mx,
                                                  bool strict, uint32_t* slot, uint32_t* bins, Shared& sh, Emit emit) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, m = hi - lo;
    uint64_t* cut = reinterpret_cast<uint64_t*>(slot);
    Part* part = reinterpret_cast<Part*>(cut + kCuts);
    uint16_t* start = reinterpret_cast<uint16_t*>(bins);
    __syncthreads();  // the arrays are no longer read
    {
      uint4* z = reinterpret_cast<uint4*>(bins) + tid * 2u;
      z[0] = make_uint4(0, 0, 0, 0);
      z[1] = make_uint4(0, 0, 0, 0);
      if (tid == 0) start[kBins] = (uint16_t)m;
    }
    // the cuts, by bitonic exchanges
    uint64_t v = in[lo + tid * m / kCuts].key;
#pragma unroll
    for (uint32_t k = 2; k <= kCuts; k <<= 1) {
#pragma unroll
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        uint64_t o;
        if (j >= 32u) {
          __syncthreads();
          cut[tid] = v;
          __syncthreads();
          o = cut[tid ^ j];
        } else {
          o = __shfl_xor_sync(0xffffffffu, v, (int)j);
        }
        const bool lower = ((tid & k) == 0u) == ((tid & j) == 0u);
        v = lower == (o < v) ? o : v;
      }
    }
    __syncthreads();
    cut[tid] = v;
    __syncthreads();
    if (__syncthreads_count(tid > 0u && cut[tid - 1u] == v) > (int)(kCuts / 8u) && strict) return false;
    for (uint32_t i = tid; i <= kCuts; i += THREADS) {  // part i: keys from cut i - 1 up to below cut i
      const uint64_t a = i ? cut[i - 1u] : mn, b = i < kCuts ? cut[i] : mx;
      const uint64_t range = b > a ? b - a : 1ull;
      const uint32_t up = (uint32_t)__clzll((long long)range);
      const uint32_t xr = (uint32_t)((range << up) >> 32);
      part[i] = Part{a, up, (uint32_t)(__fdividef((float)kPartBins * 4294967296.0f, (float)xr + 1.0f) * (1.0f - 1.0f / 524288.0f))};
    }
    __syncthreads();
    uint32_t place[K], frac[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      const bool on = p - lo < m;
      const uint64_t key = in[on ? p : lo].key;
      uint32_t i = 0;  // cuts not above the key
#pragma unroll
      for (uint32_t s = kCuts / 2u; s > 0; s >>= 1) i += cut[i + s - 1u] <= key ? s : 0u;
      i += cut[i] <= key ? 1u : 0u;
      const Part c = part[i];
      const uint64_t x = (uint64_t)(uint32_t)(((key - c.base) << c.up) >> 32) * c.f;
      frac[k] = (uint32_t)x;
      const uint32_t b = i * kPartBins + (uint32_t)(x >> 32);
      const uint32_t s16 = (b & 1u) << 4;
      const uint32_t old = atom_add_if(on, bins + (b >> 1), 1u << s16);
      place[k] = b << 16 | ((old >> s16) & 0xffffu);
    }
    __syncthreads();
    {
      uint32_t w8[8], maxc = 0, sum = 0;
      uint4* q = reinterpret_cast<uint4*>(bins) + tid * 2u;
      {
        const uint4 a = q[0], b = q[1];
        w8[0] = a.x, w8[1] = a.y, w8[2] = a.z, w8[3] = a.w;
        w8[4] = b.x, w8[5] = b.y, w8[6] = b.z, w8[7] = b.w;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        maxc = __vmaxu2(maxc, w8[i]);
        const uint32_t c0 = w8[i] & 0xffffu, c1 = w8[i] >> 16;
        w8[i] = sum | (sum + c0) << 16;
        sum += c0 + c1;
      }
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      if (lane == 31) sh.wtot[warp] = inc;
      maxc = max(maxc & 0xffffu, maxc >> 16);
      if (__syncthreads_or(maxc > kSlotsBin)) return false;
      uint32_t off = inc - sum;
      const uint32_t wt = lane < (uint32_t)kWarps ? sh.wtot[lane] : 0u;
      off += __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
      const uint32_t both = off | off << 16;
      q[0] = make_uint4(w8[0] + both, w8[1] + both, w8[2] + both, w8[3] + both);
      q[1] = make_uint4(w8[4] + both, w8[5] + both, w8[6] + both, w8[7] + both);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      st_shared_if(p - lo < m, slot + start[place[k] >> 16] + (place[k] & 0xffffu), (frac[k] & ~kPosMask) | p);
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p - lo < m) {
        const uint32_t b = place[k] >> 16, s = start[b];
        place[k] = s + rank_exact(in, slot + s, start[b + 1u] - s, (frac[k] & ~kPosMask) | p, in[p].key);
      }
    }
    __syncthreads();
    uint16_t* order = reinterpret_cast<uint16_t*>(slot);
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      if (p - lo < m) order[place[k]] = (uint16_t)p;
    }
    __syncthreads();
    for (uint32_t i = tid; i < m; i += THREADS) emit(true, i, in[order[i]]);
    return true;
  }

  // The sort by bins; false when a bin has too many elements (HEAVY: too many
  // different keys; then some may have been emitted).
  template <bool HEAVY, typename Emit>
  static __device__ __forceinline__ bool sort_even(const Elem* in, uint32_t lo, uint32_t hi, const Scale sc,
                                                   uint32_t* slot, uint32_t* bins, Shared& sh, Emit emit) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t m = hi - lo;
    uint16_t* start = reinterpret_cast<uint16_t*>(bins);
    // keys within 2^31 of each other: next keys are at least 2 f >= 2 (kBins - 1)
    // >= 2^kPosBits apart on the scale, so slots that agree in the key bits hold one key
    static_assert(2u * (kBins - 1u) >= (1u << kPosBits), "exact slots");
    const bool whole = sc.up >= 33u;
    {
      uint4* z = reinterpret_cast<uint4*>(bins) + tid * 2u;
      z[0] = make_uint4(0, 0, 0, 0);
      z[1] = make_uint4(0, 0, 0, 0);
      if (tid == 0) start[kBins] = (uint16_t)m, sh.heavy_n = 0u;
    }
    __syncthreads();
    // 1. bin, place among the bin's elements and fraction of each element
    uint32_t place[K], frac[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      const bool on = p - lo < m;
      const uint32_t b = bin_of(sc, in[on ? p : lo].key, &frac[k]);
      const uint32_t s16 = (b & 1u) << 4;
      const uint32_t old = atom_add_if(on, bins + (b >> 1), 1u << s16);
      place[k] = b << 16 | ((old >> s16) & 0xffffu);
    }
    __syncthreads();
    // 2. exclusive scan of the counts; thread t owns bins [16 t, 16 t + 16)
    bool over;
    {
      uint32_t w8[8], maxc = 0, sum = 0;
      uint4* q = reinterpret_cast<uint4*>(bins) + tid * 2u;
      {
        const uint4 a = q[0], b = q[1];
        w8[0] = a.x, w8[1] = a.y, w8[2] = a.z, w8[3] = a.w;
        w8[4] = b.x, w8[5] = b.y, w8[6] = b.z, w8[7] = b.w;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        maxc = __vmaxu2(maxc, w8[i]);
        const uint32_t c0 = w8[i] & 0xffffu, c1 = w8[i] >> 16;
        w8[i] = sum | (sum + c0) << 16;
        sum += c0 + c1;
      }
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      if (lane == 31) sh.wtot[warp] = inc;
      maxc = max(maxc & 0xffffu, maxc >> 16);
      over = __syncthreads_or(maxc > kMaxBin) != 0;
      if (over && !HEAVY) return false;
      uint32_t off = inc - sum;
      const uint32_t wt = lane < (uint32_t)kWarps ? sh.wtot[lane] : 0u;
      off += __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
      const uint32_t both = off | off << 16;
      q[0] = make_uint4(w8[0] + both, w8[1] + both, w8[2] + both, w8[3] + both);
      q[1] = make_uint4(w8[4] + both, w8[5] + both, w8[6] + both, w8[7] + both);
      if (HEAVY && maxc > kSlotsBin) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const uint32_t s0 = (w8[i >> 1] >> (16 * (i & 1))) & 0xffffu;
          const uint32_t s1 = i < 15 ? (w8[(i + 1) >> 1] >> (16 * ((i + 1) & 1))) & 0xffffu : sum;
          if (s1 - s0 > kSlotsBin) sh.heavy[atomicAdd(&sh.heavy_n, 1u)] = (off + s0) << 16 | (s1 - s0);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t p = tid + (uint32_t)k * THREADS;
      const uint32_t q = start[place[k] >> 16] + (place[k] & 0xffffu);
      st_shared_if(p - lo < m, slot + q, (frac[k] & ~kPosMask) | p);
    }
    __syncthreads();
    if (HEAVY) {  // a large bin of many keys: nothing here helps
      const uint32_t count = sh.heavy_n;
      bool lost = false;
      for (uint32_t h = warp; h < count; h += kWarps) {
        const uint32_t c = sh.heavy[h] & 0xffffu;
        lost |= probe_keys(in, slot, sh.heavy[h] >> 16, c) > kFewKeys;
      }
      if (__syncthreads_or(lost)) return false;
    }
    // 3. rank inside the bin, elements out: three rows of the tile at a time,
    // their loads in flight together; the first four slots of the bin without
    // a branch (slots past the tile's last are read but not counted)
    constexpr int R = K % 3 == 0 ? 3 : K % 2 == 0 ? 2 : 1;
    auto exact = [&](const uint32_t* q, uint32_t cnt, uint32_t v, uint64_t key) { return rank_exact(in, q, cnt, v, key); };
    bool lost = false;
    auto load_rows = [&](uint32_t row, uint32_t (&v)[R], Elem (&e)[R]) {
#pragma unroll
      for (int i = 0; i < R; i++) v[i] = slot[min(row + (uint32_t)i * THREADS, m - 1u)];
#pragma unroll
      for (int i = 0; i < R; i++) e[i] = in[v[i] & kPosMask];
    };
    auto rank_rows = [&](const bool by_slots, const uint32_t (&v)[R], const Elem (&e)[R], uint32_t* r) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        uint32_t f;
        const uint32_t b = bin_of(sc, e[i].key, &f);
        const uint32_t s = start[b], cnt = start[b + 1u] - s;
        const uint32_t* q = slot + s;
        bool close = cnt > 4u;
        r[i] = s;
#pragma unroll
        for (uint32_t j = 0; j < 4u; j++) {
          const uint32_t u = q[j];
          if (j < cnt) {
            r[i] += u < v[i] ? 1u : 0u;
            close |= ((u ^ v[i]) - 1u) < kPosMask;
          }
        }
        if (HEAVY && by_slots && cnt > kSlotsBin) {
          r[i] = kCap;  // heavy_bins emits it
        } else if (HEAVY && by_slots && cnt > 4u) {
          // slots alone: right when all that agree in the key bits hold the same
          // key, and so when each holds the key of the lowest of them
          uint32_t low = v[i];
          for (uint32_t j = 4u; j < cnt; j += 4u) {
            uint32_t u[4];
#pragma unroll
            for (uint32_t x = 0; x < 4u; x++) u[x] = q[min(j + x, cnt - 1u)];
#pragma unroll
            for (uint32_t x = 0; x < 4u; x++) r[i] += j + x < cnt && u[x] < v[i] ? 1u : 0u;
#pragma unroll
            for (uint32_t x = 0; x < 4u; x++) low = min(low, u[x] >= (v[i] & ~kPosMask) ? u[x] : low);
          }
#pragma unroll
          for (uint32_t x = 0; x < 4u; x++) low = min(low, q[x] >= (v[i] & ~kPosMask) ? q[x] : low);
          lost |= !whole && in[low & kPosMask].key != e[i].key;
        } else if (close && (cnt > 4u || !whole)) {  // more slots, or key bits that agree
          r[i] = s + exact(q, cnt, v[i], e[i].key);
        }
      }
    };
    uint32_t v[R], r[K];
    Elem e[R];
    if (!HEAVY || !over) {
#pragma unroll 1
      for (uint32_t row = tid; row - tid < m; row += R * THREADS) {
        load_rows(row, v, e);
        rank_rows(false, v, e, r);
#pragma unroll
        for (int i = 0; i < R; i++) emit(row + (uint32_t)i * THREADS < m, r[i], e[i]);
      }
      return true;
    }
    // All ranks before the first element goes out, since some may be wrong: then
    // bins of five and more are ranked again, by whole keys.
#pragma unroll
    for (int k = 0; k < K; k += R) {
      load_rows(tid + (uint32_t)k * THREADS, v, e);
      rank_rows(HEAVY, v, e, r + k);
    }
    lost = __syncthreads_or(lost);
#pragma unroll
    for (int k = 0; k < K; k += R) {
      load_rows(tid + (uint32_t)k * THREADS, v, e);
#pragma unroll
      for (int i = 0; i < R; i++) {
        if (lost && r[k + i] < kCap) {
          uint32_t f;
          const uint32_t b = bin_of(sc, e[i].key, &f);
          const uint32_t s = start[b], cnt = start[b + 1u] - s;
          if (cnt > 4u) r[k + i] = s + exact(slot + s, cnt, v[i], e[i].key);
        }
        emit(tid + (uint32_t)(k + i) * THREADS < m && r[k + i] < kCap, r[k + i], e[i]);
      }
    }
    return sh.heavy_n == 0u || heavy_bins(in, slot, bins, sh, emit);
  }

  // The heavy bins' elements, one warp per bin and the whole CTA for the largest:
  // for each key of the bin from the smallest, a bitmap of its elements'
  // positions in the tile, whose prefix counts are the ranks. A bin of many
  // different keys is left (false).
  static constexpr uint32_t kWords = (kCap + 31u) / 32u, kPerLane = (kWords + 31u) / 32u;
  static constexpr uint32_t kMapWords = kWords + kWords / 2u + 1u;  // the bitmap and 16-bit prefix counts
  static constexpr uint32_t kFit = (uint32_t)(kBinBytes / 4u) / kMapWords;
  static constexpr uint32_t kTakers = kFit < (uint32_t)kWarps ? kFit : (uint32_t)kWarps;
  // Elements from which the whole CTA takes a bin: 9000 Zipf keys 32.8 us, with 2048 45.1;
  // batches of half zeros 90 and 107. Keys that occur a thousand times each are 5 to 17 %
  // faster with 2048 (9000: 37.0 -> 30.8); with 256 all is within 4 %.
  static constexpr uint32_t kLargeBin = 512;

  // One warp: before[w] = bits in the words below w of the bitmap; all bits in it.
  static __device__ __forceinline__ uint32_t count_map(const uint32_t* map, uint16_t* before) {
    const uint32_t lane = lane_id();
    uint32_t sum = 0, part[kPerLane];
#pragma unroll
    for (uint32_t i = 0; i < kPerLane; i++) {
      part[i] = sum;
      const uint32_t x = lane * kPerLane + i;
      sum += x < kWords ? (uint32_t)__popc(map[x]) : 0u;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
#pragma unroll
    for (uint32_t i = 0; i < kPerLane; i++)
      if (lane * kPerLane + i < kWords) before[lane * kPerLane + i] = (uint16_t)(inc - sum + part[i]);
    return __shfl_sync(0xffffffffu, inc, 31);
  }
  static __device__ __forceinline__ uint32_t map_rank(const uint32_t* map, const uint16_t* before, uint32_t p) {
    return before[p >> 5] + (uint32_t)__popc(map[p >> 5] & ((1u << (p & 31u)) - 1u));
  }
  // One warp: different keys among 32 of the bin's.
  static __device__ __forceinline__ uint32_t probe_keys(const Elem* in, const uint32_t* slot, uint32_t s, uint32_t c) {
    const uint64_t key = in[slot[s + lane_id() * c / 32u] & kPosMask].key;
    const uint32_t same = __match_any_sync(0xffffffffu, (unsigned long long)key);
    return (uint32_t)__popc(__ballot_sync(0xffffffffu, __ffs((int)same) - 1 == (int)lane_id()));
  }

  template <typename Emit>
  static __device__ __noinline__ bool heavy_bins(const Elem* in, const uint32_t* slot, uint32_t* bins, Shared& sh,
                                                 Emit emit) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    bool ok = true;
    __syncthreads();  // the bins' starts are no longer read
    const uint32_t count = sh.heavy_n;
    for (uint32_t h = 0; h < count; h++) {
      const uint32_t s = sh.heavy[h] >> 16, c = sh.heavy[h] & 0xffffu;
      if (c < kLargeBin) continue;
      if (probe_keys(in, slot, s, c) > kFewKeys) {  // the same answer in every warp
        ok = false;
        continue;
      }
      uint32_t* map = bins;
      uint16_t* before = reinterpret_cast<uint16_t*>(map + kWords);
      uint32_t done = 0;
      uint64_t last = 0;
      for (uint32_t it = 0; it < 2u * kFewKeys && done < c; it++) {
        uint64_t mn = ~0ull;
        for (uint32_t j = tid; j < c; j += THREADS) {
          const uint64_t key = in[slot[s + j] & kPosMask].key;
          if ((done == 0 || key > last) && key < mn) mn = key;
        }
        mn = warp_min(mn);
        if (lane == 0) sh.wmin[warp] = mn;
        for (uint32_t i = tid; i < kWords; i += THREADS) map[i] = 0u;
        __syncthreads();
        mn = warp_min(lane < (uint32_t)kWarps ? sh.wmin[lane] : ~0ull);
        for (uint32_t j = tid; j < c; j += THREADS) {
          const uint32_t p = slot[s + j] & kPosMask;
          if (in[p].key == mn) atomicOr(&map[p >> 5], 1u << (p & 31u));
        }
        __syncthreads();
        if (warp == 0) {
          const uint32_t all = count_map(map, before);
          if (lane == 0) sh.wtot[0] = all;
        }
        __syncthreads();
        for (uint32_t j = tid; j < c; j += THREADS) {
          const uint32_t p = slot[s + j] & kPosMask;
          const Elem e = in[p];
          if (e.key == mn) emit(true, s + done + map_rank(map, before, p), e);
        }
        done += sh.wtot[0];
        last = mn;
        __syncthreads();
      }
      ok = ok && done >= c;
    }
    uint32_t* map = bins + warp * kMapWords;
    uint16_t* before = reinterpret_cast<uint16_t*>(map + kWords);
    for (uint32_t h = warp; warp < kTakers && h < count; h += kTakers) {
      const uint32_t s = sh.heavy[h] >> 16, c = sh.heavy[h] & 0xffffu;
      if (c >= kLargeBin) continue;
      uint32_t done = 0;
      if (probe_keys(in, slot, s, c) <= kFewKeys) {
        uint64_t last = 0;
        for (uint32_t it = 0; it < 2u * kFewKeys && done < c; it++) {
          uint64_t mn = ~0ull;
          for (uint32_t j = lane; j < c; j += 32u) {
            const uint64_t key = in[slot[s + j] & kPosMask].key;
            if ((done == 0 || key > last) && key < mn) mn = key;
          }
          mn = warp_min(mn);
          for (uint32_t i = lane; i < kWords; i += 32u) map[i] = 0u;
          __syncwarp();
          for (uint32_t j = lane; j < c; j += 32u) {
            const uint32_t p = slot[s + j] & kPosMask;
            if (in[p].key == mn) atomicOr(&map[p >> 5], 1u << (p & 31u));
          }
          __syncwarp();
          const uint32_t all = count_map(map, before);
          __syncwarp();
          for (uint32_t j = lane; j < c; j += 32u) {
            const uint32_t p = slot[s + j] & kPosMask;
            const Elem e = in[p];
            if (e.key == mn) emit(true, s + done + map_rank(map, before, p), e);
          }
          done += all;
          last = mn;
          __syncwarp();
        }
      }
      ok = ok && done >= c;
    }
    return !__syncthreads_or(!ok);
  }

  // Outputs [d, d + cnt) of the stable merge of the sorted position lists a
  // (la of them, the earlier run) and b into dst, by one thread.
  static __device__ __forceinline__ void merge_span(const Elem* in, const uint16_t* a, uint32_t la, const uint16_t* b,
                                                    uint32_t lb, uint32_t d, uint32_t cnt, uint16_t* dst) {
    uint32_t lo = d > lb ? d - lb : 0u, hi = min(d, la);
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (in[a[mid]].key <= in[b[d - 1u - mid]].key) lo = mid + 1u;
      else hi = mid;
    }
    uint32_t i = lo, j = d - lo;
    uint32_t pa = i < la ? a[i] : 0u, pb = j < lb ? b[j] : 0u;
    uint64_t ka = in[pa].key, kb = in[pb].key;
    for (uint32_t q = 0; q < cnt; q++) {
      if (j >= lb || (i < la && ka <= kb)) {
        dst[q] = (uint16_t)pa;
        if (++i < la) ka = in[pa = a[i]].key;
      } else {
        dst[q] = (uint16_t)pb;
        if (++j < lb) kb = in[pb = b[j]].key;
      }
    }
  }

  // The merge of in[0..la) and in[la..la + lb), as positions in dst; id[i] = i.
  static __device__ __forceinline__ void merge_parts(const Elem* in, const uint16_t* id, uint16_t* dst, uint32_t la,
                                                     uint32_t lb) {
    const uint32_t d0 = threadIdx.x * (uint32_t)K;
    if (d0 < la + lb) merge_span(in, id, la, id + la, lb, d0, min((uint32_t)K, la + lb - d0), dst + d0);
  }

  // Stable order of in[0, m) by the bits of `diff` (those in which keys differ).
  template <typename Emit>
  static __device__ __noinline__ void sort_bits(const Elem* in, uint32_t m, uint64_t diff, uint32_t* slot,
                                                uint32_t* bins, Shared& sh, Emit emit) {
    constexpr uint32_t WP = kWarps + 1;  // padded row of a digit's per-warp counters
    constexpr uint32_t kParts = kWarps / 8;
    static_assert(kWarps % 8 == 0 && 256u * WP * 2u <= kBinBytes, "eight counters per thread in the scan");
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, lt = lanemask_lt();
    uint16_t* cur = reinterpret_cast<uint16_t*>(slot);
    uint16_t* nxt = cur + kCap;
    uint16_t* cnt = reinterpret_cast<uint16_t*>(bins);
    const uint32_t i0 = warp * 32u * K + lane;  // this thread's places: i0 + 32 k
    for (bool first = true; diff; first = false) {
      const int s = __ffsll((long long)diff) - 1;
      diff &= ~(255ull << s);
      for (uint32_t i = tid; i < 256u * WP / 2u; i += THREADS) bins[i] = 0u;
      __syncthreads();
      uint32_t pd[K], r[K];  // position | digit << 16, rank among the warp's equal digits
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t i = i0 + 32u * (uint32_t)k;
        const uint32_t p = i < m ? (first ? i : (uint32_t)cur[i]) : 0u;
        pd[k] = p | ((uint32_t)(in[p].key >> s) & 255u) << 16;
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        const bool valid = i0 + 32u * (uint32_t)k < m;
        const uint32_t d = pd[k] >> 16;
        const uint32_t peers = warp_peers(d, 8, valid);
        uint16_t* c = &cnt[d * WP + warp];
        const uint32_t before = *c;
        r[k] = before + __popc(peers & lt);
        __syncwarp();
        if (valid) *c = (uint16_t)(before + __popc(peers));
        __syncwarp();
      }
      __syncthreads();
      {
        uint16_t* c = &cnt[tid / kParts * WP + tid % kParts * 8u];
        uint32_t v[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          v[j] = sum;
          sum += c[j];
        }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= (uint32_t)o) inc += y;
        }
        if (lane == 31) sh.wtot[warp] = inc;
        __syncthreads();
        const uint32_t wt = lane < (uint32_t)kWarps ? sh.wtot[lane] : 0u;
        const uint32_t off = inc - sum + __reduce_add_sync(0xffffffffu, lane < warp ? wt : 0u);
#pragma unroll
        for (int j = 0; j < 8; j++) c[j] = (uint16_t)(off + v[j]);
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < K; k++)
        if (i0 + 32u * (uint32_t)k < m) nxt[cnt[(pd[k] >> 16) * WP + warp] + r[k]] = (uint16_t)pd[k];
      __syncthreads();
      uint16_t* t = cur;
      cur = nxt;
      nxt = t;
    }
    for (uint32_t p = tid; p < m; p += THREADS) emit(true, p, in[cur[p]]);
  }
};

}  // namespace lsb
