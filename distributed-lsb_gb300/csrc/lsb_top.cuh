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

// Warp t scans the counts of digit t, of T: exclusive starts, and bit t of *constant
// where one value holds all n keys.
__device__ __forceinline__ void scan_digits(const uint32_t* hist, uint32_t* gstart, uint32_t n, uint32_t T, uint32_t* constant) {
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  if (warp >= T) return;
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
  if (__any_sync(0xffffffffu, one) && lane == 0) atomicOr(constant, 1u << warp);
}
// Which of T passes run, from where and to where (one thread).
__device__ __forceinline__ void chain_passes(TopPlan& q, uint32_t T, uint32_t constant) {
  uint32_t par = 0, pars = 0, run = 0;
  for (uint32_t t = 0; t < T; t++) {
    pars |= par << t;
    if (!((constant >> t) & 1u)) {
      run |= 1u << t;
      par ^= 1u;
    }
  }
  q.run_mask = run;
  q.par_mask = pars;
  q.src_parity = par;
}

// ---------------------------------------------------------------------------
// the sample

constexpr int kSampleThreads = 1024;
// S keys per thread: 1024 S sample keys. One per thread is sorted by exchanges
// between threads, whatever the keys are, more by TileSort.
template <int S>
using SampleTile = TileSort<kSampleThreads, S>;
template <int S>
constexpr size_t kSampleSmem = S == 1 ? 2u * kSampleThreads * 8u : SampleTile<S>::kSmem + (size_t)SampleTile<S>::kCap * 8u;

// What the sample's statistics are held against (from n and the tile alone).
// Times are in tenths of a pass.
struct SampleRule {
  uint32_t tmin;        // fewest passes that shorten even runs to a tile
  uint32_t heavy;       // a key this often in the sample is heavy
  uint32_t tall;        // passes that leave a heavy key alone in its run
  uint32_t far;         // this many sample keys apart in one window: a run longer than a tile
  uint32_t near_limit;  // neighbours that may share a window before the mean run is too long
  uint32_t dups;        // equal neighbours from which most keys occur eight times or more
  uint32_t far_limit;   // keys in runs longer than a tile that are put up with
  uint32_t big_passes;  // passes that leave runs for the big tile, one less than tmin; 0: it is not to be had
  uint32_t big_near;    // near_limit and far for it
  uint32_t big_far;
  uint32_t finish;      // time of the last step
  uint32_t uneven;      // more of it where keys are too unevenly spread
  uint32_t straddle;    // and where only the tiles between clusters of keys are
  uint32_t copy;        // of the copy after an odd number of passes that leave nothing to sort
  uint32_t tile;        // elements of a tile
  float per_near;       // mean run length for each two neighbours that share a window
  bool skips;           // passes over digits that are the same in all keys are left out
};
// mean_run: the mean run length up to which a pass is saved, for a tile of `tile`. Keys that occur
// more than `often` times are heavy, and the passes then have `spread` windows
// or more per element. sample: keys in the sample.
__host__ __device__ inline uint32_t passes_for(float n, float per_run) {
  uint32_t t = 1;
  for (float most = per_run * 256.0f; t < 8u && n > most; most *= 256.0f) t++;
  return t;
}
// A tile between two clusters takes some 40 us more, and the last step with it; a
// pass over n elements (8 + n / 135000) us.
__host__ __device__ inline uint32_t straddle_time(uint32_t n) { return (uint32_t)(400.0f / (8.0f + (float)n / 135000.0f)); }
__host__ __device__ inline SampleRule sample_rule(uint32_t n, uint32_t sample, uint32_t tile, uint32_t mean_run,
                                                  uint32_t often, float spread) {
  SampleRule r;
  const float per = (float)sample / (float)n;
  r.tmin = passes_for((float)n, (float)mean_run);
  r.big_passes = r.big_near = r.big_far = 0u;
  // the last step over a pass, 2^24 to 2^30 elements: 1.0 to 1.16; of uneven tiles,
  // sort_spread or bits: 2^24 pairs of 20 bits in 52, 504 us and a pass 127; 2^24
  // elements in a batch, nibbles, 2160 and 380
  r.finish = 12u;
  // (with 20 text in arrays of 2^25 takes 5.1 ms, not 4.6, and 5 10^6 keys of it 317 us, not 398;
  // with 90 batches of tagged 20-bit keys take 1.3 to 1.7 times as long)
  r.uneven = 45u;
  r.straddle = straddle_time(n);
  r.copy = 6u;
  r.tile = tile;
  r.per_near = 2.0f / per / (float)sample;
  r.skips = true;
  r.tall = passes_for((float)n, 1.0f / spread);
  const float lam = (float)mean_run * per, lom = (float)often * per, share = (float)tile * per;
  // S keys in S / lam windows of even runs: so many occupied, and three standard deviations
  const float none = expf(-lam), windows = (float)sample / lam;
  r.near_limit = (uint32_t)((float)sample - windows * (1.0f - none) + 3.0f * sqrtf(windows * none * (1.0f - (1.0f + lam) * none))) + 1u;
  // a run of a tile: its share of the sample, with room for chance where even runs
  // come near it (runs of one pass have four sample keys of 1024 on average)
  r.far = (uint32_t)(share < 8.0f ? share + 2.5f * sqrtf(share) + 2.0f : share < 64.0f ? share + sqrtf(share) : 0.95f * share);
  if (r.far < 4u) r.far = 4u;
  r.far_limit = sample / 100u;
  r.heavy = (uint32_t)(lom + 4.0f * sqrtf(lom) + 4.0f);
  // sampled twice by chance: sample^2 / (2 n) pairs; every key k times in the array: k times that
  const float pairs = 4.0f * (float)sample * per;
  r.dups = pairs > 3.0f ? (uint32_t)pairs : 3u;
  return r;
}

// The 32-bit finaliser of MurmurHash3.
__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  return x ^ x >> 16;
}

// Sorts one key of each of the 1024 threads by bitonic exchanges, within a warp by
// shuffles. buf: 2 * 1024 keys of shared memory, not in use; returns the half of it
// with the sorted keys, and no barrier is due before they are read.
__device__ __forceinline__ uint64_t* sort_sample(uint64_t v, uint64_t* buf) {
  const uint32_t i = threadIdx.x;
  uint32_t half = 0;
#pragma unroll
  for (uint32_t k = 2; k <= (uint32_t)kSampleThreads; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      uint64_t o;
      if (j >= 32u) {  // two halves in turn: one barrier per exchange
        buf[half + i] = v;
        __syncthreads();
        o = buf[half + (i ^ j)];
        half ^= (uint32_t)kSampleThreads;
      } else {
        o = __shfl_xor_sync(0xffffffffu, v, (int)j);
      }
      const bool lower = ((i & k) == 0u) == ((i & j) == 0u);  // this thread keeps the smaller key
      v = lower == (o < v) ? o : v;
    }
  }
  buf[half + i] = v;
  __syncthreads();
  return buf + half;
}

// The sample's key i. The places are drawn independently of each other, not one per
// stretch: of an array nearly in order that would be the most even sample there is.
__device__ __forceinline__ uint64_t sample_key(const Elem* data, uint32_t n, uint32_t i) {
  return ld_relaxed_u64(&data[((uint64_t)mix32(i + 1u) * n) >> 32].key);
}

// A sorted sample of the keys of data[0, n), in shared memory (smem, kSampleSmem<S>
// bytes; all kSampleThreads threads call, with smem not in use).
template <int S>
__device__ __forceinline__ const uint64_t* sample_keys(const Elem* data, uint32_t n, unsigned char* smem,
                                                       typename SampleTile<S>::Shared& sh) {
  using Sample = SampleTile<S>;
  uint64_t key[S];
#pragma unroll
  for (int k = 0; k < S; k++) key[k] = sample_key(data, n, threadIdx.x + (uint32_t)k * kSampleThreads);
  if constexpr (S == 1) {
    return sort_sample(key[0], reinterpret_cast<uint64_t*>(smem));
  } else {
    Elem* in = reinterpret_cast<Elem*>(smem);
    uint32_t* slot = reinterpret_cast<uint32_t*>(smem + Sample::kElemBytes);
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + Sample::kElemBytes + Sample::kSlotBytes);
    uint64_t* s = reinterpret_cast<uint64_t*>(smem + Sample::kSmem);
#pragma unroll
    for (int k = 0; k < S; k++) in[threadIdx.x + (uint32_t)k * kSampleThreads] = Elem{key[k], 0};
    __syncthreads();
    Sample::sort(in, 0, Sample::kCap, 0, 0, slot, bins, sh, false, Uneven::kBits, [&](bool on, uint32_t r, const Elem& e) {
      if (on) s[r] = e.key;
    });
    __syncthreads();
    return s;
  }
}

// The bits [pos - bits, pos), those of them that there are.
__device__ __forceinline__ uint64_t bits_below(uint32_t pos, uint32_t bits) {
  const uint64_t upto = pos >= 64u ? ~0ull : (1ull << pos) - 1ull;
  return pos > bits ? upto & ~((1ull << (pos - bits)) - 1ull) : upto;
}
// Runs of keys that agree down to bit `pos` are sorted in bins that cut the keys'
// range equally: `below` bits under pos in a run, and, with several runs in a tile,
// `above` bits that vary from there up. Do bits that never vary lie among those
// (under bits that do)? Two of them put four times as many elements in a bin.
__device__ __forceinline__ bool ragged(uint32_t pos, uint32_t below, uint32_t above, uint64_t varies) {
  const uint64_t lowest = varies & (~varies + 1ull);
  const uint32_t in_run = (uint32_t)__popcll(bits_below(pos, below) & ~varies & ~(lowest - 1ull));
  const uint64_t up = pos < 64u ? varies >> pos : 0ull;
  uint64_t rest = up;
  for (uint32_t i = 0; i < above; i++) rest &= rest - 1ull;
  const uint64_t taken = up & ~rest;
  const uint32_t between = taken ? 64u - (uint32_t)__clzll((long long)taken) - (uint32_t)__popcll(taken) : 0u;
  return in_run + between >= 2u;
}

// How to sort: by the `passes` highest bytes below bit hb1 and, if that does not
// cover the key, in runs on chip; or, when `plain`, by every byte of the key.
struct SampleChoice {
  uint32_t passes;
  bool plain;
  bool skewed;  // a key is heavy, and tiles of runs are mostly in order
  bool dups;    // most keys, or a heavy one, occur often
  bool big;     // the runs are for the big tile
};

// Counts over the sorted sample; zeroed by its owner before the sample is sorted.
struct SampleStats {
  uint32_t near[8], far[8];  // keys that share T windows with the next one, with the one rule.far - 1 places on
  uint32_t big_far;          // keys that share rule.big_passes windows with the one rule.big_far - 1 places on
  uint32_t equal, diff[2];   // equal neighbours, bits in which keys differ
  SampleChoice choice;
};
__device__ __forceinline__ void clear_stats(SampleStats& st) {
  if (threadIdx.x < sizeof(SampleStats) / 4u) reinterpret_cast<uint32_t*>(&st)[threadIdx.x] = 0u;
}

// The choice that the sorted sample s (keys below bit hb1 differ) lets expect to be
// the fastest, the same answer in every thread. The passes must leave runs of at most
// a tile, whose keys are spread evenly enough for the last step's bins: where they
// are not (bits below the windows that never vary, or that the windows already
// tell: tags, sentinels, signs, text, exponents) that step takes several times as
// long, and more windows are passed over, up to all of them. plain_passes: passes of
// a sort by every byte, 0: those in which the sample differs. low_bit(t): the lowest
// bit of the key in t windows; key_bits: those that vary (0: the sample's). BIG: there
// is a kernel for the big tile.
template <int S, bool BIG = false, class LowBit>
__device__ __forceinline__ SampleChoice choose_passes(const uint64_t* s, uint32_t hb1, const SampleRule& rule,
                                                      uint32_t plain_passes, SampleStats& st, uint64_t key_bits, LowBit low_bit) {
  // nibble T-1 of near / far: this thread's keys that share T windows (but
  // not all 64 bits) with the next key / with the key `far` places on
  constexpr uint32_t kSample = (uint32_t)(S * kSampleThreads);
  uint32_t near = 0, farm = 0, equal = 0, big_far = 0;
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
    if (BIG && rule.big_passes && i + rule.big_far - 1u < kSample && s[i + rule.big_far - 1u] != ki)
      big_far += shared_windows(i + rule.big_far - 1u) >> (4u * (rule.big_passes - 1u)) & 1u;
    heavy |= i + rule.heavy - 1u < kSample && s[i + rule.heavy - 1u] == ki;
  }
  {
    const uint32_t n0 = __reduce_add_sync(0xffffffffu, near & 0x0F0F0F0Fu);
    const uint32_t n1 = __reduce_add_sync(0xffffffffu, (near >> 4) & 0x0F0F0F0Fu);
    const uint32_t f0 = __reduce_add_sync(0xffffffffu, farm & 0x0F0F0F0Fu);
    const uint32_t f1 = __reduce_add_sync(0xffffffffu, (farm >> 4) & 0x0F0F0F0Fu);
    const uint32_t d0 = __reduce_or_sync(0xffffffffu, (uint32_t)diff), d1 = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    equal = __reduce_add_sync(0xffffffffu, equal);
    if (BIG) big_far = __reduce_add_sync(0xffffffffu, big_far);
    const uint32_t l = lane_id();
    if (l < 8) {
      atomicAdd(&st.near[l], ((l & 1u ? n1 : n0) >> (8u * (l >> 1))) & 0xFFu);
      atomicAdd(&st.far[l], ((l & 1u ? f1 : f0) >> (8u * (l >> 1))) & 0xFFu);
    }
    if (l == 0) {
      if (equal) atomicAdd(&st.equal, equal);
      if (BIG && big_far) atomicAdd(&st.big_far, big_far);
      atomicOr(&st.diff[0], d0);
      atomicOr(&st.diff[1], d1);
    }
  }
  heavy = __syncthreads_or(heavy);
  if (threadIdx.x < 32u) {  // lane t weighs t passes, and windows and bytes are looked at by a lane each
    const uint64_t varies = (uint64_t)st.diff[1] << 32 | st.diff[0], key = key_bits ? key_bits : varies;
    const uint32_t full = (hb1 + 7u) / 8u, t = lane_id();
    const bool many_dups = st.equal >= rule.dups, counts = t >= 1u && t <= full;
    const uint32_t near_t = counts ? st.near[t - 1u] : 0u, near_more = t >= 1u && t < 8u ? st.near[t] : 0u;  // share t windows, and one more
    const bool at_all = counts && t >= min(rule.tmin, full);
    auto enough = [&](uint32_t near_limit) {
      return near_t <= near_limit && st.far[t - 1u] <= rule.far_limit && (!heavy || t >= rule.tall);
    };
    bool even = true;
    if (counts && t < full) {
      // x sample keys in a run: where keys are even, x / 512 of the neighbours share a window more
      const float f = (float)near_t / (float)kSample;
      const float x = fminf(f < 0.5f ? 2.6f * f : 64.0f, 2.0f / rule.per_near * (float)rule.tile / (float)kSample);
      even = near_more < 3u || (float)near_more <= 8.0f / 512.0f * x * (float)kSample;
      // the mean run's length is this at most (one neighbour more than were seen), and half of it
      // at least, if some were
      const float most = fminf(rule.per_near * (float)(near_t + 1u), (float)rule.tile);
      const uint32_t below = (uint32_t)__log2f(2.0f * most) + 1u, above = near_t >= 3u ? (uint32_t)__log2f(2.0f * (float)rule.tile / most) : 16u;
      // (four keys that agree in a window more are no crowd wherever they fall)
      even = even && (rule.per_near * (float)(near_more + 1u) <= 4.0f || !ragged(low_bit(t), below, above, key));
    }
    // windows that tell nothing new: most keys that share the ones above share them too
    const uint32_t flat = __ballot_sync(0xffffffffu, counts && t < full && near_more >= 8u && near_more * 2u > near_t);
    const uint32_t windows = __ballot_sync(0xffffffffu, t < full && (varies & bits_below(hb1 - 8u * t, 8u)) != 0ull);
    const uint32_t bytes = __ballot_sync(0xffffffffu, t < 8u && ((varies >> (8u * (t & 7u))) & 255u) != 0ull);
    const uint32_t runs = rule.skips ? (uint32_t)__popc(windows & ((1u << t) - 1u)) : t;
    uint32_t time = 10u * runs + (t > 4u ? 3u : 0u);
    if (t < full)
      time += rule.finish + (many_dups ? 4u : 0u) + (!even ? rule.uneven : (flat & ((1u << t) - 1u)) ? rule.straddle : 0u);
    else
      time += (runs & 1u) ? rule.copy : 0u;
    // the first t that is enough, evenly or not, and evenly any from there on
    const uint32_t ok = __ballot_sync(0xffffffffu, at_all && (t == full || enough(rule.near_limit)));
    const uint32_t first = (uint32_t)__ffs((int)ok) - 1u;
    const uint32_t best = __reduce_min_sync(0xffffffffu, at_all && t >= first && (t == first || even) ? time << 8 | t : ~0u);
    // a pass less for the big tile, whose runs are even and of the one or two top windows
    const bool fits_big = BIG && counts && t == rule.big_passes && full > t + 1u && even && near_t <= rule.big_near && st.big_far <= rule.far_limit &&
                          !heavy && !many_dups && varies == bits_below(hb1, 64u);
    const bool big = BIG && first == rule.big_passes + 1u && __any_sync(0xffffffffu, fits_big);
    const uint32_t passes = big ? rule.big_passes : varies == 0ull ? min(rule.tmin, full) : best & 255u;
    const uint32_t every = plain_passes ? plain_passes : (uint32_t)__popc(bytes);
    const uint32_t plain = 10u * every + (every > 4u || full <= 4u ? 3u : 0u) + ((every & 1u) ? rule.copy : 0u);
    const uint32_t near_of = __shfl_sync(0xffffffffu, near_t, (int)passes);
    if (t == 0u) {
      SampleChoice c;
      c.passes = passes;
      c.big = big;
      // (digits at byte boundaries are kinder to the counters' banks)
      c.plain = !big && varies != 0ull && (passes == full ? plain <= best >> 8 : plain < best >> 8);
      // heavy keys alone in their runs, and hardly two keys share one: tiles mostly in order
      c.skewed = heavy && passes < full && near_of * 256u <= kSample;
      c.dups = heavy || many_dups;
      st.choice = c;
    }
  }
  __syncthreads();
  return st.choice;
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

// Sorts the runs that start in [g, limit) of src[0, n) into X (src = X: in
// place), as many whole runs at a time as fit in a tile: a tile's worth comes
// in from where the CTA stands (the piece of a run at its end comes again with
// the next tile), the last run start in it is found, and the runs up to there
// are sorted. known: g is a run's start. load(from, count) brings src[from,
// from + count) into in[], a barrier before it and one after, and returns false
// for the whole CTA on an error; long_run(b, e), called by warp 0, takes a run of at
// least a tile. False after a failed load.
// dups: most keys are duplicates.
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
                                          const RunKey& w, const bool& clamped, const bool& skewed, const bool& dups, uint32_t shift, const Elem* in, uint32_t* slot,
                                          uint32_t* bins, typename TS::Shared& sh, RunMarks& marks, Load load,
                                          Long long_run) {
  constexpr uint32_t kNone = 0xffffffffu;
  constexpr int kMaxMixed = 2;                     // runs fixed one by one
  // threads that see an inversion: few and the runs are small, many and it is one long
  // one; else several are out of order and the whole tile is sorted. Zipf keys with 0
  // for few: 1.1 10^6 136 -> 165 us, 2 10^6 150 -> 168 (half zeros are 5 to 12 % faster so);
  // with 16, or with 5 or 1025 for many, within 2 % but for a batch of two arrays
  // (half zeros 3.09 -> 3.26 ms with 16 or 5; a tenth of sentinels 4.47 -> 4.16 with 1025).
  constexpr int kFewThreads = 4, kManyThreads = 64;
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
            TS::sort_any(in, a, b, slot, bins, sh, true, in_place, Uneven::kBits,
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
      auto emit = [=](bool on, uint32_t r, const Elem& e) { store_elem_if(on, out + r, e); };
      if (range == 0 || !TS::template sort_even<false>(in, from, end, TS::make_scale(base, range), slot, bins, sh, emit))
        TS::sort_any(in, from, end, slot, bins, sh, range == 0, in_place, dups ? Uneven::kDups : Uneven::kSpread, emit);
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
