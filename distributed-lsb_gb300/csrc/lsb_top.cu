// lsb_top.cu -- the "top" kernel family: whole sorts that do not go through
// every digit of the key.
//
// mySort (mpi/mpi_lsbsort.cpp:592-597) sorts by all 64/RADIX digits, lowest
// first, each digit one pass over memory. Its result is the stable order of
// the keys, and that is what the kernels here produce: an array that fits in
// one CTA's shared memory is sorted there, in one launch.
#include <algorithm>

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
  Elem* in = reinterpret_cast<Elem*>(smem);
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + TS::kElemBytes + TS::kSlotBytes);
  for (uint32_t i = threadIdx.x; i < kCtrlBytes / 4u; i += THREADS) reinterpret_cast<uint32_t*>(ctrl)[i] = 0u;
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
    }
  }
  __syncthreads();
  uint64_t diff = 0;
  TS::sort(in, n, slot, bins, sh, true, [&](uint32_t r, const Elem& e) { store_elem(a + r, e); }, &diff);
  if (threadIdx.x == 0) write_plan(ctrl, diff, n, bits, num_digits, api_bits, sub);
}

// 1024 threads hold up to 9216 elements (212 KB of shared memory); up to half
// that 512 threads do, whose barriers cost less.
using SmallHalf = TileSort<512, 9>;
using SmallFull = TileSort<1024, 9>;

uint32_t top_small_limit() { return SmallFull::kCap; }

template <int THREADS>
static int small_sort(Elem* X, const Layout& L, Ctrl* ctrl, cudaStream_t st) {
  auto kern = k_small_sort<THREADS, 9>;
  const size_t smem = TileSort<THREADS, 9>::kSmem;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 5;
  ProfScope prof("small_sort", st);
  kern<<<1, THREADS, smem, st>>>(X, L.n, L.stat_bits, L.stat_digits, L.api_bits, L.sub, ctrl);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 5;
}

int top_run(Elem* X, Elem* Y, unsigned char* ws, const Layout& L, cudaStream_t st) {
  (void)Y;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(ws);
  return L.n <= SmallHalf::kCap ? small_sort<512>(X, L, ctrl, st) : small_sort<1024>(X, L, ctrl, st);
}

}  // namespace lsb
