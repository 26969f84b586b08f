// Tiles, digit counts and the scatter of one radix digit, shared by the sort (sort.cu) and by
// the pair stage's writes in rank order (pair.cu).
#pragma once

#include <algorithm>

#include "mlc_internal.h"
#include "scan.cuh"

namespace mlc {

static constexpr int SORT_THREADS = 512;
static constexpr int SORT_ITEMS = 16;
static constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;  // 8192
static constexpr int SORT_WARPS = SORT_THREADS / 32;

// The digit of a key that a pass goes by; make() once per thread.
struct ShiftDigit {
  int shift;
  __device__ __forceinline__ ShiftDigit make() const { return *this; }
  template <typename K>
  __device__ __forceinline__ unsigned operator()(K k) const {
    return (unsigned)(k >> shift) & 0xffu;
  }
};
// What radix_sort_range_u64_u32 left: the sorted keys, the keys as they were, or keys in no order
// (the last two have to be sorted by all their bits).
enum class RangeSort { DONE, UNTOUCHED, LOST };

// Byte `byte` of the top 32 bits of the keys' range: (key - lo) >> shift, lo and hi the least and
// the largest key (range[0], ~range[1], as two minima gather them).
struct RangeDigit {
  const unsigned long long* range;
  int byte;
  struct Made {
    uint64_t lo;
    int shift;
    __device__ __forceinline__ unsigned operator()(uint64_t k) const { return (unsigned)((k - lo) >> shift) & 0xffu; }
  };
  static __device__ __forceinline__ int base_shift(const unsigned long long* range) {
    return max(0, 32 - __clzll((long long)(~range[1] - range[0])));  // the top 32 bits of the range
  }
  __device__ __forceinline__ Made make() const { return Made{range[0], base_shift(range) + 8 * byte}; }
};

// Exclusive scan, in digit-major order, of hist[pass] (256 x ntiles) -> offsets (same
// layout).  One CTA per digit scans that digit's tiles, starting from the digit's
// global base: the count of all keys with a smaller digit, from the 256 digit totals.
static __global__ void __launch_bounds__(1024) k_scan_digit(const uint32_t* __restrict__ hist, int ntiles,
                                                     const unsigned long long* __restrict__ totals,
                                                     uint32_t* __restrict__ offs) {
  __shared__ uint32_t wsum[32];
  const int d = blockIdx.x;
  uint32_t running;
  block_exclusive_sum(threadIdx.x < (unsigned)d ? (uint32_t)totals[threadIdx.x] : 0u, &running, wsum);
  __syncthreads();  // wsum is rewritten by the first round
  for (int t0 = 0; t0 < ntiles; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x;
    const uint32_t v = (t < ntiles) ? hist[(long)d * ntiles + t] : 0;
    uint32_t agg;
    const uint32_t ex = block_exclusive_sum(v, &agg, wsum);
    if (t < ntiles) offs[(long)d * ntiles + t] = running + ex;
    running += agg;
    __syncthreads();  // wsum is rewritten by the next round
  }
}

// Per-tile counts of one digit position in the current key order: hist [digit][tile].
template <typename K, typename D>
__global__ void __launch_bounds__(SORT_THREADS) k_tile_hist(const K* __restrict__ keys, long n, int ntiles, D digit,
                                                            uint32_t* __restrict__ hist) {
  __shared__ uint32_t cnt[256];
  const auto dg = digit.make();
  for (int i = threadIdx.x; i < 256; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  const long t0 = (long)blockIdx.x * SORT_TILE;
#pragma unroll 4
  for (int q = 0; q < SORT_ITEMS; q++) {
    const long i = t0 + (long)q * SORT_THREADS + threadIdx.x;
    if (i < n) atomicAdd(&cnt[dg(keys[i])], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[(long)d * ntiles + blockIdx.x] = cnt[d];
}

// totals[p*256 + d] = number of keys whose digit p is d
static __global__ void __launch_bounds__(256) k_digit_totals(const uint32_t* __restrict__ hist, int ntiles,
                                                      unsigned long long* __restrict__ totals) {
  const long row = blockIdx.x;  // p*256 + d
  unsigned long long s = 0;
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x) s += hist[row * ntiles + t];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ unsigned long long red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; w++) t += red[w];
    totals[row] = t;
  }
}

// Rank of a lane's element among the elements of digit d that its warp has seen: those of
// earlier calls (cnt, the warp's counters) and of lower lanes.  Lanes without an element
// (!ok) count nowhere.  The lanes of the same digit by one vote per bit: eight votes issue
// faster than one __match_any_sync of an 8-bit value.
__device__ __forceinline__ uint32_t warp_digit_rank(unsigned d, bool ok, uint32_t* cnt, unsigned lt) {
  unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const unsigned v = __ballot_sync(0xffffffffu, (d >> k) & 1u);
    peers &= (d >> k) & 1u ? v : ~v;
  }
  uint32_t r = 0;
  if (ok) r = cnt[d] + __popc(peers & lt);
  __syncwarp();
  if (ok && (peers & lt) == 0) cnt[d] += __popc(peers);
  __syncwarp();
  return r;
}

// Turns the warps' digit counts wcnt[w][d] into each warp's first place of the digit in the
// CTA's digit order, and sets base[d] to the digit's own first place.  Every thread calls it
// after a barrier; ends with one.
template <int WARPS>
__device__ __forceinline__ void digit_places(uint32_t (*wcnt)[256], uint32_t* base, uint32_t* wsum) {
  uint32_t tot = 0;
  if (threadIdx.x < 256) {
#pragma unroll 4
    for (int w = 0; w < WARPS; w++) {
      const uint32_t c = wcnt[w][threadIdx.x];
      wcnt[w][threadIdx.x] = tot;
      tot += c;
    }
  }
  uint32_t agg;
  const uint32_t ex = block_exclusive_sum(tot, &agg, wsum);
  if (threadIdx.x < 256) {
    base[threadIdx.x] = ex;
#pragma unroll 4
    for (int w = 0; w < WARPS; w++) wcnt[w][threadIdx.x] += ex;
  }
  __syncthreads();
}

// One tile into digit order and out: key K with its digit, payload V from load(i) for element
// i of the input.  8.5e7 keys of 8 + 4 bytes: 2.37 ms a pass when every thread wrote the
// keys it had ranked (tiles of 4096: runs of 16 keys in random order), 0.64 ms in digit order
// from shared memory.  Two CTAs of 512 threads per SM.  A place of n or more is not written and sets
// *err, where there is one.
template <typename K, typename V, typename D, typename Load>
__global__ void __launch_bounds__(SORT_THREADS, 2) k_scatter(const K* __restrict__ kin, Load load, K* __restrict__ kout,
                                                             V* __restrict__ vout, long n, int ntiles, D digit,
                                                             const uint32_t* __restrict__ offs, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t wcnt[SORT_WARPS][256];  // per-warp running digit counts, then places
  __shared__ uint32_t gofs[256];              // global place of a digit's first key minus its place in the tile
  __shared__ uint32_t base[256];
  __shared__ uint32_t wsum[32];
  K* ks = reinterpret_cast<K*>(smem_raw);
  V* vs = reinterpret_cast<V*>(smem_raw);
  const auto dg = digit.make();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < SORT_WARPS * 256; i += SORT_THREADS) (&wcnt[0][0])[i] = 0;
  if (threadIdx.x < 256) gofs[threadIdx.x] = offs[(long)threadIdx.x * ntiles + blockIdx.x];
  // warp w owns tile elements [w*512, (w+1)*512): item q of lane l is element w*512 + 32q + l
  const long tile0 = (long)blockIdx.x * SORT_TILE;
  const int cnt = (int)min((long)SORT_TILE, n - tile0), e0 = warp * (SORT_ITEMS * 32) + lane;
  const K* kt = kin + tile0 + e0;
  K key[SORT_ITEMS];
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++) key[q] = e0 + q * 32 < cnt ? kt[q * 32] : (K)0;
  __syncthreads();
  uint32_t pos[SORT_ITEMS];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++) pos[q] = warp_digit_rank(dg(key[q]), e0 + q * 32 < cnt, wcnt[warp], lt);
  __syncthreads();
  digit_places<SORT_WARPS>(wcnt, base, wsum);
  if (threadIdx.x < 256) gofs[threadIdx.x] -= base[threadIdx.x];
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++)
    if (e0 + q * 32 < cnt) {
      pos[q] += wcnt[warp][dg(key[q])];
      ks[pos[q]] = key[q];
    }
  __syncthreads();
  const uint32_t un = (uint32_t)n;  // (n < 2^32)
  uint32_t dst[SORT_ITEMS];
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++) {
    const int i = threadIdx.x + q * SORT_THREADS;
    if (i < cnt) {
      const K k = ks[i];
      dst[q] = gofs[dg(k)] + (uint32_t)i;
      if (dst[q] < un) kout[dst[q]] = k;
      else if (err) atomicExch(err, 1);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++)
    if (e0 + q * 32 < cnt) vs[pos[q]] = load(tile0 + e0 + q * 32);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < SORT_ITEMS; q++) {
    const int i = threadIdx.x + q * SORT_THREADS;
    if (i < cnt && dst[q] < un) vout[dst[q]] = vs[i];
  }
}

struct LoadU32 {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(long i) const { return p[i]; }
};

template <typename K, typename V, typename D, typename Load>
static void scatter(mlc_ctx* ctx, const char* name, const K* kin, Load load, K* kout, V* vout, long n, int ntiles,
                    D digit, const uint32_t* offs, int* derr) {
  auto k = k_scatter<K, V, D, Load>;
  const size_t smem = (size_t)SORT_TILE * std::max(sizeof(K), sizeof(V));
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, name);
    k<<<ntiles, SORT_THREADS, smem, ctx->stream>>>(kin, load, kout, vout, n, ntiles, digit, offs, derr);
  }
  MLC_CHECK_LAUNCH();
}

// out[idx[i]] = load(i) for i < n; an idx of n or more writes nothing.  From BINNED_PUT_FROM values
// on they go through bins of nearby places: where out is larger than L2 (129 MB), writing each
// value by itself moves a 32-byte sector per value and reads it back first.  The values
// are put in the order of idx >> shift (256 bins, a digit of the sort) and then written bin
// by bin, whose places of out (1/256 of it) stay in L2 until their sectors are whole; one
// more trip of index and value through memory, in order.  8.5e7 values: ranks (4 bytes) 2.77
// ms directly, 1.27 ms; chi2 (8 bytes, with the FP64 arithmetic that makes them) 3.23 ms, 2.67 ms.
// Where the bins' 8 or 12 bytes a value do not fit the device, each value is written by itself.
// 4.2e7: 1.00 and 0.64; 1.46 and 1.33.  2.7e7: 0.33 and 0.41; 0.83 and 0.87.
template <typename V>
static __global__ void __launch_bounds__(256) k_put(const uint32_t* __restrict__ idx, const V* __restrict__ val, long n,
                                                    V* __restrict__ out) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t p = idx[i];
    if ((long)p < n) out[p] = val[i];
  }
}
template <typename V, typename Load>
static __global__ void __launch_bounds__(256) k_put_direct(const uint32_t* __restrict__ idx, Load load, long n,
                                                           V* __restrict__ out) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const uint32_t p = idx[i];
    if ((long)p < n) out[p] = load(i);
  }
}

constexpr long BINNED_PUT_FROM = 30'000'000;

template <typename V, typename Load>
static void put_by_index(mlc_ctx* ctx, const char* name, const uint32_t* idx, Load load, long n, V* out) {
  if (n <= 0) return;
  const int ntiles = (int)((n + SORT_TILE - 1) / SORT_TILE);
  if (n < BINNED_PUT_FROM || !ws_try(ctx, WS_SORT_KEYS, sizeof(V) * n) || !ws_try(ctx, WS_SORT_VALS, sizeof(uint32_t) * n) ||
      !ws_try(ctx, WS_SORT_HIST, sizeof(uint32_t) * 256 * (size_t)ntiles * 2 + 256 * 8)) {
    {
      MLC_KSCOPE(ctx, name);
      const int grid = (int)std::max<long>(1, std::min<long>((n + 255) / 256, (long)ctx->sm_count * 16));
      k_put_direct<V, Load><<<grid, 256, 0, ctx->stream>>>(idx, load, n, out);
    }
    MLC_CHECK_LAUNCH();
    return;
  }
  int shift = 0;
  while (((n - 1) >> shift) > 255) shift++;
  V* val = (V*)ws_get(ctx, WS_SORT_KEYS, sizeof(V) * n);
  uint32_t* key = (uint32_t*)ws_get(ctx, WS_SORT_VALS, sizeof(uint32_t) * n);
  uint32_t* hist = (uint32_t*)ws_get(ctx, WS_SORT_HIST, sizeof(uint32_t) * 256 * (size_t)ntiles * 2 + 256 * 8);
  uint32_t* offs = hist + (size_t)256 * ntiles;
  unsigned long long* dtot = reinterpret_cast<unsigned long long*>(offs + (size_t)256 * ntiles);
  {
    MLC_KSCOPE(ctx, name);
    k_tile_hist<uint32_t, ShiftDigit><<<ntiles, SORT_THREADS, 0, ctx->stream>>>(idx, n, ntiles, ShiftDigit{shift}, hist);
    k_digit_totals<<<256, 256, 0, ctx->stream>>>(hist, ntiles, dtot);
    k_scan_digit<<<256, 1024, 0, ctx->stream>>>(hist, ntiles, dtot, offs);
  }
  MLC_CHECK_LAUNCH();
  // (no error word: the places are counts of the same idx, below n whatever its values)
  scatter(ctx, name, idx, load, key, val, n, ntiles, ShiftDigit{shift}, offs, nullptr);
  {
    MLC_KSCOPE(ctx, name);
    k_put<V><<<(unsigned)((n + 2047) / 2048), 256, 0, ctx->stream>>>(key, val, n, out);
  }
  MLC_CHECK_LAUNCH();
}

}  // namespace mlc
