// Hand-written stable LSD radix sort (8-bit digits) of 64-bit keys carrying 32-bit
// values, a stable-order scatter through bins for random writes, and warp-aggregated
// shared-memory histograms.
//
// Up to 16384 keys: one CTA sorts them in shared memory, all passes in one launch
// (10^4 keys: 0.25 ms of launches, scans and a host round trip before, 64 us now).
//
// More: k_digit_hist counts all eight digits of every tile in one read of the keys;
// their totals give each digit's global start and let passes where all keys share a
// digit be skipped.  Then one pass per remaining digit: (1) per-tile counts of that
// digit in the keys' current order (the up-front counts serve the first pass only,
// since each scatter permutes the keys); (2) k_scan_digit turns them into scatter
// offsets; (3) k_scatter ranks each key inside its tile in element order (stable; one
// vote per bit of the digit), puts the tile in digit order in shared memory and writes it
// from there: the keys of one digit are consecutive, 32 on average in a tile of 8192, so
// a warp writes a few whole runs (writing each key from the thread that ranked it cost
// 2.4 ms a pass for 8.5e7 keys, this 0.64; see k_scatter).  Every scatter address is checked against
// n; a violation sets an error flag instead of writing.

#include <mutex>
#include <unordered_map>

#include "mlc_internal.h"
#include "radix.cuh"

namespace mlc {

// Order-preserving map of an IEEE double to an unsigned key, and back.
__host__ __device__ __forceinline__ uint64_t f64_key(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double key_f64(uint64_t k) {
  return __longlong_as_double((k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k);
}

uint64_t f64_to_key(double d) { return f64_key(d); }

// hist layout: [pass][digit][tile]
__global__ void __launch_bounds__(SORT_THREADS) k_digit_hist(const uint64_t* __restrict__ keys, long n,
                                                             int ntiles, uint32_t* __restrict__ hist) {
  __shared__ uint32_t cnt[8][256];
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const long t0 = (long)blockIdx.x * SORT_TILE;
  for (int q = 0; q < SORT_ITEMS; q++) {
    const long i = t0 + (long)q * SORT_THREADS + threadIdx.x;
    if (i < n) {
      const uint64_t k = keys[i];
#pragma unroll
      for (int p = 0; p < 8; p++) atomicAdd(&cnt[p][(k >> (8 * p)) & 0xff], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) {
    const int p = i / 256, d = i % 256;
    hist[((long)p * 256 + d) * ntiles + blockIdx.x] = cnt[p][d];
  }
}

// The longest run of keys with equal sorted bits that one thread or warp puts in order.
constexpr int FIX_RUN = 64;

// Insertion of elements [b, e): a key passes only larger ones.
__device__ __forceinline__ void fix_run(uint64_t* ks, uint32_t* vals, int b, int e) {
  for (int i = b + 1; i < e; i++) {
    const uint64_t k = ks[i];
    if (ks[i - 1] <= k) continue;
    const uint32_t v = vals[i];
    int j = i;
    for (; j > b && ks[j - 1] > k; j--) {
      ks[j] = ks[j - 1];
      vals[j] = vals[j - 1];
    }
    ks[j] = k;
    vals[j] = v;
  }
}

// First place of the run of equal bits (key >> sh) that the descent at i (ks[i] > ks[i + 1])
// belongs to; -1 where an earlier descent of the run exists (which lists it), -2 where the run
// is too long.
__device__ __forceinline__ int run_of_descent(const uint64_t* ks, int i, uint64_t lo, int sh) {
  const uint64_t tp = (ks[i] - lo) >> sh;
  int b = i;
  while (b > 0 && i - b <= FIX_RUN && (ks[b - 1] - lo) >> sh == tp) {
    if (ks[b - 1] > ks[b]) return -1;
    b--;
  }
  return i - b > FIX_RUN ? -2 : b;
}

// Up to 1024 ITEMS keys in one CTA: stable LSD passes, keys and values in shared memory, held in
// registers while they change places.  Four passes over the 32 bits below the highest in
// which keys differ, then runs of equal bits that are out of order put right by a thread
// each; all other digits too where a run is too long for that (equal keys never are out of
// order).  F64: the keys are doubles, mapped on the way in and back out.
constexpr int SMALL_THREADS = 1024, SMALL_WARPS = SMALL_THREADS / 32, SMALL_MAX_ITEMS = 16;
constexpr long SMALL_MAX = (long)SMALL_THREADS * SMALL_MAX_ITEMS;

// One stable pass by the digit at `shift` over the CTA's THREADS x ITEMS keys and values in shared
// memory; item q of a thread is element e0 + 32 q.
template <int ITEMS, int THREADS>
__device__ __forceinline__ void cta_pass(uint64_t* ks, uint32_t* vs, uint64_t (&key)[ITEMS], uint32_t (*wcnt)[256],
                                         uint32_t* base, uint32_t* wsum, int e0, int shift) {
  constexpr int WARPS = THREADS / 32;
  const int warp = threadIdx.x >> 5;
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
  for (int i = threadIdx.x; i < WARPS * 256; i += THREADS) (&wcnt[0][0])[i] = 0;
#pragma unroll
  for (int q = 0; q < ITEMS; q++) key[q] = ks[e0 + 32 * q];
  __syncthreads();
  uint32_t pos[ITEMS];
#pragma unroll
  for (int q = 0; q < ITEMS; q++) pos[q] = warp_digit_rank((unsigned)(key[q] >> shift) & 0xffu, true, wcnt[warp], lt);
  __syncthreads();
  digit_places<WARPS>(wcnt, base, wsum);
#pragma unroll
  for (int q = 0; q < ITEMS; q++) {
    pos[q] += wcnt[warp][(unsigned)(key[q] >> shift) & 0xffu];
    ks[pos[q]] = key[q];
  }
  uint32_t v[ITEMS];
#pragma unroll
  for (int q = 0; q < ITEMS; q++) v[q] = vs[e0 + 32 * q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < ITEMS; q++) vs[pos[q]] = v[q];
  __syncthreads();
}

template <int ITEMS, bool F64>
__global__ void __launch_bounds__(SMALL_THREADS) k_sort_small(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                              int n) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int CAP = SMALL_THREADS * ITEMS;
  uint64_t* ks = reinterpret_cast<uint64_t*>(smem_raw);
  uint32_t* vs = reinterpret_cast<uint32_t*>(ks + CAP);
  uint32_t (*wcnt)[256] = reinterpret_cast<uint32_t (*)[256]>(vs + CAP);
  uint16_t* list = reinterpret_cast<uint16_t*>(vs + CAP);  // (the counters' space, after the passes)
  __shared__ uint32_t base[256];
  __shared__ uint32_t wsum[32];
  __shared__ unsigned long long differ;
  __shared__ int nlist, too_long;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = warp * (ITEMS * 32) + lane;  // item q is element e0 + 32 q
  if (threadIdx.x == 0) differ = 0, nlist = 0, too_long = 0;
  __syncthreads();
  uint64_t first = keys[0];
  if (F64) first = f64_key(__longlong_as_double((long long)first));
  uint64_t key[ITEMS];
  uint64_t m = 0;
#pragma unroll
  for (int q = 0; q < ITEMS; q++) {
    const int e = e0 + 32 * q;
    key[q] = ~0ull;  // (places past n: all bits set, and after the others of their digit, so they stay last)
    if (e < n) {
      const uint64_t k = keys[e];
      key[q] = F64 ? f64_key(__longlong_as_double((long long)k)) : k;
      m |= key[q] ^ first;
      vs[e] = vals[e];
    }
    ks[e] = key[q];
  }
  if (m) atomicOr(&differ, (unsigned long long)m);
  __syncthreads();
  const uint64_t diff = differ;
  auto pass = [&](int shift) { cta_pass<ITEMS, SMALL_THREADS>(ks, vs, key, wcnt, base, wsum, e0, shift); };
  const int sh = diff ? max(0, 32 - __clzll((long long)diff)) : 64;  // the lowest sorted bit
#pragma unroll 1
  for (int shift = sh; shift < min(64, sh + 32); shift += 8)
    if ((diff >> shift) & 0xff) pass(shift);
  if (sh > 0 && sh < 64) {
    for (int i = threadIdx.x; i + 1 < n; i += SMALL_THREADS) {
      if (!(ks[i] > ks[i + 1])) continue;
      const int b = run_of_descent(ks, i, 0, sh);
      if (b >= 0) list[atomicAdd(&nlist, 1)] = (uint16_t)b;
      else if (b == -2) too_long = 1;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nlist; r += SMALL_THREADS) {
      const int b = list[r];
      int e = b + 1;
      while (e < n && e - b <= FIX_RUN && (ks[e] >> sh) == (ks[b] >> sh)) e++;
      if (e - b > FIX_RUN) too_long = 1;
      else fix_run(ks, vs, b, e);
    }
    __syncthreads();
    if (too_long) {
#pragma unroll 1
      for (int shift = 0; shift < 64; shift += 8)
        if ((diff >> shift) & 0xff) pass(shift);
    }
  }
#pragma unroll
  for (int q = 0; q < ITEMS; q++) {
    const int e = e0 + 32 * q;
    if (e < n) {
      const uint64_t k = ks[e];
      keys[e] = F64 ? (uint64_t)__double_as_longlong(key_f64(k)) : k;
      vals[e] = vs[e];
    }
  }
}

template <bool F64>
static void sort_small(mlc_ctx* ctx, int n, uint64_t* keys, uint32_t* vals) {
  using K = void (*)(uint64_t*, uint32_t*, int);
  const int items = (n + SMALL_THREADS - 1) / SMALL_THREADS;
  K k = k_sort_small<16, F64>;
  int cap = 16;
  if (items <= 1) k = k_sort_small<1, F64>, cap = 1;
  else if (items <= 2) k = k_sort_small<2, F64>, cap = 2;
  else if (items <= 4) k = k_sort_small<4, F64>, cap = 4;
  else if (items <= 8) k = k_sort_small<8, F64>, cap = 8;
  const size_t smem = (size_t)cap * SMALL_THREADS * 12 + sizeof(uint32_t) * SMALL_WARPS * 256;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, "sort_small");
    k<<<1, SMALL_THREADS, smem, ctx->stream>>>(keys, vals, n);
  }
  MLC_CHECK_LAUNCH();
}

// Sorts keys/vals (device, n) stably; uses two workspace buffers.  Result in place.
void radix_sort_u64_u32(mlc_ctx* ctx, long n, uint64_t* keys, uint32_t* vals) {
  if (n <= 1) return;
  if (n <= SMALL_MAX) {
    sort_small<false>(ctx, (int)n, keys, vals);
    return;
  }
  MLC_REQUIRE(n <= 0xFFFFFFFFl, MLC_ERR_LIMIT, "sort length above 2^32-1");
  const int ntiles = (int)((n + SORT_TILE - 1) / SORT_TILE);
  uint64_t* k2 = (uint64_t*)ws_get(ctx, WS_SORT_KEYS, sizeof(uint64_t) * n);
  uint32_t* v2 = (uint32_t*)ws_get(ctx, WS_SORT_VALS, sizeof(uint32_t) * n);
  uint32_t* hist = (uint32_t*)ws_get(ctx, WS_SORT_HIST, sizeof(uint32_t) * 256 * (size_t)ntiles * 9 + 8 * 256 * 8 + 64);
  uint32_t* offs = hist + (size_t)8 * 256 * ntiles;
  unsigned long long* dtot = reinterpret_cast<unsigned long long*>(offs + (size_t)256 * ntiles);
  int* derr = reinterpret_cast<int*>(dtot + 8 * 256);
  MLC_CUDA(cudaMemsetAsync(derr, 0, sizeof(int), ctx->stream));
  {
    MLC_KSCOPE(ctx, "sort_digit_hist");
    k_digit_hist<<<ntiles, SORT_THREADS, 0, ctx->stream>>>(keys, n, ntiles, hist);
  }
  MLC_CHECK_LAUNCH();
  {
    MLC_KSCOPE(ctx, "sort_digit_totals");
    k_digit_totals<<<8 * 256, 256, 0, ctx->stream>>>(hist, ntiles, dtot);
  }
  MLC_CHECK_LAUNCH();
  // Digit totals to the host: positions where all keys agree are skipped.
  std::vector<unsigned long long> h(8 * 256);
  MLC_CUDA(cudaMemcpyAsync(h.data(), dtot, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                           ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));
  uint64_t* ka = keys;
  uint32_t* va = vals;
  uint64_t* kb = k2;
  uint32_t* vb = v2;
  bool first = true;
  for (int p = 0; p < 8; p++) {
    bool trivial = false;
    for (int d = 0; d < 256; d++) trivial |= h[p * 256 + d] == (unsigned long long)n;
    if (trivial) continue;
    if (!first) {  // per-tile counts of digit p in the current order
      MLC_KSCOPE(ctx, "sort_tile_hist");
      k_tile_hist<uint64_t, ShiftDigit><<<ntiles, SORT_THREADS, 0, ctx->stream>>>(ka, n, ntiles, ShiftDigit{8 * p},
                                                                                  hist + (size_t)p * 256 * ntiles);
    }
    MLC_CHECK_LAUNCH();
    first = false;
    {
      MLC_KSCOPE(ctx, "sort_scan");
      k_scan_digit<<<256, 1024, 0, ctx->stream>>>(hist + (size_t)p * 256 * ntiles, ntiles, dtot + p * 256, offs);
    }
    MLC_CHECK_LAUNCH();
    scatter(ctx, "sort_scatter", ka, LoadU32{va}, kb, vb, n, ntiles, ShiftDigit{8 * p}, offs, derr);
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    MLC_CUDA(cudaMemcpyAsync(keys, ka, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
    MLC_CUDA(cudaMemcpyAsync(vals, va, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
  }
  int herr = 0;
  MLC_CUDA(cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));
  MLC_REQUIRE(herr == 0, MLC_ERR_CUDA, "radix sort: scatter offset out of range (inconsistent digit counts)");
}

// ---- keys spread over their range: four passes instead of eight
//
// Of the 64 key bits of values that fill a range, the top 32 of (key - least key) almost
// decide the order: of 8.5e7 quotients over some twenty octaves about one key in six has a
// neighbour of the same 32 bits.  Four stable passes order the keys by them; where two
// neighbours of the same top bits then stand in the wrong order (a descent), their run is
// sorted by its full keys, stably, by a thread or a warp: within tiles of the keys in shared memory
// (k_fix_tiles), then across the tiles' edges (k_fix_edges).  Runs of equal keys are in order
// as they stand, however long.  A run with a descent that is longer than FIX_RUN is noted
// (long_run) and sorted by a CTA, up to RUN_MAX keys in shared memory (k_sort_runs), longer ones
// through the second buffers (k_sort_big), by its keys less the least of them: a digit or two.  A
// few beyond BIG_MAX are sorted as ranges of their own.  Quotients of ray counts come in runs
// of 10^2 to 10^4 equal keys, and equal fractions of different counts share their top bits.  Rank
// of 1500 and 2200 locations with counts around 300: 0.51 and 0.93 ms by all bits, 0.82 and
// 1.68 with long runs sorted by comparison or one by one from the host, 0.40 and 0.55 as here.
constexpr int FIX_TILE = 4096, FIX_THREADS = 256;
constexpr int RUN_SLOTS = 8192, BIG_RUNS = 1024, HOST_RUNS = 8;
constexpr int RUN_THREADS = 256, RUN_ITEMS = 8, RUN_MAX = RUN_THREADS * RUN_ITEMS;
constexpr int BIG_THREADS = 1024, BIG_ITEMS = 8, BIG_TILE = BIG_THREADS * BIG_ITEMS;
constexpr unsigned long long BIG_MAX = 1 << 18;
struct LongRuns {
  int scatter_err, full, nbig;  // full: more runs than there is room for, the order is not made
  unsigned long long at[RUN_SLOTS];  // first key of a noted run (~0: none), by a hash of it
  unsigned long long big_at[BIG_RUNS], big_end[BIG_RUNS];
};

// First of the n keys, ordered by their top bits, whose top bits are at least tp.
__device__ __forceinline__ long lower_bound_top(const uint64_t* __restrict__ keys, long n, uint64_t lo, int sh, uint64_t tp) {
  long b = 0, e = n;
  while (b < e) {
    const long m = (b + e) / 2;
    if (((keys[m] - lo) >> sh) < tp) b = m + 1;
    else e = m;
  }
  return b;
}
// start: the run's first place, -1 where it has to be searched for.
__device__ __noinline__ void long_run(const uint64_t* keys, long n, uint64_t lo, int sh, uint64_t tp, long start,
                                      LongRuns* lr) {
  const unsigned long long b = (unsigned long long)(start >= 0 ? start : lower_bound_top(keys, n, lo, sh, tp));
  const unsigned h = ((unsigned)b * 2654435761u) >> 16;
  for (unsigned r = 0; r < 64; r++) {
    const unsigned long long was = atomicCAS(&lr->at[(h + r) % RUN_SLOTS], ~0ull, b);
    if (was == ~0ull || was == b) return;
  }
  atomicExch(&lr->full, 1);
}
// A CTA per slot: the noted run, stably sorted by its keys less the least of them.
__global__ void __launch_bounds__(RUN_THREADS) k_sort_runs(uint64_t* keys, uint32_t* vals, long n,
                                                           const unsigned long long* __restrict__ range,
                                                           LongRuns* __restrict__ lr) {
  __shared__ uint64_t ks[RUN_MAX];
  __shared__ uint32_t vs[RUN_MAX];
  __shared__ uint32_t wcnt[RUN_THREADS / 32][256];
  __shared__ uint32_t base[256], wsum[32];
  __shared__ unsigned long long least, most;
  __shared__ int len_s;
  const unsigned long long b = lr->at[blockIdx.x];
  if (b == ~0ull) return;
  if (threadIdx.x == 0) least = ~0ull, most = 0, len_s = 0;
  __syncthreads();
  const uint64_t lo = range[0];
  const int sh = RangeDigit::base_shift(range);
  const uint64_t tp = (keys[b] - lo) >> sh;
  const long rest = n - (long)b;
  const int e0 = (threadIdx.x >> 5) * (RUN_ITEMS * 32) + (threadIdx.x & 31);
  uint64_t key[RUN_ITEMS], kmin = ~0ull, kmax = 0;
  int in = 0;
#pragma unroll
  for (int q = 0; q < RUN_ITEMS; q++) {
    const int e = e0 + 32 * q;
    if (e < rest) {
      const uint64_t k = keys[b + e];
      if ((k - lo) >> sh == tp) {
        key[q] = k;
        vs[e] = vals[b + e];
        kmin = min(kmin, k);
        kmax = max(kmax, k);
        in++;
      }
    }
  }
  if (in) {
    atomicAdd(&len_s, in);
    atomicMin(&least, (unsigned long long)kmin);
    atomicMax(&most, (unsigned long long)kmax);
  }
  __syncthreads();
  const int len = len_s;
  if (len == RUN_MAX && rest > RUN_MAX && (keys[b + RUN_MAX] - lo) >> sh == tp) {
    if (threadIdx.x == 0) {
      const int r = atomicAdd(&lr->nbig, 1);
      if (r < BIG_RUNS) lr->big_at[r] = b, lr->big_end[r] = b + lower_bound_top(keys + b, rest, lo, sh, tp + 1);
      else atomicExch(&lr->full, 1);
    }
    return;
  }
  const uint64_t k0 = least, spread = most - k0;
  // (places past the run: all bits set, and after the others of their digit, so they stay there)
#pragma unroll
  for (int q = 0; q < RUN_ITEMS; q++) ks[e0 + 32 * q] = e0 + 32 * q < len ? key[q] - k0 : ~0ull;
  __syncthreads();
#pragma unroll 1
  for (int shift = 0; shift < 64 && spread >> shift; shift += 8)
    cta_pass<RUN_ITEMS, RUN_THREADS>(ks, vs, key, wcnt, base, wsum, e0, shift);
#pragma unroll
  for (int q = 0; q < RUN_ITEMS; q++) {
    const int e = e0 + 32 * q;
    if (e < len) {
      keys[b + e] = ks[e] + k0;
      vals[b + e] = vs[e];
    }
  }
}

// The same for runs beyond RUN_MAX (a CTA each, up to BIG_MAX keys): tile by tile from one buffer
// to the other, each digit's next place in shared memory.
__global__ void __launch_bounds__(BIG_THREADS) k_sort_big(uint64_t* keys, uint32_t* vals, uint64_t* k2, uint32_t* v2,
                                                          const LongRuns* __restrict__ lr) {
  constexpr int WARPS = BIG_THREADS / 32;
  __shared__ uint32_t wcnt[WARPS][256];
  __shared__ uint32_t base[256], next[256], wsum[32];
  __shared__ unsigned long long least, most;
  const unsigned long long b = lr->big_at[blockIdx.x], all = lr->big_end[blockIdx.x] - b;
  if (all > BIG_MAX) return;
  const int len = (int)all, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e0 = warp * (BIG_ITEMS * 32) + lane;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t *ka = keys + b, *kb = k2 + b;
  uint32_t *va = vals + b, *vb = v2 + b;
  if (threadIdx.x == 0) least = ~0ull, most = 0;
  __syncthreads();
  // few digits occur, so that one atomic per warp and digit does
  auto count = [&](int n, auto at) {
    for (int i0 = 0; i0 < n; i0 += BIG_THREADS) {
      const int i = i0 + threadIdx.x;
      const unsigned d = i < n ? at(i) : 256u, peers = __match_any_sync(0xffffffffu, d);
      if (d < 256 && (peers & lt) == 0) atomicAdd(&next[d], (uint32_t)__popc(peers));
    }
  };
  uint64_t kmin = ~0ull, kmax = 0;
#pragma unroll 4
  for (int i = threadIdx.x; i < len; i += BIG_THREADS) {
    const uint64_t k = ka[i];
    kmin = min(kmin, k);
    kmax = max(kmax, k);
  }
  atomicMin(&least, (unsigned long long)kmin);
  atomicMax(&most, (unsigned long long)kmax);
  __syncthreads();
  const uint64_t k0 = least, spread = most - k0;
#pragma unroll 1
  for (int shift = 0; shift < 64 && spread >> shift; shift += 8) {
    auto digit = [&](uint64_t k) { return (unsigned)((k - k0) >> shift) & 0xffu; };
    if (threadIdx.x < 256) next[threadIdx.x] = 0;
    __syncthreads();
    count(len, [&](int i) { return digit(ka[i]); });
    __syncthreads();
    uint32_t agg;
    const uint32_t ex = block_exclusive_sum(threadIdx.x < 256 ? next[threadIdx.x] : 0u, &agg, wsum);
    __syncthreads();
    if (threadIdx.x < 256) next[threadIdx.x] = ex;
#pragma unroll 1
    for (int t0 = 0; t0 < len; t0 += BIG_TILE) {
      const int cnt = min(BIG_TILE, len - t0);
      for (int i = threadIdx.x; i < WARPS * 256; i += BIG_THREADS) (&wcnt[0][0])[i] = 0;
      __syncthreads();
      uint64_t key[BIG_ITEMS];
      uint32_t pos[BIG_ITEMS];
#pragma unroll
      for (int q = 0; q < BIG_ITEMS; q++) key[q] = e0 + 32 * q < cnt ? ka[t0 + e0 + 32 * q] : 0ull;
#pragma unroll
      for (int q = 0; q < BIG_ITEMS; q++)
        pos[q] = warp_digit_rank(digit(key[q]), e0 + 32 * q < cnt, wcnt[warp], lt);
      __syncthreads();
      digit_places<WARPS>(wcnt, base, wsum);
#pragma unroll
      for (int q = 0; q < BIG_ITEMS; q++)
        if (e0 + 32 * q < cnt) {
          const unsigned d = digit(key[q]);
          const uint32_t dst = next[d] + pos[q] + wcnt[warp][d] - base[d];  // (below len)
          kb[dst] = key[q];
          vb[dst] = va[t0 + e0 + 32 * q];
        }
      __syncthreads();
      if (threadIdx.x < 256) next[threadIdx.x] += (threadIdx.x < 255 ? base[threadIdx.x + 1] : cnt) - base[threadIdx.x];
      __syncthreads();
    }
    uint64_t* tk = ka;
    ka = kb;
    kb = tk;
    uint32_t* tv = va;
    va = vb;
    vb = tv;
  }
  if (ka != keys + b)
    for (int i = threadIdx.x; i < len; i += BIG_THREADS) {
      kb[i] = ka[i];
      vb[i] = va[i];
    }
}

// A run of up to 32 KPL keys, stably sorted by one warp that counts the keys before each.  (A
// thread's insertions move keys and values in memory one after another: 160 us where a run of
// 60 was among them.)
constexpr int THREAD_RUN = 8;  // keys of a run that one thread sorts by insertion
template <int KPL>
__device__ __forceinline__ void warp_run(uint64_t* keys, uint32_t* vals, int len) {
  const int lane = threadIdx.x & 31;
  uint64_t k[KPL];
  uint32_t v[KPL];
  int r[KPL];
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    const bool in = lane + 32 * q < len;
    k[q] = in ? keys[lane + 32 * q] : ~0ull;
    v[q] = in ? vals[lane + 32 * q] : 0u;
    r[q] = 0;
  }
#pragma unroll
  for (int p = 0; p < KPL; p++)
    for (int l = 0; l < 32 && 32 * p + l < len; l++) {
      const uint64_t o = __shfl_sync(0xffffffffu, k[p], l);
#pragma unroll
      for (int q = 0; q < KPL; q++) r[q] += o < k[q] || (o == k[q] && 32 * p + l < lane + 32 * q);
    }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < KPL; q++)
    if (lane + 32 * q < len) {
      keys[r[q]] = k[q];
      vals[r[q]] = v[q];
    }
}

__global__ void __launch_bounds__(FIX_THREADS) k_fix_tiles(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                           long n, const unsigned long long* __restrict__ range,
                                                           LongRuns* __restrict__ lr) {
  __shared__ uint64_t ks[FIX_TILE];
  __shared__ uint16_t list[FIX_TILE / 2];  // first elements of the runs to sort (two keys or more each)
  __shared__ uint32_t wide[FIX_TILE / THREAD_RUN];  // those of more than THREAD_RUN keys: first element and length
  __shared__ int nlist, nwide;
  const uint64_t lo = range[0];
  const int sh = RangeDigit::base_shift(range);
  const long t0 = (long)blockIdx.x * FIX_TILE;
  const int cnt = (int)min((long)FIX_TILE, n - t0);
  if (threadIdx.x == 0) nlist = nwide = 0;
  for (int i = threadIdx.x; i < cnt; i += FIX_THREADS) ks[i] = keys[t0 + i];
  __syncthreads();
  auto top = [&](uint64_t k) { return (k - lo) >> sh; };
  for (int i = threadIdx.x; i + 1 < cnt; i += FIX_THREADS) {
    if (!(ks[i] > ks[i + 1])) continue;  // (a descent has equal top bits: the keys are in their order)
    int b = run_of_descent(ks, i, lo, sh);
    // (a long run may be listed for each descent that has none in the FIX_RUN keys before it)
    if (b == -2) b = (int)lower_bound_top(ks, i, lo, sh, top(ks[i]));
    if (b >= 0) list[atomicAdd(&nlist, 1)] = (uint16_t)b;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < nlist; r += FIX_THREADS) {
    const int b = list[r];
    const uint64_t tp = top(ks[b]);
    int e = b + 1;
    while (e < cnt && e - b <= FIX_RUN && top(ks[e]) == tp) e++;
    if (e - b > FIX_RUN) {
      long_run(keys, n, lo, sh, tp, b > 0 ? t0 + b : -1, lr);
      continue;
    }
    // (a run that goes on in a neighbouring tile is k_fix_edges')
    if ((b == 0 && t0 > 0 && top(keys[t0 - 1]) == tp) || (e == cnt && t0 + e < n && top(keys[t0 + e]) == tp)) continue;
    if (e - b > THREAD_RUN) {
      wide[atomicAdd(&nwide, 1)] = (uint32_t)b | (uint32_t)(e - b) << 16;
      continue;
    }
    fix_run(ks, vals + t0, b, e);
    for (int i = b; i < e; i++) keys[t0 + i] = ks[i];
  }
  __syncthreads();
  for (int r = threadIdx.x >> 5; r < nwide; r += FIX_THREADS / 32) {
    const uint32_t w = wide[r];
    warp_run<2>(keys + t0 + (w & 0xffffu), vals + t0 + (w & 0xffffu), (int)(w >> 16));
  }
}

// The runs across the edge at the start of tile 1, 2, ...: a warp each, whose lanes look at the keys
// on both sides at once (one thread's walk through a long run took 40 us).
__global__ void __launch_bounds__(256) k_fix_edges(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, long n,
                                                   const unsigned long long* __restrict__ range,
                                                   LongRuns* __restrict__ lr) {
  static_assert(FIX_RUN == 64, "two keys a lane");
  const uint64_t lo = range[0];
  const int sh = RangeDigit::base_shift(range), lane = threadIdx.x & 31;
  const long j = (((long)blockIdx.x * blockDim.x + threadIdx.x) / 32 + 1) * FIX_TILE;
  if (j >= n) return;  // (a whole warp)
  const uint64_t tp = (keys[j] - lo) >> sh;
  auto same = [&](long i) { return i >= 0 && i < n && (keys[i] - lo) >> sh == tp; };
  // keys of the run from place i on in steps of dir, counted up to FIX_RUN + 1
  auto length = [&](long i, int dir) {
    const unsigned a = __ballot_sync(0xffffffffu, same(i + dir * lane)), b = __ballot_sync(0xffffffffu, same(i + dir * (32 + lane)));
    if (a != ~0u) return __ffs(~a) - 1;
    if (b != ~0u) return 32 + __ffs(~b) - 1;
    return same(i + dir * 64) ? 65 : 64;
  };
  const int before = length(j - 1, -1), after = length(j, 1);
  if (before == 0) return;
  const long b = j - before, e = j + after;
  bool descent = false;
  for (long i = b + lane; i + 1 < e; i += 32) descent |= keys[i] > keys[i + 1];
  if (!__any_sync(0xffffffffu, descent)) return;
  if (before <= FIX_RUN && after <= FIX_RUN) warp_run<4>(keys + b, vals + b, (int)(e - b));
  else if (lane == 0) long_run(keys, n, lo, sh, tp, before <= FIX_RUN ? b : -1, lr);
}

// An even sample of the keys, and how many neighbours of the sorted sample are unequal but share
// their top bits with each other and with a third.
constexpr int CLOSE_SAMPLE = 4096, CLOSE_LIMIT = 16;
constexpr uint64_t ZERO_KEY = 1ull << 63, INF_KEY = ZERO_KEY | 0x7ff0000000000000ull;  // of doubles (f64_key)
constexpr long CLOSE_FROM = 1L << 24;  // (the sample takes 40 us, the four passes of 2.3e6 keys 200)
__global__ void __launch_bounds__(256) k_sample_keys(const uint64_t* __restrict__ keys, long n,
                                                     uint64_t* __restrict__ out, uint32_t* __restrict__ vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= CLOSE_SAMPLE) return;
  out[i] = keys[(long)((double)i * (double)n / CLOSE_SAMPLE)];  // (below n for i < CLOSE_SAMPLE <= n)
  vals[i] = i;
}
__global__ void __launch_bounds__(256) k_count_close(const uint64_t* __restrict__ keys,
                                                     const unsigned long long* __restrict__ range,
                                                     int* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t lo = range[0];
  const int sh = RangeDigit::base_shift(range);
  auto same = [&](int a, int b) { return a >= 0 && b < CLOSE_SAMPLE && (keys[a] - lo) >> sh == (keys[b] - lo) >> sh; };
  if (same(i, i + 1) && keys[i] != keys[i + 1] && (same(i - 1, i) || same(i + 1, i + 2))) atomicAdd(count, 1);
}

// Sorts keys/vals stably by the top of their range, then fixes what that leaves.  range (device):
// the least key, and the least ~key.  Where many keys lie in long runs (counts of a convolved map,
// each with its own rounding in the last bits) a sample tells so before the four passes are
// spent; a range that zeros, infinities or NaN stretch over all exponents is not tried (9216
// locations of a ray-shot map, one in seventeen without a ray: 17.9 -> 10.8 ms).
RangeSort radix_sort_range_u64_u32(mlc_ctx* ctx, long n, uint64_t* keys, uint32_t* vals, const unsigned long long* range) {
  MLC_REQUIRE(n <= 0xFFFFFFFFl, MLC_ERR_LIMIT, "sort length above 2^32-1");
  const int ntiles = (int)((n + SORT_TILE - 1) / SORT_TILE);
  uint64_t* k2 = (uint64_t*)ws_get(ctx, WS_SORT_KEYS, sizeof(uint64_t) * n);
  uint32_t* v2 = (uint32_t*)ws_get(ctx, WS_SORT_VALS, sizeof(uint32_t) * n);
  uint32_t* hist = (uint32_t*)ws_get(ctx, WS_SORT_HIST, sizeof(uint32_t) * 256 * (size_t)ntiles * 2 + 256 * 8 +
                                                                sizeof(LongRuns));
  uint32_t* offs = hist + (size_t)256 * ntiles;
  unsigned long long* dtot = reinterpret_cast<unsigned long long*>(offs + (size_t)256 * ntiles);
  LongRuns* dl = reinterpret_cast<LongRuns*>(dtot + 256);
  MLC_CUDA(cudaMemsetAsync(dl, 0, offsetof(LongRuns, at), ctx->stream));
  MLC_CUDA(cudaMemsetAsync(dl->at, 0xff, sizeof dl->at, ctx->stream));
  if (n >= CLOSE_FROM) {
    {
      MLC_KSCOPE(ctx, "sort_sample");
      k_sample_keys<<<CLOSE_SAMPLE / 256, 256, 0, ctx->stream>>>(keys, n, k2, v2);
    }
    sort_small<false>(ctx, CLOSE_SAMPLE, k2, v2);
    {
      MLC_KSCOPE(ctx, "sort_sample");
      k_count_close<<<CLOSE_SAMPLE / 256, 256, 0, ctx->stream>>>(k2, range, &dl->nbig);
    }
    MLC_CHECK_LAUNCH();
    int close = 0;
    unsigned long long r[2];
    MLC_CUDA(cudaMemcpyAsync(&close, &dl->nbig, sizeof close, cudaMemcpyDeviceToHost, ctx->stream));
    MLC_CUDA(cudaMemcpyAsync(r, range, sizeof r, cudaMemcpyDeviceToHost, ctx->stream));
    MLC_CUDA(cudaStreamSynchronize(ctx->stream));
    if (close >= CLOSE_LIMIT || r[0] <= ZERO_KEY || ~r[1] >= INF_KEY) return RangeSort::UNTOUCHED;
    MLC_CUDA(cudaMemsetAsync(&dl->nbig, 0, sizeof(int), ctx->stream));
  }
  uint64_t* ka = keys;
  uint32_t* va = vals;
  uint64_t* kb = k2;
  uint32_t* vb = v2;
  for (int p = 0; p < 4; p++) {
    const RangeDigit dg{range, p};
    {
      MLC_KSCOPE(ctx, "sort_tile_hist");
      k_tile_hist<uint64_t, RangeDigit><<<ntiles, SORT_THREADS, 0, ctx->stream>>>(ka, n, ntiles, dg, hist);
    }
    MLC_CHECK_LAUNCH();
    {
      MLC_KSCOPE(ctx, "sort_scan");
      k_digit_totals<<<256, 256, 0, ctx->stream>>>(hist, ntiles, dtot);
      k_scan_digit<<<256, 1024, 0, ctx->stream>>>(hist, ntiles, dtot, offs);
    }
    MLC_CHECK_LAUNCH();
    scatter(ctx, "sort_scatter", ka, LoadU32{va}, kb, vb, n, ntiles, dg, offs, &dl->scatter_err);
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  // (four passes: the result is back in keys)
  {
    MLC_KSCOPE(ctx, "sort_fix");
    const long tiles = (n + FIX_TILE - 1) / FIX_TILE;
    k_fix_tiles<<<(unsigned)tiles, FIX_THREADS, 0, ctx->stream>>>(keys, vals, n, range, dl);
    k_fix_edges<<<(unsigned)((tiles + 7) / 8), 256, 0, ctx->stream>>>(keys, vals, n, range, dl);
    k_sort_runs<<<RUN_SLOTS, RUN_THREADS, 0, ctx->stream>>>(keys, vals, n, range, dl);
  }
  MLC_CHECK_LAUNCH();
  struct {
    int scatter_err, full, nbig;
  } h;
  MLC_CUDA(cudaMemcpyAsync(&h, dl, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));
  MLC_REQUIRE(h.scatter_err == 0, MLC_ERR_CUDA, "radix sort: scatter offset out of range (inconsistent digit counts)");
  if (h.full) return RangeSort::LOST;
  if (h.nbig == 0) return RangeSort::DONE;
  {
    MLC_KSCOPE(ctx, "sort_big_runs");
    k_sort_big<<<h.nbig, BIG_THREADS, 0, ctx->stream>>>(keys, vals, k2, v2, dl);
  }
  MLC_CHECK_LAUNCH();
  std::vector<unsigned long long> big(2 * BIG_RUNS);
  MLC_CUDA(cudaMemcpyAsync(big.data(), dl->big_at, sizeof dl->big_at + sizeof dl->big_end, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<int> host;
  for (int r = 0; r < h.nbig; r++)
    if (big[BIG_RUNS + r] - big[r] > BIG_MAX) host.push_back(r);
  if ((int)host.size() > HOST_RUNS) return RangeSort::LOST;
  // (their keys agree in most digits, whose passes are skipped)
  for (int r : host) radix_sort_u64_u32(ctx, (long)(big[BIG_RUNS + r] - big[r]), keys + big[r], vals + big[r]);
  return RangeSort::DONE;
}

__global__ void k_f64_to_keys(double* __restrict__ v, long n) {
  uint64_t* u = reinterpret_cast<uint64_t*>(v);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    u[i] = f64_key(v[i]);
}
__global__ void k_keys_to_f64(double* __restrict__ v, long n) {
  uint64_t* u = reinterpret_cast<uint64_t*>(v);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    v[i] = key_f64(u[i]);
}

void sort_f64_u32(mlc_ctx* ctx, long n, double* keys, uint32_t* vals) {
  if (n <= 1) return;
  if (n <= SMALL_MAX) {
    sort_small<true>(ctx, (int)n, reinterpret_cast<uint64_t*>(keys), vals);
    return;
  }
  const int grid = (int)std::min<long>((n + 255) / 256, (long)ctx->sm_count * 16);
  {
    MLC_KSCOPE(ctx, "sort_keys_in");
    k_f64_to_keys<<<grid, 256, 0, ctx->stream>>>(keys, n);
  }
  MLC_CHECK_LAUNCH();
  radix_sort_u64_u32(ctx, n, reinterpret_cast<uint64_t*>(keys), vals);
  {
    MLC_KSCOPE(ctx, "sort_keys_out");
    k_keys_to_f64<<<grid, 256, 0, ctx->stream>>>(keys, n);
  }
  MLC_CHECK_LAUNCH();
}

// Histogram with warp-aggregated shared-memory counters; counts (uint64, nbins) must
// be zeroed by the caller.
__global__ void __launch_bounds__(256) k_hist_f64(const double* __restrict__ v, long n, int nbins, double lo,
                                                  double width, int logscale, unsigned long long* __restrict__ counts) {
  extern __shared__ uint32_t hs[];
  for (int i = threadIdx.x; i < nbins; i += blockDim.x) hs[i] = 0;
  __syncthreads();
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
  for (long base = blockIdx.x * (long)blockDim.x; base < n; base += (long)gridDim.x * blockDim.x) {
    const long i = base + threadIdx.x;
    int b = -1;
    if (i < n) {
      double x = v[i];
      bool ok = true;
      if (logscale) {
        ok = x > 0;
        x = ok ? log10(x) : 0.0;
      }
      const double hi = lo + width * nbins;
      if (ok && x >= lo && x < hi) {
        b = (int)floor((x - lo) / width);
        b = b < 0 ? 0 : (b >= nbins ? nbins - 1 : b);
      }
    }
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    if (b >= 0 && (peers & lt) == 0) atomicAdd(&hs[b], (uint32_t)__popc(peers));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nbins; i += blockDim.x)
    if (hs[i]) atomicAdd(&counts[i], (unsigned long long)hs[i]);
}

void histogram_f64(mlc_ctx* ctx, long n, const double* v, int nbins, double lo, double hi, int logscale,
                   unsigned long long* counts_dev) {
  MLC_CUDA(cudaMemsetAsync(counts_dev, 0, sizeof(unsigned long long) * nbins, ctx->stream));
  if (n <= 0) return;
  const size_t smem = sizeof(uint32_t) * nbins;
  set_max_smem((const void*)k_hist_f64, smem);
  const int grid = (int)std::min<long>((n + 255) / 256, (long)ctx->sm_count * 8);
  {
    MLC_KSCOPE(ctx, "histogram");
    k_hist_f64<<<grid, 256, smem, ctx->stream>>>(v, n, nbins, lo, (hi - lo) / nbins, logscale, counts_dev);
  }
  MLC_CHECK_LAUNCH();
}

}  // namespace mlc

// ---------------------------------------------------------------- histogram without allocation
//
// For callers that must not allocate device memory: code running while another
// framework has reserved the whole device memory pool for its own allocator, and host
// callbacks and plugins that may only use the buffers they were handed.  The per-bin
// counters live in a fixed file-scope device array instead of the
// context's workspace, so this entry point calls no cudaMalloc, cudaFree or allocating
// library routine.  The array is loaded with the library and stays allocated on every
// device that loads it until the process exits.
namespace mlc {
namespace {

constexpr int kNoAllocMaxBins = 12000;  // 96 KB of uint64 counters per device
static __device__ __align__(256) unsigned long long g_noalloc_hist[kNoAllocMaxBins];

std::mutex g_noalloc_mu;
std::unordered_map<int, void*> g_noalloc_addr;  // device ordinal -> device address of the array

// Device address of the array on the current device, resolved once per device.  In host
// code the symbol is only a host-side stand-in, never a device address.
void* noalloc_counters(int device) {
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  auto it = g_noalloc_addr.find(device);
  if (it != g_noalloc_addr.end()) return it->second;
  void* p = nullptr;
  MLC_CUDA(cudaGetSymbolAddress(&p, g_noalloc_hist));
  g_noalloc_addr[device] = p;
  return p;
}

}  // namespace
}  // namespace mlc

extern "C" int mlc_histogram_f64_noalloc(mlc_ctx* ctx, long n, const double* v, int nbins, double lo, double hi,
                                         int logscale, uint64_t* counts_host) {
  using namespace mlc;
  if (!ctx) return MLC_ERR_ARG;
  if ((n > 0 && !v) || !counts_host || n < 0 || !(hi > lo)) {
    ctx->err = "mlc_histogram_f64_noalloc: null pointer, negative n or hi <= lo";
    return MLC_ERR_ARG;
  }
  if (nbins < 1 || nbins > kNoAllocMaxBins) {
    ctx->err = "mlc_histogram_f64_noalloc: nbins must be in [1, 12000] (fixed counter array)";
    return MLC_ERR_LIMIT;
  }
  try {
    DeviceGuard g(ctx->device);
    unsigned long long* counts = (unsigned long long*)noalloc_counters(ctx->device);
    // the array keeps the previous call's counts: clear the bins this call uses
    MLC_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned long long) * nbins, ctx->stream));
    if (n > 0) {
      const size_t smem = sizeof(uint32_t) * nbins;
      set_max_smem((const void*)k_hist_f64, smem);
      const int grid = (int)std::min<long>((n + 255) / 256, (long)ctx->sm_count * 8);
      {
        MLC_KSCOPE(ctx, "histogram_noalloc");
        k_hist_f64<<<grid, 256, smem, ctx->stream>>>(v, n, nbins, lo, (hi - lo) / nbins, logscale, counts);
      }
      MLC_CHECK_LAUNCH();
    }
    MLC_CUDA(cudaMemcpyAsync(counts_host, counts, sizeof(uint64_t) * nbins, cudaMemcpyDeviceToHost, ctx->stream));
    MLC_CUDA(cudaStreamSynchronize(ctx->stream));
    return MLC_OK;
  } catch (const Error& e) {
    ctx->err = e.what();
    return e.code;
  }
}
