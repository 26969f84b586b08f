// Transforms by radices chosen at run time (AnyLevels): the places of their points in shared
// memory, and how many threads run them.
#pragma once

#include <algorithm>

#include "fft_impl.cuh"

namespace mlc {

__device__ __forceinline__ int any_div(int x, int d, uint32_t magic) { return d == 1 ? x : (int)__umulhi((uint32_t)x, magic); }

// Place of sub-block `blk` of level i: its digits over r[0 .. i-1], the last one fastest.
__device__ __forceinline__ int any_outer(const AnyLevels& lv, int i, int blk) {
  int p = 0;
  for (int j = i - 1; j >= 0; j--) {
    const int q = any_div(blk, lv.r[j], lv.mr[j]);
    p += (blk - q * lv.r[j]) * lv.tn[j];
    blk = q;
  }
  return p;
}
// Place of point m of a block of level i (level i = 0: of the whole transform).
__device__ __forceinline__ int any_inner(const AnyLevels& lv, int i, int m) {
  int p = 0;
  for (int j = i; j < lv.n - 1; j++) {
    const int q = any_div(m, lv.bn[j], lv.mbn[j]);
    p += q * lv.tn[j];
    m -= q * lv.bn[j];
  }
  return p + m;
}
// Place of output k: output digit j (radix r[j], digit 0 fastest) is the place's digit j.
__device__ __forceinline__ int any_output(const AnyLevels& lv, int k) {
  int p = 0;
  for (int j = 0; j < lv.n; j++) {
    const int q = any_div(k, lv.r[j], lv.mr[j]);
    p += (k - q * lv.r[j]) * lv.tn[j];
    k = q;
  }
  return p;
}

// f(integral_constant<R>) for the radix r, 2 to 10.
template <typename F>
__device__ __forceinline__ void any_radix(int r, F f) {
  switch (r) {
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    default: f(std::integral_constant<int, 2>{}); break;
  }
}

constexpr size_t ANY_SMEM = 224 * 1024;  // (and static arrays beside it)

// Threads of a row's CTA: the fewest turns of a level's items over the CTAs that an SM holds at
// once, by its registers (resident threads), shared memory and the rows there are.
static inline int any_row_threads(mlc_ctx* ctx, const AnyLevels& lv, size_t smem, int nrows, int resident) {
  const int fit = std::max(1, std::min((int)(ANY_SMEM / (smem + 1024)), ceil_div(nrows, ctx->sm_count)));
  int best = 0;
  float least = 0.f;
  for (int nt = 64; nt <= 512; nt += 32) {
    int turns = 0;
    for (int i = 0; i < lv.n; i++) turns += ceil_div(lv.L / lv.r[i], nt) * lv.r[i];
    const float cost = (float)turns / std::min(fit, resident / nt);
    if (!best || cost < least) best = nt, least = cost;
  }
  return best;
}
// Threads of a column strip's CTA: the number that leaves the fewest idle ones over the levels.
static inline int any_col_threads(const AnyLevels& lv, int cw, int max) {
  int best = 0;
  long least = 0;
  for (int nt = 64; nt <= max; nt += 32) {
    long cost = 0;
    for (int i = 0; i < lv.n; i++) cost += (long)ceil_div(lv.L / lv.r[i] * cw, nt) * nt * lv.r[i];
    if (!best || cost <= least) best = nt, least = cost;
  }
  return best;
}

}  // namespace mlc
