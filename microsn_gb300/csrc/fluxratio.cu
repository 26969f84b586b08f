// Multi-filter flux-ratio likelihood of every pair of simulated locations, replacing
// getChi2GPU / getChi2CPU (chi2/chi2_functions.cuh:93-190):
//
//   chi2[x, y] = 1/2 sum_f sum_t ((f_obs[f,t] - mu1[x,f,t] / mu2[y,f,t]) / df_obs[f,t])^2
//   likelihood = sum over (x, y) of exp(-chi2[x, y])
//
// with the CPU twin's indexing (the reference's kernel reads mu2 at x, so its chi2 never
// depends on y).  The reference runs one thread per (x, y, filter) with a float atomic
// per filter into a managed N^2 array zero-filled on the host, then sums the N^2 exp()
// on one host core.  Here one CTA owns a tile of pairs, its K = F*T values staged through shared
// memory in chunks, and a pair costs two FP32 operations per (filter, time):
//
//   t = o - mu1 B,  acc += t^2,   o = RN(f/df),  B = RN(rho/mu2),  rho = o/f (to twice the precision)
//
// f/df is rounded, but rho follows it, so t = rho (f - mu1/mu2) with the one rounding of B inside
// the difference, as 1/mu2 would have, and a factor rho within 2^-24 of 1/df.  (f = 0: rho =
// RN(1/df).)  Few locations, or an f or df that is not of moderate size, or a B beyond the exponents that
// 1/mu2 still has: t = (f - mu1 RN(1/mu2)) RN(1/df), three operations.
// exp(-chi2) is summed per thread relative to its smallest chi2 (FP32 terms, one FP64-range
// exp per thread), per CTA in FP64, and the CTA sums are added in a fixed order
// (deterministic).  chi2 is stored only when asked for.
//
// Bound by the FP32 pipe: 1.4e10 operations for 10^4 x 10^4 pairs of 70 values, 0.36 ms at the
// measured 39 T/s.  Large N: 128 x 128 pairs per CTA, 8 x 8 per thread (five shared-memory loads
// for 128 operations), the values laid out [k][location] and B formed once by a kernel before,
// the next chunk copied while one is worked on; measured 0.57 ms (4 x 4 per thread, three
// operations, reciprocals formed in every CTA: 1.15 ms).  Few locations: 64 x 64 pairs, which
// fill the SMs from a quarter of the pairs on, and one launch less (at 3000 locations both
// forms take 0.15 ms).
#include <cmath>
#include <vector>

#include "mlc_internal.h"

namespace mlc {

constexpr int FR_TILE = 64;   // locations per tile side, few locations
constexpr int FR_KC = 32;     // (filter, time) values per shared-memory chunk
constexpr int FR_BIG = 128;   // locations per tile side, many
constexpr int FR_BIG_KC = 16;

// Tables of K values each, one after another: o, or f; 1/df; rho high, rho low.
struct FluxTables {
  const float* p;
  int K;
  __device__ __forceinline__ float o(int k) const { return __ldg(p + k); }
  __device__ __forceinline__ float b(int k, float mu2) const {
    const float rh = __ldg(p + 2 * K + k), rl = __ldg(p + 3 * K + k);
    const float q = __fdiv_rn(rh, mu2);
    const float r = fmaf(-q, mu2, rh) + rl;
    return isfinite(q) && q != 0.f && isfinite(r) ? q + r / mu2 : q;
  }
};

// chi2 (halved sums) of a thread's 8 x 8 pairs out, and the sum of their exp(-chi2): column i is
// x = x0 + (i / 4) 64 + i % 4, rows likewise.  FULL: all of them are inside N.
template <bool FULL>
__device__ __forceinline__ double flux_finish(const float (&acc)[8][8], int x0, int y0, int N,
                                              float* __restrict__ chi2) {
  auto at = [](int b, int i) { return b + (i / 4) * 64 + i % 4; };
  const int nx = N - x0, ny = N - y0;
  // as in k_flux_ratio: exp(-cmin) * sum expf(cmin - chi2)
  float amin = INFINITY;
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (FULL || (at(0, i) < nx && at(0, j) < ny)) amin = fminf(amin, acc[j][i]);
  const float cmin = 0.5f * amin;
  const bool vec = (N & 3) == 0;
  float esum = 0.f;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    if (!FULL && at(0, j) >= ny) continue;
    float* row = chi2 ? chi2 + (long)at(y0, j) * N + x0 : nullptr;
#pragma unroll
    for (int g = 0; g < 8; g += 4) {
      float c[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        c[i] = 0.5f * acc[j][g + i];
        if (FULL || at(0, g + i) < nx) esum += expf(cmin - c[i]);
      }
      if (row) {
        float* dst = row + (g / 4) * 64;
        if (vec && (FULL || at(0, g + 3) < nx)) {
          *reinterpret_cast<float4*>(dst) = make_float4(c[0], c[1], c[2], c[3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (FULL || at(0, g + i) < nx) dst[i] = c[i];
        }
      }
    }
  }
  return esum > 0.f ? (cmin < 80.f ? (double)expf(-cmin) : exp(-(double)cmin)) * (double)esum : 0.0;
}

__global__ void __launch_bounds__(256) k_flux_ratio(const float* __restrict__ mu1, const float* __restrict__ mu2,
                                                    const float* __restrict__ obs, const float* __restrict__ sinv,
                                                    int N, int K, float* __restrict__ chi2,
                                                    double* __restrict__ partial) {
  __shared__ __align__(16) float sa[FR_KC][FR_TILE];  // mu1 of the tile's x locations
  __shared__ __align__(16) float sr[FR_KC][FR_TILE];  // 1 / mu2 of the tile's y locations
  __shared__ float so[FR_KC], ss[FR_KC];
  __shared__ double red[8];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int x0 = blockIdx.x * FR_TILE, y0 = blockIdx.y * FR_TILE;
  float acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[j][i] = 0.f;

  for (int k0 = 0; k0 < K; k0 += FR_KC) {
    // stage: 64 locations x 32 values of each image into [k][location] (lanes along the
    // location: conflict-free stores; the 8 values of a 32-byte sector are read by
    // consecutive k steps from L1); padding (k >= K or location >= N) contributes 0
    for (int e = tid; e < FR_TILE * FR_KC; e += 256) {
      const int loc = e % FR_TILE, kk = e / FR_TILE;
      const int k = k0 + kk;
      const bool kin = k < K;
      const int xa = x0 + loc, yb = y0 + loc;
      sa[kk][loc] = (kin && xa < N) ? __ldg(mu1 + (long)xa * K + k) : 0.f;
      sr[kk][loc] = (kin && yb < N) ? 1.0f / __ldg(mu2 + (long)yb * K + k) : 0.f;
    }
    if (tid < FR_KC) {
      const int k = k0 + tid;
      so[tid] = k < K ? __ldg(obs + k) : 0.f;
      ss[tid] = k < K ? __ldg(sinv + k) : 0.f;
    }
    __syncthreads();
    const int kn = min(FR_KC, K - k0);
    for (int kk = 0; kk < kn; kk++) {
      const float4 a = *reinterpret_cast<const float4*>(&sa[kk][tx * 4]);
      const float4 r = *reinterpret_cast<const float4*>(&sr[kk][ty * 4]);
      const float o = so[kk], s = ss[kk];
      const float av[4] = {a.x, a.y, a.z, a.w};
      const float rv[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float d = fmaf(-av[i], rv[j], o) * s;
          acc[j][i] = fmaf(d, d, acc[j][i]);
        }
    }
    __syncthreads();
  }

  // sum of exp(-chi2) over this thread's pairs as exp(-cmin) * sum expf(cmin - chi2): the
  // FP32 terms are in (0, 1] and only those below e^-87 of the largest underflow, and
  // one exp per thread takes the FP64 path when cmin is beyond the FP32 exp range
  float cmin = INFINITY;
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (x0 + tx * 4 + i < N && y0 + ty * 4 + j < N) cmin = fminf(cmin, 0.5f * acc[j][i]);
  float esum = 0.f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int y = y0 + ty * 4 + j;
    float c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      c[i] = 0.5f * acc[j][i];
      const int x = x0 + tx * 4 + i;
      if (x < N && y < N) esum += expf(cmin - c[i]);
    }
    if (chi2 && y < N) {
      const int x = x0 + tx * 4;
      float* dst = chi2 + (long)y * N + x;
      if (x + 3 < N && (((long)y * N + x) & 3) == 0) {
        *reinterpret_cast<float4*>(dst) = make_float4(c[0], c[1], c[2], c[3]);
      } else {
        for (int i = 0; i < 4; i++)
          if (x + i < N) dst[i] = c[i];
      }
    }
  }
  double lsum = 0.0;
  if (esum > 0.f) lsum = (cmin < 80.f ? (double)expf(-cmin) : exp(-(double)cmin)) * (double)esum;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((tid & 31) == 0) red[tid >> 5] = lsum;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; w++) t += red[w];
    partial[blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

// mu1 and B in the order [k][location] with Np locations a row (zeros past N), 32 x 32 values per
// CTA through shared memory.  blockIdx.z: 0 mu1, 1 B.  *beyond is set where a B of an ordinary
// mu2 is near or past the ends of FP32.
__global__ void __launch_bounds__(256) k_flux_layout(const float* __restrict__ mu1, const float* __restrict__ mu2,
                                                     FluxTables tab, int N, int Np, int K, float* __restrict__ a,
                                                     float* __restrict__ b, int* __restrict__ beyond) {
  __shared__ float t[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int l0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const bool side = blockIdx.z != 0;
  const float* src = side ? mu2 : mu1;
  for (int l = w; l < 32; l += 8) {
    const int loc = l0 + l, k = k0 + lane;
    float v = 0.f;
    if (loc < N && k < K) {
      v = __ldg(src + (long)loc * K + k);
      if (side) {
        const float m = v;
        v = tab.b(k, m);
        if (m != 0.f && isfinite(m) && !(fabsf(v) >= 0x1p-110f && fabsf(v) <= 0x1p110f)) *beyond = 1;
      }
    }
    t[l][lane] = v;
  }
  __syncthreads();
  float* dst = side ? b : a;
  for (int q = w; q < 32; q += 8)
    if (k0 + q < K) dst[(long)(k0 + q) * Np + l0 + lane] = t[lane][q];
}

__device__ __forceinline__ void flux_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__global__ void __launch_bounds__(256, 2) k_flux_ratio_big(const float* __restrict__ a, const float* __restrict__ b,
                                                           FluxTables tab, int N, int Np, int K,
                                                           float* __restrict__ chi2, double* __restrict__ partial) {
  __shared__ __align__(16) float sa[2][FR_BIG_KC][FR_BIG];
  __shared__ __align__(16) float sr[2][FR_BIG_KC][FR_BIG];
  __shared__ float so[2][FR_BIG_KC];
  __shared__ double red[8];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int x0 = blockIdx.x * FR_BIG, y0 = blockIdx.y * FR_BIG;
  // chunk c of 16 k's into buffer c & 1: 2 x 16 rows of 32 16-byte words
  auto stage = [&](int c) {
    const int k0 = c * FR_BIG_KC, buf = c & 1;
    for (int e = tid; e < FR_BIG_KC * 32; e += 256) {
      const int kk = e >> 5, q = (e & 31) * 4;
      if (k0 + kk < K) {
        flux_copy16(&sa[buf][kk][q], a + (long)(k0 + kk) * Np + x0 + q);
        flux_copy16(&sr[buf][kk][q], b + (long)(k0 + kk) * Np + y0 + q);
      }
    }
    if (tid < FR_BIG_KC && k0 + tid < K) so[buf][tid] = tab.o(k0 + tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[8][8];
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int i = 0; i < 8; i++) acc[j][i] = 0.f;
  const int nc = (K + FR_BIG_KC - 1) / FR_BIG_KC;
  stage(0);
  for (int c = 0; c < nc; c++) {
    if (c + 1 < nc) {
      stage(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int buf = c & 1, kn = min(FR_BIG_KC, K - c * FR_BIG_KC);
#pragma unroll 2
    for (int kk = 0; kk < kn; kk++) {
      float av[8], rv[8];
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const float4 p = *reinterpret_cast<const float4*>(&sa[buf][kk][tx * 4 + 64 * g]);
        const float4 q = *reinterpret_cast<const float4*>(&sr[buf][kk][ty * 4 + 64 * g]);
        av[4 * g] = p.x, av[4 * g + 1] = p.y, av[4 * g + 2] = p.z, av[4 * g + 3] = p.w;
        rv[4 * g] = q.x, rv[4 * g + 1] = q.y, rv[4 * g + 2] = q.z, rv[4 * g + 3] = q.w;
      }
      const float o = so[buf][kk];
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float d = fmaf(-av[i], rv[j], o);
          acc[j][i] = fmaf(d, d, acc[j][i]);
        }
    }
    __syncthreads();  // the buffer is refilled two chunks on
  }
  double lsum = x0 + FR_BIG <= N && y0 + FR_BIG <= N ? flux_finish<true>(acc, x0 + tx * 4, y0 + ty * 4, N, chi2)
                                                     : flux_finish<false>(acc, x0 + tx * 4, y0 + ty * 4, N, chi2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((tid & 31) == 0) red[tid >> 5] = lsum;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; w++) t += red[w];
    partial[blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

// Fixed-order sum of the per-CTA partial likelihoods.
__global__ void __launch_bounds__(1024) k_sum_partials(const double* __restrict__ p, long n, double* __restrict__ out) {
  __shared__ double red[32];
  double s = 0.0;
  for (long i = threadIdx.x; i < n; i += blockDim.x) s += p[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    *out = t;
  }
}

// One of the two forms; false where a B is beyond the exponents that 1/mu2 still has (big), and the
// results are not to be used.
static bool flux_ratio_run(mlc_ctx* ctx, const float* f_obs_host, const float* df_obs_host, const float* mu1,
                           const float* mu2, int N, int K, float* chi2, double* likelihood_host, bool big) {
  std::vector<float> h(4 * (size_t)K);
  for (int k = 0; k < K; k++) {
    const float f = f_obs_host[k], df = df_obs_host[k];
    h[k] = f;
    h[K + k] = 1.0f / df;
    if (!big) continue;
    h[k] = f / df;
    const double rho = f != 0.f ? (double)h[k] / (double)f : (double)h[K + k];
    h[2 * (size_t)K + k] = (float)rho;
    h[3 * (size_t)K + k] = (float)(rho - (double)(float)rho);
  }
  const int nb = (N + FR_BIG - 1) / FR_BIG, nt = big ? nb : (N + FR_TILE - 1) / FR_TILE;
  const long nblk = (long)nt * nt;
  const size_t hb = round_up((long)(4 * K * sizeof(float)), 256);
  char* ws = (char*)ws_get(ctx, WS_SMALL, hb + (size_t)nblk * sizeof(double) + 256);
  float* d_tab = (float*)ws;
  double* d_part = (double*)(ws + hb);
  struct Result {
    double like;
    int beyond;
  };
  Result* d_res = (Result*)(d_part + nblk);
  MLC_CUDA(cudaMemcpyAsync(d_tab, h.data(), (big ? 4 : 2) * (size_t)K * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
  MLC_CUDA(cudaMemsetAsync(d_res, 0, sizeof(Result), ctx->stream));
  const FluxTables tab{d_tab, K};
  if (big) {
    const int Np = nb * FR_BIG;
    float* da = (float*)ws_get(ctx, WS_SORT_KEYS, 2 * (size_t)K * Np * sizeof(float));
    float* db = da + (size_t)K * Np;
    {
      MLC_KSCOPE(ctx, "flux_layout");
      k_flux_layout<<<dim3(Np / 32, ceil_div(K, 32), 2), 256, 0, ctx->stream>>>(mu1, mu2, tab, N, Np, K, da, db,
                                                                                &d_res->beyond);
    }
    MLC_CHECK_LAUNCH();
    MLC_KSCOPE(ctx, "flux_ratio_chi2");
    k_flux_ratio_big<<<dim3(nt, nt), 256, 0, ctx->stream>>>(da, db, tab, N, Np, K, chi2, d_part);
  } else {
    MLC_KSCOPE(ctx, "flux_ratio_chi2");
    k_flux_ratio<<<dim3(nt, nt), 256, 0, ctx->stream>>>(mu1, mu2, d_tab, d_tab + K, N, K, chi2, d_part);
  }
  MLC_CHECK_LAUNCH();
  {
    MLC_KSCOPE(ctx, "flux_ratio_sum");
    k_sum_partials<<<1, 1024, 0, ctx->stream>>>(d_part, nblk, &d_res->like);
  }
  MLC_CHECK_LAUNCH();
  Result r;
  download(ctx, &r, d_res, sizeof r);
  *likelihood_host = r.like;
  return !r.beyond;
}

void flux_ratio_chi2(mlc_ctx* ctx, const float* f_obs_host, const float* df_obs_host, const float* mu1,
                     const float* mu2, int N, int F, int T, float* chi2, double* likelihood_host) {
  MLC_REQUIRE(N >= 1 && F >= 1 && T >= 1, MLC_ERR_ARG, "need N, F, T >= 1");
  MLC_REQUIRE(N <= 200000, MLC_ERR_LIMIT, "N <= 200000 locations");
  const int K = F * T;
  // 128 x 128 tiles once they fill every SM twice, two operations per term where the scaled values
  // stay in range (f and df within 2^16 of 1; B is looked at where it is formed)
  // and there is room for them (they take as much as mu1 and mu2)
  const int nb = (N + FR_BIG - 1) / FR_BIG;
  bool big = (long)nb * nb >= 2L * 2 * ctx->sm_count;
  auto moderate = [](float v) { return std::isfinite(v) && std::fabs(v) >= 0x1p-16f && std::fabs(v) <= 0x1p16f; };
  for (int k = 0; k < K && big; k++)
    big = moderate(df_obs_host[k]) && (f_obs_host[k] == 0.f || moderate(f_obs_host[k]));
  big = big && ws_try(ctx, WS_SORT_KEYS, 2 * (size_t)K * nb * FR_BIG * sizeof(float));
  if (big && flux_ratio_run(ctx, f_obs_host, df_obs_host, mu1, mu2, N, K, chi2, likelihood_host, true)) return;
  flux_ratio_run(ctx, f_obs_host, df_obs_host, mu1, mu2, N, K, chi2, likelihood_host, false);
}

}  // namespace mlc
