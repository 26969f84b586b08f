// Pair stage in the reference's flux-ratio form (simulating_lcurves/src/gpu_functions.cu:
// setup_integral_GPU :351-401, calculate_chi2_GPU :428-456, bin_chi2_GPU :483-503 and
// kernels kernel_z :643, kernel_chi2 :700, kernel_bin_chi2 :772).
//
// GB300 form: no "offset-squares" launch loop and no __constant__ tables.  The
// interpolated curves mA (Nloc x Njp) and mB are built once in FP64; pair kernels read
// them through L1/L2; the z ranking uses the hand-written radix sort; bin means are a
// parallel segmented reduction; and a fused variant computes each pair's z bin directly
// and accumulates chi2 and exp(-chi2/2) per bin without any Nloc^2 array.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mlc_internal.h"
#include "radix.cuh"

namespace mlc {

void radix_sort_u64_u32(mlc_ctx* ctx, long n, uint64_t* keys, uint32_t* vals);
RangeSort radix_sort_range_u64_u32(mlc_ctx* ctx, long n, uint64_t* keys, uint32_t* vals, const unsigned long long* range);

// The key of the reference's z sort (thrust::stable_sort_by_key on doubles, a radix sort):
// the order of the bit patterns with the sign folded in, -0.0 taken as +0.0 (the radix sort
// keeps the two in pair-index order), and NaN placed by its sign bit -- the GPU's 0/0
// (0xfff8...) and a negative NaN operand before -inf, a positive NaN operand after +inf.
__device__ __forceinline__ uint64_t key_of(double d) {
  uint64_t u = __double_as_longlong(d);
  if (u == 0x8000000000000000ull) u = 0;
  return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

// The double a key stands for (-0.0 comes back as +0.0, equal under comparison).
__device__ __forceinline__ double value_of(uint64_t k) {
  return __longlong_as_double((k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k);
}

// Correctly rounded a / b from y = 1/b as a pair (yh = RN(1/b), yl the rest): q = RN(a yh +
// RN(a yl)) is within one ulp of a/b, its residual a - q b is exact with an FMA, and
// RN(q + r yh) is then the correctly rounded quotient (Markstein's theorem; the first step as
// in Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division
// when the divisor is known in advance", IEEE Trans. Comput. 53, 2004).  Four FP64 operations
// instead of a division's dozen, for operands of moderate exponent (no step over- or
// underflows); others divide.
struct Reciprocal {
  double b, h, l;
  bool plain;
  static __device__ __forceinline__ bool moderate(double v) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    return e > 1023 - 400 && e < 1023 + 400;
  }
  __device__ __forceinline__ explicit Reciprocal(double b_) : b(b_) {
    plain = !moderate(b);
    h = 1.0 / b;
    l = h * __fma_rn(-b, h, 1.0);
  }
  __device__ __forceinline__ double quotient(double a) const {
    if (plain || !moderate(a)) return a / b;
    const double q = __fma_rn(a, h, __dmul_rn(a, l));
    return __fma_rn(__fma_rn(-q, b, a), h, q);
  }
};

// z keys and pair indices for the stable rank sort: a thread per b, Z_ROWS rows a each; and the
// least key and least ~key of all (range).
constexpr int Z_ROWS = 32;
__global__ void __launch_bounds__(256) k_pair_z(const double* __restrict__ LCA, const double* __restrict__ LCB, int Nloc,
                                                int Nprof, uint64_t* __restrict__ keys, uint32_t* __restrict__ idx,
                                                unsigned long long* __restrict__ range) {
  __shared__ unsigned long long least[2];
  if (threadIdx.x < 2) least[threadIdx.x] = ~0ull;
  __syncthreads();
  const int b = blockIdx.x * 256 + threadIdx.x;
  if (b < Nloc) {
    const Reciprocal rb(__ldg(LCB + (long)b * Nprof));
    const int a1 = min(Nloc, (int)(blockIdx.y + 1) * Z_ROWS);
    uint64_t lo = ~0ull, nhi = ~0ull;
    for (int a = blockIdx.y * Z_ROWS; a < a1; a++) {
      const long p = (long)a * Nloc + b;
      const uint64_t k = key_of(rb.quotient(__ldg(LCA + (long)a * Nprof)));
      keys[p] = k;
      idx[p] = (uint32_t)p;
      lo = min(lo, k);
      nhi = min(nhi, ~k);
    }
    atomicMin(&least[0], (unsigned long long)lo);
    atomicMin(&least[1], (unsigned long long)nhi);
  }
  __syncthreads();
  if (threadIdx.x < 2) atomicMin(&range[threadIdx.x], least[threadIdx.x]);
}

// rank[perm[r]] = r
struct LoadOwnIndex {
  __device__ __forceinline__ uint32_t operator()(long i) const { return (uint32_t)i; }
};

// upper_bound of each edge in the sorted z: the reference's binary search
// (thrust::upper_bound, gpu_functions.cu:388) step for step -- the same midpoints and the
// same FP64 comparison edge < z, so that NaN z (never greater than an edge) land where they
// land there: those before -inf count in the first bin, those after +inf in the bins the
// search's path gives them.
__global__ void k_upper_bound(const uint64_t* __restrict__ sorted, long P, const double* __restrict__ edges,
                              int nb, uint32_t* __restrict__ upper) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  const double e = edges[i];
  long lo = 0, hi = P;
  while (lo < hi) {
    const long mid = (lo + hi) >> 1;
    if (e < value_of(sorted[mid])) hi = mid;
    else lo = mid + 1;
  }
  upper[i] = (uint32_t)lo;
}

// m[i*Nloc + a] = LC[a*Nprof + ind_i] + fac_i * DLC[a*(Nprof-1) + ind_i], or 1 (ind_i = -1).
// The B side (rho given): B_i = rho_i / m, rho_i = rho[i] + rho[Njp + i], rounded once: one division
// per (epoch, location) instead of one per pair; and 1 / m in inv.  *plain is set where a B_i
// is beyond the exponents that 1 / m still has (m near the ends of FP64).
__global__ void k_interp(const double* __restrict__ LC, const double* __restrict__ DLC, int Nloc, int Nprof,
                         int Njp, const int* __restrict__ ind, const double* __restrict__ fac,
                         const double* __restrict__ rho, double* __restrict__ m, double* __restrict__ inv,
                         int* __restrict__ plain) {
  const long n = (long)Nloc * Njp;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
    const int i = (int)(q / Nloc), a = (int)(q % Nloc);
    const int k = ind[i];
    double v = (k == -1) ? 1.0 : LC[(long)a * Nprof + k] + fac[i] * DLC[(long)a * (Nprof - 1) + k];
    if (rho) {
      inv[q] = 1.0 / v;
      const double h = rho[i] / v, r = __fma_rn(-h, v, rho[i]) + rho[Njp + i];
      if (v != 0.0 && isfinite(v) && !(fabs(h) >= 0x1p-960 && fabs(h) <= 0x1p960)) *plain = 1;
      // (a quotient that is 0, infinite or NaN has no residual)
      v = isfinite(h) && h != 0.0 && isfinite(r) ? h + r / v : h;
    }
    m[q] = v;
  }
}

// Point-source values of the fused binning: the FP64 values z[a], and FP32 ones of z (side A) or
// 1/z (side B) for the search.
__global__ void k_zvalues(const double* __restrict__ LC, int Nloc, int Nprof, int invert, double* __restrict__ z,
                          float* __restrict__ zf) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < Nloc; q += gridDim.x * blockDim.x) {
    const double v = LC[(long)q * Nprof];
    z[q] = v;
    zf[q] = invert ? (float)(1.0 / v) : (float)v;
  }
}
// chi2 of pair (a, b) = sum_i ((d_i - mA_i/mB_i)/s_i)^2 in FP64.  The kernels that sum it are
// bound by the FP64 pipe (0.63 T operations/s), so each term is two FMAs:
//   t = ds_i - mA_i B_i,  c += t^2,  ds_i = RN(d_i/s_i),  B_i = RN(rho_i / mB_i),  rho_i = ds_i / d_i
// (to twice the precision).  d_i/s_i is rounded, but rho_i follows it, so that t = rho_i (d_i -
// mA_i/mB_i) with the one rounding of B_i inside the difference -- as 1/mB_i's would be -- and
// a factor rho_i within one ulp of 1/s_i.  Where d_i or s_i is zero, not finite or of an extreme
// exponent, or a B_i would be, the terms are (d_i - mA_i RN(1/mB_i)) RN(1/s_i) (*plain).
struct RatioChi2 {
  const double* mA;
  const double* iB;   // B_i
  const double* inv;  // 1 / mB_i
  const double* ds;
  const double* d;
  const double* is;  // 1 / s_i
  const int* plain;
  int Nloc, Njp;
  __device__ __forceinline__ double operator()(int a, int b, bool pl) const {
    const double* A = mA + a;
    double c = 0.0;
    if (!pl) {
      for (int i = 0; i < Njp; i++) {
        const double t = __fma_rn(-__ldg(A + (long)i * Nloc), __ldg(iB + (long)i * Nloc + b), __ldg(ds + i));
        c = __fma_rn(t, t, c);
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < Njp; i++) {
        const double t = __fma_rn(-__ldg(A + (long)i * Nloc), __ldg(inv + (long)i * Nloc + b), __ldg(d + i)) * __ldg(is + i);
        c = __fma_rn(t, t, c);
      }
    }
    return c;
  }
  __device__ __forceinline__ double operator()(long p) const {  // pair index a Nloc + b, below 2^32
    const uint32_t a = (uint32_t)p / (uint32_t)Nloc;
    return (*this)((int)a, (int)((uint32_t)p - a * (uint32_t)Nloc), __ldg(plain) != 0);
  }
};

// One pair per thread, in pair order, or at its rank (a rank beyond the pairs writes nothing).
__global__ void __launch_bounds__(256) k_pair_chi2_ratio(RatioChi2 f, const uint32_t* __restrict__ rank,
                                                         double* __restrict__ chi2) {
  const int b = blockIdx.x * 32 + (threadIdx.x & 31);
  const int a = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (a >= f.Nloc || b >= f.Nloc) return;
  const long p = (long)a * f.Nloc + b;
  const long at = rank ? (long)rank[p] : p;
  if (at < (long)f.Nloc * f.Nloc) chi2[at] = f(a, b, __ldg(f.plain) != 0);
}

// Bin means of the rank-ordered chi2 (bin_chi2_GPU): every bin's slice is cut into pieces
// of at most BIN_PIECE values, one CTA per piece sums chi2 and exp(-chi2/2) over it, and a
// second kernel adds each bin's pieces in order -- a fixed summation order (the result does
// not depend on timing), and a bin of millions of pairs is spread over many CTAs (one CTA
// per bin left most SMs idle behind the largest bins).
//
// exp(-c/2), the FP64 pipe's largest part of this kernel, from a table: exp(-c/2) =
// 2^(k/2048) e^r with k = RN(-c 1024/ln 2) and |r| <= ln 2/4096, where three terms of the
// series for e^r - 1, the fourth folded into the second where it is least off, leave 2^-57;
// 2^(j/2048) for the 2048 fractions lies in shared memory, rounded, with the relative rest.  Eight
// FP64 operations, within 0.53 ulp (the library's within 0.51; 4096 entries without the rest
// were within one ulp); outside [0, 1400] (NaN, results
// near or below the smallest normal) the library's exp, and 0 where that underflows.
constexpr int EXP_TAB = 2048;
__device__ __forceinline__ double exp_neg_half(double c, const double2* tab) {
  // (compared by its high word: FP64 comparisons run on the FP64 pipe, and a negative or NaN c
  // has a larger one)
  const unsigned hi = (unsigned)__double2hiint(c);
  if (hi >= 0x4095E000u) return hi - 0x40977000u < 0x7FF00000u - 0x40977000u ? 0.0 : exp(-0.5 * c);  // 1400; 1500 to below inf
  const double magic = 6755399441055744.0;                   // 1.5 * 2^52: the sum's low word is k
  const double t = __fma_rn(c, -1477.3197218702985, magic);  // 1024 / ln 2
  const double k = __dsub_rn(t, magic);
  double r = __fma_rn(k, 0x1.62e42fe8p-11, c);  // r' = -2 r = c + k ln 2/1024; 30 bits of it: exact
  r = __fma_rn(k, 0x1.e8e7bcd5e4f1ep-41, r);
  const int ki = __double2loint(t);
  // e^r - 1 = r' (-1/2 + r'/8 - r'^2/48 + r'^3/384), r'^4 as 0.828 (ln 2/2048)^2 r'^2
  const double p = __fma_rn(r, __fma_rn(r, -1.0 / 48.0, 0.125 + 0.828427 / 384.0 * (0x1.62e42fefa39efp-12 * 0x1.62e42fefa39efp-12)), -0.5);
  const double2 s = tab[ki & (EXP_TAB - 1)];
  const double e = __fma_rn(s.x, __fma_rn(r, p, s.y), s.x);
  return __hiloint2double(__double2hiint(e) + ((ki >> 11) << 20), __double2loint(e));
}

// 2^(j/2048) on the device, made once per context (and there for any stream it is given later).
static const double2* exp_table(mlc_ctx* ctx) {
  if (!ctx->exp_table) {
    std::vector<double2> h(EXP_TAB);
    for (int j = 0; j < EXP_TAB; j++) {
      const long double v = exp2l((long double)j / EXP_TAB);
      h[j].x = (double)v;
      h[j].y = (double)(v / h[j].x - 1.0L);
    }
    void* d = ws_get(ctx, WS_EXP_TAB, sizeof(double2) * EXP_TAB);
    upload(ctx, d, h.data(), sizeof(double2) * EXP_TAB);
    MLC_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->exp_table = d;
  }
  return (const double2*)ctx->exp_table;
}
__device__ __forceinline__ void load_exp_table(const double2* __restrict__ src, double2* dst) {
  for (int i = threadIdx.x; i < EXP_TAB; i += blockDim.x) dst[i] = __ldg(src + i);
}
constexpr uint32_t BIN_PIECE = 1u << 15;
struct BinPiece {
  uint32_t first, count;
};

__global__ void __launch_bounds__(256) k_bin_piece_sums(const double* __restrict__ chi2,
                                                        const BinPiece* __restrict__ pieces, int npieces,
                                                        const double2* __restrict__ etab, double* __restrict__ psum,
                                                        double* __restrict__ pexp) {
  __shared__ double2 tab[EXP_TAB];
  __shared__ double r1[8], r2[8];
  load_exp_table(etab, tab);
  __syncthreads();
  for (int pi = blockIdx.x; pi < npieces; pi += gridDim.x) {  // (one table for many pieces)
    const BinPiece pc = pieces[pi];
    double sc = 0.0, se = 0.0;
#pragma unroll 4
    for (uint32_t k = threadIdx.x; k < pc.count; k += blockDim.x) {
      const double c = chi2[(long)pc.first + k];
      sc += c;
      se += exp_neg_half(c, tab);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sc += __shfl_xor_sync(0xffffffffu, sc, o);
      se += __shfl_xor_sync(0xffffffffu, se, o);
    }
    if ((threadIdx.x & 31) == 0) {
      r1[threadIdx.x >> 5] = sc;
      r2[threadIdx.x >> 5] = se;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        a += r1[w];
        b += r2[w];
      }
      psum[pi] = a;
      pexp[pi] = b;
    }
    __syncthreads();  // r1, r2 are rewritten by the next piece
  }
}

// Per bin: the sum of its pieces [pfirst[bin], pfirst[bin + 1]) over its count; an empty bin
// gets the reference's values (chi2 2000, exp(-1000)).
__global__ void k_bin_combine(const uint32_t* __restrict__ pfirst, const uint32_t* __restrict__ nper,
                              const double* __restrict__ psum, const double* __restrict__ pexp, int nb,
                              double* __restrict__ bchi2, double* __restrict__ bexp) {
  const int bin = blockIdx.x * blockDim.x + threadIdx.x;
  if (bin >= nb) return;
  const uint32_t n = nper[bin];
  if (n == 0) {
    bexp[bin] = exp(-2000.0 / 2.0);
    bchi2[bin] = 2000.0;
    return;
  }
  double a = 0.0, b = 0.0;
  for (uint32_t q = pfirst[bin]; q < pfirst[bin + 1]; q++) {
    a += psum[q];
    b += pexp[q];
  }
  bexp[bin] = b / n;
  bchi2[bin] = a / n;
}

// Fused rank-free pair binning.  Bin of z = LCA_a / LCB_b: smallest i with z <= edge_i,
// z above the last edge dropped.  The search runs on float copies (z32 = zA_a * zB_b within
// 1.8e-7 of z, float edges within 6e-8 of the edges): when z32 is more than 2^-20 z32
// away from both neighbouring float edges the float order is the FP64 order; otherwise
// (and for zero, non-finite or extreme z32) the exact FP64 quotient is searched in the
// FP64 edges.
//
// A thread goes through na places a of its b and keeps the sums of its present bin in registers;
// when the bin changes they go to the bin's accumulators in global memory: an add there costs
// the SM no FP64 operation, where an FP64 add to shared memory is a compare-and-swap loop of
// them.  There are up to 1024 copies of the accumulators, so that each sums a thousand
// values or so (the rounding of one running sum of all 10^6 pairs of a bin would show), and
// k_fused_combine adds the copies up in pairs.  (With the accumulators there, having both
// sides sorted, so that bins change once in tens of pairs, measures the same.)  The next pair's
// bin is the last one's while z32 is clear of that bin's two edges.  What is left is the FP64
// pipe: 2 Njp operations for chi2, 8 for the exponential, 2 for the sums (9216 locations,
// Njp = 5: 6.24 -> 3.56 ms; the pipe needs 2.7).  A CTA: 256 b x na (at most FUSED_A) a.
constexpr int FUSED_A = 64;
struct FusedSide {
  const double* z;
  const float* zf;
};
__device__ __forceinline__ int edge_search(const double* e, int nb, double z) {
  int lo = 0, hi = nb;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (e[mid] < z) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(256) k_pair_bin_fused(RatioChi2 f, FusedSide A, FusedSide B, int na, int nb,
                                                        const double* __restrict__ edges,
                                                        const double2* __restrict__ etab, int copies,
                                                        double* __restrict__ gsum, double* __restrict__ gexp,
                                                        unsigned long long* __restrict__ gcnt) {
  extern __shared__ __align__(16) double sm[];
  double2* tab = reinterpret_cast<double2*>(sm);
  float* ef_s = reinterpret_cast<float*>(tab + EXP_TAB);
  load_exp_table(etab, tab);
  for (int i = threadIdx.x; i < nb; i += blockDim.x) ef_s[i] = (float)edges[i];
  __syncthreads();
  const long copy = (long)((blockIdx.y * gridDim.x + blockIdx.x) % copies) * nb;
  auto flush = [&](int bin, double sc, double se, unsigned cn) {
    atomicAdd(gsum + copy + bin, sc);
    atomicAdd(gexp + copy + bin, se);
    atomicAdd(gcnt + copy + bin, (unsigned long long)cn);
  };
  const bool plain = __ldg(f.plain) != 0;
  const int b = blockIdx.x * 256 + threadIdx.x;
  if (b < f.Nloc) {
    const float zb = __ldg(B.zf + b);
    const int a0 = blockIdx.y * na, a1 = min(a0 + na, f.Nloc);
    int bin = -1;                   // bin of the sums below
    float below = 0.f, above = 0.f;  // z32 strictly between them: certainly this bin
    double sc = 0.0, se = 0.0;
    unsigned cn = 0;
    for (int a = a0; a < a1; a++) {
      const float z32 = __ldg(A.zf + a) * zb;
      if (!(z32 > below && z32 < above)) {
        int lo = 0, hi = nb;  // first float edge >= z32
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (ef_s[mid] < z32) lo = mid + 1;
          else hi = mid;
        }
        bool exact = !(z32 > 0x1p-100f && z32 < 0x1p100f);
        if (!exact) {
          const float tol = z32 * 0x1p-20f;
          exact = (lo < nb && ef_s[lo] - z32 <= tol) || (lo > 0 && z32 - ef_s[lo - 1] <= tol);
        }
        if (exact) {
          // NaN: the rank order puts a negative one (the GPU's 0/0) before every z, in the
          // first bin, and a positive one (from a NaN light-curve value) after +inf, counted
          // here in no bin
          const double z = __ldg(A.z + a) / __ldg(B.z + b);
          if (z != z) lo = signbit(z) ? 0 : nb;
          else lo = edge_search(edges, nb, z);
        }
        if (lo != bin) {
          if (cn) flush(bin, sc, se, cn);
          bin = lo;
          sc = se = 0.0;
          cn = 0;
        }
        // the bin's float edges, moved in by twice the tolerance (an empty interval where that
        // leaves nothing, or beyond the exponents the float search answers for)
        below = bin > 0 ? ef_s[bin - 1] * (1.f + 0x1p-19f) : 0x1p-100f;
        above = bin < nb ? ef_s[bin] * (1.f - 0x1p-19f) : 0x1p100f;
        below = fmaxf(below, 0x1p-100f);
        above = fminf(above, 0x1p100f);
      }
      if (bin >= nb) continue;
      const double c = f(a, b, plain);
      sc += c;
      se += exp_neg_half(c, tab);
      cn++;
    }
    // what the threads hold at the end: neighbours mostly hold the same bin
    const unsigned act = __activemask();
    int same = 0;
    __match_all_sync(act, bin, &same);
    if (same && act == 0xffffffffu) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sc += __shfl_xor_sync(0xffffffffu, sc, o);
        se += __shfl_xor_sync(0xffffffffu, se, o);
        cn += __shfl_xor_sync(0xffffffffu, cn, o);
      }
      if (threadIdx.x & 31) cn = 0;
    }
    if (cn) flush(bin, sc, se, cn);
  }
}

// The copies' sums: a warp per bin, each lane the copies 32 apart, then the lanes in pairs.
__global__ void __launch_bounds__(256) k_fused_combine(int nb, int copies, double* __restrict__ gsum,
                                                       double* __restrict__ gexp,
                                                       unsigned long long* __restrict__ gcnt) {
  const int i = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= nb) return;
  double s = 0.0, e = 0.0;
  unsigned long long n = 0;
  for (int c = lane; c < copies; c += 32) {
    const long q = (long)c * nb + i;
    s += gsum[q];
    e += gexp[q];
    n += gcnt[q];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if (lane == 0) {
    gsum[i] = s;
    gexp[i] = e;
    gcnt[i] = n;
  }
}

// ---------------------------------------------------------------- host entry helpers

static int grid_for(mlc_ctx* ctx, long n) {
  return (int)std::max<long>(1, std::min<long>((n + 255) / 256, (long)ctx->sm_count * 16));
}

constexpr long RANGE_SORT_FROM = 1l << 20;  // (fewer keys are bound by the launches of either form)

void pair_setup(mlc_ctx* ctx, int Nloc, int Nprof, const double* LCA, const double* LCB, int Nbins,
                const double* edges_host, uint32_t* rank, uint32_t* lower_host, uint32_t* nper_host) {
  const long P = (long)Nloc * Nloc;
  MLC_REQUIRE(P <= 0xFFFFFFFFl, MLC_ERR_LIMIT, "Nloc^2 above 2^32-1");
  uint64_t* keys = (uint64_t*)ws_get(ctx, WS_PAIR_ACC, sizeof(uint64_t) * P + sizeof(uint32_t) * P + 4096);
  uint32_t* idx = reinterpret_cast<uint32_t*>(keys + P);
  unsigned long long* range = reinterpret_cast<unsigned long long*>(keys + P + (P + 1) / 2);
  auto make_keys = [&] {
    MLC_CUDA(cudaMemsetAsync(range, 0xff, 2 * sizeof(*range), ctx->stream));
    {
      MLC_KSCOPE(ctx, "pair_z");
      k_pair_z<<<dim3(ceil_div(Nloc, 256), ceil_div(Nloc, Z_ROWS)), 256, 0, ctx->stream>>>(LCA, LCB, Nloc, Nprof, keys,
                                                                                         idx, range);
    }
    MLC_CHECK_LAUNCH();
  };
  make_keys();
  // by the top of the keys' range where the keys are many and that decides their order (8.5e7: 3.7
  // ms, by all bits 7.7); outliers, infinities or NaN may stretch the range: then by all bits
  const RangeSort done = P < RANGE_SORT_FROM ? RangeSort::UNTOUCHED : radix_sort_range_u64_u32(ctx, P, keys, idx, range);
  if (done == RangeSort::LOST) make_keys();
  if (done != RangeSort::DONE) radix_sort_u64_u32(ctx, P, keys, idx);
  if (rank) put_by_index(ctx, "pair_rank", idx, LoadOwnIndex{}, P, rank);
  if (Nbins > 0) {
    double* dedge = (double*)ws_get(ctx, WS_SMALL, sizeof(double) * Nbins + sizeof(uint32_t) * Nbins);
    uint32_t* dup = reinterpret_cast<uint32_t*>(dedge + Nbins);
    MLC_CUDA(cudaMemcpyAsync(dedge, edges_host, sizeof(double) * Nbins, cudaMemcpyHostToDevice, ctx->stream));
    {
      MLC_KSCOPE(ctx, "pair_upper_bound");
      k_upper_bound<<<ceil_div(Nbins, 256), 256, 0, ctx->stream>>>(keys, P, dedge, Nbins, dup);
    }
    MLC_CHECK_LAUNCH();
    std::vector<uint32_t> up(Nbins);
    MLC_CUDA(cudaMemcpyAsync(up.data(), dup, sizeof(uint32_t) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
    MLC_CUDA(cudaStreamSynchronize(ctx->stream));
    // lower_ind[0] = 0, lower_ind[i] = upper[i-1]; n_per_bin = adjacent difference of upper
    for (int i = 0; i < Nbins; i++) {
      lower_host[i] = i ? up[i - 1] : 0u;
      nper_host[i] = i ? up[i] - up[i - 1] : up[0];
    }
  }
}

static bool moderate_host(double v) {
  int e = 0;
  return std::isfinite(v) && v != 0.0 && (std::frexp(v, &e), e > -400 && e < 400);
}

static RatioChi2 build_interp(mlc_ctx* ctx, int Njp, const int* indA, const int* indB, const double* facA,
                           const double* facB, const double* d, const double* s, int Nloc, int Nprof,
                           const double* LCA, const double* DLCA, const double* LCB, const double* DLCB) {
  const long n = (long)Nloc * Njp;
  for (int i = 0; i < Njp; i++) {
    MLC_REQUIRE(indA[i] >= -1 && indA[i] < Nprof - 1 && indB[i] >= -1 && indB[i] < Nprof - 1, MLC_ERR_ARG,
                "interpolation index out of the profile range");
  }
  // small tables: fac A/B, ds, d, 1/s, rho (two rows); ind A/B, plain (int)
  const size_t nd = 7 * (size_t)Njp, ni = 2 * (size_t)Njp + 1;
  char* sm = (char*)ws_get(ctx, WS_LOC, sizeof(double) * (3 * n + nd) + sizeof(int) * ni + 64);
  double* mA = (double*)sm;
  double* iB = mA + n;
  double* inv = iB + n;
  double* fA = inv + n;
  double* fB = fA + Njp;
  double* rho = fB + 4 * Njp;
  int* iA = reinterpret_cast<int*>(fA + nd);
  int* iBx = iA + Njp;
  int* plain = iBx + Njp;
  bool pl = false;
  for (int i = 0; i < Njp; i++) pl |= !moderate_host(d[i]) || !moderate_host(s[i]);
  std::vector<char> h(sizeof(double) * nd + sizeof(int) * ni);
  double* hd = reinterpret_cast<double*>(h.data());
  std::copy(facA, facA + Njp, hd);
  std::copy(facB, facB + Njp, hd + Njp);
  for (int i = 0; i < Njp; i++) {
    const double ds = d[i] / s[i];
    hd[2 * Njp + i] = ds;
    hd[3 * Njp + i] = d[i];
    hd[4 * Njp + i] = 1.0 / s[i];
    // rho = ds / d to twice the precision: its rounding, then the exact residual over d
    const double rh = pl ? 1.0 : ds / d[i];
    hd[5 * Njp + i] = rh;
    hd[6 * Njp + i] = pl ? 0.0 : std::fma(-rh, d[i], ds) / d[i];
  }
  int* hi = reinterpret_cast<int*>(hd + nd);
  std::copy(indA, indA + Njp, hi);
  std::copy(indB, indB + Njp, hi + Njp);
  hi[2 * Njp] = pl;
  upload(ctx, fA, h.data(), h.size());
  if (n > 0) {
    {
      MLC_KSCOPE(ctx, "pair_interp");
      k_interp<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(LCA, DLCA, Nloc, Nprof, Njp, iA, fA, nullptr, mA, nullptr,
                                                          nullptr);
    }
    MLC_CHECK_LAUNCH();
    {
      MLC_KSCOPE(ctx, "pair_interp");
      k_interp<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(LCB, DLCB, Nloc, Nprof, Njp, iBx, fB, rho, iB, inv, plain);
    }
    MLC_CHECK_LAUNCH();
  }
  return RatioChi2{mA, iB, inv, fB + Njp, fB + 2 * Njp, fB + 3 * Njp, plain, Nloc, Njp};
}

// Writes in rank order go through bins where the pairs are many and their terms few: the bins save
// what scattered stores cost beyond L2, but form chi2 in the order of a flat index, where a pair's
// operands are not shared by its neighbours.  5600, 9216 locations, bins and 32 x 8 tiles of
// pairs: 5 terms 0.99 and 0.99 ms, 2.79 and 3.15; 6 terms 1.21 and 1.00, 3.30 and 3.16; 12 terms 1.69
// and 1.23, 4.57 and 3.53.
constexpr int BINNED_TERMS = 5;

void pair_chi2_ratio(mlc_ctx* ctx, int Njp, const int* indA, const int* indB, const double* facA,
                     const double* facB, const double* d, const double* s, int Nloc, int Nprof, const double* LCA,
                     const double* DLCA, const double* LCB, const double* DLCB, const uint32_t* rank, double* chi2) {
  if (Nloc <= 0) return;
  const RatioChi2 f = build_interp(ctx, Njp, indA, indB, facA, facB, d, s, Nloc, Nprof, LCA, DLCA, LCB, DLCB);
  const long P = (long)Nloc * Nloc;
  if (rank && Njp <= BINNED_TERMS && P >= BINNED_PUT_FROM && P <= 0xFFFFFFFFl) {
    put_by_index(ctx, "pair_chi2_ratio", rank, f, P, chi2);
    return;
  }
  {
    MLC_KSCOPE(ctx, "pair_chi2_ratio");
    k_pair_chi2_ratio<<<dim3(ceil_div(Nloc, 32), ceil_div(Nloc, 8)), 256, 0, ctx->stream>>>(f, rank, chi2);
  }
  MLC_CHECK_LAUNCH();
}

void bin_chi2(mlc_ctx* ctx, int Nbins, const uint32_t* lower_host, const uint32_t* nper_host,
              const double* chi2_sorted, double* bchi2_host, double* bexp_host) {
  if (Nbins <= 0) return;
  std::vector<BinPiece> pieces;
  std::vector<uint32_t> pfirst(Nbins + 1), nper(nper_host, nper_host + Nbins);
  for (int b = 0; b < Nbins; b++) {
    pfirst[b] = (uint32_t)pieces.size();
    for (uint32_t k = 0; k < nper_host[b]; k += BIN_PIECE)
      pieces.push_back(BinPiece{lower_host[b] + k, std::min(BIN_PIECE, nper_host[b] - k)});
  }
  pfirst[Nbins] = (uint32_t)pieces.size();
  const size_t np = std::max<size_t>(pieces.size(), 1);
  char* sm = (char*)ws_get(ctx, WS_SMALL, sizeof(double) * (2 * Nbins + 2 * np) + sizeof(BinPiece) * np +
                                              sizeof(uint32_t) * (2 * Nbins + 1) + 256);
  double* bc = (double*)sm;
  double* be = bc + Nbins;
  double* ps = be + Nbins;
  double* pe = ps + np;
  BinPiece* dp = reinterpret_cast<BinPiece*>(pe + np);
  uint32_t* dfirst = reinterpret_cast<uint32_t*>(dp + np);
  uint32_t* dn = dfirst + Nbins + 1;
  if (!pieces.empty())
    MLC_CUDA(cudaMemcpyAsync(dp, pieces.data(), sizeof(BinPiece) * pieces.size(), cudaMemcpyHostToDevice, ctx->stream));
  MLC_CUDA(cudaMemcpyAsync(dfirst, pfirst.data(), sizeof(uint32_t) * (Nbins + 1), cudaMemcpyHostToDevice, ctx->stream));
  MLC_CUDA(cudaMemcpyAsync(dn, nper.data(), sizeof(uint32_t) * Nbins, cudaMemcpyHostToDevice, ctx->stream));
  const double2* etab = exp_table(ctx);
  if (!pieces.empty()) {
    MLC_KSCOPE(ctx, "pair_bin_means");
    const unsigned grid = (unsigned)std::min<size_t>(pieces.size(), (size_t)ctx->sm_count * 6);
    k_bin_piece_sums<<<grid, 256, 0, ctx->stream>>>(chi2_sorted, dp, (int)pieces.size(), etab, ps, pe);
  }
  MLC_CHECK_LAUNCH();
  {
    MLC_KSCOPE(ctx, "pair_bin_combine");
    k_bin_combine<<<ceil_div(Nbins, 128), 128, 0, ctx->stream>>>(dfirst, dn, ps, pe, Nbins, bc, be);
  }
  MLC_CHECK_LAUNCH();
  MLC_CUDA(cudaMemcpyAsync(bchi2_host, bc, sizeof(double) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaMemcpyAsync(bexp_host, be, sizeof(double) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));  // (also keeps the host vectors alive for the copies)
}

void pair_bin_fused(mlc_ctx* ctx, int Njp, const int* indA, const int* indB, const double* facA,
                    const double* facB, const double* d, const double* s, int Nloc, int Nprof, const double* LCA,
                    const double* DLCA, const double* LCB, const double* DLCB, int Nbins, const double* edges_host,
                    double* bchi2_host, double* bexp_host, uint32_t* nper_host) {
  MLC_REQUIRE(Nbins > 0 && Nbins <= 6000, MLC_ERR_LIMIT, "fused pair binning supports 1..6000 bins");
  // edges, sums, counts; both sides' FP64 and FP32 point-source values
  // A places per CTA: as many as leave four CTAs for every SM
  const int cols = ceil_div(Nloc, 256);
  const int na = (int)std::max<long>(4, std::min<long>(FUSED_A, (long)Nloc * cols / (4 * ctx->sm_count)));
  const dim3 grid(cols, ceil_div(Nloc, na));
  // (no more copies than CTAs: 10 locations spent 20 us on adding up 1024 of them)
  const int copies = (int)std::max<long>(1, std::min<long>(std::max(16, std::min(1024, (1 << 19) / Nbins)), (long)grid.x * grid.y));
  const size_t N = (size_t)Nloc, NC = (size_t)copies * Nbins;
  char* sm = (char*)ws_get(ctx, WS_PAIR_ACC, 8 * (3 * NC + Nbins) + 2 * (8 + 4) * N + 512);
  double* de = (double*)sm;
  double* gs = de + Nbins;
  double* ge = gs + NC;
  unsigned long long* gc = reinterpret_cast<unsigned long long*>(ge + NC);
  double* z = reinterpret_cast<double*>(gc + NC);
  float* zf = reinterpret_cast<float*>(z + 2 * N);
  if (Nloc > 0) {
    MLC_KSCOPE(ctx, "pair_interp");
    k_zvalues<<<grid_for(ctx, Nloc), 256, 0, ctx->stream>>>(LCA, Nloc, Nprof, 0, z, zf);
    k_zvalues<<<grid_for(ctx, Nloc), 256, 0, ctx->stream>>>(LCB, Nloc, Nprof, 1, z + N, zf + N);
  }
  MLC_CHECK_LAUNCH();
  const RatioChi2 f = build_interp(ctx, Njp, indA, indB, facA, facB, d, s, Nloc, Nprof, LCA, DLCA, LCB, DLCB);
  MLC_CUDA(cudaMemcpyAsync(de, edges_host, sizeof(double) * Nbins, cudaMemcpyHostToDevice, ctx->stream));
  MLC_CUDA(cudaMemsetAsync(gs, 0, 8 * 3 * NC, ctx->stream));
  const size_t smem = sizeof(double2) * EXP_TAB + sizeof(float) * Nbins;
  const double2* etab = exp_table(ctx);
  if (Nloc > 0) {
    set_max_smem((const void*)k_pair_bin_fused, smem);
    const FusedSide A{z, zf}, B{z + N, zf + N};
    {
      MLC_KSCOPE(ctx, "pair_bin_fused");
      k_pair_bin_fused<<<grid, 256, smem, ctx->stream>>>(f, A, B, na, Nbins, de, etab, copies, gs, ge, gc);
    }
    MLC_CHECK_LAUNCH();
    MLC_KSCOPE(ctx, "pair_bin_combine");
    k_fused_combine<<<ceil_div(Nbins, 8), 256, 0, ctx->stream>>>(Nbins, copies, gs, ge, gc);
  }
  MLC_CHECK_LAUNCH();
  std::vector<double> hs(Nbins), he(Nbins);
  std::vector<unsigned long long> hc(Nbins);
  MLC_CUDA(cudaMemcpyAsync(hs.data(), gs, sizeof(double) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaMemcpyAsync(he.data(), ge, sizeof(double) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaMemcpyAsync(hc.data(), gc, sizeof(unsigned long long) * Nbins, cudaMemcpyDeviceToHost, ctx->stream));
  MLC_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int i = 0; i < Nbins; i++) {
    if (hc[i]) {
      bchi2_host[i] = hs[i] / (double)hc[i];
      bexp_host[i] = he[i] / (double)hc[i];
    } else {
      bchi2_host[i] = 2000.0;
      bexp_host[i] = std::exp(-2000.0 / 2.0);
    }
    if (nper_host) nper_host[i] = (uint32_t)hc[i];
  }
}

}  // namespace mlc
