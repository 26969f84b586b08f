// Fixed-grid sums of three FP32 numbers ("limbs") for FP64 transforms.
//
// GB300 issues FP32 about sixty times faster than FP64 (measured: 39 against 0.63 T
// operations/s), and a Fourier transform is mostly additions.  A sum of floating parts needs
// two-sums (8 FP32 operations each), because the rounding error of the high parts has to be
// recovered where the exponents of the operands are not known.  Here every value of one
// transform is first scaled by one power of two so that |x| < 1, and its high limbs are
// multiples of fixed grids: h of 2^-22, m of 2^-39, and l the rest, about 62 bits.  High limbs
// then add exactly in a single FP32 addition, and a sum costs one addition per limb.
//
// Why |x| < 1 holds throughout a transform: the scale comes from S, the sum of |re| + |im|
// over all of its inputs, and every intermediate value of an FFT is a sum of distinct inputs
// times factors of modulus one, so its modulus is at most S -- whatever the inputs.
//
// An operation's error is absolute, about 2^-62 of the scale, and S is far above the values of a
// long transform until its last levels: rows of 5000 points under the scale of S throughout
// kept 2^-47.7 of their rms (forward) and 2^-49.4 (back), where FP64 keeps 2^-51.8.  The rows
// therefore start under a scale from their largest input and go over to a larger one from
// level to level, as far as the radices since then can have made the values grow (LimbGrow):
// 2^-52.7 and 2^-51.7.  Columns, of 128 points or so, gain nothing from that.
// (Two limbs, 46 bits, in place of float-float lost the faint pixels of FP32 maps: 2^-30 of
// the map's rms at 10000^2.)
//
// Products return to the grid with the additive constant 3 = 1.5 * 2: t = 3 + x c is
// rounded to 2^-22 (t lies in [2, 4)), t - 3 is the high limb, and fma(x, c, -(t - 3)) is the
// rest, exactly.  The same with 1.5 * 2^-16 for the second limb.  All operations are
// explicitly rounded intrinsics: nothing may be contracted or reassociated.
#pragma once

#include "mlc_common.cuh"

namespace mlc {

constexpr float LIMB_G1 = 3.0f;         // 1.5 * 2: rounds to multiples of 2^-22
constexpr float LIMB_G2 = 0x1.8p-16f;   // rounds to multiples of 2^-39
constexpr float LIMB_G3 = 0x1.8p-39f;   // rounds to multiples of 2^-62

// A constant's high limb is cut to multiples of 2^-24, so that its product with a value's
// high limb leaves an exact remainder.
__host__ __device__ constexpr double limb_cut24(double d) {
  return (double)(long long)(d * 16777216.0 + (d < 0 ? -0.5 : 0.5)) / 16777216.0;
}

struct lf3 {
  float h, m, l;
  lf3() = default;
  __host__ __device__ constexpr lf3(float h_, float m_, float l_) : h(h_), m(m_), l(l_) {}
  __host__ __device__ constexpr lf3(double d)
      : h((float)limb_cut24(d)),
        m((float)(d - limb_cut24(d))),
        l((float)((d - limb_cut24(d)) - (double)(float)(d - limb_cut24(d)))) {}
};

template <>
struct C2<lf3> {
  lf3 x, y;
};

// ---------------------------------------------------------------- lf3

__device__ __forceinline__ lf3 operator+(lf3 a, lf3 b) {
  return lf3(__fadd_rn(a.h, b.h), __fadd_rn(a.m, b.m), __fadd_rn(a.l, b.l));
}
__device__ __forceinline__ lf3 operator-(lf3 a, lf3 b) {
  return lf3(__fsub_rn(a.h, b.h), __fsub_rn(a.m, b.m), __fsub_rn(a.l, b.l));
}
__device__ __forceinline__ lf3 operator-(lf3 a) { return lf3(-a.h, -a.m, -a.l); }
__device__ __forceinline__ lf3 operator*(lf3 a, lf3 b) {
  const float h = __fsub_rn(__fmaf_rn(a.h, b.h, LIMB_G1), LIMB_G1);
  const float r = __fmaf_rn(a.h, b.h, -h);  // a multiple of 2^-46 below 2^-22: exact
  const float u0 = __fadd_rn(r, LIMB_G2), u1 = __fmaf_rn(a.h, b.m, u0), u2 = __fmaf_rn(a.m, b.h, u1);
  float e = __fsub_rn(r, __fsub_rn(u0, LIMB_G2));
  float f = __fmaf_rn(a.h, b.m, -__fsub_rn(u1, u0));
  f = __fadd_rn(f, __fmaf_rn(a.m, b.h, -__fsub_rn(u2, u1)));
  e = __fmaf_rn(a.h, b.l, e);
  f = __fmaf_rn(a.l, b.h, f);
  e = __fmaf_rn(a.m, b.m, e);
  return lf3(h, __fsub_rn(u2, LIMB_G2), __fadd_rn(e, f));
}
// c x + d y (34 operations).  NORM carries the lower limbs' excess upwards (6 more): between
// two carries a limb may gather up to 2^7 of its own grid steps, the exact range of an FP32
// addition, so every twiddle product carries and the additions between them do not.
template <bool NORM>
__device__ __forceinline__ lf3 limb_lin2(lf3 c, lf3 x, lf3 d, lf3 y) {
  const float t1 = __fmaf_rn(c.h, x.h, LIMB_G1), t2 = __fmaf_rn(d.h, y.h, t1);
  const float r = __fadd_rn(__fmaf_rn(c.h, x.h, -__fsub_rn(t1, LIMB_G1)), __fmaf_rn(d.h, y.h, -__fsub_rn(t2, t1)));
  const float u0 = __fadd_rn(r, LIMB_G2), u1 = __fmaf_rn(c.m, x.h, u0), u2 = __fmaf_rn(c.h, x.m, u1);
  const float u3 = __fmaf_rn(d.m, y.h, u2), u4 = __fmaf_rn(d.h, y.m, u3);
  float e = __fsub_rn(r, __fsub_rn(u0, LIMB_G2));
  float f = __fmaf_rn(c.m, x.h, -__fsub_rn(u1, u0));
  e = __fadd_rn(e, __fmaf_rn(c.h, x.m, -__fsub_rn(u2, u1)));
  f = __fadd_rn(f, __fmaf_rn(d.m, y.h, -__fsub_rn(u3, u2)));
  e = __fadd_rn(e, __fmaf_rn(d.h, y.m, -__fsub_rn(u4, u3)));
  e = __fmaf_rn(c.l, x.h, e);
  f = __fmaf_rn(d.l, y.h, f);
  e = __fmaf_rn(c.m, x.m, e);
  f = __fmaf_rn(d.m, y.m, f);
  e = __fmaf_rn(c.h, x.l, e);
  f = __fmaf_rn(d.h, y.l, f);
  e = __fadd_rn(e, f);
  if (!NORM) return lf3(__fsub_rn(t2, LIMB_G1), __fsub_rn(u4, LIMB_G2), e);
  const float u5 = __fadd_rn(u4, e);
  const float m = __fsub_rn(u5, LIMB_G2), t3 = __fadd_rn(t2, m);
  return lf3(__fsub_rn(t3, LIMB_G1), __fsub_rn(m, __fsub_rn(t3, t2)), __fsub_rn(e, __fsub_rn(u5, u4)));
}
// ---------------------------------------------------------------- complex products

// a x + b y of the small DFTs' constants: the limb forms make one trip over the grid.
template <typename T>
__device__ __forceinline__ T lin2(T a, T x, T b, T y) {
  return a * x + b * y;
}
__device__ __forceinline__ lf3 lin2(lf3 a, lf3 x, lf3 b, lf3 y) { return limb_lin2<false>(a, x, b, y); }

// Complex forms on both components.
template <typename T>
__device__ __forceinline__ C2<T> crmul(T c, C2<T> a) {
  return C2<T>{c * a.x, c * a.y};
}
template <typename T>
__device__ __forceinline__ C2<T> cscale2(C2<T> a, float s) {
  return C2<T>{scale2(a.x, s), scale2(a.y, s)};
}
template <typename T>
__device__ __forceinline__ C2<T> clin2(T a, C2<T> x, T b, C2<T> y) {
  return C2<T>{lin2(a, x.x, b, y.x), lin2(a, x.y, b, y.y)};
}

// ---------------------------------------------------------------- packed pairs

// The real and imaginary limbs of a complex value as one register pair: packed FP32
// instructions do the same roundings on both halves for one issue slot.  The small transforms
// use them (P1 of FP64 at 10000^2: 8.1 -> 7.7 ms); twiddle products stay scalar, as the swap of one
// factor's components took back what the packing gave (7.8 ms).
struct f32p {
  unsigned long long v;
};
__device__ __forceinline__ f32p pk(float a, float b) {
  f32p r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32p pk(float a) { return pk(a, a); }
__device__ __forceinline__ void unpk(f32p a, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ f32p operator+(f32p a, f32p b) {
  f32p r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32p operator-(f32p a, f32p b) {
  f32p r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32p pfma(f32p a, f32p b, f32p c) {
  f32p r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
template <typename T>
struct Packed;
template <>
struct Packed<lf3> {
  f32p h, m, l;
  static __device__ __forceinline__ Packed of(lf3 x, lf3 y) {
    return Packed{pk(x.h, y.h), pk(x.m, y.m), pk(x.l, y.l)};
  }
  __device__ __forceinline__ C2<lf3> c() const {
    C2<lf3> r;
    unpk(h, r.x.h, r.y.h);
    unpk(m, r.x.m, r.y.m);
    unpk(l, r.x.l, r.y.l);
    return r;
  }
};
template <>
struct Packed<ff> {
  f32p h, l;
  static __device__ __forceinline__ Packed of(ff x, ff y) { return Packed{pk(x.hi, y.hi), pk(x.lo, y.lo)}; }
  __device__ __forceinline__ C2<ff> c() const {
    C2<ff> r;
    unpk(h, r.x.hi, r.y.hi);
    unpk(l, r.x.lo, r.y.lo);
    return r;
  }
};
using P3 = Packed<lf3>;
template <typename T>
__device__ __forceinline__ Packed<T> pc(C2<T> a) { return Packed<T>::of(a.x, a.y); }

__device__ __forceinline__ C2<lf3> cadd(C2<lf3> a, C2<lf3> b) {
  const P3 x = pc(a), y = pc(b);
  return P3{x.h + y.h, x.m + y.m, x.l + y.l}.c();
}
__device__ __forceinline__ C2<lf3> csub(C2<lf3> a, C2<lf3> b) {
  const P3 x = pc(a), y = pc(b);
  return P3{x.h - y.h, x.m - y.m, x.l - y.l}.c();
}
// (the operations of the scalar forms above, one for one; -(t - G) as G - t)
__device__ __forceinline__ P3 pmul(P3 a, P3 b) {
  const f32p G1 = pk(LIMB_G1), G2 = pk(LIMB_G2), t = pfma(a.h, b.h, G1);
  const f32p r = pfma(a.h, b.h, G1 - t);
  const f32p u0 = r + G2, u1 = pfma(a.h, b.m, u0), u2 = pfma(a.m, b.h, u1);
  f32p e = r - (u0 - G2);
  f32p f = pfma(a.h, b.m, u0 - u1);
  f = f + pfma(a.m, b.h, u1 - u2);
  e = pfma(a.h, b.l, e);
  f = pfma(a.l, b.h, f);
  e = pfma(a.m, b.m, e);
  return P3{t - G1, u2 - G2, e + f};
}
__device__ __forceinline__ P3 plin2(P3 c, P3 x, P3 d, P3 y) {
  const f32p G1 = pk(LIMB_G1), G2 = pk(LIMB_G2);
  const f32p t1 = pfma(c.h, x.h, G1), t2 = pfma(d.h, y.h, t1);
  const f32p r = pfma(c.h, x.h, G1 - t1) + pfma(d.h, y.h, t1 - t2);
  const f32p u0 = r + G2, u1 = pfma(c.m, x.h, u0), u2 = pfma(c.h, x.m, u1);
  const f32p u3 = pfma(d.m, y.h, u2), u4 = pfma(d.h, y.m, u3);
  f32p e = r - (u0 - G2);
  f32p f = pfma(c.m, x.h, u0 - u1);
  e = e + pfma(c.h, x.m, u1 - u2);
  f = f + pfma(d.m, y.h, u2 - u3);
  e = e + pfma(d.h, y.m, u3 - u4);
  e = pfma(c.l, x.h, e);
  f = pfma(d.l, y.h, f);
  e = pfma(c.m, x.m, e);
  f = pfma(d.m, y.m, f);
  e = pfma(c.h, x.l, e);
  f = pfma(d.h, y.l, f);
  return P3{t2 - G1, u4 - G2, e + f};
}
__device__ __forceinline__ C2<lf3> crmul(lf3 c, C2<lf3> a) { return pmul(P3::of(c, c), pc(a)).c(); }
__device__ __forceinline__ C2<lf3> clin2(lf3 a, C2<lf3> x, lf3 b, C2<lf3> y) {
  return plin2(P3::of(a, a), pc(x), P3::of(b, b), pc(y)).c();
}
// s a power of two, at least 2^-16: the remainder of the high limb is on the second grid.
__device__ __forceinline__ C2<lf3> cscale2(C2<lf3> a, float s) {
  const P3 x = pc(a);
  const f32p G1 = pk(LIMB_G1), G2 = pk(LIMB_G2), S = pk(s), t = pfma(x.h, S, G1), u = pfma(x.m, S, G2);
  const f32p r = pfma(x.h, S, G1 - t);
  return P3{t - G1, r + (u - G2), pfma(x.l, S, pfma(x.m, S, G2 - u))}.c();
}

// Float-float, the operations of ff's + and - one for one.  (Its products stay scalar: a packed
// product ended up fused into the addition that followed it, and a two-sum needs the rounded one.)
using PF = Packed<ff>;
__device__ __forceinline__ C2<ff> cadd(C2<ff> a, C2<ff> b) {
  const PF x = pc(a), y = pc(b);
  const f32p s = x.h + y.h, bb = s - x.h, e = (x.h - (s - bb)) + (y.h - bb);
  return PF{s, e + (x.l + y.l)}.c();
}
__device__ __forceinline__ C2<ff> csub(C2<ff> a, C2<ff> b) {
  const PF x = pc(a), y = pc(b);
  const f32p s = x.h - y.h, bb = s - x.h, e = (x.h - (s - bb)) - (y.h + bb);
  return PF{s, e + (x.l - y.l)}.c();
}
__device__ __forceinline__ C2<ff> clin2(ff a, C2<ff> x, ff b, C2<ff> y) { return cadd(crmul(a, x), crmul(b, y)); }

// v w or v conj(w); every product carries.
template <bool CONJ, typename T>
__device__ __forceinline__ C2<T> limb_tw(C2<T> v, C2<T> w) {
  if (CONJ) return C2<T>{limb_lin2<true>(w.x, v.x, w.y, v.y), limb_lin2<true>(w.x, v.y, -w.y, v.x)};
  return C2<T>{limb_lin2<true>(w.x, v.x, -w.y, v.y), limb_lin2<true>(w.x, v.y, w.y, v.x)};
}
__device__ __forceinline__ C2<lf3> limb_cnorm(C2<lf3> v) {
  const P3 a = pc(v);
  const f32p G1 = pk(LIMB_G1), G2 = pk(LIMB_G2), q = (a.l + G2) - G2, m = a.m + q, p = (m + G1) - G1;
  return P3{a.h + p, m - p, a.l - q}.c();
}

// ---------------------------------------------------------------- scale of one transform

// Partial sum of |re| + |im| over the inputs of one transform: s 2^(e - 1023) with the exponent
// field e kept apart (in place, bits 20..30), s from the high words alone.
template <typename S>
struct LimbSum;
template <>
struct LimbSum<double> {
  int e;
  float s;
};

// 2^(a - b) for exponent fields a <= b in place (bits 20..30); 0 where it underflows FP32.
__device__ __forceinline__ float limb_pow_diff(int a, int b) {
  return __int_as_float(max(a - b + (127 << 20), 0) << 3);
}
template <int N>
__device__ __forceinline__ LimbSum<double> limb_sum(const C2<double>* v) {
  int top = 0;
#pragma unroll
  for (int i = 0; i < N; i++)
    top = max(top, max(__double2hiint(v[i].x) & 0x7fffffff, __double2hiint(v[i].y) & 0x7fffffff));
  const int e = top & 0x7ff00000;
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < N; i++) {
    s = __fadd_rn(s, limb_pow_diff(__double2hiint(v[i].x) & 0x7fffffff, e));
    s = __fadd_rn(s, limb_pow_diff(__double2hiint(v[i].y) & 0x7fffffff, e));
  }
  return LimbSum<double>{e, s};
}
__device__ __forceinline__ LimbSum<double> limb_sum_add(LimbSum<double> a, LimbSum<double> b) {
  const int e = max(a.e, b.e);
  return LimbSum<double>{e, __fmaf_rn(a.s, limb_pow_diff(a.e, e), __fmul_rn(b.s, limb_pow_diff(b.e, e)))};
}
__device__ __forceinline__ LimbSum<double> limb_sum_warp(LimbSum<double> a) {
  const int e = __reduce_max_sync(0xffffffffu, a.e);
  a.s = __fmul_rn(a.s, limb_pow_diff(a.e, e));
  a.e = e;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a.s = __fadd_rn(a.s, __shfl_xor_sync(0xffffffffu, a.s, o));
  return a;
}

// The same with the largest |re| + |im| of a value, or of the G values that one input of the
// transform is made of: p 2^(e - 1023).
struct LimbPeak {
  int e;
  float s, p;
};
template <int N, int G>
__device__ __forceinline__ LimbPeak limb_peak(const C2<double>* v) {
  static_assert(N % G == 0, "whole groups");
  int top = 0;
#pragma unroll
  for (int i = 0; i < N; i++)
    top = max(top, max(__double2hiint(v[i].x) & 0x7fffffff, __double2hiint(v[i].y) & 0x7fffffff));
  const int e = top & 0x7ff00000;
  float s = 0.f, p = 0.f;
#pragma unroll
  for (int i = 0; i < N; i += G) {
    float g = 0.f;
#pragma unroll
    for (int k = 0; k < G; k++) {
      g = __fadd_rn(g, limb_pow_diff(__double2hiint(v[i + k].x) & 0x7fffffff, e));
      g = __fadd_rn(g, limb_pow_diff(__double2hiint(v[i + k].y) & 0x7fffffff, e));
    }
    s = __fadd_rn(s, g);
    p = fmaxf(p, g);
  }
  return LimbPeak{e, s, p};
}
__device__ __forceinline__ LimbPeak limb_peak_add(LimbPeak a, LimbPeak b) {
  const int e = max(a.e, b.e);
  const float fa = limb_pow_diff(a.e, e), fb = limb_pow_diff(b.e, e);
  return LimbPeak{e, __fmaf_rn(a.s, fa, __fmul_rn(b.s, fb)), fmaxf(__fmul_rn(a.p, fa), __fmul_rn(b.p, fb))};
}
__device__ __forceinline__ LimbPeak limb_peak_warp(LimbPeak a) {
  const int e = __reduce_max_sync(0xffffffffu, a.e);
  const float f = limb_pow_diff(a.e, e);
  a.s = __fmul_rn(a.s, f);
  a.p = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(__fmul_rn(a.p, f))));  // (p >= 0)
  a.e = e;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a.s = __fadd_rn(a.s, __shfl_xor_sync(0xffffffffu, a.s, o));
  return a;
}

// The power of two that brings a transform below 1 and back: the exponent fields to add to a
// double before its conversion to a 62-bit fixed-point integer and after the way back.  A sum
// that is not finite makes every output NaN.
template <typename T>
struct LimbScale;
template <>
struct LimbScale<lf3> {
  int e;  // |x| < 2^e
  bool bad;
};
// Least e with s 2^(field - 1023) < 2^e; the margin covers the cut to high words and the
// rounding of some ten thousand FP32 additions.
__device__ __forceinline__ int limb_above(int field, float s) {
  return (field >> 20) - 1023 + ((__float_as_int(__fmul_rn(s, 1.f + 0x1p-17f)) >> 23) - 127) + 1;
}
__device__ __forceinline__ LimbScale<lf3> limb_scale(LimbSum<double> a) {
  return LimbScale<lf3>{limb_above(a.e, a.s), a.e >= 0x7ff00000};
}

// The scales of a row transform's levels: the values are at most p r_0 ... r_i in level i, p the
// largest of the inputs, and at most the sum s.  first(): the scale of the inputs, for level 0
// of radix r; next(): the factor that takes the values over to the scale of a level of radix r.
struct LimbGrow {
  int field, top, e;
  float p;
  bool bad;
  // bs, bp: what the transform's sum and its largest input are at most, in s and p of a
  static __device__ __forceinline__ LimbGrow of(LimbPeak a, float bs, float bp) {
    return LimbGrow{a.e, limb_above(a.e, __fmul_rn(a.s, bs)), 0, __fmul_rn(a.p, bp), a.e >= 0x7ff00000};
  }
  __device__ __forceinline__ int level(int r) {
    p = __fmul_rn(p, (float)r);
    return min(top, limb_above(field, p));
  }
  __device__ __forceinline__ LimbScale<lf3> first(int r) {
    e = level(r);
    return LimbScale<lf3>{e, bad};
  }
  __device__ __forceinline__ float next(int r) {
    const int was = e;
    e = level(r);
    return __int_as_float((127 + was - e) << 23);
  }
  __device__ __forceinline__ LimbScale<lf3> scale() const { return LimbScale<lf3>{e, bad}; }
};

// ---------------------------------------------------------------- in and out

// FP64 in: the exponent moved by an integer addition, one conversion to a fixed-point
// integer of 62 fractional bits, and its bit fields 22 | 17 | 23 as the three limbs.  Subnormal
// values count as zero: where the sum is so small that they matter, limb_lift comes first.
__device__ __forceinline__ lf3 limb_in(double v, LimbScale<lf3> s) {
  const int hi = __double2hiint(v), d = (62 - s.e) * (1 << 20);
  const int ex = hi & 0x7ff00000;
  const bool z = ex == 0 || ex + d <= 0;
  const long long q = __double2ll_rn(z ? 0.0 : __hiloint2double(hi + d, __double2loint(v)));
  const int qh = (int)(q >> 32);
  const unsigned ql = (unsigned)q;
  const float h = __fsub_rn(__int_as_float(0x40400000 + (qh >> 8)), LIMB_G1);
  const float m = __fsub_rn(__int_as_float(0x37800000 | (int)(__funnelshift_r(ql, (unsigned)qh, 23) & 0x1ffffu)), 0x1p-16f);
  const float l = __fsub_rn(__int_as_float(0x2C000000 | (int)(ql & 0x7fffffu)), 0x1p-39f);
  return lf3(h, m, l);
}
__device__ __forceinline__ double limb_out(lf3 v, LimbScale<lf3> s) {
  const float c = __fsub_rn(__fadd_rn(v.l, LIMB_G2), LIMB_G2);
  const float mm = __fadd_rn(v.m, c), ll = __fsub_rn(v.l, c);
  const int ih = __float_as_int(__fadd_rn(v.h, LIMB_G1)) - 0x40400000;
  const int im = __float_as_int(__fadd_rn(mm, LIMB_G2)) - 0x37C00000;
  const int il = __float_as_int(__fadd_rn(ll, LIMB_G3)) - 0x2C400000;
  const long long q = ((long long)ih << 40) + ((long long)im << 23) + il;
  const double d = __ll2double_rn(q);
  if (s.bad) return __longlong_as_double(0x7ff8000000000000ll);
  const int hi = __double2hiint(d), lo = __double2loint(d), ef = (hi >> 20) & 0x7ff, sh = s.e - 62, r = ef + sh;
  if (ef == 0 || (unsigned)(r - 1) >= 2046u) {  // zero; beyond the exponents: infinite; below: rounded to a subnormal
    if (ef == 0 || r < -60) return 0.0;
    if (r > 0) return __hiloint2double((hi & 0x80000000) | 0x7ff00000, 0);
    return __dmul_rn(__hiloint2double(hi + (sh + 64) * (1 << 20), lo), 0x1p-64);
  }
  return __hiloint2double(hi + (int)((unsigned)sh << 20), lo);
}
__device__ __forceinline__ double limb_round(lf3 v, LimbScale<lf3> s) { return limb_out(v, s); }

template <typename S, typename T>
__device__ __forceinline__ C2<T> limb_cin(C2<S> v, LimbScale<T> s) {
  return C2<T>{limb_in(v.x, s), limb_in(v.y, s)};
}
template <typename S, typename T>
__device__ __forceinline__ C2<S> limb_cout(C2<T> v, LimbScale<T> s) {
  return C2<S>{limb_out(v.x, s), limb_out(v.y, s)};
}

// The inputs of a transform and its scale, times 2^128 where the sum is below 2^-880: subnormal
// inputs become normal.  (Asked once for all of them: asked for in every conversion it cost 7 %.)
template <int N>
__device__ __forceinline__ LimbScale<lf3> limb_lift(C2<double>* v, LimbScale<lf3> s) {
  if (s.e < -880) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      v[i].x = __dmul_rn(v[i].x, 0x1p128);
      v[i].y = __dmul_rn(v[i].y, 0x1p128);
    }
    s.e += 128;
  }
  return s;
}

// ---------------------------------------------------------------- arrays of limbs

// Complex limbs in shared memory: 16 bytes (high and middle limbs) and 8 bytes (low limbs) in
// two planes, so that every access is one aligned vector.
template <typename T>
struct LimbArr;
template <>
struct LimbArr<lf3> {
  float4* a;
  float2* b;
  static __host__ __device__ constexpr size_t bytes(long n) { return (size_t)((n + 1) & ~1L) * 24; }
  static __device__ __forceinline__ LimbArr at(unsigned char* raw, long n) {
    return LimbArr{reinterpret_cast<float4*>(raw), reinterpret_cast<float2*>(raw + (size_t)((n + 1) & ~1L) * 16)};
  }
  __device__ __forceinline__ C2<lf3> ld(int i) const {
    const float4 u = a[i];
    const float2 v = b[i];
    return C2<lf3>{lf3(u.x, u.z, v.x), lf3(u.y, u.w, v.y)};
  }
  __device__ __forceinline__ void st(int i, C2<lf3> v) const {
    a[i] = make_float4(v.x.h, v.y.h, v.x.m, v.y.m);
    b[i] = make_float2(v.x.l, v.y.l);
  }
};

// Twiddle tables in global memory: two planes likewise.
template <typename T>
struct LimbTab;
template <>
struct LimbTab<lf3> {
  const float4* a;
  const float2* b;
  __device__ __forceinline__ C2<lf3> ld(long i) const {
    const float4 u = __ldg(a + i);
    const float2 v = __ldg(b + i);
    return C2<lf3>{lf3(u.x, u.z, v.x), lf3(u.y, u.w, v.y)};
  }
};

}  // namespace mlc
