// FP64 square root, reciprocal, log, exp, acos and sin/cos of the polar
// power on the integer pipe.
//
// On sm_103a the FP64 pipe runs at 1/64 of the FP32 and integer rate, so one
// FP64 instruction costs as much as 64 integer ones; the device library's
// functions took about 150 of the 200 FP64 instructions of one root term.
// Here a positive double is unpacked to a 64-bit fixed-point mantissa and an
// exponent, and each function is evaluated with 64-bit integer products
// (four 32-bit multiply-adds for the high half), a table at a nearby point
// and a short series of the remainder whose higher terms need 32 bits only.
// The method is Tang's table-driven one and Newton's iteration for the
// reciprocal square root and reciprocal, from a 22-bit hardware seed; no
// library's code.  Absolute errors are about 2^-58 of a mantissa in [1/2, 1)
// before the one rounding to 53 bits, so a result is the correctly rounded
// one but for about 3% of arguments (the device library's acos, sin and cos:
// 14-17%, its exp: 6%) and off by at most 0.53 ulp.  Results much smaller
// than 1 (a logarithm near 0, an angle below 2^-5, a sine near a zero) keep
// that absolute accuracy, 2^-58 or better, not the relative one: the power
// they go into is of size |q|^e.
//
// Arguments outside the stated ranges are the caller's to send elsewhere.
// The same source compiles for the host, where the tests check it.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define FX_FN static __device__ __forceinline__
#define FX_TAB static __device__ const
#else
#include <math.h>
#include <string.h>
#define FX_FN static inline
#define FX_TAB static const
#endif

typedef struct __attribute__((aligned(16))) {
  unsigned long long a, b;
} fx_pair;

#include "qj_fxmath_tables.h"

typedef unsigned long long fx_u64;
typedef long long fx_i64;

// value m 2^(e - 64), m with its top bit set
typedef struct {
  fx_u64 m;
  int e;
} fx_num;

FX_FN fx_u64 fx_bits(double x) {
#ifdef __CUDACC__
  return (fx_u64)__double_as_longlong(x);
#else
  fx_u64 b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
FX_FN double fx_from(fx_u64 b) {
#ifdef __CUDACC__
  return __longlong_as_double((fx_i64)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
// high half of a 64-bit product
FX_FN fx_u64 fx_mulhi(fx_u64 a, fx_u64 b) {
#ifdef __CUDACC__
  return __umul64hi(a, b);
#else
  return (fx_u64)(((unsigned __int128)a * b) >> 64);
#endif
}
FX_FN fx_i64 fx_smulhi(fx_i64 a, fx_i64 b) {
#ifdef __CUDACC__
  return __mul64hi(a, b);
#else
  return (fx_i64)(((__int128)a * b) >> 64);
#endif
}
FX_FN uint32_t fx_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((fx_u64)a * b) >> 32); }
FX_FN int fx_clz(fx_u64 a) {
#ifdef __CUDACC__
  return __clzll((fx_i64)a);
#else
  return __builtin_clzll(a);
#endif
}
// 22-bit seeds: 1/sqrt(x) and 1/x for x in [1/4, 1]
FX_FN float fx_seed_rsqrt(float x) {
#ifdef __CUDACC__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / sqrtf(x);
#endif
}
FX_FN float fx_seed_rcp(float x) {
#ifdef __CUDACC__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}

// A positive normal double.
FX_FN fx_num fx_unpack(double x) {
  const fx_u64 b = fx_bits(x);
  fx_num r;
  r.e = (int)((b >> 52) & 0x7ff) - 1022;
  r.m = (b << 11) | 0x8000000000000000ull;
  return r;
}
// The mantissa rounded to 53 bits (2^53 when it rounds up to the next power).
FX_FN fx_u64 fx_round53(fx_u64 m) { return (m >> 11) + ((m >> 10) & 1); }
// m with its top bit set, to the nearest double (normal results only).
FX_FN double fx_pack(fx_u64 m, int e) {
  return fx_from(((fx_u64)(uint32_t)(e + 1021) << 52) + fx_round53(m));
}
// v 2^-frac for v > 0 of any size.
FX_FN double fx_pack_fix(fx_u64 v, int frac) {
  const int z = fx_clz(v);
  return fx_pack(v << z, 64 - frac - z);
}

// 1/sqrt(x) for x in [1/4, 1) in 2^-64, result in [1, 2] in 2^-62.  The seed
// y0 leaves d = 1 - x y0^2 below 2^-21; y0 (1 + d/2 + 3/8 d^2) is exact to
// d^3, 2^-63.
FX_FN fx_u64 fx_rsqrt(fx_u64 x) {
  const float xf = (float)(uint32_t)(x >> 32) * 2.3283064365386963e-10f;
  const uint32_t y0 = (uint32_t)(fx_seed_rsqrt(xf) * 1073741824.0f);  // 2^-30
  const fx_i64 d = (fx_i64)((1ull << 60) - fx_mulhi(x, (fx_u64)y0 * y0));  // 2^-60
  const int32_t ds = (int32_t)(d >> 14);                                   // 2^-46
  const fx_i64 g = d + ((3 * ((fx_i64)ds * ds)) >> 34);                    // d + 3/4 d^2
  const fx_i64 gh = g >> 16, gl = g & 0xffff;
  return ((fx_u64)y0 << 32) + (fx_u64)(((fx_i64)y0 * gh + (((fx_i64)y0 * gl) >> 16)) >> 13);
}

// x (top bit set) as sqrt's mantissa in [1/4, 1) and the root's exponent.
FX_FN fx_u64 fx_even(fx_num x, int* e) {
  *e = (x.e + 1) >> 1;
  return (x.e & 1) ? x.m >> 1 : x.m;
}

// sqrt(x) to a double and 1 / (that double) to a double and, in *inv, to
// 2^-62 as in_m 2^-62 2^(in_e).
typedef struct {
  double root;
  fx_u64 inv;  // 1 / root = inv 2^(-62 - e)
  int e;
} fx_roots;
FX_FN fx_roots fx_sqrt_inv(double x) {
  fx_roots r;
  const fx_u64 f = fx_even(fx_unpack(x), &r.e);
  const fx_u64 y = fx_rsqrt(f);
  const fx_u64 s = fx_mulhi(f, y) << 2;  // sqrt in [1/2, 1), 2^-64
  const fx_u64 s53 = fx_round53(s);
  r.root = fx_from(((fx_u64)(uint32_t)(r.e + 1021) << 52) + s53);
  // 1 / (s + rho) = y - y^2 rho, rho the rounding of the root (11 bits)
  const fx_i64 rho = (fx_i64)((s53 << 11) - s);  // 2^-64 (wraps right where s53 = 2^53)
  const uint32_t yh = (uint32_t)(y >> 32);       // 2^-30
  const fx_i64 ry = (rho * (fx_i64)yh) >> 16;    // 2^-78
  r.inv = y - (fx_u64)((ry * (fx_i64)yh) >> 46);
  return r;
}

// v > 0 in 2^-62, below 4, times 2^e, to a double.
FX_FN double fx_pack62(fx_u64 v, int e) {
  const int z = fx_clz(v);
  return fx_pack(v << z, e + 2 - z);
}

// 1/x of a positive normal double.
FX_FN double fx_rcp(double x) {
  const fx_num n = fx_unpack(x);  // m in [1/2, 1)
  const float xf = (float)(uint32_t)(n.m >> 32) * 2.3283064365386963e-10f;
  const uint32_t y0 = (uint32_t)(fx_seed_rcp(xf) * 1073741824.0f);  // 2^-30, in [1, 2]
  // d = 1 - m y0 (2^-62); y0 (1 + d + d^2) exact to d^3
  const fx_i64 d = (fx_i64)((1ull << 62) - fx_mulhi(n.m, (fx_u64)y0 << 32));
  const int32_t ds = (int32_t)(d >> 16);                    // 2^-46
  const fx_i64 g = d + (((fx_i64)ds * ds) >> 30);           // 2^-62
  const fx_i64 gh = g >> 16, gl = g & 0xffff;
  const fx_u64 y = ((fx_u64)y0 << 32) + (fx_u64)(((fx_i64)y0 * gh + (((fx_i64)y0 * gl) >> 16)) >> 14);
  return fx_pack62(y, -n.e);
}

// log x of a positive normal double with |log x| < 100.
FX_FN double fx_log(double x) {
  const fx_u64 b = fx_bits(x);
  const fx_u64 m = (b & 0xfffffffffffffull) | 0x10000000000000ull;  // [1, 2) in 2^-52
  const fx_pair t = fx_tab_log[(int)(m >> 44) & 255];
  const uint32_t c = (uint32_t)t.b & 0xffff;
  const int k = (int)(b >> 52) - 1023 + (int)(t.b >> 16);
  const fx_i64 r = (fx_i64)(m * c - 0x8000000000000000ull);  // m c - 1 in 2^-63, below 2^-8.3
  // log(1 + r) = r - r^2/2 + r^3 (1/3 - r/4 + r^2/5 - r^3/6 + r^4/7)
  const fx_u64 r2 = (fx_u64)fx_smulhi(r << 8, r << 8);       // 2^-78
  const int32_t rs = (int32_t)(r >> 24);                     // 2^-39
  const uint32_t r2s = (uint32_t)(r2 >> 30);                 // 2^-48
  // in 2^-33; rs 2^-39 * 2^-33 -> 2^-33 by >> 39
  int32_t p = 1431655765 - (int32_t)(((fx_i64)rs * 1227133513) >> 39);  // 1/6 - r/7
  p = 1717986918 - (int32_t)(((fx_i64)rs * p) >> 39);                   // 1/5 - ...
  fx_i64 q = 2147483648ll - (((fx_i64)rs * p) >> 39);                   // 1/4 - ...
  q = 2863311531ll - (((fx_i64)rs * q) >> 39);                          // 1/3 - ..., 2^-33
  const uint32_t c3 = (uint32_t)(((fx_u64)r2s * (uint32_t)q) >> 31);    // 2^-50
  const fx_i64 s = r - (fx_i64)(r2 >> 16) + (((fx_i64)rs * (fx_i64)c3) >> 26);
  fx_i64 v = (fx_i64)t.a + s;  // 2^-63
  int sh = 0;
  if (k) {
    // k log 2, with as many bits below the point as k leaves
    sh = fx_clz((fx_u64)(k < 0 ? -k : k));
    sh = 65 - sh;
    v = (v >> sh) + (((fx_i64)k * 0x58b90bfb) << (32 - sh)) + (((fx_i64)k * 0xe8e7bcd6ll) >> sh);
  }
  if (v == 0) return 0.0;
  const double a = fx_pack_fix(v < 0 ? (fx_u64)-v : (fx_u64)v, 63 - sh);
  return v < 0 ? -a : a;
}

// exp x for 2^-60 < |x| < 700.
FX_FN double fx_exp(double x) {
  const fx_num n = fx_unpack(x);
  // |x| log2 e = (hi, lo) 2^(e + 1), log2(e)/2 in 2^-64
  const fx_u64 L = 0xb8aa3b295c17f0bcull;
  fx_u64 hi = fx_mulhi(n.m, L), lo = n.m * L;
  const int s = n.e + 1;
  int k = 0;
  fx_u64 f;
  if (s > 0) {
    k = (int)(hi >> (64 - s));
    f = (hi << s) | (lo >> (64 - s));
  } else {
    f = s > -64 ? hi >> -s : 0;
  }
  if (fx_bits(x) >> 63) {
    k = -k - (f != 0);
    f = 0 - f;
  }
  const fx_u64 T = fx_tab_exp[(int)(f >> 56)];
  // t = (f - j/256) log 2, 2^-72
  const fx_u64 t = fx_mulhi(f << 8, 0xb17217f7d1cf79acull);
  const fx_u64 t2 = fx_mulhi(t, t);         // 2^-80
  const uint32_t ts = (uint32_t)(t >> 32);  // 2^-40
  const uint32_t t2s = (uint32_t)(t2 >> 31);  // 2^-49
  // 1/6 + t/24 + t^2/120 + t^3/720 in 2^-34; ts p: 2^-40 2^-34 -> >> 40
  uint32_t p = 143165577u + (uint32_t)(((fx_u64)ts * 23860929u) >> 40);
  p = 715827883u + (uint32_t)(((fx_u64)ts * p) >> 40);
  p = 2863311531u + (uint32_t)(((fx_u64)ts * p) >> 40);
  const uint32_t c3 = fx_mulhi32(t2s, p);  // 2^-51
  const fx_u64 E = (t >> 8) + (t2 >> 17) + (((fx_u64)ts * c3) >> 27);  // e^t - 1, 2^-64
  fx_u64 m = T + fx_mulhi(T, E);
  if (m < T) m = ~0ull;  // rounded past 2
  return fx_pack(m, k + 1);
}

// acos u for |u| < 1 - 2^-17: u = w inv 2^(-62 - e), w's mantissa and
// exponent in n (n.m = 0 for w = 0), rounded to a double first; neg: u < 0.
FX_FN double fx_acos(fx_num n, fx_u64 inv, int e, int neg, int* far) {
  const fx_u64 HALF_PI = 0x6487ed5110b4611aull;  // 2^-62
  // u in 2^-64 (nothing left below 2^-64)
  fx_u64 U = 0;
  if (n.m) {
    fx_u64 p = fx_mulhi(n.m, inv);  // 2^-62, in [1/2, 2)
    const int z = fx_clz(p);
    p <<= z;
    const int eu = n.e - e + 2 - z;
    if (eu > 0) {  // |u| >= 1 but for rounding
      *far = 1;
      return 0.0;
    }
    const fx_u64 u53 = fx_round53(p);
    if (eu > -64) U = u53 >> 53 ? (eu == 0 ? ~0ull : 1ull << (64 + eu)) : (u53 << 11) >> -eu;
  }
  if (U >= 0xffff800000000000ull) {  // within 2^-17 of 1
    *far = 1;
    return 0.0;
  }
  // s = sqrt((1 - u)(1 + u)), the first factor normalized
  const fx_u64 w = 0 - U;  // 1 - u (0 where u = 0)
  fx_u64 S;
  if (U == 0) {
    S = ~0ull;
  } else {
    const int z = fx_clz(w);
    fx_num v;
    v.m = fx_mulhi(w << z, 0x8000000000000000ull + (U >> 1));  // (1 - u)(1 + u)/2
    const int y = fx_clz(v.m);
    v.m <<= y;
    v.e = 1 - z - y;
    int h;
    const fx_u64 f = fx_even(v, &h);
    const fx_u64 r = fx_mulhi(f, fx_rsqrt(f));  // 2^-62, in [1/2, 1)
    S = (r >> 62 ? ~0ull : r << 2) >> -h;  // h <= 0; the root may round up to 1
  }
  const int small = U <= S;
  const fx_u64 a = small ? U : S, b = small ? S : U;
  const int j = (int)(a >> 55);
  const fx_pair t = fx_tab_asin[j];
  // sin(asin a - asin a_j) = a cos_j - b a_j
  const fx_i64 x = (fx_i64)(fx_mulhi(a, t.b) - fx_mulhi(b, (fx_u64)(2 * j + 1) << 54));  // 2^-64
  // below 2^-9.4; asin x = x + x^3 (1/6 + 3/40 x^2)
  const int32_t xs = (int32_t)(x >> 24);                                 // 2^-40
  const uint32_t x2 = (uint32_t)(((fx_i64)xs * xs) >> 30);               // 2^-50
  const uint32_t p = 2863311531u + fx_mulhi32(x2, 4915u);                // 2^-34
  const uint32_t c3 = (uint32_t)(((fx_u64)x2 * p) >> 31);                // 2^-53
  const fx_i64 d = (x + (((fx_i64)xs * (fx_i64)c3) >> 29)) >> 2;         // 2^-62
  const fx_u64 as = t.a + (fx_u64)d;                                     // asin a
  fx_u64 th;
  if (small) th = neg ? HALF_PI + as : HALF_PI - as;
  else th = neg ? 2 * HALF_PI - as : as;
  return fx_pack62(th, 0);
}

// sin x and cos x for 2^-20 < x < 2^11.
FX_FN void fx_sincos(double x, double* sn, double* cs) {
  const fx_num n = fx_unpack(x);
  // x 2/pi in quarter turns, 2/pi in 2^-64
  const fx_u64 C = 0xa2f9836e4e44152aull;
  const fx_u64 hi = fx_mulhi(n.m, C), lo = n.m * C;
  int k = 0;
  fx_u64 f;
  if (n.e > 0) {
    k = (int)(hi >> (64 - n.e));
    f = (hi << n.e) | (lo >> (64 - n.e));
  } else {
    f = hi >> -n.e;
  }
  const int j = (int)((f >> 55) + 1) >> 1;  // nearest of 0..256
  const fx_i64 r = (fx_i64)(f - ((fx_u64)j << 56));  // below 2^-9 in size
  // eps = r pi/2: (r << 7) pi/4, 2^-70
  const fx_i64 eps = fx_smulhi((fx_i64)((fx_u64)r << 7), 0x6487ed5110b4611all) << 1;
  const fx_u64 e2 = (fx_u64)fx_smulhi(eps << 1, eps << 1);  // 2^-78
  const int32_t es = (int32_t)(eps >> 31);                  // 2^-39
  const uint32_t e2s = (uint32_t)(e2 >> 30);                // 2^-48
  // sin eps = eps - eps^3 (1/6 - eps^2/120)
  const uint32_t p = 2863311531u - fx_mulhi32(e2s, 2185u);  // 2^-34 (1/120 in 2^-18)
  const uint32_t c3 = (uint32_t)(((fx_u64)e2s * p) >> 31);  // 2^-51
  const fx_i64 se = eps - (((fx_i64)es * (fx_i64)c3) >> 20);  // 2^-70
  // 1 - cos eps = eps^2/2 - eps^4/24
  const uint32_t e4 = fx_mulhi32(e2s, e2s);                              // 2^-64
  const fx_u64 V = (e2 >> 15) - fx_mulhi32(e4, 178956971u);              // 2^-64 (1/24: 2^-32)
  const fx_pair t = fx_tab_sin[j];
  const fx_i64 S = (fx_i64)t.a, Cc = (fx_i64)t.b;                        // 2^-62
  fx_i64 si = S + (fx_smulhi(Cc, se << 1) >> 7) - (fx_i64)(fx_mulhi((fx_u64)S, V << 17) >> 17);
  fx_i64 co = Cc - (fx_smulhi(S, se << 1) >> 7) - (fx_i64)(fx_mulhi((fx_u64)Cc, V << 17) >> 17);
  if (k & 1) {
    const fx_i64 u = si;
    si = co;
    co = -u;
  }
  if (k & 2) {
    si = -si;
    co = -co;
  }
  const fx_u64 sb = si < 0 ? 0x8000000000000000ull : 0, cb = co < 0 ? 0x8000000000000000ull : 0;
  *sn = si ? fx_from(fx_bits(fx_pack62(si < 0 ? (fx_u64)-si : (fx_u64)si, 0)) | sb) : 0.0;
  *cs = co ? fx_from(fx_bits(fx_pack62(co < 0 ? (fx_u64)-co : (fx_u64)co, 0)) | cb) : 0.0;
}

// ---- quaternion products in fixed point ---------------------------------
// A Hamilton product costs 28 FP64 instructions in the reference's order, as
// much of that pipe's time as 1792 integer ones would take on theirs.  Here a
// quaternion is four 64-bit integers with one exponent, value c 2^(e - 62),
// the largest |c| in [2^61, 2^62): a product is 16 high halves of 64-bit
// products of magnitudes and a renormalization.  Against |a b| it is off by
// at most 2^-55 (four halves cut towards 0, and the largest component of a
// product of norm 2^58 is at least 2^57), an FP64 product by 2^-52.
//
// Every step cuts magnitudes, so that values of opposite sign are treated
// alike: terms that cancel exactly in FP64 (conjugate factors) cancel here,
// and mirror images have the same bits.  The error is one of the whole
// quaternion, FP64's of each component.  Where a component is small in every
// one of its terms (near the real axis or a coordinate plane with roots in
// it), FP64 keeps it to 2^-53 of itself, and whether it is zero decides the
// polar power's branch.  Maps with roots in such places are known when they
// are uploaded (fx_beside); elsewhere `odd` says that FP64's product is
// wanted, as soon as all four terms of a component are below 2^-16 of the
// largest they could be without all being zero, or the vector part as a whole
// is below 2^-20.  (At 2^-9, where fewer than 53 bits are left, a square's
// small vector part met a small component of the product before it in 1e-3 of
// a map's first applications, whose FP64 error is as large as ever.)
typedef struct {
  fx_i64 w, x, y, z;       // the components, and as magnitude and sign (0 or
  fx_u64 mw, mx, my, mz;   // -1): the compiler drops what a caller leaves
  int32_t sw, sx, sy, sz;  // unused
  int e;
  int odd;  // not held as FP64 would hold it (of a difference: bit c, component c is small)
} fx_quat;

FX_FN uint32_t fx_high(fx_u64 v) { return (uint32_t)(v >> 32); }
FX_FN uint32_t fx_least(uint32_t a, uint32_t b) { return a < b ? a : b; }
// the sign of c, and a sign in both halves of a word
FX_FN int32_t fx_sign(fx_i64 c) { return (int32_t)(c >> 32) >> 31; }
FX_FN fx_u64 fx_mask(int32_t s) {
#ifdef __CUDACC__
  fx_u64 m;
  asm("mov.b64 %0, {%1, %1};" : "=l"(m) : "r"(s));
  return m;
#else
  return (fx_u64)(fx_i64)s;
#endif
}
FX_FN fx_u64 fx_abs(fx_i64 c) {
  const fx_u64 s = fx_mask(fx_sign(c));
  return ((fx_u64)c ^ s) - s;
}
FX_FN fx_i64 fx_signed(fx_u64 m, int32_t s) { return (fx_i64)((m ^ fx_mask(s)) - fx_mask(s)); }
// v 2^-s, its magnitude cut; 0 <= s < 64
FX_FN fx_i64 fx_cut(fx_i64 v, int s) { return fx_signed(fx_abs(v) >> s, fx_sign(v)); }

// magnitudes and signs from the components, and back
FX_FN fx_quat fx_split(fx_quat q) {
  q.sw = fx_sign(q.w);
  q.sx = fx_sign(q.x);
  q.sy = fx_sign(q.y);
  q.sz = fx_sign(q.z);
  q.mw = fx_abs(q.w);
  q.mx = fx_abs(q.x);
  q.my = fx_abs(q.y);
  q.mz = fx_abs(q.z);
  return q;
}
FX_FN fx_quat fx_joined(fx_quat q) {
  q.w = fx_signed(q.mw, q.sw);
  q.x = fx_signed(q.mx, q.sx);
  q.y = fx_signed(q.my, q.sy);
  q.z = fx_signed(q.mz, q.sz);
  return q;
}
FX_FN int fx_clz32(uint32_t a) {
#ifdef __CUDACC__
  return __clz((int)a);
#else
  return a ? __builtin_clz(a) : 32;
#endif
}
// The largest magnitude's top bit to 2^61; none is 2^62 or more, and one has
// a high half (or all are zero: so they stay).
FX_FN fx_quat fx_norm(fx_quat q) {
  const int s = fx_clz32(fx_high(q.mw) | fx_high(q.mx) | fx_high(q.my) | fx_high(q.mz)) - 2;
  q.mw <<= s;
  q.mx <<= s;
  q.my <<= s;
  q.mz <<= s;
  q.e -= s;
  return fx_joined(q);
}

FX_FN int fx_field(double v) { return (int)(fx_bits(v) >> 52) & 0x7ff; }
// v's mantissa in units of 2^(top - 62), top at least v's exponent; 0 for
// zeros and subnormals.
FX_FN fx_u64 fx_align(double v, int top) {
  const int f = fx_field(v), sh = 2 + top - (f - 1022);
  return f == 0 || sh > 63 ? 0 : ((fx_bits(v) << 11) | 0x8000000000000000ull) >> sh;
}
// The exponent of the largest component.
FX_FN int fx_top(double w, double x, double y, double z) {
  int f = fx_field(w), g = fx_field(x);
  f = f > g ? f : g;
  g = fx_field(y);
  f = f > g ? f : g;
  g = fx_field(z);
  return (f > g ? f : g) - 1022;
}
// The components in units of 2^(top - 62), top at least fx_top's.
FX_FN fx_quat fx_quat_at(double w, double x, double y, double z, int top) {
  fx_quat q;
  q.e = top;
  q.odd = 0;
  q.sw = fx_sign((fx_i64)fx_bits(w));
  q.sx = fx_sign((fx_i64)fx_bits(x));
  q.sy = fx_sign((fx_i64)fx_bits(y));
  q.sz = fx_sign((fx_i64)fx_bits(z));
  q.mw = fx_align(w, top);
  q.mx = fx_align(x, top);
  q.my = fx_align(y, top);
  q.mz = fx_align(z, top);
  return fx_joined(q);
}
// odd where a component that is not zero has fewer than 11 bits left
FX_FN fx_quat fx_quat_of(double w, double x, double y, double z) {
  const int top = fx_top(w, x, y, z), least = top + 1022 - 51;
  fx_quat q = fx_quat_at(w, x, y, z, top);
  if (fx_field(w) < least || fx_field(x) < least || fx_field(y) < least || fx_field(z) < least)
    q.odd = (w != 0.0 && fx_field(w) < least) || (x != 0.0 && fx_field(x) < least) ||
            (y != 0.0 && fx_field(y) < least) || (z != 0.0 && fx_field(z) < least);
  return q;
}

// a - b, each kept to 2^-62 of the larger exponent: off by at most 2^-53 of
// |a - b| unless fx_near says that more bits cancelled.  odd: bit c where
// component c has fewer than 33 bits; such a one is exact where the operands'
// components are equal.  (Of the operands only w to z and e count.)
FX_FN fx_quat fx_qsub(fx_quat a, fx_quat b) {
  fx_quat o;
  o.e = a.e > b.e ? a.e : b.e;
  if (a.e != b.e) {
    const int sa = o.e - a.e < 63 ? o.e - a.e : 63, sb = o.e - b.e < 63 ? o.e - b.e : 63;
    a.w = fx_cut(a.w, sa);
    a.x = fx_cut(a.x, sa);
    a.y = fx_cut(a.y, sa);
    a.z = fx_cut(a.z, sa);
    b.w = fx_cut(b.w, sb);
    b.x = fx_cut(b.x, sb);
    b.y = fx_cut(b.y, sb);
    b.z = fx_cut(b.z, sb);
  }
  o.w = a.w - b.w;
  o.x = a.x - b.x;
  o.y = a.y - b.y;
  o.z = a.z - b.z;
  o = fx_split(o);
  o.odd = (fx_high(o.mw) == 0) | (fx_high(o.mx) == 0) << 1 | (fx_high(o.my) == 0) << 2 |
          (fx_high(o.mz) == 0) << 3;
  // below 2^63: the top bit to 2^62, then half (no high half: fx_near)
  const int s = fx_clz32(fx_high(o.mw) | fx_high(o.mx) | fx_high(o.my) | fx_high(o.mz)) - 1;
  o.mw = o.mw << s >> 1;
  o.mx = o.mx << s >> 1;
  o.my = o.my << s >> 1;
  o.mz = o.mz << s >> 1;
  o.e -= s - 1;
  return fx_joined(o);
}
// Whether d = fx_qsub(a, b) came out below 2^-6 of the larger of a and b.
FX_FN int fx_near(fx_quat d, fx_quat a, fx_quat b) {
  return d.e < (a.e > b.e ? a.e : b.e) - 5;
}

// m with sign s but for the 1 that a negative one lacks
FX_FN fx_u64 fx_flip(fx_u64 m, int32_t s) { return m ^ fx_mask(s); }
// The sum of four products of magnitudes, each cut, with signs s1 to s4.
FX_FN fx_i64 fx_sum4(fx_u64 a1, fx_u64 b1, int32_t s1, fx_u64 a2, fx_u64 b2, int32_t s2, fx_u64 a3,
                     fx_u64 b3, int32_t s3, fx_u64 a4, fx_u64 b4, int32_t s4) {
  const uint32_t minus = (uint32_t)-(s1 + s2 + s3 + s4);
  return (fx_i64)((fx_flip(fx_mulhi(a1, b1), s1) + fx_flip(fx_mulhi(a2, b2), s2) + minus) +
                  (fx_flip(fx_mulhi(a3, b3), s3) + fx_flip(fx_mulhi(a4, b4), s4)));
}
// Whether all four terms are below 2^44 of at most 2^60 (by the high halves)
// and not all zero.
FX_FN int fx_lost(fx_u64 a1, fx_u64 b1, fx_u64 a2, fx_u64 b2, fx_u64 a3, fx_u64 b3, fx_u64 a4,
                  fx_u64 b4) {
  const fx_u64 most = (fx_u64)fx_high(a1) * fx_high(b1) | (fx_u64)fx_high(a2) * fx_high(b2) |
                      (fx_u64)fx_high(a3) * fx_high(b3) | (fx_u64)fx_high(a4) * fx_high(b4);
  return most < (1ull << 44) && ((a1 && b1) || (a2 && b2) || (a3 && b3) || (a4 && b4));
}
// The product; `strict`: of two factors of the map, odd as said above.
FX_FN fx_quat fx_hamilton(fx_quat a, fx_quat b, int strict) {
  fx_quat o;
  o.w = fx_sum4(a.mw, b.mw, a.sw ^ b.sw, a.mx, b.mx, ~(a.sx ^ b.sx), a.my, b.my, ~(a.sy ^ b.sy),
                a.mz, b.mz, ~(a.sz ^ b.sz));
  o.x = fx_sum4(a.mw, b.mx, a.sw ^ b.sx, a.mx, b.mw, a.sx ^ b.sw, a.my, b.mz, a.sy ^ b.sz, a.mz,
                b.my, ~(a.sz ^ b.sy));
  o.y = fx_sum4(a.mw, b.my, a.sw ^ b.sy, a.mx, b.mz, ~(a.sx ^ b.sz), a.my, b.mw, a.sy ^ b.sw, a.mz,
                b.mx, a.sz ^ b.sx);
  o.z = fx_sum4(a.mw, b.mz, a.sw ^ b.sz, a.mx, b.my, a.sx ^ b.sy, a.my, b.mx, ~(a.sy ^ b.sx), a.mz,
                b.mw, a.sz ^ b.sw);
  o.e = a.e + b.e + 2;
  o.odd = a.odd | b.odd;
  o = fx_norm(fx_split(o));
  if (strict) {
    // no small component on one side: its product with the other side's
    // largest is a term of 2^44 or more in every component
    const uint32_t p = fx_least(fx_least(fx_high(a.mw), fx_high(a.mx)), fx_least(fx_high(a.my), fx_high(a.mz)));
    const uint32_t q = fx_least(fx_least(fx_high(b.mw), fx_high(b.mx)), fx_least(fx_high(b.my), fx_high(b.mz)));
    const int real = fx_high(o.mx | o.my | o.mz) < (1u << 10);
    if ((p < (1u << 15) && q < (1u << 15)) || real)
      o.odd |= (real && ((a.mx | a.my | a.mz) || (b.mx | b.my | b.mz))) ||
               fx_lost(a.mw, b.mw, a.mx, b.mx, a.my, b.my, a.mz, b.mz) ||
               fx_lost(a.mw, b.mx, a.mx, b.mw, a.my, b.mz, a.mz, b.my) ||
               fx_lost(a.mw, b.my, a.mx, b.mz, a.my, b.mw, a.mz, b.mx) ||
               fx_lost(a.mw, b.mz, a.mx, b.my, a.my, b.mx, a.mz, b.mw);
  }
  return o;
}
// The product of two factors of the map.
FX_FN fx_quat fx_qmul(fx_quat a, fx_quat b) { return fx_hamilton(a, b, 1); }
// ... and of a power and its base.  Their vectors are parallel, so the terms
// of a component are small together on a 2^-8 of all bases; a later factor's
// terms then count beside them, and the product with it is tested.
FX_FN fx_quat fx_qpower(fx_quat a, fx_quat b) { return fx_hamilton(a, b, 0); }
FX_FN fx_quat fx_conj(fx_quat a) {
  a.sx = ~a.sx;
  a.sy = ~a.sy;
  a.sz = ~a.sz;
  return fx_joined(a);
}
// Maps whose roots all lie on the real axis or in a coordinate plane through
// it, but for 2^-9 of their size: bits 0 to 2, components x to z small in
// every root; bits 3 to 5, and not zero in all of them.  0 for other maps.
FX_FN int fx_beside_of(const double (*r)[4], int n, int top) {
  int small = 7, some = 0;
  for (int i = 0; i < n; i++)
    for (int c = 0; c < 3; c++) {
      if (fx_field(r[i][c + 1]) >= top + 1022 - 9) small &= ~(1 << c);
      if (r[i][c + 1] != 0.0) some |= 8 << c;
    }
  return small == 7 || small == 3 || small == 5 || small == 6 ? small | some : 0;
}
// Whether q lies beside that axis or plane: every difference q - root then has
// those components below 2^-9 of its largest (top, the larger exponent of q
// and the roots) and not zero.  A single plane needs both components off it
// small; on the axis each counts, for all vector parts are q's multiples.
FX_FN int fx_beside(int map, double x, double y, double z, int top) {
  const int least = top + 1022 - 9;
  const int s = (fx_field(x) < least) | (fx_field(y) < least) << 1 | (fx_field(z) < least) << 2;
  const int some = (x != 0.0) | (y != 0.0) << 1 | (z != 0.0) << 2 | map >> 3;
  const int small = map & 7, hit = s & some & small;
  return hit && (small == 7 || (s & small) == small);
}
// v 2^k for a normal result, by the exponent field (0, infinities and NaN stay).
FX_FN double fx_scale(double v, int k) {
  const fx_u64 b = fx_bits(v);
  const int f = (int)(b >> 52) & 0x7ff;
  if (f == 0 || f == 0x7ff) return v;
  if (f + k <= 0) return 0.0 * v;
  if (f + k >= 0x7ff) return fx_from((b & 0x8000000000000000ull) | 0x7ff0000000000000ull);
  return fx_from(b + ((fx_u64)(fx_i64)k << 52));
}
// odd where a component 2 w c has fewer than 33 bits and is not zero
FX_FN fx_quat fx_qsq(fx_quat a) {
  fx_quat o;
  o.w = (fx_i64)(fx_mulhi(a.mw, a.mw) - fx_mulhi(a.mx, a.mx) - fx_mulhi(a.my, a.my) -
                 fx_mulhi(a.mz, a.mz));
  o.sw = fx_sign(o.w);
  o.mw = fx_abs(o.w);
  o.mx = fx_mulhi(a.mw << 1, a.mx);
  o.my = fx_mulhi(a.mw << 1, a.my);
  o.mz = fx_mulhi(a.mw << 1, a.mz);
  o.sx = a.sw ^ a.sx;
  o.sy = a.sw ^ a.sy;
  o.sz = a.sw ^ a.sz;
  o.odd = a.odd;
  if (fx_least(fx_high(o.mx), fx_least(fx_high(o.my), fx_high(o.mz))) == 0)
    o.odd |= a.mw && ((a.mx && !fx_high(o.mx)) || (a.my && !fx_high(o.my)) || (a.mz && !fx_high(o.mz)));
  o.e = a.e + a.e + 2;
  return fx_norm(o);
}
