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
// A Hamilton product costs 16 FP64 instructions, as much of that pipe's time
// as 1024 integer ones would take on theirs.  Here a quaternion is four
// 64-bit integers with one exponent, value c 2^(e - 62), the largest |c| in
// [2^61, 2^62): a product is 16 high halves of 64-bit products and a
// renormalization, about 230 integer instructions.  Against |a b| it is off
// by at most 2^-55 (four truncated halves, and the largest component of a
// product of norm 2^58 is at least 2^57), FP64's fused product by 2^-52.
typedef struct {
  fx_i64 w, x, y, z;
  int e;
} fx_quat;

// v's mantissa in units of 2^(top - 62), top at least v's exponent; 0 for
// zeros and subnormals.
FX_FN fx_i64 fx_align(double v, int top) {
  const fx_u64 b = fx_bits(v);
  const int f = (int)(b >> 52) & 0x7ff;
  const int sh = 2 + top - (f - 1022);
  if (f == 0 || sh > 63) return 0;
  const fx_i64 m = (fx_i64)(((b << 11) | 0x8000000000000000ull) >> sh);
  return (fx_i64)b < 0 ? -m : m;
}
FX_FN fx_quat fx_quat_of(double w, double x, double y, double z) {
  int f = (int)(fx_bits(w) >> 52) & 0x7ff, g = (int)(fx_bits(x) >> 52) & 0x7ff;
  f = f > g ? f : g;
  g = (int)(fx_bits(y) >> 52) & 0x7ff;
  f = f > g ? f : g;
  g = (int)(fx_bits(z) >> 52) & 0x7ff;
  f = f > g ? f : g;
  fx_quat q;
  q.e = f - 1022;
  q.w = fx_align(w, q.e);
  q.x = fx_align(x, q.e);
  q.y = fx_align(y, q.e);
  q.z = fx_align(z, q.e);
  return q;
}
FX_FN fx_quat fx_norm(fx_quat q) {
  // the bits of |c| - 1 or |c|: enough to place the top bit (none: 0 or -1)
  const fx_u64 any = (fx_u64)((q.w ^ q.w >> 63) | (q.x ^ q.x >> 63) | (q.y ^ q.y >> 63) |
                              (q.z ^ q.z >> 63));
  const int s = any ? fx_clz(any) - 2 : 61;
  q.w = (fx_i64)((fx_u64)q.w << s);
  q.x = (fx_i64)((fx_u64)q.x << s);
  q.y = (fx_i64)((fx_u64)q.y << s);
  q.z = (fx_i64)((fx_u64)q.z << s);
  q.e -= s;
  return q;
}
// a - b, each kept to 2^-61 of the larger one's largest component: off by
// at most 2^-53 of |a - b| unless fx_near says that more bits cancelled.
FX_FN fx_quat fx_qsub(fx_quat a, fx_quat b) {
  fx_quat o;
  o.e = (a.e > b.e ? a.e : b.e) + 1;
  const int sa = o.e - a.e < 63 ? o.e - a.e : 63, sb = o.e - b.e < 63 ? o.e - b.e : 63;
  o.w = (a.w >> sa) - (b.w >> sb);
  o.x = (a.x >> sa) - (b.x >> sb);
  o.y = (a.y >> sa) - (b.y >> sb);
  o.z = (a.z >> sa) - (b.z >> sb);
  return fx_norm(o);
}
// Whether d = fx_qsub(a, b) came out below 2^-6 of the larger of a and b.
FX_FN int fx_near(fx_quat d, fx_quat a, fx_quat b) {
  return d.e < (a.e > b.e ? a.e : b.e) - 5;
}
FX_FN fx_quat fx_qmul(fx_quat a, fx_quat b) {
  fx_quat o;
  o.w = fx_smulhi(a.w, b.w) - fx_smulhi(a.x, b.x) - fx_smulhi(a.y, b.y) - fx_smulhi(a.z, b.z);
  o.x = fx_smulhi(a.w, b.x) + fx_smulhi(a.x, b.w) + fx_smulhi(a.y, b.z) - fx_smulhi(a.z, b.y);
  o.y = fx_smulhi(a.w, b.y) - fx_smulhi(a.x, b.z) + fx_smulhi(a.y, b.w) + fx_smulhi(a.z, b.x);
  o.z = fx_smulhi(a.w, b.z) + fx_smulhi(a.x, b.y) - fx_smulhi(a.y, b.x) + fx_smulhi(a.z, b.w);
  o.e = a.e + b.e + 2;
  return fx_norm(o);
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
FX_FN fx_quat fx_qsq(fx_quat a) {
  fx_quat o;
  o.w = fx_smulhi(a.w, a.w) - fx_smulhi(a.x, a.x) - fx_smulhi(a.y, a.y) - fx_smulhi(a.z, a.z);
  o.x = fx_smulhi(a.w << 1, a.x);
  o.y = fx_smulhi(a.w << 1, a.y);
  o.z = fx_smulhi(a.w << 1, a.z);
  o.e = a.e + a.e + 2;
  return fx_norm(o);
}
