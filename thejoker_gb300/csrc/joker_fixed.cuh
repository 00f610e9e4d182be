// The unit-K velocity column and the epoch sums in 64-bit fixed point.
//
// One FP64 instruction of a warp holds this GPU's FP64 pipe for 16 cycles of
// an SM, an FP32 or integer one a quarter of a cycle, so the column and its
// sums are carried as integers: 62-bit values in two 31-bit limbs, a product
// one 32 x 32 -> 64 multiply and two high halves.  FP32 serves where a term is
// already small (the starter, the first Newton step, the last correction).
// Every fixed-point step is good to about 2^-59 whatever the phase; near
// pericentre the column's error is that over f'^2, f' = 1 - e cos E.  In doubles
// the same formulas round the phase by 2^-53 of the unreduced angle, over f'^2
// too, and the rest by 2^-53 over f': as_exact() below is where the first is no
// larger.
//
// Notation: Qn is a real number times 2^n held in an integer.  The eccentric
// anomaly and the mean anomaly are in turns (Q32, Q63, Q64); a limb pair
// (h, l) stands for h 2^31 + l with 0 <= l < 2^31.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define JOKER_FX __host__ __device__ __forceinline__
#else
#define JOKER_FX inline
#endif
#include "joker_trig_table.cuh"

namespace joker {
namespace fx {

constexpr int64_t ONE61 = (int64_t)1 << 61;
constexpr int64_t ONE62 = (int64_t)1 << 62;
constexpr int64_t PI_4_Q62 = 0x3243F6A8885A308D;
constexpr int32_t PI_4_H = (int32_t)(PI_4_Q62 >> 31), PI_4_L = (int32_t)(PI_4_Q62 & 0x7fffffff);
constexpr int64_t LN2_Q62 = 0x2C5C85FDF473DE6A;
constexpr uint64_t INV_2PI_Q66 = 0xA2F9836E4E44152Aull, INV_2PI_Q64 = 0x28BE60DB9391054Aull;
constexpr float TWO_PI_FX = 6.28318530717958648f;

// Largest |ri|: 2^16 r^2 stays below 1/2.  A node is within 2^20, and
// Markley's starter within 4.4e-4 rad (300000) of the anomaly.
constexpr int32_t RI_MAX = 1850000;

struct limbs { int32_t h, l; };

JOKER_FX int64_t wide(int32_t a, int32_t b) { return (int64_t)a * (int64_t)b; }
JOKER_FX limbs split(int64_t v) {
    limbs r;
    r.h = (int32_t)(v >> 31);
    r.l = (int32_t)(v & 0x7fffffff);
    return r;
}
JOKER_FX int64_t join(limbs a) { return ((int64_t)a.h << 31) + a.l; }
// node k of the table, k in [0, TRIG_N)
JOKER_FX trig_entry trig_node(int k) {
#ifdef __CUDA_ARCH__
    const longlong2 v = __ldg(reinterpret_cast<const longlong2 *>(kTrig) + k);
    trig_entry t;
    t.s = v.x;
    t.c = v.y;
    return t;
#elif defined(__CUDACC__)
    return trig_entry();                 // no host caller
#else
    return kTrig[k];
#endif
}
JOKER_FX int32_t hi32(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return (int32_t)(wide(a, b) >> 32);
#endif
}
JOKER_FX uint32_t uhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// a b 2^-62 to 5 units (truncated): Qi x Qj -> Q(i + j - 62).  The sum of the
// two high halves stays in 32 bits: each is below 2^30 in size.
JOKER_FX int64_t mul(limbs a, limbs b) {
    return wide(a.h, b.h) + 2 * (int64_t)(hi32(a.h, b.l) + hi32(a.l, b.h));
}
// u v, with u v's 64 bits: the three partial products above 2^32 of the four
JOKER_FX uint64_t hi64(uint64_t u, uint64_t v) {
    const uint32_t uh = (uint32_t)(u >> 32), ul = (uint32_t)u;
    const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
    return (uint64_t)uh * vh + (((uint64_t)uh * vl) >> 32) + (((uint64_t)ul * vh) >> 32);
}

#ifdef __CUDA_ARCH__
JOKER_FX int clz64(uint64_t v) { return __clzll((long long)v); }
JOKER_FX float rcp_a(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
JOKER_FX float rsqrt_a(float x) { float r; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
JOKER_FX float lg2_a(float x) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
JOKER_FX float ex2_a(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
JOKER_FX int32_t rint_a(float x) { return __float2int_rn(x); }   // saturates, NaN -> 0
JOKER_FX float fma_a(float a, float b, float c) { return __fmaf_rn(a, b, c); }
JOKER_FX float max_a(float a, float b) { return fmaxf(a, b); }
JOKER_FX int32_t max_a(int32_t a, int32_t b) { return max(a, b); }
#else
JOKER_FX int clz64(uint64_t v) { return v ? __builtin_clzll(v) : 64; }
JOKER_FX float rcp_a(float x) { return 1.0f / x; }
JOKER_FX float rsqrt_a(float x) { return 1.0f / std::sqrt(x); }
JOKER_FX float lg2_a(float x) { return std::log2(x); }
JOKER_FX float ex2_a(float x) { return std::exp2(x); }
JOKER_FX int32_t rint_a(float x) {
    if (!(x == x)) return 0;
    if (x >= 2147483648.0f) return 2147483647;
    if (x <= -2147483648.0f) return (int32_t)0x80000000;
    return (int32_t)std::nearbyint(x);
}
JOKER_FX float fma_a(float a, float b, float c) { return std::fma(a, b, c); }
JOKER_FX float max_a(float a, float b) { return a < b ? b : a; }
JOKER_FX int32_t max_a(int32_t a, int32_t b) { return a < b ? b : a; }
#endif

// num / den in Q61 for 0 < den < 2^62 and |num| <= den (1 + 2^-40), to 16
// units: the quotient in two digits, each the product with an FP32 reciprocal
// that one Newton step takes to 2^-30.  The first digit is within 2 units of
// Q30 (rounded, and the middle of the bits that nh drops added), so the
// remainder is below 2^33 and the second loses 8 (dropped bits), 4 (the
// reciprocal) and 3 (truncations) units.
JOKER_FX int64_t div61(int64_t num, int64_t den) {
    const int sh = clz64((uint64_t)den) - 2;
    const int64_t dn = den << sh, nn = num << sh;        // dn in [2^61, 2^62)
    const int32_t dh = (int32_t)(dn >> 31), dl = (int32_t)(dn & 0x7fffffff);
    // r = 2^60 / dh in (2^29, 2^30]
    int32_t r = rint_a(rcp_a((float)dh) * 0x1p60f);
    const int64_t t = ((int64_t)1 << 60) - wide(dh, r);  // |t| < 2^38
    r += (hi32(r, (int32_t)(t >> 8)) + (1 << 19)) >> 20;
    const int32_t nh = (int32_t)(nn >> 32);
    const int32_t q0 = (int32_t)((wide(nh, r) + (5ll << 27)) >> 29);     // Q30
    const int64_t rem = nn - 2 * wide(q0, dh) - (wide(q0, dl) >> 30);
    return ((int64_t)q0 << 31) + (wide((int32_t)(rem >> 3), r) >> 27);
}

// A signed 64-bit integer as a float with a float's relative accuracy.
JOKER_FX float to_float(int64_t v) {
    const int32_t l = (int32_t)(uint32_t)v;               // the nearest multiple of 2^32 and
    const int32_t h = (int32_t)((v - l) >> 32);           // the signed rest
    return fma_a((float)h, 0x1p32f, (float)l);
}

// sin and cos (Q61) of a node's angle plus r (Q62), |r| < 2^-8.4: the Taylor
// series of sin r and cos r to r^5, then the addition formulas.
JOKER_FX void turn_by(trig_entry tab, limbs S, limbs C, int64_t rq, int64_t &s1, int64_t &c1) {
    const limbs r = split(rq);
    const int32_t rh = (int32_t)(rq >> 23);                           // 2^39 r
    const int64_t R2 = mul(r, r);                                     // r^2 (Q62)
    const int32_t R2h = (int32_t)(R2 >> 14);                          // 2^48 r^2
    const int32_t R4h = hi32(R2h, R2h);                               // 2^64 r^4
    const int32_t g = hi32(R2h, 715827883) - hi32(R4h, 546);          // 2^48 (r^2/6 - r^4/120)
    const limbs sr = split(rq - (wide(rh, g) >> 25));                 // sin r (Q62)
    const limbs nc = split((R2 >> 1) - hi32(R4h, 44739243));          // 1 - cos r (Q62)
    s1 = tab.s + mul(sr, C) - mul(nc, S);
    c1 = tab.c - mul(sr, S) - mul(nc, C);
}

// ------------------------------------------------- doubles to fixed point
JOKER_FX uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
JOKER_FX double double_of(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
JOKER_FX uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
JOKER_FX float float_of(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}
// |v| 2^k for a magnitude v, bits below the unit dropped; k >= 64 is not asked for
JOKER_FX uint64_t shift(uint64_t v, int k) {
    return k >= 0 ? v << k : (k > -64 ? v >> -k : 0);
}
JOKER_FX int64_t clamp62(int64_t v) { return v > ONE62 - 1 ? ONE62 - 1 : v; }
JOKER_FX int64_t twice(int64_t v) { return clamp62(v + v); }
// x in [0, 1] (-0 too) as Q62, at most 1 - 2^-62
JOKER_FX int64_t fixed62(double x) {
    const uint64_t b = bits_of(x);
    return clamp62((int64_t)shift((b & 0xfffffffffffffull) | 0x10000000000000ull,
                                  ((int)(b >> 52) & 0x7ff) - 1013));
}
// x 2^q, the bits below the unit dropped, for |x| 2^q < 2^63
JOKER_FX int64_t fixed_signed(double x, int q) {
    const uint64_t b = bits_of(x);
    const int be = (int)(b >> 52) & 0x7ff;
    if (be == 0) return 0;
    const int64_t v = (int64_t)shift((b & 0xfffffffffffffull) | 0x10000000000000ull,
                                     be - 1075 + q);
    return (b >> 63) ? -v : v;
}
// a (radians, |a| < 2^10) in turns mod 1, Q64
JOKER_FX uint64_t turns64(double a) {
    const uint64_t b = bits_of(a);
    const int be = (int)(b >> 52) & 0x7ff;
    const uint64_t mn = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
    const uint64_t t = shift(hi64(mn, INV_2PI_Q66), be - 1024);
    return (b >> 63) ? 0 - t : t;
}
// 2^124 / dn for dn in [2^61, 2^62), relative error below 2^-58: an FP32
// reciprocal, one Newton step to 30 bits, one to 60
JOKER_FX uint64_t rcp62(uint64_t dn) {
    const int32_t dh = (int32_t)(dn >> 31), dl = (int32_t)(dn & 0x7fffffff);
    int32_t r = rint_a(rcp_a((float)dh) * 0x1p60f);
    const int64_t t = ((int64_t)1 << 60) - wide(dh, r);
    r += hi32(r, (int32_t)(t >> 8)) >> 20;
    // 2^91 - r dn, exact (mod 2^64)
    const int64_t rem = 0 - (int64_t)((uint64_t)wide(r, dl) + ((uint64_t)wide(r, dh) << 31));
    int32_t rh = (int32_t)(rem >> 31);                    // units of 2^-60
    rh += hi32(rh, rh) >> 28;                             // t + t^2
    return ((uint64_t)r << 33) + (uint64_t)(wide(rh, r) >> 27);
}
// sqrt(y) (Q62) for y (Q62) in (0, 2^62]: a Q31 root from FP32, refined twice
JOKER_FX int64_t sqrt62(int64_t y) {
    const float yf = to_float(y) * 0x1p-62f;
    const float h = rsqrt_a(yf);
    int32_t s = rint_a(yf * h * 0x1p31f);
    const uint32_t s1 = (uint32_t)s + (uint32_t)rint_a(to_float(y - wide(s, s)) * 0.5f * h * 0x1p-31f);
    s = (int32_t)(s1 > 0x7fffffffu ? 0x7fffffffu : s1);   // y near 1: at most 2^31 - 1
    return ((int64_t)s << 31) + (int64_t)rint_a(to_float(y - wide(s, s)) * 0.5f * h);
}

// 2^(n + f) for f (Q62) in [0, 1) and a normal result: 2^(j/512) times
// e^z = 1 + z + z^2/2 + z^3 (1/6 + z/24 + z^2/120), z < 2^-9.5, good to 2^-58
// before the rounding to a double (the truncations leave 0 to -16 units of
// Q61; 7 are added).
JOKER_FX double exp2_fixed(int n, int64_t f) {
#ifdef __CUDA_ARCH__
    const limbs T = split(__ldg(kExp2 + (int)(f >> 53)));
#elif defined(__CUDACC__)
    const limbs T = split(0);            // no host caller
#else
    const limbs T = split(kExp2[f >> 53]);
#endif
    const limbs z = split(mul(split(f & (((int64_t)1 << 53) - 1)), split(LN2_Q62)));
    const int64_t zq = join(z);
    const uint32_t zz = (uint32_t)(zq >> 21);                        // 2^41 z
    const float zf = (float)zz * 0x1p-41f;
    const uint32_t h = 2863311531u +                                 // 2^34 / 6
                       (uint32_t)rint_a(zf * fma_a(zf, 1.0f / 120.0f, 1.0f / 24.0f) * 0x1p34f);
    const uint32_t z3 = uhi32(uhi32(zz, zz), zz);                    // 2^59 z^3
    const int64_t p = zq + (mul(z, z) >> 1) + 2 * (int64_t)uhi32(z3, h);
    const int64_t v = join(T) + mul(T, split(p));                    // Q61, [1, 2)
    return double_of(((uint64_t)(1022 + n) << 52) + (uint64_t)((v + 263) >> 9));
}

// Whether an orbit's column is at least as exact in fixed point as in doubles,
// for times |dt| 2^tsh < 2^62 whose largest is above half of that: span / P is
// then above 2^(s-5).  Column errors (rms near pericentre) in fixed point over
// those in doubles, measured against quadruple precision:
//   span / P        1 - e = 2^-3..2^-2   2^-6..2^-5   2^-8..2^-7   2^-10..2^-9
//   1/2 .. 1                  0.27          0.34         0.43          0.70
//   1/4 .. 1/2                0.43          0.68         0.80          1.4
//   1/8 .. 1/4                0.59          1.4          1.6           2.7
//   1/256 .. 1/8              0.42..0.77    2.2..2.9     3.1..9        5..29
JOKER_FX bool as_exact(int tsh, double P, double e) {
    const int s = 1088 - tsh - ((int)(bits_of(P) >> 52) & 0x7ff);
    // by the upper word (a sign or a NaN is Orbit::init's matter): 63/64 and 7/8
    return s >= 4 || (int32_t)(bits_of(e) >> 32) <= (s == 3 ? 0x3fef8000 : 0x3fec0000);
}

// One orbit against one star's time scale.
struct Orbit {
    uint32_t Ri;               // 2^64 turns per unit of the integer epoch times:
    uint64_t Rf;               //   Ri + Rf 2^-64
    uint64_t ph0;              // phase at integer time 0, Q64 turns
    limbs e, ep;               // e (Q62), e / 2 pi (Q64)
    limbs A, B;                // cos w, -sin w sqrt(1 - e^2) (Q62)
    int64_t D;                 // e cos w (Q61)
    float ef, omef, a1f;       // e, 1 - e, Markley's a1
    float ef30;                // e 2^-30
    float cs;                  // 2^(61 - sg): scale of the last correction
    int32_t psg;               // 2^sg
    int32_t far_r;             // the largest |ri| and |dl| of the columns so far
    float far_d;

    // No column yet; what bad() reads of an orbit that init refused or never saw.
    JOKER_FX void clear() { far_r = 0; far_d = cs = 0.0f; }

    // Integer times are t = dt 2^tsh - t0.  False: outside the fixed-point
    // form's range, whose lines are the phase's 2^32 turns per time scale,
    // angles below 2^10, and e <= 0.999 (see as_exact for its exactness).
    JOKER_FX bool init(int tsh, int64_t t0, double P, double e_, double om, double M0) {
        clear();
        const uint64_t pb = bits_of(P);
        const int pe = (int)(pb >> 52);                       // sign bit too
        const int s = 1088 - tsh - pe;
        const int oe = (int)(bits_of(om) >> 52) & 0x7ff, me = (int)(bits_of(M0) >> 52) & 0x7ff;
        if (!(pe > 0 && pe < 2047 && s <= 32 && e_ >= 0.0 && e_ <= 0.999 && oe < 1033 && me < 1033))
            return false;
        const uint64_t X = rcp62(((pb & 0xfffffffffffffull) | 0x10000000000000ull) << 9);
        Rf = shift(X, s);
        Ri = s > 0 ? (uint32_t)(X >> (64 - s)) : 0u;
        ph0 = 0 - turns64(M0);
        if (t0 != 0) {
            const uint64_t u = (uint64_t)(t0 < 0 ? -t0 : t0);
            const uint64_t p = u * Ri + hi64(u, Rf);
            ph0 += t0 < 0 ? 0 - p : p;
        }
        const int64_t e62 = fixed62(e_);
        e = split(e62);
        ep = split((int64_t)hi64((uint64_t)e62 << 2, INV_2PI_Q64));
        ef = to_float(e62) * 0x1p-62f;
        ef30 = ef * 0x1p-30f;
        omef = to_float(ONE62 - e62) * 0x1p-62f;
        a1f = 1.6f * 3.14159265358979f / (9.8696044011f - 6.0f) * rcp_a(1.0f + ef);
        const int sg = 5 + 126 - (int)(float_bits(omef) >> 23);
        cs = float_of((uint32_t)(127 + 61 - sg) << 23);
        psg = 1 << sg;
        // omega: the node nearest to |turn| and the rest of the angle, r = 2 pi 2^-64 rest
        const uint64_t w = turns64(om);
        const bool neg = (int64_t)w < 0;
        const uint64_t aw = neg ? 0 - w : w;                   // [0, 2^63]
        const int k = (int)((aw + (1ull << 52)) >> 53);        // 0..1024
        const trig_entry tab = trig_node(k);
        const int64_t rho = (int64_t)(aw - ((uint64_t)k << 53)) << 9;   // r = rho 2^-62 pi/4 2^-8
        int64_t sw, cw;
        turn_by(tab, split(tab.s), split(tab.c), mul(split(rho), split(PI_4_Q62)) >> 8, sw, cw);
        D = mul(e, split(cw));
        A = split(twice(cw));
        const int64_t om2 = ONE62 - mul(e, e);
        const int64_t b = mul(split(clamp62(sqrt62(clamp62(om2)))), split(sw));
        B = split(twice(neg ? b : -b));
        return true;
    }
    // The column m = cos(w + f) + e cos(w) (Q61) at integer time t.
    JOKER_FX int64_t column(uint64_t t) {
        // phase in turns mod 1, Q64; its sign and its size in [0, 1/2] (to a
        // unit: the complement stands for the negative)
        const uint64_t turn = ph0 + t * Ri + hi64(t, Rf);
        const int64_t sgn = (int64_t)turn >> 63;
        const uint64_t x = turn ^ (uint64_t)sgn;
        const int64_t x63 = (int64_t)(x >> 1);
        const float xf = fma_a((float)(uint32_t)(x >> 32), TWO_PI_FX * 0x1p-32f,
                               (float)(uint32_t)x * (TWO_PI_FX * 0x1p-64f));
        // Markley's starter in FP32 (markley_starter_f32), in Q32 turns
        const float PI = 3.14159265358979f;
        const float alpha = fma_a(a1f, PI - xf, 3.0f * 9.8696044011f / (9.8696044011f - 6.0f));
        const float d = fma_a(alpha, ef, 3.0f * omef);
        const float x2 = xf * xf;
        const float ad = alpha * d;
        const float q = fma_a(ad, 2.0f * omef, -x2);
        const float r = xf * fma_a(ad, fma_a(3.0f, d, -3.0f * omef), x2);
        const float qq = q * q;
        const float disc = max_a(fma_a(qq, q, r * r), 1e-30f);
        const float w = ex2_a(0.6666667f * lg2_a(fma_a(disc, rsqrt_a(disc), r)));
        const float den3 = fma_a(w, w + q, qq);
        const float E0 = fma_a(xf, den3, 2.0f * r * w) * rcp_a(den3 * d);
        int32_t i0 = rint_a(E0 * (0x1p32f / TWO_PI_FX));
        i0 = i0 < 0 ? 0 : i0;
        // node k of the table (2048 a turn) nearest to it
        const int k = (int)(((uint32_t)i0 + (1u << 20)) >> 21);          // 0..1024
        const trig_entry tab = trig_node(k);
        const limbs S = split(tab.s), C = split(tab.c);                   // Q61
        const float Sf = (float)S.h, Cf = (float)C.h;                     // 2^30 sin, cos
        int32_t ri = (int32_t)((uint32_t)i0 - ((uint32_t)k << 21));       // Q32 turns
        // first step: f(E0) to 2^-34 turns, Halley's correction in FP32
        const float rf = (float)ri * (TWO_PI_FX * 0x1p-32f);
        const float hr2 = 0.5f * rf * rf;
        const float srf = fma_a(rf * hr2, -1.0f / 3.0f, rf);
        const float ds0 = fma_a(Cf, srf, -Sf * hr2);                      // 2^30 (sin E0 - S)
        const float c0 = fma_a(-Sf, srf, fma_a(-Cf, hr2, Cf));
        const int64_t f0i = ((int64_t)i0 << 31) - x63 - wide(ep.h, S.h);  // Q63
        const float f0 = fma_a((float)(int32_t)(f0i >> 21), TWO_PI_FX * 0x1p-42f, -ef30 * ds0);
        const float f2 = ef30 * (Sf + ds0);
        const float f1 = fma_a(-ef30, c0, 1.0f);
        const float dl0 = f0 * f1 * rcp_a(fma_a(f1, f1, -0.5f * f0 * f2));   // -delta
        ri -= rint_a(dl0 * (0x1p32f / TWO_PI_FX));
        far_r = max_a(far_r, ri < 0 ? -ri : ri);
        // sin E1, cos E1 (Q61) from the node and r = 2 pi ri 2^-32 (Q62)
        const int32_t rho = (int32_t)((uint32_t)ri << 10);
        int64_t s1, c1;
        turn_by(tab, S, C, (wide(rho, PI_4_H) >> 8) + (hi32(rho, PI_4_L) >> 7), s1, c1);
        // last step: f(E1) (Q63 turns) in fixed point, the correction in FP32
        const limbs s1l = split(s1);
        const int64_t E1 = ((int64_t)k << 52) + ((int64_t)ri << 31);
        const float u0 = to_float(E1 - x63 - mul(ep, s1l)) * (TWO_PI_FX * 0x1p-63f);
        const int64_t omc = ONE61 - c1;
        const float omcf = fma_a((float)(int32_t)(omc >> 32), 0x1p-29f,
                                 (float)(uint32_t)omc * 0x1p-61f);
        const float i1 = rcp_a(fma_a(ef, omcf, omef));
        const float s1f = (float)s1l.h * 0x1p-30f, c1f = 1.0f - omcf;
        const float u = -u0 * i1;
        const float dl = fma_a(u * u, -0.5f * ef * s1f * i1, u);
        const float hd2 = -0.5f * dl * dl;
        const float dsf = fma_a(c1f, dl, hd2 * s1f) * cs;
        const float dcf = fma_a(-s1f, dl, hd2 * c1f) * cs;
        far_d = max_a(far_d, fabsf(dl));
        const limbs cE = split(c1 + wide(rint_a(dcf), psg));
        const limbs sE = split(s1 + wide(rint_a(dsf), psg));
        // (A cos E + B sin E - D) / (1 - e cos E) + D
        const int64_t num = mul(A, cE) + (mul(B, sE) ^ sgn) - D;
        return div61(num, ONE61 - mul(e, cE)) + D;
    }

    // Whether an iteration left its range in a column so far.
    JOKER_FX bool bad() const { return far_r > RI_MAX || !(far_d * cs < 0x1p30f); }
};

// A signed 96-bit sum of 64-bit terms.
struct Sum96 {
    uint64_t lo;
    int32_t hi;
    JOKER_FX void zero() { lo = 0; hi = 0; }
    JOKER_FX void add(int64_t v) { add(v, (int32_t)(v >> 63)); }
    JOKER_FX void add(int64_t v, int32_t vh) {
#ifdef __CUDA_ARCH__
        uint32_t l = (uint32_t)lo, m = (uint32_t)(lo >> 32);
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
            : "+r"(l), "+r"(m), "+r"(hi) : "r"((uint32_t)v), "r"((uint32_t)(v >> 32)), "r"(vh));
        lo = ((uint64_t)m << 32) | l;
#else
        lo += (uint64_t)v;
        hi += vh + (lo < (uint64_t)v);
#endif
    }
    JOKER_FX double value() const {
        const int64_t top = (int64_t)(((uint64_t)(uint32_t)hi << 32) | (lo >> 32));
        return (double)top * 4294967296.0 + (double)(uint32_t)lo;
    }
#ifdef __CUDACC__
    // the sum over the 32 lanes of a warp, in every lane
    __device__ __forceinline__ void warp_sum() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int64_t v = (int64_t)__shfl_xor_sync(0xffffffffu, (unsigned long long)lo, o);
            add(v, __shfl_xor_sync(0xffffffffu, hi, o));
        }
    }
#endif
};

// One epoch's integers: time, weight (ivar 2^-ew, Q62), velocity (y' 2^-ey,
// Q62), the trend columns j >= 2 (T_j 2^-eT_j, Q62).  64 bytes.
struct alignas(16) EpochFx {
    uint64_t t;
    limbs w;
    limbs y;
    limbs T[4];
    int64_t pad;
};

}  // namespace fx
}  // namespace joker
