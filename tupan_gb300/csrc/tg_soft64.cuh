// Correctly rounded binary64 multiplication, reciprocal and square root on
// the integer pipe.
//
// Why: an FP64 warp instruction costs this GPU's SM 19 cycles, an IEEE
// division 86 and a square root 143; a 32-bit integer one half a cycle, on a
// pipe that is otherwise idle.  Measured (SM cycles a warp, 16 warps an SM):
// product 14.4 against 19.1, reciprocal 16 against 86, root 29 against 143.
// Every result is the IEEE round-to-nearest-even one (1.6e9 random and
// structured operands on the GPU against its own division and root), so
// sweeps built on these keep the reference's bits.
//
// Method (from the mathematics): significands are held as integers.  A
// product is the exact 106-bit integer product, normalised by at most one
// bit and rounded with its sticky bits.  Reciprocal, quotient and root start
// from the MUFU approximation, take a second-order correction in fixed point
// (error below 0.4 ulp), truncate, and decide the last bit exactly: the sign
// of the integer remainder at the midpoint of the two candidates (S H -
// 2^106, B H - 2^53 A or H^2 - 2^44 W, H odd) says which is nearer.  None
// can be zero: no quotient or root of 53-bit significands is a 54-bit odd
// one.  The correction needs |1 - x r| < 2^-21 and |1 - w t^2| < 2^-21.2;
// over all 2^23 and 2^24 seeds, with the truncation of the operand, MUFU's
// errors are at most 2^-22.4 (r) and 2^-22.5 (t)
// (tests/test_soft64_seed_bounds.py: every seed, and seeds at those limits).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define TG_HD __host__ __device__ __forceinline__
#else
#define TG_HD inline
#endif
#if !defined(__CUDA_ARCH__)
#include <math.h>
#include <string.h>
// host builds check the method; they may perturb the seeds
#ifndef TG_HOST_SEED
#define TG_HOST_SEED(y) (y)
#endif
#endif

namespace tg {
namespace soft {

TG_HD uint32_t hi32(double a)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(a);
#else
    uint64_t u;
    memcpy(&u, &a, 8);
    return (uint32_t)(u >> 32);
#endif
}

TG_HD uint32_t lo32(double a)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(a);
#else
    uint64_t u;
    memcpy(&u, &a, 8);
    return (uint32_t)u;
#endif
}

TG_HD double make(uint32_t hi, uint32_t lo)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    uint64_t u = ((uint64_t)hi << 32) | lo;
    double a;
    memcpy(&a, &u, 8);
    return a;
#endif
}

// (hi:lo << n) >> 32 and low word of (hi:lo >> n), 0 <= n <= 31.
TG_HD uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t n)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, n);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << (n & 31)) >> 32);
#endif
}

TG_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

TG_HD float as_float(uint32_t u)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

TG_HD float seed_rcp(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return TG_HOST_SEED(1.0f / x);
#endif
}

TG_HD float seed_rsq(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return TG_HOST_SEED((float)(1.0 / sqrt((double)x)));
#endif
}

TG_HD uint32_t to_u32(float x)
{
#ifdef __CUDA_ARCH__
    return __float2uint_rz(x);
#else
    return (uint32_t)x;
#endif
}

// Operands the integer forms take: biased exponents in [EXP_LO, EXP_LO +
// EXP_SPAN), so that every product, reciprocal and root is normal.
// range_key(a) < RANGE says a is one; keys of several operands combine with
// max.  Zeros, subnormals, infinities and NaN all fail it.
constexpr uint32_t EXP_LO = (1023u - 500u) << 20;
constexpr uint32_t RANGE = 1000u << 20;

TG_HD uint32_t range_key(double a)
{
    return (hi32(a) & 0x7fffffffu) - EXP_LO;
}

TG_HD uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }

// a * b for operands in range.
TG_HD double mul(double a, double b)
{
    const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
    // a's significand at the top of 64 bits, b's as 53 bits: the product is
    // in [2^115, 2^117), its integer part above bit 64
    const uint32_t A1 = fsl(al, ah, 11) | 0x80000000u, A0 = al << 11;
    const uint32_t B1 = (bh & 0xfffffu) | 0x100000u;
    const uint64_t p00 = wide(A0, bl);
    const uint64_t p01 = wide(A0, B1) + (p00 >> 32);
    const uint64_t p10 = wide(A1, bl) + (uint32_t)p01;
    const uint64_t p11 = wide(A1, B1) + (p01 >> 32) + (p10 >> 32);
    uint32_t w3 = (uint32_t)(p11 >> 32), w2 = (uint32_t)p11;
    uint32_t w1 = (uint32_t)p10;
    const uint32_t p0 = (uint32_t)p00;
    w1 |= p0 < 1u ? p0 : 1u;                       // sticky
    const uint32_t n = (w3 >> 20) ^ 1u;            // 1: below 2^116
    w3 = fsl(w2, w3, n);
    w2 = fsl(w1, w2, n);
    w1 <<= n;
    // round to nearest even: carry out of fraction + (half - 1) + odd
    const uint64_t f = (uint64_t)w1 + 0x7fffffffu + (w2 & 1u);
    const uint64_t m = (((uint64_t)w3 << 32) | w2) + (f >> 32);
    const uint32_t e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) -
                       (1023u << 20) - (n << 20);
    const uint32_t sg = (ah ^ bh) & 0x80000000u;
    return make((uint32_t)(m >> 32) + e + sg, (uint32_t)m);
}

// Y within 4 of 2^116 / S (2^64 / x for x = S / 2^52 in [1, 2)) of the
// significand S = S1:sl; 2^64 - 1 for S = 2^52.
TG_HD uint64_t recip64(uint32_t S1, uint32_t sl)
{
    // r = 2^-31 R within 2^-22.4 of 1/x (all 2^23 seeds checked)
    const float r = seed_rcp(as_float((fsl(sl, S1, 3) & 0x7fffffu) |
                                      0x3f800000u));
    const uint32_t R = to_u32(r * 2147483648.0f);
    // D = 2^83 - S R = 2^83 (1 - x r) in 64 bits, less 1 (so x = 1 gives
    // 2^64 - 1 and rounds up); 1/x = r (1 + d + d^2 + ..), d = D / 2^83
    const uint64_t D = ~(wide(sl, R) + ((uint64_t)(S1 * R) << 32));
    const int32_t Dh = (int32_t)(D >> 32);
    const uint64_t E = D + ((uint64_t)((int64_t)Dh * Dh) >> 19);
    const int64_t T = (int64_t)(wide((uint32_t)E, R) >> 32) +
                      (int64_t)(int32_t)(E >> 32) * (int64_t)R;
    return ((uint64_t)R << 33) + (uint64_t)(T >> 18);
}

// 1 / s for s > 0 in range.
TG_HD double rcp(double s)
{
    const uint32_t sh = hi32(s), sl = lo32(s);
    const uint32_t S1 = (sh & 0xfffffu) | 0x100000u;
    const uint64_t Y = recip64(S1, sl);
    // candidates Y >> 11 and the next; H their midpoint in half units;
    // the sign of S H - 2^106 (below 2^63 in magnitude) decides
    const uint64_t H = (Y >> 10) | 1u;
    const uint32_t H0 = (uint32_t)H, H1 = (uint32_t)(H >> 32);
    const uint32_t rem = (uint32_t)(wide(sl, H0) >> 32) + sl * H1 + S1 * H0;
    const uint64_t Q = (Y >> 11) + (rem >> 31);
    // value Q 2^-53 2^(1023 - e), Q in [2^52, 2^53]
    const uint32_t e = (2044u << 20) - (sh & 0x7ff00000u);
    return make((uint32_t)(Q >> 32) + e, (uint32_t)Q);
}

// a / b for operands in range.
TG_HD double quo(double a, double b)
{
    const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
    const uint32_t A1 = (ah & 0xfffffu) | 0x100000u;
    const uint32_t B1 = (bh & 0xfffffu) | 0x100000u;
    const uint64_t Y = recip64(B1, bl);
    // n: 1 where |significand of a| is the smaller one; A = 2^n a's, top
    // aligned at 2^62, so P = 2^62 A / B in [2^62, 2^63)
    const uint64_t A = ((uint64_t)A1 << 32) | al;
    const uint32_t n = A < (((uint64_t)B1 << 32) | bl) ? 1u : 0u;
    const uint32_t C1 = fsl(al, A1, 10u + n), C0 = al << (10u + n);
    const uint32_t Y1 = (uint32_t)(Y >> 32), Y0 = (uint32_t)Y;
    const uint64_t p01 = wide(C0, Y1) + (wide(C0, Y0) >> 32);
    const uint64_t p10 = wide(C1, Y0) + (uint32_t)p01;
    const uint64_t P = wide(C1, Y1) + (p01 >> 32) + (p10 >> 32);
    // midpoint H of P >> 10 and the next; sign of B H - 2^53 A decides
    const uint64_t H = (P >> 9) | 1u;
    const uint32_t H0 = (uint32_t)H, H1 = (uint32_t)(H >> 32);
    const uint32_t rem = (uint32_t)(wide(bl, H0) >> 32) + bl * H1 + B1 * H0 -
                         (al << (21u + n));
    const uint64_t Q = (P >> 10) + (rem >> 31);
    const uint32_t e = (ah & 0x7ff00000u) - (bh & 0x7ff00000u) +
                       ((1022u - n) << 20);
    return make((uint32_t)(Q >> 32) + e + ((ah ^ bh) & 0x80000000u),
                (uint32_t)Q);
}

// sqrt(q) for q > 0 in range.
TG_HD double root(double q)
{
    const uint32_t qh = hi32(q), ql = lo32(q);
    // q = w 4^k, w = W / 2^62 in [1, 4); odd: 1 where w >= 2
    const uint32_t odd = (~qh >> 20) & 1u;
    const float wf = as_float(((fsl(ql, qh, 3) & 0x7fffffu) | 0x3f800000u) +
                              (odd << 23));
    const uint32_t T = to_u32(seed_rsq(wf) * 2147483648.0f);   // 2^31 t
    const uint32_t n = 10u + odd;
    const uint32_t W1 = fsl(ql, (qh & 0xfffffu) | 0x100000u, n);
    const uint32_t W0 = ql << n;
    // M = W T^2 / 2^64 = 2^60 w t^2; D = 2^60 d with w t^2 = 1 - d
    const uint64_t T2 = wide(T, T);
    const uint32_t t0 = (uint32_t)T2, t1 = (uint32_t)(T2 >> 32);
    const uint64_t c0 = wide(W0, t1) + (wide(W0, t0) >> 32);
    const uint64_t c1 = wide(W1, t0) + (uint32_t)c0;
    const uint64_t M = wide(W1, t1) + (c0 >> 32) + (c1 >> 32);
    const int64_t D = (int64_t)((1ull << 60) - M);       // |D| < 2^39
    // sqrt(w) = w t (1 + c), c = d/2 + 3 d^2 / 8 + .. in units of 2^-60
    const int32_t dh = (int32_t)(D >> 9);
    const int32_t sq = (int32_t)(((int64_t)dh * dh) >> 32);   // 2^70 d^2
    const int64_t C = (D >> 1) + (int64_t)((3 * sq) >> 13);
    // G = 2^61 w t (1 + c).  The correction takes w t (at most 2 and a
    // little) rounded to 2^-30: 2^-31 |c|, 0.4 ulp, which the midpoint
    // decision absorbs.  G0 carries that rounding's 2^30.
    const uint64_t G0 = wide(W1, T) + ((wide(W0, T) + (1ull << 62)) >> 32);
    const uint32_t g = (uint32_t)(G0 >> 31);
    const int64_t V = (int64_t)(wide((uint32_t)C, g) >> 32) +
                      (int64_t)(int32_t)(C >> 32) * (int64_t)g;
    const uint64_t G = G0 - (1ull << 30) + ((uint64_t)V << 3);
    // candidates G >> 9 and the next; sign of H^2 - W 2^44 decides
    const uint64_t H = (G >> 8) | 1u;
    const uint32_t H0 = (uint32_t)H, H1 = (uint32_t)(H >> 32);
    const uint32_t rem = (uint32_t)(wide(H0, H0) >> 32) + 2u * H0 * H1 -
                         (W0 << 12);
    const uint64_t F = (G >> 9) + (rem >> 31);
    // biased exponent floor((e + 1023) / 2), less the implicit bit
    const uint32_t e = ((qh >> 1) + (1021u << 19)) & 0x7ff00000u;
    return make((uint32_t)(F >> 32) + e, (uint32_t)F);
}

}  // namespace soft
}  // namespace tg
