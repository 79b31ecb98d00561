// Pair arithmetic of the tupan kernels in REAL precision (double or float),
// evaluated in the same order as the reference C so that, compiled without
// multiply-add contraction (-fmad=false) and with IEEE division and square
// root (nvcc's defaults), every pair term rounds exactly as in
// tupan/lib/src/*_common.h.  Used by the EXACT sweeps and by Sakura/Kepler.
//
// Attribute order of a particle record p[]: m, rx, ry, rz, e2, vx, vy, vz,
// ax, ay, az, jx, jy, jz (NREG_V: m, vx, vy, vz, ax, ay, az).
#pragma once

#include "tg_common.cuh"
#include "tg_soft64.cuh"

namespace tg {

template <typename R>
__device__ __forceinline__ R masked_inv_r2(R r2, R h2)
{
    // smoothing.h:10-184: 1/(r2+h2), zeroed where r2 == 0 (self pairs)
    R q = R(1) / (r2 + h2);
    return (r2 > R(0)) ? q : R(0);
}

// Products, reciprocals, roots and quotients of the pair terms.  In double
// they run on the integer pipe (tg_soft64.cuh: the same bits, and the FP64
// pipe, 19 cycles of the SM for each warp instruction, is left to the
// additions) wherever every operand of a group lies in soft::RANGE; a lane
// with a zero, subnormal, infinite or NaN operand takes the FP64 forms.
// `key` is the largest range_key of a group's operands: one test a group.
// float takes the hardware's IEEE operations throughout.
template <typename R>
__device__ __forceinline__ uint32_t key_of(R) { return 0u; }

template <>
__device__ __forceinline__ uint32_t key_of<double>(double a)
{
    return soft::range_key(a);
}

template <typename R, typename... T>
__device__ __forceinline__ uint32_t key_of(R a, T... rest)
{
    return soft::umax(key_of(a), key_of(rest...));
}

// o[k] = a[k] * b[k]
template <int N>
__device__ __forceinline__ void muls(uint32_t, const float (&a)[N],
                                     const float (&b)[N], float (&o)[N])
{
#pragma unroll
    for (int k = 0; k < N; ++k) o[k] = a[k] * b[k];
}

template <int N>
__device__ __forceinline__ void muls(uint32_t key, const double (&a)[N],
                                     const double (&b)[N], double (&o)[N])
{
    if (__builtin_expect(key < soft::RANGE, 1)) {
#pragma unroll
        for (int k = 0; k < N; ++k) o[k] = soft::mul(a[k], b[k]);
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) o[k] = a[k] * b[k];
    }
}

__device__ __forceinline__ float quotient(float a, float b) { return a / b; }

__device__ __forceinline__ double quotient(double a, double b)
{
    return key_of(a, b) < soft::RANGE ? soft::quo(a, b) : a / b;
}

__device__ __forceinline__ float square_root(float a) { return sqrt(a); }

__device__ __forceinline__ double square_root(double a)
{
    // a negative a fails the range test by its sign bit being dropped from
    // the key, so it is tested too
    return soft::range_key(a) < soft::RANGE && (int)soft::hi32(a) > 0
               ? soft::root(a) : sqrt(a);
}

// 2 a, exact
__device__ __forceinline__ float twice(float a) { return 2.0f * a; }

__device__ __forceinline__ double twice(double a)
{
    return soft::range_key(a) < soft::RANGE
               ? soft::make(soft::hi32(a) + 0x100000u, soft::lo32(a))
               : 2.0 * a;
}

// 64 a, exact
__device__ __forceinline__ float times64(float a) { return 64.0f * a; }

__device__ __forceinline__ double times64(double a)
{
    return soft::range_key(a) < soft::RANGE
               ? soft::make(soft::hi32(a) + (6u << 20), soft::lo32(a))
               : 64.0 * a;
}

// r2 > 0 for an r2 that is not negative; fmax(a, o) for o not negative or
// NaN (comparisons of doubles run on the FP64 pipe, those of their bits,
// which order the same way, do not)
__device__ __forceinline__ bool positive(float r2) { return r2 > 0.0f; }

__device__ __forceinline__ bool positive(double r2)
{
    const long long b = __double_as_longlong(r2);
    return b > 0 && b <= 0x7ff0000000000000ll;
}

// a > b for b not negative, or either of them NaN (of any sign: 0 / 0 is one
// with the sign set).  Unsigned, negative values and NaN lie above infinity.
__device__ __forceinline__ bool greater(float a, float b) { return a > b; }

__device__ __forceinline__ bool greater(double a, double b)
{
    const unsigned long long x = (unsigned long long)__double_as_longlong(a),
                             y = (unsigned long long)__double_as_longlong(b);
    return x > y && x <= 0x7ff0000000000000ull;
}

__device__ __forceinline__ float larger(float a, float o) { return fmax(a, o); }

__device__ __forceinline__ double larger(double a, double o)
{
    return greater(a, o) ? a : o;
}

// e2_i + e2_j, kept while e2_j keeps its bits from one j to the next
// (uniform softening, the common case: one FP64 addition a pair less).
template <typename R>
struct Softening {
    R e2, h2;
    __device__ __forceinline__ void set(R ei, R ej)
    {
        e2 = ej;
        h2 = ei + ej;
    }
    __device__ __forceinline__ R sum(R ei, R ej);
};

template <>
__device__ __forceinline__ float Softening<float>::sum(float ei, float ej)
{
    return ei + ej;
}

template <>
__device__ __forceinline__ double Softening<double>::sum(double ei, double ej)
{
    if (__builtin_expect(__double_as_longlong(ej) !=
                             __double_as_longlong(e2), 0)) {
        e2 = ej;
        h2 = ei + ej;
    }
    return h2;
}

// q = masked 1/(r2+h2) and w = sqrt(q)
__device__ __forceinline__ void inv_root(float r2, float h2, float *q,
                                         float *w)
{
    *q = masked_inv_r2(r2, h2);
    *w = sqrt(*q);
}

__device__ __forceinline__ void inv_root(double r2, double h2, double *q,
                                         double *w)
{
    // s in [2^-320, 2^320): q, w, q w and products with one factor of
    // soft::RANGE stay normal; a NaN r2 makes s one, r2 is never negative
    constexpr uint32_t lo = (1023u - 320u) << 20, span = 640u << 20;
    const double s = r2 + h2;
    if (__builtin_expect(soft::hi32(s) - lo < span &&
                             (soft::hi32(r2) | soft::lo32(r2)) != 0u, 1)) {
        *q = soft::rcp(s);
        *w = soft::root(*q);
    } else {
        *q = masked_inv_r2(r2, h2);
        *w = sqrt(*q);
    }
}

// Each operator gives the terms one j adds to the sums of one i (terms),
// how a term joins its sum (join: added, subtracted or the larger kept; sums
// start from zero; fold does it), whether an output's terms nearly all have
// one sign (one_signed: ordered_sum's fast case) and the last step of each
// output (finish).  MANY: the i from which a float sweep does best with one
// i a thread.  Terms of different j are independent, so they
// may be formed in any order; folding them in j order keeps the
// reference's bits.
enum Join : int { JOIN_ADD = 0, JOIN_SUB = 1, JOIN_MAX = 2 };

template <class Op, typename R>
__device__ __forceinline__ R fold(int c, R o, R t)
{
    const int j = Op::join(c);
    return j == JOIN_MAX ? larger(t, o) : j == JOIN_SUB ? o - t : o + t;
}

template <class Op, typename R>
__device__ __forceinline__ void fold_pair(const R *ip, const R *jp, R *o,
                                          const Sweep &s,
                                          Softening<R> &soft2)
{
    R t[Op::NO];
    Op::terms(ip, jp, t, s, soft2);
#pragma unroll
    for (int c = 0; c < Op::NO; ++c) o[c] = fold<Op>(c, o[c], t[c]);
}

// phi_kernel_common.h:7-32
template <typename R>
struct PhiPair {
    static constexpr int NA = 5, NO = 1;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 64000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &,
                                                 Softening<R> &soft2)
    {
        const R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        R p[3], q, w;
        muls<3>(key_of(d[0], d[1], d[2]), d, d, p);
        inv_root(p[0] + p[1] + p[2], h2, &q, &w);
        const R a[1] = {jp[0]}, b[1] = {w};
        R x[1];
        muls<1>(key_of(a[0], w), a, b, x);
        t[0] = x[0];
    }
    __device__ static constexpr int join(int) { return JOIN_SUB; }
    __device__ static constexpr bool one_signed(int) { return true; }
    __device__ static R finish(int, const R *, R o, const Sweep &) { return o; }
};

// acc_kernel_common.h:7-38
template <typename R>
struct AccPair {
    static constexpr int NA = 5, NO = 3;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 42000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &,
                                                 Softening<R> &soft2)
    {
        const R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        const uint32_t kd = key_of(d[0], d[1], d[2]);
        R p[3], q, w;
        muls<3>(kd, d, d, p);
        inv_root(p[0] + p[1] + p[2], h2, &q, &w);
        R k[1];
        muls<1>(key_of(q, w), {q}, {w}, k);
        muls<1>(key_of(k[0], jp[0]), {k[0]}, {jp[0]}, k);
        const R kk[3] = {k[0], k[0], k[0]};
        R x[3];
        muls<3>(soft::umax(kd, key_of(k[0])), kk, d, x);
        t[0] = x[0];
        t[1] = x[1];
        t[2] = x[2];
    }
    __device__ static constexpr int join(int) { return JOIN_SUB; }
    __device__ static constexpr bool one_signed(int) { return false; }
    __device__ static R finish(int, const R *, R o, const Sweep &) { return o; }
};

// acc_jerk_kernel_common.h:7-56
template <typename R>
struct AccJerkPair {
    static constexpr int NA = 8, NO = 6;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 42000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &,
                                                 Softening<R> &soft2)
    {
        const R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        R u[3] = {ip[5] - jp[5], ip[6] - jp[6], ip[7] - jp[7]};
        const uint32_t kd = key_of(d[0], d[1], d[2]);
        R p[6], q, w;
        muls<6>(soft::umax(kd, key_of(u[0], u[1], u[2])),
                {d[0], d[1], d[2], d[0], d[1], d[2]},
                {d[0], d[1], d[2], u[0], u[1], u[2]}, p);
        R r2 = p[0] + p[1] + p[2];
        R rv = p[3] + p[4] + p[5];
        inv_root(r2, h2, &q, &w);
        // k = q w and 3 rv, then k m and alpha = 3 rv q
        R k[2], g[2];
        muls<2>(key_of(q, w, rv), {q, R(3)}, {w, rv}, k);
        muls<2>(key_of(k[0], k[1], jp[0], q), {k[0], k[1]}, {jp[0], q}, g);
        const R al[3] = {g[1], g[1], g[1]};
        R x[3];
        muls<3>(soft::umax(kd, key_of(g[1])), al, d, x);
        u[0] -= x[0];
        u[1] -= x[1];
        u[2] -= x[2];
        R y[6];
        muls<6>(soft::umax(kd, key_of(g[0], u[0], u[1], u[2])),
                {g[0], g[0], g[0], g[0], g[0], g[0]},
                {d[0], d[1], d[2], u[0], u[1], u[2]}, y);
#pragma unroll
        for (int c = 0; c < 6; ++c) t[c] = y[c];
    }
    __device__ static constexpr int join(int) { return JOIN_SUB; }
    __device__ static constexpr bool one_signed(int) { return false; }
    __device__ static R finish(int, const R *, R o, const Sweep &) { return o; }
};

// snap_crackle_kernel_common.h:7-95
template <typename R>
struct SnapCracklePair {
    static constexpr int NA = 14, NO = 6;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 40000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &,
                                                 Softening<R> &soft2)
    {
        const R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        R u[3] = {ip[5] - jp[5], ip[6] - jp[6], ip[7] - jp[7]};
        R A[3] = {ip[8] - jp[8], ip[9] - jp[9], ip[10] - jp[10]};
        R J[3] = {ip[11] - jp[11], ip[12] - jp[12], ip[13] - jp[13]};
        const uint32_t kd = key_of(d[0], d[1], d[2]);
        const uint32_t ku = key_of(u[0], u[1], u[2]);
        const uint32_t ka = key_of(A[0], A[1], A[2]);
        R p[9], s[9];
        muls<9>(soft::umax(kd, ku),
                {d[0], d[1], d[2], d[0], d[1], d[2], u[0], u[1], u[2]},
                {d[0], d[1], d[2], u[0], u[1], u[2], u[0], u[1], u[2]}, p);
        muls<9>(soft::umax(soft::umax(kd, ku),
                           soft::umax(ka, key_of(J[0], J[1], J[2]))),
                {d[0], d[1], d[2], d[0], d[1], d[2], u[0], u[1], u[2]},
                {J[0], J[1], J[2], A[0], A[1], A[2], A[0], A[1], A[2]}, s);
        R r2 = p[0] + p[1] + p[2];
        R rv = p[3] + p[4] + p[5];
        R v2 = p[6] + p[7] + p[8];
        R rJ = s[0] + s[1] + s[2];
        R rA = s[3] + s[4] + s[5];
        R vA = s[6] + s[7] + s[8];
        R q, w;
        inv_root(r2, h2, &q, &w);
        // k = q w, al = rv q, (v2 + rA) q, 3 vA
        R a[4];
        const R vr = v2 + rA;
        muls<4>(key_of(q, w, rv, vr, vA), {q, rv, vr, R(3)}, {w, q, q, vA},
                a);
        // k m, al^2, (3 vA + rJ) q
        R b[3];
        const R vj = a[3] + rJ;
        R al = a[1];
        muls<3>(key_of(a[0], jp[0], al, vj, q), {a[0], al, vj},
                {jp[0], al, q}, b);
        R k = b[0];
        const R al2 = b[1];
        // be = 3 ((v2 + rA) q + al^2), 4 al^2, al 3
        R c[3];
        const R bs = a[2] + al2;
        muls<3>(key_of(bs, al2, al), {R(3), R(4), al}, {bs, al2, R(3)}, c);
        R be = c[0];
        // al (be - 4 al^2)
        R e[1];
        const R bd = be - c[1];
        muls<1>(key_of(al, bd), {al}, {bd}, e);
        R ga = b[2] + e[0];
        al = c[2];
        // ga 3, al d, two_al = 2 al
        R f[5];
        muls<5>(soft::umax(kd, key_of(ga, al)), {ga, al, al, al, R(2)},
                {R(3), d[0], d[1], d[2], al}, f);
        ga = f[0];
        u[0] -= f[1];
        u[1] -= f[2];
        u[2] -= f[3];
        const R two_al = f[4];
        // A -= two_al u + be d; then al 3, be 3
        const uint32_t ku1 = key_of(u[0], u[1], u[2]);
        R g[8];
        muls<8>(soft::umax(soft::umax(kd, ku1), key_of(two_al, be, al)),
                {two_al, two_al, two_al, be, be, be, al, be},
                {u[0], u[1], u[2], d[0], d[1], d[2], R(3), R(3)}, g);
        A[0] -= g[0] + g[3];
        A[1] -= g[1] + g[4];
        A[2] -= g[2] + g[5];
        al = g[6];
        be = g[7];
        const uint32_t ka1 = key_of(A[0], A[1], A[2]);
        R h[9];
        muls<9>(soft::umax(soft::umax(kd, ku1),
                           soft::umax(ka1, key_of(al, be, ga))),
                {al, al, al, be, be, be, ga, ga, ga},
                {A[0], A[1], A[2], u[0], u[1], u[2], d[0], d[1], d[2]}, h);
        J[0] -= h[0] + h[3] + h[6];
        J[1] -= h[1] + h[4] + h[7];
        J[2] -= h[2] + h[5] + h[8];
        R y[6];
        muls<6>(soft::umax(ka1, key_of(k, J[0], J[1], J[2])),
                {k, k, k, k, k, k}, {A[0], A[1], A[2], J[0], J[1], J[2]}, y);
#pragma unroll
        for (int n = 0; n < 6; ++n) t[n] = y[n];
    }
    __device__ static constexpr int join(int) { return JOIN_SUB; }
    __device__ static constexpr bool one_signed(int) { return false; }
    __device__ static R finish(int, const R *, R o, const Sweep &) { return o; }
};

// tstep_kernel_common.h:7-60 and tstep_kernel.c:43-47
template <typename R>
struct TstepPair {
    static constexpr int NA = 8, NO = 2;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 64000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &s,
                                                 Softening<R> &soft2)
    {
        R eta = R(s.scal[0]);
        const R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        const R u[3] = {ip[5] - jp[5], ip[6] - jp[6], ip[7] - jp[7]};
        R msum = ip[0] + jp[0];
        R p[9], q, w;
        muls<9>(key_of(d[0], d[1], d[2], u[0], u[1], u[2]),
                {d[0], d[1], d[2], d[0], d[1], d[2], u[0], u[1], u[2]},
                {d[0], d[1], d[2], u[0], u[1], u[2], u[0], u[1], u[2]}, p);
        R r2 = p[0] + p[1] + p[2];
        R rv = p[3] + p[4] + p[5];
        R v2 = p[6] + p[7] + p[8];
        const bool mask = positive(r2);
        inv_root(r2, h2, &q, &w);
        // phi; b = 2 q and two phi are exact
        R f[1], g[2], e[1];
        muls<1>(key_of(msum, w), {msum}, {w}, f);
        const R phi = f[0], b = twice(q);
        const R sum = v2 + twice(phi);
        muls<2>(key_of(q, sum, b, phi), {q, b}, {sum, phi}, g);
        R w2 = g[0];
        const R gs = w2 + g[1];
        const R ew = quotient(eta, square_root(w2));
        muls<1>(key_of(q, gs), {q}, {gs}, e);
        muls<1>(key_of(e[0], ew), {e[0]}, {ew}, e);
        muls<1>(key_of(e[0], rv), {e[0]}, {rv}, e);
        w2 -= e[0];
        w2 = mask ? w2 : R(0);
        t[0] = w2;
        t[1] = w2;
    }
    __device__ static constexpr int join(int c)
    {
        return c == 0 ? JOIN_ADD : JOIN_MAX;
    }
    __device__ static constexpr bool one_signed(int c) { return c == 0; }
    __device__ static R finish(int, const R *, R o, const Sweep &s)
    {
        R eta = R(s.scal[0]);
        return eta / sqrt(R(1) + o);
    }
};

// nreg_kernels_common.h:7-61 and nreg_kernels.c:59-66
template <typename R>
struct NregXPair {
    static constexpr int NA = 8, NO = 7;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 33000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &s,
                                                 Softening<R> &soft2)
    {
        R dt = R(s.scal[0]);
        R d[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        R h2 = soft2.sum(ip[4], jp[4]);
        const R u[3] = {ip[5] - jp[5], ip[6] - jp[6], ip[7] - jp[7]};
        R p[3], q, w;
        muls<3>(key_of(u[0], u[1], u[2], dt), u, {dt, dt, dt}, p);
        d[0] += p[0];
        d[1] += p[1];
        d[2] += p[2];
        const uint32_t kd = key_of(d[0], d[1], d[2]);
        muls<3>(kd, d, d, p);
        inv_root(p[0] + p[1] + p[2], h2, &q, &w);
        R jm = jp[0];
        R k[1], y[7];
        muls<1>(key_of(q, w), {q}, {w}, k);
        muls<1>(key_of(k[0], jm), {k[0]}, {jm}, k);
        muls<7>(soft::umax(kd, key_of(k[0], jm, w)),
                {jm, jm, jm, k[0], k[0], k[0], jm},
                {d[0], d[1], d[2], d[0], d[1], d[2], w}, y);
#pragma unroll
        for (int n = 0; n < 7; ++n) t[n] = y[n];
    }
    __device__ static constexpr int join(int c)
    {
        return c < 3 || c == 6 ? JOIN_ADD : JOIN_SUB;
    }
    __device__ static constexpr bool one_signed(int c) { return c == 6; }
    __device__ static R finish(int c, const R *ip, R o, const Sweep &)
    {
        return c == 6 ? ip[0] * o : o;
    }
};

// nreg_kernels_common.h:63-102 and nreg_kernels.c:107-114
template <typename R>
struct NregVPair {
    static constexpr int NA = 7, NO = 4;
    static constexpr bool WIDE = false;
    static constexpr uint64_t MANY = 10000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &s,
                                                 Softening<R> &)
    {
        R dt = R(s.scal[0]);
        R u[3] = {ip[1] - jp[1], ip[2] - jp[2], ip[3] - jp[3]};
        const R w[3] = {ip[4] - jp[4], ip[5] - jp[5], ip[6] - jp[6]};
        R p[3], y[4];
        muls<3>(key_of(w[0], w[1], w[2], dt), w, {dt, dt, dt}, p);
        u[0] += p[0];
        u[1] += p[1];
        u[2] += p[2];
        const uint32_t ku = key_of(u[0], u[1], u[2]);
        muls<3>(ku, u, u, p);
        R v2 = p[0] + p[1] + p[2];
        R jm = jp[0];
        muls<4>(soft::umax(ku, key_of(jm, v2)), {jm, jm, jm, jm},
                {u[0], u[1], u[2], v2}, y);
#pragma unroll
        for (int n = 0; n < 4; ++n) t[n] = y[n];
    }
    __device__ static constexpr int join(int) { return JOIN_ADD; }
    __device__ static constexpr bool one_signed(int c) { return c == 3; }
    __device__ static R finish(int c, const R *ip, R o, const Sweep &)
    {
        return c == 3 ? ip[0] * o : o;
    }
};

}  // namespace tg
