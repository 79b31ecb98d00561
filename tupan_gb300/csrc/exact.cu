// EXACT-mode sweeps: the terms of the pairs are formed in parallel over i
// and j (or by one thread an i, where that is the faster form) and added to
// each i's sums in source order.  With the pair
// arithmetic of tg_pairs.cuh and this file compiled with -fmad=false, every
// output is bit-identical to the reference C kernel (tupan/lib/src/*.c) on
// the same inputs, for REAL = double and REAL = float.
//
// Sakura and Kepler share the pair/solver code of tg_kepler.cuh; their
// leapfrog branch is bit-identical, their Kepler branch agrees to the
// accuracy of CUDA's transcendental functions.

#include <type_traits>

#include "tg_common.cuh"
#include "tg_launch.cuh"
#include "tg_kepler.cuh"
#include "tg_ordered.cuh"
#include "tg_pairs.cuh"
#include "tg_pn.cuh"

namespace tg {

constexpr int EXACT_THREADS = 128;

// The pair terms of a tile, I = 2^li particles i (a block's) against
// J = T P / I consecutive j, P pairs (P i's, one j) a thread; the terms go
// through shared memory to the I x NO threads that hold the sums and fold
// them in j order.  Double buffered: one barrier a tile, a warp that holds
// no sum goes on to the next tile's pairs.
//
// Why: a sum's additions have to stay in order, the terms need not.  One i a
// thread over all j (exact_sweep, the only form before) put a 256-body sweep
// on two SMs and a 3001-body one on 24, each at the latency of a chain of
// whole pairs; here only the additions are a chain (64 cycles each in double)
// and any ni fills the chip.  Bound: the FP64 pipe (20 additions of 19 SM cycles a
// warp of AccJerk pairs; ncu at N = 8192: 71 % of its peak, the integer pipe
// that carries the products 57 %).  No j prefetch and 64 registers (eight
// blocks of 128 an SM) beat a prefetch at four blocks by 10 %: the chains of
// dependent additions want warps.  Measured, double: AccJerk / SnapCrackle at
// N = 3001 6.09 / 14.1 ms before, 0.53 / 1.40 ms now; Phi / AccJerk /
// SnapCrackle / Tstep at N = 32768 61 / 128 / 302 / 157 ms, now 21 / 51 /
// 141 / 54 ms.  float takes four i a thread (one load of a j for four pairs,
// one 16-byte store of a term): Phi + Acc at N = 10007 2.3 ms before, 0.62.
// SKIP: rows past the last j form no term (else one that nobody reads: the
// branch costs 1 to 2 % of a long sweep).
template <class Op, typename R, int T, int P, int BLK, bool SKIP>
__global__ void __launch_bounds__(T, BLK)
exact_terms(const Sweep s, const int li)
{
    constexpr int NA = Op::NA, NO = Op::NO;
    constexpr int LP = P == 1 ? 0 : P == 2 ? 1 : 2;
    static_assert(P == 1 << LP, "P is 1, 2 or 4");
    __shared__ __align__(16) R buf[2][NO][T * P];
    chain_begin();
    const uint64_t ni = s.ni_dev ? (uint64_t)*s.ni_dev : s.ni, nj = s.nj;
    const uint64_t i0 = (uint64_t)blockIdx.x << li;
    // blocks past a device-side count have no i (the whole block leaves)
    if (i0 >= ni) return;
    const int tid = threadIdx.x;
    const int g = tid & ((1 << (li - LP)) - 1), row = tid >> (li - LP);
    const int J = T * P >> li;
    const int c = tid >> li, ii = tid & ((1 << li) - 1);
    const bool sums = c < NO;
    R o = R(0);
    if (nj) {
        R ip[P][NA], jp[NA];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const uint64_t i = i0 + g * P + p < ni ? i0 + g * P + p : ni - 1;
#pragma unroll
            for (int a = 0; a < NA; ++a) ip[p][a] = ((const R *)s.ip[a])[i];
        }
        Softening<R> soft2[P];
#pragma unroll
        for (int p = 0; p < P; ++p)
            soft2[p].set(ip[p][4], ((const R *)s.jp[4])[0]);
        int b = 0;
        for (uint64_t j0 = 0; j0 < nj; j0 += J, b ^= 1) {
            const uint64_t j = j0 + row < nj ? j0 + row : nj - 1;
#pragma unroll
            for (int a = 0; a < NA; ++a) jp[a] = ((const R *)s.jp[a])[j];
            R t[NO][P];
#pragma unroll
            for (int p = 0; p < P; ++p) {
                R tp[NO];
                if (!SKIP || j0 + row < nj)
                    Op::terms(ip[p], jp, tp, s, soft2[p]);
#pragma unroll
                for (int k = 0; k < NO; ++k) t[k][p] = tp[k];
            }
#pragma unroll
            for (int k = 0; k < NO; ++k) {
                R *w = &buf[b][k][tid * P];
                if constexpr (P == 4)
                    *(float4 *)w = make_float4(t[k][0], t[k][1], t[k][2],
                                               t[k][3]);
                else
#pragma unroll
                    for (int p = 0; p < P; ++p) w[p] = t[k][p];
            }
            __syncthreads();
            if (sums) {
                const int n = nj - j0 < (uint64_t)J ? (int)(nj - j0) : J;
                const R *q = &buf[b][c][ii];
#pragma unroll 8
                for (int k = 0; k < n; ++k) o = fold<Op>(c, o, q[k << li]);
            }
        }
    }
    if (sums && i0 + ii < ni) {
        R ip[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) ip[a] = ((const R *)s.ip[a])[i0 + ii];
        ((R *)s.out[c])[i0 + ii] = Op::finish(c, ip, o, s);
    }
}

// Few i against many j, double: one i a block, eight warps form the terms of
// 256 j a tile while others sum the tile before.  A one-signed or max output
// has a warp of its own (ordered_sum, or a maximum in any order); the others
// share one, an output a lane, that adds term by term.  Bound: that chain of
// additions, 64 cycles a term (AccJerk 100 x 8192 336 us, 273 of them the
// chain), else the latency of a tile's pairs.  ordered_sum and a warp each
// for the signed outputs too, on terms of zero mean: slower to some thousand
// j (AccJerk 100 x 1024 45 us and 73, x 8192 333 and 398; 3001 x 3001 529
// and 1383), as their sums keep leaving their binade and six warps add where
// one did, faster for long ones (x 65536 2.63 and 1.67 ms).  Measured against exact_terms
// at one i a block: Phi 100 x 8192 387 -> 66 us, Tstep 576 -> 115, AccJerk
// 447 -> 336, SnapCrackle 690 -> 405; NREG X at N = 256 33 -> 19 us.
constexpr int FEW_T = 256;
constexpr uint64_t FEW_I = 2 * 152;     // two blocks an SM

template <class Op>
__host__ __device__ constexpr bool few_own(int c)
{
    return Op::one_signed(c) || Op::join(c) == JOIN_MAX;
}

template <class Op>
__host__ __device__ constexpr int few_owned()
{
    int n = 0;
    for (int c = 0; c < Op::NO; ++c) n += few_own<Op>(c) ? 1 : 0;
    return n;
}

template <class Op>
constexpr int few_threads()
{
    return FEW_T + 32 * (few_owned<Op>() + (few_owned<Op>() < Op::NO ? 1 : 0));
}

// The n-th output that has (own) or has not a warp of its own; NO if none.
template <class Op>
__device__ __forceinline__ int few_output(int n, bool own)
{
    int at = Op::NO;
#pragma unroll
    for (int c = Op::NO - 1; c >= 0; --c) {
        int before = 0;
        for (int q = 0; q < c; ++q) before += few_own<Op>(q) == own ? 1 : 0;
        if (few_own<Op>(c) == own && before == n) at = c;
    }
    return at;
}

template <class Op>
__global__ void __launch_bounds__(few_threads<Op>())
exact_few(const Sweep s)
{
    constexpr int NA = Op::NA, NO = Op::NO;
    constexpr int RUNS = FEW_T / ORD_RUN, SPAN = ORD_PITCH * ORD_K;
    constexpr int ROW = RUNS * SPAN + 1;      // odd: outputs on other banks
    __shared__ double buf[2][NO][ROW];
    chain_begin();
    const uint64_t i = blockIdx.x, nj = s.nj;
    if (s.ni_dev && i >= (uint64_t)*s.ni_dev) return;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool forms = tid < FEW_T;
    const int w = (tid - FEW_T) >> 5;
    const bool own = w < few_owned<Op>();
    const int c = few_output<Op>(own ? w : lane, own);
    double ip[NA], o = 0.0;
#pragma unroll
    for (int a = 0; a < NA; ++a) ip[a] = ((const double *)s.ip[a])[i];
    Softening<double> soft2;
    if (nj) soft2.set(ip[4], ((const double *)s.jp[4])[0]);
    // tile k is formed in step k and summed in step k + 1
    const uint64_t tiles = (nj + FEW_T - 1) / FEW_T;
    for (uint64_t k = 0; k <= tiles; ++k) {
        if (forms) {
            const uint64_t j = k * FEW_T + tid;
            if (j < nj) {
                double jp[NA], t[NO];
#pragma unroll
                for (int a = 0; a < NA; ++a)
                    jp[a] = ((const double *)s.jp[a])[j];
                Op::terms(ip, jp, t, s, soft2);
#pragma unroll
                for (int q = 0; q < NO; ++q)
                    buf[k & 1][q][few_own<Op>(q)
                                      ? tid / ORD_RUN * SPAN +
                                            ord_at(tid % ORD_RUN)
                                      : tid] =
                        Op::join(q) == JOIN_SUB ? -t[q] : t[q];
            }
        } else if (k > 0 && c < NO) {
            const uint64_t j0 = (k - 1) * FEW_T;
            const int n = nj - j0 < (uint64_t)FEW_T ? (int)(nj - j0) : FEW_T;
            const double *q = buf[(k - 1) & 1][c];
            if (!own) {
                // the next eight loads are under way while eight terms add
                double x[8], y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = e < n ? q[e] : -0.0;
                for (int u = 0; u < n; u += 8) {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        y[e] = u + 8 + e < n ? q[u + 8 + e] : -0.0;
#pragma unroll
                    for (int e = 0; e < 8; ++e) o = o + x[e];
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = y[e];
                }
            } else if (Op::join(c) == JOIN_MAX) {
                for (int u = lane; u < n; u += 32)
                    o = larger(q[u / ORD_RUN * SPAN + ord_at(u % ORD_RUN)], o);
            } else {
                for (int r = 0; r * ORD_RUN < n; ++r)
                    o = ordered_sum(o, q + r * SPAN,
                                    n - r * ORD_RUN < ORD_RUN
                                        ? n - r * ORD_RUN : ORD_RUN);
            }
        }
        __syncthreads();
    }
    if (forms || c == NO) return;
    if (own && Op::join(c) == JOIN_MAX) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            o = larger(__shfl_xor_sync(0xffffffffu, o, d), o);
    }
    if (!own || lane == 0) ((double *)s.out[c])[i] = Op::finish(c, ip, o, s);
}

// One i a thread over all j, j through shared memory in tiles: for many i,
// where the threads fill the chip without the terms' way through shared
// memory, in float, whose additions are cheap; and against a handful of j,
// which would leave most rows of a tile of exact_terms idle.  Bound: issue
// slots (float), the FP64 pipe.  float, 70000 x 16384 against exact_terms:
// Acc 2.04 ms and 2.53, AccJerk 2.91 and 3.91, SnapCrackle 5.61 and 7.12;
// double, 70000 x 1: AccJerk 6 us and 27, SnapCrackle 12 and 71.
constexpr int SWEEP_T = 128;

template <typename R> struct SakuraPair;

// Whether exact_sweep takes a call that exact_terms would serve with J rows a
// tile.  The lines lie where the two take equally long, measured at 1 to
// 16384 j.  double: one j always (SnapCrackle at 1000 20 us and 7), two but
// against few i (SnapCrackle at 1000 20 and 13, Tstep at 20000 8 and 10),
// three from 30000 i (SnapCrackle 34 and 21, Tstep 11 and 12; at 3000 Tstep
// 8 and 10).  float: up to 8 j (equal at few i, SnapCrackle at 35000 11 and
// 4), else from MANY i (AccJerk x 16384 at 40000 2.35 and 2.37 ms, at 45000
// 2.62 and 2.38), or from as many fewer as the tiles' empty rows make of them
// (SnapCrackle at 35000 x 33, where exact_terms takes two tiles of 32, 18 us
// and 9).  Sakura, whose terms are solves: lanes of a warp that solve for
// different i diverge, so the i have to be many (double x 1 at 3000 96 us
// and 112, at 7000 142 and 124; x 3 at 20000 275 and 353, at 50000 589 and
// 535; x 5 at 200000 3.14 and 2.80 ms; float x 64 at 100000 640 and 624 us,
// at 200000 1.30 and 1.15 ms).
template <class Op, typename R>
bool one_i_a_thread(uint64_t ni, uint64_t nj, uint64_t J)
{
    constexpr bool solves = std::is_same<Op, SakuraPair<R>>::value;
    if (solves && ((nj <= 1 && ni >= 6000) || (nj <= 3 && ni >= 32000) ||
                   (nj <= 5 && ni >= 200000)))
        return true;
    if (sizeof(R) == 4)
        return (!solves && nj <= 8) || (double)ni * ((nj + J - 1) / J * J) >=
                                           (double)Op::MANY * nj;
    return !solves && (nj <= 1 || (nj == 2 && ni > FEW_I) ||
                       (nj == 3 && ni >= 30000));
}

template <class Op, typename R>
__global__ void __launch_bounds__(SWEEP_T)
exact_sweep(const Sweep s)
{
    constexpr int NA = Op::NA, NO = Op::NO;
    __shared__ R tile[NA][SWEEP_T];
    chain_begin();
    const uint64_t ni = s.ni_dev ? (uint64_t)*s.ni_dev : s.ni, nj = s.nj;
    // blocks past a device-side count have no i (the whole block leaves)
    if ((uint64_t)blockIdx.x * SWEEP_T >= ni) return;
    const uint64_t i = (uint64_t)blockIdx.x * SWEEP_T + threadIdx.x;
    R ip[NA], jp[NA], o[NO];
#pragma unroll
    for (int a = 0; a < NA; ++a) ip[a] = ((const R *)s.ip[a])[i < ni ? i : ni - 1];
#pragma unroll
    for (int c = 0; c < NO; ++c) o[c] = R(0);
    Softening<R> soft2;
    if (nj) soft2.set(ip[4], ((const R *)s.jp[4])[0]);
    for (uint64_t j0 = 0; j0 < nj; j0 += SWEEP_T) {
        const int n = nj - j0 < SWEEP_T ? (int)(nj - j0) : SWEEP_T;
        __syncthreads();
        if ((int)threadIdx.x < n)
#pragma unroll
            for (int a = 0; a < NA; ++a)
                tile[a][threadIdx.x] = ((const R *)s.jp[a])[j0 + threadIdx.x];
        __syncthreads();
        for (int jj = 0; jj < n; ++jj) {
#pragma unroll
            for (int a = 0; a < NA; ++a) jp[a] = tile[a][jj];
            fold_pair<Op>(ip, jp, o, s, soft2);
        }
    }
    if (i >= ni) return;
#pragma unroll
    for (int c = 0; c < NO; ++c)
        ((R *)s.out[c])[i] = Op::finish(c, ip, o[c], s);
}

// sakura_kernel.c:33-62: Sigma_j (m_j/M)(two-body step - initial state).
template <typename R>
struct SakuraPair {
    static constexpr int NA = 8, NO = 6;
    static constexpr bool WIDE = true;
    static constexpr uint64_t MANY = 150000;
    __device__ __forceinline__ static void terms(const R *ip, const R *jp,
                                                 R *t, const Sweep &s,
                                                 Softening<R> &)
    {
        R p0[6], p1[6], m, e2;
        pair_state(ip, jp, p0, &m, &e2);
        KepCtx<R> c = {0, s.budget, 0, false, false, R(0)};
        evolve_pair(R(s.scal[0]), s.iscal, m, e2, p0, p1, c);
        if (c.exhausted) atomicOr(s.err, (unsigned)DERR_KEPLER_BUDGET);
        pair_term(jp[0], m, p0, p1, t);
    }
    __device__ static constexpr int join(int) { return JOIN_ADD; }
    __device__ static constexpr bool one_signed(int) { return false; }
    __device__ static R finish(int, const R *, R o, const Sweep &) { return o; }
};

// kepler_solver_kernel.c:5-49 with kepler_solver_kernel_common.h:8-80: two
// particles evolved in their centre-of-mass frame; outputs may alias inputs.
template <typename R>
__global__ void exact_kepler(const Sweep s, long long budget, unsigned *err)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    R a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        a[k] = ((const R *)s.ip[k])[0];
        b[k] = ((const R *)s.ip[k])[1];
    }
    const R dt = R(s.scal[0]);
    KepCtx<R> ctx = {0, budget, 0, false, false, R(0)};
    R a1[6], b1[6];
    kepler_two_body(a, b, dt, a1, b1, ctx);
    for (int q = 0; q < 6; ++q) {
        ((R *)s.out[q])[0] = a1[q];
        ((R *)s.out[q])[1] = b1[q];
    }
    if (ctx.exhausted) atomicOr(err, (unsigned)DERR_KEPLER_BUDGET);
}

template <class Op, typename R>
static cudaError_t run_exact(const Sweep &s, cudaStream_t st)
{
    constexpr int T = EXACT_THREADS;
    constexpr int P = sizeof(R) == 8 ? 1 : Op::WIDE ? 1 : 4;
    constexpr int BLK = sizeof(R) == 8 ? (Op::WIDE ? 4 : 8) : 6;
    // As many i a block as leave 600 blocks (four an SM): more i share a j
    // load and fill the warps that add, fewer leave SMs idle (AccJerk at
    // N = 3001: 751 blocks of 4 i 0.55 ms, 376 of 8 i 0.70 ms; at 32768
    // 8 or 16 i within 1 %).  The I x NO sums have to fit the block.
    int li = 5;
    while ((Op::NO << li) > T) --li;
    while ((1 << li) > P && (s.ni >> li) < 600) --li;
    if (one_i_a_thread<Op, R>(s.ni, s.nj, T * P >> li)) {
        const unsigned b = (unsigned)((s.ni + SWEEP_T - 1) / SWEEP_T);
        g_launch_count += 1;
        return launch_chained(exact_sweep<Op, R>, b, SWEEP_T, 0, st, s);
    }
    if constexpr (sizeof(R) == 8) {
        // One i a block where its sums are the bound: while no SM has more
        // than two blocks (AccJerk 300 x 8192 380 us against 477, 600 x 3000
        // equal, 1000 x 1000 137 against 107), and up to 5000 i if each sum
        // has a warp of its own (Phi at 3001 x 3001 267 us against 320, at
        // 8192 equal; Tstep at 5000 x 5000 1.61 against 1.81 ms, at 8192 7 %
        // slower) and j enough to fill it (Phi at 1500 x 512 53 us against
        // 41, x 1024 73 and 80; at 5000 x 1024 208 and 174, x 2048 318 and
        // 345; Tstep at 5000 x 16 73 and 9).
        constexpr uint64_t most = few_owned<Op>() == Op::NO ? 5000 : FEW_I;
        if (s.ni <= FEW_I || (s.ni <= most && 3 * s.nj >= s.ni)) {
            g_launch_count += 1;
            return launch_chained(exact_few<Op>, (unsigned)s.ni,
                                  few_threads<Op>(), 0, st, s);
        }
    }
    const unsigned blocks = (unsigned)((s.ni + (1u << li) - 1) >> li);
    g_launch_count += 1;
    // A dear term is left out where nobody reads it: a Sakura solve (1000 x 4
    // 246 us without, 97 with), and PnAcc's in double against fewer j than a
    // tile may have rows (1000 x 4 46 us and 17; in a long sweep it would
    // cost up to 13 %).
    constexpr bool solves = std::is_same<Op, SakuraPair<R>>::value;
    if constexpr (Op::WIDE && !solves && sizeof(R) == 8)
        if (s.nj < T)
            return launch_chained(exact_terms<Op, R, T, P, BLK, true>, blocks,
                                  T, 0, st, s, li);
    return launch_chained(exact_terms<Op, R, T, P, BLK, solves>, blocks, T, 0,
                          st, s, li);
}

template <typename R>
cudaError_t launch_exact(const Sweep &s, cudaStream_t st, long long budget,
                         unsigned *err)
{
    if (s.kernel == K_KEPLER) {
        exact_kepler<R><<<1, 32, 0, st>>>(s, budget, err);
        g_launch_count += 1;
        return cudaGetLastError();
    }
    if (s.ni == 0) return cudaSuccess;
    switch (s.kernel) {
    case K_PHI: return run_exact<PhiPair<R>, R>(s, st);
    case K_ACC: return run_exact<AccPair<R>, R>(s, st);
    case K_ACC_JERK: return run_exact<AccJerkPair<R>, R>(s, st);
    case K_SNAP_CRACKLE: return run_exact<SnapCracklePair<R>, R>(s, st);
    case K_TSTEP: return run_exact<TstepPair<R>, R>(s, st);
    case K_PNACC: return run_exact<PnAccPair<R>, R>(s, st);
    case K_NREG_X: return run_exact<NregXPair<R>, R>(s, st);
    case K_NREG_V: return run_exact<NregVPair<R>, R>(s, st);
    case K_SAKURA: {
        Sweep k = s;
        k.budget = budget;
        k.err = err;
        return run_exact<SakuraPair<R>, R>(k, st);
    }
    default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_exact<double>(const Sweep &, cudaStream_t,
                                          long long, unsigned *);
template cudaError_t launch_exact<float>(const Sweep &, cudaStream_t,
                                         long long, unsigned *);

}  // namespace tg
