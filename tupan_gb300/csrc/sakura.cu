// Sakura sweep with the Kepler-branch pairs solved as a separate queue, and
// a standalone universal-Kepler pair solver with an optional learned start.
//
// tupan's sakura_kernel (sakura_kernel.c:33-62) evolves every (i, j) pair as
// a two-body problem over dt: about 99 % of pairs take the leapfrog branch
// (r^2 > (64 m / v^2)^2, sakura_kernel_common.h:111-117), the rest the
// iterative universal-variable solver.  Run inline, one Kepler pair stalls
// its whole warp.  Here, for the flags the Sakura integrator uses (-1, +1):
//   1. sum the leapfrog pairs in j order, append the Kepler pairs (i, j and
//      the rank among their i's) to a queue and count them per i;
//   2. exclusive scan of the counts: pair (i, rank)'s place in j order;
//   3. solve the queue, one thread per pair (coherent work);
//   4. add each i's Kepler contributions, in j order, to its leapfrog sum.
// The counts stay on the device; a queue that turns out too small is grown
// and the sweep repeated.
// The leapfrog branch is bit-identical to the reference (compiled without
// contraction); the result differs from the reference's interleaved sum only
// by the order of the additions, and the Kepler branch by CUDA's
// transcendental functions.
//
// The pair solver is also the engine of the learned start: an MLP
// (4 -> 64 -> 64 -> 1, SiLU, bf16 weights, FP32 accumulation) predicts the
// ratio of the converged universal anomaly to the plain first guess; the
// plain Laguerre iteration then runs to the unchanged tolerance.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <mutex>
#include <unordered_map>

#include "tg_common.cuh"
#include "tg_kepler.cuh"
#include "tg_split_ops.cuh"

#define TG_EXPORT extern "C" __attribute__((visibility("default")))

namespace tg {

cudaError_t launch_pack_both(int kernel, uint64_t ni, const unsigned *ni_dev,
                             const void *const *iattrs, float4 *iout,
                             uint64_t nj, const void *const *jattrs,
                             float4 *jout, cudaStream_t st);

// ---------------------------------------------------------------------------
// Learned start: parameters in device memory.
// ---------------------------------------------------------------------------
constexpr int MLP_IN = 4, MLP_H = 64;

struct MlpParams {
    const __nv_bfloat16 *w1;   // MLP_H x MLP_IN
    const float *b1;           // MLP_H
    const __nv_bfloat16 *w2;   // MLP_H x MLP_H
    const float *b2;           // MLP_H
    const __nv_bfloat16 *w3;   // MLP_H
    const float *b3;           // 1
    const float *norm;         // mean[4], 1/std[4] of the features
    float gate;                // learned start only where feature 3 exceeds it
};

__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }

// Features of a single-step solve, from the quantities of kep_setup, in
// FP32 (they only feed the network's guess): log r0, log |v0|, the cosine of
// the angle between r0 and v0, and the orbital phase of the step
// log(|dt| sqrt(m / r0^3)), formed from logarithms so that no power
// overflows.  kep_phase alone decides whether the network is evaluated.
__device__ __forceinline__ float kep_phase(const KepArg<double> &k)
{
    const float lr = __logf((float)k.r0);
    return __logf(fabsf((float)k.dt)) + 0.5f * (__logf((float)k.m) - 3.0f * lr);
}

__device__ __forceinline__ void kep_features(const KepArg<double> &k,
                                             const double *p, float *f)
{
    const float vx = (float)p[3], vy = (float)p[4], vz = (float)p[5];
    const float v = sqrtf(vx * vx + vy * vy + vz * vz);
    const float vs = v > 0.f ? v : 1e-30f;
    const float r = (float)k.r0;
    f[0] = __logf(r);
    f[1] = __logf(vs);
    f[2] = (float)k.rv0 / (r * vs);
    f[3] = kep_phase(k);
}

// Learned start of one solve: s0 scaled by exp(network); false (keep the
// plain guess) when the network's output is not finite.
__device__ __forceinline__ bool learned_start(double s0, double *start,
                                              float y)
{
    if (!isfinite(y)) return false;
    *start = s0 * (double)__expf(y);
    return true;
}

// Weights are shared by every thread of a block: staged once in shared memory
// (bf16), activations in registers, FP32 fused multiply-adds.
struct MlpSmem {
    __nv_bfloat16 w1[MLP_H * MLP_IN];
    __nv_bfloat16 w2[MLP_H * MLP_H];
    __nv_bfloat16 w3[MLP_H];
    float b1[MLP_H], b2[MLP_H], b3, norm[8];
};

__device__ void mlp_stage(MlpSmem &S, const MlpParams &P)
{
    for (int t = threadIdx.x; t < MLP_H * MLP_H; t += blockDim.x) {
        S.w2[t] = P.w2[t];
        if (t < MLP_H * MLP_IN) S.w1[t] = P.w1[t];
        if (t < MLP_H) {
            S.w3[t] = P.w3[t];
            S.b1[t] = P.b1[t];
            S.b2[t] = P.b2[t];
        }
        if (t < 8) S.norm[t] = P.norm[t];
        if (t == 0) S.b3 = P.b3[0];
    }
}

__device__ float mlp_eval(const MlpSmem &S, const float *x_raw)
{
    float x[MLP_IN];
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k)
        x[k] = (x_raw[k] - S.norm[k]) * S.norm[4 + k];
    float h1[MLP_H];
#pragma unroll
    for (int o = 0; o < MLP_H; ++o) {
        float a = S.b1[o];
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k)
            a = __fmaf_rn(__bfloat162float(S.w1[o * MLP_IN + k]), x[k], a);
        h1[o] = silu(a);
    }
    float y = S.b3;
    for (int o = 0; o < MLP_H; ++o) {
        float a = S.b2[o];
#pragma unroll
        for (int k = 0; k < MLP_H; ++k)
            a = __fmaf_rn(__bfloat162float(S.w2[o * MLP_H + k]), h1[k], a);
        y = __fmaf_rn(__bfloat162float(S.w3[o]), silu(a), y);
    }
    return y;
}

// ---------------------------------------------------------------------------
// Standalone pair solver: one universal_kepler_solver per pair (as the Kepler
// branch of twobody_solver calls it), optional learned start, optional record
// of (features, log(root / plain guess)) of each pair's first single-step
// solve for training.
// ---------------------------------------------------------------------------
struct PairSolve {
    uint64_t n;
    double dt;
    const double *m, *e2, *state;   // state: n x 6 (r, v)
    double *out;                    // n x 6
    int *iters;                     // Laguerre updates per pair (or null)
    float *rec_x, *rec_y;           // n x 4 features, n targets (or null)
    long long budget;
    int use_mlp;
    int form;                       // KeplerForm of the single-step solves
    MlpParams mlp;
};

__global__ void __launch_bounds__(128)
k_pair_solve(const PairSolve P, unsigned *err)
{
    __shared__ MlpSmem S;
    if (P.use_mlp) mlp_stage(S, P.mlp);
    __syncthreads();
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    double p0[6], p1[6];
    for (int c = 0; c < 6; ++c) p0[c] = P.state[6 * q + c];
    const double m = P.m[q], e2 = P.e2[q];
    KepCtx<double> ctx = {0, P.budget, 0, false, false, 0.0};
    ctx.form = P.form;
    KepArg<double> ka;
    double s0;
    const bool moving = kep_setup(P.dt, m, e2, p0, &ka, &s0);
    if (moving && P.use_mlp && !P.rec_x && kep_phase(ka) > P.mlp.gate) {
        float f[MLP_IN];
        kep_features(ka, p0, f);
        ctx.use_start = learned_start(s0, &ctx.start, mlp_eval(S, f));
    }
    if (moving && P.rec_x) {
        float f[MLP_IN];
        kep_features(ka, p0, f);
        if (P.use_mlp && f[3] > P.mlp.gate)
            ctx.use_start = learned_start(s0, &ctx.start, mlp_eval(S, f));
        for (int k = 0; k < MLP_IN; ++k) P.rec_x[4 * q + k] = f[k];
        double root;
        int it = 0;
        const int st = kep_laguerre(s0, &root, ka, &it);
        P.rec_y[q] = (st == 0 && root / s0 > 0)
                         ? (float)log(root / s0) : __int_as_float(0x7fc00000);
    }
    kep_solve(P.dt, m, e2, p0, p1, ctx);
    for (int c = 0; c < 6; ++c) P.out[6 * q + c] = p1[c];
    if (P.iters) P.iters[q] = (int)ctx.iterations;
    if (ctx.exhausted) atomicOr(err, (unsigned)DERR_KEPLER_BUDGET);
}

// ---------------------------------------------------------------------------
// Queued Sakura sweep (flags -1 and +1).
// ---------------------------------------------------------------------------
constexpr int SK_THREADS = 128;

// What a sweep reports back: Kepler pairs found, Laguerre-update histogram
// (bin k: solves with k updates, the last 64 or more), error word.
struct SakuraReport {
    unsigned long long pairs;
    unsigned long long hist[65];
    unsigned err;
};

struct SakuraArgs {
    uint64_t ni, nj;
    const double *ip[8], *jp[8];
    double *out[6];
    double dt;
    long long flag;
    unsigned *cnt;          // ni counts (step 1), then offsets (step 2)
    unsigned *queue_j;      // Kepler pairs: j index
    unsigned *queue_i;      // Kepler pairs: i index
    unsigned *queue_r;      // Kepler pairs: rank among their i's, in j order
    unsigned long long cap; // queue entries
    double *contrib;        // 6 per queued pair, in (i, j) order
    SakuraReport *rep;
    long long budget;
    int use_mlp;
    int form;               // KeplerForm of the Kepler-branch solves
    MlpParams mlp;
};

// Drift applied before the two-body step for flag -1 (sakura_kernel_common.h
// :151-157); flag +1 evolves first and drifts after (:158-164).
__device__ __forceinline__ void sk_start(const double *ip, const double *jp,
                                         double dt, long long flag,
                                         double *p0, double *pre, double *m,
                                         double *e2)
{
    pair_state(ip, jp, p0, m, e2);
    for (int c = 0; c < 6; ++c) pre[c] = p0[c];
    if (flag == -1) pair_drift(pre, pre + 3, dt, true);
}

// Pairs in parallel over i and j, I = 2^li i a block, one pair a thread; the
// leapfrog terms are folded in j order through shared memory (as
// exact_terms does), the Kepler pairs of each i are queued in j order (their
// terms enter the sum as +0, which changes no sum).
//
// One i a thread over all j, in two passes (count, then sum), the form this
// replaces, ran a 4096-body sweep on 32 SMs with its quotients on the FP64
// pipe: 23.9 ms a sweep with its solves, now 2.3 (N = 256: 1.70 ms, now
// 0.18).  Bound: the FP64 pipe, 39 additions a pair at 19 SM cycles a warp
// (1.3 ms of the 1.8 the kernel takes at N = 4096); eight blocks of 64
// registers an SM beat five of 96 by 11 %.
__global__ void __launch_bounds__(SK_THREADS, 8)
k_sakura_pass(const SakuraArgs A, const int li)
{
    constexpr int T = SK_THREADS, NO = 6;
    __shared__ double buf[2][NO][T];
    __shared__ unsigned near[2][T / 32];
    const int tid = threadIdx.x, ii = tid & ((1 << li) - 1), row = tid >> li;
    const int J = T >> li;
    const uint64_t i0 = (uint64_t)blockIdx.x << li;
    const uint64_t i = i0 + ii < A.ni ? i0 + ii : A.ni - 1;
    double ip[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) ip[a] = A.ip[a][i];
    const double dt = A.dt;
    const long long flag = A.flag;
    const bool sums = row < NO, queues = row == NO && i0 + ii < A.ni;
    double o = 0.0;
    unsigned count = 0;
    unsigned lanes = 0;             // this i's lanes of a warp
    for (int k = 0; k < 32; k += 1 << li) lanes |= 1u << (k + ii);
    int b = 0;
    for (uint64_t j0 = 0; j0 < A.nj; j0 += J, b ^= 1) {
        const uint64_t j = j0 + row < A.nj ? j0 + row : A.nj - 1;
        double jp[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) jp[a] = A.jp[a][j];
        double p0[6], pre[6], m, e2;
        sk_start(ip, jp, dt, flag, p0, pre, &m, &e2);
        const bool far = takes_leapfrog(m, pre);
        double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (far) {
            double p1[6];
            two_body_leapfrog(dt, m, e2, pre, p1);
            if (flag == 1) pair_drift(p1, p1 + 3, dt, true);
            pair_term(jp[0], m, p0, p1, t);
        }
#pragma unroll
        for (int c = 0; c < NO; ++c) buf[b][c][tid] = t[c];
        const unsigned v = __ballot_sync(0xffffffffu,
                                         !far && j0 + row < A.nj);
        if ((tid & 31) == 0) near[b][tid >> 5] = v;
        __syncthreads();
        if (sums) {
            const int n = A.nj - j0 < (uint64_t)J ? (int)(A.nj - j0) : J;
            const double *q = &buf[b][row][ii];
#pragma unroll 8
            for (int k = 0; k < n; ++k) o += q[k << li];
        } else if (queues) {
            unsigned f[T / 32], n = 0;
#pragma unroll
            for (int k = 0; k < T / 32; ++k) {
                f[k] = near[b][k] & lanes;
                n += __popc(f[k]);
            }
            if (n) {
                unsigned long long at = atomicAdd(&A.rep->pairs,
                                                  (unsigned long long)n);
#pragma unroll
                for (int k = 0; k < T / 32; ++k)
                    for (; f[k]; f[k] &= f[k] - 1, ++at, ++count)
                        if (at < A.cap) {
                            const int l = 32 * k + __ffs((int)f[k]) - 1;
                            A.queue_j[at] = (unsigned)(j0 + (l >> li));
                            A.queue_i[at] = (unsigned)i;
                            A.queue_r[at] = count;
                        }
            }
        }
    }
    if (sums && i0 + ii < A.ni) A.out[row][i] = o;
    if (queues) A.cnt[i] = count;
}

// The i's a block of the pass: as many (up to 16, the six sums and the
// queue of each have to fit the block) as leave 600 blocks.
int sk_li(uint64_t ni)
{
    int li = 4;
    while (li > 0 && (ni >> li) < 600) --li;
    return li;
}

// SPLIT mode of the pass (flags -1 and +1): FP32 pair arithmetic on
// the packed double-single records.  In the leapfrog branch the pair's
// change over the step has a closed form: with the midpoint position
// b = r0 + flag v0 dt/2 and a = -m b / |b|^3 (softened), the velocity
// changes by a dt and the position by -flag a dt^2/2 (the algebra of
// sakura_kernel_common.h:45-91 with :151-164), so each pair is one
// acceleration evaluation formed directly as increments (no difference of
// nearly equal FP32 states).  The branch test is the reference's
// (r^2 > (64 m / v^2)^2, sakura_kernel_common.h:109-123) in FP32.  Kepler-branch pairs go to the same
// queue and fp64 solver as in EXACT mode.
constexpr int SKS_TILE = 256;

__global__ void __launch_bounds__(SK_THREADS)
k_sakura_split_pass(const SakuraArgs A, const float4 *irec, const float4 *jrec)
{
    __shared__ float4 tile[SKS_TILE * 3];
    const uint64_t i = (uint64_t)blockIdx.x * SK_THREADS + threadIdx.x;
    const uint64_t ic = i < A.ni ? i : A.ni - 1;
    const float4 ia = irec[3 * ic], ib = irec[3 * ic + 1], iv = irec[3 * ic + 2];
    const float fl = (float)A.flag;
    const float dt = (float)A.dt, hdt = 0.5f * dt, dt2h = 0.5f * dt * dt;
    double o[6] = {0, 0, 0, 0, 0, 0};
    float part[6] = {0, 0, 0, 0, 0, 0};
    int run = 0;
    unsigned count = 0;
    for (uint64_t j0 = 0; j0 < A.nj; j0 += SKS_TILE) {
        const int n = (int)((A.nj - j0) < SKS_TILE ? (A.nj - j0) : SKS_TILE);
        __syncthreads();
        for (int t = threadIdx.x; t < 3 * n; t += SK_THREADS)
            tile[t] = jrec[3 * j0 + t];
        __syncthreads();
        for (int jj = 0; jj < n; ++jj) {
            const float4 ja = tile[3 * jj], jb = tile[3 * jj + 1],
                         jv = tile[3 * jj + 2];
            const float dx = (ia.x - ja.x) + (ib.x - jb.x);
            const float dy = (ia.y - ja.y) + (ib.y - jb.y);
            const float dz = (ia.z - ja.z) + (ib.z - jb.z);
            const float ux = iv.x - jv.x, uy = iv.y - jv.y, uz = iv.z - jv.z;
            const float m = ia.w + ja.w, e2 = ib.w + jb.w;
            // state the two-body step starts from: flag -1 drifts back first
            const float sh = fl < 0.f ? -dt : 0.f;
            const float px = fmaf(ux, sh, dx), py = fmaf(uy, sh, dy),
                        pz = fmaf(uz, sh, dz);
            const float r2p = fmaf(pz, pz, fmaf(py, py, px * px));
            const float v2 = fmaf(uz, uz, fmaf(uy, uy, ux * ux));
            const float R = 64.0f * (m / v2);
            if (!(r2p > R * R)) {           // Kepler branch
                if (i < A.ni) {
                    const unsigned long long at =
                        atomicAdd(&A.rep->pairs, 1ull);
                    if (at < A.cap) {
                        A.queue_j[at] = (unsigned)(j0 + jj);
                        A.queue_i[at] = (unsigned)i;
                        A.queue_r[at] = count;
                    }
                }
                ++count;
                continue;
            }
            const float bx = fmaf(ux, fl * hdt, dx), by = fmaf(uy, fl * hdt, dy),
                        bz = fmaf(uz, fl * hdt, dz);
            const float r2b = fmaf(bz, bz, fmaf(by, by, bx * bx));
            float y = rsqrt_nr(r2b + e2);
            y = r2b > 0.f ? y : 0.f;
            const float jmk = -ja.w * (y * y) * y;      // -(m_j/m) m k
            const float av = jmk * dt, ar = -fl * jmk * dt2h;
            part[0] = fmaf(ar, bx, part[0]);
            part[1] = fmaf(ar, by, part[1]);
            part[2] = fmaf(ar, bz, part[2]);
            part[3] = fmaf(av, bx, part[3]);
            part[4] = fmaf(av, by, part[4]);
            part[5] = fmaf(av, bz, part[5]);
            if (++run == 16) {
                for (int q = 0; q < 6; ++q) {
                    o[q] += (double)part[q];
                    part[q] = 0.f;
                }
                run = 0;
            }
        }
    }
    if (i >= A.ni) return;
    A.cnt[i] = count;
    for (int q = 0; q < 6; ++q) A.out[q][i] = o[q] + (double)part[q];
}

// Exclusive scan of n counts in place (one block).
__global__ void k_scan(unsigned *x, uint64_t n)
{
    __shared__ unsigned long long carry;
    __shared__ unsigned long long part[1024];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t b = 0; b < n; b += blockDim.x) {
        const uint64_t i = b + threadIdx.x;
        unsigned long long v = i < n ? x[i] : 0;
        part[threadIdx.x] = v;
        __syncthreads();
        for (int off = 1; off < (int)blockDim.x; off <<= 1) {
            unsigned long long t =
                threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0;
            __syncthreads();
            part[threadIdx.x] += t;
            __syncthreads();
        }
        if (i < n) x[i] = (unsigned)(carry + part[threadIdx.x] - v);
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += part[threadIdx.x];
        __syncthreads();
    }
}

// Step 3: one thread per queued pair; its contribution goes to its place in
// (i, j) order.
__device__ __forceinline__ void sk_solve(const SakuraArgs &A, uint64_t q,
                                         const MlpSmem &S, unsigned *bins)
{
    const uint64_t i = A.queue_i[q], j = A.queue_j[q];
    const uint64_t at = (uint64_t)A.cnt[i] + A.queue_r[q];
    double ip[8], jp[8];
    for (int a = 0; a < 8; ++a) {
        ip[a] = A.ip[a][i];
        jp[a] = A.jp[a][j];
    }
    double p0[6], pre[6], m, e2, p1[6];
    sk_start(ip, jp, A.dt, A.flag, p0, pre, &m, &e2);
    KepCtx<double> ctx = {0, A.budget, 0, false, false, 0.0};
    ctx.form = A.form;
    if (A.use_mlp) {
        KepArg<double> ka;
        double s0;
        if (kep_setup(A.dt, m, e2, pre, &ka, &s0) &&
            kep_phase(ka) > A.mlp.gate) {
            float f[MLP_IN];
            kep_features(ka, pre, f);
            ctx.use_start = learned_start(s0, &ctx.start, mlp_eval(S, f));
        }
    }
    kep_solve(A.dt, m, e2, pre, p1, ctx);
    if (A.flag == 1) {
        p1[0] -= p1[3] * A.dt;
        p1[1] -= p1[4] * A.dt;
        p1[2] -= p1[5] * A.dt;
    }
    const double mu = jp[0] / m;
    for (int c = 0; c < 6; ++c) A.contrib[6 * at + c] = mu * (p1[c] - p0[c]);
    atomicAdd(&bins[ctx.iterations < 64 ? ctx.iterations : 64], 1u);
    if (ctx.exhausted) atomicOr(&A.rep->err, (unsigned)DERR_KEPLER_BUDGET);
}

__global__ void __launch_bounds__(SK_THREADS)
k_sakura_kepler(const SakuraArgs A)
{
    __shared__ MlpSmem S;
    __shared__ unsigned bins[65];
    const uint64_t nq = A.rep->pairs;
    if (nq > A.cap) return;           // the host repeats the sweep
    if (A.use_mlp) mlp_stage(S, A.mlp);
    if (threadIdx.x < 65) bins[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nq;
         q += (uint64_t)gridDim.x * blockDim.x)
        sk_solve(A, q, S, bins);
    __syncthreads();
    if (threadIdx.x < 65 && bins[threadIdx.x])
        atomicAdd(&A.rep->hist[threadIdx.x],
                  (unsigned long long)bins[threadIdx.x]);
}

// Step 4: add each i's queued contributions in queue (= j) order.  A warp an
// i: 32 contributions at a time come to shared memory coalesced, the next
// 32 while six lanes add (one thread an i, 48-byte strides, the form this
// replaces: 1.42 ms at N = 4096, where the heaviest body has thousands; now
// 0.18 ms).
__global__ void __launch_bounds__(SK_THREADS)
k_sakura_gather(const SakuraArgs A)
{
    __shared__ double part[SK_THREADS / 32][6 * 32];
    const uint64_t nq = A.rep->pairs;
    if (nq > A.cap) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t i = (uint64_t)blockIdx.x * (SK_THREADS / 32) + w;
    if (i >= A.ni) return;
    const uint64_t b = 6 * (uint64_t)A.cnt[i];
    const uint64_t e = 6 * ((i + 1 < A.ni) ? (uint64_t)A.cnt[i + 1] : nq);
    double o = lane < 6 ? A.out[lane][i] : 0.0, x[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
        x[k] = b + 32 * k + lane < e ? A.contrib[b + 32 * k + lane] : 0.0;
    for (uint64_t q = b; q < e; q += 192) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 6; ++k) part[w][32 * k + lane] = x[k];
        __syncwarp();
        const uint64_t nx = q + 192 + lane;
#pragma unroll
        for (int k = 0; k < 6; ++k)
            x[k] = nx + 32 * k < e ? A.contrib[nx + 32 * k] : 0.0;
        if (lane < 6) {
            const int n = e - q < 192 ? (int)(e - q) : 192;
#pragma unroll 8
            for (int k = lane; k < n; k += 6) o += part[w][k];
        }
    }
    if (lane < 6) A.out[lane][i] = o;
}

}  // namespace tg

using namespace tg;

namespace {

// Workspace of the queued sweeps and the pair solver on one device, grown as
// needed.  A call holds `mu` until its stream has finished with it, so calls
// from several threads or streams take turns.
struct SakuraWork {
    std::mutex mu;
    unsigned *cnt = nullptr;
    size_t cnt_cap = 0;
    unsigned *qi = nullptr, *qj = nullptr, *qr = nullptr;
    double *contrib = nullptr;
    size_t q_cap = 0;
    SakuraReport *rep = nullptr;
    unsigned *err = nullptr;          // kepler_pairs' error word
    float4 *rec = nullptr;            // SPLIT mode: packed i and j records
    size_t rec_cap = 0;
    int sms = 0;
};

MlpParams g_mlp;
bool g_have_mlp = false;
int g_kepler_form = KEP_REFERENCE;   // tupan_gb300_kepler_set_form

// The current device's workspace, or null without a device.
SakuraWork *device_work()
{
    static std::mutex mu;
    static std::unordered_map<int, SakuraWork *> works;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    SakuraWork *&w = works[dev];
    if (!w) w = new SakuraWork();
    return w;
}

// Status of a call that failed part way: what it launched is waited for, as
// the workspace goes to the next call, and the runtime's error is cleared,
// which the next sweep's launch would report as its own.
int failed(cudaStream_t st)
{
    cudaStreamSynchronize(st);
    cudaGetLastError();
    return ST_CUDA;
}

int grow_queue(SakuraWork &W, size_t cap)
{
    if (cap <= W.q_cap) return 0;
    cudaFree(W.qi);
    cudaFree(W.qj);
    cudaFree(W.qr);
    cudaFree(W.contrib);
    W.qi = W.qj = W.qr = nullptr;
    W.contrib = nullptr;
    W.q_cap = 0;
    if (cudaMalloc((void **)&W.qi, cap * sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc((void **)&W.qj, cap * sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc((void **)&W.qr, cap * sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc((void **)&W.contrib, cap * 6 * sizeof(double)) != cudaSuccess)
        return 1;
    W.q_cap = cap;
    return 0;
}

}  // namespace

// ===========================================================================
// C-ABI (no counterpart in the reference).
// ===========================================================================

// Installs (or, with w1 == NULL, removes) the learned-start network: DEVICE
// pointers to bf16 weights w1 (64x4), w2 (64x64), w3 (64), fp32 biases b1,
// b2, b3 and the feature normalisation norm[8] = mean[4], 1/std[4].  The
// network is evaluated only for solves whose feature log(|dt| sqrt(m/r^3))
// exceeds `gate` (where the plain guess needs more than the minimum two
// updates); elsewhere the plain guess is kept.  The arrays must stay valid
// while the network is installed.
TG_EXPORT int tupan_gb300_kepler_set_mlp(const void *w1, const float *b1,
                                         const void *w2, const float *b2,
                                         const void *w3, const float *b3,
                                         const float *norm, float gate)
{
    if (!w1) {
        g_have_mlp = false;
        return ST_OK;
    }
    g_mlp.w1 = (const __nv_bfloat16 *)w1;
    g_mlp.b1 = b1;
    g_mlp.w2 = (const __nv_bfloat16 *)w2;
    g_mlp.b2 = b2;
    g_mlp.w3 = (const __nv_bfloat16 *)w3;
    g_mlp.b3 = b3;
    g_mlp.norm = norm;
    g_mlp.gate = gate;
    g_have_mlp = true;
    return ST_OK;
}

// Form of the universal-Kepler root solve used by the pair solver, the
// queued Sakura sweep and the device Sakura integrator: 0 the reference's
// structure (default), 1 the same arithmetic with one cos/sin (cosh/sinh)
// per Laguerre update (bit-identical), 2 FP32 Laguerre updates then FP64
// updates to the reference's 2^-42 tolerance (see tg_kepler.cuh).  The ten
// libtupan.h entry points always use form 0.  Returns the previous form, or
// -1 for an unknown one.
TG_EXPORT int tupan_gb300_kepler_set_form(int form)
{
    if (form < KEP_REFERENCE || form > KEP_MIXED) return -1;
    const int old = g_kepler_form;
    g_kepler_form = form;
    return old;
}

// Solves n independent pairs (DEVICE arrays: m, e2, state n x 6, out n x 6)
// over dt with universal_kepler_solver's full retry logic; iters, rec_x
// (n x 4) and rec_y (n) are optional.  use_mlp selects the learned start.
// Synchronous, callable from several threads at once; returns a status code
// (3: a solve hit the budget).
TG_EXPORT int tupan_gb300_kepler_pairs(uint64_t n, double dt, const double *m,
                                       const double *e2, const double *state,
                                       double *out, int *iters, float *rec_x,
                                       float *rec_y, int use_mlp,
                                       long long budget, void *stream)
{
    if (use_mlp && !g_have_mlp) return ST_BAD_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    SakuraWork *const work = device_work();
    if (!work) return ST_CUDA;
    SakuraWork &W = *work;
    std::lock_guard<std::mutex> lock(W.mu);
    if (!W.err &&
        cudaMalloc((void **)&W.err, sizeof(unsigned)) != cudaSuccess)
        return failed(st);
    cudaMemsetAsync(W.err, 0, sizeof(unsigned), st);
    PairSolve P;
    memset(&P, 0, sizeof(P));
    P.n = n;
    P.dt = dt;
    P.m = m;
    P.e2 = e2;
    P.state = state;
    P.out = out;
    P.iters = iters;
    P.rec_x = rec_x;
    P.rec_y = rec_y;
    P.budget = budget > 0 ? budget : (1LL << 20);
    P.use_mlp = use_mlp;
    P.form = g_kepler_form;
    P.mlp = g_mlp;
    if (n) {
        k_pair_solve<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(P, W.err);
        g_launch_count += 1;
    }
    unsigned h = 0;
    if (cudaMemcpyAsync(&h, W.err, sizeof(unsigned), cudaMemcpyDeviceToHost,
                        st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return failed(st);
    return h ? ST_DEVICE : ST_OK;
}

// sakura_kernel (libtupan.h:203-229) on DEVICE arrays with the Kepler-branch
// pairs solved as a queue; flag must be -1 or +1 (the integrator's flags).
// i_attrs/j_attrs: 8 device pointers each (m r e2 v); outs: 6.  Optional
// iteration histogram: kepler_iters (host, 65 bins; bin k counts solves with
// k Laguerre updates, the last bin k >= 64).  Returns the number of queued
// (Kepler-branch) pairs in *n_kepler.  Synchronous, callable from several
// threads and streams at once.
TG_EXPORT int tupan_gb300_sakura_queue(uint64_t ni, const void *const *i_attrs,
                                       uint64_t nj, const void *const *j_attrs,
                                       double dt, int64_t flag,
                                       void *const *outs, int use_mlp,
                                       long long budget, void *stream,
                                       unsigned long long *n_kepler,
                                       long long *kepler_iters, int mode)
{
    if (flag != -1 && flag != 1) return ST_BAD_ARGUMENT;
    if (mode != MODE_EXACT && mode != MODE_SPLIT) return ST_BAD_ARGUMENT;
    if (use_mlp && !g_have_mlp) return ST_BAD_ARGUMENT;
    if (ni == 0) return ST_OK;
    cudaStream_t st = (cudaStream_t)stream;
    SakuraWork *const work = device_work();
    if (!work) return ST_CUDA;
    SakuraWork &W = *work;
    std::lock_guard<std::mutex> lock(W.mu);
    if (!W.rep) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&W.sms, cudaDevAttrMultiProcessorCount,
                                   dev) != cudaSuccess ||
            cudaMalloc((void **)&W.rep, sizeof(SakuraReport)) != cudaSuccess)
            return failed(st);
    }
    if (ni > W.cnt_cap) {
        cudaFree(W.cnt);
        W.cnt = nullptr;
        W.cnt_cap = 0;
        if (cudaMalloc((void **)&W.cnt, ni * sizeof(unsigned)) != cudaSuccess)
            return failed(st);
        W.cnt_cap = ni;
    }
    SakuraArgs A;
    memset(&A, 0, sizeof(A));
    A.ni = ni;
    A.nj = nj;
    for (int a = 0; a < 8; ++a) {
        A.ip[a] = (const double *)i_attrs[a];
        A.jp[a] = (const double *)j_attrs[a];
    }
    for (int c = 0; c < 6; ++c) A.out[c] = (double *)outs[c];
    A.dt = dt;
    A.flag = flag;
    A.cnt = W.cnt;
    A.budget = budget > 0 ? budget : (1LL << 20);
    A.use_mlp = use_mlp;
    A.form = g_kepler_form;
    A.mlp = g_mlp;
    A.rep = W.rep;
    const unsigned blocks = (unsigned)((ni + SK_THREADS - 1) / SK_THREADS);
    const int li = sk_li(ni);
    const unsigned eblocks = (unsigned)((ni + (1u << li) - 1) >> li);
    const float4 *irec = nullptr, *jrec = nullptr;
    if (mode == MODE_SPLIT) {
        bool same = ni == nj;
        for (int a = 0; a < 8 && same; ++a) same = i_attrs[a] == j_attrs[a];
        const size_t need = (ni + (same ? 0 : nj)) * 3;
        if (need > W.rec_cap) {
            cudaFree(W.rec);
            W.rec = nullptr;
            W.rec_cap = 0;
            if (cudaMalloc((void **)&W.rec, need * sizeof(float4)) !=
                cudaSuccess)
                return failed(st);
            W.rec_cap = need;
        }
        if (launch_pack_both(K_ACC_JERK, ni, nullptr, i_attrs, W.rec,
                             same ? 0 : nj, j_attrs, W.rec + ni * 3,
                             st) != cudaSuccess)
            return failed(st);
        irec = W.rec;
        jrec = same ? W.rec : W.rec + ni * 3;
    }
    // room for a pair in 32 (Salpeter spheres: 1 in 16 at N = 256, 125 at
    // 4096), at most 2^20 to begin with; the counts decide
    unsigned long long want = ni * nj / 32 + 4096;
    if (want > 1ull << 20) want = 1ull << 20;
    SakuraReport r;
    for (;;) {
        if (grow_queue(W, want)) return failed(st);
        A.queue_i = W.qi;
        A.queue_j = W.qj;
        A.queue_r = W.qr;
        A.cap = W.q_cap;
        A.contrib = W.contrib;
        cudaMemsetAsync(W.rep, 0, sizeof(SakuraReport), st);
        if (mode == MODE_SPLIT)
            k_sakura_split_pass<<<blocks, SK_THREADS, 0, st>>>(A, irec, jrec);
        else
            k_sakura_pass<<<eblocks, SK_THREADS, 0, st>>>(A, li);
        k_scan<<<1, 1024, 0, st>>>(W.cnt, ni);
        // the solves stride over the queue, whose length only the device
        // knows: five blocks of 96 registers a thread fill an SM
        k_sakura_kepler<<<(unsigned)(5 * W.sms), SK_THREADS, 0, st>>>(A);
        k_sakura_gather<<<(unsigned)((ni + 3) / 4), SK_THREADS, 0, st>>>(A);
        g_launch_count += 4;
        if (cudaMemcpyAsync(&r, W.rep, sizeof(r), cudaMemcpyDeviceToHost,
                            st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return failed(st);
        if (r.pairs <= A.cap) break;
        want = r.pairs + r.pairs / 4;
    }
    if (n_kepler) *n_kepler = r.pairs;
    if (kepler_iters)
        for (int k = 0; k < 65; ++k) kepler_iters[k] = (long long)r.hist[k];
    return r.err ? ST_DEVICE : ST_OK;
}

// ===========================================================================
// Device-resident Sakura integrator (sakura.py:22-50, fixed step): per step
// drift tau/2, queued Sakura sweeps with flag -1 then +1 at dt = tau/2, each
// followed by r += dr, v += dv, and a final drift tau/2.  State in HBM.
// ===========================================================================
namespace {

__global__ void k_drift(double *r0, double *r1, double *r2, const double *v0,
                        const double *v1, const double *v2, uint64_t n,
                        double tau)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        r0[i] = r0[i] + v0[i] * tau / 2;
        r1[i] = r1[i] + v1[i] * tau / 2;
        r2[i] = r2[i] + v2[i] * tau / 2;
    }
}

__global__ void k_kick(double *const *x, const double *const *d, uint64_t n)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        for (int c = 0; c < 6; ++c) x[c][i] = x[c][i] + d[c][i];
}

struct SakuraSys {
    uint64_t n = 0;
    double *pool = nullptr;          // m e2 r3 v3 d6
    double *a[8];                    // m r(3) e2 v(3), the kernels' order
    double *d[6];
    double **xd = nullptr, **dd = nullptr;   // device arrays of pointers
    cudaStream_t stream = nullptr;
    int use_mlp = 0;
    int mode = MODE_EXACT;           // Sakura sweeps: EXACT or SPLIT
    long long kepler_total = 0, steps = 0;
    long long hist[65] = {0};
    double t = 0.0;
};

}  // namespace

TG_EXPORT int tupan_gb300_sakura_destroy(void *handle);

TG_EXPORT int tupan_gb300_sakura_create(uint64_t n, const double *m,
                                        const double *e2, const double *rx,
                                        const double *ry, const double *rz,
                                        const double *vx, const double *vy,
                                        const double *vz, void **handle)
{
    if (!handle || n == 0) return ST_BAD_ARGUMENT;
    SakuraSys *S = new SakuraSys();
    CreateGuard guard{S, tupan_gb300_sakura_destroy};
    S->n = n;
    if (cudaStreamCreateWithFlags(&S->stream, cudaStreamNonBlocking) !=
            cudaSuccess ||
        cudaMalloc((void **)&S->pool, 14 * n * sizeof(double)) != cudaSuccess ||
        cudaMalloc((void **)&S->xd, 6 * sizeof(double *)) != cudaSuccess ||
        cudaMalloc((void **)&S->dd, 6 * sizeof(double *)) != cudaSuccess)
        return ST_CUDA;
    for (int k = 0; k < 8; ++k) S->a[k] = S->pool + (size_t)k * n;
    for (int k = 0; k < 6; ++k) S->d[k] = S->pool + (size_t)(8 + k) * n;
    const double *src[8] = {m, rx, ry, rz, e2, vx, vy, vz};
    for (int k = 0; k < 8; ++k)
        if (cudaMemcpy(S->a[k], src[k], n * sizeof(double),
                       cudaMemcpyHostToDevice) != cudaSuccess)
            return ST_CUDA;
    double *xs[6] = {S->a[1], S->a[2], S->a[3], S->a[5], S->a[6], S->a[7]};
    cudaMemcpy(S->xd, xs, sizeof(xs), cudaMemcpyHostToDevice);
    cudaMemcpy(S->dd, S->d, sizeof(S->d), cudaMemcpyHostToDevice);
    *handle = S;
    guard.keep();
    return ST_OK;
}

// Fixed-step Sakura steps of size tau until t >= t_end (t_end - t a multiple
// of tau is the intended use).  use_mlp: learned Kepler start.  kepler_iters
// (host, 65 bins) accumulates the Laguerre-update histogram if not NULL.
TG_EXPORT int tupan_gb300_sakura_evolve(void *handle, double tau, double t_end,
                                        int use_mlp, double *t_out,
                                        long long *steps_out,
                                        long long *kepler_out,
                                        long long *kepler_iters)
{
    SakuraSys *S = (SakuraSys *)handle;
    if (!S || !(tau > 0)) return ST_BAD_ARGUMENT;
    const uint64_t n = S->n;
    const unsigned g = (unsigned)((n + 255) / 256 < 1216 ? (n + 255) / 256 : 1216);
    void *ia[8];
    for (int k = 0; k < 8; ++k) ia[k] = S->a[k];
    void *oa[6];
    for (int k = 0; k < 6; ++k) oa[k] = S->d[k];
    long long h[65];
    while (S->t < t_end) {
        k_drift<<<g, 256, 0, S->stream>>>(S->a[1], S->a[2], S->a[3], S->a[5],
                                          S->a[6], S->a[7], n, tau);
        g_launch_count += 1;
        for (int flag = -1; flag <= 1; flag += 2) {
            unsigned long long nk = 0;
            int st = tupan_gb300_sakura_queue(n, ia, n, ia, tau / 2, flag, oa,
                                              use_mlp, 0, S->stream, &nk,
                                              kepler_iters ? h : nullptr,
                                              S->mode);
            if (st) return st;
            S->kepler_total += (long long)nk;
            if (kepler_iters)
                for (int k = 0; k < 65; ++k) kepler_iters[k] += h[k];
            k_kick<<<g, 256, 0, S->stream>>>(S->xd, S->dd, n);
            g_launch_count += 1;
        }
        k_drift<<<g, 256, 0, S->stream>>>(S->a[1], S->a[2], S->a[3], S->a[5],
                                          S->a[6], S->a[7], n, tau);
        g_launch_count += 1;
        S->t += tau;
        S->steps += 1;
    }
    if (cudaStreamSynchronize(S->stream) != cudaSuccess) return ST_CUDA;
    if (t_out) *t_out = S->t;
    if (steps_out) *steps_out = S->steps;
    if (kepler_out) *kepler_out = S->kepler_total;
    return ST_OK;
}

// Sakura sweeps of the integrator: mode 0 EXACT (default), 1 SPLIT.
TG_EXPORT int tupan_gb300_sakura_set_mode(void *handle, int mode)
{
    SakuraSys *S = (SakuraSys *)handle;
    if (!S || (mode != MODE_EXACT && mode != MODE_SPLIT)) return ST_BAD_ARGUMENT;
    S->mode = mode;
    return ST_OK;
}

TG_EXPORT int tupan_gb300_sakura_get_state(void *handle, double *rx,
                                           double *ry, double *rz, double *vx,
                                           double *vy, double *vz)
{
    SakuraSys *S = (SakuraSys *)handle;
    if (!S) return ST_BAD_ARGUMENT;
    double *dst[6] = {rx, ry, rz, vx, vy, vz};
    double *src[6] = {S->a[1], S->a[2], S->a[3], S->a[5], S->a[6], S->a[7]};
    for (int k = 0; k < 6; ++k)
        if (cudaMemcpy(dst[k], src[k], S->n * sizeof(double),
                       cudaMemcpyDeviceToHost) != cudaSuccess)
            return ST_CUDA;
    return ST_OK;
}

TG_EXPORT int tupan_gb300_sakura_destroy(void *handle)
{
    SakuraSys *S = (SakuraSys *)handle;
    if (!S) return ST_BAD_ARGUMENT;
    cudaStreamSynchronize(S->stream);
    cudaFree(S->pool);
    cudaFree(S->xd);
    cudaFree(S->dd);
    if (S->stream) cudaStreamDestroy(S->stream);
    delete S;
    return ST_OK;
}
