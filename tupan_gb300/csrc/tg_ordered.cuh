// Sequential binary64 sums by a whole warp, with the bits of the one-by-one
// additions.
//
// While a running sum o stays in one binade, its ulp g is fixed and adding a
// term rounds to the grid g: o + t becomes o + g r, r the integer nearest
// t / g.  The r do not depend on o, so they are formed in parallel and added
// as integers, where the order does not matter.  What has to be shown for a
// run of terms is that every prefix stays strictly inside the binade (in
// units of g: 2^52 < |prefix| < 2^53; at 2^52 itself the grid below is
// finer) and that no t / g is a tie (which would round by o's parity).  The
// first group of terms that breaks this is added one by one, then the run
// goes on from there.
//
// Why: a chain of dependent FP64 additions takes 64 cycles a term on this
// GPU.  Measured on one warp (cycles a term, sums of 1024 / 8192 terms):
// one-signed uniform terms 21 / 10, heavy-tailed ones of both signs (a body's
// force components) 26 .. 34 / 11 .. 14, uniform terms of zero mean, whose
// sum keeps crossing binades, 81 / 52.
#pragma once

#include <stdint.h>

namespace tg {

// Terms of a group, and terms of a full run (one group a lane).
constexpr int ORD_K = 4;
constexpr int ORD_RUN = 32 * ORD_K;
// Place of term n of a run in shared memory (lane n / ORD_K reads its terms
// without bank conflicts); a run takes ORD_PITCH * ORD_K doubles.
constexpr int ORD_PITCH = 33;
__device__ __forceinline__ int ord_at(int n)
{
    return (n % ORD_K) * ORD_PITCH + n / ORD_K;
}

// ((o + t[0]) + t[1]) + .. over n <= ORD_RUN terms laid out by ord_at.  All
// 32 lanes call it and get the result.
__device__ __forceinline__ double ordered_sum(double o, const double *t, int n)
{
    const int lane = threadIdx.x & 31;
    const int groups = (n + ORD_K - 1) / ORD_K;
    double x[ORD_K];
#pragma unroll
    for (int k = 0; k < ORD_K; ++k) {
        // terms past the end are -0, which leaves every o as it is
        x[k] = lane * ORD_K + k < n ? t[k * ORD_PITCH + lane] : -0.0;
    }
    int first = 0;          // groups before it are in o
    int alone = 1;          // groups added one by one after a break
    while (first < groups) {
        const uint32_t oh = (uint32_t)__double2hiint(o);
        const int eo = (int)((oh >> 20) & 0x7ffu);
        const uint32_t so = oh & 0x80000000u;
        const bool zero = eo == 0;
        int stop = first;   // first group that cannot be taken in this pass
        if (eo > 64 && eo < 2047) {
            const long long M =
                (long long)(((unsigned long long)((oh & 0xfffffu) | 0x100000u)
                             << 32) | (uint32_t)__double2loint(o));
            long long p[ORD_K], s = 0;
            bool bad = false;
#pragma unroll
            for (int k = 0; k < ORD_K; ++k) {
                const uint32_t h = (uint32_t)__double2hiint(x[k]);
                const int et = (int)((h >> 20) & 0x7ffu);
                const unsigned long long m =
                    ((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) |
                    (uint32_t)__double2loint(x[k]);
                const int sh = eo - et;
                // |t| / g = m 2^-sh: below 1/2 from sh = 54 on (and for
                // et = 0, where eo > 64)
                const int c = sh < 1 ? 0 : sh;
                const unsigned long long half = (1ull << (c < 63 ? c : 63)) >> 1;
                const unsigned long long q =
                    sh > 53 ? 0ull : (m + half) >> (c < 63 ? c : 63);
                bad |= sh < 0 ||
                       (sh > 0 && sh < 54 &&
                        ((m + half) & (2 * half - 1)) == 0ull);
                s += (h ^ so) & 0x80000000u ? -(long long)q : (long long)q;
                p[k] = s;
            }
            const bool mine = lane >= first && lane < groups;
            bad = bad && mine;
            if (!mine || bad) s = 0;
            long long incl = s;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const long long u = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += u;
            }
            const long long before = M + (incl - s);
            if (mine && !bad) {
                bad = before <= (1ll << 52) && first != lane;
#pragma unroll
                for (int k = 0; k < ORD_K; ++k)
                    bad |= (unsigned long long)(before + p[k] -
                                                ((1ll << 52) + 1)) >=
                           (1ull << 52) - 1;
                // adding to exactly 2^52 g
                bad |= before == (1ll << 52);
            }
            const unsigned b = __ballot_sync(0xffffffffu, bad);
            stop = b ? __ffs((int)b) - 1 : groups;
            const long long P = __shfl_sync(0xffffffffu, b ? before : M + incl,
                                            b ? stop : 31);
            o = __hiloint2double(
                (int)((uint32_t)((unsigned long long)P >> 32) +
                      ((uint32_t)(eo - 1) << 20) + so),
                (int)(uint32_t)P);
        }
        // a sum that keeps leaving its binade takes longer stretches one by
        // one, so that no input costs much more than the plain chain
        alone = zero ? 32 : stop == first ? 4 : 1;
        first = stop;
        for (int k = 0; k < alone && first < groups; ++k, ++first)
#pragma unroll
            for (int c = 0; c < ORD_K; ++c)
                o = o + __shfl_sync(0xffffffffu, x[c], first);
    }
    return o;
}

}  // namespace tg
