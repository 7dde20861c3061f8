// permutation.cu -- the training's shuffled order, drawn on the device.
//
// The order is the one that the sequential shuffle gives: A = 0 .. n - 1, then for
// i = n - 1 down to 1 swap A[i] with A[h_i], h_i = splitmix64's (n - i)-th word mod
// (i + 1).  The swaps commute unless they share a place, so they run in rounds
// (deterministic reservations; Shun, Gu, Blelloch, Fineman, Gibbons, "Sequential random
// permutation, list contraction and tree contraction are highly parallel", SODA 2015):
// every swap left writes its i, by maximum, on its two places, and the swaps that find
// their own i on both are the ones that the sequential order would do next there.  The
// number of rounds grows with log n (about 40 for 10^5); a round is two grid barriers of
// one cooperative kernel.  On a host core the shuffle of 124,519 rows took 720 us, as
// long as twelve training steps.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "surrogate_internal.h"

namespace cg = cooperative_groups;

namespace cgppd {

namespace {

constexpr int kPermThreads = 1024;

__device__ __forceinline__ uint64_t splitmix64_at(uint64_t state, uint64_t k)
{
    uint64_t z = state + k * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// place[p]: (round, i) of the last reservation of p, later rounds above earlier ones, so
// nothing is cleared between rounds.  partner[i] = h_i, -1 once swapped.  left[3]: swaps
// left after rounds of each residue mod 3 (every block reads a round's count before the
// next barrier, and it is cleared two rounds on: all blocks leave after the same round).
__global__ void __launch_bounds__(kPermThreads) k_permutation(int n, uint64_t state, int *perm, int *partner,
                                                              unsigned long long *place, unsigned *left)
{
    cg::grid_group grid = cg::this_grid();
    const int t = (int)grid.thread_rank(), T = (int)grid.size();
    for (int i = t; i < n; i += T) {
        perm[i] = i;
        place[i] = 0ull;
        partner[i] = i > 0 ? (int)(splitmix64_at(state, (uint64_t)(n - i)) % (uint64_t)(i + 1)) : -1;
    }
    if (t < 3)
        left[t] = 0u;
    grid.sync();
    for (unsigned long long round = 1; round <= (unsigned)n; ++round) {  // (a round does at least one swap)
        for (int i = t; i < n; i += T) {
            const int h = partner[i];
            if (h >= 0) {
                atomicMax(&place[i], round << 32 | (unsigned)i);
                atomicMax(&place[h], round << 32 | (unsigned)i);
            }
        }
        if (t == 0)
            left[(round + 1) % 3] = 0u;
        grid.sync();
        int mine = 0;
        for (int i = t; i < n; i += T) {
            const int h = partner[i];
            if (h < 0)
                continue;
            const unsigned long long own = round << 32 | (unsigned)i;
            if (__ldcg(&place[i]) == own && __ldcg(&place[h]) == own) {
                const int a = __ldcg(&perm[i]), b = __ldcg(&perm[h]);
                __stcg(&perm[i], b);
                __stcg(&perm[h], a);
                partner[i] = -1;
            } else {
                ++mine;
            }
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0 && mine)
            atomicAdd(&left[round % 3], (unsigned)mine);
        grid.sync();
        if (__ldcg(&left[round % 3]) == 0u)
            return;
    }
}

}  // namespace

cudaError_t launch_permutation(int n, uint64_t state, int *perm, int *partner, unsigned long long *place,
                               unsigned *left, int max_ctas, cudaStream_t st)
{
    // one CTA an SM (fewer arrivals at the barriers), no more than there are rows for
    int ctas = (n + kPermThreads - 1) / kPermThreads;
    ctas = ctas < max_ctas ? ctas : max_ctas;
    void *args[] = {&n, &state, &perm, &partner, &place, &left};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_permutation), dim3(ctas), dim3(kPermThreads),
                                       args, 0, st);
}

}  // namespace cgppd
