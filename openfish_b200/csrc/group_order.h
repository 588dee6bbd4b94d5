// group_order.h -- the order in which a scan that runs ahead of its checks takes its groups of timesteps, and which
// group its checker is told to look at, without the means: plain C++, so that it can be tried without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define OF_HD __host__ __device__ __forceinline__
#else
#define OF_HD inline
#endif

constexpr uint32_t kAllAnew = 1u << 31;  // a verdict: too many guesses to check, the scan takes the whole group exactly

// The scan warps' side; a barrier that scan warps and checker pass together ends every group.  While the scan takes
// a group, the checker looks at the one that ended at the last barrier and puts its wrong guesses right; the
// verdict (bit q: a guess of timestep q was wrong) is looked at in the group after.
struct GroupOrder {
    int g = 0;       // the group under way
    int from = 0;    // its first timestep to be taken: behind a corrected one when the scan has gone back
    int ignore = 2;  // verdicts to come that are about nothing
    int par = 0;     // parity of the barriers passed

    OF_HD bool goes_back(uint32_t verdict) const { return ignore == 0 && verdict != 0; }
    // to the group before the last, behind its first wrong timestep or, with kAllAnew, to its start; no barrier is
    // passed for it
    OF_HD void go_back(uint32_t verdict) {
        g -= 2;
#ifdef __CUDA_ARCH__
        from = verdict & kAllAnew ? 0 : __ffs((int)verdict);
#else
        from = verdict & kAllAnew ? 0 : __builtin_ffs((int)verdict);
#endif
        ignore = 2;
    }
    // the verdict just looked at was about group g-2 and found it right: its input rows are final
    OF_HD bool verified() const { return ignore == 0; }
    // By one thread, when the scan takes up a group (or goes back to it), for the barrier that ends it.  The checker writes
    // into the rows of the group that it is told, so it must be one that is still to be verified, whenever it gets round to
    // reading which: a check that the scan goes back beside is of the group in between, all of whose rows are taken
    // again.  Hence a note for each parity, which stays as it is from its barrier to the next; a single count that the
    // scan changed on going back could send a late checker to a group whose rows were final and whose scores were
    // gone.
    OF_HD void tell(volatile int *ended) const { ended[par] = g; }
    OF_HD void next() {
        ++g;
        from = 0;
        ignore -= ignore > 0;
        par ^= 1;
    }
};

// The checker's side: the group that ended at barrier `at` (0, 1, 2 ...).
OF_HD int group_told(const volatile int *ended, int at) { return ended[at & 1]; }
