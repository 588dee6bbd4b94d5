// copy_ring.h -- the order in which a copy warp fills its ring of stages, without the means: plain C++, so that
// it can be tried without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define OF_HD __host__ __device__ __forceinline__
#else
#define OF_HD inline
#endif

// Copies `groups` groups in order, group i into stage i % ring:
//   released(stage, parity)  waits until the readers have let go of what the stage holds (its (i / ring)-th
//                            release, of phase parity `parity`), or the block has given up
//   given_up()               the block has given up: no more copies
//   issue(i, stage)          starts the copies of group i
//   landed(stage, parity)    waits, with a limit, until the stage's copies of that phase parity are there
// It returns only when the newest copies have landed (or `landed` has run out), whether or not the block has
// given up by then: a reader whose own wait runs out after the last group was issued ends the block, and a copy
// still under way would write into shared memory that has passed to another one.
template <class Released, class GivenUp, class Issue, class Landed>
OF_HD void fill_ring(int groups, int ring, Released released, GivenUp given_up, Issue issue, Landed landed) {
    int issued = 0, stage = 0;
    uint32_t parity = 1;  // (of the stage's previous release)
    for (; issued < groups; ++issued) {
        if (issued >= ring) released(stage, parity);
        if (given_up()) break;
        issue(issued, stage);
        if (++stage == ring) {
            stage = 0;
            parity ^= 1u;
        }
    }
    for (int i = issued > ring ? issued - ring : 0; i < issued; ++i) landed(i % ring, (uint32_t)(i / ring) & 1u);
}
