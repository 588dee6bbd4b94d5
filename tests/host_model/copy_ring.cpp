// Host run of the copy warp's order (copy_ring.h) over a made-up ring: barriers count phases, copies land when
// somebody waits for them, readers let go on demand.  Test code only.
#include <vector>

#include "../../openfish_b200/csrc/copy_ring.h"

// Runs `groups` groups through a ring of `ring` stages; the block gives up just before group `stop` is issued
// (or, with stop >= groups, after the last one).  Returns how many copies are still under way at the end, or a
// negative number for a mistake on the way: -1 a stage filled before its readers let go, -2 a wait for a phase
// that is not the stage's newest, -3 a group out of order or after the block has given up.
extern "C" int copies_left(int groups, int ring, int stop) {
    std::vector<int> filled(ring, 0), released(ring, 0);  // phases of `full` begun and of `empty` completed
    std::vector<char> under_way(ring, 0);
    int next = 0, bad = 0;
    fill_ring(
        groups, ring,
        [&](int stage, uint32_t parity) {
            // the readers of a stage need its copies to have landed before they can let go
            under_way[stage] = 0;
            if ((uint32_t)(released[stage] & 1) == parity) ++released[stage];
            else bad = -2;
        },
        [&]() { return next >= stop; },
        [&](int i, int stage) {
            if (i != next || stage != i % ring || next >= stop) bad = -3;
            if (under_way[stage] || released[stage] != filled[stage]) bad = bad ? bad : -1;
            ++next;
            ++filled[stage];
            under_way[stage] = 1;
        },
        [&](int stage, uint32_t parity) {
            if ((uint32_t)((filled[stage] - 1) & 1) != parity) bad = -2;
            under_way[stage] = 0;
        });
    if (bad) return bad;
    int left = 0;
    for (char c : under_way) left += c;
    return left;
}
