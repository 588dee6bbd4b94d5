// Host run of a scan that runs ahead of its checks (group_order.h) over made-up timesteps: a row is one number, the
// next one a hash of it and of the timestep's score, a guess now and then another number.  The checker gets round
// to its check anywhere between two barriers, and what is verified leaves, and has its scores replaced, as early or
// as late as it may.  Test code only.
#include <random>
#include <vector>

#include "../../openfish_b200/csrc/group_order.h"

static uint32_t next_row(uint32_t row, uint32_t score) {
    uint32_t x = row * 2654435761u ^ (score + 0x9e3779b9u) * 2246822519u;
    return x ^ x >> 15;
}

// Scans T timesteps in groups of E through a ring of S groups.  marked, wrong: percentages of timesteps whose value
// is a guess, and of guesses that are wrong; many: guesses that are too many for a check.  Returns how many of the T+1 rows left with a wrong value; *backs the times the
// scan has gone back, *late the checks that ran after the scan had gone back beside them; negative: -1 a row that
// has not left is written over, -2 a group checked that is not there.
extern "C" int wrong_rows(int T, int E, int S, int marked, int wrong, int many, unsigned seed, int *backs, int *late) {
    std::mt19937 rng(seed);
    auto percent = [&](int p) { return (int)(rng() % 100) < p; };
    const int groups = (T + E - 1) / E, H = E * (S + 1);
    auto score_of = [&](int t) { return (uint32_t)t * 40503u + seed; };
    std::vector<uint32_t> rows(H, 0), ring(S * E), out;
    std::vector<int> holds(S);  // the group whose scores a stage has
    int bad = 0;
    *backs = *late = 0;
    auto fill = [&](int g) {
        for (int q = 0; q < E; ++q) ring[g % S * E + q] = score_of(g * E + q);
        holds[g % S] = g;
    };
    for (int g = 0; g < S && g < groups; ++g) fill(g);

    GroupOrder at;
    int ended[2] = {0, 0};
    uint32_t mask[2] = {0, 0}, verdict[2] = {0, 0};
    int barrier = -1;          // the last one passed
    bool check_due = false, went_back = false, exactly = false;
    int verified = 0, left = 0;  // groups

    auto check = [&]() {
        check_due = false;
        const int g = group_told(ended, barrier);
        uint32_t m = g < groups ? mask[barrier & 1] : 0, v = 0;
        if (g < 0 || g > groups + 1) bad = -2;
        if (went_back && m) ++*late;
        int checked = 0;
        for (int q = 0; q < E; ++q) {
            if (!(m >> q & 1)) continue;
            if (++checked == many) {
                v = kAllAnew;
                break;
            }
            const int h = (g * E + q) % H;
            const uint32_t x = next_row(rows[h], ring[g % S * E + q]);
            if (x != rows[(h + 1) % H]) {
                rows[(h + 1) % H] = x;
                v |= 1u << q;
            }
        }
        verdict[barrier & 1] = v;
    };
    auto group_leaves = [&]() {
        for (int t = left * E; t < left * E + E && t < T; ++t) out.push_back(rows[t % H]);
        if (left + S < groups) fill(left + S);
        ++left;
    };
    auto meanwhile = [&]() {
        if (check_due && percent(15)) check();
        while (left < verified && percent(40)) group_leaves();
    };

    while (at.g <= groups + 1) {
        const uint32_t seen = verdict[at.par];
        at.tell(ended);
        const bool back = at.goes_back(seen);
        uint32_t guesses = 0;
        meanwhile();
        if (at.g < groups) {
            for (int q = 0; q < E; ++q) {
                if (q < at.from) continue;
                const int t = at.g * E + q;
                uint32_t x = next_row(rows[t % H], ring[at.g % S * E + q]);
                if (!exactly && percent(marked)) {
                    if (t < T) guesses |= 1u << q;
                    if (percent(wrong)) x ^= 1u;
                }
                if (q == 0 && back) break;
                if (t + 1 - H >= left * E && t + 1 - H >= 0) bad = -1;
                rows[(t + 1) % H] = x;
                meanwhile();
            }
        }
        if (back) {
            at.go_back(seen);
            exactly = seen & kAllAnew;
            went_back = true;
            ++*backs;
            meanwhile();
            continue;
        }
        if (at.verified() && verified < groups) ++verified;
        mask[at.par] = guesses;
        meanwhile();
        while (at.g + 1 < groups && holds[(at.g + 1) % S] != at.g + 1) {
            if (left == verified) return -3;  // nothing could ever bring those scores
            group_leaves();
        }
        if (check_due) check();
        ++barrier;
        check_due = true;
        went_back = false;
        exactly = false;
        at.next();
    }
    while (left < verified) group_leaves();
    out.push_back(rows[T % H]);
    if (bad) return bad;
    int n = 0;
    uint32_t row = 0;
    for (int t = 0; t <= T; ++t) {
        n += out.size() <= (size_t)t || out[t] != row;
        row = next_row(row, score_of(t));
    }
    return n;
}
