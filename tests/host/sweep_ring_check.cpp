// The ring of shared-memory stages of a sweeping CTA (csrc/sweep.cu), as a model: a producer
// fills the stages in the order of the rounds, its copies land when they land, groups take the
// rounds in turn, and a warp knows a stage's barrier by the parity of its phase only.
#include <cstdio>
#include <random>

#include "sweep_plan.hpp"

using namespace ssv;

// Whether every warp finds its own round in the stage that it passed the wait of.
static bool ring_is_sound(int stages, int rounds, unsigned seed) {
    std::mt19937 g(seed);
    struct Stage {
        int phase = 0;    // phases of the full barrier that are complete
        int round = -1;   // round whose copy is under way or has landed
        bool flying = false;
        int held = -1;    // round in the memory
        int left = 0;     // warps that still have to release it
    };
    std::vector<Stage> st(stages);
    constexpr int W = kSweepWarps * kSweepGroups;
    std::vector<int> at(W);  // each warp's round
    for (int w = 0; w < W; ++w) at[w] = w / kSweepWarps;
    int next = 0;
    for (long turn = 0; turn < 200L * rounds; ++turn) {
        const int what = g() % (W + 2);
        if (what == W) {  // the producer
            Stage& s = st[next % stages];
            if (next < rounds && !s.flying && s.left == 0) {
                s.round = next++;
                s.flying = true;
                s.left = kSweepWarps;
            }
        } else if (what == W + 1) {  // a copy lands: now and then, and any of them
            Stage& s = st[g() % stages];
            if (s.flying && g() % 8 == 0) {
                s.flying = false;
                s.held = s.round;
                ++s.phase;
            }
        } else if (at[what] < rounds) {
            Stage& s = st[at[what] % stages];
            const int parity = at[what] / stages & 1;
            if ((s.phase & 1) == parity) continue;  // the phase of that parity is not complete
            if (s.flying || s.held != at[what]) return false;
            --s.left;
            at[what] += kSweepGroups;
        }
    }
    return true;
}

int main() {
    int fails = 0;
    SweepPlanHost P;
    for (int stage : {96, 1024, 4128, 13344, 40960}) {
        P.stage_bytes = stage;
        for (int bytes = kSweepMinStages * stage; bytes < 11 * stage; bytes += stage / 3 + 1) {
            const int n = P.ring_stages(bytes);
            bool ok = n >= kSweepMinStages && n <= kSweepMaxStages && n * stage <= bytes && n % kSweepGroups == 0;
            for (unsigned seed = 0; ok && seed < 3; ++seed) ok = ring_is_sound(n, 200, seed);
            if (!ok) {
                std::printf("%d bytes, stages of %d: a ring of %d\n", bytes, stage, n);
                ++fails;
            }
        }
    }
    // the model finds what is wrong with the sizes between
    for (int n : {5, 6, 7}) {
        bool found = false;
        for (unsigned seed = 0; seed < 50 && !found; ++seed) found = !ring_is_sound(n, 200, seed);
        if (!found) {
            std::printf("a ring of %d passes\n", n);
            ++fails;
        }
    }
    if (!fails) std::printf("ok\n");
    return fails ? 1 : 0;
}
