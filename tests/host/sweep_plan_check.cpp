// Runs SweepPlanHost plans of random and grid patterns on the CPU the way the
// device kernel walks them: chunk by chunk, every CTA at its own pace, values
// of other CTAs only from what the masks send and the byte counts announce.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <set>

#include "host_order.hpp"
#include "sweep_plan.hpp"

using namespace ssv;

static int fails = 0;
#define CHECK(c, ...)                                     \
    do {                                                  \
        if (!(c)) {                                       \
            std::printf(__VA_ARGS__);                     \
            std::printf(" [%s:%d]\n", __FILE__, __LINE__); \
            ++fails;                                      \
            return;                                       \
        }                                                 \
    } while (0)

struct Csr {
    int n;
    std::vector<int> rp, ci;
};

static Csr random_csr(int n, int most, int reach, unsigned seed) {
    std::srand(seed);
    std::vector<std::set<int>> r(n);
    for (int i = 0; i < n; ++i) {
        r[i].insert(i);
        const int m = most > 0 ? std::rand() % (most + 1) : 0;
        for (int k = 0; k < m; ++k) {
            const int j = i - 1 - std::rand() % reach;
            if (j >= 0) {
                r[i].insert(j);
                r[j].insert(i);
            }
        }
    }
    Csr A;
    A.n = n;
    A.rp.push_back(0);
    for (auto& s : r) {
        A.ci.insert(A.ci.end(), s.begin(), s.end());
        A.rp.push_back((int)A.ci.size());
    }
    return A;
}

static Csr grid(int nx, int ny, int nz) {
    Csr A;
    A.n = nx * ny * nz;
    A.rp.push_back(0);
    for (int i = 0; i < A.n; ++i) {
        const int x = i % nx, y = i / nx % ny, z = i / (nx * ny);
        if (z) A.ci.push_back(i - nx * ny);
        if (y) A.ci.push_back(i - nx);
        if (x) A.ci.push_back(i - 1);
        A.ci.push_back(i);
        if (x + 1 < nx) A.ci.push_back(i + 1);
        if (y + 1 < ny) A.ci.push_back(i + nx);
        if (z + 1 < nz) A.ci.push_back(i + nx * ny);
        A.rp.push_back((int)A.ci.size());
    }
    return A;
}

// two levels of n rows, row n + i coupled to row i
static Csr pairs(int n) {
    Csr A;
    A.n = 2 * n;
    A.rp.push_back(0);
    for (int i = 0; i < A.n; ++i) {
        if (i >= n) A.ci.push_back(i - n);
        A.ci.push_back(i);
        if (i < n) A.ci.push_back(i + n);
        A.rp.push_back((int)A.ci.size());
    }
    return A;
}

static void run(const char* name, const Csr& A, bool fwd, int sbytes, int smem, int stage, int ctas_max, bool expect) {
    std::vector<int> lev, rows, off;
    const int nl = build_levels(A.n, A.rp.data(), A.ci.data(), !fwd, lev);
    group_by_level(lev, nl, rows, off);
    SweepPlanHost P;
    const bool ok = P.build(A.n, A.rp.data(), A.ci.data(), fwd, rows, off, sbytes, smem, stage, ctas_max);
    CHECK(ok == expect, "%s: build %d, expected %d", name, (int)ok, (int)expect);
    if (!ok) return;
    CHECK(P.ctas <= ctas_max, "%s: limits", name);
    for (int vb : {sbytes / 2, sbytes}) {
        P.layout(vb);
        CHECK(P.stage_bytes <= stage && P.slots * sbytes + kSweepMinStages * P.stage_bytes <= smem, "%s: shared memory", name);
        size_t at = 0;
        for (auto& r : P.rounds) {
            CHECK((size_t)r.off16 * 16 == at && r.bytes % 16 == 0 && r.pos0 % 32 == 0, "%s: stream", name);
            at += r.bytes;
        }
        CHECK(at == P.stream_bytes, "%s: stream length", name);
    }
    // positions
    std::vector<int> seen(A.n, 0);
    for (size_t p = 0; p < P.rowpos.size(); ++p)
        if (P.rowpos[p] >= 0) {
            ++seen[P.rowpos[p]];
            CHECK(P.pos[P.rowpos[p]] == (int)p, "%s: position", name);
        }
    for (int i = 0; i < A.n; ++i) CHECK(seen[i] == 1, "%s: row %d at %d positions", name, i, seen[i]);
    // every CTA's window, chunk by chunk; a CTA may run any distance ahead inside a chunk, so
    // a row may use a value of its chunk only if that value was sent to its CTA from an
    // earlier level, and the bytes of every level add up to what the CTA waits for
    std::vector<double> x(A.n), ref(A.n), out(A.n, NAN);
    for (int i = 0; i < A.n; ++i) x[i] = std::sin(0.7 * i + 1.0);
    auto coef = [&](int i, int j) { return 0.3 * std::cos(1.3 * i + 0.4 * j); };
    for (int q = 0; q < A.n; ++q) {
        const int i = fwd ? q : A.n - 1 - q;
        double s = x[i];
        for (int k = A.rp[i]; k < A.rp[i + 1]; ++k)
            if (fwd ? A.ci[k] < i : A.ci[k] > i) s -= coef(i, A.ci[k]) * ref[A.ci[k]];
        ref[i] = s / 2.0;
    }
    for (int c = 0; c < P.nchunks; ++c) {
        std::vector<std::vector<double>> window(P.ctas, std::vector<double>(P.slots, NAN));
        for (auto& w : window) w[0] = 0.0;
        std::vector<std::pair<int, double>> done;
        for (int l = P.chunk_lev[c]; l < P.chunk_lev[c + 1]; ++l) {
            struct Sent {
                int cta, slot;
                double v;
            };
            std::vector<Sent> sent;
            std::vector<uint32_t> got(P.ctas, 0u);
            for (int t = 0; t < P.ctas; ++t)
                for (int q = P.round_ptr[t]; q < P.round_ptr[t + 1]; ++q) {
                    const SweepRound& r = P.rounds[q];
                    if (r.chunk != c || r.lev != l - P.chunk_lev[c]) continue;
                    CHECK(r.nsl >= 1 && r.nsl <= kSweepWarps && r.lev < kSweepMaxLevels, "%s: round", name);
                    for (int p = r.pos0; p < r.pos0 + 32 * r.nsl; ++p) {
                        const int i = P.rowpos[p];
                        CHECK(P.slice_round[p / 32] == q, "%s: slice", name);
                        if (i < 0) continue;
                        CHECK(lev[i] == l && P.lev[i] == l && P.cta[i] == t, "%s: owner of row %d", name, i);
                        const int c0 = P.slice_chunk0[p / 32];
                        double s = x[i];
                        int ke = 0, kl = 0;
                        for (int k = A.rp[i]; k < A.rp[i + 1]; ++k) {
                            const int j = A.ci[k];
                            if (!(fwd ? j < i : j > i)) continue;
                            const bool here = P.pos[j] >= c0;
                            (here && P.lev[j] == l - 1 ? kl : ke) += 1;
                            double v = out[j];
                            if (here) {
                                const int sl = P.slot_of(j, t);
                                CHECK(sl > 0 && sl < P.slots, "%s: slot of row %d in CTA %d", name, j, t);
                                v = window[t][sl];
                            }
                            s -= coef(i, j) * v;
                        }
                        CHECK(ke <= (r.ke_kl & 0xffff) && kl <= r.ke_kl >> 16, "%s: entries", name);
                        CHECK(P.tgt_ptr[i + 1] - P.tgt_ptr[i] <= r.nt, "%s: targets", name);
                        done.push_back({i, s / 2.0});
                        for (int k = P.tgt_ptr[i]; k < P.tgt_ptr[i + 1]; ++k) {
                            sent.push_back({P.tgt[k] >> 24, P.tgt[k] & 0xffffff, s / 2.0});
                            got[P.tgt[k] >> 24] += sbytes;
                        }
                    }
                }
            for (auto& v : sent) {
                CHECK(std::isnan(window[v.cta][v.slot]), "%s: slot used twice", name);
                window[v.cta][v.slot] = v.v;
            }
            for (int t = 0; t < P.ctas; ++t)
                CHECK(got[t] == P.tx[(size_t)l * P.ctas + t], "%s: bytes of level %d", name, l);
            CHECK(l + 1 < P.chunk_lev[c + 1] || sent.empty(), "%s: a chunk's last level is sent", name);
        }
        for (auto& d : done) out[d.first] = d.second;
    }
    for (int i = 0; i < A.n; ++i) CHECK(out[i] == ref[i], "%s: row %d %g %g", name, i, out[i], ref[i]);
}

int main() {
    for (bool fwd : {true, false}) {
        for (int n : {1, 31, 32, 33, 257, 1000})
            for (int most : {0, 1, 7})
                for (int reach : {1, 9, 400})
                    for (int sb : {8, 16}) {
                        run("random", random_csr(n, most, reach, n + most), fwd, sb, 1 << 18, 1 << 16, 16, true);
                        run("random, small window", random_csr(n, most, reach, n), fwd, sb, 90000, 1 << 14, 16, true);
                    }
        run("wide rows", random_csr(300, 120, 300, 5), fwd, 8, 1 << 19, 1 << 17, 16, true);
        run("row past a round", random_csr(300, 120, 300, 5), fwd, 8, 1 << 19, 2048, 16, false);
        run("level past the window", pairs(40000), fwd, 8, 1 << 16, 8192, 2, false);
        run("level past two windows", pairs(40000), fwd, 8, 1 << 16, 8192, 16, true);
        run("grid", grid(16, 16, 16), fwd, 8, 224256, 40960, 16, true);
        run("grid, many chunks", grid(61, 23, 37), fwd, 16, 65536, 12288, 16, true);
        run("grid, 16 CTAs", grid(50, 50, 50), fwd, 8, 224256, 40960, 16, true);
        run("grid, 4 CTAs", grid(50, 50, 30), fwd, 8, 224256, 40960, 4, true);
        run("chain", random_csr(700, 3, 1, 9), fwd, 8, 224256, 40960, 16, true);
    }
    if (!fails) std::printf("ok\n");
    return fails ? 1 : 0;
}
