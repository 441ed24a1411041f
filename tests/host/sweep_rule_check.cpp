// Which of the two ways a level-scheduled sweep is planned to go: one launch for all levels
// (16 SMs at most) or a launch per level. The expectations are the measured outcomes: forward
// and backward time of both ways, in us, beside each pattern.
#include <algorithm>
#include <cstdio>
#include <random>

#include "host_order.hpp"
#include "sweep_plan.hpp"

using namespace ssv;

struct Csr {
    int n;
    std::vector<int> rp, ci;
};

// the 7-point grid of m^3 rows, row i numbered perm[i]
static Csr grid(int m, const std::vector<int>* perm = nullptr) {
    const int n = m * m * m;
    auto num = [&](int i) { return perm ? (*perm)[i] : i; };
    std::vector<std::vector<int>> row(n);
    for (int i = 0; i < n; ++i) {
        const int x = i % m, y = i / m % m, z = i / (m * m);
        auto& r = row[num(i)];
        r.push_back(num(i));
        if (z) r.push_back(num(i - m * m));
        if (y) r.push_back(num(i - m));
        if (x) r.push_back(num(i - 1));
        if (x + 1 < m) r.push_back(num(i + 1));
        if (y + 1 < m) r.push_back(num(i + m));
        if (z + 1 < m) r.push_back(num(i + m * m));
        std::sort(r.begin(), r.end());
    }
    Csr A{n, {0}, {}};
    for (auto& r : row) {
        A.ci.insert(A.ci.end(), r.begin(), r.end());
        A.rp.push_back((int)A.ci.size());
    }
    return A;
}

static std::vector<int> random_numbers(int n) {
    std::vector<int> p(n);
    for (int i = 0; i < n; ++i) p[i] = i;
    std::mt19937 g(1);
    std::shuffle(p.begin(), p.end(), g);
    return p;
}

// numbers by colour: 2 = red-black, 8 = by the parities of x, y and z
static std::vector<int> colour_numbers(int m, int colours) {
    std::vector<int> p(m * m * m), next(9, 0);
    auto colour = [&](int i) {
        const int x = i % m, y = i / m % m, z = i / (m * m);
        return colours == 2 ? (x + y + z) % 2 : x % 2 + 2 * (y % 2) + 4 * (z % 2);
    };
    for (int i = 0; i < (int)p.size(); ++i) ++next[colour(i) + 1];
    for (int c = 0; c < 8; ++c) next[c + 1] += next[c];
    for (int i = 0; i < (int)p.size(); ++i) p[i] = next[colour(i)]++;
    return p;
}

// L levels of w rows, each coupled to K neighbouring rows of the level before
static Csr layers(int w, int L, int K) {
    const int n = w * L;
    Csr A{n, {0}, {}};
    for (int i = 0; i < n; ++i) {
        std::vector<int> r{i};
        for (int k = 0; k < K; ++k) {
            const int p = ((i % w + k - K / 2) % w + w) % w, l = i / w;
            if (l > 0) r.push_back((l - 1) * w + p);
            const int q = ((i % w - k + K / 2) % w + w) % w;
            if (l + 1 < L) r.push_back((l + 1) * w + q);
        }
        std::sort(r.begin(), r.end());
        r.erase(std::unique(r.begin(), r.end()), r.end());
        A.ci.insert(A.ci.end(), r.begin(), r.end());
        A.rp.push_back((int)A.ci.size());
    }
    return A;
}

static int fails = 0;

static void expect(const char* name, const Csr& A, int sbytes, bool one_launch) {
    bool both = true;
    double us[2], launches[2];
    for (bool fwd : {true, false}) {
        std::vector<int> lev, rows, off, rp{0}, ci;
        for (int i = 0; i < A.n; ++i) {  // the triangle with its diagonal, as an IC factor stores it
            for (int k = A.rp[i]; k < A.rp[i + 1]; ++k)
                if (fwd ? A.ci[k] <= i : A.ci[k] >= i) ci.push_back(A.ci[k]);
            rp.push_back((int)ci.size());
        }
        const int nl = build_levels(A.n, rp.data(), ci.data(), !fwd, lev);
        group_by_level(lev, nl, rows, off);
        SweepPlanHost P;
        launches[fwd] = level_launches_us(A.n, rp.data(), rows, off, sbytes);
        both = P.build(A.n, rp.data(), ci.data(), fwd, rows, off, sbytes, 221000, 40960, 16, launches[fwd]) && both;
        us[fwd] = P.us;
    }
    if (both != one_launch) {
        std::printf("%s, %d bytes: one launch %d (%.1f %.1f us), a launch per level %.1f %.1f us\n", name, sbytes, (int)both,
                    us[1], us[0], launches[1], launches[0]);
        ++fails;
    }
}

int main() {
    const auto r41 = random_numbers(41 * 41 * 41), r64 = random_numbers(64 * 64 * 64);
    const auto rb30 = colour_numbers(30, 2), rb64 = colour_numbers(64, 2), c64 = colour_numbers(64, 8);
    expect("grid 16", grid(16), 8, true);                    // 22 / 20 against 128 / 128
    expect("grid 16", grid(16), 16, true);                   // 40 / 39 against 136 / 134
    expect("grid 64", grid(64), 8, true);                    // 108 / 102 against 603 / 607
    expect("grid 100", grid(100), 8, true);                  // 289 / 266 against 1195 / 1160
    expect("grid 100", grid(100), 16, true);                 // 763 / 765 against 1589 / 1564
    expect("random 41", grid(41, &r41), 8, true);            // 26 / 24 against 69 / 62
    expect("layers of 2048", layers(2048, 97, 3), 8, true);  // 44 / 40 against 254 / 254
    expect("layers of 8192", layers(8192, 24, 3), 8, true);  // 37 / 34 against 63 / 65
    expect("random 64", grid(64, &r64), 8, false);           // 123 / 119 against 76 / 71
    expect("random 64", grid(64, &r64), 16, false);          // (past the windows) against 84 / 90
    expect("red-black 30", grid(30, &rb30), 8, false);       // 9.2 / 7.3 against 5.5 / 5.2
    expect("red-black 30", grid(30, &rb30), 16, false);      // 20.7 / 18.7 against 5.9 / 6.0
    expect("red-black 64", grid(64, &rb64), 8, false);       // 46.9 / 44.7 against 6.8 / 7.2
    expect("8 colours 64", grid(64, &c64), 8, false);        // 55.3 / 51.8 against 11.6 / 11.7
    expect("layers of 8192", layers(8192, 24, 3), 16, false);    // 119 / 116 against 69 / 69
    expect("layers of 16384", layers(16384, 16, 3), 16, false);  // 137 / 137 against 45 / 46
    expect("4 layers of 60000", layers(60000, 4, 3), 8, false);  // 43 / 40 against 10.7 / 10.5
    expect("diagonal", layers(1000, 1, 0), 8, false);        // 4.8 / 2.9 against 2.0 / 2.0
    expect("diagonal", layers(60000, 1, 0), 8, false);       // 13.8 / 11.8 against 2.2 / 2.1
    // a device that places smaller clusters, or none
    for (int most : {0, 1, 2, 8}) {
        const Csr A = grid(20);
        std::vector<int> lev, rows, off;
        const int nl = build_levels(A.n, A.rp.data(), A.ci.data(), false, lev);
        group_by_level(lev, nl, rows, off);
        SweepPlanHost P;
        const bool ok = P.build(A.n, A.rp.data(), A.ci.data(), true, rows, off, 8, 221000, 40960, most);
        if (ok != (most > 0) || (ok && P.ctas > most)) {
            std::printf("clusters of %d at most: built %d with %d\n", most, (int)ok, P.ctas);
            ++fails;
        }
    }
    if (!fails) std::printf("ok\n");
    return fails ? 1 : 0;
}
