// sweep_plan.cpp -- see sweep_plan.hpp.
#include "sweep_plan.hpp"

#include <algorithm>

namespace ssv {

// Cluster size from the mean level width: about one slice of a level per CTA. Measured
// per sweep with 2 / 4 / 8 / 16 CTAs: 22.1 / 22.1 / 22.1 / 21.9 us at a mean of 89 rows
// (46 levels), 38 / 31 / 31 / 31 us at 197 (70), 233 / 148 / 119 / 89 us at 479 (213,
// 8 entries a row), 276 / 166 / 115 / 79 us at 1090 (169). One CTA with a barrier per
// level in place of the pushes: 34 us at 89.
static int pick_ctas(int n, int nlev, int ctas_max) {
    const int mean = nlev > 0 ? n / nlev : 0;
    int c = 2;
    while (c < ctas_max && mean > 32 * c) c *= 2;
    return std::min(c, ctas_max);
}

// What a sweep takes, in us. A level takes what its busiest CTA takes for its rounds: so much
// a round, a slice, an entry and a target of the padded rows, and an entry of an earlier level
// in a chunk after the first (read one by one); changing to another chunk and starting the
// sweep come on top. Fitted to 150 real and 110 complex sweeps of 5 to 1400 us (grids of 12^3
// to 160^3 rows in natural, random and coloured order, edge matrices, scattered and layered
// patterns), which it meets to 7 and 14 % (standard deviation).
struct SweepCost {
    double round, slice, entry, target, far, chunk;
};
constexpr SweepCost kCostReal{0.264, 0.0, 0.005, 0.039, 0.033, 10.2};
constexpr SweepCost kCostComplex{0.384, 0.154, 0.016, 0.098, 0.063, 1.9};
constexpr double kCostStart = 3.9;  // 4.8 with the load of the inputs (forward), 3.0 without

// A launch takes 2.3 us on a few short rows. A thread walks its row alone (0.08 us an entry of
// the longest row), and rows that do not follow one another are read in pieces: longer by the
// entry and by the row, and by up to 1.7 us where the factor and the vectors no longer stay in
// L2. Within 13 % of 260 measured sweeps of 2 to 7000 us, which fails only where no cluster
// competes (coloured levels of 100,000 rows and more, twice the estimate).
double level_launches_us(int n, const int* rp, const std::vector<int>& rows, const std::vector<int>& off, int sbytes) {
    const double bytes = (double)rp[n] * (4 + sbytes) + (double)n * (8 + 3 * sbytes);
    const double miss = std::min(1.0, std::max(0.0, (bytes - 40e6) / 60e6));
    double us = 0.0;
    for (size_t l = 0; l + 1 < off.size(); ++l) {
        int longest = 0, pieces = 0;
        for (int q = off[l]; q < off[l + 1]; ++q) {
            longest = std::max(longest, rp[rows[q] + 1] - rp[rows[q]]);
            pieces += q == off[l] || rows[q] != rows[q - 1] + 1;
        }
        const int w = off[l + 1] - off[l];
        if (w <= 0) continue;
        const double apart = (double)pieces / w;
        us += 2.27 + (0.08 + 0.10 * apart) * longest * (sbytes > 8 ? 1.6 : 1.0) + apart * (36e-6 * w + 1.7 * miss);
    }
    return us;
}

double sweep_least_us(const std::vector<int>& off, int sbytes, int ctas) {
    const SweepCost& cost = sbytes > 8 ? kCostComplex : kCostReal;
    double us = kCostStart;
    for (size_t l = 0; l + 1 < off.size(); ++l) {
        const int sl = ((off[l + 1] - off[l] + 31) / 32 + ctas - 1) / ctas;
        us += cost.round * ((sl + kSweepWarps - 1) / kSweepWarps) + cost.slice * sl;
    }
    return us;
}

bool SweepPlanHost::build(int n_, const int* rp, const int* ci, bool fwd, const std::vector<int>& rows,
                          const std::vector<int>& off, int sbytes_, int smem, int stage, int ctas_max, double worth) {
    n = n_;
    nlev = (int)off.size() - 1;
    sbytes = sbytes_;
    if (n <= 0 || nlev <= 0 || ctas_max < 1) return false;
    ctas = pick_ctas(n, nlev, std::min(ctas_max, kSweepMaxCtas));
    const SweepCost& cost = sbytes > 8 ? kCostComplex : kCostReal;
    us = sweep_least_us(off, sbytes, ctas);
    if (us > worth) return false;
    // positions, owners, levels
    rowpos.clear();
    rowpos.reserve((size_t)n + (size_t)nlev * 16 + 64);
    pos.resize(n);
    lev.resize(n);
    cta.resize(n);
    std::vector<int> lev_pos(nlev + 1, 0);  // first position of each level
    int wmax = 0;
    for (int l = 0; l < nlev; ++l) {
        const int w = off[l + 1] - off[l], sl = (w + 31) / 32, parts = std::min(ctas, sl);
        wmax = std::max(wmax, sl);
        for (int p = 0; p < parts; ++p) {
            const int a = off[l] + sl * p / parts * 32, b = std::min(off[l] + sl * (p + 1) / parts * 32, off[l + 1]);
            for (int t = a; t < b; ++t) {
                const int i = rows[t];
                pos[i] = lev_pos[l] + (t - off[l]);
                lev[i] = l;
                cta[i] = (uint8_t)(p * ctas / parts);
                rowpos.push_back(i);
            }
        }
        rowpos.resize((size_t)lev_pos[l] + sl * 32, -1);
        lev_pos[l + 1] = (int)rowpos.size();
    }
    nslices = (int)rowpos.size() / 32;
    // entries by slice: late ones and all; owners with a dependent row, by row
    std::vector<int> late(nslices, 0), early(nslices, 0), ents(nslices, 0);
    std::vector<uint32_t> need(n, 0u);
    for (int i = 0; i < n; ++i) {
        const uint32_t bit = 1u << cta[i];
        int kl = 0, k = 0;
        for (int q = rp[i]; q < rp[i + 1]; ++q) {
            const int j = ci[q];
            if (!(fwd ? j < i : j > i)) continue;
            ++k;
            kl += lev[j] == lev[i] - 1;
            need[j] |= bit;
        }
        const int s = pos[i] / 32;
        late[s] = std::max(late[s], kl);
        early[s] = std::max(early[s], k - kl);
        ents[s] = std::max(ents[s], k);
    }
    // chunks: windows of what kSweepMinStages of the largest rounds leave
    int kmax = 0;
    for (int s = 0; s < nslices; ++s) kmax = std::max(kmax, std::max(ents[s], early[s] + late[s]));
    const int rsl = std::min(kSweepWarps, (wmax + ctas - 1) / ctas);
    const int round = std::min(stage, kSweepHeader + rsl * 32 * (row_bytes(kmax, std::min(ctas, 4), sbytes, sbytes) + sbytes));
    const int win = (smem - 128 - kSweepMinStages * round) / sbytes / 32 * 32;
    chunk_lev.assign(1, 0);
    std::vector<int> used(ctas, 1), add(ctas);
    slots = 1;
    for (int l = 0; l < nlev; ++l) {
        std::fill(add.begin(), add.end(), 0);
        for (int q = off[l]; q < off[l + 1]; ++q)
            for (uint32_t m = need[rows[q]]; m; m &= m - 1) ++add[__builtin_ctz(m)];
        bool fits = l - chunk_lev.back() < kSweepMaxLevels;
        for (int c = 0; c < ctas; ++c) {
            if (1 + add[c] > win) return false;
            fits = fits && used[c] + add[c] <= win;
        }
        if (!fits) {
            chunk_lev.push_back(l);
            std::fill(used.begin(), used.end(), 1);
        }
        for (int c = 0; c < ctas; ++c) slots = std::max(slots, used[c] += add[c]);
    }
    chunk_lev.push_back(nlev);
    nchunks = (int)chunk_lev.size() - 1;
    // the chunk of each level; owners with a dependent row inside the chunk
    std::vector<int> lev_chunk(nlev);
    for (int c = 0; c < nchunks; ++c)
        for (int l = chunk_lev[c]; l < chunk_lev[c + 1]; ++l) lev_chunk[l] = c;
    if (nchunks > 1) {
        std::fill(need.begin(), need.end(), 0u);
        for (int i = 0; i < n; ++i)
            for (int q = rp[i]; q < rp[i + 1]; ++q) {
                const int j = ci[q];
                if ((fwd ? j < i : j > i) && lev_chunk[lev[j]] == lev_chunk[lev[i]]) need[j] |= 1u << cta[i];
            }
    }
    std::vector<int> nt(nslices, 0);
    for (int i = 0; i < n; ++i) nt[pos[i] / 32] = std::max(nt[pos[i] / 32], __builtin_popcount(need[i]));
    // rounds: slices of one CTA and level, as many as the warps and a stage take
    std::vector<std::vector<SweepRound>> rc(ctas);
    slice_round.assign(nslices, 0);
    slice_chunk0.assign(nslices, 0);
    for (int l = 0; l < nlev; ++l) {
        const int c0 = lev_pos[chunk_lev[lev_chunk[l]]];
        const bool first = l == chunk_lev[lev_chunk[l]];
        for (int s = lev_pos[l] / 32; s < lev_pos[l + 1] / 32; ++s) {
            slice_chunk0[s] = c0;
            const int c = cta[rowpos[s * 32]];
            // in a chunk's first level all entries belong to earlier chunks
            const int ke = first ? ents[s] : early[s], kl = first ? 0 : late[s];
            SweepRound* r = rc[c].empty() ? nullptr : &rc[c].back();
            if (r && r->lev == l - chunk_lev[lev_chunk[l]] && r->chunk == lev_chunk[l] && r->nsl < kSweepWarps) {
                const int E = std::max(r->ke_kl & 0xffff, ke), L = std::max(r->ke_kl >> 16, kl), T = std::max(r->nt, nt[s]);
                if (kSweepHeader + (r->nsl + 1) * 32 * (row_bytes(E + L, T, sbytes, sbytes) + sbytes) <= stage) {
                    r->ke_kl = E | L << 16;
                    r->nt = T;
                    ++r->nsl;
                    slice_round[s] = (int)rc[c].size() - 1;
                    continue;
                }
            }
            if (ke + kl > 0x7fff || kSweepHeader + 32 * (row_bytes(ke + kl, nt[s], sbytes, sbytes) + sbytes) > stage)
                return false;
            SweepRound q{};
            q.pos0 = s * 32;
            q.nsl = 1;
            q.ke_kl = ke | kl << 16;
            q.nt = nt[s];
            q.lev = l - chunk_lev[lev_chunk[l]];
            q.chunk = lev_chunk[l];
            rc[c].push_back(q);
            slice_round[s] = (int)rc[c].size() - 1;
        }
    }
    // what these rounds take, level by level
    std::vector<double> level(nlev, 0.0), part(nlev);
    for (int c = 0; c < ctas; ++c) {
        std::fill(part.begin(), part.end(), 0.0);
        for (const SweepRound& r : rc[c]) {
            const int ke = r.ke_kl & 0xffff;
            part[chunk_lev[r.chunk] + r.lev] += cost.round + cost.slice * r.nsl + cost.entry * (ke + (r.ke_kl >> 16)) +
                                                cost.target * r.nt + cost.far * (r.chunk > 0 ? ke : 0);
        }
        for (int l = 0; l < nlev; ++l) level[l] = std::max(level[l], part[l]);
    }
    us = kCostStart + cost.chunk * (nchunks - 1);
    for (double l : level) us += l;
    if (us > worth) return false;
    // targets inside the chunk, and the bytes each level sends where
    tgt_ptr.assign(n + 1, 0);
    for (int i = 0; i < n; ++i) tgt_ptr[i + 1] = tgt_ptr[i] + __builtin_popcount(need[i]);
    tgt.resize(tgt_ptr[n]);
    tx.assign((size_t)nlev * ctas, 0u);
    for (int l = 0; l < nlev; ++l) {
        if (l == chunk_lev[lev_chunk[l]]) std::fill(used.begin(), used.end(), 1);
        for (int q = off[l]; q < off[l + 1]; ++q) {
            const int i = rows[q];
            int k = tgt_ptr[i];
            for (uint32_t m = need[i]; m; m &= m - 1) {
                const int c = __builtin_ctz(m);
                tgt[k++] = c << 24 | used[c]++;
                tx[(size_t)l * ctas + c] += (uint32_t)sbytes;
            }
        }
    }
    round_ptr.assign(ctas + 1, 0);
    rounds.clear();
    for (int c = 0; c < ctas; ++c) {
        rounds.insert(rounds.end(), rc[c].begin(), rc[c].end());
        round_ptr[c + 1] = (int)rounds.size();
    }
    for (int s = 0; s < nslices; ++s) slice_round[s] += round_ptr[cta[rowpos[s * 32]]];
    layout(sbytes);
    return slots * sbytes + 128 + kSweepMinStages * stage_bytes <= smem;
}

void SweepPlanHost::layout(int vbytes) {
    slice_off16.assign(nslices, 0);
    size_t at = 0;
    stage_bytes = 0;
    for (auto& r : rounds) {
        const int rec = 32 * row_bytes((r.ke_kl & 0xffff) + (r.ke_kl >> 16), r.nt, vbytes, sbytes);
        r.off16 = (uint32_t)(at / 16);
        r.bytes = kSweepHeader + r.nsl * rec;
        for (int u = 0; u < r.nsl; ++u) slice_off16[r.pos0 / 32 + u] = (int)((at + kSweepHeader + (size_t)u * rec) / 16);
        at += r.bytes;
        stage_bytes = std::max(stage_bytes, r.bytes + r.nsl * 32 * sbytes);
    }
    stream_bytes = at;
}

}  // namespace ssv
