// sweep_plan.hpp -- host side of the one-launch level-scheduled triangular
// sweeps (sweep.cuh): which CTA of the cluster owns which rows of a level, the
// rounds each CTA streams through, and where each result is needed.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ssv {

constexpr int kSweepWarps = 4;        // computing warps of a group: slices of 32 rows in a round
constexpr int kSweepGroups = 4;       // groups of a CTA, which take its rounds in turn
// Stages of a CTA's ring: at least one for each group's next round, or a group that waits for
// the others between chunks waits for ever; and a whole multiple of the groups, so that each
// stage belongs to one group. A warp then has waited for every phase of its stages' barriers.
// On a stage that another group used last, it could come while that group's copy is still under
// way, take the phase before it, which has the parity it waits for, for its own, and work on
// what lies there.
constexpr int kSweepMinStages = kSweepGroups;
constexpr int kSweepMaxStages = 2 * kSweepGroups;
constexpr int kSweepMaxLevels = 512;  // levels of a chunk (one mbarrier each)
constexpr int kSweepMaxCtas = 16;
constexpr int kSweepHeader = 32;      // bytes in front of a round's records

// What one CTA processes at a time: up to kSweepWarps slices of one level. Its
// records lie at byte off16 * 16 of the stream, its inputs at position pos0.
struct SweepRound {
    uint32_t off16;
    int32_t bytes;  // header + records
    int32_t pos0;
    int32_t nsl;    // slices
    int32_t ke_kl;  // entries a row is padded to: early | late << 16
    int32_t nt;     // targets a row is padded to
    int32_t lev;    // level within the chunk
    int32_t chunk;
};

// Positions order the rows by (level, row), each level padded to whole slices of
// 32 that are dealt to the CTAs in order, so that neighbouring rows stay together.
// Every CTA holds a window of the results that its own rows use; slot 0 stays
// zero. A chunk is a run of levels whose results fit all windows. A row's entry
// is late when its column lies in the level just before, else early (earlier
// chunks included).
struct SweepPlanHost {
    int n = 0, ctas = 1, nlev = 0, nchunks = 0, nslices = 0;
    int slots = 0;        // largest window, slot 0 included
    int stage_bytes = 0;  // largest round: records and inputs (layout())
    int sbytes = 8;       // bytes of a vector entry
    size_t stream_bytes = 0;
    std::vector<int> rowpos;         // position -> row, -1 padding
    std::vector<int> pos, lev;       // row -> position, level
    std::vector<uint8_t> cta;        // row -> owner
    std::vector<int> tgt_ptr;        // row -> its targets: cta << 24 | slot
    std::vector<int> tgt;
    std::vector<int> slice_round, slice_chunk0, slice_off16;  // round, first position of the chunk, record
    std::vector<SweepRound> rounds;
    std::vector<int> round_ptr;      // ctas + 1
    std::vector<int> chunk_lev;      // nchunks + 1: first level of each chunk
    std::vector<uint32_t> tx;        // level * ctas + cta: bytes the level sends to that CTA
    double us = 0.0;      // estimated time of the sweep

    // Plans the sweep over the entries j < i (fwd) or j > i of the CSR pattern,
    // rows grouped by level (rows, off). `smem` = bytes for the window and
    // kSweepMinStages rounds, `stage` = most bytes of a round, ctas_max = largest
    // cluster (0: none). False where a level does not fit the windows or a row a round, or where
    // the sweep is estimated to take more than `worth` us, the time of the other way: at
    // most 16 of the SMs work, so wide levels are better launched one by one.
    bool build(int n, const int* rp, const int* ci, bool fwd, const std::vector<int>& rows,
               const std::vector<int>& off, int sbytes, int smem, int stage, int ctas_max, double worth = 1e300);
    // Stream offsets for coefficients of vbytes each.
    void layout(int vbytes);
    // stages of a ring in that many bytes
    int ring_stages(int bytes) const {
        return std::min(kSweepMaxStages, bytes / stage_bytes / kSweepGroups * kSweepGroups);
    }
    // a row's record: input scale, K coefficients, K columns, output index, targets
    static constexpr int row_bytes(int K, int nt, int vbytes, int sbytes) {
        return sbytes + K * (vbytes + 4) + 4 + 4 * nt;
    }
    int slot_of(int row, int c) const {  // slot of a row's result in CTA c's window
        for (int k = tgt_ptr[row]; k < tgt_ptr[row + 1]; ++k)
            if (tgt[k] >> 24 == c) return tgt[k] & 0xffffff;
        return -1;
    }
};

// The least that a sweep over levels of these offsets can take on so many CTAs, in us, from their
// widths alone: wide levels need no plan to be refused.
double sweep_least_us(const std::vector<int>& off, int sbytes, int ctas = kSweepMaxCtas);
// Estimated time in us of the same sweep with a launch per level, a thread per row.
double level_launches_us(int n, const int* rp, const std::vector<int>& rows, const std::vector<int>& off, int sbytes);

}  // namespace ssv
