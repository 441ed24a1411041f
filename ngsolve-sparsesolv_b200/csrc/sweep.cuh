// sweep.cuh -- level-scheduled triangular sweeps in one launch.
//
// A sweep y_i = f(x_i, sum over j before i of a_ij y_j) is a chain of level
// sets: 100 to 600 of them on nodal and edge-element matrices, a few hundred to
// a few thousand rows each. One launch per level costs 2.3 - 6 us a level, little
// of it by its width. Here one thread-block cluster (2 - 16 CTAs, by the mean
// level width and what the device can place) walks all levels, 0.4 us a level
// while it fills the cluster's rounds once (2048 real rows), in proportion
// beyond. Wide, few or scattered levels keep their launches (SweepPlanHost). In it:
//   - every CTA owns a part of each level; its rows' records (coefficients,
//     columns, diagonal, output index) are one contiguous stream, and a
//     producer warp moves it and the inputs, which lie in the same order, into
//     a ring of 4 or 8 shared-memory stages with bulk copies, ahead of the
//     chain; four groups of four warps take the rounds in turn, each with stages
//     of its own;
//   - a row's result goes to the shared-memory windows of exactly those CTAs
//     that need it, by st.async, which also counts the bytes into the level's
//     mbarrier there: no barrier over the cluster and no fence on the chain;
//   - where the windows cannot hold all results, the levels form chunks; between
//     chunks the cluster meets once, and couplings to earlier chunks are read
//     from the output in memory.
// A record holds the row's coefficients already scaled by its diagonal, so that
// y_i = scale_i x_i - sum a'_ij y_j has no division and no multiplication after
// the sum. Entries of levels before the last one ("early") are summed before the
// last level's results are waited for.
#pragma once

#include "ssv_common.cuh"
#include "sweep_plan.hpp"

namespace ssv {

struct KState;

// Whether every wait inside the sweeps gives up at once (ssv_set_sweep_wait).
bool sweep_no_waits();
void set_sweep_wait(int tries);

// What a sweep computes, with d the row's diagonal value of fill():
enum SweepOp : int {
    SW_DIV = 0,  // y = (x - sum) / d
    SW_MUL,      // y = (x - sum) * d
    SW_ICB,      // y = x - sum * d (also (x / d - sum) * d)
};

// where a row's d comes from
enum SweepDiag : int { SD_LAST = 0, SD_FIRST = 1, SD_ARRAY = 2 };

// What the sweeps of one object report that run outside a solve's state.
struct SweepFlag {
    DevBuf<int> dev;
    void init(cudaStream_t s);
    int* get() const { return dev.get(); }
    // Waits for the stream; takes the report back and raises SSV_ERR_TIMEOUT if there is one.
    void check(cudaStream_t s) const;
};

// One direction's rows: the triangular part of a CSR pattern (entries j < i, or j > i, of every
// row), the rows by level, and the time in us of the other way to sweep it (< 0: a launch per
// level).
struct SweepRows {
    int n;
    const std::vector<int>&rp, &ci;
    bool fwd;
    const std::vector<int>&rows, &off;
    double worth = -1.0;
};

template <typename S>
struct Sweep {
    SweepPlanHost plan;
    bool ready = false;
    bool fwd = true;
    int stages = 0, smem = 0;
    bool lo = false;
    // One allocation, the forward sweep's, holds the plans' lists, the rounds, the inputs by
    // position (xs) and the streams of both directions: 28 took 2 ms at 30,000 rows, one 0.5.
    DevBuf<unsigned char> mem;
    std::vector<size_t> places;  // byte offsets of the parts, their size at the end
    std::vector<unsigned char> packed;
    template <typename T>
    struct Part {
        T* p = nullptr;
        T* get() const { return p; }
    };
    Part<unsigned char> stream;
    Part<int> rowpos, pos, lev, tgt_ptr, tgt, slice_round, slice_chunk0, slice_off16, round_ptr, chunk_lev;
    Part<uint8_t> cta;
    Part<uint32_t> tx;
    Part<SweepRound> rounds;
    Part<S> xs;

    bool plan_host(const SweepRows& q, int ctas_max);
    void upload(unsigned char* at, cudaStream_t s);
    // Writes the records from the CSR values: d from the row's last or first
    // entry or from darr; omap = output index of every row (null = the row).
    // lo_ stores the coefficients in the FP32 form.
    void fill(SweepOp op, const int* rp, const int* ci, const S* v, int dmode, const S* darr, const int* omap,
              bool lo_, cudaStream_t s);
    // xs[position] = sc * a - b of its row (sc, b may be null)
    void load(const S* a, const S* b, const double* sc, const KState* st, cudaStream_t s) const;
    // Sweeps from xs into out (at the rows' output indices). A bounded wait that gives up
    // is reported in st, or in err where there is no state.
    void run(S* out, const KState* st, int* err, cudaStream_t s) const;
    int positions() const { return plan.nslices * 32; }
};

// Plans both sweeps of an object. They stay not ready where one does not fit or is estimated to
// take longer than the caller's other way.
template <typename S>
void build_sweeps(Sweep<S>& f, Sweep<S>& b, const SweepRows& qf, const SweepRows& qb, cudaStream_t s);

}  // namespace ssv
