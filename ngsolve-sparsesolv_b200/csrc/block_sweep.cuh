// block_sweep.cuh -- colour-by-colour triangular sweeps of the ABMC-ordered IC
// factor.
//
// One launch per colour and run of ordinary blocks (a sub-warp per block, a lane
// per row), one launch per oversized block (the rows that the aggregation left
// over). A launch is a chain of dependent loads around very little work: 4 to 5
// us each when it walked row pointers, columns, values and gathered results in
// turn, whatever the colour held. So the layout takes the walk out of the chain:
//   - the entries of 32 rows lie side by side (sliced ELL, padded to the longest
//     row), with the rows' diagonal already multiplied in, y_i = r_i x_i - sum
//     a'_ij y_j, so that no division is left;
//   - a launch reads all that (rows, columns, coefficients) before it waits for
//     the launch before it (programmatic dependent launch), and only gathers,
//     sums and resolves the block's own couplings by shuffles after that;
//   - an oversized block is staged in shared memory the same way, and its level
//     sets are swept by one CTA with the next level's operands already in
//     registers at each barrier. Rows are padded to the longest one where that
//     fits, else to the width that takes the least, the rest of a row following
//     row by row; a block that does not fit at all keeps its CSR rows.
#pragma once

#include <vector>

#include "ssv_common.cuh"

namespace ssv {

struct KState;

template <typename S>
struct BlockSweep {
    using SL = typename ST<S>::lo;
    // kind 0: slices [a, b); kind 2: the oversized block of level offsets lev[a .. b],
    // staged in smem bytes (0: too large, swept from the CSR factor)
    struct Step {
        int kind, a, b;
        // first row of the list, rows, internal entries a row, entries past them, first of all these
        int smem = 0, qa = 0, nr = 0, width = 0, rest = 0, base = 0;
    };
    // one run of blocks or one oversized block, in processing order
    struct Run {
        int kind, a, b;  // 0: blocks [a, b); 2: level offsets [a, b] of the direction's list
    };
    struct Dir {
        std::vector<Step> steps;
        DevBuf<int> off, col, src, isrc;  // slices: first entry row and count; columns, sources
        DevBuf<S> v, iv;
        DevBuf<SL> v_lo, iv_lo;
        DevBuf<int> lev, rows;            // oversized blocks: level offsets, rows by level
        DevBuf<int> loc, lsrc, rrp, xrp, xcol, xsrc;  // rrp: a row's entries past the width, by row of the list
        DevBuf<S> lv, xv;
        DevBuf<SL> lv_lo, xv_lo;
    };
    int lanes = 0;
    bool lo = false;
    DevBuf<int> prow;  // position (slice * 32 + lane) -> row, -1 padding
    DevBuf<S> r;       // position -> 1 / L_ii
    Dir f, b;
    const int *Lrp = nullptr, *Lci = nullptr, *Urp = nullptr, *Uci = nullptr;  // the factor's CSR form
    const S *Lv = nullptr, *Uv = nullptr, *inv = nullptr;
    const SL *Lv_lo = nullptr, *Uv_lo = nullptr, *inv_lo = nullptr;

    // Layouts of the factor L (rows sorted, diagonal last) and U = L^T (diagonal
    // first; usrc = positions in L) over blocks boff, both directions' runs, and the
    // oversized blocks' rows by level.
    void build(int lanes, const std::vector<int>& boff, const std::vector<Run>& run_f, const std::vector<Run>& run_b,
               const std::vector<int>& rows_f, const std::vector<int>& lev_f, const std::vector<int>& rows_b,
               const std::vector<int>& lev_b, const std::vector<int>& lrp, const std::vector<int>& lci,
               const std::vector<int>& urp, const std::vector<int>& uci, const std::vector<int>& usrc, cudaStream_t s);
    // Values from the factor; lo_ stores the coefficients in the FP32 form.
    void fill(bool lo_, cudaStream_t s);
    void forward(const S* x, const double* sc, S* y, const KState* st, cudaStream_t s) const;
    void backward(const S* x, S* y, const KState* st, cudaStream_t s) const;
};

}  // namespace ssv
