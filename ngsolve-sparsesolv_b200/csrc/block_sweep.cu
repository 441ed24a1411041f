// block_sweep.cu -- see block_sweep.cuh.
#include "block_sweep.cuh"

#include "host_threads.hpp"
#include "objects.cuh"

namespace ssv {

// entries of a row read before the wait for the launch before
template <typename S>
constexpr int kBlkAhead = ST<S>::cplx ? 4 : 8;
constexpr int kBigThreads = 256;
constexpr int kBigWidth = 4;  // internal entries of an oversized block's row kept in registers

// One colour's run of blocks. iv holds, per slice, LANES - 1 rows of 32 couplings:
// forward, row t the coupling to the block's row t; backward, to its row t + 1.
template <typename S, typename SL, int LANES, bool FWD>
__global__ void __launch_bounds__(128)
k_blk_sweep(int s0, int s1, const int* __restrict__ prow, const int* __restrict__ off, const int* __restrict__ col,
            const SL* __restrict__ v, const SL* __restrict__ iv, const S* __restrict__ r, const S* __restrict__ x,
            const double* __restrict__ sc, S* y, const KState* st) {
    constexpr int A = kBlkAhead<S>;
    constexpr int NI = LANES <= 8 ? LANES - 1 : 0;  // couplings held in registers
    const int sl = s0 + blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, j = lane % LANES;
    const bool on = sl < s1;
    int row = -1, K = 0, c[A];
    SL vv[A], ii[NI > 0 ? NI : 1];
    const SL* vp = v;
    const int* cp = col;
    const SL* ip = iv;
    S rr = ST<S>::one();
    double ss = 1.0;
    if (on) {
        row = prow[sl * 32 + lane];
        const int o = off[2 * sl];
        K = off[2 * sl + 1];
        vp = v + (size_t)o * 32 + lane;
        cp = col + (size_t)o * 32 + lane;
        ip = iv + (size_t)sl * (LANES - 1) * 32 + lane;
        if (FWD) rr = r[sl * 32 + lane];
        if (FWD && sc && row >= 0) ss = sc[row];
#pragma unroll
        for (int t = 0; t < NI; ++t) ii[t] = ip[t * 32];
    }
#pragma unroll
    for (int u = 0; u < A; ++u) {
        c[u] = u < K ? cp[u * 32] : -1;
        if (u < K) vv[u] = vp[u * 32];
    }
    pdl_gate();
    if ((st && st->done) || !on) return;
    S s = ST<S>::zero(), g[A];
    if (row >= 0) {
        s = x[row];
        if (FWD) s = rr * (sc ? ST<S>::scale(ss, s) : s);
    }
#pragma unroll
    for (int u = 0; u < A; ++u)
        if (c[u] >= 0) g[u] = y[c[u]];
    S s2 = ST<S>::zero();
#pragma unroll
    for (int u = 0; u < A; u += 2) {  // two chains
        if (c[u] >= 0) s = s - hi_of_any(vv[u]) * g[u];
        if (c[u + 1] >= 0) s2 = s2 + hi_of_any(vv[u + 1]) * g[u + 1];
    }
    for (int k = A; k < K; ++k) {
        const int ck = cp[k * 32];
        if (ck >= 0) s = s - hi_of_any(vp[k * 32]) * y[ck];
    }
    s = s - s2;
#pragma unroll
    for (int q = 0; q + 1 < LANES; ++q) {
        const int t = FWD ? q : LANES - 1 - q;  // the row that is final now
        const S yt = shfl_s(s, t, LANES);
        const int e = FWD ? t : t - 1;
        SL w;
        if constexpr (NI > 0) w = ii[e];
        else w = ip[e * 32];
        if (FWD ? j > t : j < t) s = s - hi_of_any(w) * yt;
    }
    if (row >= 0) y[row] = s;
}

// An oversized block: its internal couplings (loc, lv: `width` columns of nr, padded with
// 0 * slot nr; REST: then `rest` entries past the width, those of row q from rrp[q]) and level
// offsets go to shared memory before the wait, the couplings to other blocks are folded into
// the right-hand side after it.
template <typename S, typename SL, bool FWD, bool REST>
__global__ void __launch_bounds__(kBigThreads)
k_big_sweep(int nlev, int nr, int width, int rest, const int* __restrict__ lev, const int* __restrict__ rows,
            const int* __restrict__ loc, const SL* __restrict__ lv, const int* __restrict__ rrp,
            const int* __restrict__ xrp, const int* __restrict__ xcol, const SL* __restrict__ xv,
            const S* __restrict__ inv, const S* __restrict__ x, const double* __restrict__ sc, S* y, const KState* st) {
    extern __shared__ __align__(16) unsigned char big_smem[];
    const int tid = threadIdx.x;
    const int qa = lev[0];
    S* ys = reinterpret_cast<S*>(big_smem);
    S* xs = ys + nr + 1;
    SL* sv = reinterpret_cast<SL*>(xs + nr + 1);
    const int pad = width * nr, all = pad + (REST ? rest : 0);
    int* sl = reinterpret_cast<int*>(sv + all + (all & 1));
    int* slev = sl + all;
    int* srp = slev + nlev + 1;
    for (int e = tid; e < all; e += kBigThreads) {
        sv[e] = lv[e];
        sl[e] = loc[e];
    }
    for (int l = tid; l <= nlev; l += kBigThreads) slev[l] = lev[l] - qa;
    if constexpr (REST)
        for (int q = tid; q <= nr; q += kBigThreads) srp[q] = pad + (q < nr ? rrp[qa + q] : rest);
    auto past_width = [&](S a, int q) {
        if constexpr (REST)
            for (int e = srp[q]; e < srp[q + 1]; ++e) a = a - hi_of_any(sv[e]) * ys[sl[e]];
        return a;
    };
    if (tid == 0) ys[nr] = ST<S>::zero();
    pdl_gate();
    if (st && st->done) return;
    for (int q = tid; q < nr; q += kBigThreads) {
        const int i = rows[qa + q];
        S s = x[i];
        if (FWD) s = inv[i] * (sc ? ST<S>::scale(sc[i], s) : s);
        const int e1 = xrp[qa + q + 1];
        for (int e = xrp[qa + q]; e < e1; ++e) s = s - hi_of_any(xv[e]) * y[xcol[e]];
        xs[q] = s;
    }
    __syncthreads();
    S s = ST<S>::zero();
    SL w[kBigWidth];
    int c[kBigWidth], q = 0;
    bool on = false;
    auto operands = [&](int l) {  // of this thread's row of level l
        q = slev[l] + tid;
        on = q < slev[l + 1];
        if (!on) return;
        s = xs[q];
#pragma unroll
        for (int u = 0; u < kBigWidth; ++u)
            if (u < width) {
                w[u] = sv[u * nr + q];
                c[u] = sl[u * nr + q];
            }
    };
    operands(0);
    for (int l = 0; l < nlev; ++l) {
        if (on) {
            S g[kBigWidth];
#pragma unroll
            for (int u = 0; u < kBigWidth; ++u)
                if (u < width) g[u] = ys[c[u]];
#pragma unroll
            for (int u = 0; u < kBigWidth; ++u)
                if (u < width) s = s - hi_of_any(w[u]) * g[u];
            for (int u = kBigWidth; u < width; ++u) s = s - hi_of_any(sv[u * nr + q]) * ys[sl[u * nr + q]];
            ys[q] = past_width(s, q);
        }
        for (int p = slev[l] + tid + kBigThreads; p < slev[l + 1]; p += kBigThreads) {
            S a = xs[p];
            for (int u = 0; u < width; ++u) a = a - hi_of_any(sv[u * nr + p]) * ys[sl[u * nr + p]];
            ys[p] = past_width(a, p);
        }
        if (l + 1 < nlev) operands(l + 1);
        __syncthreads();
    }
    for (int p = tid; p < nr; p += kBigThreads) y[rows[qa + p]] = ys[p];
}

template <typename S, typename SL>
static size_t big_bytes(int nr, int width, size_t rest, int nlev) {
    const size_t all = (size_t)width * nr + rest;
    return 2 * (size_t)(nr + 1) * sizeof(S) + (all + 1) * sizeof(SL) + all * 4 + (size_t)(nlev + 1) * 4 +
           (rest > 0 ? (size_t)(nr + 1) * 4 : 0) + 16;
}

// coefficients of the slices: forward L_ij / L_ii, backward L_ji * (1 / L_ii)
template <typename S, typename SO>
__global__ void k_blk_fill(int slices, int lanes, int fwd, const int* __restrict__ prow, const int* __restrict__ off,
                           const int* __restrict__ src, const int* __restrict__ isrc, const int* __restrict__ Lrp,
                           const S* __restrict__ Lv, const S* __restrict__ inv, SO* __restrict__ v,
                           SO* __restrict__ iv, S* __restrict__ r) {
    auto put = [](S x) {
        if constexpr (std::is_same<S, SO>::value) return x;
        else return lo_of(x);
    };
    const int lane = threadIdx.x & 31, nw = gridDim.x * blockDim.x / 32;
    for (int sl = (blockIdx.x * blockDim.x + threadIdx.x) / 32; sl < slices; sl += nw) {
        const int i = prow[sl * 32 + lane];
        S d = ST<S>::one(), w = ST<S>::one();
        if (i >= 0) {
            d = Lv[Lrp[i + 1] - 1];
            w = inv[i];
        }
        if (fwd) r[sl * 32 + lane] = w;
        auto scaled = [&](int k) {
            if (k < 0) return put(ST<S>::zero());
            return put(fwd ? ST<S>::div(Lv[k], d) : Lv[k] * w);
        };
        const size_t o = (size_t)off[2 * sl] * 32 + lane;
        for (int k = 0; k < off[2 * sl + 1]; ++k) v[o + k * 32] = scaled(src[o + k * 32]);
        for (int t = 0; t + 1 < lanes; ++t) {
            const size_t e = ((size_t)sl * (lanes - 1) + t) * 32 + lane;
            iv[e] = scaled(isrc[e]);
        }
    }
}

// coefficients of an oversized block's rows q of rows[qa ..]
template <typename S, typename SO>
__global__ void k_big_fill(int nr, int qa, int width, int rest, int fwd, const int* __restrict__ rows,
                           const int* __restrict__ lsrc, const int* __restrict__ rrp, const int* __restrict__ xrp,
                           const int* __restrict__ xsrc,
                           const int* __restrict__ Lrp, const S* __restrict__ Lv, const S* __restrict__ inv,
                           SO* __restrict__ lv, SO* __restrict__ xv) {
    auto put = [](S x) {
        if constexpr (std::is_same<S, SO>::value) return x;
        else return lo_of(x);
    };
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nr; q += gridDim.x * blockDim.x) {
        const int i = rows[qa + q];
        const S d = Lv[Lrp[i + 1] - 1], w = inv[i];
        auto scaled = [&](int k) {
            if (k < 0) return put(ST<S>::zero());
            return put(fwd ? ST<S>::div(Lv[k], d) : Lv[k] * w);
        };
        for (int u = 0; u < width; ++u) lv[u * nr + q] = scaled(lsrc[u * nr + q]);
        if (rest > 0)
            for (int e = rrp[qa + q]; e < (q + 1 < nr ? rrp[qa + q + 1] : rest); ++e)
                lv[width * nr + e] = scaled(lsrc[width * nr + e]);
        for (int e = xrp[qa + q]; e < xrp[qa + q + 1]; ++e) xv[e] = scaled(xsrc[e]);
    }
}

template <typename S>
void BlockSweep<S>::build(int lanes_, const std::vector<int>& boff, const std::vector<Run>& run_f,
                          const std::vector<Run>& run_b, const std::vector<int>& rows_f,
                          const std::vector<int>& lev_f, const std::vector<int>& rows_b,
                          const std::vector<int>& lev_b, const std::vector<int>& lrp, const std::vector<int>& lci,
                          const std::vector<int>& urp, const std::vector<int>& uci, const std::vector<int>& usrc,
                          cudaStream_t s) {
    lanes = lanes_;
    const int bps = 32 / lanes;  // blocks of a slice
    const int n = (int)lrp.size() - 1, nb = (int)boff.size() - 1;
    // positions: the runs' blocks in forward order, a run starting a slice
    std::vector<int> h_prow, first(nb, -1), blk;  // first slice of the run that starts at a block; slice slot -> block
    for (const Run& q : run_f) {
        if (q.kind != 0) continue;
        first[q.a] = (int)h_prow.size() / 32;
        for (int t = q.a; t < q.b; ++t) {
            blk.push_back(t);
            for (int j = 0; j < lanes; ++j) h_prow.push_back(boff[t] + j < boff[t + 1] ? boff[t] + j : -1);
        }
        while (h_prow.size() % 32) h_prow.push_back(-1);
        while ((int)blk.size() % bps) blk.push_back(-1);
    }
    const int slices = (int)h_prow.size() / 32;
    int smem_optin = 0;
    SSV_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0));
    struct Layout {
        std::vector<int> off, col, src, isrc, rrp, xrp, xcol, xsrc, loc, lsrc;
        int big_max = 0;
    } lay[2];
    auto direction = [&](bool fwd, Dir& D, Layout& h, const std::vector<Run>& runs, const std::vector<int>& rows,
                         const std::vector<int>& lv) {
        std::vector<int>&off = h.off, &col = h.col, &src = h.src, &isrc = h.isrc, &xrp = h.xrp, &xcol = h.xcol,
                        &xsrc = h.xsrc, &loc = h.loc, &lsrc = h.lsrc;
        const std::vector<int>& rp = fwd ? lrp : urp;
        const std::vector<int>& ci = fwd ? lci : uci;
        // a row's off-diagonal entries and their positions in L
        auto e0 = [&](int i) { return fwd ? rp[i] : rp[i] + 1; };
        auto e1 = [&](int i) { return fwd ? rp[i + 1] - 1 : rp[i + 1]; };
        auto from = [&](int k) { return fwd ? k : usrc[k]; };
        off.resize((size_t)slices * 2);
        isrc.assign((size_t)slices * (lanes - 1) * 32, -1);
        std::vector<int> cnt(32);
        col.reserve(rp[n]);
        src.reserve(rp[n]);
        for (int sl = 0; sl < slices; ++sl) {
            int K = 0;
            for (int t = 0; t < 32; ++t) {
                cnt[t] = 0;
                const int i = h_prow[sl * 32 + t];
                if (i < 0) continue;
                const int bk = blk[sl * bps + t / lanes], r0 = boff[bk], r1 = boff[bk + 1];
                for (int k = e0(i); k < e1(i); ++k) {
                    const int c = ci[k];
                    if (c < r0 || c >= r1) ++cnt[t];
                    else isrc[((size_t)sl * (lanes - 1) + (fwd ? c - r0 : c - r0 - 1)) * 32 + t] = from(k);
                }
                K = std::max(K, cnt[t]);
            }
            const size_t o = col.size();
            off[2 * sl] = (int)(o / 32);
            off[2 * sl + 1] = K;
            col.resize(o + (size_t)K * 32, -1);
            src.resize(o + (size_t)K * 32, -1);
            for (int t = 0; t < 32; ++t) {
                const int i = h_prow[sl * 32 + t];
                if (i < 0) continue;
                const int bk = blk[sl * bps + t / lanes], r0 = boff[bk], r1 = boff[bk + 1];
                int e = 0;
                for (int k = e0(i); k < e1(i); ++k)
                    if (ci[k] < r0 || ci[k] >= r1) {
                        col[o + (size_t)e * 32 + t] = ci[k];
                        src[o + (size_t)e * 32 + t] = from(k);
                        ++e;
                    }
            }
        }
        // oversized blocks
        xrp.assign(rows.size() + 1, 0);
        h.rrp.assign(rows.size(), 0);
        std::vector<int> at(n > 0 && !rows.empty() ? n : 0, -1);
        D.steps.clear();
        for (const Run& q : runs) {
            Step st{q.kind, q.a, q.b};
            if (q.kind == 0) {
                st.a = first[q.a];
                st.b = st.a + (q.b - q.a + bps - 1) / bps;
            } else {
                const int qa = lv[q.a], qb = lv[q.b], nr = qb - qa;
                for (int p = qa; p < qb; ++p) at[rows[p]] = p - qa;
                std::vector<int> has(nr, 0);  // internal entries of each row
                for (int p = qa; p < qb; ++p)
                    for (int k = e0(rows[p]); k < e1(rows[p]); ++k) has[p - qa] += at[ci[k]] >= 0;
                int width = nr > 0 ? *std::max_element(has.begin(), has.end()) : 0;
                size_t rest = 0;
                auto fits = [&] { return big_bytes<S, S>(nr, width, rest, q.b - q.a) + 1024 <= (size_t)smem_optin; };
                if (!fits()) {  // a few long rows: the width that takes the fewest entries in all
                    std::vector<int> by = has;
                    std::sort(by.begin(), by.end());
                    size_t past = 0, least = ~size_t(0);  // entries past the width by[t]
                    for (int t = nr - 1; t >= 0; --t) {
                        if (t + 1 < nr) past += (size_t)(nr - 1 - t) * (by[t + 1] - by[t]);
                        if ((size_t)by[t] * nr + past < least) {
                            least = (size_t)by[t] * nr + past;
                            width = by[t];
                            rest = past;
                        }
                    }
                }
                st.qa = qa;
                st.nr = nr;
                if (fits()) {
                    st.smem = (int)big_bytes<S, S>(nr, width, rest, q.b - q.a);
                    st.width = width;
                    st.rest = (int)rest;
                    st.base = (int)loc.size();
                    const size_t pad = st.base + (size_t)width * nr;
                    loc.resize(pad, nr);
                    lsrc.resize(pad, -1);
                }
                for (int p = qa; p < qb; ++p) {
                    int c = 0;
                    if (st.smem > 0) {
                        h.rrp[p] = (int)(loc.size() - st.base - (size_t)width * nr);
                        for (int k = e0(rows[p]); k < e1(rows[p]); ++k) {
                            const int a = at[ci[k]];
                            if (a < 0) {
                                xcol.push_back(ci[k]);
                                xsrc.push_back(from(k));
                            } else if (c < width) {
                                loc[st.base + (size_t)c * nr + p - qa] = a;
                                lsrc[st.base + (size_t)c * nr + p - qa] = from(k);
                                ++c;
                            } else {
                                loc.push_back(a);
                                lsrc.push_back(from(k));
                            }
                        }
                    }
                    xrp[p + 1] = (int)xcol.size();
                }
                for (int p = qa; p < qb; ++p) at[rows[p]] = -1;
                h.big_max = std::max(h.big_max, st.smem);
            }
            D.steps.push_back(st);
        }
    };
    run_threads(2, [&](int t) {  // the directions' layouts side by side
        if (t == 0) direction(true, f, lay[0], run_f, rows_f, lev_f);
        else direction(false, b, lay[1], run_b, rows_b, lev_b);
    });
    auto up = [&](DevBuf<int>& d, const std::vector<int>& h) {
        if (h.empty()) d.release();
        else d.upload(h.data(), h.size(), s);
    };
    for (int t = 0; t < 2; ++t) {
        Dir& D = t == 0 ? f : b;
        const Layout& h = lay[t];
        up(D.off, h.off); up(D.col, h.col); up(D.src, h.src); up(D.isrc, h.isrc);
        up(D.lev, t == 0 ? lev_f : lev_b); up(D.rows, t == 0 ? rows_f : rows_b);
        up(D.loc, h.loc); up(D.lsrc, h.lsrc); up(D.rrp, h.rrp); up(D.xrp, h.xrp); up(D.xcol, h.xcol); up(D.xsrc, h.xsrc);
    }
    const int big_max = std::max(lay[0].big_max, lay[1].big_max);
    if (h_prow.empty()) prow.release();
    else prow.upload(h_prow.data(), h_prow.size(), s);
    r.alloc(h_prow.size());
    SSV_CUDA(cudaStreamSynchronize(s));
    if (big_max > 0) {
        const auto kind = cudaFuncAttributeMaxDynamicSharedMemorySize;
        auto allow = [&](auto... k) { (SSV_CUDA(cudaFuncSetAttribute(k, kind, smem_optin - 1024)), ...); };
        allow(k_big_sweep<S, S, true, false>, k_big_sweep<S, S, false, false>, k_big_sweep<S, SL, true, false>,
              k_big_sweep<S, SL, false, false>, k_big_sweep<S, S, true, true>, k_big_sweep<S, S, false, true>,
              k_big_sweep<S, SL, true, true>, k_big_sweep<S, SL, false, true>);
    }
}

template <typename S>
void BlockSweep<S>::fill(bool lo_, cudaStream_t s) {
    lo = lo_;
    const int slices = (int)(prow.size() / 32);
    auto direction = [&](bool fwd, Dir& D) {
        auto values = [&](auto& v, auto& iv, auto& lv, auto& xv) {
            v.alloc(D.src.size());
            iv.alloc(D.isrc.size());
            lv.alloc(D.lsrc.size());
            xv.alloc(D.xsrc.size());
            if (slices > 0)
                k_blk_fill<S><<<grid_for((int64_t)slices * 32, 128, 16), 128, 0, s>>>(
                    slices, lanes, fwd, prow.get(), D.off.get(), D.src.get(), D.isrc.get(), Lrp, Lv, inv, v.get(),
                    iv.get(), r.get());
            for (const Step& q : D.steps)
                if (q.kind == 2 && q.smem > 0)
                    k_big_fill<S><<<grid_for(q.nr, 128), 128, 0, s>>>(
                        q.nr, q.qa, q.width, q.rest, fwd, D.rows.get(), D.lsrc.get() + q.base, D.rrp.get(), D.xrp.get(),
                        D.xsrc.get(), Lrp, Lv, inv, lv.get() + q.base, xv.get());
            SSV_LAUNCH_CHECK();
        };
        if (lo) values(D.v_lo, D.iv_lo, D.lv_lo, D.xv_lo);
        else values(D.v, D.iv, D.lv, D.xv);
    };
    direction(true, f);
    direction(false, b);
}

template <typename... KArgs, typename... Args>
static void launch_big(void (*k)(KArgs...), int smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(kBigThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    SSV_CUDA(cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...));
}

template <typename S, typename SL, bool FWD>
static void run_blocks(const BlockSweep<S>& w, const typename BlockSweep<S>::Dir& D, const SL* v, const SL* iv,
                       const SL* lv, const SL* xv, const SL* full, const SL* inv_full, const S* x, const double* sc,
                       S* y, const KState* st, cudaStream_t s) {
    for (const auto& q : D.steps) {
        if (q.kind == 0) {
            auto go = [&](auto l) {
                launch_k(k_blk_sweep<S, SL, decltype(l)::value, FWD>, (q.b - q.a + 3) / 4, 128, s, q.a, q.b,
                         w.prow.get(), D.off.get(), D.col.get(), v, iv, w.r.get(), x, sc, y, st);
            };
            switch (w.lanes) {
                case 1: go(std::integral_constant<int, 1>()); break;
                case 2: go(std::integral_constant<int, 2>()); break;
                case 4: go(std::integral_constant<int, 4>()); break;
                case 8: go(std::integral_constant<int, 8>()); break;
                case 16: go(std::integral_constant<int, 16>()); break;
                default: go(std::integral_constant<int, 32>()); break;
            }
        } else if (q.smem > 0) {
            launch_big(q.rest > 0 ? k_big_sweep<S, SL, FWD, true> : k_big_sweep<S, SL, FWD, false>, q.smem, s, q.b - q.a,
                       q.nr, q.width, q.rest, D.lev.get() + q.a, D.rows.get(), D.loc.get() + q.base, lv + q.base,
                       D.rrp.get(), D.xrp.get(), D.xcol.get(), xv, w.inv, x, sc, y, st);
        } else if (FWD) {
            launch_k(k_ic_fwd_cta<S, SL>, 1, 256, s, q.b - q.a, D.lev.get() + q.a, D.rows.get(), w.Lrp, w.Lci, full, x,
                     sc, y, st);
        } else {
            launch_k(k_ic_bwd_cta<S, SL>, 1, 256, s, q.b - q.a, D.lev.get() + q.a, D.rows.get(), w.Urp, w.Uci, full,
                     inv_full, x, y, st);
        }
    }
    SSV_LAUNCH_CHECK();
}

template <typename S>
void BlockSweep<S>::forward(const S* x, const double* sc, S* y, const KState* st, cudaStream_t s) const {
    if (lo)
        run_blocks<S, SL, true>(*this, f, f.v_lo.get(), f.iv_lo.get(), f.lv_lo.get(), f.xv_lo.get(), Lv_lo, inv_lo, x,
                                sc, y, st, s);
    else
        run_blocks<S, S, true>(*this, f, f.v.get(), f.iv.get(), f.lv.get(), f.xv.get(), Lv, inv, x, sc, y, st, s);
}

template <typename S>
void BlockSweep<S>::backward(const S* x, S* y, const KState* st, cudaStream_t s) const {
    if (lo)
        run_blocks<S, SL, false>(*this, b, b.v_lo.get(), b.iv_lo.get(), b.lv_lo.get(), b.xv_lo.get(), Uv_lo, inv_lo, x,
                                 nullptr, y, st, s);
    else
        run_blocks<S, S, false>(*this, b, b.v.get(), b.iv.get(), b.lv.get(), b.xv.get(), Uv, inv, x, nullptr, y, st, s);
}

template struct BlockSweep<double>;
template struct BlockSweep<zdouble>;

}  // namespace ssv
