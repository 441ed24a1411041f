// sweep.cu -- see sweep.cuh.
#include "host_threads.hpp"
#include "objects.cuh"
#include "sweep.cuh"

#include <atomic>
#include <cstring>
#include <type_traits>

namespace ssv {

// shared memory of a sweeping CTA: at least kSweepMinStages rounds of at most
// kStageBytes each, the window of results the rest
constexpr int kSmemBytes = 220 * 1024;
constexpr int kStageBytes = 40 * 1024;
constexpr int kMaxStages = kSweepMaxStages;
constexpr int kComputeWarps = kSweepWarps * kSweepGroups;
constexpr int kSweepThreads = (kComputeWarps + 1) * 32;
// late entries and targets of a row that are in registers before its level is due
constexpr int kAhead = 4;
constexpr int kBarBytes = (2 * kMaxStages + kSweepMaxLevels + 2) * 8;
// tries of a wait before it gives up (a try suspends for up to 3.9 us: a second in all)
constexpr int kWaitTries = 1 << 18;
static std::atomic<bool> g_no_waits{false};
bool sweep_no_waits() { return g_no_waits; }
void set_sweep_wait(int tries) { g_no_waits = tries == 0; }

// rows from which on the plans of the two directions are made on two host threads (50 ns a row
// each, a thread some 30 us)
constexpr int kSideBySide = 2000;

struct SweepArgs {
    const unsigned char* stream;
    const SweepRound* rounds;
    const int* round_ptr;
    const int* chunk_lev;
    const uint32_t* tx;
    int nchunks, bars, ctas, win_bytes, stage_bytes, stages, no_waits;
    int* err;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(unsigned a, unsigned cta) {
    unsigned m;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(cta));
    return m;
}
__device__ __forceinline__ unsigned cta_in_cluster() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void bar_init(unsigned b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
// arrives on the barrier at the cluster address b; what the warp has written is visible to its waiters
__device__ __forceinline__ void bar_arrive_cluster(unsigned b) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(b) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory");
}
// Waits for the phase of the given parity; false after kWaitTries (a constant: a limit in a
// register costs the sweep 5 %). CLUSTER: what other CTAs wrote to global memory before they
// arrived is visible too.
template <bool CLUSTER = false>
__device__ __forceinline__ bool bar_try(unsigned b, unsigned parity) {
    unsigned ok;
    if constexpr (CLUSTER)
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(b), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(b), "r"(parity)
            : "memory");
    return ok != 0;
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool bar_wait(unsigned b, unsigned parity) {
    for (int t = 0; t < kWaitTries; ++t)
        if (bar_try<CLUSTER>(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push(unsigned a, double v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push(unsigned a, zdouble v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(a),
                 "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(bar)
                 : "memory");
}

template <typename S, typename SL>
__global__ void __launch_bounds__(kSweepThreads)
k_sweep(SweepArgs a, const S* __restrict__ xs, S* out, KState* st) {
    extern __shared__ __align__(128) unsigned char sweep_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    S* win = reinterpret_cast<S*>(sweep_smem);
    unsigned char* ring = sweep_smem + a.win_bytes;
    const unsigned full = smem_u32(ring + (size_t)a.stages * a.stage_bytes), empty = full + 8 * kMaxStages;
    const unsigned cbar = empty + 8 * kMaxStages;  // where the computing warps of all CTAs meet
    const unsigned lbar = cbar + 16;               // results of each level of the chunk
    const unsigned me = cta_in_cluster();
    const int r0 = a.round_ptr[me], nr = a.round_ptr[me + 1] - r0;
    if (threadIdx.x < kMaxStages) {
        bar_init(full + 8 * threadIdx.x, 1);
        bar_init(empty + 8 * threadIdx.x, kSweepWarps);
    }
    if (threadIdx.x == 0) {
        bar_init(cbar, kComputeWarps * a.ctas);
        win[0] = ST<S>::zero();
    }
    for (int l = threadIdx.x; l < a.bars; l += kSweepThreads) bar_init(lbar + 8 * l, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    // arms the level barriers of a chunk: one phase each, complete when the
    // bytes that this CTA waits for have arrived
    auto arm = [&](int chunk) {
        const int l0 = a.chunk_lev[chunk], nl = a.chunk_lev[chunk + 1] - l0;
        for (int l = lane; l < a.bars; l += 32)
            bar_expect(lbar + 8 * l, l < nl ? a.tx[(size_t)(l0 + l) * a.ctas + me] : 0u);
    };
    if (warp == 0) arm(0);
    cluster_arrive();
    cluster_wait();
    pdl_gate();
    // a finished solve: no round is issued or waited for (the whole cluster reads the same state)
    const bool idle = st && st->done;
    // A wait that gives up ends this warp's part; the others' waits on it then give up too.
    bool bad = a.no_waits != 0;
    if (warp == kComputeWarps) {  // producer: streams the rounds
        int issued = 0;
        int sg = 0;
        unsigned turn = 1;  // parity of the wait for a stage's previous use
        for (int q0 = 0; q0 < nr && !bad && !idle; q0 += 32) {
            uint4 d = make_uint4(0, 0, 0, 0);
            if (q0 + lane < nr) {
                const SweepRound& r = a.rounds[r0 + q0 + lane];
                d = make_uint4(r.off16, (unsigned)r.bytes, (unsigned)r.pos0, (unsigned)r.nsl);
            }
            for (int q = q0; q < min(q0 + 32, nr); ++q) {
                const unsigned off = __shfl_sync(0xffffffffu, d.x, q - q0), bytes = __shfl_sync(0xffffffffu, d.y, q - q0);
                const unsigned pos = __shfl_sync(0xffffffffu, d.z, q - q0), nsl = __shfl_sync(0xffffffffu, d.w, q - q0);
                if (q >= a.stages) bad = __any_sync(0xffffffffu, !bar_wait(empty + 8 * sg, turn));
                if (bad) break;
                if (lane == 0) {
                    const unsigned xb = nsl * 32 * (unsigned)sizeof(S);
                    const unsigned dst = smem_u32(ring) + sg * a.stage_bytes;
                    bar_expect(full + 8 * sg, bytes + xb);
                    bulk_load(dst, a.stream + (size_t)off * 16, bytes, full + 8 * sg);
                    bulk_load(dst + bytes, xs + pos, xb, full + 8 * sg);
                }
                __syncwarp();
                issued = q + 1;
                if (++sg == a.stages) {
                    sg = 0;
                    turn ^= 1;
                }
            }
        }
        // every copy has landed before the CTA ends
        for (int q = max(0, issued - a.stages); q < issued; ++q) bar_wait(full + 8 * (q % a.stages), (q / a.stages) & 1);
    } else {
        int chunk = 0, waited = 0;  // levels of the chunk whose values have arrived
        auto meet = [&] {  // the computing warps of all CTAs
            __syncwarp();
            if (lane < a.ctas) bar_arrive_cluster(peer_addr(cbar, lane));
            bad = __any_sync(0xffffffffu, bad || !bar_wait<true>(cbar, chunk & 1));
        };
        // The groups take the rounds in turn: while one finishes a level, the next ones have
        // their records and early entries behind them.
        const int grp = warp / kSweepWarps, wg = warp % kSweepWarps;
        int sg = grp % a.stages;
        unsigned turn = (grp / a.stages) & 1;
        for (int q = grp; q < nr && !idle; q += kSweepGroups) {
            bad = __any_sync(0xffffffffu, bad || !bar_wait(full + 8 * sg, turn));
            if (bad) break;
            const unsigned char* stage = ring + (size_t)sg * a.stage_bytes;
            const SweepRound h = *reinterpret_cast<const SweepRound*>(stage);
            // levels whose results have arrived (a wait that gave up is agreed on by the warp below)
            auto wait_levels = [&](int upto) {
                for (; waited < upto; ++waited) bad |= !bar_wait(lbar + 8 * waited, chunk & 1);
            };
            for (; chunk < h.chunk; ++chunk) {
                meet();
                if (bad) break;
                waited = 0;
                if (warp == 0) arm(chunk + 1);
            }
            if (bad) break;
            if (wg < h.nsl) {
                const int ke = h.ke_kl & 0xffff, kl = h.ke_kl >> 16;
                const unsigned char* rec =
                    stage + kSweepHeader + wg * 32 * SweepPlanHost::row_bytes(ke + kl, h.nt, sizeof(SL), sizeof(S));
                const SL* v = reinterpret_cast<const SL*>(rec + 32 * sizeof(S)) + lane;
                const int* c = reinterpret_cast<const int*>(v - lane + 32 * (ke + kl)) + lane;
                const int* op = c + 32 * (ke + kl);
                const int o = op[0];
                S s = reinterpret_cast<const S*>(rec)[lane] * reinterpret_cast<const S*>(stage + h.bytes)[wg * 32 + lane];
                constexpr int kEarly = ST<S>::cplx ? 4 : 8;
                SL vl[kAhead], ve[kEarly];
                int cl[kAhead], ce[kEarly];
                unsigned ta[kAhead], tb[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    cl[u] = u < kl ? c[(ke + u) * 32] : 0;
                    if (u < kl) vl[u] = v[(ke + u) * 32];
                }
#pragma unroll
                for (int u = 0; u < kEarly; ++u) {
                    ce[u] = u < ke ? c[u * 32] : 0;
                    if (u < ke) ve[u] = v[u * 32];
                }
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    ta[u] = 0;
                    if (u < h.nt) {
                        const int t = op[(1 + u) * 32];
                        if (t >= 0) {
                            ta[u] = peer_addr(smem_u32(win + (t & 0xffffff)), t >> 24);
                            tb[u] = peer_addr(lbar + 8 * h.lev, t >> 24);
                        }
                    }
                }
                wait_levels(h.lev - 1);
                if (h.chunk == 0) {
                    S w[kEarly], s2 = ST<S>::zero();
#pragma unroll
                    for (int u = 0; u < kEarly; ++u)
                        if (u < ke) w[u] = win[ce[u]];
#pragma unroll
                    for (int u = 0; u < kEarly; u += 2) {  // two chains
                        if (u < ke) s = s - hi_of_any(ve[u]) * w[u];
                        if (u + 1 < ke) s2 = s2 + hi_of_any(ve[u + 1]) * w[u + 1];
                    }
                    for (int k = kEarly; k < ke; ++k) s = s - hi_of_any(v[k * 32]) * win[c[k * 32]];
                    s = s - s2;
                } else {  // some columns may lie in earlier chunks
                    for (int k = 0; k < ke; ++k) {
                        const int ck = c[k * 32];
                        const S w = ck < 0 ? ld_cg(out + (-1 - ck)) : win[ck];
                        s = s - hi_of_any(v[k * 32]) * w;
                    }
                }
                wait_levels(h.lev);
                S g[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (u < kl) g[u] = win[cl[u]];
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (u < kl) s = s - hi_of_any(vl[u]) * g[u];
                for (int k = ke + kAhead; k < ke + kl; ++k) s = s - hi_of_any(v[k * 32]) * win[c[k * 32]];
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (u < h.nt && ta[u]) push(ta[u], s, tb[u]);
                for (int u = kAhead; u < h.nt; ++u) {
                    const int t = op[(1 + u) * 32];
                    if (t >= 0)
                        push(peer_addr(smem_u32(win + (t & 0xffffff)), t >> 24), s, peer_addr(lbar + 8 * h.lev, t >> 24));
                }
                if (o >= 0) out[o] = s;
            } else {
                wait_levels(h.lev);
            }
            __syncwarp();
            if (lane == 0) bar_arrive(empty + 8 * sg);
            for (sg += kSweepGroups; sg >= a.stages; sg -= a.stages) turn ^= 1;
        }
        bad = __any_sync(0xffffffffu, bad);
        for (; chunk < a.nchunks - 1 && !bad && !idle; ++chunk) {
            meet();
            if (warp == 0) arm(chunk + 1);
        }
    }
    cluster_arrive();  // no CTA ends while another may still write to it
    cluster_wait();
    if (bad) {
        // Every CTA has sent its last result; those on their way to a CTA that no longer waits
        // for them land before it ends.
        for (int t = 0; t < 16; ++t) __nanosleep(4096);
        if (st) {
            st->status = SSV_ERR_TIMEOUT;
            st->done = 1;
        } else {
            atomicExch(a.err, 1);
        }
    }
}

// Records of a slice (one warp each): input scale, scaled coefficients and window
// slots of the early and the late entries (padded with 0 * slot 0; an entry of an
// earlier chunk refers to its output index o as -1 - o), output index, targets.
struct SweepLists {
    const int *rowpos, *pos, *lev, *tgt_ptr, *tgt, *slice_round, *slice_chunk0, *slice_off16;
    const uint8_t* cta;
    const SweepRound* rounds;
};

template <typename S, typename SL>
__global__ void k_sweep_fill(int nslices, unsigned char* stream, SweepLists a, const int* __restrict__ omap,
                             const int* __restrict__ rp, const int* __restrict__ ci, const S* __restrict__ vals,
                             int op, int fwd, int dmode, const S* __restrict__ darr) {
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * blockDim.x / 32;
    auto put = [](S x) {
        if constexpr (std::is_same<S, SL>::value) return x;
        else return lo_of(x);
    };
    for (int sl = (blockIdx.x * blockDim.x + threadIdx.x) / 32; sl < nslices; sl += nw) {
        const SweepRound h = a.rounds[a.slice_round[sl]];
        const int ke = h.ke_kl & 0xffff, K = ke + (h.ke_kl >> 16), c0 = a.slice_chunk0[sl];
        unsigned char* rec = stream + (size_t)a.slice_off16[sl] * 16;
        S* r = reinterpret_cast<S*>(rec) + lane;
        SL* v = reinterpret_cast<SL*>(rec + 32 * sizeof(S)) + lane;
        int* c = reinterpret_cast<int*>(v - lane + 32 * K) + lane;
        int* o = c + 32 * K;
        const int i = a.rowpos[sl * 32 + lane];
        int e = 0, l = ke, t = 0;
        S scale = ST<S>::zero();
        if (i >= 0) {
            const int k0 = rp[i], k1 = rp[i + 1], me = a.cta[i], late = a.lev[i] - 1;
            const S d = dmode == SD_ARRAY ? darr[i] : dmode == SD_LAST ? vals[k1 - 1] : vals[k0];
            scale = op == SW_DIV ? ST<S>::div(ST<S>::one(), d) : op == SW_MUL ? d : ST<S>::one();
            for (int k = k0; k < k1; ++k) {
                const int j = ci[k];
                if (!(fwd ? j < i : j > i)) continue;
                const bool here = a.pos[j] >= c0;
                const int at = here && a.lev[j] == late ? l++ : e++;
                v[at * 32] = put(op == SW_DIV ? ST<S>::div(vals[k], d) : vals[k] * d);
                int code = -1 - (omap ? omap[j] : j);
                if (here)
                    for (int q = a.tgt_ptr[j]; q < a.tgt_ptr[j + 1]; ++q)
                        if (a.tgt[q] >> 24 == me) code = a.tgt[q] & 0xffffff;
                c[at * 32] = code;
            }
            for (int q = a.tgt_ptr[i]; q < a.tgt_ptr[i + 1]; ++q) o[(1 + t++) * 32] = a.tgt[q];
        }
        for (; e < ke; ++e) {
            v[e * 32] = put(ST<S>::zero());
            c[e * 32] = 0;
        }
        for (; l < K; ++l) {
            v[l * 32] = put(ST<S>::zero());
            c[l * 32] = 0;
        }
        *r = scale;
        o[0] = i < 0 ? -1 : omap ? omap[i] : i;
        for (; t < h.nt; ++t) o[(1 + t) * 32] = -1;
    }
}

__global__ void k_sweep_heads(int n, const SweepRound* __restrict__ rounds, unsigned char* stream) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) *reinterpret_cast<SweepRound*>(stream + (size_t)rounds[q].off16 * 16) = rounds[q];
}

template <typename S>
__global__ void __launch_bounds__(kBlock)
k_sweep_load(int np, const int* __restrict__ rowpos, const S* __restrict__ a, const S* __restrict__ b,
             const double* __restrict__ sc, S* __restrict__ xs, const KState* st) {
    pdl_gate();
    if (st && st->done) return;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
        const int i = rowpos[p];
        S v = ST<S>::zero();
        if (i >= 0) {
            v = a[i];
            if (sc) v = ST<S>::scale(sc[i], v);
            if (b) v = v - b[i];
        }
        xs[p] = v;
    }
}

// calls f with the kernel of the FP64 or the FP32 form
template <typename S, typename F>
static void sweep_kernel(bool lo, F&& f) {
    using SLo = typename ST<S>::lo;
    if (lo) f(k_sweep<S, SLo>);
    else f(k_sweep<S, S>);
}

template <typename S>
static void allow_clusters(bool lo) {
    sweep_kernel<S>(lo, [](auto k) {
        SSV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        SSV_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    });
}

// Most CTAs of a cluster that the device can place with all the shared memory they may take:
// 16 on a whole B200, fewer (or none: 0) on a partition of one. Asked once for each device.
template <typename S>
static int placeable_ctas() {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];  // ctas + 1
    int dev = 0;
    SSV_CUDA(cudaGetDevice(&dev));
    if (dev < kDevices && known[dev] > 0) return known[dev] - 1;
    int ctas = kSweepMaxCtas;
    for (bool lo : {false, true}) {
        allow_clusters<S>(lo);
        sweep_kernel<S>(lo, [&](auto k) {
            for (; ctas > 0; ctas /= 2) {
                cudaLaunchAttribute at[1];
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim.x = ctas;
                at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(ctas);
                cfg.blockDim = dim3(kSweepThreads);
                cfg.dynamicSmemBytes = kSmemBytes;
                cfg.attrs = at;
                cfg.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters > 0) break;
                cudaGetLastError();
            }
        });
    }
    if (dev < kDevices) known[dev] = ctas + 1;
    return ctas;
}

template <typename S>
bool Sweep<S>::plan_host(const SweepRows& q, int ctas_max) {
    const double worth = q.worth >= 0.0 ? q.worth : level_launches_us(q.n, q.rp.data(), q.rows, q.off, (int)sizeof(S));
    if (!plan.build(q.n, q.rp.data(), q.ci.data(), q.fwd, q.rows, q.off, (int)sizeof(S), kSmemBytes - kBarBytes, kStageBytes,
                    ctas_max, worth)) {
        plan = SweepPlanHost();
        return false;
    }
    // the lists side by side, as they lie on the device; only the kernels need them from here on
    places.clear();
    size_t at = 0;
    auto room = [&](size_t bytes) {
        places.push_back(at);
        at += (bytes + 255) / 256 * 256;
    };
    auto lists = [&](auto&& f) {
        f(plan.rowpos); f(plan.pos); f(plan.lev); f(plan.tgt_ptr); f(plan.tgt); f(plan.slice_round); f(plan.slice_chunk0);
        f(plan.round_ptr); f(plan.chunk_lev); f(plan.tx); f(plan.cta);
    };
    lists([&](auto& v) { room(v.size() * sizeof(v[0])); });
    packed.resize(at);
    size_t k = 0;
    lists([&](auto& v) {
        if (!v.empty()) std::memcpy(packed.data() + places[k], v.data(), v.size() * sizeof(v[0]));
        ++k;
    });
    room(plan.rounds.size() * sizeof(SweepRound));
    room(plan.slice_off16.size() * sizeof(int));
    room(plan.rowpos.size() * sizeof(S));
    room(plan.stream_bytes);  // (the FP32 form takes less)
    places.push_back(at);
    auto drop = [](auto& v) { std::remove_reference_t<decltype(v)>().swap(v); };
    drop(plan.rowpos); drop(plan.pos); drop(plan.lev); drop(plan.tgt_ptr); drop(plan.tgt); drop(plan.slice_round);
    drop(plan.slice_chunk0); drop(plan.tx); drop(plan.cta);
    return true;
}

template <typename S>
void build_sweeps(Sweep<S>& f, Sweep<S>& b, const SweepRows& qf, const SweepRows& qb, cudaStream_t s) {
    f.ready = b.ready = false;
    f.fwd = qf.fwd;
    b.fwd = qb.fwd;
    const int ctas = placeable_ctas<S>();
    bool ok[2] = {false, false};
    auto one = [&](int t) { ok[t] = t == 0 ? f.plan_host(qf, ctas) : b.plan_host(qb, ctas); };
    if (qf.n >= kSideBySide) {
        run_threads(2, one);
    } else {
        one(0);
        if (ok[0]) one(1);
    }
    if (!ok[0] || !ok[1]) {
        f.plan = b.plan = SweepPlanHost();
        std::vector<unsigned char>().swap(f.packed);
        std::vector<unsigned char>().swap(b.packed);
        return;
    }
    f.mem.alloc(f.places.back() + b.places.back());
    f.upload(f.mem.get(), s);
    b.upload(f.mem.get() + f.places.back(), s);
    SSV_CUDA(cudaStreamSynchronize(s));
    std::vector<unsigned char>().swap(f.packed);
    std::vector<unsigned char>().swap(b.packed);
    f.ready = b.ready = true;
}

template <typename S>
void Sweep<S>::upload(unsigned char* at, cudaStream_t s) {
    size_t k = 0;
    auto set = [&](auto& v) {
        v.p = reinterpret_cast<decltype(v.p)>(at + places[k++]);
    };
    set(rowpos); set(pos); set(lev); set(tgt_ptr); set(tgt); set(slice_round); set(slice_chunk0); set(round_ptr);
    set(chunk_lev); set(tx); set(cta); set(rounds); set(slice_off16); set(xs); set(stream);
    h2d_staged(at, packed.data(), packed.size(), s);
    SSV_CUDA(cudaMemsetAsync(xs.get(), 0, sizeof(S) * (size_t)positions(), s));
    stages = 0;  // laid out by the first fill()
}

template <typename S>
void Sweep<S>::fill(SweepOp op, const int* rp, const int* ci, const S* v, int dmode, const S* darr, const int* omap,
                    bool lo_, cudaStream_t s) {
    using SLo = typename ST<S>::lo;
    if (!stages || lo != lo_) {
        lo = lo_;
        stages = 0;
        plan.layout((int)(lo ? sizeof(SLo) : sizeof(S)));  // FP32 rounds are no larger than the planned ones
        auto put = [&](void* d, const void* h, size_t bytes) {
            SSV_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s));
        };
        put(rounds.get(), plan.rounds.data(), plan.rounds.size() * sizeof(SweepRound));
        put(slice_off16.get(), plan.slice_off16.data(), plan.slice_off16.size() * sizeof(int));
        const int wb = (plan.slots * (int)sizeof(S) + 127) / 128 * 128;
        const int st = plan.ring_stages(kSmemBytes - wb - kBarBytes);
        smem = wb + st * plan.stage_bytes + kBarBytes;
        allow_clusters<S>(lo);
        const int nq = (int)plan.rounds.size();
        k_sweep_heads<<<(nq + 255) / 256, 256, 0, s>>>(nq, rounds.get(), stream.get());
        SSV_LAUNCH_CHECK();
        SSV_CUDA(cudaStreamSynchronize(s));
        stages = st;
    }
    const int g = grid_for((int64_t)plan.nslices * 32, 128, 16);
    const SweepLists ls{rowpos.get(), pos.get(), lev.get(), tgt_ptr.get(), tgt.get(), slice_round.get(),
                        slice_chunk0.get(), slice_off16.get(), cta.get(), rounds.get()};
    if (lo)
        k_sweep_fill<S, SLo><<<g, 128, 0, s>>>(plan.nslices, stream.get(), ls, omap, rp, ci, v, op, fwd, dmode, darr);
    else
        k_sweep_fill<S, S><<<g, 128, 0, s>>>(plan.nslices, stream.get(), ls, omap, rp, ci, v, op, fwd, dmode, darr);
    SSV_LAUNCH_CHECK();
}

template <typename S>
void Sweep<S>::load(const S* a, const S* b, const double* sc, const KState* st, cudaStream_t s) const {
    launch_k(k_sweep_load<S>, grid_for(positions(), kBlock), kBlock, s, positions(), rowpos.get(), a, b, sc, xs.get(),
             st);
}

template <typename S>
void Sweep<S>::run(S* out, const KState* st, int* err, cudaStream_t s) const {
    int bars = 0;  // levels of the longest chunk
    for (int c = 0; c < plan.nchunks; ++c) bars = std::max(bars, plan.chunk_lev[c + 1] - plan.chunk_lev[c]);
    SweepArgs a{stream.get(), rounds.get(), round_ptr.get(), chunk_lev.get(), tx.get(), plan.nchunks, bars,
                plan.ctas, (plan.slots * (int)sizeof(S) + 127) / 128 * 128, plan.stage_bytes, stages, sweep_no_waits(), err};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.ctas);
    cfg.blockDim = dim3(kSweepThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int na = 0;
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = plan.ctas;
    at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1;
    ++na;
    if (pdl_enabled()) {
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = at;
    cfg.numAttrs = na;
    sweep_kernel<S>(lo, [&](auto k) {
        SSV_CUDA(cudaLaunchKernelEx(&cfg, k, a, (const S*)xs.get(), out, const_cast<KState*>(st)));
    });
}

void SweepFlag::init(cudaStream_t s) {
    if (!dev.get()) dev.alloc(1);
    dev.zero(s);
}

void SweepFlag::check(cudaStream_t s) const {
    int e = 0;
    SSV_CUDA(cudaMemcpyAsync(&e, dev.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    SSV_CUDA(cudaStreamSynchronize(s));
    if (!e) return;
    dev.zero(s);
    fail(SSV_ERR_TIMEOUT, "triangular sweep: a wait gave up");
}

template struct Sweep<double>;
template struct Sweep<zdouble>;
template void build_sweeps(Sweep<double>&, Sweep<double>&, const SweepRows&, const SweepRows&, cudaStream_t);
template void build_sweeps(Sweep<zdouble>&, Sweep<zdouble>&, const SweepRows&, const SweepRows&, cudaStream_t);

}  // namespace ssv
