/*
 * Jacobi PageRank of a small graph in one cooperative launch.
 *
 * Replaces, for graphs below RESIDENT_MAX_EDGES, the queue of three kernels per
 * sweep of gcg_pagerank.cu (graphchi_engine::run() driving the PageRank update(),
 * src/engine/graphchi_engine.hpp:718-992, example_apps/pagerank.cpp:73-144). There
 * a sweep of a small graph is all latency: three launches that each drain before
 * the next may read, and a pass of its own over the rows that cross chunks.
 *
 * Here one 1024-thread CTA per SM keeps a contiguous range of the plan's 256-edge
 * chunks for the whole solve, cut so that edges plus rows are even, and applies
 * the rows that begin in it itself: gather and reduce its chunks, add up its rows
 * that cross chunks, apply its rows, and meet the other CTAs once per sweep, when
 * all new contributions are written. A row that runs on into the next CTAs' chunks
 * waits for those CTAs' edge phase by a flag per CTA, not for the grid. The
 * residual of a sweep is added up by one warp while the next sweep's gathers run;
 * a solve that has met its tolerance leaves before it writes anything more.
 * Initial vector and result assembly are in the same launch.
 *
 * Chunks, sums and their order are those of k_pr_edges / k_pr_fix / k_pr_vertex,
 * so the ranks are the same bits; only the FP64 residual is added in another
 * (fixed) order.
 *
 * What bounds it: at 1 M edges the chain of one sweep, 8.0 us (hub 1.2, gathers 2.4,
 * rows across chunks 1.2, apply 1.9, barrier 1.6 at ~1.9 GHz); from ~2 M edges the L1's
 * requests to L2 on gathers that miss the hub (2.4 M uniform edges: 11.5 of 18 us).
 *
 * Every wait is bounded: when one runs out the kernel sets an error flag, every
 * CTA leaves, and the call returns GCG_ERR_TIMEOUT.
 */
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "gcg_internal.cuh"
#include "gcg_pr_device.cuh"

namespace gcg {
namespace {

constexpr uint32_t WARPS = EDGE_THREADS / 32;
/* after the edge phase one warp of a CTA keeps its boundary with the other CTAs, the
 * others apply its rows */
constexpr uint32_t ROW_WARPS = WARPS - 1, ROW_THREADS = ROW_WARPS * 32;
constexpr int VB = 4; /* rows a thread applies at a time */
/* cost of applying a row, in edges, when the chunks are divided among the CTAs */
constexpr uint64_t ROW_COST = 3;
/* A source is staged in shared memory when that saves more than it costs: an entry
 * costs a CTA ~0.11 cycles a sweep (41,724 entries in 4,700 cycles), a gather that
 * misses the hub ~1 cycle, and a source of out-degree d is gathered d / CTAs times
 * per CTA */
constexpr uint32_t HUB_MIN_DEGREE = 16;
/* Vertices without in-edges to a CTA, where the chunks alone ask for fewer CTAs: the CTAs
 * walk them four times a solve, each step a chain of dependent loads. One to a thread: 4 M
 * vertices with 4,096 edges, 3 sweeps: 9.7 ms by the chunks' one CTA, 0.11 by 148; 65,536
 * with 4,096: 0.183, 0.053 (0.056 with 2,048 to a CTA, 0.059 with 4,096). */
constexpr uint32_t ZERO_ROWS = EDGE_THREADS;
/* polls of a wait: each takes at least an L2 round trip (~0.6 us), so seconds */
constexpr long long RES_SPIN = 1ll << 23;

struct ResArgs {
    SweepArgs a;
    float *c[2], *rnz[2];
    const ResRange *rg;
    uint32_t *bar;  /* arrivals at the grid barrier, counted up over the solve */
    uint32_t *flag; /* per CTA: sweeps whose edge phase is complete */
    int *err;
    double2 *bres;  /* [2][CTAs]: residual sums of a sweep, by its parity */
    float init;
    const float *init_rank;
    float *out;       /* result by vertex id, or null */
    ResStatus *status; /* pinned host memory */
    long long spin_limit; /* polls of a wait */
    uint32_t max_sweeps;
};

__device__ __forceinline__ uint64_t res_cost(const uint32_t *chunk_nz, uint32_t nchunks, uint32_t nnz, uint32_t c) {
    return (uint64_t)c * CH + ROW_COST * (c < nchunks ? chunk_nz[c] : nnz);
}

/* the range of each CTA: thread k of one block takes CTA k */
__global__ void k_res_ranges(const uint32_t *__restrict__ chunk_nz, const uint16_t *__restrict__ meta,
                             const uint4 *__restrict__ split, uint32_t nchunks, uint32_t nnz, uint32_t nsplit,
                             uint32_t ncta, const uint32_t *__restrict__ od_nz,
                             const uint32_t *__restrict__ nz_cidx, ResRange *__restrict__ out,
                             uint32_t *__restrict__ hub) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == ncta) { /* sources with at least HUB_MIN_DEGREE out-edges: the first ids */
        uint32_t lo = 0, hi = nnz;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (od_nz[mid] >= HUB_MIN_DEGREE) lo = mid + 1; else hi = mid;
        }
        *hub = lo < nnz ? nz_cidx[lo] : HUB_MAX;
    }
    if (k >= ncta) return;
    const uint64_t total = res_cost(chunk_nz, nchunks, nnz, nchunks);
    auto target = [&](uint32_t b) { return total * b / ncta; };
    auto bound = [&](uint32_t b) { /* first chunk whose cost prefix reaches b's share */
        const uint64_t t = target(b);
        uint32_t lo = 0, hi = nchunks;
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (res_cost(chunk_nz, nchunks, nnz, mid) < t) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    auto first_row = [&](uint32_t c) { /* first row that begins at or after chunk c */
        if (c >= nchunks) return nnz;
        return chunk_nz[c] + ((meta[meta_slot(c, 0)] & 1u) ? 0u : 1u);
    };
    auto first_split = [&](uint32_t row) {
        uint32_t lo = 0, hi = nsplit;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (split[mid].x < row) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    ResRange r;
    r.c0 = bound(k);
    r.c1 = bound(k + 1);
    r.r0 = first_row(r.c0);
    r.r1 = first_row(r.c1);
    r.s0 = first_split(r.r0);
    r.s1 = first_split(r.r1);
    r.cross = 0;
    r.blast = k;
    if (r.s1 > r.s0) {
        const uint32_t ce = split[r.s1 - 1].z;
        if (ce >= r.c1) { /* the last CTA whose range begins at or before chunk ce */
            r.cross = 1;
            const uint64_t cost = res_cost(chunk_nz, nchunks, nnz, ce);
            uint32_t b = k;
            while (b + 1 < ncta && target(b + 1) <= cost) ++b;
            r.blast = b;
        }
    }
    out[k] = r;
}

__device__ __forceinline__ uint32_t ld_acq(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
/* A contribution that other CTAs wrote before the last grid barrier: an ordinary
 * load, never the non-coherent path */
__device__ __forceinline__ float ld_contrib(const float *p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

/* waits (bounded) until *p reaches target; false when the limit ran out here or in
 * another CTA */
__device__ __forceinline__ bool wait_reach(const ResArgs &m, const uint32_t *p, uint32_t target) {
    for (long long spins = 0; (int32_t)(ld_acq(p) - target) < 0; ++spins) {
        if ((spins & 255) == 255 && *(volatile int *)m.err) return false;
        if (spins > m.spin_limit) {
            atomicExch(m.err, 1);
            m.status->err = 1;
            __threadfence_system();
            return false;
        }
    }
    return true;
}

/* grid barrier: every CTA arrives once per use, target = CTAs x uses */
__device__ bool res_sync(const ResArgs &m, uint32_t target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(m.bar, 1u);
        s_ok = wait_reach(m, m.bar, target);
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ float init_value(const ResArgs &m, uint32_t v) {
    if (m.init_rank) return m.init_rank[v];
    return m.a.source == GCG_NO_SOURCE ? m.init : (v == m.a.source ? 1.0f : 0.0f);
}

__global__ void __launch_bounds__(EDGE_THREADS, 1) k_pr_resident(ResArgs m) {
    extern __shared__ __align__(16) float s_hub[];
    __shared__ double2 s_red[WARPS];
    __shared__ int s_stop;
    __shared__ double s_res;
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t gtid = blockIdx.x * EDGE_THREADS + tid, gthreads = gridDim.x * EDGE_THREADS;
    const uint64_t pol_stream = policy_evict_first();
    const ResRange rg = m.rg[blockIdx.x];
    SweepArgs a = m.a;
    const bool pers = a.source != GCG_NO_SOURCE;

    /* initial state of this CTA's rows and of its share of the constant vertices */
    for (uint32_t i = rg.r0 + tid; i < rg.r1; i += EDGE_THREADS) {
        const float x = init_value(m, (m.init_rank || pers) ? a.nz_rows[i] : 0u);
        const uint32_t od = a.od_nz[i];
        m.rnz[0][i] = x;
        m.c[0][a.nz_cidx[i]] = od ? __fdiv_rn(x, (float)od) : 0.0f;
    }
    for (uint32_t i = gtid; i < a.nzero; i += gthreads) {
        const uint32_t v = a.zero_rows[i], od = a.outdeg[v];
        m.c[0][a.zero_cidx[i]] = od ? __fdiv_rn(init_value(m, v), (float)od) : 0.0f;
    }
    if (tid == 0) s_stop = 0;

    /* the first chunk's columns do not change: they are loaded ahead of each barrier */
    uint32_t col[EPL], meta = 0, base = 0;
    const uint32_t first = rg.c0 + warp;
    if (first < rg.c1) load_chunk(a, first, lane, pol_stream, col, meta, base);
    uint32_t meets = gridDim.x;
    if (!res_sync(m, meets)) return;

    /* one warp adds the CTAs' sums of sweep s in a fixed order and decides */
    auto residual = [&](uint32_t s) {
        double d = 0.0, n = 0.0;
        for (uint32_t k = lane; k < gridDim.x; k += 32u) {
            const double2 p = __ldcg(m.bres + (size_t)(s & 1u) * gridDim.x + k);
            d += p.x;
            n += p.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d += __shfl_xor_sync(FULL, d, o);
            n += __shfl_xor_sync(FULL, n, o);
        }
        if (lane == 0) {
            if (s >= 2) n += a.norm_const;
            const double res = n > 0.0 ? d / n : 0.0;
            s_res = res;
            if (a.tol > 0.0 && res <= a.tol) s_stop = 1;
            if (blockIdx.x == 0) {
                a.res_log[s] = res;
                if (a.delta_log) a.delta_log[s] = d;
            }
        }
    };

    uint32_t sweep = 0;
    for (;;) {
        const float *c_old = m.c[sweep & 1];
        float *c_new = m.c[(sweep + 1) & 1];
        const float *r_old = m.rnz[sweep & 1];
        float *r_new = m.rnz[(sweep + 1) & 1];

        /* ---- this CTA's chunks ---- */
        const uint32_t hub4 = a.hub >> 2;
        for (uint32_t i = tid; i < hub4; i += EDGE_THREADS) cp_async16(s_hub + 4 * i, c_old + 4 * i);
        for (uint32_t i = 4 * hub4 + tid; i < a.hub; i += EDGE_THREADS) s_hub[i] = __ldcg(c_old + i);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (sweep && warp == WARPS - 1) residual(sweep - 1); /* the warp with the fewest chunks */
        for (uint32_t ch = first; ch < rg.c1;) {
            float val[EPL];
#pragma unroll
            for (int j = 0; j < EPL; ++j) {
                const uint32_t x = col[j];
                val[j] = x < a.hub ? s_hub[x] : ld_contrib(c_old + x);
            }
            const uint32_t cur = ch, cm = meta, cb = base;
            ch += WARPS;
            if (ch < rg.c1) load_chunk(a, ch, lane, pol_stream, col, meta, base);
            reduce_chunk(a, cur, lane, val, cm, cb, a.ne);
        }
        /* rows and split rows that need nothing of other CTAs, and the one that does; a
         * thread's first split row is on its way during the wait */
        const uint32_t r1 = rg.r1 - rg.cross, s1 = rg.s1 - rg.cross;
        const uint32_t k00 = warp < ROW_WARPS ? rg.s0 + lane * ROW_WARPS + warp : s1;
        const uint4 sp0 = k00 < (warp < ROW_WARPS ? s1 : rg.s1) ? a.split[k00] : make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        if (s_stop) break;
        double d = 0.0, n = 0.0;
        auto apply = [&](uint32_t i, float sum, float old, uint32_t deg, uint32_t at) {
            const double tele = (!pers || a.nz_rows[i] == a.source) ? a.teleport : 0.0;
            const float rn = (float)__dadd_rn(tele, __dmul_rn(a.damping, (double)sum));
            r_new[i] = rn;
            c_new[at] = deg ? __fdiv_rn(rn, (float)deg) : 0.0f;
            d += fabs((double)rn - (double)old);
            n += fabs((double)rn);
        };
        if (warp == WARPS - 1) {
            /* ---- the boundary warp: the CTA's partials are published for the rows of
             *      earlier CTAs, then the row that runs on into later CTAs' chunks ---- */
            if (lane == 0) {
                __threadfence();
                atomicExch(m.flag + blockIdx.x, sweep + 1);
            }
            if (rg.cross) {
                const uint4 last = sp0;
                const float old = r_old[last.x];
                const uint32_t deg = a.od_nz[last.x], at = a.nz_cidx[last.x];
                for (uint32_t b = blockIdx.x + 1 + lane; b <= rg.blast; b += 32u)
                    if (!wait_reach(m, m.flag + b, sweep + 1)) break; /* the barrier below then ends the solve */
                __threadfence();
                __syncwarp();
                float sum;
                if (last.z - last.y > LONG_SPAN) {
                    const float t = long_row_sum_warp<true>(a.head_part, last.y, last.z, lane);
                    sum = __ldcg(a.tail_part + last.y) + t;
                } else {
                    sum = short_row_sum<true>(a.tail_part, a.head_part, last.y, last.z);
                }
                if (lane == 0) apply(last.x, sum, old, deg, at);
            }
        } else {
            /* the first rows' state does not wait for their sums */
            float ro[VB];
            uint32_t od[VB], cid[VB];
            auto load_rows = [&](uint32_t i0) {
#pragma unroll
                for (int u = 0; u < VB; ++u) {
                    const uint32_t i = i0 + u * ROW_THREADS;
                    if (i < r1) {
                        ro[u] = r_old[i];
                        od[u] = a.od_nz[i];
                        cid[u] = a.nz_cidx[i];
                    }
                }
            };
            load_rows(rg.r0 + tid);

            /* ---- rows that cross chunks, dealt to the warps one by one (long rows lie
             *      next to each other) ---- */
            for (uint32_t k0 = rg.s0; k0 < s1; k0 += ROW_THREADS) {
                const uint32_t k = k0 + lane * ROW_WARPS + warp;
                const bool have = k < s1;
                const uint4 sp = k0 == rg.s0 ? sp0 : have ? a.split[k] : make_uint4(0u, 0u, 0u, 0u);
                const bool is_long = have && sp.z - sp.y > LONG_SPAN;
                if (have && !is_long) a.nzsum[sp.x] = short_row_sum<true>(a.tail_part, a.head_part, sp.y, sp.z);
                for (uint32_t todo = __ballot_sync(FULL, is_long); todo; todo &= todo - 1u) {
                    const int j = __ffs((int)todo) - 1;
                    const uint32_t x = __shfl_sync(FULL, sp.x, j), cs = __shfl_sync(FULL, sp.y, j),
                                   ce = __shfl_sync(FULL, sp.z, j);
                    const float t = long_row_sum_warp<true>(a.head_part, cs, ce, lane);
                    if (lane == 0) a.nzsum[x] = __ldcg(a.tail_part + cs) + t;
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(ROW_THREADS) : "memory");

            /* ---- apply ---- */
            for (uint32_t i0 = rg.r0 + tid; i0 < r1; i0 += VB * ROW_THREADS) {
                float sum[VB];
                if (i0 != rg.r0 + tid) load_rows(i0);
#pragma unroll
                for (int u = 0; u < VB; ++u)
                    if (i0 + u * ROW_THREADS < r1) sum[u] = a.nzsum[i0 + u * ROW_THREADS];
#pragma unroll
                for (int u = 0; u < VB; ++u)
                    if (i0 + u * ROW_THREADS < r1) apply(i0 + u * ROW_THREADS, sum[u], ro[u], od[u], cid[u]);
            }
        }
        if (sweep < 2) { /* vertices without in-edges: constant from the first sweep on */
            for (uint32_t i = gtid; i < a.nzero; i += gthreads) {
                const uint32_t v = a.zero_rows[i];
                const double tele = (!pers || v == a.source) ? a.teleport : 0.0;
                const float rn = (float)__dadd_rn(tele, __dmul_rn(a.damping, 0.0));
                const float ro = sweep == 0 ? init_value(m, v) : rn;
                const uint32_t od = a.outdeg[v];
                c_new[a.zero_cidx[i]] = od ? __fdiv_rn(rn, (float)od) : 0.0f;
                d += fabs((double)rn - (double)ro);
                n += fabs((double)rn);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d += __shfl_down_sync(FULL, d, o);
            n += __shfl_down_sync(FULL, n, o);
        }
        if (lane == 0) s_red[warp] = make_double2(d, n);
        if (first < rg.c1) load_chunk(a, first, lane, pol_stream, col, meta, base);
        __syncthreads();
        if (warp == 0) {
            const double2 w = s_red[lane];
            double x = w.x, y = w.y;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x += __shfl_xor_sync(FULL, x, o);
                y += __shfl_xor_sync(FULL, y, o);
            }
            if (lane == 0) m.bres[(size_t)(sweep & 1u) * gridDim.x + blockIdx.x] = make_double2(x, y);
        }
        meets += gridDim.x;
        if (!res_sync(m, meets)) return;
        if (++sweep == m.max_sweeps) {
            if (warp == WARPS - 1) residual(sweep - 1);
            __syncthreads();
            break;
        }
    }

    if (m.out) {
        const float *r = m.rnz[sweep & 1];
        for (uint32_t i = rg.r0 + tid; i < rg.r1; i += EDGE_THREADS) m.out[a.nz_rows[i]] = r[i];
        const float t = (float)a.teleport;
        for (uint32_t i = gtid; i < a.nzero; i += gthreads) {
            const uint32_t v = a.zero_rows[i];
            m.out[v] = (!pers || v == a.source) ? t : 0.0f;
        }
    }
    if (gtid == 0) {
        m.status->sweeps = (int)sweep;
        m.status->done = s_stop;
        m.status->residual = s_res;
        __threadfence_system();
    }
}

}  // namespace

/* Where the line lies (host time of solves to 1e-8, this launch against the queued
 * kernels): 1.0 M edges 0.63 against 1.43 ms (3 sweeps: 60 against 125 us), 2.4 M
 * uniform 1.06 against 2.08, R-MAT of 3.9 M 1.13 against 2.16, 16 M 3.07 against 4.62,
 * 32 M 6.31 against 6.89; 67 M, with the limit lifted, 16.7 against 13.8: there the
 * CTAs' fixed ranges, cut by edges and rows alone, are less even than chunks dealt one
 * by one, and the scattered gathers want the texture path. Explicit launch configurations, source tiers and
 * per-sweep timing belong to the queued kernels. */
bool resident_applies(const gcg_graph *g, const gcg_pr_params *p) {
    const ChunkPlan &pl = *g->cplan;
    return !pl.configured && pl.tune_tiers <= 1 && !(p->flags & GCG_PR_TIME_SWEEPS) && p->max_sweeps > 0 &&
           pl.nchunks > 0 && g->ne <= RESIDENT_MAX_EDGES && g->nv <= RESIDENT_MAX_VERTICES;
}

int pagerank_resident(gcg_graph *g, const gcg_pr_params *p, float *out_rank, gcg_pr_stats *stats, bool *ran) {
    *ran = false;
    cudaStream_t s = g->stream;
    ChunkPlan &pl = *g->cplan;
    PrWork &w = pl.work;
    const uint32_t nv = g->nv;
    const size_t cstride = pr_contrib_stride(nv);

    if (!w.res_ctas) { /* once per graph: the CTAs' ranges, counters, events */
        int dev = 0, coop = 0, per_sm = 0;
        GCG_CUDA(cudaGetDevice(&dev));
        GCG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        GCG_CUDA(cudaFuncSetAttribute(k_pr_resident, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(HUB_MAX * 4)));
        GCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pr_resident, EDGE_THREADS,
                                                               HUB_DEFAULT * 4u));
        if (!coop || per_sm < 1) return GCG_OK; /* the queued kernels take it */
        const uint32_t ncta = std::min((uint32_t)num_sms(), std::max((pl.nchunks + WARPS / 2 - 1) / (WARPS / 2),
                                                                     (pl.nzero + ZERO_ROWS - 1) / ZERO_ROWS));
        GCG_TRY(w.res_rg.alloc(ncta));
        GCG_TRY(w.res_ctl.alloc(2 + ncta));
        GCG_TRY(w.res_bres.alloc(2 * (size_t)ncta));
        for (cudaEvent_t &e : w.ev)
            if (!e) GCG_CUDA(cudaEventCreate(&e));
        k_res_ranges<<<ncta / 32 + 1, 32, 0, s>>>(pl.chunk_nz.get(), pl.lane_meta.get(),
                                                     pl.split.get(), pl.nchunks, pl.nnz, pl.nsplit, ncta,
                                              pl.od_nz.get(), pl.nz_cidx.get(), w.res_rg.get(), w.res_ctl.get());
        GCG_LAUNCH_CHECK();
        GCG_CUDA(cudaMemcpyAsync(w.h_flags, w.res_ctl.get(), 4, cudaMemcpyDeviceToHost, s));
        GCG_CUDA(cudaStreamSynchronize(s));
        w.res_hub = std::min({(uint32_t)w.h_flags[0], pl.hub, HUB_DEFAULT});
        w.res_ctas = ncta;
    }

    const uint32_t hub = w.res_hub, hub_bytes = hub * 4u;
    tbuf<float> init_stage;
    const float *init_dev = nullptr;
    if (p->init_rank) {
        if (is_device_ptr(p->init_rank)) {
            init_dev = p->init_rank;
        } else {
            GCG_TRY(init_stage.alloc(nv, s));
            GCG_TRY(copy_in(init_stage.get(), p->init_rank, (size_t)nv * 4, s));
            init_dev = init_stage.get();
        }
    }
    const bool direct = out_rank && is_local_device_ptr(out_rank);

    ResArgs m;
    memset(&m, 0, sizeof(m));
    SweepArgs &a = m.a;
    a.col = pl.col_r.get();
    a.outdeg = g->outdeg.get();
    a.meta = pl.lane_meta.get();
    a.chunk_nz = pl.chunk_nz.get();
    a.nz_rows = pl.nz_rows.get();
    a.zero_rows = pl.zero_rows.get();
    a.split = pl.split.get();
    a.ne = g->ne;
    a.nchunks = pl.nchunks;
    a.nnz = pl.nnz;
    a.nzero = pl.nzero;
    a.nsplit = pl.nsplit;
    a.hub = hub;
    a.nz_cidx = pl.nz_cidx.get();
    a.zero_cidx = pl.zero_cidx.get();
    a.od_nz = pl.od_nz.get();
    a.nzsum = w.nzsum.get();
    a.head_part = w.parts.get();
    a.tail_part = w.parts.get() + pl.nchunks + 1;
    a.res_log = w.dres.get();
    a.delta_log = p->delta_log ? w.dres.get() + p->max_sweeps : nullptr;
    a.teleport = p->teleport;
    a.damping = p->damping;
    a.tol = p->tol;
    a.source = p->source;
    GCG_TRY(pr_norm_const(g, p, &a.norm_const));
    for (int h = 0; h < 2; ++h) {
        m.c[h] = w.c.get() + (size_t)h * cstride;
        m.rnz[h] = w.rnz.get() + (size_t)h * pl.nnz;
    }
    m.rg = w.res_rg.get();
    m.bar = w.res_ctl.get();
    m.err = (int *)(w.res_ctl.get() + 1);
    m.flag = w.res_ctl.get() + 2;
    m.bres = w.res_bres.get();
    m.init = p->init;
    m.init_rank = init_dev;
    m.out = !out_rank ? nullptr : direct ? out_rank : w.r.get();
    m.status = (ResStatus *)w.h_flags;
    m.max_sweeps = (uint32_t)p->max_sweeps;
    memset(w.h_flags, 0, sizeof(ResStatus));

    GCG_CUDA(cudaMemsetAsync(w.res_ctl.get(), 0, (2 + (size_t)w.res_ctas) * 4, s));
    m.spin_limit = RES_SPIN;
    if (p->flags & GCG_PR_TEST_BARRIER_TIMEOUT) { /* one arrival short */
        m.spin_limit = GCG_TEST_SPIN;
        GCG_CUDA(cudaMemsetAsync(m.bar, 0xFF, 4, s));
    }
    GCG_CUDA(cudaEventRecord(w.ev[0], s));
    void *kargs[] = {&m};
    const cudaError_t launched = cudaLaunchCooperativeKernel(
        (const void *)k_pr_resident, dim3(w.res_ctas), dim3(EDGE_THREADS), kargs, (size_t)hub_bytes, s);
    if (launched == cudaErrorCooperativeLaunchTooLarge) { /* fewer SMs than the device has: the queued kernels */
        cudaGetLastError();
        return GCG_OK;
    }
    GCG_CUDA(launched);
    GCG_CUDA(cudaEventRecord(w.ev[1], s));
    GCG_CUDA(cudaStreamSynchronize(s));
    *ran = true;
    ResStatus st; /* complete: the stream has been waited for */
    memcpy(&st, w.h_flags, sizeof(st));
    if (st.err) return fail(GCG_ERR_TIMEOUT, "pagerank: a wait between the CTAs of the solve ran out");
    float ms = 0.0f;
    GCG_CUDA(cudaEventElapsedTime(&ms, w.ev[0], w.ev[1]));
    GCG_TRY(pr_copy_logs(g, p, st.sweeps, a.res_log, a.delta_log));
    if (out_rank && !direct) {
        GCG_TRY(copy_out(out_rank, w.r.get(), (size_t)nv * sizeof(float), s));
        GCG_CUDA(cudaStreamSynchronize(s));
    }
    if (stats) {
        stats->sweeps = st.sweeps;
        stats->converged = st.done;
        stats->residual = st.residual;
        stats->device_ms = ms;
        stats->kernel_launches = 1;
    }
    return GCG_OK;
}

}  // namespace gcg
