/*
 * Batched personalised PageRank: k sources at once as a dense rank matrix.
 *
 * No reference counterpart (the reference runs one vector per engine run,
 * example_apps/pagerank.cpp); the per-source semantics are those of the
 * personalised scalar path: r_s[v] = (float)(tele_s(v) + damping*(double)sum_{u->v}
 * c_s[u]) with tele_s(v) = teleport if v == source_s else 0, c_s[u] = r_s[u]/outdeg[u]
 * in float, r_s starting at the indicator of source_s, and each source stopping
 * after its own first sweep with normalised L1 change (FP64) <= tol.
 *
 * Layout: vertex-major matrices R[V][kp], C[V][kp] (kp = k rounded up to 8, at most
 * 256 per group; larger k run group by group), so the contribution row of a source
 * vertex is one contiguous 4*kp-byte line, gathered with 128-bit loads by 8 or 16
 * lanes, a slice of at most 64 columns at a time.
 * Work: in-edge rows are cut into segments of at most 256 edges; one group of lanes
 * per segment broadcasts the segment's source ids with shuffles, keeps eight row
 * gathers in flight, and accumulates in registers. A row of one
 * segment is applied at once; longer rows leave per-segment partials that a
 * fix-up pass adds in segment order. Vertices without in-edges are constant after
 * the first sweep and are written only in sweeps 0 and 1. Per-column FP64
 * residuals are reduced in a fixed order. A column that converges is copied to the
 * result at that sweep (k_ppr_retire) and keeps being swept in place; when the
 * columns still iterating fit a layout at most 3/4 as wide, they are compacted into it.
 * Algorithmic traffic per sweep: E*(4 + 4*kp) + 3*V*4*kp bytes.
 */
#include <math.h>

#include <string.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "gcg_internal.cuh"

namespace gcg {
namespace {

constexpr uint32_t SEG = 256;     /* edges per segment */
constexpr int PPR_THREADS = 256;  /* 8 warps */
constexpr uint32_t KMAX = 256;    /* columns per group */
constexpr uint32_t NONE = 0xFFFFFFFFu;
constexpr int SEG_BLOCKS_MAX = 8; /* per SM, of the segment kernel */

/* A matrix row of kp columns is worked on in slices of at most SLICE columns by G lanes
 * with one float4 each (G = 16, or 8 for up to 32 columns), so a warp has two or four rows
 * under way. The slices of a sweep come one after another: each reads the source ids
 * again (4 bytes an edge beside 256 gathered), but the lines gathered meanwhile are a part
 * of the matrix only. With one row per warp and its columns spread over all lanes, a load
 * of 64 columns asked for 256 bytes, and four in flight were bound by their latency
 * (3.8 TB/s from L2). Per sweep, before -> now: R-MAT scale 20 with 57 of 100 columns
 * live 1.44 -> 0.44 ms (10.6 TB/s), 143 of 256 2.40 -> 1.23; scale 22, 126 of 256
 * 6.02 -> 4.05; uniform scale 20, 256 4.44 -> 3.18. What bounds it now is L2: 70 % of
 * its sectors hit, 17 M of 137 M come from the other die's half. */
constexpr uint32_t SLICE = 64;

/* the lanes' float4 of a row's slice; lanes past it, and rows that are off, hold zeros */
struct RowPart {
    float4 v;
};
__device__ __forceinline__ RowPart load_row(const float *row, uint32_t lanes, uint32_t gl, bool on) {
    RowPart x;
    x.v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (on && gl < lanes) x.v = __ldg((const float4 *)row + gl);
    return x;
}
__device__ __forceinline__ void store_row(float *row, uint32_t lanes, uint32_t gl, const RowPart &x) {
    if (gl < lanes) ((float4 *)row)[gl] = x.v;
}
__device__ __forceinline__ void add_row(RowPart &s, const RowPart &x) {
    s.v.x += x.v.x;
    s.v.y += x.v.y;
    s.v.z += x.v.z;
    s.v.w += x.v.w;
}

/* A slice: columns [c0, c0 + 4 lanes) */
struct Slice {
    uint32_t c0, lanes;
};

struct PprArgs {
    const uint32_t *col, *outdeg;
    const uint4 *seg;        /* (row, edge begin, edge end, partial slot or NONE) */
    const uint4 *multi;      /* (row, first slot, segment count, 0) */
    const uint32_t *zero_rows;
    uint32_t nseg, nmulti, nzero, kp, k;
    uint32_t slice;          /* columns per slice (the last may have fewer), a multiple of 8 */
    const uint32_t *src;     /* kp source ids (NONE for padding columns) */
    const float *c_old, *r_old;
    float *c_new, *r_new, *partial;
    double2 *bpart;          /* per block, per column (|dr|, |r|) */
    uint32_t nbseg;          /* blocks of the segment kernel (their partials come first) */
    uint32_t *ticket;
    int *done, *sweeps_done;
    double *res_log, *last_res;
    const double *norm_const; /* per column: |r| of constant vertices once no longer visited */
    int *col_sweeps;          /* per column: 0 while iterating, else the sweeps after which it converged */
    double *col_res;          /* per column: residual of its last iterated sweep */
    double teleport, damping, tol;
};

__device__ __forceinline__ Slice slice_at(const PprArgs &a, uint32_t c0) {
    return Slice{c0, min(a.slice, a.kp - c0) >> 2};
}

/* a lane's columns of the residual's two sums, and its columns' sources */
struct LaneColumns {
    double d[4], n[4];
    uint32_t src[4];
};
__device__ __forceinline__ void lane_columns(const PprArgs &a, Slice sl, uint32_t gl, LaneColumns &l) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        l.d[j] = l.n[j] = 0.0;
        l.src[j] = gl < sl.lanes ? a.src[sl.c0 + 4u * gl + j] : NONE;
    }
}

/* apply one row: r' = tele + damping*sum, c' = r'/outdeg, residual per column */
__device__ __forceinline__ void ppr_apply(const PprArgs &a, Slice sl, uint32_t v, const RowPart &sum, uint32_t gl,
                                          LaneColumns &l) {
    const size_t off = (size_t)v * a.kp + sl.c0;
    const RowPart ro = load_row(a.r_old + off, sl.lanes, gl, true);
    RowPart rn, cn;
    const uint32_t od = a.outdeg[v];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float s = (&sum.v.x)[j], old = (&ro.v.x)[j];
        const double tele = l.src[j] == v ? a.teleport : 0.0;
        const float r = (float)__dadd_rn(tele, __dmul_rn(a.damping, (double)s));
        (&rn.v.x)[j] = r;
        (&cn.v.x)[j] = od ? __fdiv_rn(r, (float)od) : 0.0f;
        l.d[j] += fabs((double)r - (double)old);
        l.n[j] += fabs((double)r);
    }
    store_row(a.r_new + off, sl.lanes, gl, rn);
    store_row(a.c_new + off, sl.lanes, gl, cn);
}

/* the block's sums per column of a slice, in a fixed order: the groups of a warp, then
 * the warps, then nmore partials of earlier blocks, `stride` apart */
template <int G>
__device__ __forceinline__ void block_columns(const PprArgs &a, Slice sl, LaneColumns &l, double2 (*s_part)[4 * G],
                                              double2 *out, const double2 *more, uint32_t nmore, uint32_t stride) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int o = G; o < 32; o <<= 1) {
            l.d[j] += __shfl_xor_sync(0xFFFFFFFFu, l.d[j], o);
            l.n[j] += __shfl_xor_sync(0xFFFFFFFFu, l.n[j], o);
        }
        if (lane < sl.lanes) s_part[warp][4u * lane + j] = make_double2(l.d[j], l.n[j]);
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < 4u * sl.lanes; c += blockDim.x) {
        double2 t = make_double2(0.0, 0.0);
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
            t.x += s_part[w][c].x;
            t.y += s_part[w][c].y;
        }
        for (uint32_t m = 0; m < nmore; ++m) {
            const double2 x = __ldcg(more + (size_t)m * stride * a.kp + sl.c0 + c);
            t.x += x.x;
            t.y += x.y;
        }
        out[sl.c0 + c] = t;
    }
    __syncthreads();
}

/* One group of lanes per segment of a slice (blockIdx.y: the slices come one after
 * another as the blocks do). The segments are sorted by length, so the groups of a warp take about
 * the same number of steps; a group past its end loads
 * nothing. The loads are written as they are because the rate hangs on it: as explicitly
 * predicated loads, all eight of a step leave at once and the sweep takes 570 us instead
 * of 440 (same sectors, same hit rates). */
template <int G>
__global__ void __launch_bounds__(PPR_THREADS) k_ppr_seg(PprArgs a) {
    if (*(volatile const int *)a.done) return;
    __shared__ double2 s_part[PPR_THREADS / 32][4 * G];
    const uint32_t FULL = 0xFFFFFFFFu;
    constexpr int U = 8; /* row gathers in flight per group */
    const uint32_t lane = threadIdx.x & 31u, gl = lane % G;
    const uint32_t gg = (blockIdx.x * blockDim.x + threadIdx.x) / G, ng = (gridDim.x * blockDim.x) / G;
    const uint32_t wfirst = gg - lane / G; /* the warp's first group: every lane loops alike */
    const uint32_t c0 = blockIdx.y * a.slice;
    const Slice sl = slice_at(a, c0);
    LaneColumns l;
    lane_columns(a, sl, gl, l);
    const float *c_old = a.c_old + c0;
    for (uint32_t k0 = wfirst; k0 < a.nseg; k0 += ng) {
        const uint32_t k = k0 + lane / G;
        const uint4 sg = k < a.nseg ? a.seg[k] : make_uint4(0u, 0u, 0u, 0u); /* row, eb, ee, slot */
        const uint32_t len = sg.z - sg.y, most = __reduce_max_sync(FULL, len);
        RowPart acc;
        acc.v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint32_t mine = gl < len ? __ldg(a.col + sg.y + gl) : 0u;
        for (uint32_t e0 = 0; e0 < most; e0 += G) {
            const uint32_t cur = mine, nx = e0 + G + gl;
            mine = nx < len ? __ldg(a.col + sg.y + nx) : 0u;
#pragma unroll
            for (int j = 0; j < G; j += U) {
                if (e0 + j >= most) break;
                RowPart x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t w = __shfl_sync(FULL, cur, j + u, G);
                    x[u] = load_row(c_old + (size_t)w * a.kp, sl.lanes, gl, e0 + j + u < len);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) add_row(acc, x[u]); /* past the end: + 0 */
            }
        }
        if (k < a.nseg) {
            if (sg.w == NONE) ppr_apply(a, sl, sg.x, acc, gl, l);
            else store_row(a.partial + (size_t)sg.w * a.kp + c0, sl.lanes, gl, acc);
        }
    }
    block_columns<G>(a, sl, l, s_part, a.bpart + (size_t)blockIdx.x * a.kp, nullptr, 0u, 0u);
}

/* rows of more than one segment (partials in segment order, eight in flight; the rows
 * of most segments first), the constant vertices in sweeps 0 and 1, then, in the last
 * block, the fixed-order per-column residual reduction and the stopping test. Each
 * block also adds its share of the segment kernel's partials, so the last block has
 * one per block of this kernel left to add (with all of them left to one thread per
 * column this kernel took 204 us at R-MAT scale 20, now 41). */
template <int G>
__global__ void __launch_bounds__(PPR_THREADS) k_ppr_fix(PprArgs a, int sweep, int const_pass) {
    if (*(volatile const int *)a.done) return;
    __shared__ double2 s_part[PPR_THREADS / 32][4 * G];
    __shared__ double s_res[KMAX];
    __shared__ int s_act[KMAX];
    __shared__ int s_last;
    constexpr int U = 8;
    const uint32_t gl = threadIdx.x % G;
    const uint32_t gg = (blockIdx.x * blockDim.x + threadIdx.x) / G, ng = (gridDim.x * blockDim.x) / G;
    double2 *const mypart = a.bpart + (size_t)a.nbseg * a.kp;
    const uint32_t c0 = blockIdx.y * a.slice;
    const Slice sl = slice_at(a, c0);
    LaneColumns l;
    lane_columns(a, sl, gl, l);
    for (uint32_t k = gg; k < a.nmulti; k += ng) {
        const uint4 m = a.multi[k]; /* row, first slot, count */
        const float *part = a.partial + (size_t)m.y * a.kp + c0;
        RowPart acc = load_row(part, sl.lanes, gl, true);
        for (uint32_t s = 1; s < m.z; s += U) {
            RowPart x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = load_row(part + (size_t)(s + u) * a.kp, sl.lanes, gl, s + u < m.z);
#pragma unroll
            for (int u = 0; u < U; ++u) add_row(acc, x[u]);
        }
        ppr_apply(a, sl, m.x, acc, gl, l);
    }
    if (const_pass) {
        RowPart zero;
        zero.v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t i = gg; i < a.nzero; i += ng) ppr_apply(a, sl, a.zero_rows[i], zero, gl, l);
    }
    __syncwarp();
    block_columns<G>(a, sl, l, s_part, mypart + (size_t)blockIdx.x * a.kp, a.bpart + (size_t)blockIdx.x * a.kp,
                     blockIdx.x < a.nbseg ? (a.nbseg - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u, gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(a.ticket, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    /* per column: residual of this sweep; a column stops after its own first
     * sweep with residual <= tol (it keeps being swept in place until the next
     * compaction, but its answer is taken at that sweep). SPLIT threads of a column
     * add a quarter of the blocks each, in block order */
    constexpr uint32_t SPLIT = 4;
    for (uint32_t c0 = 0; c0 < KMAX; c0 += PPR_THREADS / SPLIT) {
        const uint32_t c = c0 + threadIdx.x / SPLIT, part = threadIdx.x % SPLIT;
        const bool live = c < a.k && a.col_sweeps[c] == 0;
        double x = 0.0, y = 0.0;
        if (live) {
            const uint32_t per = (gridDim.x + SPLIT - 1) / SPLIT, b1 = min(gridDim.x, (part + 1) * per);
#pragma unroll 8
            for (uint32_t b = part * per; b < b1; ++b) {
                const double2 p = __ldcg(mypart + (size_t)b * a.kp + c);
                x += p.x;
                y += p.y;
            }
        }
#pragma unroll
        for (int o = 1; o < (int)SPLIT; o <<= 1) {
            x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
            y += __shfl_xor_sync(0xFFFFFFFFu, y, o);
        }
        if (part == 0) {
            int act = 0;
            double res = 0.0;
            if (live) {
                if (!const_pass) y += a.norm_const[c];
                res = y > 0.0 ? x / y : 0.0;
                a.col_res[c] = res;
                if (a.tol > 0.0 && res <= a.tol) a.col_sweeps[c] = sweep + 1;
                else act = 1;
            }
            s_res[c] = res;
            s_act[c] = act;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32u) {
        double worst = 0.0;
        int active = 0;
        for (uint32_t c = threadIdx.x; c < a.k; c += 32u) {
            worst = s_res[c] > worst ? s_res[c] : worst;
            active += s_act[c];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_xor_sync(0xFFFFFFFFu, worst, o);
            worst = w > worst ? w : worst;
            active += __shfl_xor_sync(0xFFFFFFFFu, active, o);
        }
        if (threadIdx.x == 0) {
            a.res_log[sweep] = worst;
            *a.last_res = worst;
            *a.sweeps_done = sweep + 1;
            if (active == 0) *a.done = 1;
            *a.ticket = 0u;
        }
    }
}

/* the columns that converged in this sweep (col_sweeps == sweep + 1) are copied
 * from the sweep's rank matrix to their place in the result */
__global__ void __launch_bounds__(256) k_ppr_retire(const float *__restrict__ r, uint32_t kp, uint32_t k, uint32_t nv,
                                                    const int *__restrict__ col_sweeps, int sweep_done,
                                                    const uint32_t *__restrict__ gcol, float *__restrict__ dst,
                                                    size_t dpitch) {
    __shared__ uint32_t s_l[KMAX], s_g[KMAX];
    __shared__ uint32_t s_n;
    if (threadIdx.x < 32u) { /* one warp lists them, 32 columns at a time */
        uint32_t n = 0;
        for (uint32_t c0 = 0; c0 < k; c0 += 32u) {
            const uint32_t c = c0 + threadIdx.x;
            const bool is = c < k && col_sweeps[c] == sweep_done;
            const uint32_t hit = __ballot_sync(0xFFFFFFFFu, is);
            if (is) {
                const uint32_t at = n + __popc(hit & ((1u << threadIdx.x) - 1u));
                s_l[at] = c;
                s_g[at] = gcol[c];
            }
            n += __popc(hit);
        }
        if (threadIdx.x == 0) s_n = n;
    }
    __syncthreads();
    const uint32_t n = s_n;
    if (n == 0) return;
    const uint64_t tot = (uint64_t)nv * n;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < tot; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)(i / n), j = (uint32_t)(i % n);
        dst[(size_t)v * dpitch + s_g[j]] = r[(size_t)v * kp + s_l[j]];
    }
}

/* copies columns of a V x kp matrix: dst[v*dpitch + dcol[j]] = src[v*kp + scol[j]] */
__global__ void k_ppr_columns(const float *__restrict__ src, uint32_t kp, uint32_t nv, const uint32_t *__restrict__ scol,
                              const uint32_t *__restrict__ dcol, uint32_t n, float *__restrict__ dst, size_t dpitch) {
    const uint64_t tot = (uint64_t)nv * n;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < tot; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)(i / n), j = (uint32_t)(i % n);
        dst[(size_t)v * dpitch + dcol[j]] = src[(size_t)v * kp + scol[j]];
    }
}

__global__ void k_ppr_seed(const uint32_t *__restrict__ src, uint32_t k, uint32_t kp, const uint32_t *__restrict__ outdeg,
                           float *__restrict__ r, float *__restrict__ c) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= k) return;
    const uint32_t v = src[j], od = outdeg[v];
    r[(size_t)v * kp + j] = 1.0f;
    c[(size_t)v * kp + j] = od ? __fdiv_rn(1.0f, (float)od) : 0.0f;
}

}  // namespace

/* Segments of the in-CSR for the batched sweeps, built once per graph. */
struct PprPlan {
    uint32_t nseg = 0, nmulti = 0, nzero = 0, nslots = 0;
    dbuf<uint4> seg, multi;
    dbuf<uint32_t> zero_rows;
    std::vector<uint32_t> indeg; /* host copy: constant-vertex test of the sources */
};

void free_ppr_plan(PprPlan *p) { delete p; }

static int ensure_ppr_plan(gcg_graph *g) {
    if (g->pplan) return GCG_OK;
    const uint32_t nv = g->nv;
    std::vector<uint32_t> rp((size_t)nv + 1);
    GCG_CUDA(cudaMemcpy(rp.data(), g->in_rowptr.get(), ((size_t)nv + 1) * 4, cudaMemcpyDeviceToHost));
    /* Segments longest first, so that the groups of a warp share rows of equal length, rows of
     * most segments first, otherwise in row order. Counted before they are placed: the host
     * builds this before the first sweep (4 M rows, a first call of two sweeps: 97 ms with lists that
     * grow, 133 with a sort after them, 55 so). */
    constexpr uint32_t MANY = 4096; /* segments of a row, from where on rows are sorted, not counted */
    std::vector<uint32_t> seg_at(SEG + 2, 0), multi_at(MANY + 2, 0);
    uint32_t nzero = 0, nslots = 0;
    for (uint32_t v = 0; v < nv; ++v) {
        const uint32_t d = rp[v + 1] - rp[v], full = d / SEG, rest = d % SEG;
        nzero += d == 0;
        seg_at[1] += full; /* of SEG edges */
        if (rest) ++seg_at[SEG - rest + 1];
        if (d > SEG) {
            const uint32_t ns = full + (rest != 0);
            ++multi_at[MANY - std::min(ns, MANY) + 1];
            nslots += ns;
        }
    }
    for (uint32_t i = 1; i < SEG + 2; ++i) seg_at[i] += seg_at[i - 1];
    for (uint32_t i = 1; i < MANY + 2; ++i) multi_at[i] += multi_at[i - 1];
    const uint32_t nseg = seg_at[SEG + 1], nmulti = multi_at[MANY + 1], nmany = multi_at[1];
    std::unique_ptr<uint4[]> seg(new uint4[nseg]), multi(new uint4[nmulti]);
    std::unique_ptr<uint32_t[]> zero(new uint32_t[nzero]);
    PprPlan *p = new PprPlan();
    p->indeg.resize(nv);
    uint32_t slot = 0, z = 0;
    for (uint32_t v = 0; v < nv; ++v) {
        const uint32_t b = rp[v], e = rp[v + 1], d = e - b;
        p->indeg[v] = d;
        if (d == 0) {
            zero[z++] = v;
        } else if (d <= SEG) {
            seg[seg_at[SEG - d]++] = make_uint4(v, b, e, NONE);
        } else {
            const uint32_t ns = (d + SEG - 1) / SEG;
            multi[multi_at[MANY - std::min(ns, MANY)]++] = make_uint4(v, slot, ns, 0u);
            for (uint32_t s = 0; s < ns; ++s) {
                const uint32_t s0 = b + s * SEG, s1 = e - s0 > SEG ? s0 + SEG : e;
                seg[seg_at[SEG - (s1 - s0)]++] = make_uint4(v, s0, s1, slot + s);
            }
            slot += ns;
        }
    }
    std::stable_sort(multi.get(), multi.get() + nmany, [](const uint4 &x, const uint4 &y) { return x.z > y.z; });
    p->nseg = nseg;
    p->nmulti = nmulti;
    p->nzero = nzero;
    p->nslots = nslots;
    if (p->seg.alloc(std::max(nseg, 1u)) || p->multi.alloc(std::max(nmulti, 1u)) ||
        p->zero_rows.alloc(std::max(nzero, 1u))) {
        delete p;
        return GCG_ERR_NOMEM;
    }
    cudaMemcpy(p->seg.get(), seg.get(), nseg * sizeof(uint4), cudaMemcpyHostToDevice);
    cudaMemcpy(p->multi.get(), multi.get(), nmulti * sizeof(uint4), cudaMemcpyHostToDevice);
    cudaMemcpy(p->zero_rows.get(), zero.get(), nzero * sizeof(uint32_t), cudaMemcpyHostToDevice);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        delete p;
        return fail(GCG_ERR_CUDA, std::string("ppr plan: ") + cudaGetErrorString(e));
    }
    g->pplan = p;
    return GCG_OK;
}

namespace {

/* rank / contribution matrices of one layout width, and its per-column state */
struct PprLayout {
    uint32_t kp = 0, k = 0;           /* padded width, columns in use */
    dbuf<float> r, c;                 /* 2 x V x kp each (the two sweep parities) */
    dbuf<uint32_t> src, gcol;         /* kp source ids (NONE for padding); group column of each */
    dbuf<double> norm_const, col_res; /* kp */
    dbuf<int> col_sweeps;             /* kp */
    int alloc(uint32_t nv, uint32_t width) {
        kp = width;
        /* room for whole 32 columns: later calls, with other numbers of columns left,
         * find these blocks in the cache */
        const size_t mat = (size_t)nv * ((kp + 31u) & ~31u);
        if (r.alloc(2 * mat) || c.alloc(2 * mat) || src.alloc(kp) || gcol.alloc(kp) || norm_const.alloc(kp) ||
            col_res.alloc(kp) || col_sweeps.alloc(kp))
            return GCG_ERR_NOMEM;
        return GCG_OK;
    }
};

/* Row width: whole 32-byte sectors; above one slice whole 128-byte lines, so that the
 * slices of a row share none (uniform scale 20, 100 columns: 104 wide 1.86 ms a sweep,
 * 112 1.79, 128 1.59; R-MAT scale 22, 126 live: 4.21, 4.95, 4.05). Narrow rows gain
 * nothing from whole lines (36 live as 40 or 64: 449, 460 us). */
uint32_t width_for(uint32_t n) { return n <= SLICE ? (n + 7u) & ~7u : (n + 31u) & ~31u; }

/* blocks of the segment kernel: what the SMs hold at once */
int seg_grid(uint32_t slice) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, slice <= 32 ? k_ppr_seg<8> : k_ppr_seg<16>, PPR_THREADS,
                                                      0) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    return num_sms() * std::min(per_sm, SEG_BLOCKS_MAX);
}

void ppr_sweep(const PprArgs &a, int nbfix, int sw, cudaStream_t s, std::vector<cudaEvent_t> *sev) {
    cudaEvent_t e0, e1;
    if (sev) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, s);
    }
    const uint32_t ns = (a.kp + a.slice - 1) / a.slice;
    if (a.slice <= 32) k_ppr_seg<8><<<dim3(a.nbseg, ns), PPR_THREADS, 0, s>>>(a);
    else k_ppr_seg<16><<<dim3(a.nbseg, ns), PPR_THREADS, 0, s>>>(a);
    if (sev) {
        cudaEventRecord(e1, s);
        sev->push_back(e0);
        sev->push_back(e1);
    }
    if (a.slice <= 32) k_ppr_fix<8><<<dim3(nbfix, ns), PPR_THREADS, 0, s>>>(a, sw, sw < 2 ? 1 : 0);
    else k_ppr_fix<16><<<dim3(nbfix, ns), PPR_THREADS, 0, s>>>(a, sw, sw < 2 ? 1 : 0);
}

/* columns scol[j] of src (V x kp) -> columns dcol[j] of dst (row pitch dpitch) */
int copy_columns(const float *src, uint32_t kp, uint32_t nv, const std::vector<uint32_t> &scol,
                 const std::vector<uint32_t> &dcol, float *dst, size_t dpitch, cudaStream_t s) {
    const uint32_t n = (uint32_t)scol.size();
    if (n == 0 || nv == 0) return GCG_OK;
    tbuf<uint32_t> d;
    GCG_TRY(d.alloc(2 * (size_t)n, s));
    std::vector<uint32_t> h(scol);
    h.insert(h.end(), dcol.begin(), dcol.end());
    GCG_CUDA(cudaMemcpyAsync(d.get(), h.data(), h.size() * 4, cudaMemcpyHostToDevice, s));
    const uint64_t tot = (uint64_t)nv * n;
    const unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((tot + 255) / 256, num_sms() * 16ull));
    k_ppr_columns<<<blocks, 256, 0, s>>>(src, kp, nv, d.get(), d.get() + n, n, dst, dpitch);
    GCG_LAUNCH_CHECK();
    GCG_CUDA(cudaStreamSynchronize(s)); /* h is host stack memory */
    return GCG_OK;
}

/* One group of k <= 256 sources. Each column stops after its own first sweep
 * with residual <= tol (the scalar path's rule): it is copied to the result at
 * that sweep; whenever the columns still iterating fit a layout at most 3/4 as
 * wide, they are compacted into it, so later sweeps gather narrower rows. */
int ppr_group(gcg_graph *g, const PprPlan &pl, const uint32_t *src_host, uint32_t k, const gcg_pr_params *p,
              float *out, uint32_t out_pitch, gcg_pr_stats *st, std::vector<double> *res_log,
              std::vector<int> *col_sweeps) {
    cudaStream_t s = g->stream;
    const uint32_t nv = g->nv;
    const int max_sweeps = p->max_sweeps;
    const int nbfix = num_sms() * 2;
    dbuf<float> partial, stage;
    dbuf<double2> bpart;
    dbuf<uint32_t> ctl;
    dbuf<double> dres;
    GCG_TRY(partial.alloc((size_t)std::max<uint32_t>(pl.nslots, 1) * KMAX));
    GCG_TRY(bpart.alloc((size_t)(num_sms() * SEG_BLOCKS_MAX + nbfix) * KMAX));
    GCG_TRY(ctl.alloc(4));
    GCG_TRY(dres.alloc((size_t)max_sweeps + 1));
    /* finished columns go straight to a device output, else to a staging matrix */
    const bool dev_out = is_device_ptr(out);
    float *res_dst = out;
    size_t res_pitch = out_pitch;
    if (!dev_out) {
        GCG_TRY(stage.alloc((size_t)nv * k));
        res_dst = stage.get();
        res_pitch = k;
    }
    std::vector<uint32_t> act(k); /* layout column -> group column */
    for (uint32_t j = 0; j < k; ++j) act[j] = j;
    std::vector<int> fin_sweeps(k, 0);
    std::vector<double> fin_res(k, 0.0);

    auto lay = std::make_unique<PprLayout>();
    GCG_TRY(lay->alloc(nv, width_for(k)));
    lay->k = k;
    auto upload_state = [&](PprLayout &L) -> int {
        std::vector<uint32_t> srcv(L.kp, NONE), gc(L.kp, 0u);
        std::vector<double> nc(L.kp, 0.0);
        for (uint32_t j = 0; j < L.k; ++j) {
            srcv[j] = src_host[act[j]];
            gc[j] = act[j];
            if (pl.indeg[srcv[j]] == 0) nc[j] = fabs((double)(float)p->teleport);
        }
        GCG_CUDA(cudaMemcpyAsync(L.src.get(), srcv.data(), L.kp * 4, cudaMemcpyHostToDevice, s));
        GCG_CUDA(cudaMemcpyAsync(L.gcol.get(), gc.data(), L.kp * 4, cudaMemcpyHostToDevice, s));
        GCG_CUDA(cudaMemcpyAsync(L.norm_const.get(), nc.data(), L.kp * 8, cudaMemcpyHostToDevice, s));
        GCG_CUDA(cudaMemsetAsync(L.col_sweeps.get(), 0, L.kp * 4, s));
        GCG_CUDA(cudaMemsetAsync(L.col_res.get(), 0, L.kp * 8, s));
        GCG_CUDA(cudaStreamSynchronize(s));
        return GCG_OK;
    };
    GCG_TRY(upload_state(*lay));
    GCG_CUDA(cudaMemsetAsync(ctl.get(), 0, 16, s));
    GCG_CUDA(cudaMemsetAsync(lay->r.get(), 0, (size_t)nv * lay->kp * 4, s));
    GCG_CUDA(cudaMemsetAsync(lay->c.get(), 0, (size_t)nv * lay->kp * 4, s));
    k_ppr_seed<<<(k + 255) / 256, 256, 0, s>>>(lay->src.get(), k, lay->kp, g->outdeg.get(), lay->r.get(), lay->c.get());
    GCG_LAUNCH_CHECK();

    PprArgs a;
    memset(&a, 0, sizeof(a));
    a.col = g->in_col.get();
    a.outdeg = g->outdeg.get();
    a.seg = pl.seg.get();
    a.multi = pl.multi.get();
    a.zero_rows = pl.zero_rows.get();
    a.nseg = pl.nseg;
    a.nmulti = pl.nmulti;
    a.nzero = pl.nzero;
    a.partial = partial.get();
    a.bpart = bpart.get();
    a.ticket = ctl.get();
    a.done = (int *)(ctl.get() + 1);
    a.sweeps_done = (int *)(ctl.get() + 2);
    a.res_log = dres.get();
    a.last_res = dres.get() + max_sweeps;
    a.teleport = p->teleport;
    a.damping = p->damping;
    a.tol = p->tol;
    auto bind = [&](PprLayout &L) {
        a.kp = L.kp;
        a.k = L.k;
        a.slice = std::min(L.kp, SLICE);
        a.nbseg = (uint32_t)seg_grid(a.slice);
        a.src = L.src.get();
        a.norm_const = L.norm_const.get();
        a.col_sweeps = L.col_sweeps.get();
        a.col_res = L.col_res.get();
    };
    bind(*lay);

    const bool time_sweeps = (p->flags & GCG_PR_TIME_SWEEPS) != 0;
    cudaEvent_t ev0, ev1;
    GCG_CUDA(cudaEventCreate(&ev0));
    GCG_CUDA(cudaEventCreate(&ev1));
    std::vector<cudaEvent_t> sev;
    GCG_CUDA(cudaEventRecord(ev0, s));
    int sweep = 0, launches = 1, compactions = 0;
    bool done = false;
    std::vector<int> hsw(KMAX);
    std::vector<double> hres(KMAX);
    while (sweep < max_sweeps && !done) {
        const int n = std::min(4, max_sweeps - sweep);
        const size_t mat = (size_t)nv * lay->kp;
        for (int i = 0; i < n; ++i) {
            const int sw = sweep + i;
            a.r_old = lay->r.get() + (size_t)(sw & 1) * mat;
            a.c_old = lay->c.get() + (size_t)(sw & 1) * mat;
            a.r_new = lay->r.get() + (size_t)((sw + 1) & 1) * mat;
            a.c_new = lay->c.get() + (size_t)((sw + 1) & 1) * mat;
            ppr_sweep(a, nbfix, sw, s, time_sweeps ? &sev : nullptr);
            if (p->tol > 0.0)
                k_ppr_retire<<<num_sms(), 256, 0, s>>>(a.r_new, lay->kp, lay->k, nv, lay->col_sweeps.get(), sw + 1,
                                                       lay->gcol.get(), res_dst, res_pitch);
        }
        GCG_LAUNCH_CHECK();
        launches += (p->tol > 0.0 ? 3 : 2) * n;
        sweep += n;
        if (!(p->tol > 0.0)) continue;
        uint32_t h[4];
        GCG_CUDA(cudaMemcpyAsync(h, ctl.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
        GCG_CUDA(cudaMemcpyAsync(hsw.data(), lay->col_sweeps.get(), lay->k * 4, cudaMemcpyDeviceToHost, s));
        GCG_CUDA(cudaStreamSynchronize(s));
        if (h[1]) {
            done = true;
            sweep = (int)h[2];
            break;
        }
        uint32_t nact = 0;
        for (uint32_t j = 0; j < lay->k; ++j) nact += hsw[j] == 0;
        if (sweep >= max_sweeps || 4 * width_for(nact) > 3 * lay->kp) continue;
        /* compact the columns still iterating into a narrower layout (the others
         * are already in the result) */
        GCG_CUDA(cudaMemcpyAsync(hres.data(), lay->col_res.get(), lay->k * 8, cudaMemcpyDeviceToHost, s));
        GCG_CUDA(cudaStreamSynchronize(s));
        const float *rcur = lay->r.get() + (size_t)(sweep & 1) * mat;
        const float *ccur = lay->c.get() + (size_t)(sweep & 1) * mat;
        std::vector<uint32_t> ks, kd, nact_cols;
        for (uint32_t j = 0; j < lay->k; ++j) {
            if (hsw[j]) {
                fin_sweeps[act[j]] = hsw[j];
                fin_res[act[j]] = hres[j];
            } else {
                ks.push_back(j);
                kd.push_back((uint32_t)nact_cols.size());
                nact_cols.push_back(act[j]);
            }
        }
        auto nxt = std::make_unique<PprLayout>();
        GCG_TRY(nxt->alloc(nv, width_for(nact)));
        nxt->k = nact;
        const size_t nmat = (size_t)nv * nxt->kp;
        GCG_CUDA(cudaMemsetAsync(nxt->r.get(), 0, 2 * nmat * 4, s));
        GCG_CUDA(cudaMemsetAsync(nxt->c.get(), 0, 2 * nmat * 4, s));
        for (int par = 0; par < 2; ++par) { /* both parities: rows not swept any more keep their values */
            GCG_TRY(copy_columns(rcur, lay->kp, nv, ks, kd, nxt->r.get() + (size_t)par * nmat, nxt->kp, s));
            GCG_TRY(copy_columns(ccur, lay->kp, nv, ks, kd, nxt->c.get() + (size_t)par * nmat, nxt->kp, s));
        }
        act = nact_cols;
        GCG_TRY(upload_state(*nxt));
        lay = std::move(nxt);
        bind(*lay);
        launches += 4;
        ++compactions;
    }
    GCG_CUDA(cudaEventRecord(ev1, s));
    GCG_CUDA(cudaEventSynchronize(ev1));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    uint32_t ctlh[4];
    GCG_CUDA(cudaMemcpy(ctlh, ctl.get(), sizeof(ctlh), cudaMemcpyDeviceToHost));
    const int sweeps = (int)ctlh[2];
    double seg_ms = 0.0;
    int timed = 0;
    for (size_t i = 0; i + 1 < sev.size(); i += 2) {
        float t = 0.0f;
        if (cudaEventElapsedTime(&t, sev[i], sev[i + 1]) == cudaSuccess && (int)(i / 2) < sweeps) {
            seg_ms += t;
            ++timed;
        }
        cudaEventDestroy(sev[i]);
        cudaEventDestroy(sev[i + 1]);
    }
    cudaGetLastError();
    /* the columns still in the layout: final values are in the buffer of the last sweep */
    GCG_CUDA(cudaMemcpy(hsw.data(), lay->col_sweeps.get(), lay->k * 4, cudaMemcpyDeviceToHost));
    GCG_CUDA(cudaMemcpy(hres.data(), lay->col_res.get(), lay->k * 8, cudaMemcpyDeviceToHost));
    {
        /* columns that never converged: the buffer of the last sweep */
        std::vector<uint32_t> ks, kd;
        for (uint32_t j = 0; j < lay->k; ++j) {
            fin_sweeps[act[j]] = hsw[j] ? hsw[j] : sweeps;
            fin_res[act[j]] = hres[j];
            if (!hsw[j]) {
                ks.push_back(j);
                kd.push_back(act[j]);
            }
        }
        const float *rfin = lay->r.get() + (size_t)(sweeps & 1) * (size_t)nv * lay->kp;
        GCG_TRY(copy_columns(rfin, lay->kp, nv, ks, kd, res_dst, res_pitch, s));
        launches += ks.empty() ? 0 : 1;
    }
    if (res_log && sweeps > 0) {
        std::vector<double> lg((size_t)sweeps);
        GCG_CUDA(cudaMemcpy(lg.data(), dres.get(), (size_t)sweeps * 8, cudaMemcpyDeviceToHost));
        if (res_log->size() < lg.size()) res_log->resize(lg.size(), 0.0);
        for (size_t i = 0; i < lg.size(); ++i) (*res_log)[i] = std::max((*res_log)[i], lg[i]);
    }
    if (!dev_out)
        GCG_CUDA(cudaMemcpy2DAsync(out, (size_t)out_pitch * 4, stage.get(), (size_t)k * 4, (size_t)k * 4, nv,
                                   cudaMemcpyDeviceToHost, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    bool conv = p->tol > 0.0;
    double worst = 0.0;
    int mx = 0;
    for (uint32_t j = 0; j < k; ++j) {
        mx = std::max(mx, fin_sweeps[j]);
        worst = std::max(worst, fin_res[j]);
        if (!(p->tol > 0.0 && fin_res[j] <= p->tol)) conv = false;
    }
    if (col_sweeps) col_sweeps->insert(col_sweeps->end(), fin_sweeps.begin(), fin_sweeps.end());
    st->sweeps = std::max(st->sweeps, mx);
    st->converged = st->converged && conv;
    st->residual = std::max(st->residual, worst);
    st->device_ms += ms;
    st->sweep_kernel_ms += seg_ms;
    st->timed_sweeps += timed;
    st->kernel_launches += launches;
    (void)compactions;
    return GCG_OK;
}

}  // namespace
}  // namespace gcg

using namespace gcg;

extern "C" int gcg_ppr_batched(gcg_graph *g, const uint32_t *sources, uint32_t nsources, const gcg_pr_params *params,
                               float *out, gcg_pr_stats *stats) {
    if (!g || !sources || !params || !out) return fail(GCG_ERR_INVALID, "gcg_ppr_batched: null argument");
    if (nsources == 0) return fail(GCG_ERR_INVALID, "gcg_ppr_batched: nsources must be > 0");
    if (params->mode != GCG_PR_JACOBI || params->init_rank || params->source != GCG_NO_SOURCE)
        return fail(GCG_ERR_UNSUPPORTED,
                    "gcg_ppr_batched: Jacobi from the source indicators only (no init_rank, no source field)");
    if (params->max_sweeps < 0) return fail(GCG_ERR_INVALID, "gcg_ppr_batched: max_sweeps < 0");
    std::vector<uint32_t> src(nsources);
    GCG_CUDA(cudaMemcpy(src.data(), sources, (size_t)nsources * 4, cudaMemcpyDefault));
    for (uint32_t j = 0; j < nsources; ++j)
        if (src[j] >= g->nv) return fail(GCG_ERR_INVALID, "gcg_ppr_batched: source id >= num_vertices");
    GCG_TRY(ensure_ppr_plan(g));
    gcg_pr_stats st = {0, 1, 0.0, 0.0, 0.0, 0, 0};
    std::vector<double> lg;
    std::vector<int> col_sweeps; /* sweeps each source took */
    for (uint32_t g0 = 0; g0 < nsources; g0 += KMAX) {
        const uint32_t k = std::min(KMAX, nsources - g0);
        GCG_TRY(ppr_group(g, *g->pplan, src.data() + g0, k, params, out + g0, nsources, &st, &lg, &col_sweeps));
    }
    if (params->residuals && !lg.empty()) GCG_TRY(copy_out(params->residuals, lg.data(), lg.size() * 8, g->stream));
    if (params->work_log && params->max_sweeps > 0) {
        /* cumulative work of the sources still iterating: sweep i updates every
         * vertex and gathers every in-edge once per source with more than i sweeps */
        const int S = params->max_sweeps;
        std::vector<uint64_t> active((size_t)S + 1, 0);
        for (int c : col_sweeps) ++active[(size_t)std::min(c, S)];
        std::vector<uint64_t> wl(2 * (size_t)S);
        uint64_t left = col_sweeps.size(), upd = 0, gat = 0;
        for (int i = 0; i < S; ++i) {
            left -= active[(size_t)i]; /* sources that took exactly i sweeps are done */
            upd += left * (uint64_t)g->nv;
            gat += left * g->ne;
            wl[2 * (size_t)i] = upd;
            wl[2 * (size_t)i + 1] = gat;
        }
        GCG_TRY(copy_out(params->work_log, wl.data(), wl.size() * 8, g->stream));
    }
    if (stats) *stats = st;
    return GCG_OK;
}
