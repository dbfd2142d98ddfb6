/*
 * Exact vertex-API PageRank: the in-memory program of example_apps/pagerank.cpp
 * (:121-146) as the engine runs it with deterministic parallelism
 * (src/engine/graphchi_engine.hpp:396-454): one Gauss-Seidel sweep per iteration
 * in ascending vertex id order, each vertex reading the values its smaller-id
 * in-neighbours wrote in this sweep and its larger-id in-neighbours' values from
 * the previous sweep, summing them in ascending source order in float.
 *
 * Parallel form: vertex v depends on in-neighbours u < v only, so v's level
 * (1 + max level of those u, 0 if none) orders the sweep: every level is a set of
 * independent vertices. Within a sweep, levels run in order; each vertex sums
 * sequentially (bit-exact float order), reading new values below its id and old
 * values above it. Levels come from topological rounds over the in-CSR and a radix
 * sort of (level, id); a sweep is one cooperative launch with a grid barrier between
 * levels, and the sums of long rows, though sequential by definition, are evaluated
 * in parallel with the same bits (group_add).
 *
 * The same schedule runs the edge-value program of the app (PagerankProgram,
 * example_apps/pagerank.cpp:73-113, taken when num_vertices * 4 >= membudget):
 * there the value on every out-edge of u is u's pagerank / outdeg in float,
 * initially (float)(1.0/outdeg), the vertex value is the pagerank itself, and
 * each iteration logs the sum of |pagerank - old| (pagerank.cpp:108).
 */
#include <algorithm>
#include <vector>

#include "gcg_internal.cuh"

namespace gcg {
namespace {

/* Levels of the id-ordered dependency DAG (edges u -> v with u < v) by
 * topological rounds (Kahn): a vertex's level is 1 + the largest level of its
 * smaller-id in-neighbours, i.e. the round after its last such neighbour's. */

/* pending[v] = number of in-neighbours u < v (sources ascending: a binary search) */
__global__ void k_gs_pending(const uint32_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t nv,
                             uint32_t *__restrict__ pending) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        uint32_t lo = rowptr[v], hi = rowptr[v + 1]; /* first position with col >= v */
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (col[mid] < v) lo = mid + 1; else hi = mid;
        }
        pending[v] = lo - rowptr[v];
    }
}

/* keys (u << vbits) | v of the edges u -> v with u < v, compacted by a scan
 * over the per-vertex counts */
__global__ void k_gs_fwd_keys(const uint32_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t nv,
                              const uint32_t *__restrict__ pending, const uint32_t *__restrict__ pos, uint32_t vbits,
                              uint64_t *__restrict__ keys) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const uint32_t b = rowptr[v], n = pending[v], o = pos[v];
        for (uint32_t j = 0; j < n; ++j) keys[o + j] = ((uint64_t)col[b + j] << vbits) | v;
    }
}

/* fwd_off[u] = first sorted key with source >= u (keys sorted by source) */
__global__ void k_gs_fwd_off(const uint64_t *__restrict__ keys, uint64_t n, uint32_t vbits, uint32_t nv,
                             uint32_t *__restrict__ off, uint32_t *__restrict__ dst) {
    const uint64_t mask = (1ull << vbits) - 1ull;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        dst[i] = (uint32_t)(k & mask);
        const int64_t u = (int64_t)(k >> vbits);
        const int64_t prev = i == 0 ? -1 : (int64_t)(keys[i - 1] >> vbits);
        for (int64_t x = prev + 1; x <= u; ++x) off[x] = (uint32_t)i;
        if (i == n - 1)
            for (int64_t x = u + 1; x <= (int64_t)nv; ++x) off[x] = (uint32_t)n;
    }
}

/* round 0: the vertices without smaller-id in-neighbours */
__global__ void k_gs_roots(const uint32_t *__restrict__ pending, uint32_t nv, uint32_t *__restrict__ front,
                           uint32_t *__restrict__ count) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
        if (pending[v] == 0) front[atomicAdd(count, 1u)] = v;
}

/* one round: a warp per vertex of the current frontier (level r) releases its
 * forward edges; a vertex whose last pending in-neighbour this is joins the next
 * frontier with level r + 1. Counts per round: cnt[r] = frontier size of round
 * r; rounds whose frontier is empty return at once (several are queued). */
__global__ void __launch_bounds__(256) k_gs_round(uint32_t r, const uint32_t *__restrict__ fwd_off,
                                                  const uint32_t *__restrict__ fwd_dst, uint32_t *pending,
                                                  uint32_t *level, const uint32_t *__restrict__ front_cur,
                                                  uint32_t *front_next, uint32_t *cnt) {
    const uint32_t n = *(volatile const uint32_t *)(cnt + r);
    if (n == 0) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
        const uint32_t u = front_cur[i];
        for (uint32_t j = fwd_off[u] + lane; j < fwd_off[u + 1]; j += 32) {
            const uint32_t v = fwd_dst[j];
            if (atomicSub(pending + v, 1u) == 1u) {
                level[v] = r + 1;
                front_next[atomicAdd(cnt + r + 1, 1u)] = v;
            }
        }
    }
}

/* Vertex classes of a level, by in-degree: a thread sums a row of at most
 * GS_THREAD_MAX in-edges, a warp one of at most GS_WARP_MAX, a group of threads a
 * longer one. The result is always that of adding the in-edges one after another in
 * ascending source order (a float sum is not associative). A thread's and a warp's
 * row have all their loads in flight at once: with 32 in-edges per thread, eight at a
 * time, and a warp's batches one ahead, their latencies made most of a small level
 * (scale 14: 8.4 against 6.0 us a level).
 *
 * A wide level has more rows than threads wait for: there what counts is how many rows are
 * under way. Where its rows of up to GS_WIDE_THREAD in-edges outnumber the warps they go to
 * the threads (3 sweeps of a uniform graph of 16 in-edges, 4 M vertices: 8.8 ms by warps,
 * 1.83 by threads; one launch per level, a full grid each, took 3.2), and where its rows of
 * up to GS_WIDE_WARP outnumber half the warps, four a group, they go to the warps (100,000
 * rows of 300 in-edges in one level: 2.89 -> 0.68 ms). */
constexpr uint32_t GS_THREAD_MAX = 8, GS_WARP_MAX = 256;
constexpr uint32_t GS_WIDE_THREAD = 32, GS_WIDE_WARP = 4096;
/* Rows that a warp of a level takes one by one, adding from shuffles: the quickest for one
 * row. Beyond, it loads what it needs of 32 rows at once, and the next row's columns behind
 * a row's adds, which go through shared memory: with all warps at it shuffles are bound by
 * their rate (500,000 rows of 100 in-edges: 1.59 -> 1.12 ms). */
constexpr uint32_t GS_FEW_ROUNDS = 4;
constexpr int GS_CLASSES = 4; /* segments per level: thread, thread in a wide level, warp, block */

/* rows of level l with up to GS_WIDE_THREAD in-edges that are beyond the thread class: mid[2 l];
 * with up to GS_WIDE_WARP that are beyond the warp class: mid[2 l + 1] */
__global__ void k_level_mid(const uint32_t *__restrict__ level, const uint32_t *__restrict__ rowptr, uint32_t nv,
                            uint32_t *__restrict__ mid) {
    const uint64_t end = ((uint64_t)nv + 31u) & ~31ull; /* whole warps: the ballot below */
    for (uint64_t v = blockIdx.x * blockDim.x + threadIdx.x; v < end; v += gridDim.x * blockDim.x) {
        const uint32_t d = v < nv ? rowptr[v + 1] - rowptr[v] : 0u;
        const bool counts = (d > GS_THREAD_MAX && d <= GS_WIDE_THREAD) || (d > GS_WARP_MAX && d <= GS_WIDE_WARP);
        const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, counts);
        if (!counts) continue;
        uint32_t *const at = mid + 2 * (size_t)level[v] + (d > GS_WARP_MAX);
        const uint32_t same = __match_any_sync(lanes, (unsigned long long)at);
        if ((threadIdx.x & 31u) == (uint32_t)__ffs((int)same) - 1u) atomicAdd(at, (uint32_t)__popc(same));
    }
}

/* sort key: level, class, vertex id */
__global__ void k_level_keys(const uint32_t *__restrict__ level, const uint32_t *__restrict__ rowptr, uint32_t nv,
                             const uint32_t *__restrict__ mid, uint32_t warps, uint32_t vbits, uint64_t *keys) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const uint32_t d = rowptr[v + 1] - rowptr[v], l = level[v], *m = mid + 2 * (size_t)l;
        const uint64_t cls = d <= GS_THREAD_MAX                       ? 0u
                             : d <= GS_WIDE_THREAD && m[0] > warps    ? 1u
                             : d <= GS_WARP_MAX                       ? 2u
                             : d <= GS_WIDE_WARP && m[1] > warps / 2u ? 2u
                                                                      : 3u;
        keys[v] = ((((uint64_t)l << 2) | cls) << vbits) | v;
    }
}

/* order[i] = vertex of sorted key i; off[x] = first i whose segment
 * (level * GS_CLASSES + class) is >= x, for x in [0, nseg] */
__global__ void k_level_bounds(const uint64_t *__restrict__ keys, uint32_t nv, uint32_t vbits, uint32_t nseg,
                               uint32_t *__restrict__ off, uint32_t *__restrict__ order) {
    const uint64_t mask = (1ull << vbits) - 1ull;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
        uint64_t k = keys[i];
        order[i] = (uint32_t)(k & mask);
        int64_t l = (int64_t)(k >> vbits);
        int64_t prev = i == 0 ? -1 : (int64_t)(keys[i - 1] >> vbits);
        for (int64_t x = prev + 1; x <= l; ++x) off[x] = i;
        if (i == nv - 1)
            for (int64_t x = l + 1; x <= (int64_t)nseg; ++x) off[x] = nv;
    }
}

/* what a sweep reads of a level: where its thread, warp and block class begin, and its end */
__global__ void k_level_pack(const uint32_t *__restrict__ seg, uint32_t nlev, uint4 *__restrict__ off) {
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < nlev; l += gridDim.x * blockDim.x) {
        const uint32_t *s = seg + (size_t)GS_CLASSES * l;
        off[l] = make_uint4(s[0], s[2], s[3], s[4]);
    }
}

/* pagerank.cpp:124,137-139: pr starts at 0.15; iteration 0 sets 1/outc when outc > 0 */
__global__ void k_gs_init(uint32_t nv, const uint32_t *__restrict__ outdeg, float reset, float *pr) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        uint32_t oc = outdeg[v];
        pr[v] = oc > 0 ? __fdiv_rn(1.0f, (float)oc) : reset;
    }
}

/* pagerank.cpp:80-83 (edge-value program, iteration 0): out-edges hold
 * (float)(1.0 / outdeg) */
__global__ void k_gs_edge_init(uint32_t nv, const uint32_t *__restrict__ outdeg, float *c) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const uint32_t oc = outdeg[v];
        c[v] = oc > 0 ? __double2float_rn(__ddiv_rn(1.0, (double)oc)) : 0.0f;
    }
}

/* 4-byte asynchronous copy global -> shared (through L1), in commit groups */
__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
/* The apply of one vertex. In-memory program (EDGE = false), pagerank.cpp:127-136:
 * pr = (float)((0.15 + 0.85 * (double)sum) / outc). Edge-value program (EDGE =
 * true), pagerank.cpp:89-111: pagerank = (float)(0.15 + 0.85 * (double)sum), the
 * out-edge value pagerank / outc in float. TRACK (always with EDGE): the vertex's
 * pagerank goes to val[v] and |pagerank - previous| (float) to delta[v], for
 * the progress log and the residual stop. Explicit round-to-nearest ops: no FMA
 * contraction, the same rounding as the reference's separate double multiply
 * and add. */
template <bool EDGE, bool TRACK>
__device__ __forceinline__ void gs_apply(uint32_t v, float sum, uint32_t outdeg, float *pr_new,
                                         float *val, float *delta, double reset, double damping) {
    const int outc = (int)outdeg;
    const double t = __dadd_rn(reset, __dmul_rn(damping, (double)sum));
    if (EDGE) pr_new[v] = outc > 0 ? __fdiv_rn(__double2float_rn(t), (float)outc) : 0.0f;
    else pr_new[v] = outc > 0 ? (float)__ddiv_rn(t, (double)outc) : (float)t;
    if (TRACK) {
        const float pagerank = __double2float_rn(t);
        delta[v] = fabsf(__fsub_rn(pagerank, val[v]));
        val[v] = pagerank;
    }
}

/* ---- exact sums of long rows ------------------------------------------------
 * A row's value is the float sum of its in-edge values one after another, each add
 * rounded: a chain of dependent adds. It can be evaluated in parallel, bit for bit,
 * as long as the running sum stays in one binade: there the sum is a whole number m
 * of its ulp u, and adding x >= 0 makes it m + round(x / u), to nearest, ties to the
 * even result. The increment depends on m only through m's parity, and only in a tie,
 * so each value is a function of the parity (two increments), and such functions
 * compose associatively: a prefix scan gives every partial sum. With E the binade's
 * first float (even) and E' the next one (odd), the two increments are
 * bits(E + x) - bits(E) and bits(E' + x) - bits(E'): one float add each. The first
 * partial sum that leaves the binade is formed by an ordinary add, and the scan starts
 * again behind it in the new binade, at most once per doubling of the sum. Sums that
 * are zero, subnormal or not finite and values that are negative or NaN go one by one.
 *
 * A thread adds in ~4.5 cycles a value; a pass takes ~500 cycles for up to 1,024
 * values, ~1,100 where the sum leaves its binade. R-MAT, per sweep, against one launch
 * per level and one thread's adds: scale 20 10.6 -> 6.1 ms, scale 22 29.1 -> 15.2 ms
 * (1,340 levels, 11.3 us each: barrier and value latency ~4, the longest row's sum the
 * rest). */
constexpr uint32_t GS_GROUP = 256;                /* threads that take a block-class row */
constexpr uint32_t GS_STEP = 4 * GS_GROUP;        /* values of a step, four per thread */
constexpr uint32_t GS_DEPTH = 3;                  /* steps in flight */
constexpr uint32_t GS_THREADS = 512;              /* one CTA per SM, two groups */
constexpr uint32_t GS_GROUPS = GS_THREADS / GS_GROUP;
constexpr uint32_t GS_TAIL = 64;                  /* so few values are added by one thread */
constexpr uint32_t GS_HEAD = 256;                 /* a row's first values: the sum doubles too often for the scan
                                                     (scale 20: 128 6.72 ms, 256 6.47, 512 6.50) */
constexpr uint32_t BINADE = 1u << 23;             /* ulps in a binade */
constexpr uint32_t INC_MAX = 1u << 24;            /* increments are cut here: past any binade's end */

constexpr uint32_t GS_WARPS = GS_GROUP / 32;
constexpr uint32_t ODD_VALUES = 0xFFFFFFFFu;      /* in place of a warp's increment */

/* Shared memory of a group. What one pass or thread tells the group alternates between
 * two places: between two uses of one place lies a barrier that every reader of the
 * first has passed after reading. */
struct GsGroup {
    float val[GS_DEPTH][GS_STEP];
    uint2 total[2][GS_WARPS]; /* each warp's increment for an even and an odd start */
    struct {
        float sum;
        uint32_t pos;
    } told[2];
};

static_assert(sizeof(GsGroup) % 16 == 0, "the second group's 128-bit reads");

__device__ __forceinline__ void group_sync(uint32_t grp) {
    asm volatile("bar.sync %0, %1;" ::"r"(grp + 1u), "n"(GS_GROUP) : "memory");
}

/* s + sv[k] + ... + sv[end - 1], one after another */
__device__ __forceinline__ float add_in_order(float s, const float *sv, uint32_t k, uint32_t end) {
    for (; k < end && (k & 3u); ++k) s += sv[k];
    for (; k + 16 <= end; k += 16) { /* four loads, then the sixteen adds */
        float4 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *(const float4 *)(sv + k + 4 * i);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s += q[i].x;
            s += q[i].y;
            s += q[i].z;
            s += q[i].w;
        }
    }
    for (; k < end; ++k) s += sv[k];
    return s;
}

/* sum + sv[0] + ... + sv[n - 1] in this order, by a group; every thread has sum and
 * gets the result. head: values that one thread adds first. par: which of the two
 * places are next, bit 0 for total, bit 1 for told. */
__device__ __forceinline__ float group_add(GsGroup &g, const float *sv, uint32_t n, uint32_t head, uint32_t grp,
                                           uint32_t tid, float sum, uint32_t &par) {
    const uint32_t FULL = 0xFFFFFFFFu, lane = tid & 31u, warp = tid >> 5;
    auto one_thread = [&](uint32_t pos, uint32_t end) {
        par ^= 2u;
        auto &told = g.told[par >> 1];
        if (tid == 0) told.sum = add_in_order(sum, sv, pos, end);
        group_sync(grp);
        sum = told.sum;
    };
    uint32_t pos = n <= head + GS_TAIL && head ? n : min(head, n);
    if (pos) one_thread(0, pos);
    const float4 q = *(const float4 *)(sv + 4u * tid);
    while (pos < n) {
        const uint32_t sb = __float_as_uint(sum), E = sb & 0x7F800000u;
        /* few values; or a negative, zero, subnormal, huge or not finite sum */
        if (n - pos <= GS_TAIL || sb >= 0x7F000000u || E == 0u) {
            one_thread(pos, n);
            return sum;
        }
        const float e0 = __uint_as_float(E), e1 = __uint_as_float(E + 1u);
        float x[4] = {q.x, q.y, q.z, q.w};
        uint32_t a0[4], a1[4];
        bool tie = false, odd = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = 4u * tid + k;
            if (i < pos || i >= n) x[k] = 0.0f;
            odd |= !(x[k] >= 0.0f);
            a0[k] = min(__float_as_uint(__fadd_rn(e0, x[k])) - E, INC_MAX);
            a1[k] = min(__float_as_uint(__fadd_rn(e1, x[k])) - (E + 1u), INC_MAX);
            tie |= a0[k] != a1[k];
        }
        /* this thread's function (t0, t1) and its warp's (w0, w1). Without a tie both are
         * whole numbers, and unless the sum leaves the binade among this warp's values
         * only the total is wanted. */
        uint32_t t0, t1, w0, w1, p0 = 0u, p1 = 0u;
        const bool ties = __any_sync(FULL, tie);
        if (!ties) {
            t0 = t1 = (a0[0] + a0[1]) + (a0[2] + a0[3]);
            w0 = w1 = min(__reduce_add_sync(FULL, t0), INC_MAX); /* 128 increments: at most 2^31 */
        } else {
            t0 = t1 = 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                t0 += (t0 & 1u) ? a1[k] : a0[k];
                t1 += (t1 & 1u) ? a0[k] : a1[k];
            }
            w0 = t0;
            w1 = t1;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y0 = __shfl_up_sync(FULL, w0, d), y1 = __shfl_up_sync(FULL, w1, d);
                if (lane >= (uint32_t)d) { /* first the lower lanes' function, then this one */
                    const uint32_t n0 = y0 + ((y0 & 1u) ? w1 : w0), n1 = y1 + ((y1 & 1u) ? w0 : w1);
                    w0 = min(n0, INC_MAX);
                    w1 = min(n1, INC_MAX);
                }
            }
            p0 = __shfl_up_sync(FULL, w0, 1);
            p1 = __shfl_up_sync(FULL, w1, 1);
            if (lane == 0u) p0 = p1 = 0u;
        }
        if (__any_sync(FULL, odd)) w0 = w1 = ODD_VALUES;
        par ^= 1u;
        uint2 *const total = g.total[par & 1u];
        if (lane == 31u) total[warp] = make_uint2(w0, w1);
        group_sync(grp);
        /* ulps past the binade's first float: now, before this warp, after all warps */
        uint32_t m = sb - E, before = 0u;
        bool odd_values = false;
#pragma unroll
        for (uint32_t w = 0; w < GS_WARPS; ++w) {
            const uint2 t = total[w];
            if (w == warp) before = m;
            odd_values |= t.x == ODD_VALUES;
            m = min(m + ((m & 1u) ? t.y : t.x), INC_MAX);
        }
        if (odd_values) {
            one_thread(pos, n);
            return sum;
        }
        if (m < BINADE) { /* the sum stays in its binade: every thread has it */
            sum = __uint_as_float(E + m);
            return sum;
        }
        par ^= 2u;
        auto &told = g.told[par >> 1];
        const uint32_t through = before + ((before & 1u) ? w1 : w0); /* (lane 31's is the warp's) */
        if (before < BINADE && __shfl_sync(FULL, through, 31) >= BINADE) { /* it leaves it among this warp's values */
            if (!ties) {
                uint32_t incl = t0;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, incl, d);
                    if (lane >= (uint32_t)d) incl += y;
                }
                p0 = p1 = incl - t0;
            }
            uint32_t at = before + ((before & 1u) ? p1 : p0);
            if (at < BINADE && at + ((at & 1u) ? t1 : t0) >= BINADE) { /* this thread's */
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t next = at + ((at & 1u) ? a1[k] : a0[k]);
                    if (at < BINADE && next >= BINADE) {
                        told.sum = __fadd_rn(__uint_as_float(E + at), x[k]);
                        told.pos = 4u * tid + k + 1u;
                    }
                    at = next;
                }
            }
        }
        group_sync(grp);
        sum = told.sum;
        pos = told.pos;
    }
    return sum;
}

struct GsArgs {
    const uint32_t *order;
    const uint4 *off; /* per level: first vertex of the thread, warp and block class, end */
    uint32_t nlev;
    const uint32_t *rowptr, *col, *outdeg;
    const float *pr_old;
    float *pr_new, *val, *delta;
    const int *done;
    uint32_t *bar; /* arrivals at the grid barrier, counted up over the call */
    uint32_t meets; /* arrivals before this sweep */
    int *err;
    long long spin_limit;
    double reset, damping;
};

/* polls of the grid barrier: seconds */
constexpr long long GS_SPIN = 1ll << 23;

/* the grid barrier in two halves, so that what follows need not wait for static loads:
 * every CTA arrives; then waits, false when the (bounded) wait ran out here or in
 * another CTA */
__device__ __forceinline__ void gs_arrive(const GsArgs &a) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
}
__device__ __forceinline__ bool gs_wait(const GsArgs &a, uint32_t target) {
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        int ok = 1;
        for (long long spins = 0;; ++spins) {
            uint32_t seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
            if ((int32_t)(seen - target) >= 0) break;
            if ((spins & 255) == 255 && *(volatile int *)a.err) ok = 0;
            if (spins > a.spin_limit) {
                atomicExch(a.err, 1);
                ok = 0;
            }
            if (!ok) break;
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

/* One sweep: the levels in order, a grid barrier between them (one cooperative
 * launch, one CTA per SM). A level's vertices are independent. A block-class vertex
 * is taken by a group of 256 threads: the threads copy the in-edge values of a step
 * into shared memory, GS_DEPTH - 1 steps ahead, and group_add adds a step. A
 * warp-class vertex by a warp: 256 values in flight, then added in order from
 * shuffles (or shared memory, GS_FEW_ROUNDS). A thread-class vertex by a thread, eight
 * loads in flight, then the adds. Block-class vertices go to the CTAs from the first on,
 * the others from the last warp down, so that a small level's rows lie on different SMs. What does not change within a sweep (a level's vertices, row bounds
 * and first columns) is loaded while the CTA waits for the others. */
template <bool EDGE, bool TRACK>
__global__ void __launch_bounds__(GS_THREADS, 1) k_gs_sweep(GsArgs a) {
    if (TRACK && *(volatile const int *)a.done) return; /* sweeps queued after the tolerance was met */
    extern __shared__ __align__(16) unsigned char s_raw[];
    const uint32_t grp = threadIdx.x / GS_GROUP, tid = threadIdx.x % GS_GROUP, lane = threadIdx.x & 31u;
    GsGroup &g = ((GsGroup *)s_raw)[grp];
    const uint32_t ngroups = gridDim.x * GS_GROUPS, nwarps = gridDim.x * (GS_THREADS / 32u);
    const uint32_t gid = grp * gridDim.x + blockIdx.x;
    const uint32_t rev = nwarps - 1u - ((threadIdx.x >> 5) * gridDim.x + blockIdx.x); /* warps from the last down */
    const float *pr_old = a.pr_old;
    float *pr_new = a.pr_new;
    uint32_t par = 0;

    constexpr uint32_t GQ = GS_STEP / GS_GROUP;
    auto value = [&](uint32_t u, uint32_t v) { return __ldcg((u < v ? pr_new : pr_old) + u); };
    auto columns = [&](uint32_t jb, uint32_t je, uint32_t b, uint32_t *u) {
#pragma unroll
        for (uint32_t q = 0; q < GQ; ++q) {
            const uint64_t j = (uint64_t)jb + (uint64_t)b * GS_STEP + q * GS_GROUP + tid;
            u[q] = j < je ? __ldg(a.col + j) : 0u;
        }
    };

    auto row_columns = [&](uint32_t jb, uint32_t je, uint32_t *u) { /* a warp-class row, 32 at a time */
#pragma unroll
        for (uint32_t q = 0; q < GS_WARP_MAX / 32; ++q) {
            const uint64_t j = (uint64_t)jb + 32u * q + lane;
            u[q] = j < je ? __ldg(a.col + j) : 0u;
        }
    };

    /* the first vertex that this warp takes in a level: its id, row and first columns */
    uint32_t pv = 0, pjb = 0, pje = 0, pod = 0, pc[8];
    auto prefetch = [&](uint4 o) {
        const uint32_t nb = o.w - o.z, nw = o.z - o.y, nt = o.y - o.x;
        uint32_t i = 0xFFFFFFFFu;
        if (gid < nb) i = o.z + gid;
        else if (rev < nw) i = o.y + rev;
        else if ((uint64_t)(rev - nw) * 32u + lane < nt) i = o.x + (rev - nw) * 32u + lane;
        pv = pjb = pje = 0;
        if (i != 0xFFFFFFFFu) {
            pv = __ldg(a.order + i);
            pjb = __ldg(a.rowptr + pv);
            pje = __ldg(a.rowptr + pv + 1);
            pod = __ldg(a.outdeg + pv);
        }
        if (gid < nb) {
            columns(pjb, pje, 0, pc);
            columns(pjb, pje, 1, pc + 4);
        } else if (rev < nw) {
            row_columns(pjb, pje, pc);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) pc[k] = pjb + k < pje ? __ldg(a.col + pjb + k) : 0u;
        }
    };

    /* one row of many by this warp: the values through shared memory, then every lane adds them in
     * order. pc: its first columns, then those of the warp's next row [njb, nje) */
    float *const wv = (float *)(s_raw + GS_GROUPS * sizeof(GsGroup)) + (threadIdx.x >> 5) * GS_WARP_MAX;
    auto warp_row = [&](uint32_t v, uint32_t jb, uint32_t je, uint32_t od, uint32_t njb, uint32_t nje) {
        float sum = 0.0f;
        for (uint32_t left = je - jb;;) {
            const uint32_t n = min(left, GS_WARP_MAX);
            float x[GS_WARP_MAX / 32];
#pragma unroll
            for (uint32_t q = 0; q < GS_WARP_MAX / 32; ++q) x[q] = 32u * q + lane < n ? value(pc[q], v) : 0.0f;
            left -= n;
            row_columns(left ? je - left : njb, left ? je : nje, pc);
#pragma unroll
            for (uint32_t q = 0; q < GS_WARP_MAX / 32; ++q)
                if (32u * q < n) wv[32u * q + lane] = x[q];
            __syncwarp();
            sum = add_in_order(sum, wv, 0u, n);
            __syncwarp();
            if (!left) break;
        }
        if (lane == 0) gs_apply<EDGE, TRACK>(v, sum, od, pr_new, a.val, a.delta, a.reset, a.damping);
    };

    uint4 o = a.off[0], on = a.nlev > 1 ? a.off[1] : o;
    prefetch(o);
    uint32_t target = a.meets;
    for (uint32_t l = 0; l < a.nlev; ++l) {
        const uint32_t nb = o.w - o.z, nw = o.z - o.y, nt = o.y - o.x;
        bool ready = true; /* the prefetched vertex is the next one */
        for (uint32_t k = gid; k < nb; k += ngroups) { /* block class */
            uint32_t v = pv, jb = pjb, je = pje, od = pod, c0[GQ], c1[GQ];
            if (!ready) {
                v = __ldg(a.order + o.z + k);
                jb = __ldg(a.rowptr + v);
                je = __ldg(a.rowptr + v + 1);
                od = __ldg(a.outdeg + v);
                columns(jb, je, 0, pc);
                columns(jb, je, 1, pc + 4);
            }
            ready = false;
#pragma unroll
            for (uint32_t q = 0; q < GQ; ++q) {
                c0[q] = pc[q];
                c1[q] = pc[4 + q];
            }
            const uint32_t nstep = (je - jb + GS_STEP - 1) / GS_STEP;
            auto issue = [&](uint32_t b) { /* c0 holds step b's columns; one commit group per step */
#pragma unroll
                for (uint32_t q = 0; q < GQ; ++q)
                    if ((uint64_t)jb + (uint64_t)b * GS_STEP + q * GS_GROUP + tid < je)
                        cp_async4(&g.val[b % GS_DEPTH][q * GS_GROUP + tid], (c0[q] < v ? pr_new : pr_old) + c0[q]);
                cp_async_commit();
#pragma unroll
                for (uint32_t q = 0; q < GQ; ++q) c0[q] = c1[q];
                columns(jb, je, b + 2, c1);
            };
            float sum = 0.0f;
            issue(0);
            issue(1);
            for (uint32_t b = 0; b < nstep; ++b) {
                cp_async_wait<1>(); /* this thread's values of step b have landed */
                group_sync(grp);    /* everyone's; step b - 1 is added */
                issue(b + 2);       /* into step b - 1's buffer */
                sum = group_add(g, g.val[b % GS_DEPTH], min(GS_STEP, je - (jb + b * GS_STEP)), b ? 0u : GS_HEAD, grp,
                                tid, sum, par);
            }
            cp_async_wait<0>(); /* no copy in flight when the buffers are used again */
            if (tid == 0) gs_apply<EDGE, TRACK>(v, sum, od, pr_new, a.val, a.delta, a.reset, a.damping);
            group_sync(grp);
        }
        uint32_t kw = rev; /* warp class */
        for (; kw < nw && nw <= GS_FEW_ROUNDS * nwarps; kw += nwarps) {
            uint32_t v = pv, jb = pjb, je = pje, od = pod;
            if (!ready) {
                v = __ldg(a.order + o.y + kw);
                jb = __ldg(a.rowptr + v);
                je = __ldg(a.rowptr + v + 1);
                od = __ldg(a.outdeg + v);
                row_columns(jb, je, pc);
            }
            ready = false;
            float x[GS_WARP_MAX / 32], sum = 0.0f;
            for (uint32_t left = je - jb;;) {
#pragma unroll
                for (uint32_t q = 0; q < GS_WARP_MAX / 32; ++q) x[q] = 32u * q + lane < left ? value(pc[q], v) : 0.0f;
                const bool more = left > GS_WARP_MAX;
                if (more) row_columns(je - left + GS_WARP_MAX, je, pc);
#pragma unroll
                for (uint32_t q = 0; q < GS_WARP_MAX / 32; ++q) {
                    const uint32_t n = left > 32u * q ? left - 32u * q : 0u;
                    if (n == 0u) break;
#pragma unroll
                    for (uint32_t i = 0; i < 32u; ++i) { /* in order, in every lane */
                        const float z = __shfl_sync(0xFFFFFFFFu, x[q], (int)i);
                        if (i < n) sum += z;
                    }
                }
                if (!more) break;
                left -= GS_WARP_MAX;
            }
            if (lane == 0) gs_apply<EDGE, TRACK>(v, sum, od, pr_new, a.val, a.delta, a.reset, a.damping);
        }
        for (; kw < nw; kw += 32u * nwarps) { /* a lane loads what the warp needs of one row in 32 */
            uint32_t v = 0, jb = 0, je = 0, od = 0;
            if (kw + (uint64_t)lane * nwarps < nw) {
                v = __ldg(a.order + o.y + kw + lane * nwarps);
                jb = __ldg(a.rowptr + v);
                je = __ldg(a.rowptr + v + 1);
                od = __ldg(a.outdeg + v);
            }
            ready = false;
            row_columns(__shfl_sync(0xFFFFFFFFu, jb, 0), __shfl_sync(0xFFFFFFFFu, je, 0), pc);
            for (uint32_t r = 0; r < 32u && kw + r * nwarps < nw; ++r) {
                const uint32_t njb = __shfl_sync(0xFFFFFFFFu, jb, (int)r + 1), nje = __shfl_sync(0xFFFFFFFFu, je, (int)r + 1);
                warp_row(__shfl_sync(0xFFFFFFFFu, v, (int)r), __shfl_sync(0xFFFFFFFFu, jb, (int)r),
                         __shfl_sync(0xFFFFFFFFu, je, (int)r), __shfl_sync(0xFFFFFFFFu, od, (int)r),
                         r < 31u ? njb : 0u, r < 31u ? nje : 0u);
            }
        }
        /* thread class: warps past those of the warp class first */
        for (uint64_t k = (uint64_t)(rev >= nw % nwarps ? rev - nw % nwarps : rev + nwarps - nw % nwarps) * 32u + lane;
             k < nt; k += (uint64_t)nwarps * 32u) {
            uint32_t v = pv, jb = pjb, je = pje, od = pod;
            const bool have = ready && rev >= nw;
            if (!have) {
                v = __ldg(a.order + o.x + k);
                jb = __ldg(a.rowptr + v);
                je = __ldg(a.rowptr + v + 1);
                od = __ldg(a.outdeg + v);
            }
            float sum = 0.0f;
            if (!have) {
#pragma unroll
                for (uint32_t i = 0; i < GS_THREAD_MAX; ++i) pc[i] = jb + i < je ? __ldg(a.col + jb + i) : 0u;
            }
            for (uint32_t j = jb; j < je; j += GS_THREAD_MAX) { /* the next columns with these values in flight */
                float x[GS_THREAD_MAX];
#pragma unroll
                for (uint32_t i = 0; i < GS_THREAD_MAX; ++i) x[i] = j + i < je ? value(pc[i], v) : 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < GS_THREAD_MAX; ++i)
                    if (j + GS_THREAD_MAX + i < je) pc[i] = __ldg(a.col + j + GS_THREAD_MAX + i);
#pragma unroll
                for (uint32_t i = 0; i < GS_THREAD_MAX; ++i)
                    if (j + i < je) sum += x[i];
            }
            ready = false;
            gs_apply<EDGE, TRACK>(v, sum, od, pr_new, a.val, a.delta, a.reset, a.damping);
        }
        if (l + 1 == a.nlev) break;
        gs_arrive(a);
        o = on;
        if (l + 2 < a.nlev) on = a.off[l + 2];
        prefetch(o);
        target += gridDim.x;
        if (!gs_wait(a, target)) return;
    }
}

/* The sweep's sums of delta[] and |val[]|: each block adds a fixed slice in
 * FP64, the last block to finish adds the block sums in block order, logs
 * delta_log[k] = sum delta and res_log[k] = sum delta / sum |val| for the k-th
 * sweep (k = *slot, then advanced) and raises *done when the residual is <= tol. */
constexpr int DSUM_BLOCKS = 256;
__global__ void __launch_bounds__(256) k_gs_delta_sum(const float *__restrict__ delta, const float *__restrict__ val,
                                                      uint32_t nv, double2 *part, uint32_t *ticket, uint32_t *slot,
                                                      int *done, double tol, double *delta_log, double *res_log) {
    if (*(volatile const int *)done) return;
    __shared__ double2 s[8];
    __shared__ int s_last;
    const uint32_t per = (nv + gridDim.x - 1) / gridDim.x;
    const uint32_t b0 = blockIdx.x * per, b1 = min(nv, b0 + per);
    double x = 0.0, y = 0.0;
    for (uint32_t v = b0 + threadIdx.x; v < b1; v += blockDim.x) {
        x += (double)delta[v];
        y += fabs((double)val[v]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_down_sync(0xFFFFFFFFu, x, o);
        y += __shfl_down_sync(0xFFFFFFFFu, y, o);
    }
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = make_double2(x, y);
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 t = make_double2(0.0, 0.0);
        for (int w = 0; w < 8; ++w) {
            t.x += s[w].x;
            t.y += s[w].y;
        }
        part[blockIdx.x] = t;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    double dx = 0.0, ny = 0.0;
    for (uint32_t b = 0; b < gridDim.x; ++b) {
        const double2 p = __ldcg(part + b);
        dx += p.x;
        ny += p.y;
    }
    const uint32_t k = *slot;
    const double res = ny > 0.0 ? dx / ny : 0.0;
    delta_log[k] = dx;
    res_log[k] = res;
    *slot = k + 1;
    if (tol > 0.0 && res <= tol) *done = 1;
    *ticket = 0u;
}

/* the vertex values before the first sweep, for the progress log: the edge-value
 * program's 0.15 (pagerank.cpp:84), the in-memory program's pr * outc = 1 (or
 * 0.15 without out-edges, pagerank.cpp:137-139) */
__global__ void k_gs_val_init(uint32_t nv, const uint32_t *__restrict__ outdeg, float reset, int edge, float *val) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
        val[v] = (edge || outdeg[v] == 0) ? reset : 1.0f;
}

/* pagerank.cpp:140-143: the stored value is pr * outc on the last iteration */
__global__ void k_gs_final(uint32_t nv, const uint32_t *__restrict__ outdeg, const float *__restrict__ pr, float *out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        uint32_t oc = outdeg[v];
        out[v] = oc > 0 ? __fmul_rn(pr[v], (float)oc) : pr[v];
    }
}

inline unsigned vgrid(uint32_t n) {
    uint64_t b = ((uint64_t)n + 255) / 256;
    uint64_t cap = (uint64_t)num_sms() * 16;
    return (unsigned)std::max<uint64_t>(1, std::min(b, cap));
}

}  // namespace

/* Level schedule of the id-ordered dependency DAG: order[] (vertices by
 * (level, class, id)) and where each of the nlev levels' classes lie in it. */
struct GsPlan {
    uint32_t nlev = 0;
    dbuf<uint32_t> order;
    dbuf<uint4> off;
};

void free_gs_plan(GsPlan *p) { delete p; }

static int build_gs_plan(gcg_graph *g, GsPlan &pl) {
    cudaStream_t s = g->stream;
    const uint32_t nv = g->nv;
    tbuf<uint32_t> level, pending, pos, total;
    GCG_TRY(level.alloc(nv, s));
    GCG_TRY(pending.alloc(nv, s));
    GCG_TRY(pos.alloc(nv, s));
    GCG_TRY(total.alloc(1, s));
    GCG_CUDA(cudaMemsetAsync(level.get(), 0, (size_t)nv * 4, s));
    k_gs_pending<<<vgrid(nv), 256, 0, s>>>(g->in_rowptr.get(), g->in_col.get(), nv, pending.get());
    GCG_TRY(scan_u32(pending.get(), pos.get(), nv, total.get(), s));
    uint32_t nfwd = 0;
    GCG_CUDA(cudaMemcpyAsync(&nfwd, total.get(), 4, cudaMemcpyDeviceToHost, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    uint32_t maxl = 0;
    if (nfwd) {
        /* the forward (u < v) edges grouped by source */
        tbuf<uint64_t> keys, tmp;
        tbuf<uint32_t> fwd_off, fwd_dst, front, cnt;
        GCG_TRY(keys.alloc(nfwd, s));
        GCG_TRY(tmp.alloc(nfwd, s));
        GCG_TRY(fwd_off.alloc((size_t)nv + 1, s));
        GCG_TRY(fwd_dst.alloc(nfwd, s));
        GCG_TRY(front.alloc((size_t)2 * nv, s));
        k_gs_fwd_keys<<<vgrid(nv), 256, 0, s>>>(g->in_rowptr.get(), g->in_col.get(), nv, pending.get(), pos.get(),
                                                g->vbits, keys.get());
        uint64_t *sorted = nullptr;
        GCG_TRY(radix_sort_u64(keys.get(), tmp.get(), nfwd, (int)g->vbits, (int)(2 * g->vbits), &sorted, s));
        k_gs_fwd_off<<<vgrid(nfwd), 256, 0, s>>>(sorted, nfwd, g->vbits, nv, fwd_off.get(), fwd_dst.get());
        /* rounds, queued in batches of 64 (empty rounds return at once); the host
         * checks the last frontier count of each batch. A vertex joins a frontier
         * once, so at most nv rounds. */
        const uint32_t CAP = nv + 2;
        GCG_TRY(cnt.alloc(CAP, s));
        GCG_CUDA(cudaMemsetAsync(cnt.get(), 0, (size_t)CAP * 4, s));
        k_gs_roots<<<vgrid(nv), 256, 0, s>>>(pending.get(), nv, front.get(), cnt.get());
        GCG_LAUNCH_CHECK();
        uint32_t r = 0;
        for (;;) {
            const uint32_t nb = std::min<uint32_t>(64, CAP - 2 - r);
            for (uint32_t k = 0; k < nb; ++k, ++r) {
                uint32_t *cur = front.get() + (size_t)(r & 1) * nv, *nxt = front.get() + (size_t)((r + 1) & 1) * nv;
                k_gs_round<<<vgrid(nv), 256, 0, s>>>(r, fwd_off.get(), fwd_dst.get(), pending.get(), level.get(), cur,
                                                     nxt, cnt.get());
            }
            GCG_LAUNCH_CHECK();
            uint32_t last = 0;
            GCG_CUDA(cudaMemcpyAsync(&last, cnt.get() + r, 4, cudaMemcpyDeviceToHost, s));
            GCG_CUDA(cudaStreamSynchronize(s));
            if (last == 0 || r + 2 >= CAP) break;
        }
        /* the deepest non-empty round */
        std::vector<uint32_t> hc(r + 1);
        GCG_CUDA(cudaMemcpyAsync(hc.data(), cnt.get(), (size_t)(r + 1) * 4, cudaMemcpyDeviceToHost, s));
        GCG_CUDA(cudaStreamSynchronize(s));
        uint64_t placed = 0;
        for (uint32_t k = 0; k <= r; ++k) {
            placed += hc[k];
            if (hc[k]) maxl = k;
        }
        if (placed != nv) return fail(GCG_ERR_CUDA, "level schedule: a vertex was not reached");
    }
    pl.nlev = maxl + 1;
    uint32_t lbits = 1;
    while (lbits < 32 && (1ull << lbits) <= maxl) ++lbits;
    if (g->vbits + 2 + lbits > 64) return fail(GCG_ERR_UNSUPPORTED, "level schedule: too many levels");
    tbuf<uint64_t> keys, tmp;
    GCG_TRY(keys.alloc(nv, s));
    GCG_TRY(tmp.alloc(nv, s));
    tbuf<uint32_t> mid, seg;
    GCG_TRY(mid.alloc(2 * (size_t)pl.nlev, s));
    GCG_CUDA(cudaMemsetAsync(mid.get(), 0, (size_t)pl.nlev * 8, s));
    k_level_mid<<<vgrid(nv), 256, 0, s>>>(level.get(), g->in_rowptr.get(), nv, mid.get());
    k_level_keys<<<vgrid(nv), 256, 0, s>>>(level.get(), g->in_rowptr.get(), nv, mid.get(),
                                           (uint32_t)num_sms() * (GS_THREADS / 32), g->vbits, keys.get());
    uint64_t *sorted = nullptr;
    GCG_TRY(radix_sort_u64(keys.get(), tmp.get(), nv, (int)g->vbits, (int)(g->vbits + 2 + lbits), &sorted, s));
    const size_t nseg = (size_t)GS_CLASSES * pl.nlev;
    GCG_TRY(seg.alloc(nseg + 1, s));
    GCG_CUDA(cudaMemsetAsync(seg.get(), 0, (nseg + 1) * 4, s));
    GCG_TRY(pl.off.alloc(pl.nlev));
    GCG_TRY(pl.order.alloc(nv));
    k_level_bounds<<<vgrid(nv), 256, 0, s>>>(sorted, nv, g->vbits, (uint32_t)nseg, seg.get(), pl.order.get());
    k_level_pack<<<vgrid(pl.nlev), 256, 0, s>>>(seg.get(), pl.nlev, pl.off.get());
    GCG_LAUNCH_CHECK();
    GCG_CUDA(cudaStreamSynchronize(s));
    return GCG_OK;
}

/* GCG_PR_GS_EXACT (in-memory program) and GCG_PR_GS_EDGE (edge-value program).
 * With tol > 0, residuals or delta_log (always for GS_EDGE) every sweep also
 * tracks the vertices' pageranks: delta_log gets sum |pagerank - previous| and
 * residuals that sum over sum |pagerank| (the Jacobi residual's definition); the
 * run stops after the first sweep whose residual is <= tol. */
int pagerank_gs_exact(gcg_graph *g, const gcg_pr_params *p, float *out_rank, gcg_pr_stats *stats) {
    cudaStream_t s = g->stream;
    const uint32_t nv = g->nv;
    const bool edge = p->mode == GCG_PR_GS_EDGE;
    const bool track = edge || p->tol > 0.0 || p->residuals || p->delta_log;
    if (!g->gsplan) { /* built once per graph, dropped when its edges change */
        GsPlan *np = new GsPlan();
        const int st = build_gs_plan(g, *np);
        if (st != GCG_OK) {
            delete np;
            return st;
        }
        g->gsplan = np;
    }
    const GsPlan &pl = *g->gsplan;
    const int nsw = p->max_sweeps;
    tbuf<float> pr, val, delta;
    tbuf<double> logs; /* delta_log[nsw], res_log[nsw] */
    tbuf<double2> part;
    tbuf<uint32_t> ctl; /* ticket, slot, done, error, barrier arrivals */
    GCG_TRY(pr.alloc((size_t)2 * nv, s));
    GCG_TRY(ctl.alloc(8, s));
    GCG_CUDA(cudaMemsetAsync(ctl.get(), 0, 8 * sizeof(uint32_t), s));
    int *done = (int *)(ctl.get() + 2);
    float *const buf[2] = {pr.get(), pr.get() + nv}; /* sweep k reads buf[k & 1], writes the other */
    const float reset = (float)p->teleport;
    if (track) {
        GCG_TRY(val.alloc(nv, s));
        GCG_TRY(delta.alloc(nv, s));
        GCG_TRY(logs.alloc(2 * (size_t)std::max(1, nsw), s));
        GCG_TRY(part.alloc(DSUM_BLOCKS, s));
        k_gs_val_init<<<vgrid(nv), 256, 0, s>>>(nv, g->outdeg.get(), reset, edge ? 1 : 0, val.get());
    }
    if (edge) k_gs_edge_init<<<vgrid(nv), 256, 0, s>>>(nv, g->outdeg.get(), buf[0]);
    else k_gs_init<<<vgrid(nv), 256, 0, s>>>(nv, g->outdeg.get(), reset, buf[0]);
    GCG_LAUNCH_CHECK();

    EventPair ev;
    GCG_TRY(ev.create());
    GsArgs a{};
    a.order = pl.order.get();
    a.off = pl.off.get();
    a.nlev = pl.nlev;
    a.rowptr = g->in_rowptr.get();
    a.col = g->in_col.get();
    a.outdeg = g->outdeg.get();
    a.val = val.get();
    a.delta = delta.get();
    a.done = done;
    a.err = (int *)(ctl.get() + 3);
    a.bar = ctl.get() + 4;
    a.spin_limit = GS_SPIN;
    if (p->flags & GCG_PR_TEST_BARRIER_TIMEOUT) { /* one arrival short */
        a.spin_limit = GCG_TEST_SPIN;
        GCG_CUDA(cudaMemsetAsync(a.bar, 0xFF, 4, s));
    }
    a.reset = p->teleport;
    a.damping = p->damping;
    const void *kern = edge    ? (const void *)k_gs_sweep<true, true>
                       : track ? (const void *)k_gs_sweep<false, true>
                               : (const void *)k_gs_sweep<false, false>;
    const size_t smem = sizeof(GsGroup) * GS_GROUPS + (size_t)(GS_THREADS / 32) * GS_WARP_MAX * sizeof(float);
    GCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    unsigned grid = (unsigned)num_sms();
    int queued = 0;
    /* one cooperative launch per sweep; where fewer SMs are to be had, a smaller grid */
    auto launch_sweep = [&]() -> int {
        a.pr_old = buf[queued & 1];
        a.pr_new = buf[(queued + 1) & 1];
        void *kargs[] = {&a};
        cudaError_t e;
        for (;;) {
            a.meets = (uint32_t)queued * (pl.nlev - 1) * grid;
            e = cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(GS_THREADS), kargs, smem, s);
            if (e != cudaErrorCooperativeLaunchTooLarge || queued || grid == 1) break;
            cudaGetLastError();
            grid = (grid + 1) / 2;
        }
        GCG_CUDA(e);
        if (track)
            k_gs_delta_sum<<<DSUM_BLOCKS, 256, 0, s>>>(delta.get(), val.get(), nv, part.get(), ctl.get(),
                                                       ctl.get() + 1, done, p->tol, logs.get(),
                                                       logs.get() + std::max(1, nsw));
        ++queued;
        return GCG_OK;
    };
    /* sweeps are queued in chunks of 8; with a tolerance the host checks the
     * sweep count after each chunk (sweeps queued past convergence return at once) */
    uint32_t h_ctl[4] = {0, 0, 0, 0};
    GCG_CUDA(cudaEventRecord(ev.first, s));
    for (int sw = 0; sw < nsw;) {
        const int n = std::min(8, nsw - sw);
        for (int k = 0; k < n; ++k) GCG_TRY(launch_sweep());
        sw += n;
        if (p->tol > 0.0 && sw < nsw) {
            GCG_CUDA(cudaMemcpyAsync(h_ctl, ctl.get(), sizeof(h_ctl), cudaMemcpyDeviceToHost, s));
            GCG_CUDA(cudaStreamSynchronize(s));
            if (h_ctl[2]) break;
        }
    }
    GCG_CUDA(cudaEventRecord(ev.last, s));
    GCG_CUDA(cudaMemcpyAsync(h_ctl, ctl.get(), sizeof(h_ctl), cudaMemcpyDeviceToHost, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    if (h_ctl[3]) return fail(GCG_ERR_TIMEOUT, "pagerank: a wait between the levels of a sweep ran out");
    const int sweeps = track ? (int)h_ctl[1] : nsw;
    float *const pr_last = buf[sweeps & 1], *const pr_out = buf[(sweeps + 1) & 1];
    if (!edge) {
        k_gs_final<<<vgrid(nv), 256, 0, s>>>(nv, g->outdeg.get(), pr_last, pr_out);
        GCG_LAUNCH_CHECK();
    }
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev.first, ev.last);
    double last_res = 0.0;
    if (track && sweeps > 0)
        GCG_CUDA(cudaMemcpy(&last_res, logs.get() + std::max(1, nsw) + sweeps - 1, sizeof(double),
                            cudaMemcpyDeviceToHost));
    if (out_rank) GCG_TRY(copy_out(out_rank, edge ? val.get() : pr_out, (size_t)nv * 4, s));
    if (track && p->delta_log && sweeps > 0)
        GCG_TRY(copy_out(p->delta_log, logs.get(), (size_t)sweeps * sizeof(double), s));
    if (track && p->residuals && sweeps > 0)
        GCG_TRY(copy_out(p->residuals, logs.get() + std::max(1, nsw), (size_t)sweeps * sizeof(double), s));
    if (p->work_log && sweeps > 0) { /* every vertex updated per sweep; its in-edges (+ out-edges with edge values) */
        std::vector<uint64_t> wl(2 * (size_t)sweeps);
        for (int i = 0; i < sweeps; ++i) {
            wl[2 * i] = (uint64_t)nv * (uint64_t)(i + 1);
            wl[2 * i + 1] = (edge ? 2 : 1) * g->ne * (uint64_t)(i + 1);
        }
        GCG_TRY(copy_out(p->work_log, wl.data(), wl.size() * sizeof(uint64_t), s));
    }
    GCG_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        stats->sweeps = sweeps;
        stats->converged = (int)h_ctl[2];
        stats->residual = last_res;
        stats->device_ms = ms;
        stats->sweep_kernel_ms = ms;
        stats->timed_sweeps = sweeps;
        stats->kernel_launches = 1 + (track ? 1 : 0) + (edge ? 0 : 1) + (track ? 2 : 1) * queued;
        stats->levels = (int)pl.nlev;
    }
    return GCG_OK;
}

}  // namespace gcg
