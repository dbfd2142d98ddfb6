/*
 * Triangle counting: replaces order_by_degree + the dynamic-graph engine running
 * TriangleCountingProgram + sum_vertices / 3
 * (src/preprocessing/util/orderbydegree.hpp:59-143,
 *  example_apps/trianglecounting.cpp:95-357, :476-477).
 *
 * Device form:
 *   1. rank vertices by (in+out degree, id) ascending with one radix sort
 *      (orderbydegree.hpp:16-25, 71-89): vertexmap[v] = rank.
 *   2. orient every edge from the lower to the higher rank, radix sort and
 *      deduplicate (reciprocal edges collapse, like the reference's lastvid
 *      checks, trianglecounting.cpp:182,309) -> CSR of higher-ranked neighbours,
 *      each list ascending.
 *   3. group the edges (a, b) by b; a warp lays out N+(b) as bits in shared memory
 *      and streams the rest of N+(a) behind b past them for each of b's edges. A match
 *      c is a triangle (a,b,c): c's count is bumped per match, a's and b's by the match
 *      totals (counts of the top-ranked vertices gathered in shared memory first) — the
 *      per-rank incident-triangle counts of <base>_degord.4B.vout. Where lists are short
 *      (TC_SHORT) the edges are not grouped; the shorter list is searched in the longer.
 */
#include <algorithm>

#include "gcg_internal.cuh"
#include "gcg_mergepath.cuh"

namespace gcg {
namespace {

inline unsigned vgrid(uint64_t n) {
    uint64_t b = (n + 255) / 256;
    uint64_t cap = (uint64_t)num_sms() * 16;
    return (unsigned)std::max<uint64_t>(1, std::min(b, cap));
}

/* of the in + out degrees */
struct DegreeStat {
    double squares; /* their sum */
    uint32_t most;
};

__global__ void __launch_bounds__(256) k_degree_keys(const uint32_t *__restrict__ indeg, const uint32_t *__restrict__ outdeg, uint32_t nv,
                              uint32_t vbits, uint64_t *__restrict__ keys, DegreeStat *stat) {
    __shared__ uint32_t s_m[8];
    __shared__ double s_s[8];
    uint32_t m = 0;
    double sq = 0.0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        uint64_t d = (uint64_t)indeg[v] + outdeg[v];
        keys[v] = (d << vbits) | v;
        m = max(m, d > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)d);
        sq += (double)d * (double)d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_down_sync(0xFFFFFFFFu, m, o));
        sq += __shfl_down_sync(0xFFFFFFFFu, sq, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_m[threadIdx.x >> 5] = m;
        s_s[threadIdx.x >> 5] = sq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            m = max(m, s_m[w]);
            sq += s_s[w];
        }
        atomicMax(&stat->most, m);
        atomicAdd(&stat->squares, sq);
    }
}

__global__ void k_rank_scatter(const uint64_t *__restrict__ sorted, uint32_t nv, uint32_t vbits,
                               uint32_t *__restrict__ rank) {
    const uint64_t mask = (1ull << vbits) - 1ull;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x)
        rank[(uint32_t)(sorted[i] & mask)] = i;
}

/* key of edge e (row v, source u): (min rank << vbits) | max rank */
__global__ void __launch_bounds__(MP_THREADS) k_orient_keys(const uint32_t *__restrict__ rowptr,
                                                            const uint32_t *__restrict__ col,
                                                            const uint32_t *__restrict__ tile_row,
                                                            const uint32_t *__restrict__ tile_edge, uint32_t ntiles,
                                                            const uint32_t *__restrict__ rank, uint32_t vbits, int half,
                                                            uint32_t *__restrict__ count, uint64_t *__restrict__ keys) {
    __shared__ uint32_t s_rowend[MP_TILE];
    __shared__ uint32_t s_wsum[MP_THREADS / 32];
    __shared__ uint32_t s_base;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t r0 = tile_row[t], r1 = tile_row[t + 1];
        const uint32_t e0 = tile_edge[t], e1 = tile_edge[t + 1];
        const uint32_t nrows = r1 - r0, nedges = e1 - e0;
        for (uint32_t k = threadIdx.x; k < nrows; k += MP_THREADS) s_rowend[k] = rowptr[r0 + k + 1] - e0;
        __syncthreads();
        const uint32_t items = nrows + nedges;
        const uint32_t d0 = min((uint32_t)threadIdx.x * MP_ITEMS, items);
        const uint32_t d1 = min(d0 + MP_ITEMS, items);
        const uint32_t ti0 = mp_search(s_rowend, nrows, nedges, d0);
        if (!half) {
            uint32_t ti = ti0, tj = d0 - ti0;
            for (uint32_t d = d0; d < d1; ++d) {
                if (ti < nrows && s_rowend[ti] <= tj) {
                    ++ti;
                } else {
                    uint64_t a = rank[__ldg(col + e0 + tj)], b = rank[r0 + ti];
                    keys[e0 + tj] = a < b ? ((a << vbits) | b) : ((b << vbits) | a);
                    ++tj;
                }
            }
        } else {
            /* symmetric graph: every edge is stored both ways and both give the
             * same key, so only the copy in the higher-ranked endpoint's row is
             * kept, compacted: count, block prefix sum, one global claim per
             * tile, write (the sort that follows fixes the order) */
            uint32_t kept = 0;
            {
                uint32_t ti = ti0, tj = d0 - ti0;
                for (uint32_t d = d0; d < d1; ++d) {
                    if (ti < nrows && s_rowend[ti] <= tj) {
                        ++ti;
                    } else {
                        kept += rank[__ldg(col + e0 + tj)] <= rank[r0 + ti];
                        ++tj;
                    }
                }
            }
            uint32_t incl = kept;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            if (lane == 31) s_wsum[w] = incl;
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t run = 0;
                for (uint32_t k = 0; k < MP_THREADS / 32; ++k) {
                    const uint32_t x = s_wsum[k];
                    s_wsum[k] = run;
                    run += x;
                }
                s_base = run ? atomicAdd(count, run) : 0u;
            }
            __syncthreads();
            uint64_t pos = (uint64_t)s_base + s_wsum[w] + (incl - kept);
            uint32_t ti = ti0, tj = d0 - ti0;
            for (uint32_t d = d0; d < d1; ++d) {
                if (ti < nrows && s_rowend[ti] <= tj) {
                    ++ti;
                } else {
                    const uint64_t a = rank[__ldg(col + e0 + tj)], b = rank[r0 + ti];
                    if (a <= b) keys[pos++] = (a << vbits) | b;
                    ++tj;
                }
            }
        }
        __syncthreads();
    }
}

/* ---- counting ---------------------------------------------------------------
 * Every triangle a < b < c (ranks) is found at its edge (a, b): c is in N+(a) after b
 * and in N+(b). The edges are taken grouped by b, so that N+(b) is laid out once, as
 * bits, and each edge only streams the rest of N+(a) past it: one coalesced load and one
 * shared-memory bit per candidate, sum over edges of |N+(a) after b| of them. Searching
 * the shorter list in the longer took that many searches of log2 steps, each a dependent
 * uncoalesced load (R-MAT scale 20: 1.2 G candidates against 10.6 G search steps; the
 * counting 9.4 -> 2.7 ms with 0.36 ms for the grouping, the whole call 11.0 -> 4.8, scale
 * 22 62 -> 26 ms). What bounds it is instruction issue, ~50 per 32 candidates.
 *
 * Ranks grow with degree, so nearly every candidate is among the top ranks (scale 20:
 * 99.1 % among 16,384): those have a bit each, indexed from the top rank down. For the
 * elements of N+(b) below them a filter of TC_FILTER hashed bits says no to nearly all
 * candidates; the few that pass are searched in N+(b). */
constexpr uint32_t TC_WARPS = 32;      /* one 1024-thread block per SM */
constexpr uint32_t TC_TOP = 16384;     /* top ranks with a bit (per warp) and a shared counter (per block) each */
constexpr uint32_t TC_FILTER = 4096;   /* bits */
constexpr int TC_WINDOWS = 4;          /* loads of 32 candidates in flight per warp */
constexpr uint32_t TC_TASK_MIN = 32, TC_TASK_MAX = 256; /* edges of one b that a warp takes at a time */
constexpr uint32_t TC_WARP_WORDS = (TC_TOP + TC_FILTER) / 32 + 64; /* bits, filter, 32 lists' places and hits */
/* Where the degrees are alike (an edge's end has less than TC_FLAT times the mean degree) the
 * top ranks hold few of the candidates, and N+(b)'s elements below them may be many: from
 * TC_PAIRS on, where the filter lets many candidates through, they are searched two at a
 * time (uniform, 200 K vertices of degree 2,000: 1,078 -> 932 ms, of 500: 50.4 -> 48.1). In a
 * kernel of its own: the same code costs R-MAT scale 20 1.6 %. */
constexpr double TC_FLAT = 4.0;
constexpr uint32_t TC_PAIRS = 32;
/* Below this many neighbours of an edge's end, on average over the edges, grouping the edges
 * costs more than it saves, and the shorter list is searched in the longer, edge by edge
 * (k_tc_search). Uniform graphs, grouped and searched: 4 M vertices of degree 16 6.43 and
 * 4.69 ms, 48 20.0 and 16.7; 128 K of 64 1.06 and 1.05; 200 K of 100 2.49 and 2.79; 16 K of
 * 64 0.376 and 0.353; 1 M in communities of 50 2.11 and 1.62. R-MAT graphs of more than a few
 * edges a vertex are above it (scale 14 with 4: 143, scale 20 with 1: 217). */
constexpr double TC_SHORT = 96.0;
constexpr size_t TC_SMEM = ((size_t)TC_TOP + TC_WARPS * TC_WARP_WORDS) * 4;

/* Edges with candidates (b is not the last of N+(a)) grouped by b, in two passes over
 * the sorted keys: FILL false counts them per b (at[b]), FILL true writes the lists,
 * rev[..] = (position of b in cl, a), from their starts at[b] on, which it moves to their
 * ends. A block takes a contiguous share of the edges and counts those of the top ranks
 * in shared memory first, so that a hot b costs one global atomic per block and pass
 * (straight global atomics: 584 us a pass at R-MAT scale 20). The order within a list
 * does not matter, every count is a sum of whole numbers. */
template <bool FILL>
__global__ void __launch_bounds__(1024, 1) k_tc_group(const uint64_t *__restrict__ keys, uint64_t m, uint32_t vbits,
                                                      const uint32_t *__restrict__ rp, uint32_t nv, uint32_t top,
                                                      uint32_t *__restrict__ at, uint32_t *__restrict__ part,
                                                      uint2 *__restrict__ rev) {
    extern __shared__ uint32_t s_cnt[]; /* rank nv - 1 - r at r */
    const uint64_t mask = (1ull << vbits) - 1ull;
    const uint64_t per = (m + gridDim.x - 1) / gridDim.x;
    const uint64_t j0 = blockIdx.x * per, j1 = j0 + per < m ? j0 + per : m;
    auto each = [&](auto f) { /* f(position, a, b); four edges' loads in flight */
        for (uint64_t j = j0 + threadIdx.x; j < j1; j += 4ull * blockDim.x) {
            uint64_t k[4];
            uint32_t end[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = j + u * (uint64_t)blockDim.x < j1 ? keys[j + u * (uint64_t)blockDim.x] : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) end[u] = rp[(uint32_t)(k[u] >> vbits) + 1];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint64_t p = j + u * (uint64_t)blockDim.x;
                if (p < j1 && p + 1 < end[u]) f((uint32_t)p, (uint32_t)(k[u] >> vbits), (uint32_t)(k[u] & mask));
            }
        }
    };
    uint32_t *const mine = part + (size_t)blockIdx.x * top; /* this block's counts, from pass to pass */
    if constexpr (!FILL) {
        for (uint32_t i = threadIdx.x; i < top; i += blockDim.x) s_cnt[i] = 0u;
        __syncthreads();
        each([&](uint32_t, uint32_t, uint32_t b) {
            const uint32_t r = nv - 1u - b;
            if (r < top) atomicAdd(s_cnt + r, 1u);
            else atomicAdd(at + b, 1u);
        });
        __syncthreads();
        for (uint32_t r = threadIdx.x; r < top; r += blockDim.x) {
            mine[r] = s_cnt[r];
            if (s_cnt[r]) atomicAdd(at + (nv - 1u - r), s_cnt[r]);
        }
        return;
    } else {
        for (uint32_t r = threadIdx.x; r < top; r += blockDim.x) { /* where this block's part of each list begins */
            const uint32_t c = mine[r];
            if (c) s_cnt[r] = atomicAdd(at + (nv - 1u - r), c);
        }
        __syncthreads();
        each([&](uint32_t j, uint32_t a, uint32_t b) {
            const uint32_t r = nv - 1u - b;
            rev[r < top ? atomicAdd(s_cnt + r, 1u) : atomicAdd(at + b, 1u)] = make_uint2(j, a);
        });
    }
}

/* tasks per b: `size` of its edges each, none when N+(b) is empty */
__global__ void k_tc_task_count(const uint32_t *__restrict__ count, const uint32_t *__restrict__ rp, uint32_t nv,
                                uint32_t size, uint32_t *__restrict__ ntask) {
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nv; b += gridDim.x * blockDim.x)
        ntask[b] = rp[b + 1] > rp[b] ? (count[b] + size - 1) / size : 0u;
}
/* task t of b: (b, its first edge); end[b]: the end of b's edges, end[b - 1] their start */
__global__ void k_tc_tasks(const uint32_t *__restrict__ end, const uint32_t *__restrict__ pos,
                           const uint32_t *__restrict__ rp, uint32_t nv, uint32_t size, uint2 *__restrict__ task) {
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nv; b += gridDim.x * blockDim.x) {
        if (rp[b + 1] == rp[b]) continue;
        uint32_t t = pos[b];
        for (uint64_t e = b ? end[b - 1] : 0u; e < end[b]; e += size) task[t++] = make_uint2(b, (uint32_t)e);
    }
}

constexpr uint32_t NO_ONE = 0xFFFFFFFFu;
static_assert(TC_FILTER == 4096, "the hash's bits");
__device__ __forceinline__ uint32_t tc_hash(uint32_t c) { return (c * 2654435761u) >> 20; }

/* candidate c below the top ranks that passed the filter: is it among the first nlow elements of N+(b) (list)? */
__device__ __noinline__ bool low_candidate(uint32_t c, const uint32_t *__restrict__ list, uint32_t nlow,
                                           uint32_t *__restrict__ cnt) {
    uint32_t at = 0, len = nlow; /* the last element <= c */
    while (len > 1) {
        const uint32_t half = len >> 1;
        if (__ldg(list + at + half) <= c) at += half;
        len -= half;
    }
    if (__ldg(list + at) != c) return false;
    atomicAdd(cnt + c, 1u);
    return true;
}

/* The same of two candidates at once (want: bits 0, 1), returned as bits: what a search waits
 * for is one dependent load after another. */
__device__ __noinline__ uint32_t low_candidates(uint32_t c0, uint32_t c1, uint32_t want,
                                                const uint32_t *__restrict__ list, uint32_t nlow,
                                                uint32_t *__restrict__ cnt) {
    uint32_t at0 = 0, at1 = 0, len = nlow; /* the last element <= c */
    while (len > 1) {
        const uint32_t half = len >> 1;
        const uint32_t x0 = __ldg(list + at0 + half), x1 = __ldg(list + at1 + half);
        if (x0 <= c0) at0 += half;
        if (x1 <= c1) at1 += half;
        len -= half;
    }
    const uint32_t x0 = __ldg(list + at0), x1 = __ldg(list + at1);
    if (x0 != c0) want &= 2u;
    if (x1 != c1) want &= 1u;
    if (want & 1u) atomicAdd(cnt + c0, 1u);
    if (want & 2u) atomicAdd(cnt + c1, 1u);
    return want;
}

/* A warp takes tasks from a device counter, those of the highest b first. Counts of the
 * top ranks are gathered in the block's shared memory and added to `cnt` at the end:
 * one global atomic per triangle on those few addresses queues at the L2. */
template <bool FLAT>
__global__ void __launch_bounds__(1024, 1) k_tc_count(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ cl,
                                                      uint32_t nv, uint32_t top, const uint2 *__restrict__ rev,
                                                      const uint32_t *__restrict__ rev_end,
                                                      const uint2 *__restrict__ task,
                                                      const uint32_t *__restrict__ ntasks, uint32_t size,
                                                      uint32_t full, uint32_t *ticket,
                                                      uint32_t *__restrict__ cnt, unsigned long long *total) {
    extern __shared__ uint32_t s_mem[];
    uint32_t *const s_top = s_mem; /* rank nv - 1 - r at r */
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t *const bits = s_mem + TC_TOP + w * TC_WARP_WORDS, *const filter = bits + TC_TOP / 32;
    uint32_t *const list_off = filter + TC_FILTER / 32, *const list_hit = list_off + 32;
    for (uint32_t i = threadIdx.x; i < TC_TOP + TC_WARPS * TC_WARP_WORDS; i += blockDim.x) s_mem[i] = 0u;
    __syncthreads();
    const uint32_t last_rank = nv - 1u;
    auto bump = [&](uint32_t v, uint32_t inc) {
        const uint32_t r = last_rank - v;
        if (r < top) atomicAdd(s_top + r, inc);
        else atomicAdd(cnt + v, inc);
    };
    auto hashed = [](uint32_t c) { return tc_hash(c); };
    const uint32_t n = *ntasks;
    unsigned long long mine = 0;
    const uint32_t upto = FULL >> (31u - lane);
    uint32_t t0 = 0;
    for (;;) {
        /* one by one among the tasks of the many-edged top ranks, then eight at a time */
        const uint32_t grab = t0 > full ? 8u : 1u;
        if (lane == 0) t0 = atomicAdd(ticket, grab);
        t0 = __shfl_sync(FULL, t0, 0);
        if (t0 >= n) break;
        const uint32_t nt = min(grab, n - t0);
        uint32_t tb = 0, te0 = 0, te1 = 0, tB = 0, tn = 0; /* lane q: the claim's task q */
        if (lane < nt) {
            const uint2 tk = task[n - 1u - t0 - lane];
            tb = tk.x;
            te0 = tk.y;
            te1 = (uint32_t)min((uint64_t)te0 + size, (uint64_t)rev_end[tb]);
            tB = __ldg(rp + tb);
            tn = __ldg(rp + tb + 1) - tB;
        }
        for (uint32_t q0 = 0; q0 < nt; ++q0) {
            const uint32_t b = __shfl_sync(FULL, tb, q0), first = __shfl_sync(FULL, te0, q0),
                           e1 = __shfl_sync(FULL, te1, q0), B = __shfl_sync(FULL, tB, q0),
                           nb = __shfl_sync(FULL, tn, q0);
            uint32_t nlow = 0; /* elements of N+(b) without a bit of their own: its first ones */
            for (uint32_t i = lane; i < ((nb + 31u) & ~31u); i += 32u) {
                bool low = false;
                if (i < nb) {
                    const uint32_t c = __ldg(cl + B + i), r = last_rank - c;
                    low = r >= top;
                    if (!low) {
                        atomicOr(bits + (r >> 5), 1u << (r & 31u));
                    } else {
                        const uint32_t h = hashed(c);
                        atomicOr(filter + (h >> 5), 1u << (h & 31u));
                    }
                }
                nlow += __popc(__ballot_sync(FULL, low));
            }
            __syncwarp();
            /* which of the candidates (one per lane, NO_ONE where there is none) are in N+(b),
             * each counted; those without a bit of their own go the long way, out of line */
            auto probe = [&](uint32_t c) -> uint32_t {
                const uint32_t r = last_rank - c; /* NO_ONE: nv */
                bool hit = false;
                if (r < top) hit = (bits[r >> 5] >> (r & 31u)) & 1u;
                if (hit) atomicAdd(s_top + r, 1u);
                uint32_t m = __ballot_sync(FULL, hit);
                if (nlow) {
                    const uint32_t h = tc_hash(c);
                    const bool maybe = r - top < nv - top && ((filter[h >> 5] >> (h & 31u)) & 1u);
                    if (__any_sync(FULL, maybe))
                        m |= __ballot_sync(FULL, maybe && low_candidate(c, cl + B, nlow, cnt));
                }
                return m;
            };
            /* the same of two candidates per lane, for many such elements: there the filter lets
             * many through */
            auto probe2 = [&](uint32_t c0, uint32_t c1, uint32_t &m0, uint32_t &m1) {
                const uint32_t r0 = last_rank - c0, r1 = last_rank - c1;
                bool hit0 = false, hit1 = false;
                if (r0 < top) hit0 = (bits[r0 >> 5] >> (r0 & 31u)) & 1u;
                if (r1 < top) hit1 = (bits[r1 >> 5] >> (r1 & 31u)) & 1u;
                if (hit0) atomicAdd(s_top + r0, 1u);
                if (hit1) atomicAdd(s_top + r1, 1u);
                const uint32_t h0 = tc_hash(c0), h1 = tc_hash(c1);
                uint32_t want = r0 - top < nv - top ? (filter[h0 >> 5] >> (h0 & 31u)) & 1u : 0u;
                if (r1 - top < nv - top) want |= ((filter[h1 >> 5] >> (h1 & 31u)) & 1u) << 1;
                if (want) want = low_candidates(c0, c1, want, cl + B, nlow, cnt);
                __syncwarp();
                m0 = __ballot_sync(FULL, hit0 || (want & 1u));
                m1 = __ballot_sync(FULL, hit1 || (want & 2u));
            };
            const bool pairs = FLAT && nlow >= TC_PAIRS;
            uint32_t bsum = 0;
            for (uint32_t e0 = first; e0 < e1; e0 += 32u) {
                const uint32_t ne = min(32u, e1 - e0);
                uint32_t base = 0, len = 0, a = 0, hits = 0;
                if (lane < ne) {
                    const uint2 e = rev[e0 + lane];
                    a = e.y;
                    base = e.x + 1u;
                    len = __ldg(rp + a + 1) - base;
                }
                /* whole windows of 32 candidates list by list */
                const uint32_t nf = len >> 5;
                for (uint32_t many = __ballot_sync(FULL, nf != 0u); many; many &= many - 1u) {
                    const int l = __ffs((int)many) - 1;
                    const uint32_t *at = cl + __shfl_sync(FULL, base, l) + lane;
                    const uint32_t n32 = __shfl_sync(FULL, nf, l);
                    uint32_t m = 0, o = 0;
                    if (pairs)
                        for (; o + 1u < n32; o += 2u) {
                            uint32_t m0, m1;
                            probe2(__ldg(at + 32u * o), __ldg(at + 32u * o + 32u), m0, m1);
                            m += __popc(m0) + __popc(m1);
                        }
                    for (; o + 1u < n32; o += 2u) {
                        const uint32_t x = __ldg(at + 32u * o), y = __ldg(at + 32u * o + 32u);
                        m += __popc(probe(x));
                        m += __popc(probe(y));
                    }
                    if (o < n32) m += __popc(probe(__ldg(at + 32u * o)));
                    if ((int)lane == l) hits = m;
                }
                /* what is left of the lists end to end. The list of a position: the number
                 * of lists begun up to it; lists with nothing left are passed over */
                const uint32_t rest = len & 31u, some = __ballot_sync(FULL, rest != 0u);
                const uint32_t mine_at = __popc(some & (upto >> 1));
                uint32_t incl = rest;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, incl, d);
                    if (lane >= (uint32_t)d) incl += y;
                }
                const uint32_t W = __shfl_sync(FULL, incl, 31), excl = incl - rest;
                if (rest) {
                    list_off[mine_at] = base + (len - rest) - excl;
                    list_hit[mine_at] = 0u;
                }
                __syncwarp();
                uint32_t begun = 0;
                for (uint32_t w1 = 0; w1 < W; w1 += 32u * TC_WINDOWS) {
                    uint32_t x[TC_WINDOWS], q[TC_WINDOWS];
#pragma unroll
                    for (int u = 0; u < TC_WINDOWS; ++u) {
                        const uint32_t w0 = w1 + 32u * u, d = excl - w0;
                        const uint32_t starts = __reduce_or_sync(FULL, rest && d < 32u ? 1u << d : 0u);
                        q[u] = begun + __popc(starts & upto) - 1u;
                        begun += __popc(starts);
                        x[u] = w0 + lane < W ? __ldg(cl + (list_off[q[u]] + w0 + lane)) : NO_ONE;
                    }
                    if (pairs) {
#pragma unroll
                        for (int u = 0; u < TC_WINDOWS; u += 2) {
                            if (w1 + 32u * u >= W) break;
                            uint32_t m0, m1;
                            probe2(x[u], x[u + 1], m0, m1);
                            if ((m0 >> lane) & 1u) atomicAdd(list_hit + q[u], 1u);
                            if ((m1 >> lane) & 1u) atomicAdd(list_hit + q[u + 1], 1u);
                        }
                        continue;
                    }
#pragma unroll
                    for (int u = 0; u < TC_WINDOWS; ++u)
                        if (w1 + 32u * u < W && ((probe(x[u]) >> lane) & 1u)) atomicAdd(list_hit + q[u], 1u);
                }
                __syncwarp();
                if (rest) hits += list_hit[mine_at];
                __syncwarp();
                if (hits) bump(a, hits);
                bsum += hits;
            }
            bsum = __reduce_add_sync(FULL, bsum);
            if (lane == 0 && bsum) {
                bump(b, bsum);
                mine += bsum;
            }
            __syncwarp();
            for (uint32_t i = lane; i < nb; i += 32u) { /* the bits are cleared for the next task */
                const uint32_t c = __ldg(cl + B + i), r = last_rank - c;
                if (r < top) bits[r >> 5] = 0u;
                else filter[hashed(c) >> 5] = 0u;
            }
            __syncwarp();
        }
    }
    if (lane == 0 && mine) atomicAdd(total, mine);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < top; i += blockDim.x)
        if (s_top[i]) atomicAdd(cnt + (last_rank - i), s_top[i]);
}

/* ---- counting where lists are short (TC_SHORT) --------------------------------- */

/* One halving of the search for the last element <= x in the sorted,
 * duplicate-free cl[base .. base + n), n >= 2: the range that still holds that
 * element shrinks to ceil(n / 2) values. After ceil(log2 n) halvings n is 1 and
 * x is present exactly when cl[base] equals it. */
__device__ __forceinline__ uint32_t last_le_step(const uint32_t *__restrict__ cl, uint32_t base, uint32_t &n,
                                                 uint32_t x) {
    const uint32_t h = n >> 1;
    if (__ldg(cl + base + h) <= x) base += h;
    n -= h;
    return base;
}

constexpr uint32_t TC_SPLIT = 64;   /* top-range vertices with more higher-ranked neighbours go batch by batch */

/* Longest higher-ranked neighbour list among rows lo .. nv - 1 (atomicMax into *out). */
__global__ void k_max_rowlen(const uint32_t *__restrict__ rp, uint32_t lo, uint32_t nv, uint32_t *out) {
    uint32_t m = 0;
    for (uint32_t r = lo + blockIdx.x * blockDim.x + threadIdx.x; r < nv; r += gridDim.x * blockDim.x)
        m = max(m, rp[r + 1] - rp[r]);
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

/* Triangles through vertex a, 32 of its higher-ranked neighbours b at a time (a
 * batch). For each b the shorter of (N+(a) after b) and N+(b) is searched element
 * by element in the longer; the searches of the batch's b's are laid end to end
 * (a warp prefix sum of their lengths) and dealt to the lanes two at a time, so
 * every lane runs two independent searches whatever the lengths. A match c is the
 * triangle (a, b, c): c's count is bumped per match, b's by its match total, a's
 * by the batch's sum. A b whose two lists are both long is not searched: the
 * whole warp merges the two lists instead, after the searches.
 * Work is spread two ways. Vertex a goes to warp (a mod warps), numbered block
 * fastest, so the heavy vertices, which sit together in the upper ranks, land on
 * every SM. Vertices among the top `nsplit` ranks with more than TC_SPLIT
 * higher-ranked neighbours are not taken whole: their batches are dealt out one
 * by one after the other vertices, so no warp is left with a whole heavy vertex.
 * Ranks grow with degree, so the highest-ranked vertex of a triangle is nearly
 * always among the top few thousand ranks: their counts are kept in the block's
 * shared memory (dynamic, `top` entries for ranks nv - top .. nv - 1) and added
 * to `cnt` once at the end, which keeps the per-triangle increments off a few
 * hot global addresses. */
__global__ void __launch_bounds__(1024, 2) k_tc_search(const uint32_t *__restrict__ rp, const uint32_t *__restrict__ cl,
                                                       uint32_t nv, uint32_t top, uint32_t nsplit,
                                                      const uint32_t *__restrict__ split_maxlen,
                                                      uint32_t *__restrict__ cnt, unsigned long long *total) {
    extern __shared__ uint32_t s_top[];
    __shared__ uint32_t s_pre[TC_WARPS][32], s_so[TC_WARPS][32], s_lo[TC_WARPS][32], s_nl[TC_WARPS][32],
        s_hit[TC_WARPS][32];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t *pre = s_pre[w], *so_ = s_so[w], *lo_ = s_lo[w], *nl_ = s_nl[w], *hit = s_hit[w];
    const uint32_t warp = w * gridDim.x + blockIdx.x;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t lo_top = nv - top, lo_split = nv - nsplit;
    for (uint32_t i = threadIdx.x; i < top; i += blockDim.x) s_top[i] = 0;
    __syncthreads();
    auto bump = [&](uint32_t v, uint32_t inc) {
        if (v >= lo_top)
            atomicAdd(s_top + (v - lo_top), inc);
        else
            atomicAdd(cnt + v, inc);
    };
    /* the batch of a's neighbours j0 .. j0 + 31 (ab <= j0, j0 + 1 < ae); returns
     * this lane's b's match total (0 for lanes past the list) */
    auto batch = [&](uint32_t ab, uint32_t ae, uint32_t j0) -> uint32_t {
        const uint32_t j = j0 + lane;
        uint32_t ns = 0, so = 0, lo = 0, nl = 0, b = 0;
        bool mrg = false;
        if (j + 1 < ae) {
            b = __ldg(cl + j);
            const uint32_t na = ae - j - 1, bb = __ldg(rp + b), nb = __ldg(rp + b + 1) - bb;
            if (nb) {
                if (na <= nb) {
                    ns = na, so = j + 1, lo = bb, nl = nb;
                } else {
                    ns = nb, so = bb, lo = j + 1, nl = na;
                }
                /* both lists long: a merge of the two (a warp walking na + nb
                 * values, one partition search per lane) when the ns searches of
                 * log2(nl) steps would take more than three steps per merged value
                 * (a merge step is a dependent load; 1.5, 2, 3, 4 and 6 were
                 * measured) */
                const uint32_t tot = na + nb;
                if (ns * (32 - __clz((nl - 1) | 1)) > 3 * tot + 32 * (32 - __clz((tot - 1) | 1))) {
                    mrg = true, ns = 0;
                }
            }
        }
        uint32_t inc = ns;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += t;
        }
        const uint32_t W = __shfl_sync(FULL, inc, 31);
        const uint32_t merges = __ballot_sync(FULL, mrg);
        if (W == 0 && merges == 0) return 0u;
        pre[lane] = inc, so_[lane] = so, lo_[lane] = lo, nl_[lane] = nl, hit[lane] = 0;
        __syncwarp();
        for (uint32_t t0 = 0; t0 < W; t0 += 64) {
            uint32_t x[2], base[2], n[2], q[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t t = t0 + 32 * u + lane;
                n[u] = 0, x[u] = 0, base[u] = 0, q[u] = 0;
                if (t < W) {
                    /* owner: how many of the 32 inclusive prefix sums are <= t
                     * (t < W = pre[31], so at most 31; indexes stay below 31) */
                    uint32_t qq = 0;
#pragma unroll
                    for (uint32_t st = 16; st; st >>= 1)
                        if (pre[qq + st - 1] <= t) qq += st;
                    const uint32_t k = t - (qq ? pre[qq - 1] : 0);
                    x[u] = __ldg(cl + so_[qq] + k);
                    base[u] = lo_[qq], n[u] = nl_[qq], q[u] = qq;
                }
            }
            while (n[0] > 1 || n[1] > 1) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (n[u] > 1) base[u] = last_le_step(cl, base[u], n[u], x[u]);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (n[u] == 1 && __ldg(cl + base[u]) == x[u]) {
                    bump(x[u], 1u);
                    atomicAdd(hit + q[u], 1u);
                }
        }
        __syncwarp();
        /* the merged pairs, one at a time by the whole warp: A = N+(a) after b,
         * B = N+(b); lane l walks diagonals [l per, (l + 1) per) of the merge that
         * takes A[i] when A[i] <= B[j], so B[j] is the least B value not below
         * A[i] and A[i] is in B exactly when they are equal */
        for (uint32_t m = merges; m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const uint32_t jl = j0 + (uint32_t)l, A = jl + 1, na = ae - jl - 1;
            const uint32_t bl = __shfl_sync(FULL, b, l), B = __ldg(rp + bl), nb = __ldg(rp + bl + 1) - B;
            const uint32_t tot = na + nb, per = (tot + 31) / 32;
            const uint32_t d0 = min(lane * per, tot), d1 = min(d0 + per, tot);
            uint32_t i = d0 > nb ? d0 - nb : 0, hi = min(d0, na);
            while (i < hi) { /* first i with A[i] > B[d0 - 1 - i] */
                const uint32_t mid = (i + hi) >> 1;
                if (__ldg(cl + A + mid) <= __ldg(cl + B + d0 - 1 - mid))
                    i = mid + 1;
                else
                    hi = mid;
            }
            uint32_t k = d0 - i, found = 0;
            uint32_t av = i < na ? __ldg(cl + A + i) : 0u, bv = k < nb ? __ldg(cl + B + k) : 0u;
            for (uint32_t d = d0; d < d1; ++d) {
                if (i < na && (k >= nb || av <= bv)) {
                    if (k < nb && av == bv) {
                        bump(av, 1u);
                        ++found;
                    }
                    ++i;
                    if (i < na) av = __ldg(cl + A + i);
                } else {
                    ++k;
                    if (k < nb) bv = __ldg(cl + B + k);
                }
            }
            found = __reduce_add_sync(FULL, found);
            if (lane == 0 && found) hit[l] += found;
            __syncwarp();
        }
        const uint32_t h = hit[lane];
        if (h) bump(b, h);
        __syncwarp(); /* the tables are rewritten by the next batch */
        return h;
    };
    unsigned long long mine = 0;
    auto finish = [&](uint32_t a, uint32_t acc) {
        const uint32_t A = __reduce_add_sync(FULL, acc);
        if (A && lane == 0) {
            bump(a, A);
            mine += A;
        }
    };
    for (uint32_t a = warp; a < nv; a += nwarps) {
        const uint32_t ab = __ldg(rp + a), ae = __ldg(rp + a + 1);
        if (ae - ab < 2) continue; /* a triangle needs two higher-ranked neighbours */
        if (a >= lo_split && ae - ab > TC_SPLIT) continue; /* dealt out batch by batch below */
        uint32_t acc = 0;
        for (uint32_t j0 = ab; j0 + 1 < ae; j0 += 32) acc += batch(ab, ae, j0);
        finish(a, acc);
    }
    /* the split vertices' batches: item t is batch t / nsplit of vertex
     * lo_split + t % nsplit, and goes to warp t mod warps (neighbouring vertices'
     * batches to different warps); each lane checks one of its warp's items, the
     * warp runs the real ones */
    const uint64_t items = (uint64_t)nsplit * ((*split_maxlen + 31) / 32);
    for (uint64_t k0 = 0; warp + (uint64_t)nwarps * k0 < items; k0 += 32) {
        const uint64_t t = warp + (uint64_t)nwarps * (k0 + lane);
        uint32_t a = 0, ab = 0, ae = 0, j0 = 0;
        bool real = false;
        if (t < items) {
            a = lo_split + (uint32_t)(t % nsplit);
            ab = __ldg(rp + a), ae = __ldg(rp + a + 1);
            j0 = ab + 32u * (uint32_t)(t / nsplit);
            real = ae - ab > TC_SPLIT && j0 + 1 < ae;
        }
        for (uint32_t m = __ballot_sync(FULL, real); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const uint32_t va = __shfl_sync(FULL, a, l), vab = __shfl_sync(FULL, ab, l),
                           vae = __shfl_sync(FULL, ae, l), vj0 = __shfl_sync(FULL, j0, l);
            finish(va, batch(vab, vae, vj0));
        }
    }
    if (lane == 0 && mine) atomicAdd(total, mine);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < top; i += blockDim.x)
        if (s_top[i]) atomicAdd(cnt + lo_top + i, s_top[i]);
}

}  // namespace
}  // namespace gcg

using namespace gcg;

extern "C" int gcg_triangle_count(gcg_graph *g, uint64_t *total, uint32_t *per_rank, uint32_t *vertexmap,
                                  gcg_tc_stats *stats) {
    if (!g) return fail(GCG_ERR_INVALID, "gcg_triangle_count: null graph");
    GCG_TRY(ensure_plan(g));
    cudaStream_t s = g->stream;
    const uint32_t nv = g->nv, vbits = g->vbits;
    const uint64_t ne = g->ne;
    const PrPlan &pl = *g->plan;

    cudaEvent_t ev0, ev1;
    GCG_CUDA(cudaEventCreate(&ev0));
    GCG_CUDA(cudaEventCreate(&ev1));
    GCG_CUDA(cudaEventRecord(ev0, s));

    /* 1. degree ranking */
    tbuf<uint64_t> keys, tmp;
    tbuf<uint32_t> rank;
    tbuf<DegreeStat> dstat;
    GCG_TRY(keys.alloc(std::max<uint64_t>(nv, ne), s));
    GCG_TRY(tmp.alloc(std::max<uint64_t>(nv, ne), s));
    GCG_TRY(rank.alloc(nv, s));
    GCG_TRY(dstat.alloc(1, s));
    GCG_CUDA(cudaMemsetAsync(dstat.get(), 0, sizeof(DegreeStat), s));
    k_degree_keys<<<vgrid(nv), 256, 0, s>>>(g->indeg.get(), g->outdeg.get(), nv, vbits, keys.get(), dstat.get());
    DegreeStat deg = {};
    GCG_CUDA(cudaMemcpyAsync(&deg, dstat.get(), sizeof(deg), cudaMemcpyDeviceToHost, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    uint32_t dbits = 1;
    while (dbits < 33 && (1ull << dbits) <= deg.most) ++dbits;
    /* neighbours of an edge's end, on average over the edges (a symmetric graph counts each twice) */
    const double twice = g->symmetric ? 2.0 : 1.0;
    const double edge_degree = ne ? deg.squares / (2.0 * (double)ne) / twice : 0.0;
    const double mean_degree = 2.0 * (double)ne / (double)nv / twice;
    if (vbits + dbits > 64) return fail(GCG_ERR_UNSUPPORTED, "gcg_triangle_count: degree and id do not fit 64 bits");
    uint64_t *sorted = nullptr;
    GCG_TRY(radix_sort_u64(keys.get(), tmp.get(), nv, 0, (int)(vbits + dbits), &sorted, s));
    k_rank_scatter<<<vgrid(nv), 256, 0, s>>>(sorted, nv, vbits, rank.get());
    GCG_LAUNCH_CHECK();

    /* 2. oriented, deduplicated edges in rank space */
    uint64_t m_or = 0;
    uint64_t *okeys = nullptr; /* the oriented edges' sorted keys */
    uint2 *rev = nullptr;      /* room for the edges grouped by their second vertex */
    dbuf<uint32_t> rp, cl;
    GCG_TRY(rp.alloc((size_t)nv + 1));
    if (ne > 0) {
        int per_sm = 4;
        unsigned tb = (unsigned)std::max<uint32_t>(1, std::min<uint32_t>(pl.ntiles, (uint32_t)(num_sms() * per_sm)));
        /* a symmetric graph keeps one of the two stored copies of every edge */
        const int half = g->symmetric ? 1 : 0;
        tbuf<uint32_t> fl, d_tot;
        GCG_TRY(d_tot.alloc(1, s));
        GCG_CUDA(cudaMemsetAsync(d_tot.get(), 0, 4, s));
        k_orient_keys<<<tb, MP_THREADS, 0, s>>>(g->in_rowptr.get(), g->in_col.get(), pl.tile_row.get(),
                                               pl.tile_edge.get(), pl.ntiles, rank.get(), vbits, half, d_tot.get(),
                                               keys.get());
        GCG_LAUNCH_CHECK();
        uint64_t nk = ne;
        if (half) {
            uint32_t kept = 0;
            GCG_CUDA(cudaMemcpyAsync(&kept, d_tot.get(), 4, cudaMemcpyDeviceToHost, s));
            GCG_CUDA(cudaStreamSynchronize(s));
            nk = kept;
        }
        if (nk > 0) {
            GCG_TRY(radix_sort_u64(keys.get(), tmp.get(), nk, 0, 2 * (int)vbits, &sorted, s));
            /* unique: flags + scan + scatter, then CSR by the low-rank half */
            GCG_TRY(fl.alloc(nk, s));
            uint64_t *other = sorted == keys.get() ? tmp.get() : keys.get();
            GCG_TRY(unique_u64(sorted, nk, fl.get(), d_tot.get(), other, s));
            uint32_t tot = 0;
            GCG_CUDA(cudaMemcpyAsync(&tot, d_tot.get(), 4, cudaMemcpyDeviceToHost, s));
            GCG_CUDA(cudaStreamSynchronize(s));
            m_or = tot;
            GCG_TRY(cl.alloc(m_or));
            GCG_TRY(csr_from_sorted_keys(other, m_or, vbits, nv, rp.get(), cl.get(), s));
            okeys = other;
            rev = (uint2 *)sorted; /* no longer read once the unique keys are out */
        } else {
            GCG_TRY(cl.alloc(1));
            GCG_CUDA(cudaMemsetAsync(rp.get(), 0, ((size_t)nv + 1) * 4, s));
        }
    } else {
        GCG_TRY(cl.alloc(1));
        GCG_CUDA(cudaMemsetAsync(rp.get(), 0, ((size_t)nv + 1) * 4, s));
    }

    /* 3. count */
    tbuf<uint32_t> cnt;
    tbuf<unsigned long long> d_total;
    uint32_t *cnt_ptr;
    const bool dev_counts = per_rank && is_device_ptr(per_rank);
    if (dev_counts) {
        cnt_ptr = per_rank;
    } else {
        GCG_TRY(cnt.alloc(nv, s));
        cnt_ptr = cnt.get();
    }
    GCG_TRY(d_total.alloc(1, s));
    GCG_CUDA(cudaMemsetAsync(cnt_ptr, 0, (size_t)nv * 4, s));
    GCG_CUDA(cudaMemsetAsync(d_total.get(), 0, 8, s));
    const uint32_t top = std::min(nv, TC_TOP);
    const unsigned sms = (unsigned)num_sms();
    if (m_or > 0 && edge_degree < TC_SHORT) {
        const uint32_t nsplit = std::min(nv, std::max<uint32_t>(65536u, nv / 16));
        tbuf<uint32_t> split_maxlen;
        GCG_TRY(split_maxlen.alloc(1, s));
        GCG_CUDA(cudaMemsetAsync(split_maxlen.get(), 0, 4, s));
        k_max_rowlen<<<vgrid(nsplit), 256, 0, s>>>(rp.get(), nv - nsplit, nv, split_maxlen.get());
        GCG_CUDA(cudaFuncSetAttribute(k_tc_search, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TC_TOP * 4)));
        /* two blocks per SM, each with its own top-rank counters */
        const unsigned cb = (unsigned)std::min<uint64_t>(((uint64_t)nv + TC_WARPS - 1) / TC_WARPS, 2ull * sms);
        k_tc_search<<<cb, TC_WARPS * 32, (size_t)top * 4, s>>>(rp.get(), cl.get(), nv, top, nsplit,
                                                               split_maxlen.get(), cnt_ptr, d_total.get());
        GCG_LAUNCH_CHECK();
    } else if (m_or > 0) {
        /* the edges grouped by b, cut into tasks */
        tbuf<uint32_t> in_cnt, ntask, ctl, part;
        tbuf<uint2> task;
        GCG_TRY(in_cnt.alloc(nv, s));
        GCG_TRY(ntask.alloc(nv, s));
        GCG_TRY(ctl.alloc(2, s)); /* tasks, ticket */
        /* about sixteen full tasks per warp, so that the last ones end together */
        const uint64_t warps = (uint64_t)num_sms() * TC_WARPS;
        const uint32_t size =
            (uint32_t)std::min<uint64_t>(TC_TASK_MAX, std::max<uint64_t>(TC_TASK_MIN, m_or / (16 * warps) & ~31ull));
        const uint64_t most = std::min<uint64_t>(nv, m_or) + m_or / size;
        const uint32_t full = (uint32_t)(2 * (m_or / size) + 8 * warps);
        GCG_TRY(task.alloc(most, s));
        GCG_CUDA(cudaMemsetAsync(in_cnt.get(), 0, (size_t)nv * 4, s));
        GCG_CUDA(cudaMemsetAsync(ctl.get(), 0, 8, s));
        GCG_TRY(part.alloc((size_t)sms * top, s));
        GCG_CUDA(cudaFuncSetAttribute(k_tc_group<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TC_TOP * 4)));
        GCG_CUDA(cudaFuncSetAttribute(k_tc_group<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(TC_TOP * 4)));
        k_tc_group<false><<<sms, 1024, top * 4, s>>>(okeys, m_or, vbits, rp.get(), nv, top, in_cnt.get(), part.get(),
                                                       nullptr);
        k_tc_task_count<<<vgrid(nv), 256, 0, s>>>(in_cnt.get(), rp.get(), nv, size, ntask.get());
        GCG_TRY(scan_u32(ntask.get(), ntask.get(), nv, ctl.get(), s));
        GCG_TRY(scan_u32(in_cnt.get(), in_cnt.get(), nv, nullptr, s));
        k_tc_group<true><<<sms, 1024, top * 4, s>>>(okeys, m_or, vbits, rp.get(), nv, top, in_cnt.get(), part.get(), rev);
        k_tc_tasks<<<vgrid(nv), 256, 0, s>>>(in_cnt.get(), ntask.get(), rp.get(), nv, size, task.get());
        auto kern = edge_degree < TC_FLAT * mean_degree ? k_tc_count<true> : k_tc_count<false>;
        GCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
        kern<<<sms, TC_WARPS * 32, TC_SMEM, s>>>(rp.get(), cl.get(), nv, top, rev, in_cnt.get(),
                                                             task.get(), ctl.get(), size, full, ctl.get() + 1,
                                                             cnt_ptr, d_total.get());
        GCG_LAUNCH_CHECK();
    }
    GCG_CUDA(cudaEventRecord(ev1, s));
    unsigned long long tri = 0;
    GCG_CUDA(cudaMemcpyAsync(&tri, d_total.get(), 8, cudaMemcpyDeviceToHost, s));
    if (per_rank && !dev_counts) GCG_TRY(copy_out(per_rank, cnt_ptr, (size_t)nv * 4, s));
    if (vertexmap) GCG_TRY(copy_out(vertexmap, rank.get(), (size_t)nv * 4, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    if (total) *total = tri;
    if (stats) {
        stats->triangles = tri;
        stats->oriented_edges = m_or;
        stats->device_ms = ms;
    }
    return GCG_OK;
}
