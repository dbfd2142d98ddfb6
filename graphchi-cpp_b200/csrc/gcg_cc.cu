/*
 * Connected components: replaces graphchi_engine::run(ConnectedComponentsProgram)
 * (example_apps/connectedcomponents.cpp:79-138), whose fixpoint labels every
 * vertex with the minimum vertex id of its weakly connected component.
 *
 * Device form: min-label propagation on roots with pointer-jumping shortcuts
 * (hook-and-compress). parent[v] starts at v; every edge (u,v) hooks the larger
 * of the two current roots under the smaller with a CAS (labels only move to
 * smaller ids, so parent[x] <= x always holds and each final root is the
 * minimum id of its component); finds shorten paths by pointer jumping (path
 * halving) as they go; a last pass jumps every vertex to its root. The edge pass
 * walks the merge-path tiles of the in-CSR, so hubs and empty rows are spread
 * evenly over the CTAs; one pass suffices because hooking is transitive.
 * The CAS loop has no waits on other threads: each failed CAS moves to a
 * strictly smaller id, so it ends.
 *
 * When every vertex's full neighbourhood is at hand (a symmetrised graph: the
 * in-list; otherwise the in-list plus the out-list), the edge pass samples
 * instead (the Afforest scheme with one round): every vertex points at the first
 * entry of its lists where that is smaller, by a plain store; the vertices whose
 * first entry is larger link it. The roots of 1024 sampled vertices then name the
 * most frequent one (the giant component; where no root has half of them, some
 * vertices link their last entry too and the sample is taken again), and only vertices
 * whose root is not it link all their neighbours (a thread per short list, a warp per
 * long one). A skipped vertex of the giant component loses nothing: each of its other edges is
 * also in the neighbour's list, and that neighbour links it unless it is in the
 * giant component too. The same hook keeps the labels (the minimum id per component).
 * R-MAT scale 24 symmetrised (521 M directed edges): 0.285 ms, of which the first pass,
 * bound by one column sector per vertex from HBM, is 0.096; with a CAS per vertex in that
 * pass, and every path climbed through L2 one step at a time, 0.889.
 */
#include <algorithm>

#include "gcg_internal.cuh"
#include "gcg_mergepath.cuh"

namespace gcg {
namespace {

__device__ __forceinline__ uint32_t find_root(uint32_t *parent, uint32_t x) {
    uint32_t p = ((volatile uint32_t *)parent)[x];
    while (p != x) {
        uint32_t gp = ((volatile uint32_t *)parent)[p];
        if (gp != p) ((volatile uint32_t *)parent)[x] = gp; /* path halving: gp < p <= x */
        x = p;
        p = gp;
    }
    return x;
}

__device__ __forceinline__ void hook(uint32_t *parent, uint32_t u, uint32_t v) {
    uint32_t a = find_root(parent, u);
    uint32_t b = find_root(parent, v);
    while (a != b) {
        uint32_t hi = a > b ? a : b, lo = a > b ? b : a;
        uint32_t old = atomicCAS(parent + hi, hi, lo);
        if (old == hi) return;
        /* hi was hooked elsewhere meanwhile: continue from its new parent */
        a = find_root(parent, old);
        b = lo == a ? a : find_root(parent, lo);
    }
}

__global__ void k_cc_init(uint32_t nv, uint32_t *parent) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) parent[v] = v;
}

__global__ void __launch_bounds__(MP_THREADS) k_cc_hook(const uint32_t *__restrict__ rowptr,
                                                        const uint32_t *__restrict__ col,
                                                        const uint32_t *__restrict__ tile_row,
                                                        const uint32_t *__restrict__ tile_edge, uint32_t ntiles,
                                                        uint32_t *parent) {
    __shared__ uint32_t s_rowend[MP_TILE];
    __shared__ uint32_t s_src[MP_TILE];
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t r0 = tile_row[t], r1 = tile_row[t + 1];
        const uint32_t e0 = tile_edge[t], e1 = tile_edge[t + 1];
        const uint32_t nrows = r1 - r0, nedges = e1 - e0;
        for (uint32_t k = threadIdx.x; k < nrows; k += MP_THREADS) s_rowend[k] = rowptr[r0 + k + 1] - e0;
        for (uint32_t k = threadIdx.x; k < nedges; k += MP_THREADS) s_src[k] = __ldg(col + e0 + k);
        __syncthreads();
        const uint32_t items = nrows + nedges;
        const uint32_t d0 = min((uint32_t)threadIdx.x * MP_ITEMS, items);
        const uint32_t d1 = min(d0 + MP_ITEMS, items);
        uint32_t ti = mp_search(s_rowend, nrows, nedges, d0);
        uint32_t tj = d0 - ti;
        for (uint32_t d = d0; d < d1; ++d) {
            if (ti < nrows && s_rowend[ti] <= tj) {
                ++ti;
            } else {
                hook(parent, s_src[tj], r0 + ti);
                ++tj;
            }
        }
        __syncthreads();
    }
}

/* neighbour i of v in the concatenation in-list(v) ++ out-list(v) (rout NULL: in-list only) */
struct Nbrs {
    const uint32_t *rin, *cin, *rout, *cout;
};
__device__ __forceinline__ uint32_t nbr_count(const Nbrs &n, uint32_t v) {
    uint32_t d = n.rin[v + 1] - n.rin[v];
    if (n.rout) d += n.rout[v + 1] - n.rout[v];
    return d;
}
__device__ __forceinline__ uint32_t nbr_at(const Nbrs &n, uint32_t v, uint32_t i) {
    const uint32_t b = n.rin[v], din = n.rin[v + 1] - b;
    return i < din ? n.cin[b + i] : n.cout[n.rout[v] + (i - din)];
}

/* Link of the sampling scheme: climbs one parent at a time and re-reads the
 * larger side's parent before the CAS, so a pair already joined by another
 * thread ends without an atomic (hub roots see many such pairs). Like hook, it
 * only ever points a root at a smaller id. */
__device__ __forceinline__ void link(uint32_t *parent, uint32_t u, uint32_t v) {
    volatile uint32_t *p = parent;
    uint32_t p1 = p[u], p2 = p[v];
    while (p1 != p2) {
        const uint32_t hi = p1 > p2 ? p1 : p2, lo = p1 > p2 ? p2 : p1;
        const uint32_t ph = p[hi];
        if (ph == lo) return;
        if (ph == hi && atomicCAS(parent + hi, hi, lo) == hi) return;
        p1 = p[p[hi]];
        p2 = p[lo];
    }
}

/* vertices in flight per thread in the passes over all vertices: what they wait for is
 * one or two dependent loads per vertex */
constexpr int CC_ILP = 4;

/* parent[v] = the smallest of v and the first entries of its lists; bit v of minima:
 * v has neighbours and none of those entries is smaller. Also zeroes the counters. No
 * atomics and no chase: every parent is at most its vertex, so this is a forest
 * whatever the graph. */
__global__ void __launch_bounds__(256) k_cc_first(Nbrs n, uint32_t nv, uint32_t *__restrict__ parent,
                                                  uint32_t *__restrict__ minima, uint32_t *cnt) {
    if (blockIdx.x == 0 && threadIdx.x < 4u) cnt[threadIdx.x] = 0u;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t end = ((uint64_t)nv + 31u) & ~31ull; /* whole warps: the ballots below */
    for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v0 < end; v0 += nth * CC_ILP) {
        uint32_t b[CC_ILP], e[CC_ILP], u[CC_ILP];
#pragma unroll
        for (int k = 0; k < CC_ILP; ++k) {
            const uint64_t v = v0 + k * nth;
            b[k] = v < nv ? __ldg(n.rin + v) : 0u;
            e[k] = v < nv ? __ldg(n.rin + v + 1) : 0u;
        }
#pragma unroll
        for (int k = 0; k < CC_ILP; ++k) u[k] = b[k] < e[k] ? __ldg(n.cin + b[k]) : GCG_NO_SOURCE;
        if (n.rout) {
#pragma unroll
            for (int k = 0; k < CC_ILP; ++k) {
                const uint64_t v = v0 + k * nth;
                b[k] = v < nv ? __ldg(n.rout + v) : 0u;
                e[k] = v < nv ? __ldg(n.rout + v + 1) : 0u;
            }
#pragma unroll
            for (int k = 0; k < CC_ILP; ++k)
                if (b[k] < e[k]) u[k] = min(u[k], __ldg(n.cout + b[k]));
        }
#pragma unroll
        for (int k = 0; k < CC_ILP; ++k) {
            const uint64_t v = v0 + k * nth;
            if (v >= end) break; /* uniform over the warp: nth and end are multiples of 32 */
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, v < nv && u[k] != GCG_NO_SOURCE && u[k] > (uint32_t)v);
            uint32_t p = min(u[k], (uint32_t)v);
            const uint32_t in_warp = p >> 5 == (uint32_t)v >> 5 && p != (uint32_t)v;
            if (__any_sync(0xFFFFFFFFu, in_warp)) /* a chain in id order comes out 32 times shorter */
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    const uint32_t pp = __shfl_sync(0xFFFFFFFFu, p, (int)(p & 31u));
                    if (p >> 5 == (uint32_t)v >> 5) p = pp;
                }
            if (v < nv) parent[v] = p;
            if ((threadIdx.x & 31u) == 0u) minima[v >> 5] = m;
        }
    }
}

/* The vertices of the bit set link their first neighbour: few where ids follow the
 * degrees, one in degree + 1 where they do not. A warp lists the set bits of up to 32
 * words (fewer where that keeps more warps busy) in shared memory first, so that its
 * lanes chase 32 of them at a time. */
__global__ void __launch_bounds__(256) k_cc_minima(Nbrs n, uint32_t nv, const uint32_t *__restrict__ minima,
                                                   uint32_t *parent) {
    __shared__ uint16_t s_list[8][1024];
    const uint32_t lane = threadIdx.x & 31u;
    uint16_t *list = s_list[threadIdx.x >> 5];
    const uint32_t words = (uint32_t)(((uint64_t)nv + 31u) >> 5);
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t per = min(32u, (words + nwarps - 1u) / nwarps);
    for (uint32_t w0 = per * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w0 < words; w0 += per * nwarps) {
        uint32_t m = lane < per && w0 + lane < words ? __ldg(minima + w0 + lane) : 0u;
        uint32_t at = (uint32_t)__popc(m);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, d);
            if (lane >= (uint32_t)d) at += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, at, 31);
        at -= (uint32_t)__popc(m);
        for (; m; m &= m - 1u) list[at++] = (uint16_t)(32u * lane + (uint32_t)__ffs((int)m) - 1u);
        __syncwarp();
        for (uint32_t k = lane; k < total; k += 32u) {
            const uint32_t v = 32u * w0 + list[k];
            link(parent, v, nbr_at(n, v, 0));
        }
        __syncwarp();
    }
}

/* Second round, only where the sampling found no giant component (cnt[2]; ids that do
 * not follow the degrees leave n / 32 trees after the first round of a uniform graph of
 * 16 neighbours a vertex): one vertex in CC_SPARSE links its last neighbour. That is two
 * links a tree there, enough for a giant component, and what these links wait for is one
 * another: all climb towards the same few roots (4 M vertices: 0.16 ms, all vertices
 * 4.4 ms; without this round the pass over the rest takes 2.4 ms). */
constexpr uint32_t CC_SPARSE = 16;
__global__ void __launch_bounds__(256) k_cc_second(Nbrs n, uint32_t nv, const uint32_t *cnt, uint32_t *parent) {
    if (cnt[2] == 0u) return;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * CC_SPARSE;
    for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * CC_SPARSE; v < nv; v += step) {
        const uint32_t d = nbr_count(n, (uint32_t)v);
        if (d > 1u) link(parent, (uint32_t)v, nbr_at(n, (uint32_t)v, d - 1u));
    }
}

/* The most frequent root among 1024 sampled vertices (ties: the smaller id), by one block
 * of 256 threads once every parent is a root: counted in a hash table in shared memory of
 * twice as many slots, the equal roots of a warp at once. cnt[1] = that root, cnt[2] =
 * fewer than half of the sampled vertices that hang below some root hang below it. With the
 * lists given (n.rin) cnt[2] also wants those of them that have neighbours to have more than
 * CC_GIANT / 8 on average: of fewer (1.58 in a uniform graph of one neighbour a vertex) no
 * giant component is made that a second round could find (uniform, 1 M vertices with 512 K
 * edges: 135 us with the round, 123 without; a core of 130,000 vertices with 1 M edges among
 * 4 M keeps it: 164 us, without 722). */
constexpr int CC_GIANT = 13;
__device__ __noinline__ int cc_dense(const Nbrs &n, uint32_t x) {
    const uint32_t d = nbr_count(n, x);
    return d ? 8 * (int)min(d, 4096u) - CC_GIANT : 0;
}
constexpr uint32_t CC_SLOTS = 2048;
static_assert(CC_SLOTS == 1u << 11, "the hash's shift");
__device__ void cc_sample(const Nbrs &n, const uint32_t *parent, uint32_t nv, uint32_t *cnt) {
    __shared__ uint32_t s_key[CC_SLOTS], s_cnt[CC_SLOTS];
    __shared__ unsigned long long s_best;
    __shared__ uint32_t s_below;
    __shared__ int s_dense;
    const uint32_t t = threadIdx.x;
    for (uint32_t k = t; k < CC_SLOTS; k += 256u) {
        s_key[k] = GCG_NO_SOURCE; /* no vertex */
        s_cnt[k] = 0u;
    }
    if (t == 0) {
        s_best = ~0ull;
        s_below = 0u;
        s_dense = n.rin ? 0 : 1;
    }
    uint32_t x[4], r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint64_t z = (uint64_t)(t + 256u * q) * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        x[q] = (uint32_t)(z % nv);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) r[q] = __ldcg(parent + x[q]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, r[q]);
        if ((t & 31u) == (uint32_t)__ffs((int)same) - 1u) {
            uint32_t at = (r[q] * 0x9E3779B1u) >> 21;
            for (uint32_t probe = 0; probe < CC_SLOTS; ++probe, at = (at + 1u) & (CC_SLOTS - 1u)) {
                const uint32_t old = atomicCAS(&s_key[at], GCG_NO_SOURCE, r[q]);
                if (old == GCG_NO_SOURCE || old == r[q]) {
                    atomicAdd(&s_cnt[at], (uint32_t)__popc(same));
                    break;
                }
            }
        }
        const uint32_t nb = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, r[q] != x[q]));
        if ((t & 31u) == 0u) atomicAdd(&s_below, nb);
        if (n.rin) atomicAdd(&s_dense, cc_dense(n, x[q]));
    }
    __syncthreads();
    for (uint32_t k = t; k < CC_SLOTS; k += 256u)
        if (s_cnt[k]) atomicMin(&s_best, ((unsigned long long)(1024u - s_cnt[k]) << 32) | s_key[k]);
    __syncthreads();
    if (t == 0) {
        cnt[1] = (uint32_t)(s_best & 0xFFFFFFFFull);
        cnt[2] = 2u * (1024u - (uint32_t)(s_best >> 32)) < s_below && s_dense > 0;
    }
}

constexpr uint32_t CC_THREAD_MAX = 8; /* neighbours a thread links itself, one after another */

/* c is v or an ancestor of v. Shortens the path as find_root does, but never past c, so
 * that what was below c stays so when c is hooked under a smaller root meanwhile. */
__device__ __forceinline__ bool below(uint32_t *parent, uint32_t v, uint32_t c) {
    volatile uint32_t *par = parent;
    uint32_t x = v, p = par[x];
    while (x != c && p != c && p != x) {
        const uint32_t gp = par[p];
        if (gp != p) par[x] = gp;
        x = p;
        p = gp;
    }
    return x == c || p == c;
}

/* Vertices outside the giant component link their neighbours (the first of a symmetric
 * graph's list is linked already): a thread a short list, the warp together a long one.
 * Every parent is a root at the start, so one coalesced load tells, CC_REST vertices at a
 * time. A warp lists the few that are left before it works on them, so that their chains
 * of dependent loads run side by side, not one per step (79.8 -> 41.2 us at R-MAT scale 24). */
constexpr int CC_REST = 8;
__global__ void __launch_bounds__(256) k_cc_rest(Nbrs n, uint32_t nv, const uint32_t *cnt, uint32_t *parent) {
    __shared__ uint32_t s_list[8][32 * CC_REST];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t c = cnt[1], lane = threadIdx.x & 31u, i0 = n.rout ? 0u : 1u;
    uint32_t *list = s_list[threadIdx.x >> 5];
    volatile uint32_t *par = parent;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t end = ((uint64_t)nv + 31u) & ~31ull; /* whole warps: the ballots below */
    for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v0 < end; v0 += nth * CC_REST) {
        uint32_t p[CC_REST], d[CC_REST];
#pragma unroll
        for (int k = 0; k < CC_REST; ++k) p[k] = v0 + k * nth < nv ? par[v0 + k * nth] : c;
#pragma unroll
        for (int k = 0; k < CC_REST; ++k) d[k] = p[k] != c ? nbr_count(n, (uint32_t)(v0 + k * nth)) : 0u;
        uint32_t total = 0;
#pragma unroll
        for (int k = 0; k < CC_REST; ++k) {
            const uint32_t m = __ballot_sync(FULL, d[k] > 1u);
            if (d[k] > 1u) list[total + __popc(m & ((1u << lane) - 1u))] = (uint32_t)(v0 + k * nth);
            total += __popc(m);
        }
        __syncwarp();
        for (uint32_t k0 = 0; k0 < total; k0 += 32u) {
            const uint32_t v = k0 + lane < total ? list[k0 + lane] : GCG_NO_SOURCE;
            const bool rest = v != GCG_NO_SOURCE && !below(parent, v, c);
            const uint32_t dv = rest ? nbr_count(n, v) : 0u;
            if (dv <= CC_THREAD_MAX)
                for (uint32_t i = i0; i < dv; ++i) link(parent, v, nbr_at(n, v, i));
            for (uint32_t m = __ballot_sync(FULL, dv > CC_THREAD_MAX); m; m &= m - 1u) {
                const int from = __ffs((int)m) - 1;
                const uint32_t u = __shfl_sync(FULL, v, from), du = __shfl_sync(FULL, dv, from);
                for (uint32_t i = i0 + lane; i < du; i += 32u) link(parent, u, nbr_at(n, u, i));
                __syncwarp();
            }
        }
        __syncwarp();
    }
}

/* Every vertex to its root, once before the sampling (SAMPLE) and once at the end, which
 * counts the roots in cnt[0]. What bounds the passes is that most paths lead through the
 * same few vertices, whose parents then come from one L2 slice, unless each SM keeps them
 * in its L1. Nothing hooks during this kernel, so a value an L1 holds from earlier in it is
 * still an ancestor, and a root is still a root: plain cached loads, and CC_ILP paths of
 * a thread climbed in step. There is no path halving here: a halving store racing with
 * another vertex's final store could put a non-root ancestor back. The only stores are
 * parent[v] = root(v) by v's own thread (258 -> 58 us before the sampling, 29 us at the end,
 * R-MAT scale 24). AGAIN: the same after the second round, if there
 * was one. The last block to finish takes the sample. */
template <bool SAMPLE, bool AGAIN>
__global__ void __launch_bounds__(256) k_cc_compress(const __grid_constant__ Nbrs n, uint32_t nv, uint32_t *parent,
                                                     uint32_t *cnt) {
    if (AGAIN && cnt[2] == 0u) return;
    uint32_t roots = 0;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v0 < nv; v0 += nth * CC_ILP) {
        uint32_t p[CC_ILP], q[CC_ILP];
#pragma unroll
        for (int k = 0; k < CC_ILP; ++k) {
            p[k] = v0 + k * nth < nv ? __ldca(parent + v0 + k * nth) : 0u; /* vertex 0 is a root */
            q[k] = p[k];
            if (!SAMPLE && v0 + k * nth < nv) roots += p[k] == (uint32_t)(v0 + k * nth);
        }
        for (bool more = true; more;) {
            more = false;
            uint32_t up[CC_ILP];
#pragma unroll
            for (int k = 0; k < CC_ILP; ++k) up[k] = __ldca(parent + q[k]);
#pragma unroll
            for (int k = 0; k < CC_ILP; ++k) {
                more |= up[k] != q[k];
                q[k] = up[k];
            }
        }
#pragma unroll
        for (int k = 0; k < CC_ILP; ++k)
            if (q[k] != p[k]) parent[v0 + k * nth] = q[k];
    }
    if constexpr (SAMPLE) {
        __shared__ uint32_t s_last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(cnt + 3, 1u) == gridDim.x - 1u;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        if (threadIdx.x == 0) cnt[3] = 0u;
        cc_sample(n, parent, nv, cnt);
    } else {
        __shared__ uint32_t s_roots[8];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) roots += __shfl_down_sync(0xFFFFFFFFu, roots, o);
        if ((threadIdx.x & 31u) == 0u) s_roots[threadIdx.x >> 5] = roots;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t w = 1; w < blockDim.x >> 5; ++w) roots += s_roots[w];
            if (roots) atomicAdd(cnt, roots);
        }
    }
}

}  // namespace
}  // namespace gcg

using namespace gcg;

extern "C" int gcg_connected_components(gcg_graph *g, uint32_t *labels, gcg_cc_stats *stats) {
    if (!g) return fail(GCG_ERR_INVALID, "gcg_connected_components: null graph");
    cudaStream_t s = g->stream;
    const uint32_t nv = g->nv;
    tbuf<uint32_t> parent_tmp, cnt;
    uint32_t *parent;
    const bool dev_out = labels && is_device_ptr(labels);
    if (dev_out) {
        parent = labels;
    } else {
        GCG_TRY(parent_tmp.alloc(nv, s));
        parent = parent_tmp.get();
    }
    /* sampling needs each vertex's whole neighbourhood: symmetric in-lists, or in + out lists */
    const bool sampled = nv > 0 && (g->symmetric || g->has_out);
    tbuf<uint32_t> minima;
    GCG_TRY(cnt.alloc(4, s));
    if (sampled) {
        GCG_TRY(minima.alloc(((size_t)nv + 31) / 32, s));
    } else { /* the edge pass walks the merge-path tiles */
        GCG_TRY(ensure_plan(g));
        GCG_CUDA(cudaMemsetAsync(cnt.get(), 0, 16, s));
    }
    const unsigned vb = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)nv + 255) / 256, (uint64_t)num_sms() * 8));
    cudaEvent_t ev0, ev1;
    GCG_CUDA(cudaEventCreate(&ev0));
    GCG_CUDA(cudaEventCreate(&ev1));
    GCG_CUDA(cudaEventRecord(ev0, s));
    if (sampled) {
        Nbrs nb;
        nb.rin = g->in_rowptr.get();
        nb.cin = g->in_col.get();
        nb.rout = g->symmetric ? nullptr : g->out_rowptr.get();
        nb.cout = g->symmetric ? nullptr : g->out_col.get();
        k_cc_first<<<vb, 256, 0, s>>>(nb, nv, parent, minima.get(), cnt.get());
        k_cc_minima<<<vb, 256, 0, s>>>(nb, nv, minima.get(), parent);
        /* fewer neighbours than vertices: the sample looks whether those that have any have enough */
        const Nbrs lists = (g->symmetric ? 1u : 2u) * g->ne > nv ? Nbrs{} : nb;
        k_cc_compress<true, false><<<vb, 256, 0, s>>>(lists, nv, parent, cnt.get());
        k_cc_second<<<vb, 256, 0, s>>>(nb, nv, cnt.get(), parent);
        k_cc_compress<true, true><<<vb, 256, 0, s>>>(Nbrs{}, nv, parent, cnt.get());
        k_cc_rest<<<vb, 256, 0, s>>>(nb, nv, cnt.get(), parent);
    } else {
        const PrPlan &pl = *g->plan;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cc_hook, MP_THREADS, 0) != cudaSuccess || per_sm <= 0) {
            cudaGetLastError();
            per_sm = 4;
        }
        const unsigned tb = (unsigned)std::max<uint32_t>(1, std::min<uint32_t>(pl.ntiles, (uint32_t)(num_sms() * per_sm)));
        k_cc_init<<<vb, 256, 0, s>>>(nv, parent);
        k_cc_hook<<<tb, MP_THREADS, 0, s>>>(g->in_rowptr.get(), g->in_col.get(), pl.tile_row.get(),
                                           pl.tile_edge.get(), pl.ntiles, parent);
    }
    k_cc_compress<false, false><<<vb, 256, 0, s>>>(Nbrs{}, nv, parent, cnt.get());
    GCG_LAUNCH_CHECK();
    GCG_CUDA(cudaEventRecord(ev1, s));
    uint32_t nroots = 0;
    GCG_CUDA(cudaMemcpyAsync(&nroots, cnt.get(), 4, cudaMemcpyDeviceToHost, s));
    if (labels && !dev_out) GCG_TRY(copy_out(labels, parent, (size_t)nv * 4, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    if (stats) {
        stats->passes = sampled ? 2 : 1;
        stats->ncomponents = nroots;
        stats->device_ms = ms;
    }
    return GCG_OK;
}

extern "C" int gcg_connected_components_ex(gcg_graph *g, const gcg_cc_params *p, uint32_t *labels,
                                           gcg_cc_stats *stats) {
    if (!g || !p) return fail(GCG_ERR_INVALID, "gcg_connected_components_ex: null argument");
    if (p->algorithm == GCG_CC_UNION_FIND) return gcg_connected_components(g, labels, stats);
    if (p->algorithm != GCG_CC_LABEL_PROPAGATION)
        return fail(GCG_ERR_INVALID, "gcg_connected_components_ex: unknown algorithm");
    const int iters = p->max_iterations > 0 ? p->max_iterations : 1000;
    return cc_label_propagation(g, p->scheduler, iters, labels, stats, p->frontier_log);
}
