/*
 * Device radix sort and scan: the B200 replacement of the sharder's shovel sort
 * (stable LSD radix sort with 8-bit digits, src/util/radixSort.hpp:50-116, used by
 * shard_flushinfo::flush sharder.hpp:192 and finish_shard sharder.hpp:640).
 *
 * Design (HBM traffic and instruction issue bound it, no tensor cores): one read
 * of the keys counts the digits of every pass; each pass is then one kernel that
 * reads and writes each key once. A tile's place in the output is found by a
 * decoupled look-back over the tiles before it, one thread per digit, while the
 * tile's keys wait in shared memory grouped by digit.
 */
#include <algorithm>

#include "gcg_internal.cuh"

namespace gcg {

namespace {

/* 256 threads x 22 keys, three blocks on an SM: 3 % faster over a build of 67 M edges than 4
 * blocks of 256 x 16 or 2 of 512 x 16 (shorter runs, or fewer phases that overlap). */
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 22;
constexpr int RS_BLOCKS = 3;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_RADIX = 256;
constexpr int RS_PASSES = RadixPlan::MAX_PASSES;
constexpr int RS_SPIN = 1 << 14;   /* polls of one tile's count before it is counted again */
constexpr int RS_RECOUNT = -1;     /* in their place: every count is taken again (a test's) */
constexpr int RS_GROUP = 16;     /* tiles that share a group word */

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

/* Digit counts of every pass from one read of the keys: counts[p][digit]. Bound
 * by the shared-memory atomics (67 M keys, 6 passes: 184 us). */
__global__ void __launch_bounds__(RadixCounter::THREADS) rs_count(const uint64_t *__restrict__ keys, uint64_t n,
                                                                  RadixPlan pl, uint32_t *__restrict__ counts) {
    __shared__ RadixCounter cnt;
    cnt.clear();
    constexpr int ITEMS = 8;
    constexpr uint64_t CH = (uint64_t)RadixCounter::THREADS * ITEMS;
    for (uint64_t c0 = blockIdx.x * CH; c0 < n; c0 += gridDim.x * CH) {
        uint64_t k[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint64_t i = c0 + (uint64_t)j * RadixCounter::THREADS + threadIdx.x;
            k[j] = i < n ? __ldg(keys + i) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (c0 + (uint64_t)j * RadixCounter::THREADS + threadIdx.x >= n) break;
            cnt.add(pl, k[j]);
        }
    }
    cnt.flush(pl, counts);
}

/* State words: the pass that wrote it and the status in the high half, a count
 * in the low half. The tag makes the words of an earlier pass read as absent, so
 * they are cleared once per sort. The word is all a reader takes from the writer,
 * so relaxed accesses do. */
constexpr uint32_t ST_AGG = 1u, ST_INC = 2u;
__device__ __forceinline__ void st_put(unsigned long long *p, uint32_t tag, uint32_t val) {
    const unsigned long long w = ((unsigned long long)tag << 32) | val;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long st_get(const unsigned long long *p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

struct RsPass {
    const uint64_t *in;
    uint64_t *out;
    uint64_t n;
    int shift, bits;
    uint32_t tag; /* pass number * 4, from 4 */
    int spin;     /* RS_SPIN or RS_RECOUNT */
    const uint32_t *counts;
    uint32_t *ticket;
    unsigned long long *tile;  /* [tile][digit]: keys of the digit in the tile, or up to its end */
    unsigned long long *group; /* [group][digit]: the same of RS_GROUP tiles */
};

/* keys of digit d among in[lo, hi): what a look-back falls back on when a word
 * does not come, so that the result needs no wait (tiles start in ticket order:
 * it does come) */
__device__ __noinline__ uint32_t rs_recount(const uint64_t *in, uint64_t lo, uint64_t hi, int shift, uint32_t dmask,
                                            uint32_t d) {
    uint32_t c = 0;
    for (uint64_t i = lo; i < hi; ++i) c += ((uint32_t)(in[i] >> shift) & dmask) == d;
    return c;
}

/* One pass. Warp w of a tile owns the contiguous keys [w*WSEG, (w+1)*WSEG) and
 * reads them as RS_ITEMS coalesced rounds of 32; keeping each warp's keys
 * contiguous lets it rank them with counters of its own and stay stable (tile
 * order = warp order, then round, then lane).
 *
 * The look-back goes over the tiles of the own group, then over whole groups.
 * All tiles of a wave count their digits at about the same time, so a look-back
 * by single tiles would have the whole wave to walk. Bound by the shared-memory
 * pipe (75% busy: random digits' bank conflicts), then by the votes on the integer
 * pipe, not by HBM: 67 M keys take 0.36 ms for 1.07 GB; a pass as three steps
 * (count per tile, scan, scatter) took 0.59. BITS >= the digit's width. */
constexpr int RS_WSEG = RS_TILE / RS_WARPS;
constexpr size_t RS_SMEM = (size_t)RS_TILE * 8 + (size_t)RS_WARPS * RS_RADIX * 4 + RS_RADIX * 4 + 64;
template <int BITS>
__global__ void __launch_bounds__(RS_THREADS, RS_BLOCKS) rs_pass(RsPass a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint64_t *s_keys = reinterpret_cast<uint64_t *>(s_raw);
    uint32_t(*s_wcnt)[RS_RADIX] = reinterpret_cast<uint32_t(*)[RS_RADIX]>(s_keys + RS_TILE);
    uint32_t *s_gofs = &s_wcnt[RS_WARPS][0];
    uint32_t *s_scan = s_gofs + RS_RADIX;
    __shared__ uint32_t s_tile;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t dmask = (1u << a.bits) - 1u;
    if (tid == 0) s_tile = atomicAdd(a.ticket, 1u);
    for (uint32_t i = tid; i < RS_WARPS * RS_RADIX; i += RS_THREADS) (&s_wcnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t t = s_tile;
    const uint64_t base = (uint64_t)t * RS_TILE;
    const uint32_t tile_n = (a.n - base) < (uint64_t)RS_TILE ? (uint32_t)(a.n - base) : (uint32_t)RS_TILE;
    const uint32_t w0 = warp * RS_WSEG + lane; /* this lane's first key of the tile */
    const uint64_t *in = a.in + base;

    /* places past the end hold all-ones keys: last in order and of the highest
     * digit, they rank behind every key of the tile */
    uint64_t key[RS_ITEMS];
    if (tile_n == (uint32_t)RS_TILE) {
#pragma unroll
        for (int k = 0; k < RS_ITEMS; ++k) key[k] = __ldg(in + w0 + k * 32);
    } else {
#pragma unroll
        for (int k = 0; k < RS_ITEMS; ++k) key[k] = (w0 + k * 32 < tile_n) ? __ldg(in + w0 + k * 32) : ~0ull;
    }

    /* warp-private ranking over the warp's rounds, in key order */
    uint32_t lrank[RS_ITEMS / 2]; /* two 16-bit ranks in each */
    uint32_t *wcnt = s_wcnt[warp];
#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        const uint32_t d = (uint32_t)(key[k] >> a.shift) & dmask;
        /* lanes holding another digit, from one vote per digit bit (cheaper here
         * than __match_any_sync, which competes with the shared-memory traffic) */
        uint32_t others = 0;
#pragma unroll
        for (int b = 0; b < BITS; ++b) {
            uint32_t vote, mine; /* written out: the compiler's form takes half as many instructions again */
            asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
                         "and.b32 t, %2, %3;\n\tsetp.ne.u32 p, t, 0;\n\t"
                         "vote.sync.ballot.b32 %0, p, 0xffffffff;\n\tselp.b32 %1, -1, 0, p;\n\t}"
                         : "=r"(vote), "=r"(mine)
                         : "r"(d), "r"(1 << b));
            others |= vote ^ mine;
        }
        const uint32_t before = wcnt[d];
        const uint32_t below = __popc(~others & lanemask_lt());
        if (k & 1) lrank[k / 2] |= (before + below) << 16;
        else lrank[k / 2] = before + below;
        __syncwarp();
        if (below == 0) wcnt[d] = before + 32u - __popc(others);
        __syncwarp();
    }
    __syncthreads();

    /* thread d: digit d's keys in this tile, published before anything else */
    uint32_t total = 0, lstart = 0, excl = 0;
    if (tid < RS_RADIX) {
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) total += s_wcnt[w][tid];
        const uint32_t held = total; /* with the places past the end */
        if (tid == dmask) total -= (uint32_t)RS_TILE - tile_n;
        if (t > 0) st_put(a.tile + (uint64_t)t * RS_RADIX + tid, a.tag | ST_AGG, total);
        uint32_t v = held;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if (lane >= (uint32_t)o) v += y;
        }
        if (lane == 31) s_scan[warp] = v;
        lstart = v - held;
        if (t == 0) { /* keys of the digits below d in all tiles: every later tile gets it from here */
            const uint32_t c = __ldg(a.counts + tid);
            v = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
                if (lane >= (uint32_t)o) v += y;
            }
            if (lane == 31) s_scan[RS_RADIX / 32 + warp] = v;
            excl = v - c;
        }
    }
    __syncthreads();
    if (tid < RS_RADIX) {
#pragma unroll
        for (uint32_t w = 0; w < RS_RADIX / 32; ++w) {
            lstart += w < warp ? s_scan[w] : 0u;
            if (t == 0) excl += w < warp ? s_scan[RS_RADIX / 32 + w] : 0u;
        }
        if (t == 0) st_put(a.tile + tid, a.tag | ST_INC, excl + total);
        /* digit-major offsets: digit d's keys of warp w start after those of warps < w */
        uint32_t run = lstart;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t c = s_wcnt[w][tid];
            s_wcnt[w][tid] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        const uint32_t d = (uint32_t)(key[k] >> a.shift) & dmask;
        s_keys[wcnt[d] + ((k & 1) ? lrank[k / 2] >> 16 : lrank[k / 2] & 0xFFFFu)] = key[k];
    }

    /* excl: keys of digit d in the tiles before this one, and of the digits below
     * d in all of them */
    if (tid < RS_RADIX) {
        const uint32_t g = t / RS_GROUP, in_g = t % RS_GROUP, pass = a.tag >> 2;
        /* a word, waited for, or else what it would hold; true: it reaches back to the start */
        auto take = [&](const unsigned long long *p, unsigned long long w, uint64_t lo, uint64_t hi) {
            for (int spin = 0; (uint32_t)(w >> 34) != pass && spin < a.spin; ++spin) w = st_get(p);
            if ((uint32_t)(w >> 34) == pass && a.spin >= 0) {
                excl += (uint32_t)w;
                return (uint32_t)(w >> 32) == (a.tag | ST_INC);
            }
            excl += rs_recount(a.in, lo * RS_TILE, hi * RS_TILE, a.shift, dmask, tid);
            if (lo == 0)
                for (uint32_t d = 0; d < tid; ++d) excl += __ldg(a.counts + d);
            return lo == 0;
        };
        bool found = t == 0;
        if (in_g) {
            const unsigned long long *p = a.tile + (uint64_t)(g * RS_GROUP) * RS_RADIX + tid;
            unsigned long long w[RS_GROUP - 1];
#pragma unroll
            for (int i = 0; i < RS_GROUP - 1; ++i) w[i] = i < (int)in_g ? st_get(p + i * RS_RADIX) : 0ull;
#pragma unroll
            for (int i = RS_GROUP - 2; i >= 0; --i)
                if (i < (int)in_g && !found)
                    found = take(p + i * RS_RADIX, w[i], (uint64_t)g * RS_GROUP + i, (uint64_t)g * RS_GROUP + i + 1);
        }
        unsigned long long *own = a.group + (uint64_t)g * RS_RADIX + tid;
        const bool last = in_g == RS_GROUP - 1;
        if (last && !found) st_put(own, a.tag | ST_AGG, excl + total);
        constexpr int WIN = 8;
        for (int64_t j = (int64_t)g - 1; !found; j -= WIN) { /* group 0's word reaches back to the start */
            const unsigned long long *p = a.group + (uint64_t)j * RS_RADIX + tid;
            unsigned long long w[WIN];
#pragma unroll
            for (int i = 0; i < WIN; ++i) w[i] = j >= i ? st_get(p - i * RS_RADIX) : 0ull;
#pragma unroll
            for (int i = 0; i < WIN; ++i)
                if (j >= i && !found)
                    found = take(p - i * RS_RADIX, w[i], (uint64_t)(j - i) * RS_GROUP,
                                 (uint64_t)(j - i + 1) * RS_GROUP);
        }
        if (t > 0) st_put(a.tile + (uint64_t)t * RS_RADIX + tid, a.tag | ST_INC, excl + total);
        if (last) st_put(own, a.tag | ST_INC, excl + total);
        /* tile position i of digit d goes to excl + (i - lstart[d]); uint32
         * wrap-around is exact: every index is below 2^32 */
        s_gofs[tid] = excl - lstart;
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = tid; i < tile_n; i += RS_THREADS) {
        const uint64_t kk = s_keys[i];
        const uint32_t d = (uint32_t)(kk >> a.shift) & dmask;
        a.out[(uint32_t)(s_gofs[d] + i)] = kk;
    }
}

/* ---- scan -------------------------------------------------------------- */

constexpr int SC_THREADS = 256;
constexpr int SC_ITEMS = 16;
constexpr int SC_TILE = SC_THREADS * SC_ITEMS;

/* Block-wide exclusive scan of one uint32 per thread (SC_THREADS threads). */
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t *s_warp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = (lane < (SC_THREADS / 32)) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < (SC_THREADS / 32)) s_warp[lane] = w;
    }
    __syncthreads();
    uint32_t before = warp ? s_warp[warp - 1] : 0u;
    return before + v - x;
}

__global__ void __launch_bounds__(SC_THREADS) sc_reduce(const uint32_t *__restrict__ in, uint64_t n,
                                                        uint32_t *__restrict__ sums) {
    __shared__ uint32_t s_warp[SC_THREADS / 32];
    const uint64_t base = (uint64_t)blockIdx.x * SC_TILE;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        uint64_t i = base + (uint64_t)k * SC_THREADS + threadIdx.x;
        if (i < n) s += in[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < SC_THREADS / 32; ++w) t += s_warp[w];
        sums[blockIdx.x] = t;
    }
}

/* Exclusive scan of one tile with a carried-in offset (offsets[blockIdx] or 0). */
__global__ void __launch_bounds__(SC_THREADS) sc_scan_tile(const uint32_t *in, uint32_t *out, uint64_t n,
                                                           const uint32_t *__restrict__ block_off,
                                                           uint32_t *total) {
    __shared__ uint32_t s_v[SC_TILE];
    __shared__ uint32_t s_warp[SC_THREADS / 32];
    const uint64_t base = (uint64_t)blockIdx.x * SC_TILE;
    const int tid = threadIdx.x;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        uint64_t i = base + (uint64_t)k * SC_THREADS + tid;
        s_v[k * SC_THREADS + tid] = (i < n) ? in[i] : 0u;
    }
    __syncthreads();
    uint32_t loc[SC_ITEMS];
    uint32_t t = 0;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        loc[k] = t;
        t += s_v[tid * SC_ITEMS + k];
    }
    uint32_t pre = block_excl_scan(t, s_warp);
    uint32_t off = block_off ? block_off[blockIdx.x] : 0u;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) s_v[tid * SC_ITEMS + k] = off + pre + loc[k];
    if (total && tid == SC_THREADS - 1 && (uint64_t)(blockIdx.x + 1) * SC_TILE >= n) *total = off + pre + t;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        uint64_t i = base + (uint64_t)k * SC_THREADS + tid;
        if (i < n) out[i] = s_v[k * SC_THREADS + tid];
    }
}

/* ---- merge of two sorted runs (merge path) ------------------------------ */

constexpr int MG_THREADS = 256;
constexpr int MG_ITEMS = 8; /* pairwise merges of the piecewise sort */
constexpr int MG_TILE = MG_THREADS * MG_ITEMS;
constexpr int MF_ITEMS = 16; /* the fused last merge: larger tiles hide its per-tile latency */
constexpr int MF_TILE = MG_THREADS * MF_ITEMS;

/* Tiles are staged in shared memory with one pad slot after every ITEMS keys, so
 * the ITEMS consecutive keys a thread writes after merging fall on distinct banks. */
template <int ITEMS>
__device__ __forceinline__ uint32_t padx(uint32_t e) { return e + e / ITEMS; }

template <int ITEMS>
struct SView { /* keys [off, off + n) of a padded tile */
    const uint64_t *s;
    uint32_t off;
    __device__ __forceinline__ uint64_t operator[](uint32_t i) const { return s[padx<ITEMS>(off + i)]; }
};

/* how many of the first diag outputs come from a (a first on equal keys) */
template <typename A, typename B, typename I>
__device__ __forceinline__ I merge_path(const A &a, I na, const B &b, I nb, I diag) {
    I lo = diag > nb ? diag - nb : 0, hi = diag < na ? diag : na;
    while (lo < hi) {
        const I mid = (lo + hi) >> 1;
        if (a[mid] <= b[diag - 1 - mid]) lo = mid + 1; else hi = mid;
    }
    return lo;
}

/* split[t] = a's share of the first t*TILE outputs, t = 0..ntiles */
template <int TILE>
__global__ void k_merge_split(const uint64_t *__restrict__ a, uint64_t na, const uint64_t *__restrict__ b,
                              uint64_t nb, uint64_t ntiles, uint64_t *__restrict__ split) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t <= ntiles;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t d = t * TILE < na + nb ? t * TILE : na + nb;
        split[t] = merge_path(a, na, b, nb, d);
    }
}

/* Stages a tile's pieces a[a0, a0+la) and b[b0, b0+lb) in s, merges them (each
 * thread ITEMS outputs from its own merge-path split) and leaves the merged tile
 * in s (padded); v[k] = merged output dg + k of this thread. */
template <int ITEMS>
__device__ __forceinline__ void tile_merge(const uint64_t *__restrict__ a, uint64_t a0, uint32_t la,
                                           const uint64_t *__restrict__ b, uint64_t b0, uint32_t lb, uint64_t *s,
                                           uint64_t (&v)[ITEMS], uint32_t &dg) {
    const uint32_t tot = la + lb;
    for (uint32_t i = threadIdx.x; i < la; i += MG_THREADS) s[padx<ITEMS>(i)] = a[a0 + i];
    for (uint32_t i = threadIdx.x; i < lb; i += MG_THREADS) s[padx<ITEMS>(la + i)] = b[b0 + i];
    __syncthreads();
    const SView<ITEMS> sa{s, 0}, sb{s, la};
    dg = threadIdx.x * ITEMS < tot ? threadIdx.x * ITEMS : tot;
    uint32_t i = merge_path(sa, la, sb, lb, dg), j = dg - i;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        v[k] = 0;
        if (dg + k < tot) {
            const bool take_a = i < la && (j >= lb || sa[i] <= sb[j]);
            v[k] = take_a ? sa[i] : sb[j];
            if (take_a) ++i; else ++j;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
        if (dg + k < tot) s[padx<ITEMS>(dg + k)] = v[k];
    __syncthreads();
}

/* One output tile per block, written back with coalesced stores. */
__global__ void __launch_bounds__(MG_THREADS) k_merge_u64(const uint64_t *__restrict__ a, uint64_t na,
                                                          const uint64_t *__restrict__ b, uint64_t nb,
                                                          const uint64_t *__restrict__ split,
                                                          uint64_t *__restrict__ out) {
    __shared__ uint64_t s_in[MG_TILE + MG_TILE / MG_ITEMS];
    const uint64_t n = na + nb;
    const uint64_t d0 = (uint64_t)blockIdx.x * MG_TILE;
    const uint64_t d1 = d0 + MG_TILE < n ? d0 + MG_TILE : n;
    const uint64_t a0 = split[blockIdx.x], a1 = split[blockIdx.x + 1];
    const uint64_t b0 = d0 - a0, b1 = d1 - a1;
    const uint32_t la = (uint32_t)(a1 - a0), lb = (uint32_t)(b1 - b0), tot = la + lb;
    uint64_t v[MG_ITEMS];
    uint32_t dg;
    tile_merge<MG_ITEMS>(a, a0, la, b, b0, lb, s_in, v, dg);
    for (uint32_t x = threadIdx.x; x < tot; x += MG_THREADS) out[d0 + x] = s_in[padx<MG_ITEMS>(x)];
}

/* ---- merge + unique + CSR in one pass ------------------------------------
 * The last merge of the sharder's sorted runs, the duplicate filter, the
 * compaction offsets and the CSR decode fused: each block merges one tile of
 * MF_TILE outputs (as k_merge_u64), flags the keys to keep, and finds where its
 * kept keys start in the output by a decoupled look-back over the tiles before
 * it (tiles are taken in ticket order, so a block only waits on blocks that are
 * already running; every wait is bounded and sets an error flag on expiry).
 * It then writes the column of every kept key, the row pointers of the rows
 * its keys open, optionally the kept keys themselves, and takes duplicates off
 * the raw out-degree counts. */
static_assert(MG_THREADS == SC_THREADS, "block_excl_scan is sized for SC_THREADS");
constexpr long long LB_SPIN = 1ll << 22;
constexpr uint32_t LB_GROUP = 32; /* tiles that share a group word */

struct FinishArgs {
    const uint64_t *a, *b;
    uint64_t na, nb, kept;
    const uint64_t *split;
    uint32_t kbits, nv;
    int dedup;
    uint32_t *rowptr, *col;
    uint64_t *keys_out;   /* kept keys, or null */
    uint32_t *outdeg_dup; /* raw out-degree counts to take duplicates off, or null */
    uint32_t *ticket;
    unsigned long long *tstate, *gstate; /* per tile; per group of tiles */
    uint32_t *total;
    int *err;
};

/* Exclusive prefix of tile t's kept keys, by one warp that publishes the tile's
 * own count and prefix: over the tiles of its group of 32 first, then over whole
 * groups, 32 at a time. All tiles of a wave count their keys at about the same
 * time: by single tiles the walk took a step per 32 of them. */
__device__ __forceinline__ uint32_t look_back(const FinishArgs &f, uint32_t t, uint32_t tile_sum, uint32_t lane) {
    const uint32_t g = t / LB_GROUP, in_g = t % LB_GROUP;
    const bool last = in_g == LB_GROUP - 1;
    uint32_t excl = 0;
    /* adds p[0], p[-1], .. p[-(n-1)] up to the first that reaches back to the start */
    auto walk = [&](const unsigned long long *p, uint32_t n) {
        unsigned long long w = 0;
        if (lane < n) {
            long long spin = 0;
            do {
                w = st_get(p - lane);
            } while ((w >> 32) == 0 && ++spin < LB_SPIN);
            if ((w >> 32) == 0) atomicExch(f.err, 1);
        }
        const uint32_t inc = __ballot_sync(0xFFFFFFFFu, (uint32_t)(w >> 32) == ST_INC);
        const uint32_t stop = inc ? (uint32_t)(__ffs(inc) - 1) : 31u;
        excl += __reduce_add_sync(0xFFFFFFFFu, lane <= stop ? (uint32_t)w : 0u);
        return inc != 0;
    };
    if (lane == 0) st_put(f.tstate + t, t == 0 ? ST_INC : ST_AGG, tile_sum);
    bool found = t == 0;
    if (in_g) found = walk(f.tstate + t - 1, in_g);
    if (lane == 0 && last && !found) st_put(f.gstate + g, ST_AGG, excl + tile_sum);
    for (int64_t j = (int64_t)g - 1; !found && j >= 0; j -= 32)
        found = walk(f.gstate + j, j + 1 < 32 ? (uint32_t)(j + 1) : 32u);
    if (lane == 0) {
        st_put(f.tstate + t, ST_INC, excl + tile_sum);
        if (last) st_put(f.gstate + g, ST_INC, excl + tile_sum);
    }
    return excl;
}

__global__ void __launch_bounds__(MG_THREADS, 4) k_merge_finish(FinishArgs f) {
    __shared__ uint64_t s_in[MF_TILE + MF_TILE / MF_ITEMS];
    __shared__ uint32_t s_warp[MG_THREADS / 32];
    __shared__ uint32_t s_tile, s_excl, s_sum;
    if (threadIdx.x == 0) s_tile = atomicAdd(f.ticket, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    const uint64_t n = f.na + f.nb;
    const uint64_t d0 = (uint64_t)t * MF_TILE;
    const uint64_t d1 = d0 + MF_TILE < n ? d0 + MF_TILE : n;
    const uint64_t a0 = f.split[t], a1 = f.split[t + 1];
    const uint64_t b0 = d0 - a0, b1 = d1 - a1;
    const uint32_t la = (uint32_t)(a1 - a0), lb = (uint32_t)(b1 - b0), tot = la + lb;
    uint64_t v[MF_ITEMS];
    uint32_t dg;
    tile_merge<MF_ITEMS>(f.a, a0, la, f.b, b0, lb, s_in, v, dg);
    /* the key before this thread's first: the previous thread's last, or the
     * previous tile's last (the larger of the last a and b keys before it) */
    uint64_t prev = 0;
    if (threadIdx.x == 0) {
        if (d0 > 0) {
            const uint64_t x = a0 ? f.a[a0 - 1] : 0ull, y = b0 ? f.b[b0 - 1] : 0ull;
            prev = x > y ? x : y;
        }
    } else if (dg > 0) {
        prev = s_in[padx<MF_ITEMS>(dg - 1)];
    }
    uint32_t fl = 0, cnt = 0;
    {
        uint64_t pk = prev;
#pragma unroll
        for (int k = 0; k < MF_ITEMS; ++k) {
            const uint64_t gi = d0 + dg + k;
            if (dg + k < tot && gi < f.kept) {
                const bool keep = !f.dedup || gi == 0 || v[k] != pk;
                fl |= (keep ? 1u : 0u) << k;
                cnt += keep ? 1u : 0u;
            }
            pk = v[k];
        }
    }
    const uint32_t local = block_excl_scan(cnt, s_warp);
    if (threadIdx.x == MG_THREADS - 1) s_sum = local + cnt;
    __syncthreads();
    const uint32_t tile_sum = s_sum;
    if (threadIdx.x < 32) {
        const uint32_t excl = look_back(f, t, tile_sum, threadIdx.x);
        if (threadIdx.x == 0) s_excl = excl;
    }
    __syncthreads();
    const uint64_t mask = (f.kbits >= 64) ? ~0ull : ((1ull << f.kbits) - 1ull);
    const uint32_t base = s_excl;
    /* the kept keys, compacted in shared memory (the merged tile is no longer
     * read), then written out with coalesced stores; row pointers and repeat
     * counts from the thread that holds the key */
    uint32_t q = local;
    uint64_t pk = prev;
#pragma unroll
    for (int k = 0; k < MF_ITEMS; ++k) {
        const uint64_t gi = d0 + dg + k;
        if (dg + k < tot && gi < f.kept) {
            const uint64_t key = v[k];
            const uint32_t row = (uint32_t)(key >> f.kbits);
            if ((fl >> k) & 1u) {
                s_in[padx<MF_ITEMS>(q)] = key;
                const int64_t prow = gi == 0 ? -1 : (int64_t)(pk >> f.kbits);
                for (int64_t r = prow + 1; r <= (int64_t)row; ++r) f.rowptr[r] = base + q;
                ++q;
            } else if (f.outdeg_dup) {
                atomicSub(f.outdeg_dup + (uint32_t)(key & mask), 1u);
            }
            if (gi == f.kept - 1) { /* rows after the last key end at the total */
                for (uint64_t r = (uint64_t)row + 1; r <= f.nv; ++r) f.rowptr[r] = base + q;
                *f.total = base + q;
            }
        }
        pk = v[k];
    }
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < tile_sum; x += MG_THREADS) {
        const uint64_t key = s_in[padx<MF_ITEMS>(x)];
        f.col[base + x] = (uint32_t)(key & mask);
        if (f.keys_out) f.keys_out[base + x] = key;
    }
}

/* The same from one sorted run (nothing to merge), in two passes of independent
 * warps: the kept keys of every 512 are counted, scanned, and written at their
 * places. The second read of the keys costs less than a look-back and merged
 * tiles staged in shared memory (67 M keys: 540 us through the merging kernel,
 * 568 in one pass with a look-back, 330 as two). */
constexpr int FR_ITEMS = 16;
constexpr int FR_WSEG = 32 * FR_ITEMS;

__global__ void __launch_bounds__(256) k_run_count(const uint64_t *__restrict__ keys, uint64_t n, uint32_t nseg,
                                                   uint32_t *__restrict__ cnt) {
    const uint32_t w = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (w >= nseg) return;
    const uint64_t i0 = (uint64_t)w * FR_WSEG + lane;
    uint32_t c = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint64_t key[FR_ITEMS / 2], prev[FR_ITEMS / 2];
#pragma unroll
        for (int k = 0; k < FR_ITEMS / 2; ++k) {
            const uint64_t i = i0 + (h * (FR_ITEMS / 2) + k) * 32;
            key[k] = i < n ? __ldg(keys + i) : 0ull;
            prev[k] = i < n && i > 0 ? __ldg(keys + i - 1) : ~key[k]; /* the first key is kept */
        }
#pragma unroll
        for (int k = 0; k < FR_ITEMS / 2; ++k)
            c += i0 + (h * (FR_ITEMS / 2) + k) * 32 < n && key[k] != prev[k] ? 1u : 0u;
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if (lane == 0) cnt[w] = c;
}

/* Empty rows are filled by the thread that opens the next one. SPARSE (few keys for the rows):
 * from this many on by its warp together (32 M vertices with 1,000 edges: a build of 19.7 ms
 * with the threads alone, 2.5 so; the same code costs a full graph 2 % of its build) */
constexpr uint32_t FR_GAP = 32;
constexpr uint64_t FR_SPARSE = 4; /* rows per key */
__device__ __forceinline__ void fill_rows(uint32_t *rowptr, uint32_t r0, uint32_t r1, uint32_t at) {
    for (uint64_t r = (uint64_t)r0 + (threadIdx.x & 31u); r <= r1; r += 32u) rowptr[r] = at;
}

/* first[w]: where the kept keys of segment w go; without duplicates to drop
 * (dedup 0, first null) every key stays where it is */
template <bool SPARSE>
__global__ void __launch_bounds__(256, 4) k_run_write(FinishArgs f, uint32_t nseg, const uint32_t *__restrict__ first) {
    const uint32_t w = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (w >= nseg) return;
    const uint64_t i0 = (uint64_t)w * FR_WSEG + lane;
    const uint32_t mask = (uint32_t)((1ull << f.kbits) - 1ull);
    uint32_t q = first ? __ldg(first + w) : w * FR_WSEG;
    RunCounts<-1> off; /* repeats, off their sources' counts */
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        uint64_t key[FR_ITEMS / 2], prev[FR_ITEMS / 2];
#pragma unroll
        for (int k = 0; k < FR_ITEMS / 2; ++k) {
            const uint64_t i = i0 + (h * (FR_ITEMS / 2) + k) * 32;
            key[k] = i < f.kept ? __ldg(f.a + i) : 0ull;
            prev[k] = i < f.kept && i > 0 ? __ldg(f.a + i - 1) : ~key[k];
        }
#pragma unroll
        for (int k = 0; k < FR_ITEMS / 2; ++k) {
            const uint64_t i = i0 + (h * (FR_ITEMS / 2) + k) * 32;
            const bool kp = i < f.kept && (!f.dedup || key[k] != prev[k]);
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, kp);
            const uint32_t at = q + __popc(b & lanemask_lt());
            q += __popc(b);
            const uint32_t row = (uint32_t)(key[k] >> f.kbits), prow = (uint32_t)(prev[k] >> f.kbits);
            const uint32_t col = (uint32_t)key[k] & mask;
            const uint32_t r0 = i == 0 ? 0u : prow + 1u; /* the first row that this key opens, when it opens one */
            bool wide = false;
            if (kp) {
                f.col[at] = col;
                if (f.keys_out) f.keys_out[at] = key[k];
                if (i == 0 || row != prow) { /* empty rows, then its own */
                    wide = SPARSE && row - r0 >= FR_GAP;
                    if (!wide)
                        for (uint32_t r = r0; r <= row; ++r) f.rowptr[r] = at;
                }
            }
            if constexpr (SPARSE)
                for (uint32_t m = __ballot_sync(0xFFFFFFFFu, wide); m; m &= m - 1u) {
                    const int l = __ffs((int)m) - 1;
                    fill_rows(f.rowptr, __shfl_sync(0xFFFFFFFFu, r0, l), __shfl_sync(0xFFFFFFFFu, row, l),
                              __shfl_sync(0xFFFFFFFFu, at, l));
                }
            const uint32_t dups = f.outdeg_dup ? __ballot_sync(0xFFFFFFFFu, i < f.kept && !kp) : 0u;
            if (dups) off.take(f.outdeg_dup, b | 1u, dups, col);
        }
    }
    off.flush(f.outdeg_dup);
    if (w == nseg - 1u) { /* rows after the last key end at the total */
        fill_rows(f.rowptr, (uint32_t)(__ldg(f.a + f.kept - 1) >> f.kbits) + 1u, f.nv, q);
        if (lane == 0) *f.total = q;
    }
}

}  // namespace

int merge_u64(const uint64_t *a, uint64_t na, const uint64_t *b, uint64_t nb, uint64_t *out, cudaStream_t s) {
    const uint64_t n = na + nb;
    if (n == 0) return GCG_OK;
    if (na == 0 || nb == 0) {
        GCG_CUDA(cudaMemcpyAsync(out, na ? a : b, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s));
        return GCG_OK;
    }
    const uint64_t ntiles = (n + MG_TILE - 1) / MG_TILE;
    if (ntiles >= 0x7FFFFFFFull) return fail(GCG_ERR_UNSUPPORTED, "merge: too many keys");
    tbuf<uint64_t> split;
    GCG_TRY(split.alloc(ntiles + 1, s));
    k_merge_split<MG_TILE><<<(unsigned)std::min<uint64_t>((ntiles + 256) / 256, (uint64_t)num_sms() * 8), 256, 0, s>>>(
        a, na, b, nb, ntiles, split.get());
    k_merge_u64<<<(unsigned)ntiles, MG_THREADS, 0, s>>>(a, na, b, nb, split.get(), out);
    GCG_LAUNCH_CHECK();
    return GCG_OK;
}

int merge_unique_csr(const uint64_t *a, uint64_t na, const uint64_t *b, uint64_t nb, uint64_t kept, bool dedup,
                     uint32_t kbits, uint32_t nv, uint32_t *rowptr, uint32_t *col, uint64_t *keys_out,
                     uint32_t *outdeg_dup, uint64_t *ne, cudaStream_t s) {
    *ne = 0;
    if (kept == 0) {
        GCG_CUDA(cudaMemsetAsync(rowptr, 0, ((size_t)nv + 1) * 4, s));
        return GCG_OK;
    }
    const uint64_t n = na + nb;
    if (kept > n || kept > 0xFFFFFFFFull) return fail(GCG_ERR_INVALID, "merge_unique_csr: bad key count");
    const bool one_run = na == 0 || nb == 0;
    tbuf<uint64_t> split;
    tbuf<unsigned long long> tstate;
    tbuf<uint32_t> seg, ctl; /* ctl: ticket, total, err */
    GCG_TRY(ctl.alloc(3, s));
    GCG_CUDA(cudaMemsetAsync(ctl.get(), 0, 3 * sizeof(uint32_t), s));
    FinishArgs f = {};
    f.a = na ? a : b;
    f.b = b;
    f.na = na;
    f.nb = nb;
    f.kept = kept;
    f.kbits = kbits;
    f.nv = nv;
    f.dedup = dedup ? 1 : 0;
    f.rowptr = rowptr;
    f.col = col;
    f.keys_out = keys_out;
    f.outdeg_dup = outdeg_dup;
    f.ticket = ctl.get();
    f.total = ctl.get() + 1;
    f.err = (int *)(ctl.get() + 2);
    if (one_run) {
        const uint32_t nseg = (uint32_t)((kept + FR_WSEG - 1) / FR_WSEG), blocks = (nseg + 7) / 8;
        if (dedup) {
            GCG_TRY(seg.alloc(nseg, s));
            k_run_count<<<blocks, 256, 0, s>>>(f.a, kept, nseg, seg.get());
            GCG_LAUNCH_CHECK();
            GCG_TRY(scan_u32(seg.get(), seg.get(), nseg, nullptr, s));
        }
        if (nv > FR_SPARSE * kept) k_run_write<true><<<blocks, 256, 0, s>>>(f, nseg, seg.get());
        else k_run_write<false><<<blocks, 256, 0, s>>>(f, nseg, seg.get());
    } else {
        const uint64_t ntiles = (kept + MF_TILE - 1) / MF_TILE, nwords = ntiles + ntiles / LB_GROUP + 1;
        GCG_TRY(split.alloc(ntiles + 1, s));
        GCG_TRY(tstate.alloc(nwords, s));
        GCG_CUDA(cudaMemsetAsync(tstate.get(), 0, nwords * sizeof(unsigned long long), s));
        k_merge_split<MF_TILE>
            <<<(unsigned)std::min<uint64_t>((ntiles + 256) / 256, (uint64_t)num_sms() * 8), 256, 0, s>>>(
                a, na, b, nb, ntiles, split.get());
        f.split = split.get();
        f.tstate = tstate.get();
        f.gstate = tstate.get() + ntiles;
        k_merge_finish<<<(unsigned)ntiles, MG_THREADS, 0, s>>>(f);
    }
    GCG_LAUNCH_CHECK();
    uint32_t h[2] = {0, 0};
    GCG_CUDA(cudaMemcpyAsync(h, ctl.get() + 1, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    GCG_CUDA(cudaStreamSynchronize(s));
    if (h[1]) return fail(GCG_ERR_TIMEOUT, "merge_unique_csr: a tile's prefix never arrived");
    *ne = h[0];
    return GCG_OK;
}

int scan_u32(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total_dev, cudaStream_t s) {
    if (n == 0) {
        if (total_dev) GCG_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s));
        return GCG_OK;
    }
    uint64_t nb = (n + SC_TILE - 1) / SC_TILE;
    if (nb == 1) {
        sc_scan_tile<<<1, SC_THREADS, 0, s>>>(in, out, n, nullptr, total_dev);
        GCG_LAUNCH_CHECK();
        return GCG_OK;
    }
    tbuf<uint32_t> sums;
    GCG_TRY(sums.alloc(nb, s));
    sc_reduce<<<(unsigned)nb, SC_THREADS, 0, s>>>(in, n, sums.get());
    GCG_LAUNCH_CHECK();
    GCG_TRY(scan_u32(sums.get(), sums.get(), nb, nullptr, s));
    sc_scan_tile<<<(unsigned)nb, SC_THREADS, 0, s>>>(in, out, n, sums.get(), total_dev);
    GCG_LAUNCH_CHECK();
    /* sums is released stream-ordered, after the kernels above. */
    return GCG_OK;
}

RadixPlan radix_plan(int begin_bit, int end_bit) {
    RadixPlan pl = {};
    for (int left = end_bit - begin_bit, passes = (left + 7) / 8; passes > 0; --passes) {
        const int bits = (left + passes - 1) / passes;
        pl.shift[pl.npass] = (uint8_t)(end_bit - left);
        pl.bits[pl.npass++] = (uint8_t)bits;
        left -= bits;
    }
    return pl;
}

int radix_passes(uint64_t *keys, uint64_t *tmp, uint64_t n, const RadixPlan &pl, int first, int last,
                 const uint32_t *counts, uint64_t **result, cudaStream_t s, bool recount) {
    *result = keys;
    if (n <= 1 || first >= last) return GCG_OK;
    if (n > 0xFFFFFFFFull) return fail(GCG_ERR_UNSUPPORTED, "radix sort: more than 2^32-1 keys");
    const uint64_t ntiles = (n + RS_TILE - 1) / RS_TILE;
    /* state words and tickets, cleared together */
    const uint64_t nwords = (ntiles + ntiles / RS_GROUP + 1) * RS_RADIX;
    tbuf<unsigned long long> work;
    GCG_TRY(work.alloc(nwords + RS_PASSES, s));
    GCG_CUDA(cudaMemsetAsync(work.get(), 0, (nwords + RS_PASSES) * 8, s));
    uint64_t *a = keys, *b = tmp;
    for (int p = first; p < last; ++p) {
        RsPass ps;
        ps.in = a;
        ps.out = b;
        ps.n = n;
        ps.shift = pl.shift[p];
        ps.bits = pl.bits[p];
        ps.tag = (uint32_t)(p + 1) << 2;
        ps.spin = recount ? RS_RECOUNT : RS_SPIN;
        ps.counts = counts + p * RS_RADIX;
        ps.ticket = reinterpret_cast<uint32_t *>(work.get() + nwords + p);
        ps.tile = work.get();
        ps.group = work.get() + ntiles * RS_RADIX;
        auto kern = ps.bits == 8 ? rs_pass<8> : ps.bits == 7 ? rs_pass<7> : rs_pass<6>;
        GCG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RS_SMEM));
        kern<<<(unsigned)ntiles, RS_THREADS, RS_SMEM, s>>>(ps);
        GCG_LAUNCH_CHECK();
        uint64_t *x = a; a = b; b = x;
    }
    *result = a;
    return GCG_OK;
}

int radix_sort_u64(uint64_t *keys, uint64_t *tmp, uint64_t n, int begin_bit, int end_bit, uint64_t **result,
                   cudaStream_t s) {
    *result = keys;
    if (n <= 1 || end_bit <= begin_bit) return GCG_OK;
    if (end_bit - begin_bit > 8 * RS_PASSES) return fail(GCG_ERR_INVALID, "radix sort: more than 64 bits");
    const RadixPlan pl = radix_plan(begin_bit, end_bit);
    tbuf<uint32_t> counts;
    GCG_TRY(counts.alloc(RS_PASSES * RS_RADIX, s));
    GCG_CUDA(cudaMemsetAsync(counts.get(), 0, RS_PASSES * RS_RADIX * 4, s));
    constexpr uint64_t per_block = (uint64_t)RadixCounter::THREADS * 8;
    rs_count<<<(unsigned)std::min<uint64_t>((n + per_block - 1) / per_block, (uint64_t)num_sms() * 4),
               RadixCounter::THREADS, 0, s>>>(keys, n, pl, counts.get());
    GCG_LAUNCH_CHECK();
    return radix_passes(keys, tmp, n, pl, 0, pl.npass, counts.get(), result, s);
}

}  // namespace gcg
