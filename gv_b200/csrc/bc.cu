// Betweenness centrality (Brandes) and single-source BFS path counts over the
// edge-block store, 32 or 64 sources per pass, sources spread over the lanes.
//
// Replaces the reference's bc (src/algorithm/bc/bc.cu:3-88) and its kernels
// initializeArrays / initbfsKernel / bfsKernel / dependencyKernel
// (src/algorithm/bc/bc_kernel.cu:3-119), which run one source per host loop
// and one level per launch with int path counts and an unordered dependency
// pass.  Here the sources of a pass share every adjacency read.  A pass keeps
// NW 32-bit words of source bits per vertex (NW = 1: 32 sources, NW = 2: 64);
// source slot s sits in lane s % 32, half s / 32.
//
//   forward, level L -> L+1, push (top-down over the union frontier): a warp takes
//   a vertex u at level L for the sources in mask F = masks[L][u]; each lane
//   holds sigma_s(u) of its NW sources.  For each neighbour w (ids read 32 at
//   a time, coalesced), want = F & ~vis[w] are the sources that reach w first
//   through this level; the neighbours with want != 0 are packed and visited:
//   one atomicOr marks want in nxt[w], each source in want adds sigma_s(u)
//   into sigma_s(w) (exact uint64 adds, so the order does not matter).
//
//   forward, pull (bottom-up, chosen per level on the device when the level
//   holds many entries; 64-source passes only): a warp takes a vertex w that
//   some source has not reached, sums sigma_s(u) over its neighbours u at level
//   L for those sources and writes its row and nxt[w] once, without atomics.
//
//   backward, level L (pull, no atomics): a warp takes v at level L for the
//   sources in A = masks[L][v]; for each neighbour w, the sources in
//   A & masks[L+1][w] (w one level deeper for them) add
//   coef_s(w) = (1 + delta_s(w)) / sigma_s(w).  Then delta_s(v) =
//   sigma_s(v) * acc_s, coef_s(v) replaces sigma_s(v) in the same 8-byte slot,
//   and each half of the pass adds the sum of its 32 deltas (fixed shuffle
//   order, fp64) into its own output row, so one pass can serve two requests.
//
// Level masks stay resident for the backward pass; sigma / coef rows are
// vertex-major ([v][32 NW] x 8 bytes), so the lanes of one vertex and half
// touch one 256-byte segment.  Vertices with more than heavy_fill entries
// are expanded by a whole CTA (block table in shared memory, warps over
// blocks), hubs in pieces with a CTA each; the backward partials of a CTA are combined in warp order, so
// results are bit-for-bit repeatable.
#include <algorithm>
#include <cstdlib>
#include <string>
#include <vector>
#include "store.cuh"
#include "group.cuh"
#include "launch.hpp"
#include "prof.hpp"

namespace gv {
namespace {

constexpr int MS_THREADS = 256;
constexpr int MS_WARPS = MS_THREADS / 32;
constexpr uint32_t MS_TAB = 2048;         // blocks per shared-memory table window
// Five times this many CTAs in the largest level launch: many small shares, so
// the block scheduler evens out the heavy-tailed work per vertex.  BC at R-MAT
// scale 25 (32 / 64 sources): 283 / 382 ms with 148 * (8 + 2) CTAs, 241 / 339 with
// twice as many, 214 / 284 with 8 times, 207 / 287 with 16 times (this), 204 / 282
// with 32 times.
constexpr unsigned MS_HEAVY_GRID = 148 * 32;
constexpr uint32_t MS_MAX_LEVELS = 1u << 16;
// Entries above which a vertex is a CTA's and not a warp's (at most 1024, a lane
// per block), and entries of a hub's piece below.  Piece / line, us a call:
//   R-MAT, 32 sources   512/256  512/512  1024/512  1024/1024  hubs whole
//   16 K vertices           329      364       366        580         403
//   64 K (64 sources)       734      739       742        990         948
//   256 K                  1775     1776      1613       1775        2440
//   1 M                    4533     4319      4321       4323        6758
//   1 M (64 sources)       6374     6184      6179       6179        8847
// Uniform graphs, which have neither, stay within 1%.
uint32_t ms_heavy_fill(uint32_t n) { return n <= (1u << 17) ? 256u : 512u; }

// Hubs: a vertex of more than two pieces' entries is cut into pieces, a CTA each,
// for otherwise one CTA's walk of the longest list is the time of a level.  The
// pieces are listed once per call, whatever level their vertex is on for some
// source; a level's launch asks its mask.  A piece has ms_piece(n) entries, or more
// where the store would come to more than ms_pieces() pieces (their sums are
// 256 or 512 bytes each; four times as many pieces on 4 M vertices, 26.0 ms
// against 24.6).  Fewer vertices have fewer: with 32,768 whatever the graph, a
// call on 16 K vertices took 29 MB of scratch (10 so), and where they have 390
// entries each 1180 us (1085 so; 128 K of 147 each, 64 sources, 3535 and 3090).
uint32_t ms_piece(uint32_t n) { return n <= (1u << 17) ? 512u : 1024u; }
uint32_t ms_pieces(uint32_t n, uint64_t slots) {
    const uint32_t by_n = n / 8 <= 32768u ? std::max(1024u, n / 8) : std::min(262144u, std::max(32768u, n / 128));
    return (uint32_t)std::min<uint64_t>(by_n, slots / ms_piece(n) + 1);
}
uint32_t ms_items_max(uint32_t pieces) {  // entries / piece, one more per vertex, which has two at least
    return pieces + pieces / 2 + 1;
}
struct MsHubs {
    unsigned long long total;  // entries of the store (used slots)
    uint32_t nitems;
    uint32_t piece;            // blocks of a piece
    uint32_t huge_fill;        // vertices with more entries are hubs
};

// CTAs of a level launch on n vertices: a warp per vertex at most (with 23,680
// CTAs for 16 K vertices, a level took 32 us, 8 so), but 740 at least, a wave, for
// few vertices with long lists (2 K vertices of 300 entries: 217 us a call with
// 320, 202 so).
unsigned ms_grid(uint32_t n) {
    const uint64_t light = ((uint64_t)n + MS_WARPS - 1) / MS_WARPS;
    const uint64_t rounds = std::min<uint64_t>((light + 3) / 4, MS_HEAVY_GRID);
    return (unsigned)(5 * std::max<uint64_t>(rounds, std::min(n, 148u)));  // a heavy CTA to four light ones (ms_share)
}

// What a level's kernels count.  A level's vertices are listed in a region of
// n words, light ones from its front and heavy ones from its back; the lists
// of the first MS_SAVED levels stay for the backward pass.
struct MsLevel {
    uint32_t light, heavy;       // vertices of the level
    uint32_t clight, cheavy;     // pull levels: vertices some source has not reached
    unsigned long long entries;  // of the level's vertices
    uint32_t blight, bheavy;     // light, heavy when the backward pass lists the level again
    // Whether it has a vertex: hubs are in neither list but have entries, and on
    // directed stores vertices may have none but are listed.
    bool empty() const { return !light && !heavy && !entries; }
};
static_assert(sizeof(MsLevel) == 32, "counters of a level");
constexpr uint32_t MS_SAVED = 5;
constexpr uint32_t MS_LEVELS = 512;  // levels with counters to begin with; deeper searches take more (slot 19)
constexpr int MS_PER_THREAD = 4;  // vertices per thread and round of the listing kernels

template <int NW> struct MaskOf;
template <> struct MaskOf<1> { using type = uint32_t; };
template <> struct MaskOf<2> { using type = unsigned long long; };

template <int NW>
struct MsBufs {
    using M = typename MaskOf<NW>::type;
    unsigned long long *row;  // [n][32 NW] sigma (u64); after its level's backward step: coef (f64 bits)
    M *vis;                   // [n] sources that reached v at a finished level
    M *nxt;                   // [n] sources that reach v at the level being built
    M *masks;                 // [levels][n]
    uint32_t *list;           // vertices of the current level: fill <= heavy_fill from [0], the rest from [n - 1] down
    uint32_t *cand;           // pull levels: vertices some source has not reached, in the same way
    uint32_t *cnt;            // [0] light, [1] heavy, [2] light candidates, [3] heavy candidates
    unsigned long long *entries;    // of the level's vertices
    unsigned long long *unreached;  // entries of the vertices some source has not reached (counted down by
                                    // k_ms_close as vertices fill up)
    double *bc;               // [outputs][n]; half k of the pass adds into row out[k]
    M full;                   // the pass's sources
    uint32_t heavy_fill;      // vertices with more entries are a CTA's, hubs a CTA's per piece
    const MsHubs *hubs;
    const uint2 *items;       // (vertex, piece), a vertex's pieces in a row
    uint32_t *arrived;        // per item: at a vertex's first, its pieces that are done
    double *part;             // per item: the sums of a dependency piece [32 NW]
    uint32_t alpha;           // pull when alpha * entries > unreached (0: always push)
    uint32_t n;
    uint32_t out[2];
};

// Scratch of one call, carved once for the widest pass it runs.
struct MsArena {
    unsigned long long *row;
    void *vis, *nxt;
    uint32_t *lists, *cand, *dsrc;   // lists: MS_SAVED + 1 regions of n
    MsLevel *lev, *hlev;             // counters per level (lev_cap of them); the host's copy of a few
    uint32_t lev_cap;
    unsigned long long *unreached;
    uint2 *items;
    uint32_t *arrived;
    MsHubs *hubs;
    double *part;
    double *bc;
    uint32_t n;

    template <int NW>
    MsBufs<NW> bufs(gv_graph *g) const {
        using M = typename MaskOf<NW>::type;
        MsBufs<NW> b;
        b.row = row;
        b.vis = (M *)vis;
        b.nxt = (M *)nxt;
        b.masks = (M *)g->aux[6];
        b.cand = cand;
        b.unreached = unreached;
        b.bc = bc;
        level(b, 0);
        b.full = 0;
        b.alpha = 0;
        b.heavy_fill = ms_heavy_fill(n);
        b.hubs = hubs;
        b.items = items;
        b.arrived = arrived;
        b.part = part;
        b.n = n;
        b.out[0] = b.out[1] = 0;
        return b;
    }

    uint32_t *region(uint32_t L) const { return lists + (size_t)std::min(L, MS_SAVED) * n; }
    uint32_t *counts(uint32_t L) const { return &lev[L].light; }
    template <int NW>
    void level(MsBufs<NW> &b, uint32_t L) const {
        b.list = region(L);
        b.cnt = counts(L);
        b.entries = &lev[L].entries;
    }
};

template <int NW>
struct alignas(8) Packed {
    uint32_t w;
    typename MaskOf<NW>::type m;
};

__device__ __forceinline__ double as_f64(unsigned long long x) { return __longlong_as_double((long long)x); }
__device__ __forceinline__ unsigned long long as_u64(double x) { return (unsigned long long)__double_as_longlong(x); }

// Source bit of lane `lane`, half k.
template <typename M>
__device__ __forceinline__ bool has_src(M m, uint32_t lane, int k) {
    return (m >> (lane + 32u * (uint32_t)k)) & 1u;
}

__device__ __forceinline__ uint32_t ms_block(const DevGraph &g, uint32_t root, uint32_t k) {
    return k == 0 ? root : cbt_block(g.left, g.right, root, k);
}

// Walks the entries of one block 32 at a time: lane j loads entry e0 + j and
// its source mask pre(w) (0: nothing to do for any source); the entries with
// a non-zero mask are packed into the warp's shared slots, and body(w, mask)
// runs for each of them with the whole warp.  In most levels few entries need
// work, so the warp skips the rest without touching them.
template <int NW, typename Pre, typename Body>
__device__ __forceinline__ void ms_block_entries(const DevGraph &g, uint32_t b, uint32_t slots, Pre &&pre,
                                                 Body &&body) {
    using M = typename MaskOf<NW>::type;
    __shared__ Packed<NW> pack_all[MS_WARPS][32];  // one row of slots per warp (MS_THREADS threads)
    const uint32_t lane = threadIdx.x & 31u;
    Packed<NW> *pack = pack_all[threadIdx.x >> 5];
    const uint32_t *bp = g.pool + ((size_t)b << g.logB);
    for (uint32_t e0 = 0; e0 < slots; e0 += 32) {
        const uint32_t e = e0 + lane;
        uint32_t w = GV_TOMB;
        M pv = 0;
        if (e < slots) {
            w = bp[e];
            if (w != GV_TOMB) pv = pre(w);
        }
        const uint32_t bal = __ballot_sync(GV_FULL_MASK, pv != 0);
        if (!bal) continue;  // warp-uniform
        if (pv) pack[__popc(bal & ((1u << lane) - 1u))] = Packed<NW>{w, pv};
        __syncwarp();
        const uint32_t c = __popc(bal);
        for (uint32_t j = 0; j < c; ++j) {
            const Packed<NW> x = pack[j];
            body(x.w, x.m);
        }
        __syncwarp();
    }
}

// Light vertex: the warp's lanes hold its (at most 32) block indices.
template <int NW, typename Pre, typename Body>
__device__ __forceinline__ void ms_walk_light(const DevGraph &g, uint4 rec, Pre &&pre, Body &&body) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t fill = rec.y, nb = blocks_for(fill, g.logB);
    const uint32_t blk = lane < nb ? ms_block(g, rec.x, lane) : GV_NIL;
    for (uint32_t k = 0; k < nb; ++k) {
        const uint32_t b = __shfl_sync(GV_FULL_MASK, blk, k);
        ms_block_entries<NW>(g, b, min(g.B, fill - (k << g.logB)), pre, body);
    }
}

// What a CTA of the heavy part takes at a time: a piece of a hub or a whole
// heavy vertex, blocks [lo, hi) of it.
struct MsUnit {
    uint32_t v, item, lo, hi;
    uint4 rec;
    bool piece;
};

// Unit i of the hubs' pieces followed by `list` (heavy vertices from its end).
template <int NW>
__device__ __forceinline__ MsUnit ms_unit(const DevGraph &g, const MsBufs<NW> &b, const uint32_t *list, uint32_t i,
                                          uint32_t nitems) {
    MsUnit u;
    const uint32_t piece = b.hubs->piece;
    u.piece = i < nitems;
    u.item = i;
    const uint2 it = u.piece ? b.items[i] : make_uint2(list[b.n - 1 - (i - nitems)], 0u);
    u.v = it.x;
    u.rec = g.vtx[it.x];
    u.lo = it.y * piece;
    u.hi = blocks_for(u.rec.y, g.logB);
    if (u.piece) u.hi = min(u.hi, u.lo + piece);
    return u;
}

// Heavy vertex: the CTA fills a shared block table window by window; warps
// take blocks w, w + MS_WARPS, ...
template <int NW, typename Pre, typename Body>
__device__ __forceinline__ void ms_walk_heavy(const DevGraph &g, uint4 rec, uint32_t lo, uint32_t nb, uint32_t *tab,
                                              Pre &&pre, Body &&body) {
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t fill = rec.y;
    for (uint32_t k0 = lo; k0 < nb; k0 += MS_TAB) {
        const uint32_t cnt = min(MS_TAB, nb - k0);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) tab[i] = ms_block(g, rec.x, k0 + i);
        __syncthreads();
        for (uint32_t i = warp; i < cnt; i += MS_WARPS) {
            const uint32_t k = k0 + i;
            ms_block_entries<NW>(g, tab[i], min(g.B, fill - (k << g.logB)), pre, body);
        }
    }
}

// Places the pass's sources: slot s (< 32 NW) holds src[s], GV_NIL for none;
// lists level 0 (a vertex once, however many slots it holds).
template <int NW>
__global__ void k_ms_init(DevGraph g, MsBufs<NW> b, const uint32_t *__restrict__ src) {
    using M = typename MaskOf<NW>::type;
    const uint32_t s = threadIdx.x;
    if (s >= 32u * NW) return;
    const uint32_t v = src[s];
    if (v == GV_NIL) return;
    const M before = atomicOr(&b.masks[v], (M)1 << s);
    atomicOr(&b.vis[v], (M)1 << s);
    b.row[(size_t)v * 32 * NW + s] = 1ull;
    if (before) return;
    const uint32_t fill = g.vtx[v].y;
    if (fill > b.hubs->huge_fill) {}  // its pieces ask the mask
    else if (fill > b.heavy_fill) b.list[b.n - 1 - atomicAdd(&b.cnt[1], 1u)] = v;
    else b.list[atomicAdd(&b.cnt[0], 1u)] = v;
    atomicAdd(b.entries, (unsigned long long)fill);
}

// Appends a CTA round's vertices to a region and its counts (MS_PER_THREAD per
// thread, bit j of on / heavy for v[j]) with two atomics; all threads call it.
__device__ __forceinline__ void ms_append(uint32_t *region, uint32_t *cnt, uint32_t n, const uint32_t *v, uint32_t on,
                                          uint32_t heavy) {
    __shared__ uint32_t wt[33], base[2];
    const uint32_t light = on & ~heavy;
    uint32_t tot;  // a round has at most MS_THREADS * MS_PER_THREAD of each: 16 bits
    const uint32_t pre = cta_excl_scan<uint32_t, MS_THREADS>(__popc(light) | __popc(on & heavy) << 16, wt, tot);
    if (!tot) return;  // CTA-uniform
    if (threadIdx.x == 0) {
        base[0] = (tot & 0xFFFFu) ? atomicAdd(&cnt[0], tot & 0xFFFFu) : 0u;
        base[1] = (tot >> 16) ? atomicAdd(&cnt[1], tot >> 16) : 0u;
    }
    __syncthreads();
    uint32_t l = base[0] + (pre & 0xFFFFu), h = base[1] + (pre >> 16);
#pragma unroll
    for (int j = 0; j < MS_PER_THREAD; ++j) {
        if (!((on >> j) & 1u)) continue;
        if ((heavy >> j) & 1u) region[n - 1 - h++] = v[j];
        else region[l++] = v[j];
    }
    __syncthreads();
}

// Entries of every vertex: what the hubs' pieces are sized by, and the pull
// levels' starting count of entries of vertices some source has not reached.
__global__ void __launch_bounds__(MS_THREADS) k_ms_total_fill(DevGraph g, unsigned long long *__restrict__ out) {
    __shared__ unsigned long long wt[33];
    unsigned long long t = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) t += g.vtx[v].y;
    t = cta_sum<unsigned long long, MS_THREADS>(t, wt);
    if (threadIdx.x == 0 && t) atomicAdd(out, t);
}

// The pieces of the hubs, once per call, from the entries of the store (total).
__global__ void k_ms_items(DevGraph g, uint32_t least, uint32_t pieces, MsHubs *hubs, uint2 *__restrict__ items) {
    const uint32_t most = pieces + pieces / 2 + 1;  // never more, by the line below
    const unsigned long long entries = max((unsigned long long)least, (hubs->total + pieces - 1) / pieces);
    const uint32_t piece = (uint32_t)((entries + g.B - 1) >> g.logB);
    const uint32_t huge_fill = 2 * (piece << g.logB);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        hubs->piece = piece;
        hubs->huge_fill = huge_fill;
    }
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
        const uint32_t fill = g.vtx[v].y;
        if (fill <= huge_fill) continue;
        const uint32_t np = (blocks_for(fill, g.logB) + piece - 1) / piece;
        const uint32_t at = atomicAdd(&hubs->nitems, np);
        for (uint32_t p = 0; p < np && at + p < most; ++p) items[at + p] = make_uint2(v, p);
    }
}

// Vertices of a level into its list, from its masks (levels whose list was not
// kept for the backward pass).
template <int NW>
__global__ void __launch_bounds__(MS_THREADS) k_ms_split(DevGraph g, MsBufs<NW> b,
                                                         const typename MaskOf<NW>::type *__restrict__ mask) {
    const uint32_t huge_fill = b.hubs->huge_fill;
    for (uint32_t base = blockIdx.x * MS_THREADS * MS_PER_THREAD; base < b.n;
         base += gridDim.x * MS_THREADS * MS_PER_THREAD) {
        uint32_t v[MS_PER_THREAD], on = 0, heavy = 0;
#pragma unroll
        for (int j = 0; j < MS_PER_THREAD; ++j) {
            v[j] = base + j * MS_THREADS + threadIdx.x;
            if (v[j] < b.n && mask[v[j]]) {
                const uint32_t fill = g.vtx[v[j]].y;
                on |= (uint32_t)(fill <= huge_fill) << j;
                heavy |= (uint32_t)(fill > b.heavy_fill) << j;
            }
        }
        ms_append(b.list, b.cnt, b.n, v, on, heavy);
    }
}

// Pull levels choose themselves on the device: the level's own entries (what a
// push level reads) against the entries of the vertices some source has not
// reached (what a pull level reads).
template <int NW>
__device__ __forceinline__ bool ms_pull_level(const MsBufs<NW> &b) {
    return b.alpha && (unsigned long long)b.alpha * *b.entries > *b.unreached;
}

// Candidates of a pull level: vertices with entries that some source of the
// pass has not reached; nothing on push levels.
template <int NW>
__global__ void __launch_bounds__(MS_THREADS) k_ms_cand(DevGraph g, MsBufs<NW> b) {
    if (!ms_pull_level(b)) return;
    const uint32_t huge_fill = b.hubs->huge_fill;
    for (uint32_t base = blockIdx.x * MS_THREADS * MS_PER_THREAD; base < b.n;
         base += gridDim.x * MS_THREADS * MS_PER_THREAD) {
        uint32_t v[MS_PER_THREAD], on = 0, heavy = 0;
#pragma unroll
        for (int j = 0; j < MS_PER_THREAD; ++j) {
            v[j] = base + j * MS_THREADS + threadIdx.x;
            if (v[j] < b.n && (b.full & ~b.vis[v[j]])) {
                const uint32_t fill = g.vtx[v[j]].y;
                on |= (uint32_t)(fill > 0 && fill <= huge_fill) << j;
                heavy |= (uint32_t)(fill > b.heavy_fill) << j;
            }
        }
        ms_append(b.cand, b.cnt + 2, b.n, v, on, heavy);
    }
}

template <typename M>
__device__ __forceinline__ M warp_or_mask(M x) {
    if (sizeof(M) == 8) {
        const uint32_t lo = __reduce_or_sync(GV_FULL_MASK, (uint32_t)x);
        const uint32_t hi = __reduce_or_sync(GV_FULL_MASK, (uint32_t)((unsigned long long)x >> 32));
        return (M)(((unsigned long long)hi << 32) | lo);
    }
    return (M)__reduce_or_sync(GV_FULL_MASK, (uint32_t)x);
}

// Pull over one block of candidate w's entries: the neighbours u at level L
// for some source that has not reached w (F = mask[u] & need) are packed,
// then each lane adds sigma_s(u) of its sources for them (exact uint64 sums)
// and ORs F into the sources that reach w at level L + 1.
template <int NW>
__device__ __forceinline__ void ms_pull_block(const DevGraph &g, const MsBufs<NW> &b,
                                              const typename MaskOf<NW>::type *__restrict__ mask, uint32_t blk,
                                              uint32_t slots, typename MaskOf<NW>::type need,
                                              unsigned long long (&acc)[NW], typename MaskOf<NW>::type &reach) {
    using M = typename MaskOf<NW>::type;
    __shared__ Packed<NW> pack_all[MS_WARPS][32];
    const uint32_t lane = threadIdx.x & 31u;
    Packed<NW> *pack = pack_all[threadIdx.x >> 5];
    const uint32_t *bp = g.pool + ((size_t)blk << g.logB);
    const unsigned long long *row = b.row;
    for (uint32_t e0 = 0; e0 < slots; e0 += 32) {
        const uint32_t e = e0 + lane;
        uint32_t u = 0;
        M f = 0;
        if (e < slots) {
            u = bp[e];
            if (u != GV_TOMB) f = mask[u] & need;
            else u = 0;
        }
        reach |= f;
        const uint32_t bal = __ballot_sync(GV_FULL_MASK, f != 0);
        if (!bal) continue;  // warp-uniform
        if (f) pack[__popc(bal & ((1u << lane) - 1u))] = Packed<NW>{u, f};
        __syncwarp();
        const uint32_t c = __popc(bal);
        constexpr int GB = NW == 1 ? 8 : 4;
        for (uint32_t j0 = 0; j0 < c; j0 += GB) {
            Packed<NW> x[GB];
#pragma unroll
            for (int t = 0; t < GB; ++t) x[t] = (j0 + t < c) ? pack[j0 + t] : Packed<NW>{0u, (M)0};
            unsigned long long v[NW][GB];
#pragma unroll
            for (int k = 0; k < NW; ++k)
#pragma unroll
                for (int t = 0; t < GB; ++t)
                    v[k][t] = has_src(x[t].m, lane, k) ? __ldg(row + (size_t)x[t].w * 32 * NW + lane + 32 * k) : 0ull;
#pragma unroll
            for (int k = 0; k < NW; ++k)
#pragma unroll
                for (int t = 0; t < GB; ++t) acc[k] += v[k][t];
        }
        __syncwarp();
    }
}

// Writes w's sigma for the sources that reach it at this level, and nxt[w].
template <int NW>
__device__ __forceinline__ void ms_pull_finish(const MsBufs<NW> &b, uint32_t w, typename MaskOf<NW>::type reach,
                                               const unsigned long long (&acc)[NW]) {
    const uint32_t lane = threadIdx.x & 31u;
    if (!reach) return;  // warp-uniform
#pragma unroll
    for (int k = 0; k < NW; ++k)
        if (has_src(reach, lane, k)) b.row[(size_t)w * 32 * NW + lane + 32 * k] = acc[k];
    if (lane == 0) b.nxt[w] = reach;
}

template <int NW>
__device__ __forceinline__ void ms_pull_light(const DevGraph &g, const MsBufs<NW> &b,
                                              const typename MaskOf<NW>::type *__restrict__ mask, uint32_t vb,
                                              uint32_t vg) {
    using M = typename MaskOf<NW>::type;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nl = b.cnt[2];
    for (uint32_t i = vb * MS_WARPS + (threadIdx.x >> 5); i < nl; i += vg * MS_WARPS) {
        const uint32_t w = b.cand[i];
        const M need = b.full & ~b.vis[w];
        unsigned long long acc[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) acc[k] = 0ull;
        M reach = 0;
        const uint4 rec = g.vtx[w];
        const uint32_t fill = rec.y, nb = blocks_for(fill, g.logB);
        const uint32_t blk = lane < nb ? ms_block(g, rec.x, lane) : GV_NIL;
        for (uint32_t k = 0; k < nb; ++k) {
            const uint32_t bk = __shfl_sync(GV_FULL_MASK, blk, k);
            ms_pull_block<NW>(g, b, mask, bk, min(g.B, fill - (k << g.logB)), need, acc, reach);
        }
        ms_pull_finish<NW>(b, w, warp_or_mask(reach), acc);
    }
}

template <int NW>
__device__ __forceinline__ void ms_pull_heavy(const DevGraph &g, const MsBufs<NW> &b,
                                              const typename MaskOf<NW>::type *__restrict__ mask, uint32_t vb,
                                              uint32_t vg) {
    using M = typename MaskOf<NW>::type;
    __shared__ uint32_t tab[MS_TAB];
    __shared__ unsigned long long red[MS_WARPS][NW][32];
    __shared__ M rred[MS_WARPS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ni = b.hubs->nitems, nh = ni + b.cnt[3];
    for (uint32_t i = vb; i < nh; i += vg) {
        const MsUnit un = ms_unit<NW>(g, b, b.cand, i, ni);
        const uint32_t w = un.v;
        const M need = b.full & ~b.vis[w];
        if (!need) continue;  // CTA-uniform: a hub that every source has reached
        unsigned long long acc[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) acc[k] = 0ull;
        M reach = 0;
        const uint32_t fill = un.rec.y;
        for (uint32_t k0 = un.lo; k0 < un.hi; k0 += MS_TAB) {
            const uint32_t cnt = min(MS_TAB, un.hi - k0);
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < cnt; t += blockDim.x) tab[t] = ms_block(g, un.rec.x, k0 + t);
            __syncthreads();
            for (uint32_t t = warp; t < cnt; t += MS_WARPS)
                ms_pull_block<NW>(g, b, mask, tab[t], min(g.B, fill - ((k0 + t) << g.logB)), need, acc, reach);
        }
#pragma unroll
        for (int k = 0; k < NW; ++k) red[warp][k][lane] = acc[k];
        reach = warp_or_mask(reach);
        if (lane == 0) rred[warp] = reach;
        __syncthreads();
        if (warp == 0) {
            unsigned long long tot[NW];
            M r = 0;
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                tot[k] = 0ull;
                for (int x = 0; x < MS_WARPS; ++x) tot[k] += red[x][k][lane];
            }
            for (int x = 0; x < MS_WARPS; ++x) r |= rred[x];
            if (!un.piece) {
                ms_pull_finish<NW>(b, w, r, tot);
            } else if (r) {  // the pieces add up in the row, which is 0 for these sources (exact sums, any order)
#pragma unroll
                for (int k = 0; k < NW; ++k)
                    if (has_src(r, lane, k)) atomicAdd(&b.row[(size_t)w * 32 * NW + lane + 32 * k], tot[k]);
                if (lane == 0) atomicOr(&b.nxt[w], r);
            }
        }
        __syncthreads();
    }
}

template <int NW>
struct FwdBody {
    using M = typename MaskOf<NW>::type;
    MsBufs<NW> b;
    M F;
    unsigned long long sig[NW];
    __device__ __forceinline__ void load(uint32_t u) {
        const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
        for (int k = 0; k < NW; ++k) sig[k] = has_src(F, lane, k) ? b.row[(size_t)u * 32 * NW + lane + 32 * k] : 0ull;
    }
    // sources that reach w first through this level
    __device__ __forceinline__ M operator()(uint32_t w) const { return F & ~b.vis[w]; }
    __device__ __forceinline__ void visit(uint32_t w, M want) const {
        const uint32_t lane = threadIdx.x & 31u;
        if (lane == 0) atomicOr(&b.nxt[w], want);
#pragma unroll
        for (int k = 0; k < NW; ++k)
            if (has_src(want, lane, k)) atomicAdd(&b.row[(size_t)w * 32 * NW + lane + 32 * k], sig[k]);
    }
};

template <int NW>
__device__ __forceinline__ void ms_fwd_light(const DevGraph &g, const MsBufs<NW> &b,
                                             const typename MaskOf<NW>::type *__restrict__ mask, uint32_t vb,
                                             uint32_t vg) {
    using M = typename MaskOf<NW>::type;
    const uint32_t nl = b.cnt[0];
    for (uint32_t i = vb * MS_WARPS + (threadIdx.x >> 5); i < nl; i += vg * MS_WARPS) {
        const uint32_t u = b.list[i];
        FwdBody<NW> f{b, mask[u], {}};
        f.load(u);
        ms_walk_light<NW>(g, g.vtx[u], f, [&](uint32_t w, M want) { f.visit(w, want); });
    }
}

template <int NW>
__device__ __forceinline__ void ms_fwd_heavy(const DevGraph &g, const MsBufs<NW> &b,
                                             const typename MaskOf<NW>::type *__restrict__ mask, uint32_t vb,
                                             uint32_t vg) {
    using M = typename MaskOf<NW>::type;
    __shared__ uint32_t tab[MS_TAB];
    const uint32_t ni = b.hubs->nitems, nh = ni + b.cnt[1];
    for (uint32_t i = vb; i < nh; i += vg) {
        const MsUnit un = ms_unit<NW>(g, b, b.list, i, ni);
        FwdBody<NW> f{b, mask[un.v], {}};
        if (!f.F) continue;  // CTA-uniform: a hub that is not on this level
        f.load(un.v);
        ms_walk_heavy<NW>(g, un.rec, un.lo, un.hi, tab, f, [&](uint32_t w, M want) { f.visit(w, want); });
    }
}

// One launch per level and direction, its CTAs shared between the heavy part (units
// of hubs and heavy vertices) and the light part in one of three ways.
// MS_SPLIT: CTA i runs the heavy part when i % 5 == 4 and the light part otherwise,
// side by side.  MS_ALL: every CTA takes its share of the heavy part, then of the
// light part.  MS_FEW: as MS_SPLIT, but where the units are more than twice the heavy
// CTAs, as on graphs with hardly a light vertex, the others take their share of them
// after the light part.
// Uniform, 16 K vertices of 900 entries, 32 sources: 1510 us with MS_SPLIT, 1020 with
// MS_FEW; 4 K of 500 905 and 280.  R-MAT, edge factor 16, 64 sources, MS_FEW against
// MS_ALL both ways: 16 K vertices 420 and 455 us, 64 K 724 and 755, 128 K 1220 and
// 1175, 1 M 6820 and 6640.  Above 64 K vertices the forward takes MS_ALL (1 M: 2890 us
// against 2920 with MS_SPLIT) and the dependencies MS_SPLIT (3555 against 3620).
enum MsWay { MS_SPLIT, MS_ALL, MS_FEW };
constexpr uint32_t MS_FEW_N = 1u << 16;
template <int WAY, typename Units, typename Light, typename Heavy>
__device__ __forceinline__ void ms_share(Units units, Light light, Heavy heavy) {
    if (WAY == MS_ALL) {
        heavy(blockIdx.x, gridDim.x);
        light(blockIdx.x, gridDim.x);
        return;
    }
    const uint32_t nh = gridDim.x / 5;
    const bool all = WAY == MS_FEW && units() > 2 * nh;
    if (blockIdx.x % 5 != 4) {
        light((blockIdx.x / 5) * 4 + blockIdx.x % 5, gridDim.x - nh);
        if (!all) return;
    }
    heavy(all ? blockIdx.x : blockIdx.x / 5, all ? gridDim.x : nh);
}

// One forward level, push or pull (bottom-up: each candidate gathers the path
// counts of its neighbours at level L; no atomics, one write of its row) as the
// level asks for.
// Five resident CTAs (48 registers, a few spilled) for the pull and the
// dependency pass: at R-MAT scale 25, 64 sources, 290 -> 268 ms (two
// requests in one pass 317 -> 302 ms) against four CTAs at 56-64 registers;
// six (40 registers) were slower.
template <int NW, int WAY>
__global__ void __launch_bounds__(MS_THREADS, 5) k_ms_fwd(DevGraph g, MsBufs<NW> b,
                                                          const typename MaskOf<NW>::type *__restrict__ mask) {
    if (ms_pull_level(b))
        ms_share<WAY>([&] { return b.hubs->nitems + b.cnt[3]; },
                 [&](uint32_t vb, uint32_t vg) { ms_pull_light<NW>(g, b, mask, vb, vg); },
                 [&](uint32_t vb, uint32_t vg) { ms_pull_heavy<NW>(g, b, mask, vb, vg); });
    else
        ms_share<WAY>([&] { return b.hubs->nitems + b.cnt[1]; },
                 [&](uint32_t vb, uint32_t vg) { ms_fwd_light<NW>(g, b, mask, vb, vg); },
                 [&](uint32_t vb, uint32_t vg) { ms_fwd_heavy<NW>(g, b, mask, vb, vg); });
}

// Closes level L: masks[L+1] = nxt, vis |= nxt, and lists level L + 1 (region,
// counts and entries of its own).  One launch with the listing, and atomics
// per CTA round: as two kernels with atomics per warp they took 40 us of a
// level on 1 M vertices, 9 so.
template <int NW>
__global__ void __launch_bounds__(MS_THREADS) k_ms_close(DevGraph g, MsBufs<NW> b,
                                                         typename MaskOf<NW>::type *__restrict__ next_mask,
                                                         uint32_t *next_list, MsLevel *next) {
    using M = typename MaskOf<NW>::type;
    __shared__ unsigned long long wt[33];
    unsigned long long entries = 0, filled = 0;
    const uint32_t huge_fill = b.hubs->huge_fill;
    for (uint32_t base = blockIdx.x * MS_THREADS * MS_PER_THREAD; base < b.n;
         base += gridDim.x * MS_THREADS * MS_PER_THREAD) {
        uint32_t v[MS_PER_THREAD], on = 0, heavy = 0;
        M x[MS_PER_THREAD];
#pragma unroll
        for (int j = 0; j < MS_PER_THREAD; ++j) {
            v[j] = base + j * MS_THREADS + threadIdx.x;
            x[j] = v[j] < b.n ? b.nxt[v[j]] : (M)0;
        }
#pragma unroll
        for (int j = 0; j < MS_PER_THREAD; ++j) {
            if (v[j] < b.n) next_mask[v[j]] = x[j];
            if (!x[j]) continue;
            const M old = b.vis[v[j]];
            b.vis[v[j]] = old | x[j];
            b.nxt[v[j]] = 0;
            const uint32_t fill = g.vtx[v[j]].y;
            on |= (uint32_t)(fill <= huge_fill) << j;
            heavy |= (uint32_t)(fill > b.heavy_fill) << j;
            entries += fill;
            // every source has reached v: its entries leave the pull levels' count
            if ((old | x[j]) == b.full && old != b.full) filled += fill;
        }
        ms_append(next_list, &next->light, b.n, v, on, heavy);
    }
    entries = cta_sum<unsigned long long, MS_THREADS>(entries, wt);
    if (threadIdx.x == 0 && entries) atomicAdd(&next->entries, entries);
    if (b.alpha) {
        filled = cta_sum<unsigned long long, MS_THREADS>(filled, wt);
        if (threadIdx.x == 0 && filled) atomicAdd(b.unreached, 0ull - filled);
    }
}

// Backward sum over one block's entries for the sources in A: the entries one
// level deeper for some of them are packed, then every lane gathers coef of
// its sources for eight (one word) or four (two words) entries at a time,
// eight predicated gathers in flight per lane, and adds them in entry order.
template <int NW>
__device__ __forceinline__ void ms_bwd_block(const DevGraph &g, const MsBufs<NW> &b,
                                             const typename MaskOf<NW>::type *__restrict__ deeper, uint32_t blk,
                                             uint32_t slots, typename MaskOf<NW>::type A, double (&acc)[NW]) {
    using M = typename MaskOf<NW>::type;
    __shared__ Packed<NW> pack_all[MS_WARPS][32];
    const uint32_t lane = threadIdx.x & 31u;
    Packed<NW> *pack = pack_all[threadIdx.x >> 5];
    const uint32_t *bp = g.pool + ((size_t)blk << g.logB);
    const unsigned long long *row = b.row;
    for (uint32_t e0 = 0; e0 < slots; e0 += 32) {
        const uint32_t e = e0 + lane;
        uint32_t w = 0;
        M mw = 0;
        if (e < slots) {
            w = bp[e];
            if (w != GV_TOMB) mw = deeper[w] & A;
            else w = 0;
        }
        const uint32_t bal = __ballot_sync(GV_FULL_MASK, mw != 0);
        if (!bal) continue;  // warp-uniform
        if (mw) pack[__popc(bal & ((1u << lane) - 1u))] = Packed<NW>{w, mw};
        __syncwarp();
        const uint32_t c = __popc(bal);
        constexpr int GB = NW == 1 ? 8 : 4;  // entries per batch: 8 gathers in flight per lane either way
        for (uint32_t j0 = 0; j0 < c; j0 += GB) {
            Packed<NW> x[GB];
#pragma unroll
            for (int t = 0; t < GB; ++t) x[t] = (j0 + t < c) ? pack[j0 + t] : Packed<NW>{0u, (M)0};
            unsigned long long v[NW][GB];
#pragma unroll
            for (int k = 0; k < NW; ++k)
#pragma unroll
                for (int t = 0; t < GB; ++t)
                    v[k][t] = has_src(x[t].m, lane, k) ? __ldg(row + (size_t)x[t].w * 32 * NW + lane + 32 * k) : 0ull;
#pragma unroll
            for (int k = 0; k < NW; ++k)
#pragma unroll
                for (int t = 0; t < GB; ++t) acc[k] += as_f64(v[k][t]);
        }
        __syncwarp();
    }
}

template <int NW>
__device__ __forceinline__ void ms_load_sig(const MsBufs<NW> &b, uint32_t v, typename MaskOf<NW>::type A,
                                            unsigned long long (&sig)[NW]) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 0; k < NW; ++k) sig[k] = has_src(A, lane, k) ? b.row[(size_t)v * 32 * NW + lane + 32 * k] : 0ull;
}

// Finishes (v, sources in A): delta = sigma * acc, coef replaces sigma, and
// each half with a source here adds the sum of its deltas over the lanes into
// its output row (lane 0, halves in order).
template <int NW>
__device__ __forceinline__ void ms_finish(const MsBufs<NW> &b, uint32_t v, typename MaskOf<NW>::type A,
                                          const unsigned long long (&sig)[NW], const double (&acc)[NW]) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
        if (NW > 1 && !(uint32_t)(A >> (32u * (uint32_t)k))) continue;  // warp-uniform: no source of this half here
        double delta = 0.0;
        if (has_src(A, lane, k)) {
            const double sv = (double)sig[k];
            delta = sv * acc[k];
            b.row[(size_t)v * 32 * NW + lane + 32 * k] = as_u64((1.0 + delta) / sv);
        }
        delta = warp_sum(delta);
        if (lane == 0) b.bc[(size_t)b.out[k] * b.n + v] += delta;
    }
}

template <int NW>
__device__ __forceinline__ void ms_bwd_light(const DevGraph &g, const MsBufs<NW> &b,
                                             const typename MaskOf<NW>::type *__restrict__ mask,
                                             const typename MaskOf<NW>::type *__restrict__ deeper, uint32_t vb,
                                             uint32_t vg) {
    using M = typename MaskOf<NW>::type;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nl = b.cnt[0];
    const uint32_t stride = vg * MS_WARPS;
    // A two-stage prefetch: while a vertex runs, the id of the vertex after
    // next and the source mask and record of the next one are in flight, and
    // the next one's sigma row is loaded before this one finishes, so a
    // vertex starts with its header at hand.  (Rows read here belong to
    // vertices of this level, which only their own warp writes.)
    uint32_t i = vb * MS_WARPS + (threadIdx.x >> 5);
    uint32_t v1 = i < nl ? b.list[i] : 0u;
    uint32_t v2 = i + stride < nl ? b.list[i + stride] : 0u;
    M A1 = i < nl ? mask[v1] : (M)0;
    uint2 rec1 = make_uint2(0u, 0u);
    if (i < nl) {
        const uint4 r = g.vtx[v1];
        rec1 = make_uint2(r.x, r.y);
    }
    unsigned long long sig1[NW];
    ms_load_sig<NW>(b, v1, A1, sig1);
    for (; i < nl; i += stride) {
        const bool has2 = i + stride < nl;
        const uint32_t v3 = i + 2 * stride < nl ? b.list[i + 2 * stride] : 0u;
        const M A2 = has2 ? mask[v2] : (M)0;
        uint2 rec2 = make_uint2(0u, 0u);
        if (has2) {
            const uint4 r = g.vtx[v2];
            rec2 = make_uint2(r.x, r.y);
        }
        double acc[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) acc[k] = 0.0;
        const uint32_t fill = rec1.y, nb = blocks_for(fill, g.logB);
        const uint32_t blk = lane < nb ? ms_block(g, rec1.x, lane) : GV_NIL;
        for (uint32_t k = 0; k < nb; ++k) {
            const uint32_t bk = __shfl_sync(GV_FULL_MASK, blk, k);
            ms_bwd_block<NW>(g, b, deeper, bk, min(g.B, fill - (k << g.logB)), A1, acc);
        }
        unsigned long long sig2[NW];
        ms_load_sig<NW>(b, v2, A2, sig2);
        ms_finish<NW>(b, v1, A1, sig1, acc);
        v1 = v2;
        v2 = v3;
        A1 = A2;
        rec1 = rec2;
#pragma unroll
        for (int k = 0; k < NW; ++k) sig1[k] = sig2[k];
    }
}

template <int NW>
__device__ __forceinline__ void ms_bwd_heavy(const DevGraph &g, const MsBufs<NW> &b,
                                             const typename MaskOf<NW>::type *__restrict__ mask,
                                             const typename MaskOf<NW>::type *__restrict__ deeper, uint32_t vb,
                                             uint32_t vg) {
    __shared__ uint32_t tab[MS_TAB];
    __shared__ double red[MS_WARPS][NW][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ni = b.hubs->nitems, nh = ni + b.cnt[1];
    for (uint32_t i = vb; i < nh; i += vg) {
        const MsUnit un = ms_unit<NW>(g, b, b.list, i, ni);
        const uint32_t v = un.v;
        const typename MaskOf<NW>::type A = mask[v];
        if (!A) continue;  // CTA-uniform: a hub that is not on this level
        double acc[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) acc[k] = 0.0;
        const uint32_t fill = un.rec.y;
        for (uint32_t k0 = un.lo; k0 < un.hi; k0 += MS_TAB) {
            const uint32_t cnt = min(MS_TAB, un.hi - k0);
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < cnt; t += blockDim.x) tab[t] = ms_block(g, un.rec.x, k0 + t);
            __syncthreads();
            for (uint32_t t = warp; t < cnt; t += MS_WARPS)
                ms_bwd_block<NW>(g, b, deeper, tab[t], min(g.B, fill - ((k0 + t) << g.logB)), A, acc);
        }
#pragma unroll
        for (int k = 0; k < NW; ++k) red[warp][k][lane] = acc[k];
        __syncthreads();
        if (warp == 0) {
            double tot[NW];
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                tot[k] = 0.0;
                for (int w = 0; w < MS_WARPS; ++w) tot[k] += red[w][k][lane];
            }
            bool finish = true;
            if (un.piece) {
                // the piece that is done last adds up all of them, in their order
                const uint32_t piece = b.hubs->piece, first = un.item - un.lo / piece;
                const uint32_t np = (blocks_for(fill, g.logB) + piece - 1) / piece;
#pragma unroll
                for (int k = 0; k < NW; ++k) b.part[(size_t)un.item * 32 * NW + 32 * k + lane] = tot[k];
                __threadfence();
                __syncwarp();
                uint32_t done = 0;
                if (lane == 0) done = atomicAdd(&b.arrived[first], 1u);
                finish = __shfl_sync(GV_FULL_MASK, done, 0) == np - 1;
                if (finish) {
                    __threadfence();
                    if (lane == 0) b.arrived[first] = 0;  // for its next level
#pragma unroll
                    for (int k = 0; k < NW; ++k) tot[k] = 0.0;
                    for (uint32_t p = 0; p < np; ++p)
#pragma unroll
                        for (int k = 0; k < NW; ++k) tot[k] += __ldcg(b.part + (size_t)(first + p) * 32 * NW + 32 * k + lane);
                }
            }
            if (finish) {
                unsigned long long sig[NW];
                ms_load_sig<NW>(b, v, A, sig);
                ms_finish<NW>(b, v, A, sig, tot);
            }
        }
        __syncthreads();
    }
}

template <int NW, int WAY>
__global__ void __launch_bounds__(MS_THREADS, 5) k_ms_bwd(DevGraph g, MsBufs<NW> b,
                                                       const typename MaskOf<NW>::type *__restrict__ mask,
                                                       const typename MaskOf<NW>::type *__restrict__ deeper) {
    ms_share<WAY>([&] { return b.hubs->nitems + b.cnt[1]; },
             [&](uint32_t vb, uint32_t vg) { ms_bwd_light<NW>(g, b, mask, deeper, vb, vg); },
             [&](uint32_t vb, uint32_t vg) { ms_bwd_heavy<NW>(g, b, mask, deeper, vb, vg); });
}

__global__ void k_ms_to_f32(const double *__restrict__ x, float *__restrict__ y, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) y[v] = (float)x[v];
}

// dist / sigma of slot 0 after a one-source forward pass.
__global__ void k_ms_extract(MsBufs<1> b, uint32_t depth, int32_t *__restrict__ dist,
                             unsigned long long *__restrict__ sigma) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < b.n; v += gridDim.x * blockDim.x) {
        int32_t d = -1;
        for (uint32_t L = 0; L <= depth; ++L)
            if (b.masks[(size_t)L * b.n + v] & 1u) {
                d = (int32_t)L;
                break;
            }
        dist[v] = d;
        sigma[v] = b.row[(size_t)v * 32];
    }
}

// Auxiliary slot `slot` becomes a new buffer of `bytes` that begins with the
// first keep_bytes of `from` (the slot's buffer or another).
gv_status ms_grow(gv_graph *g, int slot, const void *from, size_t keep_bytes, size_t bytes, cudaStream_t s) {
    void *nb = nullptr;
    if (cudaMalloc(&nb, bytes) != cudaSuccess) {
        cudaGetLastError();
        set_error("level masks allocation of " + std::to_string(bytes) + " B failed");
        return GV_ERR_NOMEM;
    }
    if (keep_bytes && from) {
        cudaError_t e = cudaMemcpyAsync(nb, from, keep_bytes, cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            cudaFree(nb);
            return cuda_status(e, "level masks copy");
        }
    }
    if (g->aux[slot]) cudaFree(g->aux[slot]);
    g->aux[slot] = nb;
    g->aux_bytes[slot] = bytes;
    return GV_OK;
}

// Level masks live in auxiliary slot 6 and grow (keeping the first
// keep_levels levels) when a BFS runs deeper than the levels allocated.
template <int NW>
gv_status masks_reserve(gv_graph *g, MsBufs<NW> &b, uint32_t levels, uint32_t keep_levels, cudaStream_t s) {
    using M = typename MaskOf<NW>::type;
    const size_t level_bytes = (size_t)b.n * sizeof(M);
    const uint32_t cap = (uint32_t)std::min<size_t>(g->aux[6] ? g->aux_bytes[6] / level_bytes : 0, MS_MAX_LEVELS);
    b.masks = (M *)g->aux[6];
    if (levels <= cap) return GV_OK;
    uint32_t want = std::max<uint32_t>(32, cap);
    while (want < levels) want *= 2;
    if (want > MS_MAX_LEVELS) {
        set_error("BFS deeper than the level table");
        return GV_ERR_UNSUPPORTED;
    }
    const gv_status st = ms_grow(g, 6, g->aux[6], (size_t)keep_levels * level_bytes, (size_t)want * level_bytes, s);
    b.masks = (M *)g->aux[6];
    return st;
}

// As masks_reserve, for the levels' counters.
gv_status levels_reserve(gv_graph *g, MsArena &a, uint32_t levels, uint32_t keep_levels, cudaStream_t s) {
    if (levels <= a.lev_cap) return GV_OK;
    uint32_t want = a.lev_cap;
    while (want < levels) want *= 2;
    const gv_status st = ms_grow(g, 19, a.lev, (size_t)keep_levels * sizeof(MsLevel), (size_t)want * sizeof(MsLevel), s);
    if (st != GV_OK) return st;
    a.lev = (MsLevel *)g->aux[19];
    a.lev_cap = want;
    return GV_OK;
}

// Forward pass for the sources placed in dsrc (32 NW slots); returns the
// deepest non-empty level.
template <int NW>
gv_status ms_forward(gv_graph *g, MsArena &a, MsBufs<NW> &b, uint32_t *depth_out, cudaStream_t s) {
    using M = typename MaskOf<NW>::type;
    const DevGraph d = g->d;
    const uint32_t n = b.n;
    gv_status st = masks_reserve<NW>(g, b, 8, 0, s);
    if (st != GV_OK) return st;
    cudaMemsetAsync(b.row, 0, (size_t)n * 256 * NW, s);
    cudaMemsetAsync(b.vis, 0, (size_t)n * sizeof(M), s);
    cudaMemsetAsync(b.nxt, 0, (size_t)n * sizeof(M), s);
    cudaMemsetAsync(b.masks, 0, (size_t)n * sizeof(M), s);
    const uint32_t chunk = 4;
    cudaMemsetAsync(a.lev, 0, (1 + chunk) * sizeof(MsLevel), s);
    a.level(b, 0);
    GV_LAUNCH(k_ms_init<NW>, 1, 32 * NW, 0, s, d, b, (const uint32_t *)a.dsrc);
    if (b.alpha) cudaMemcpyAsync(b.unreached, &a.hubs->total, 8, cudaMemcpyDeviceToDevice, s);
    const bool few = n <= MS_FEW_N;
    const unsigned grid = ms_grid(n), lgrid = grid_for(n, MS_THREADS * MS_PER_THREAD);
    uint32_t L = 0;
    for (;;) {
        st = masks_reserve<NW>(g, b, L + chunk + 2, L + 1, s);
        if (st == GV_OK) st = levels_reserve(g, a, L + chunk + 2, L + 1, s);
        if (st != GV_OK) return st;
        if (L) cudaMemsetAsync(a.lev + L + 1, 0, chunk * sizeof(MsLevel), s);
        for (uint32_t i = 0; i < chunk; ++i, ++L) {
            const M *mask = b.masks + (size_t)L * n;
            ProfScope ps(PROF_BFS_LEVEL, s);
            a.level(b, L);
            if (b.alpha) GV_LAUNCH(k_ms_cand<NW>, lgrid, MS_THREADS, 0, s, d, b);
            if (few) GV_LAUNCH((k_ms_fwd<NW, MS_FEW>), grid, MS_THREADS, 0, s, d, b, mask);
            else GV_LAUNCH((k_ms_fwd<NW, MS_ALL>), grid, MS_THREADS, 0, s, d, b, mask);
            GV_LAUNCH(k_ms_close<NW>, lgrid, MS_THREADS, 0, s, d, b, b.masks + (size_t)(L + 1) * n, a.region(L + 1),
                      a.lev + L + 1);
        }
        cudaError_t e = cudaMemcpyAsync(a.hlev, a.lev + L - chunk + 1, chunk * sizeof(MsLevel), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "bfs levels");
        for (uint32_t i = 0; i < chunk; ++i)
            if (a.hlev[i].empty()) {
                *depth_out = L - chunk + i;  // level L - chunk + 1 + i is empty
                return GV_OK;
            }
    }
}

template <int NW>
gv_status ms_backward(gv_graph *g, const MsArena &a, MsBufs<NW> &b, uint32_t depth, cudaStream_t s) {
    using M = typename MaskOf<NW>::type;
    const DevGraph d = g->d;
    const uint32_t n = b.n;
    const bool few = n <= MS_FEW_N;
    for (uint32_t L = depth; L >= 1; --L) {
        const M *mask = b.masks + (size_t)L * n;
        const M *deeper = b.masks + (size_t)(L + 1) * n;
        ProfScope ps(PROF_BC_DEP, s);
        a.level(b, L);
        if (L >= MS_SAVED) {
            b.cnt = &a.lev[L].blight;
            GV_LAUNCH(k_ms_split<NW>, grid_for(n, MS_THREADS * MS_PER_THREAD), MS_THREADS, 0, s, d, b, mask);
        }
        if (few) GV_LAUNCH((k_ms_bwd<NW, MS_FEW>), ms_grid(n), MS_THREADS, 0, s, d, b, mask, deeper);
        else GV_LAUNCH((k_ms_bwd<NW, MS_SPLIT>), ms_grid(n), MS_THREADS, 0, s, d, b, mask, deeper);
    }
    return cuda_status(cudaGetLastError(), "bc dependencies");
}

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Offsets in the analytics scratch of the buffers of passes up to nw mask words
// wide and `outputs` score rows.
struct MsLayout {
    uint32_t pieces, items;
    size_t row, vis, nxt, lists, cand, lev, unr, item, arr, part, src, bc, bytes;
    MsLayout(const DevGraph &d, uint32_t nw, uint32_t outputs) {
        const size_t n = d.n;
        pieces = ms_pieces(d.n, d.P * (uint64_t)d.B);
        items = ms_items_max(pieces);
        size_t at = 0;
        auto take = [&](size_t x) {
            const size_t o = at;
            at += al256(x);
            return o;
        };
        row = take(n * 256 * nw);
        vis = take(n * 4 * nw);
        nxt = take(n * 4 * nw);
        lists = take(n * 4 * (MS_SAVED + 1));
        cand = take(n * 4);
        lev = take(MS_LEVELS * sizeof(MsLevel));
        unr = take(256);
        item = take((size_t)items * sizeof(uint2));
        arr = take((size_t)items * 4);
        part = take((size_t)items * 256 * nw);
        src = take(256);
        bc = take(n * 8 * outputs);
        bytes = at;
    }
};

gv_status ms_setup(gv_graph *g, uint32_t nw, uint32_t outputs, MsArena &a, cudaStream_t s) {
    const uint32_t n = g->d.n;
    a.n = n;
    const MsLayout o(g->d, nw, outputs);
    char *p = (char *)analytics_scratch(g, o.bytes);
    if (!p) return GV_ERR_NOMEM;
    a.row = (unsigned long long *)(p + o.row);
    a.vis = p + o.vis;
    a.nxt = p + o.nxt;
    a.lists = (uint32_t *)(p + o.lists);
    a.cand = (uint32_t *)(p + o.cand);
    a.lev = (MsLevel *)(g->aux[19] ? g->aux[19] : p + o.lev);
    a.lev_cap = g->aux[19] ? (uint32_t)(g->aux_bytes[19] / sizeof(MsLevel)) : MS_LEVELS;
    a.unreached = (unsigned long long *)(p + o.unr);
    a.hubs = (MsHubs *)(p + o.unr + 64);
    a.items = (uint2 *)(p + o.item);
    a.arrived = (uint32_t *)(p + o.arr);
    a.part = (double *)(p + o.part);
    cudaMemsetAsync(a.hubs, 0, sizeof(MsHubs), s);
    cudaMemsetAsync(a.arrived, 0, (size_t)o.items * 4, s);
    GV_LAUNCH(k_ms_total_fill, grid_for(n, MS_THREADS * 4, 148 * 4), MS_THREADS, 0, s, g->d, &a.hubs->total);
    GV_LAUNCH(k_ms_items, grid_for(n, 256), 256, 0, s, g->d, ms_piece(n), o.pieces, a.hubs, a.items);
    a.dsrc = (uint32_t *)(p + o.src);
    a.bc = (double *)(p + o.bc);
    if (!g->host_pinned) {
        if (cudaMallocHost(&g->host_pinned, 256) != cudaSuccess) {
            cudaGetLastError();
            set_error("pinned host word allocation failed");
            return GV_ERR_NOMEM;
        }
        g->host_pinned_bytes = 256;
    }
    a.hlev = (MsLevel *)g->host_pinned;
    return GV_OK;
}

// Pull levels: a forward level of a 64-source pass pulls when MS_PULL_ALPHA
// times its own entries exceed the entries of the vertices some source has
// not reached; GV_BC_PULL=<alpha> overrides it (0: push every level).  On
// R-MAT scale 22 this takes the forward of 64 sources from 21.1 to 15.2 ms;
// 32-source passes push every level (pull levels made them slower: their
// push adds touch half the row bytes).  A pull level reads a vertex's stored
// entries as its in-neighbours, so directed stores push every level.
constexpr uint32_t MS_PULL_ALPHA = 2;
template <int NW>
uint32_t ms_pull_alpha(bool directed) {
    if (directed) return 0;
    const char *env = std::getenv("GV_BC_PULL");
    if (env) return (uint32_t)std::strtoul(env, nullptr, 10);
    return NW == 2 ? MS_PULL_ALPHA : 0;
}

// A whole pass (forward, then dependencies) over 32 NW source slots.
template <int NW>
gv_status ms_pass(gv_graph *g, MsArena &a, const uint32_t *slots, uint32_t out0, uint32_t out1,
                  cudaStream_t s) {
    using M = typename MaskOf<NW>::type;
    MsBufs<NW> b = a.bufs<NW>(g);
    b.out[0] = out0;
    b.out[1] = out1;
    for (uint32_t i = 0; i < 32u * NW; ++i)
        if (slots[i] != GV_NIL) b.full |= (M)1 << i;
    b.alpha = ms_pull_alpha<NW>(g->cfg.directed != 0);
    cudaError_t e = cudaMemcpyAsync(a.dsrc, slots, 32 * NW * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_status(e, "bc sources");
    uint32_t depth = 0;
    gv_status st = ms_forward<NW>(g, a, b, &depth, s);
    if (st != GV_OK) return st;
    return ms_backward<NW>(g, a, b, depth, s);
}

struct SourceGroup {
    uint32_t req;
    uint64_t first;
    uint32_t count;
};

}  // namespace

// Device bytes that k requests scored together take in scratch (a search of up
// to 30 levels).
uint64_t bc_scratch_bytes(const gv_graph *g, uint32_t k) {
    return MsLayout(g->d, 2, k).bytes + 32ull * 8 * g->d.n;
}

// Scores of nreq requests: request r holds hs[off[r] .. off[r+1]) (empty:
// every vertex) and adds into score row r.  Requests are cut into groups of
// up to 32 sources; consecutive groups are paired into 64-source passes (the
// last group alone runs a 32-source pass), so two requests of up to 32
// sources share every adjacency read of their BFS.
gv_status bc_requests(gv_graph *g, std::vector<uint32_t> &hs, std::vector<uint64_t> &off, uint32_t nreq,
                      float *out, int mem, cudaStream_t s) {
    const uint32_t n = g->d.n;
    for (uint32_t v : hs)
        if (v >= n) { set_error("BC source out of range"); return GV_ERR_INVALID; }
    std::vector<SourceGroup> groups;
    std::vector<uint32_t> all;
    for (uint32_t r = 0; r < nreq; ++r) {
        uint64_t lo = off[r], hi = off[r + 1];
        if (lo == hi) {  // every vertex
            if (all.empty()) {
                all.resize(n);
                for (uint32_t i = 0; i < n; ++i) all[i] = i;
            }
            lo = hs.size();
            hs.insert(hs.end(), all.begin(), all.end());
            hi = hs.size();
        }
        for (uint64_t i = lo; i < hi; i += 32) groups.push_back({r, i, (uint32_t)std::min<uint64_t>(32, hi - i)});
    }
    MsArena a;
    gv_status st = ms_setup(g, groups.size() > 1 ? 2 : 1, nreq, a, s);
    if (st != GV_OK) return st;
    cudaMemsetAsync(a.bc, 0, (size_t)n * 8 * nreq, s);
    std::vector<uint32_t> slots(64);
    for (size_t i = 0; i < groups.size() && st == GV_OK; i += 2) {
        std::fill(slots.begin(), slots.end(), GV_NIL);
        const SourceGroup &x = groups[i];
        std::copy(hs.begin() + x.first, hs.begin() + x.first + x.count, slots.begin());
        if (i + 1 < groups.size()) {
            const SourceGroup &y = groups[i + 1];
            std::copy(hs.begin() + y.first, hs.begin() + y.first + y.count, slots.begin() + 32);
            st = ms_pass<2>(g, a, slots.data(), x.req, y.req, s);
        } else {
            st = ms_pass<1>(g, a, slots.data(), x.req, x.req, s);
        }
    }
    if (st != GV_OK) return st;
    float *tmp = (float *)a.row;  // the sigma rows are free once every pass is done
    for (uint32_t r = 0; r < nreq; ++r) {
        float *dst = out + (size_t)r * n;
        GV_LAUNCH(k_ms_to_f32, grid_for(n, 256), 256, 0, s, (const double *)(a.bc + (size_t)r * n),
                  mem == GV_MEM_DEVICE ? dst : tmp, n);
        if (mem != GV_MEM_DEVICE) {
            cudaError_t e = cudaMemcpyAsync(dst, tmp, (size_t)n * 4, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // tmp is reused by the next row
            if (e != cudaSuccess) return cuda_status(e, "bc out");
        }
    }
    return cuda_status(cudaStreamSynchronize(s), "bc out");
}

gv_status bfs_sigma_impl(gv_graph *g, uint32_t source, int32_t *dist, uint64_t *sigma, int mem, cudaStream_t s) {
    const uint32_t n = g->d.n;
    MsArena a;
    gv_status st = ms_setup(g, 1, 1, a, s);
    if (st != GV_OK) return st;
    MsBufs<1> b = a.bufs<1>(g);
    uint32_t slots[32];
    std::fill(slots, slots + 32, GV_NIL);
    slots[0] = source;
    cudaError_t e = cudaMemcpyAsync(a.dsrc, slots, sizeof(slots), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // slots is a stack array
    if (e != cudaSuccess) return cuda_status(e, "bfs source");
    uint32_t depth = 0;
    st = ms_forward<1>(g, a, b, &depth, s);
    if (st != GV_OK) return st;
    // dist (int32) and sigma (u64) staged in a list and the score row (n * 4 and n * 8 bytes)
    int32_t *ddist = (int32_t *)a.lists;
    unsigned long long *dsig = (unsigned long long *)a.bc;
    GV_LAUNCH(k_ms_extract, grid_for(n, 256), 256, 0, s, b, depth, ddist, dsig);
    const cudaMemcpyKind k = mem == GV_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    e = cudaMemcpyAsync(dist, ddist, (size_t)n * 4, k, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(sigma, dsig, (size_t)n * 8, k, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return cuda_status(e, "bfs sigma");
}

// Sources from host or device memory into a host vector.
gv_status bc_host_sources(const uint32_t *sources, uint64_t ns, int mem, cudaStream_t s, std::vector<uint32_t> &hs) {
    hs.resize(ns);
    if (!ns) return GV_OK;
    if (mem == GV_MEM_DEVICE) {
        cudaError_t e = cudaMemcpyAsync(hs.data(), sources, ns * 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return cuda_status(e, "bc sources");
    }
    std::copy(sources, sources + ns, hs.begin());
    return GV_OK;
}

}  // namespace gv

using namespace gv;

extern "C" gv_status gv_bc(gv_graph *g, const uint32_t *sources, uint64_t ns, float *bc_out, int mem, void *stream) {
    if (!g || !bc_out) return GV_ERR_INVALID;
    if (!sources) ns = 0;  // every vertex
    const cudaStream_t s = (cudaStream_t)stream;
    std::vector<uint32_t> hs;
    gv_status st = bc_host_sources(sources, ns, mem, s, hs);
    if (st != GV_OK) return st;
    std::vector<uint64_t> off{0, hs.size()};
    return bc_requests(g, hs, off, 1, bc_out, mem, s);
}

extern "C" gv_status gv_bc_multi(gv_graph *g, const uint32_t *sources, const uint64_t *offsets, uint32_t nreq,
                                 float *bc_out, int mem, void *stream) {
    if (!g || !bc_out || !offsets || nreq == 0) return GV_ERR_INVALID;
    if ((uint64_t)nreq * std::max<uint32_t>(g->d.n, 1) > (1ull << 40)) {  // fp64 score rows in device scratch
        set_error("too many BC requests for one call");
        return GV_ERR_INVALID;
    }
    for (uint32_t r = 0; r < nreq; ++r)
        if (offsets[r + 1] < offsets[r]) { set_error("request offsets must not decrease"); return GV_ERR_INVALID; }
    if (offsets[0] != 0) { set_error("request offsets start at 0"); return GV_ERR_INVALID; }
    if (offsets[nreq] && !sources) return GV_ERR_INVALID;
    const cudaStream_t s = (cudaStream_t)stream;
    std::vector<uint32_t> hs;
    gv_status st = bc_host_sources(sources, offsets[nreq], mem, s, hs);
    if (st != GV_OK) return st;
    std::vector<uint64_t> off(offsets, offsets + nreq + 1);
    return bc_requests(g, hs, off, nreq, bc_out, mem, s);
}

extern "C" gv_status gv_bfs_sigma(gv_graph *g, uint32_t source, int32_t *dist, uint64_t *sigma, int mem, void *stream) {
    if (!g || !dist || !sigma || source >= g->d.n) return GV_ERR_INVALID;
    return bfs_sigma_impl(g, source, dist, sigma, mem, (cudaStream_t)stream);
}
