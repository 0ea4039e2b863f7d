// Batched edge insert / delete and compaction on the edge-block CBT store.
//
// One batch runs as a stream-ordered pipeline with no host round trip:
//   expand   pairs -> 64-bit keys (src << bits | dst), both directions on an
//            undirected graph; self-loops and out-of-range ids become the
//            sentinel key, which sorts last.  Range errors abort the batch.
//   sort     stable LSD radix sort of the keys (prims.cu) = the batch staged
//            sorted and segmented by source vertex.
//   segment  adjacent-unique compaction: bdst[] (sorted, de-duplicated
//            destinations) and one segment {vertex, start} per touched vertex.
//   member   one lane group per segment (a whole CTA for hubs) streams the
//            vertex's existing blocks with 16-byte loads and binary-searches
//            each entry in the segment: insert marks batch entries that
//            already exist, delete tombstones matching graph entries.
//   plan     blocks each segment needs; warp-aggregated atomics hand out
//            contiguous ranges of the free stack.
//   admit    rejects the whole batch if the pool cannot hold it.
//   apply    writes new entries after the last used slot, links the new
//            blocks into the CBT (children 2k+1 / 2k+2, level-order
//            predecessor) and updates the vertex record.
// Reference pipeline replaced: src/dynamicStructure/graphvine.cu:222-451 with
// kernels src/dynamicStructure/kernels/insert_kernels.cu:3-365 and
// src/dynamicStructure/kernels/delete_kernels.cu:3-48.
#include <algorithm>
#include <type_traits>
#include "store.cuh"
#include "group.cuh"
#include "prims.cuh"
#include "launch.hpp"
#include "prof.hpp"

namespace gv {

unsigned grid_for(uint64_t work_items, unsigned per_cta, unsigned max_ctas) {
    uint64_t g = (work_items + per_cta - 1) / per_cta;
    if (g < 1) g = 1;
    if (g > max_ctas) g = max_ctas;
    return (unsigned)g;
}

namespace {

constexpr int UPD_THREADS = 256;
constexpr int SEG_THREADS = 256;
constexpr int SEG_ITEMS = 8;
constexpr int SEG_TILE = SEG_THREADS * SEG_ITEMS;
constexpr int BIG_TAB = 1024;  // block-table chunk of the CTA-per-vertex paths

// What goes to a whole CTA: long segments, and vertices that would keep their
// lane group scanning long after the others are done (more than 32 quads per
// lane, see gv_create).
__device__ __forceinline__ bool is_big_vertex(const DevGraph &g, uint32_t fill, uint32_t nb) {
    return nb > BIG_BLOCKS || fill > g.big_fill;
}
__device__ __forceinline__ bool is_big(const DevGraph &g, uint32_t fill, uint32_t nb, uint32_t len) {
    return is_big_vertex(g, fill, nb) || len > BIG_SEGMENT;
}

// Lower bounds of four values in sorted D[0, len), len > 0, side by side: the
// halvings are the same for all, so the four loads of a step are in flight
// together (one value after another, a hub's scan waits for 18 loads in turn
// per entry).
__device__ __forceinline__ void lower_bound4(const uint32_t *D, uint32_t len, const uint32_t (&x)[4],
                                             uint32_t (&at)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) at[j] = 0;
    for (uint32_t n = len; n > 1;) {
        const uint32_t half = n >> 1;
#pragma unroll
        for (int j = 0; j < 4; ++j) at[j] += D[at[j] + half - 1] < x[j] ? half : 0u;
        n -= half;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) at[j] += D[at[j]] < x[j] ? 1u : 0u;
}

// Vertices that a CTA finds dirty, gathered in shared memory and appended to
// the store's list with one atomic: the list's counter is one address, and
// a return trip to it per vertex was most of a delete's time.
constexpr uint32_t DIRTY_BUF = 1024;
struct DirtyBuf {
    uint32_t v[DIRTY_BUF];
    uint32_t cnt;
    unsigned long long base;
};

__device__ __forceinline__ void dirty_push(const DevGraph &g, DirtyBuf &d, uint32_t u) {
    if (g.dirty[u]) return;
    g.dirty[u] = 1;
    const uint32_t p = atomicAdd(&d.cnt, 1u);
    if (p < DIRTY_BUF) d.v[p] = u;
    else g.dirty_list[atomicAdd(&g.ctl->ndirty, 1ull)] = u;
}

// All threads of the CTA.
__device__ __forceinline__ void dirty_flush(const DevGraph &g, DirtyBuf &d) {
    __syncthreads();
    const uint32_t n = min(d.cnt, DIRTY_BUF);
    if (threadIdx.x == 0 && n) d.base = atomicAdd(&g.ctl->ndirty, (unsigned long long)n);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) g.dirty_list[d.base + i] = d.v[i];
}

// ------------------------------------------------------------------ expand
__global__ void k_expand(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst,
                         uint64_t k, int sym, uint32_t n, uint32_t bitsn,
                         unsigned long long *__restrict__ keys, uint32_t *__restrict__ vals,
                         Ctl *ctl) {
    const unsigned long long sent = (bitsn >= 32) ? ~0ull : ((1ull << (2 * bitsn)) - 1ull);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = src[i], d = dst[i];
        const bool bad = (s >= n) || (d >= n);
        if (bad) {
            atomicOr(&ctl->status, GV_DEV_ERR_RANGE);
            ctl->batch_abort = 1;
        }
        const bool drop = bad || (s == d);
        if (sym) {
            keys[2 * i] = drop ? sent : (((unsigned long long)s << bitsn) | d);
            keys[2 * i + 1] = drop ? sent : (((unsigned long long)d << bitsn) | s);
            if (vals) {
                vals[2 * i] = (uint32_t)(2 * i);
                vals[2 * i + 1] = (uint32_t)(2 * i + 1);
            }
        } else {
            keys[i] = drop ? sent : (((unsigned long long)s << bitsn) | d);
            if (vals) vals[i] = (uint32_t)i;
        }
    }
}

// ----------------------------------------------------------------- segment
__device__ __forceinline__ void seg_flags(const unsigned long long *K, uint64_t i, uint64_t N,
                                          unsigned long long sent, uint32_t bitsn, bool &uniq,
                                          bool &head) {
    uniq = head = false;
    if (i >= N) return;
    const unsigned long long key = K[i];
    if (key == sent) return;
    if (i == 0) {
        uniq = head = true;
        return;
    }
    const unsigned long long prev = K[i - 1];
    uniq = key != prev;
    head = uniq && ((key >> bitsn) != (prev >> bitsn));
}

__global__ void __launch_bounds__(SEG_THREADS) k_seg_count(const unsigned long long *__restrict__ K,
                                                           uint64_t N, unsigned long long sent,
                                                           uint32_t bitsn,
                                                           unsigned long long *__restrict__ tile_cnt) {
    __shared__ unsigned long long wt[33];
    const uint64_t base = (uint64_t)blockIdx.x * SEG_TILE + (uint64_t)threadIdx.x * SEG_ITEMS;
    unsigned long long c = 0;
#pragma unroll
    for (int j = 0; j < SEG_ITEMS; ++j) {
        bool u, h;
        seg_flags(K, base + j, N, sent, bitsn, u, h);
        c += ((unsigned long long)u << 32) | (unsigned long long)h;
    }
    unsigned long long tot = cta_sum<unsigned long long, SEG_THREADS>(c, wt);
    if (threadIdx.x == 0) tile_cnt[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SEG_THREADS) k_seg_write(
    const unsigned long long *__restrict__ K, const uint32_t *__restrict__ V, uint64_t N,
    unsigned long long sent, uint32_t bitsn, int sym_shift,
    const unsigned long long *__restrict__ tile_off, const float *__restrict__ in_w,
    uint32_t *__restrict__ bdst, float *__restrict__ bw, uint8_t *__restrict__ found,
    uint32_t *__restrict__ seg_vertex, uint32_t *__restrict__ seg_start, uint8_t *affected,
    Ctl *ctl) {
    __shared__ unsigned long long wt[33];
    const uint64_t base = (uint64_t)blockIdx.x * SEG_TILE + (uint64_t)threadIdx.x * SEG_ITEMS;
    const unsigned long long dmask = (1ull << bitsn) - 1ull;
    unsigned long long c = 0;
    bool uf[SEG_ITEMS], hf[SEG_ITEMS];
#pragma unroll
    for (int j = 0; j < SEG_ITEMS; ++j) {
        seg_flags(K, base + j, N, sent, bitsn, uf[j], hf[j]);
        c += ((unsigned long long)uf[j] << 32) | (unsigned long long)hf[j];
    }
    unsigned long long tot;
    unsigned long long pre = cta_excl_scan<unsigned long long, SEG_THREADS>(c, wt, tot) + tile_off[blockIdx.x];
    uint32_t up = (uint32_t)(pre >> 32), hp = (uint32_t)(pre & 0xFFFFFFFFull);
#pragma unroll
    for (int j = 0; j < SEG_ITEMS; ++j) {
        if (!uf[j]) continue;
        const unsigned long long key = K[base + j];
        const uint32_t s = (uint32_t)(key >> bitsn), d = (uint32_t)(key & dmask);
        bdst[up] = d;
        found[up] = 0;
        if (bw) bw[up] = in_w[V[base + j] >> sym_shift];
        affected[s] = 1;
        affected[d] = 1;
        if (hf[j]) {
            seg_vertex[hp] = s;
            seg_start[hp] = up;
            ++hp;
        }
        ++up;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // The scan wrote the packed grand total into ctl->scratch0.
        const unsigned long long t = ctl->scratch0;
        const uint32_t nuniq = (uint32_t)(t >> 32), nseg = (uint32_t)(t & 0xFFFFFFFFull);
        ctl->nuniq = nuniq;
        ctl->nseg = nseg;
        seg_start[nseg] = nuniq;
    }
}

// ------------------------------------------------------------- small batch
// expand, sort and segment of a batch of at most SB_KEYS directed entries in
// one launch of one CTA; the results are those of the launches above, which
// cost such a batch some twenty launches of a few microseconds each.  The sort
// is the same stable LSD radix sort, 8 bits a pass: a warp owns up to SB_PER
// consecutive runs of 32 keys and ranks them against counters of its own, so a
// pass has four barriers.  1,000 pairs on 16 K vertices: 19 us, where the
// separate launches took 75 (and the driver another 35).
constexpr int SB_THREADS = 512;
constexpr int SB_WARPS = SB_THREADS / 32;
constexpr int SB_PER = 8;
constexpr uint32_t SB_KEYS = SB_THREADS * SB_PER;

template <bool VALS>
struct SbSmem {
    unsigned long long keys[SB_KEYS];
    uint32_t vals[VALS ? SB_KEYS : 1];
    uint32_t cnt[SB_WARPS][256];
    uint32_t wt[33];
    unsigned long long wt64[33];
};

template <bool VALS>
__global__ void __launch_bounds__(SB_THREADS) k_small_batch(
    const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, const float *__restrict__ in_w, uint32_t k,
    int sym, uint32_t n, uint32_t bitsn, uint32_t *__restrict__ bdst, float *__restrict__ bw,
    uint8_t *__restrict__ found, uint32_t *__restrict__ seg_vertex, uint32_t *__restrict__ seg_start, uint8_t *affected,
    Ctl *ctl) {
    extern __shared__ __align__(16) unsigned char sb_raw[];
    SbSmem<VALS> &S = *reinterpret_cast<SbSmem<VALS> *>(sb_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const unsigned long long sent = (bitsn >= 32) ? ~0ull : ((1ull << (2 * bitsn)) - 1ull);
    const uint32_t E = sym ? 2 * k : k;
    bool bad = false;
    for (uint32_t e = tid; e < SB_KEYS; e += SB_THREADS) {
        unsigned long long key = sent;
        if (e < E) {
            const uint32_t i = sym ? e >> 1 : e;
            uint32_t a = src[i], b = dst[i];
            const bool out = a >= n || b >= n;
            bad |= out;
            if (sym && (e & 1u)) {
                const uint32_t t = a;
                a = b;
                b = t;
            }
            if (!out && a != b) key = ((unsigned long long)a << bitsn) | b;
        }
        S.keys[e] = key;
        if (VALS) S.vals[e] = e;
    }
    if (bad) {
        atomicOr(&ctl->status, GV_DEV_ERR_RANGE);
        ctl->batch_abort = 1;
    }
    // whole runs of 32 keys only; the rest would be sentinels, which sort last
    const uint32_t runs = (E + 31) >> 5, per = (runs + SB_WARPS - 1) / SB_WARPS;
    for (uint32_t shift = 0; shift < 2 * bitsn; shift += 8) {
        for (uint32_t i = tid; i < SB_WARPS * 256; i += SB_THREADS) (&S.cnt[0][0])[i] = 0;
        __syncthreads();
        unsigned long long key[SB_PER];
        uint32_t val[SB_PER], rank[SB_PER];
#pragma unroll
        for (int j = 0; j < SB_PER; ++j) {
            const uint32_t run = warp * per + j;
            if (j >= per || run >= runs) break;  // warp-uniform
            key[j] = S.keys[run * 32 + lane];
            if (VALS) val[j] = S.vals[run * 32 + lane];
            const uint32_t d = (uint32_t)(key[j] >> shift) & 0xFFu;
            const uint32_t peers = digit_peers(d, true);
            const uint32_t below = __popc(peers & ((1u << lane) - 1u));
            const uint32_t before = S.cnt[warp][d];
            rank[j] = before + below;
            __syncwarp();
            if (below == 0) S.cnt[warp][d] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        // counts to places: digit by digit, and within a digit warp by warp
        uint32_t c[SB_WARPS], mine = 0;
        if (tid < 256) {
#pragma unroll
            for (int w = 0; w < SB_WARPS; ++w) {
                c[w] = S.cnt[w][tid];
                mine += c[w];
            }
        }
        uint32_t tot;
        uint32_t at = cta_excl_scan<uint32_t, SB_THREADS>(mine, S.wt, tot);
        if (tid < 256) {
#pragma unroll
            for (int w = 0; w < SB_WARPS; ++w) {
                S.cnt[w][tid] = at;
                at += c[w];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SB_PER; ++j) {
            if (j >= per || warp * per + j >= runs) break;
            const uint32_t p = S.cnt[warp][(uint32_t)(key[j] >> shift) & 0xFFu] + rank[j];
            S.keys[p] = key[j];
            if (VALS) S.vals[p] = val[j];
        }
        __syncthreads();
    }
    // segments, as k_seg_write cuts them
    unsigned long long c = 0;
    uint32_t uniq = 0, head = 0;
#pragma unroll
    for (int j = 0; j < SB_PER; ++j) {
        bool u, h;
        seg_flags(S.keys, tid * SB_PER + j, E, sent, bitsn, u, h);
        uniq |= (uint32_t)u << j;
        head |= (uint32_t)h << j;
        c += ((unsigned long long)u << 32) | (unsigned long long)h;
    }
    unsigned long long tot;
    const unsigned long long pre = cta_excl_scan<unsigned long long, SB_THREADS>(c, S.wt64, tot);
    uint32_t up = (uint32_t)(pre >> 32), hp = (uint32_t)pre;
#pragma unroll
    for (int j = 0; j < SB_PER; ++j) {
        if (!((uniq >> j) & 1u)) continue;
        const unsigned long long key = S.keys[tid * SB_PER + j];
        const uint32_t a = (uint32_t)(key >> bitsn), b = (uint32_t)(key & ((1ull << bitsn) - 1ull));
        bdst[up] = b;
        found[up] = 0;
        if (VALS) bw[up] = in_w[S.vals[tid * SB_PER + j] >> (sym ? 1 : 0)];
        affected[a] = 1;
        affected[b] = 1;
        if ((head >> j) & 1u) {
            seg_vertex[hp] = a;
            seg_start[hp] = up;
            ++hp;
        }
        ++up;
    }
    if (tid == 0) {
        const uint32_t nuniq = (uint32_t)(tot >> 32), nseg = (uint32_t)tot;
        ctl->nuniq = nuniq;
        ctl->nseg = nseg;
        seg_start[nseg] = nuniq;
    }
}

// ------------------------------------------------------------------ member
// Entries ev[0, 4) at slot, the first of them entry e of fill: marks the
// segment's entries among them as found, DEL tombstones them; returns how many.
template <bool DEL>
__device__ __forceinline__ uint32_t member_quad(uint32_t *slot, uint32_t e, uint32_t fill, const uint32_t *D,
                                                uint32_t len, uint8_t *found) {
    const uint4 v = *reinterpret_cast<const uint4 *>(slot);
    const uint32_t ev[4] = {v.x, v.y, v.z, v.w};
    uint32_t at[4], cnt = 0;
    lower_bound4(D, len, ev, at);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (e + j < fill && ev[j] != GV_TOMB && at[j] < len && D[at[j]] == ev[j]) {
            ++cnt;
            found[at[j]] = 1;
            if (DEL) slot[j] = GV_TOMB;
        }
    return cnt;
}

// A lane group per segment.  Segments are short and their vertices scattered,
// so a group waits on its chain of loads (segment, record, slots, search): the
// next segment's bounds and record are loaded while this one's slots are
// scanned, and one-block vertices skip the block table.  On R-MAT scale 22,
// 500 K pairs (1 M segments of scattered vertices): delete 1.37 -> 0.29 ms
// (with an atomic on the live count and the dirty list per segment most of it
// was those two addresses), insert 0.29 -> 0.19 ms.
template <int TPV, bool DEL>
__global__ void __launch_bounds__(UPD_THREADS) k_member(DevGraph g,
                                                        const uint32_t *__restrict__ seg_vertex,
                                                        const uint32_t *__restrict__ seg_start,
                                                        const uint32_t *__restrict__ bdst,
                                                        uint8_t *__restrict__ found,
                                                        uint32_t *__restrict__ seg_found,
                                                        uint32_t *__restrict__ big_list) {
    constexpr int GPC = UPD_THREADS / TPV;
    __shared__ uint32_t tabs[GPC][BIG_BLOCKS];
    __shared__ DirtyBuf dirty;
    if (DEL && g.ctl->batch_abort) return;
    if (DEL) {
        if (threadIdx.x == 0) dirty.cnt = 0;
        __syncthreads();
    }
    const uint32_t nseg = (uint32_t)g.ctl->nseg;
    Group<TPV> G;
    const uint32_t gcta = threadIdx.x / TPV;
    uint32_t *tab = tabs[gcta];
    const uint32_t ngroups = gridDim.x * GPC;
    uint32_t removed = 0;
    uint32_t s = blockIdx.x * GPC + gcta, u = 0, st = 0, en = 0;
    uint4 rec = make_uint4(0u, 0u, 0u, 0u);
    if (s < nseg) {
        u = seg_vertex[s];
        st = seg_start[s];
        en = seg_start[s + 1];
        rec = g.vtx[u];
    }
    while (s < nseg) {
        const uint32_t s2 = s + ngroups;
        uint32_t u2 = 0, st2 = 0, en2 = 0;
        if (s2 < nseg) {
            u2 = seg_vertex[s2];
            st2 = seg_start[s2];
            en2 = seg_start[s2 + 1];
        }
        const uint32_t len = en - st, fill = rec.y, nb = blocks_for(fill, g.logB);
        const bool big = is_big(g, fill, nb, len);
        uint32_t cnt = 0;
        if (big) {
            if (G.gl == 0) big_list[atomicAdd(&g.ctl->nbig, 1ull)] = s;
        } else {
            if (nb > 1) {
                fill_block_table(g, rec.x, 0, nb, tab, G.gl, TPV);
                G.sync();
            }
            const uint32_t nq = (fill + 3) >> 2;
            for (uint32_t q = G.gl; q < nq; q += TPV) {
                const uint32_t e = q << 2;
                const uint32_t b = nb > 1 ? tab[e >> g.logB] : rec.x;
                cnt += member_quad<DEL>(g.pool + ((size_t)b << g.logB) + (e & (g.B - 1)), e, fill, bdst + st, len,
                                        found + st);
            }
        }
        uint4 rec2 = make_uint4(0u, 0u, 0u, 0u);
        if (s2 < nseg) rec2 = g.vtx[u2];
        if (!big) {
            cnt = G.sum(cnt);
            if (G.gl == 0) {
                seg_found[s] = cnt;
                if (DEL && cnt) {
                    g.vtx[u].z = rec.z - cnt;
                    removed += cnt;
                    dirty_push(g, dirty, u);
                }
            }
        }
        G.sync();
        s = s2;
        u = u2;
        st = st2;
        en = en2;
        rec = rec2;
    }
    if (DEL) {
        removed = warp_sum(removed);
        if ((threadIdx.x & 31u) == 0 && removed)
            atomicAdd(&g.ctl->live_edges, 0ull - (unsigned long long)removed);
        dirty_flush(g, dirty);
    }
}

template <bool DEL>
__global__ void __launch_bounds__(BIG_THREADS) k_member_big(DevGraph g,
                                                            const uint32_t *__restrict__ seg_vertex,
                                                            const uint32_t *__restrict__ seg_start,
                                                            const uint32_t *__restrict__ bdst,
                                                            uint8_t *__restrict__ found,
                                                            uint32_t *__restrict__ seg_found,
                                                            const uint32_t *__restrict__ big_list) {
    __shared__ uint32_t tab[BIG_TAB];
    __shared__ uint32_t wt[33];
    if (DEL && g.ctl->batch_abort) return;
    const uint32_t nbig = (uint32_t)g.ctl->nbig;
    for (uint32_t i = blockIdx.x; i < nbig; i += gridDim.x) {
        const uint32_t s = big_list[i];
        const uint32_t u = seg_vertex[s];
        const uint32_t st = seg_start[s], len = seg_start[s + 1] - st;
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, nb = blocks_for(fill, g.logB);
        const uint32_t *D = bdst + st;
        uint32_t cnt = 0;
        for (uint32_t k0 = 0; k0 < nb; k0 += BIG_TAB) {
            const uint32_t kc = min((uint32_t)BIG_TAB, nb - k0);
            fill_block_table(g, rec.x, k0, kc, tab, threadIdx.x, BIG_THREADS);
            __syncthreads();
            const uint32_t e0 = k0 << g.logB;
            const uint32_t e1 = min(fill, (k0 + kc) << g.logB);
            const uint32_t nq = (e1 - e0 + 3) >> 2;
            for (uint32_t q = threadIdx.x; q < nq; q += BIG_THREADS) {
                const uint32_t e = e0 + (q << 2);
                const uint32_t b = tab[(e >> g.logB) - k0];
                cnt += member_quad<DEL>(g.pool + ((size_t)b << g.logB) + (e & (g.B - 1)), e, fill, D, len, found + st);
            }
            __syncthreads();
        }
        cnt = cta_sum<uint32_t, BIG_THREADS>(cnt, wt);
        if (threadIdx.x == 0) {
            seg_found[s] = cnt;
            if (DEL && cnt) {
                g.vtx[u].z = rec.z - cnt;
                atomicAdd(&g.ctl->live_edges, (unsigned long long)(-(long long)cnt));
                if (!g.dirty[u]) {
                    g.dirty[u] = 1;
                    g.dirty_list[atomicAdd(&g.ctl->ndirty, 1ull)] = u;
                }
            }
        }
        __syncthreads();
    }
}

// -------------------------------------------------------------- plan/admit
__global__ void __launch_bounds__(UPD_THREADS) k_plan(DevGraph g, const uint32_t *__restrict__ seg_vertex,
                                                      const uint32_t *__restrict__ seg_start,
                                                      const uint32_t *__restrict__ seg_found,
                                                      uint32_t *__restrict__ seg_newblocks,
                                                      uint32_t *__restrict__ seg_blkbase) {
    if (g.ctl->batch_abort) return;
    const uint32_t nseg = (uint32_t)g.ctl->nseg;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < nseg; base += stride) {
        const uint32_t s = base + threadIdx.x;
        uint32_t need = 0;
        if (s < nseg) {
            const uint32_t u = seg_vertex[s];
            const uint32_t newcnt = (seg_start[s + 1] - seg_start[s]) - seg_found[s];
            const uint32_t fill = g.vtx[u].y;
            const uint32_t cap = blocks_for(fill, g.logB) << g.logB;
            const uint32_t room = cap - fill;
            const uint32_t extra = newcnt > room ? newcnt - room : 0u;
            need = (extra + g.B - 1) >> g.logB;
            seg_newblocks[s] = need;
        }
        const unsigned long long off = warp_agg_alloc(&g.ctl->alloc_cursor, need);
        if (s < nseg) seg_blkbase[s] = (uint32_t)off;
    }
}

__global__ void k_admit(Ctl *ctl) {
    if (!ctl->batch_abort && ctl->alloc_cursor > ctl->free_top) {
        ctl->batch_abort = 1;
        ctl->status |= GV_DEV_ERR_NOMEM;
    }
}

__global__ void k_finish(Ctl *ctl) {
    if (!ctl->batch_abort) ctl->free_top -= ctl->alloc_cursor;
    ctl->alloc_cursor = 0;
    ctl->nbig = 0;
    ctl->batch_abort = 0;
}

// Commits one stage of a multi-stage window but keeps the abort flag, so a
// window rejected in an earlier stage skips the later ones too.
__global__ void k_commit_keep_abort(Ctl *ctl) {
    if (!ctl->batch_abort) ctl->free_top -= ctl->alloc_cursor;
    ctl->alloc_cursor = 0;
    ctl->nbig = 0;
}

// ------------------------------------------------------------------- apply
// Pool index of new block t of a segment (popped from the top of the stack).
__device__ __forceinline__ uint32_t new_block(const DevGraph &g, unsigned long long top, uint32_t base,
                                              uint32_t t) {
    return g.free_stack[top - 1ull - (unsigned long long)(base + t)];
}

// Initialises the new blocks, then links them into the tree (two passes so
// a parent that is itself new is initialised before its child pointer is set).
template <typename SyncF>
__device__ __forceinline__ void link_new_blocks(const DevGraph &g, uint32_t u, uint4 rec, uint32_t nb_old,
                                                uint32_t nnew, uint32_t newfill,
                                                unsigned long long top, uint32_t base,
                                                uint32_t t0, uint32_t nt, SyncF sync) {
    for (uint32_t t = t0; t < nnew; t += nt) {
        const uint32_t k = nb_old + t;
        const uint32_t b = new_block(g, top, base, t);
        g.left[b] = GV_NIL;
        g.right[b] = GV_NIL;
        g.owner[b] = u;
        g.bcount[b] = min(g.B, newfill - (k << g.logB));
        g.pred[b] = (k == 0) ? GV_NIL : (t == 0 ? rec.w : new_block(g, top, base, t - 1));
    }
    sync();
    for (uint32_t t = t0; t < nnew; t += nt) {
        const uint32_t k = nb_old + t;
        if (k == 0) continue;
        const uint32_t b = new_block(g, top, base, t);
        const uint32_t pk = (k - 1) >> 1;
        const uint32_t pb = (pk >= nb_old) ? new_block(g, top, base, pk - nb_old)
                                           : cbt_block(g.left, g.right, rec.x, pk);
        if (k & 1u) g.left[pb] = b; else g.right[pb] = b;
    }
}

template <int TPV>
__global__ void __launch_bounds__(UPD_THREADS) k_apply(DevGraph g, const uint32_t *__restrict__ seg_vertex,
                                                       const uint32_t *__restrict__ seg_start,
                                                       const uint32_t *__restrict__ bdst,
                                                       const float *__restrict__ bw,
                                                       const uint8_t *__restrict__ found,
                                                       const uint32_t *__restrict__ seg_found,
                                                       const uint32_t *__restrict__ seg_newblocks,
                                                       const uint32_t *__restrict__ seg_blkbase) {
    constexpr int GPC = UPD_THREADS / TPV;
    if (g.ctl->batch_abort) return;
    const uint32_t nseg = (uint32_t)g.ctl->nseg;
    const unsigned long long top = g.ctl->free_top;
    Group<TPV> G;
    const uint32_t ngroups = gridDim.x * GPC;
    unsigned long long added = 0;  // one atomic per warp: the counter is one address
    for (uint32_t s = blockIdx.x * GPC + threadIdx.x / TPV; s < nseg; s += ngroups) {
        const uint32_t u = seg_vertex[s];
        const uint32_t st = seg_start[s], len = seg_start[s + 1] - st;
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, nb_old = blocks_for(fill, g.logB);
        if (is_big(g, fill, nb_old, len)) continue;
        const uint32_t newcnt = len - seg_found[s];
        if (newcnt == 0) continue;
        const uint32_t nnew = seg_newblocks[s], base = seg_blkbase[s];
        const uint32_t newfill = fill + newcnt;
        uint32_t j0 = 0;
        for (uint32_t c = 0; c < len; c += TPV) {
            const uint32_t i = c + G.gl;
            const uint32_t isnew = (i < len && !found[st + i]) ? 1u : 0u;
            uint32_t tot;
            const uint32_t pre = G.excl_scan(isnew, tot);
            if (isnew) {
                const uint32_t p = fill + j0 + pre;
                const uint32_t k = p >> g.logB;
                const uint32_t b = (k < nb_old) ? rec.w : new_block(g, top, base, k - nb_old);
                const size_t at = ((size_t)b << g.logB) + (p & (g.B - 1));
                g.pool[at] = bdst[st + i];
                if (bw) g.wpool[at] = bw[st + i];
            }
            j0 += tot;
        }
        link_new_blocks(g, u, rec, nb_old, nnew, newfill, top, base, G.gl, TPV, [&] { G.sync(); });
        if (G.gl == 0) {
            if (nb_old > 0) g.bcount[rec.w] = min(g.B, newfill - ((nb_old - 1) << g.logB));
            uint4 nrec;
            nrec.x = nb_old ? rec.x : new_block(g, top, base, 0);
            nrec.y = newfill;
            nrec.z = rec.z + newcnt;
            nrec.w = nnew ? new_block(g, top, base, nnew - 1) : rec.w;
            g.vtx[u] = nrec;
            added += newcnt;
        }
        G.sync();
    }
    added = warp_sum(added);
    if ((threadIdx.x & 31u) == 0 && added) atomicAdd(&g.ctl->live_edges, added);
}

// Appends a big segment's new entries (is_new(i), in order) after slot fill;
// APP_ITEMS consecutive entries per thread and round, so a hub's segment of a
// few hundred thousand entries takes tens of rounds (and barriers), not
// hundreds.
constexpr uint32_t APP_ITEMS = 8;
template <typename IsNew>
__device__ __forceinline__ void cta_append(const DevGraph &g, uint4 rec, uint32_t nb_old, unsigned long long top,
                                           uint32_t base, const uint32_t *D, const float *W, uint32_t len,
                                           uint32_t *wt, IsNew is_new) {
    uint32_t j0 = 0;
    for (uint32_t c = 0; c < len; c += BIG_THREADS * APP_ITEMS) {
        const uint32_t i0 = c + threadIdx.x * APP_ITEMS;
        uint32_t bits = 0;
#pragma unroll
        for (uint32_t j = 0; j < APP_ITEMS; ++j)
            if (i0 + j < len && is_new(i0 + j)) bits |= 1u << j;
        uint32_t tot;
        uint32_t p = rec.y + j0 + cta_excl_scan<uint32_t, BIG_THREADS>(__popc(bits), wt, tot);
#pragma unroll
        for (uint32_t j = 0; j < APP_ITEMS; ++j)
            if ((bits >> j) & 1u) {
                const uint32_t k = p >> g.logB;
                const uint32_t b = (k < nb_old) ? rec.w : new_block(g, top, base, k - nb_old);
                const size_t at = ((size_t)b << g.logB) + (p & (g.B - 1));
                g.pool[at] = D[i0 + j];
                if (W) g.wpool[at] = W[i0 + j];
                ++p;
            }
        j0 += tot;
    }
}

__global__ void __launch_bounds__(BIG_THREADS) k_apply_big(DevGraph g, const uint32_t *__restrict__ seg_vertex,
                                                           const uint32_t *__restrict__ seg_start,
                                                           const uint32_t *__restrict__ bdst,
                                                           const float *__restrict__ bw,
                                                           const uint8_t *__restrict__ found,
                                                           const uint32_t *__restrict__ seg_found,
                                                           const uint32_t *__restrict__ seg_newblocks,
                                                           const uint32_t *__restrict__ seg_blkbase,
                                                           const uint32_t *__restrict__ big_list) {
    __shared__ uint32_t wt[33];
    if (g.ctl->batch_abort) return;
    const uint32_t nbig = (uint32_t)g.ctl->nbig;
    const unsigned long long top = g.ctl->free_top;
    for (uint32_t bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
        const uint32_t s = big_list[bi];
        const uint32_t u = seg_vertex[s];
        const uint32_t st = seg_start[s], len = seg_start[s + 1] - st;
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, nb_old = blocks_for(fill, g.logB);
        const uint32_t newcnt = len - seg_found[s];
        if (newcnt == 0) continue;  // uniform across the CTA
        const uint32_t nnew = seg_newblocks[s], base = seg_blkbase[s];
        const uint32_t newfill = fill + newcnt;
        cta_append(g, rec, nb_old, top, base, bdst + st, bw ? bw + st : nullptr, len, wt,
                   [&](uint32_t i) { return !found[st + i]; });
        link_new_blocks(g, u, rec, nb_old, nnew, newfill, top, base, threadIdx.x, BIG_THREADS,
                        [] { __syncthreads(); });
        __syncthreads();
        if (threadIdx.x == 0) {
            if (nb_old > 0) g.bcount[rec.w] = min(g.B, newfill - ((nb_old - 1) << g.logB));
            uint4 nrec;
            nrec.x = nb_old ? rec.x : new_block(g, top, base, 0);
            nrec.y = newfill;
            nrec.z = rec.z + newcnt;
            nrec.w = nnew ? new_block(g, top, base, nnew - 1) : rec.w;
            g.vtx[u] = nrec;
            atomicAdd(&g.ctl->live_edges, (unsigned long long)newcnt);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ window apply
// A window's net updates in one persistent launch.  The window has been
// reduced to the last operation per pair, so every touched vertex u has one
// segment: its destinations sorted, each marked insert or delete, and no
// pair appears twice.  Units of work are segments, taken from a device
// queue: first the big ones (is_big), one per CTA, then chunks of WIN_CHUNK small ones per warp, a
// lane group per segment.  A unit scans u's blocks once: an entry found
// among the segment's deletes becomes a tombstone, one found among its
// inserts marks that insert as already present.  The remaining inserts are
// appended after the last used slot into blocks popped from the free stack
// (warp-aggregated atomics), the new blocks are linked into the CBT and the
// vertex record is rewritten.  The caller has checked that the free stack
// holds the window's worst case (one block per segment plus one per B
// inserts), so no unit can run out; a unit that would still overrun the
// stack records GV_DEV_ERR_NOMEM and writes nothing past it.
// A window of 64 batches, 2.4 M pairs of Zipf(1.1) sources on R-MAT scale 20:
// 2.6 ms, of which the hottest vertex alone (0.3 M entries searched one load
// at a time in a segment of 0.3 M) took most; 0.67 ms with four searches side
// by side, eight entries per thread in its append, vertices above 128 slots
// per lane on the CTA side, and the counters' atomics gathered.
// Its segments are chains of loads, so warps in flight count for more than the
// registers that few of them could have: 0.57 ms with four CTAs per SM and
// chunks of 16 segments, 0.58 with three, 0.66 with the two that fit 64
// registers a thread (0.67 with chunks of 64).
constexpr uint32_t WIN_CHUNK = 16;
constexpr int WIN_CTAS = 4;

struct WinSegs {
    const uint32_t *seg_vertex, *seg_start, *bdst;
    const uint32_t *btype;       // per entry: 1 insert, 0 delete
    uint8_t *found;              // per entry: the insert is already stored
    uint32_t *big_list;          // big segments
    unsigned long long *queue;   // [0] next big unit, [1] next small chunk, [2] big units
};

__device__ __forceinline__ uint32_t win_new_blocks(uint32_t fill, uint32_t nb_old, uint32_t newcnt, uint32_t logB) {
    const uint32_t room = (nb_old << logB) - fill;
    const uint32_t extra = newcnt > room ? newcnt - room : 0u;
    return (extra + (1u << logB) - 1u) >> logB;
}

// Rewrites u's record after a unit (one thread).
__device__ __forceinline__ void win_record(const DevGraph &g, uint32_t u, uint4 rec, uint32_t nb_old, uint32_t newcnt,
                                           uint32_t nnew, uint32_t ndel, unsigned long long top, uint32_t base,
                                           DirtyBuf &dirty) {
    if (!newcnt && !ndel) return;
    uint4 nrec = rec;
    if (newcnt) {
        const uint32_t newfill = rec.y + newcnt;
        if (nb_old > 0) g.bcount[rec.w] = min(g.B, newfill - ((nb_old - 1) << g.logB));
        nrec.x = nb_old ? rec.x : new_block(g, top, base, 0);
        nrec.y = newfill;
        nrec.w = nnew ? new_block(g, top, base, nnew - 1) : rec.w;
    }
    nrec.z = rec.z - ndel + newcnt;
    g.vtx[u] = nrec;
    if (ndel) dirty_push(g, dirty, u);
}

// As member_quad for a window's segment: deletes (T 0) tombstone their entry,
// inserts (T 1) are marked as found; returns the number of deletes.
__device__ __forceinline__ uint32_t win_quad(uint32_t *slot, uint32_t e, uint32_t fill, const uint32_t *D,
                                             const uint32_t *T, uint32_t len, uint8_t *found) {
    const uint4 v = *reinterpret_cast<const uint4 *>(slot);
    const uint32_t ev[4] = {v.x, v.y, v.z, v.w};
    uint32_t at[4], ndel = 0;
    lower_bound4(D, len, ev, at);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (e + j < fill && ev[j] != GV_TOMB && at[j] < len && D[at[j]] == ev[j]) {
            if (T[at[j]]) found[at[j]] = 1;
            else {
                slot[j] = GV_TOMB;
                ++ndel;
            }
        }
    return ndel;
}

__global__ void k_window_classify(DevGraph g, WinSegs w) {
    const uint32_t nseg = (uint32_t)g.ctl->nseg;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
        const uint32_t len = w.seg_start[s + 1] - w.seg_start[s];
        const uint32_t fill = g.vtx[w.seg_vertex[s]].y;
        if (is_big(g, fill, blocks_for(fill, g.logB), len)) w.big_list[atomicAdd(&w.queue[2], 1ull)] = s;
    }
}

template <int TPV>
__global__ void __launch_bounds__(BIG_THREADS, WIN_CTAS) k_window_apply(DevGraph g, WinSegs w) {
    constexpr int GPC = BIG_THREADS / TPV;
    constexpr int GPW = 32 / TPV;
    __shared__ uint32_t tab[BIG_TAB];
    __shared__ uint32_t tabs[GPC][BIG_BLOCKS];
    __shared__ uint32_t wt[33];
    __shared__ uint32_t unit_s;
    __shared__ unsigned long long base_s;
    __shared__ DirtyBuf dirty;
    if (g.ctl->batch_abort) return;
    if (threadIdx.x == 0) dirty.cnt = 0;  // the queue's first barrier makes it seen
    long long delta = 0;                  // live entries gained, one atomic per warp
    const unsigned long long top = g.ctl->free_top;
    const uint32_t nbig = (uint32_t)w.queue[2];
    // ---- big segments: one CTA each
    for (;;) {
        if (threadIdx.x == 0) unit_s = (uint32_t)min(atomicAdd(&w.queue[0], 1ull), 0xFFFFFFFFull);
        __syncthreads();
        const uint32_t bi = unit_s;
        __syncthreads();
        if (bi >= nbig) break;
        const uint32_t s = w.big_list[bi];
        const uint32_t u = w.seg_vertex[s];
        const uint32_t st = w.seg_start[s], len = w.seg_start[s + 1] - st;
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, nb_old = blocks_for(fill, g.logB);
        const uint32_t *D = w.bdst + st;
        const uint32_t *T = w.btype + st;
        uint32_t ndel = 0;
        for (uint32_t k0 = 0; k0 < nb_old; k0 += BIG_TAB) {
            const uint32_t kc = min((uint32_t)BIG_TAB, nb_old - k0);
            fill_block_table(g, rec.x, k0, kc, tab, threadIdx.x, BIG_THREADS);
            __syncthreads();
            const uint32_t e0 = k0 << g.logB;
            const uint32_t e1 = min(fill, (k0 + kc) << g.logB);
            const uint32_t nq = (e1 - e0 + 3) >> 2;
            for (uint32_t q = threadIdx.x; q < nq; q += BIG_THREADS) {
                const uint32_t e = e0 + (q << 2);
                ndel += win_quad(g.pool + ((size_t)tab[(e >> g.logB) - k0] << g.logB) + (e & (g.B - 1)), e, e1, D, T,
                                 len, w.found + st);
            }
            __syncthreads();
        }
        ndel = cta_sum<uint32_t, BIG_THREADS>(ndel, wt);
        uint32_t c = 0;
        for (uint32_t i = threadIdx.x; i < len; i += BIG_THREADS) c += (T[i] && !w.found[st + i]) ? 1u : 0u;
        const uint32_t newcnt = cta_sum<uint32_t, BIG_THREADS>(c, wt);
        uint32_t nnew = win_new_blocks(fill, nb_old, newcnt, g.logB);
        if (threadIdx.x == 0) base_s = nnew ? atomicAdd(&g.ctl->alloc_cursor, (unsigned long long)nnew) : 0ull;
        __syncthreads();
        const unsigned long long b64 = base_s;
        uint32_t ins = newcnt;
        if (b64 + nnew > top) {  // unreachable after the host's admission check; never write past the stack
            if (threadIdx.x == 0) atomicOr(&g.ctl->status, GV_DEV_ERR_NOMEM);
            ins = 0;
            nnew = 0;
        }
        const uint32_t base = (uint32_t)b64;
        if (ins) {
            cta_append(g, rec, nb_old, top, base, D, nullptr, len, wt,
                       [&](uint32_t i) { return T[i] && !w.found[st + i]; });
            link_new_blocks(g, u, rec, nb_old, nnew, fill + ins, top, base, threadIdx.x, BIG_THREADS,
                            [] { __syncthreads(); });
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            win_record(g, u, rec, nb_old, ins, nnew, ndel, top, base, dirty);
            delta += (long long)ins - (long long)ndel;
        }
        __syncthreads();
    }
    // ---- small segments: chunks per warp, a lane group per segment
    Group<TPV> G;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gw = lane / TPV;
    uint32_t *mytab = tabs[threadIdx.x / TPV];
    const uint32_t nseg = (uint32_t)g.ctl->nseg;
    for (;;) {
        unsigned long long c0 = 0;
        if (lane == 0) c0 = atomicAdd(&w.queue[1], (unsigned long long)WIN_CHUNK);
        c0 = __shfl_sync(GV_FULL_MASK, c0, 0);
        if (c0 >= nseg) break;
        const uint32_t cend = (uint32_t)min((unsigned long long)nseg, c0 + WIN_CHUNK);
        for (uint32_t r = (uint32_t)c0; r < cend; r += GPW) {  // warp-uniform rounds
            const uint32_t s = r + gw;
            bool active = s < cend;
            uint32_t u = 0, st = 0, len = 0, fill = 0, nb_old = 0;
            uint4 rec = make_uint4(0, 0, 0, 0);
            if (active) {
                u = w.seg_vertex[s];
                st = w.seg_start[s];
                len = w.seg_start[s + 1] - st;
                rec = g.vtx[u];
                fill = rec.y;
                nb_old = blocks_for(fill, g.logB);
                active = !is_big(g, fill, nb_old, len);
            }
            const uint32_t *D = w.bdst + st;
            const uint32_t *T = w.btype + st;
            uint32_t ndel = 0;
            if (active) {
                fill_block_table(g, rec.x, 0, nb_old, mytab, G.gl, TPV);
                G.sync();
                const uint32_t nq = (fill + 3) >> 2;
                for (uint32_t q = G.gl; q < nq; q += TPV) {
                    const uint32_t e = q << 2;
                    ndel += win_quad(g.pool + ((size_t)mytab[e >> g.logB] << g.logB) + (e & (g.B - 1)), e, fill, D, T,
                                     len, w.found + st);
                }
            }
            ndel = G.sum(ndel);
            G.sync();
            uint32_t c = 0;
            if (active)
                for (uint32_t i = G.gl; i < len; i += TPV) c += (T[i] && !w.found[st + i]) ? 1u : 0u;
            const uint32_t newcnt = G.sum(c);
            uint32_t nnew = active ? win_new_blocks(fill, nb_old, newcnt, g.logB) : 0u;
            const unsigned long long off = warp_agg_alloc(&g.ctl->alloc_cursor, (G.gl == 0) ? nnew : 0u);
            const unsigned long long b64 = G.bcast(off, 0);
            uint32_t ins = active ? newcnt : 0u;
            if (b64 + nnew > top) {  // see the admission note above
                if (active && G.gl == 0) atomicOr(&g.ctl->status, GV_DEV_ERR_NOMEM);
                ins = 0;
                nnew = 0;
            }
            const uint32_t base = (uint32_t)b64;
            if (ins) {
                uint32_t j0 = 0;
                for (uint32_t cc = 0; cc < len; cc += TPV) {
                    const uint32_t i = cc + G.gl;
                    const uint32_t isnew = (i < len && T[i] && !w.found[st + i]) ? 1u : 0u;
                    uint32_t tot;
                    const uint32_t pre = G.excl_scan(isnew, tot);
                    if (isnew) {
                        const uint32_t p = fill + j0 + pre;
                        const uint32_t k = p >> g.logB;
                        const uint32_t b = (k < nb_old) ? rec.w : new_block(g, top, base, k - nb_old);
                        g.pool[((size_t)b << g.logB) + (p & (g.B - 1))] = D[i];
                    }
                    j0 += tot;
                }
                link_new_blocks(g, u, rec, nb_old, nnew, fill + ins, top, base, G.gl, TPV, [&] { G.sync(); });
            }
            G.sync();
            if (active && G.gl == 0) {
                win_record(g, u, rec, nb_old, ins, nnew, ndel, top, base, dirty);
                delta += (long long)ins - (long long)ndel;
            }
            G.sync();
        }
    }
    delta = warp_sum(delta);
    if (lane == 0 && delta) atomicAdd(&g.ctl->live_edges, (unsigned long long)delta);
    dirty_flush(g, dirty);
}

// -------------------------------------------------------------- compaction
// Stable in-place compaction of one vertex: live entries keep their order,
// tail blocks that end up empty go back to the free stack and are unlinked
// from their parents.  Replaces compactionVertexCentric
// (src/dynamicStructure/kernels/delete_kernels.cu:50-261), which fills holes
// from the tail and can drop live entries when a hole and the tail entry
// meet in the same block.
template <int TPV>
__global__ void __launch_bounds__(UPD_THREADS) k_compact(DevGraph g, uint32_t *__restrict__ big_list) {
    constexpr int GPC = UPD_THREADS / TPV;
    __shared__ uint32_t tabs[GPC][BIG_BLOCKS];
    const uint32_t nd = (uint32_t)g.ctl->ndirty;
    Group<TPV> G;
    uint32_t *tab = tabs[threadIdx.x / TPV];
    const uint32_t ngroups = gridDim.x * GPC;
    for (uint32_t di = blockIdx.x * GPC + threadIdx.x / TPV; di < nd; di += ngroups) {
        const uint32_t u = g.dirty_list[di];
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, live = rec.z, nb = blocks_for(fill, g.logB);
        if (is_big_vertex(g, fill, nb)) {
            if (G.gl == 0) big_list[atomicAdd(&g.ctl->nbig, 1ull)] = u;
            continue;
        }
        fill_block_table(g, rec.x, 0, nb, tab, G.gl, TPV);
        G.sync();
        uint32_t wpos = 0;
        const uint32_t nq = (fill + 3) >> 2;
        for (uint32_t q0 = 0; q0 < nq; q0 += TPV) {
            const uint32_t q = q0 + G.gl;
            uint32_t ev[4] = {GV_TOMB, GV_TOMB, GV_TOMB, GV_TOMB};
            float wv[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t c = 0;
            if (q < nq) {
                const uint32_t e = q << 2;
                const size_t at = ((size_t)tab[e >> g.logB] << g.logB) + (e & (g.B - 1));
                const uint4 v = *reinterpret_cast<const uint4 *>(g.pool + at);
                ev[0] = v.x; ev[1] = v.y; ev[2] = v.z; ev[3] = v.w;
                if (g.weighted) {
                    const float4 w = *reinterpret_cast<const float4 *>(g.wpool + at);
                    wv[0] = w.x; wv[1] = w.y; wv[2] = w.z; wv[3] = w.w;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (e + j >= fill) ev[j] = GV_TOMB;
                    c += (ev[j] != GV_TOMB);
                }
            }
            uint32_t tot;
            uint32_t p = wpos + G.excl_scan(c, tot);
            G.sync();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (ev[j] != GV_TOMB) {
                    if (p != (q << 2) + j) {  // entries before the first tombstone stay where they are
                        const size_t at = ((size_t)tab[p >> g.logB] << g.logB) + (p & (g.B - 1));
                        g.pool[at] = ev[j];
                        if (g.weighted) g.wpool[at] = wv[j];
                    }
                    ++p;
                }
            }
            wpos += tot;
        }
        G.sync();
        const uint32_t nb_new = blocks_for(live, g.logB);
        const uint32_t nfree = nb - nb_new;
        unsigned long long fbase = 0;
        if (G.gl == 0 && nfree) fbase = atomicAdd(&g.ctl->free_top, (unsigned long long)nfree);
        fbase = G.bcast(fbase, 0);
        for (uint32_t t = G.gl; t < nfree; t += TPV) {
            const uint32_t k = nb_new + t;
            g.free_stack[fbase + t] = tab[k];
            const uint32_t pk = (k - 1) >> 1;
            if (k > 0 && pk < nb_new) {
                if (k & 1u) g.left[tab[pk]] = GV_NIL; else g.right[tab[pk]] = GV_NIL;
            }
        }
        if (G.gl == 0) {
            if (nb_new) g.bcount[tab[nb_new - 1]] = live - ((nb_new - 1) << g.logB);
            g.vtx[u] = make_uint4(nb_new ? rec.x : GV_NIL, live, live, nb_new ? tab[nb_new - 1] : GV_NIL);
            g.dirty[u] = 0;
        }
        G.sync();
    }
}

__global__ void __launch_bounds__(BIG_THREADS) k_compact_big(DevGraph g, const uint32_t *__restrict__ big_list) {
    __shared__ uint32_t tab[BIG_TAB];
    __shared__ uint32_t wt[33];
    __shared__ unsigned long long fbase_s;
    constexpr uint32_t QPT = 4;
    const uint32_t nbig = (uint32_t)g.ctl->nbig;
    for (uint32_t bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
        const uint32_t u = big_list[bi];
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, live = rec.z, nb = blocks_for(fill, g.logB);
        uint32_t wpos = 0;
        for (uint32_t k0 = 0; k0 < nb; k0 += BIG_TAB) {
            const uint32_t kc = min((uint32_t)BIG_TAB, nb - k0);
            fill_block_table(g, rec.x, k0, kc, tab, threadIdx.x, BIG_THREADS);
            __syncthreads();
            const uint32_t e0 = k0 << g.logB;
            const uint32_t e1 = min(fill, (k0 + kc) << g.logB);
            const uint32_t nq = (e1 - e0 + 3) >> 2;
            // QPT consecutive quads per thread: a round reads 8192 entries, so
            // that a hub's barriers are few
            for (uint32_t q0 = 0; q0 < nq; q0 += BIG_THREADS * QPT) {
                uint32_t ev[QPT][4];
                float wv[QPT][4];
                uint32_t c = 0;
#pragma unroll
                for (uint32_t t = 0; t < QPT; ++t) {
                    const uint32_t q = q0 + threadIdx.x * QPT + t, e = e0 + (q << 2);
                    uint4 v = make_uint4(GV_TOMB, GV_TOMB, GV_TOMB, GV_TOMB);
                    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (q < nq) {
                        const size_t at = ((size_t)tab[(e >> g.logB) - k0] << g.logB) + (e & (g.B - 1));
                        v = *reinterpret_cast<const uint4 *>(g.pool + at);
                        if (g.weighted) w = *reinterpret_cast<const float4 *>(g.wpool + at);
                    }
                    ev[t][0] = v.x; ev[t][1] = v.y; ev[t][2] = v.z; ev[t][3] = v.w;
                    wv[t][0] = w.x; wv[t][1] = w.y; wv[t][2] = w.z; wv[t][3] = w.w;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (q < nq && e + j >= fill) ev[t][j] = GV_TOMB;
                        c += (ev[t][j] != GV_TOMB);
                    }
                }
                uint32_t tot;
                uint32_t p = wpos + cta_excl_scan<uint32_t, BIG_THREADS>(c, wt, tot);
#pragma unroll
                for (uint32_t t = 0; t < QPT; ++t)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (ev[t][j] == GV_TOMB) continue;
                        if (p != e0 + ((q0 + threadIdx.x * QPT + t) << 2) + j) {
                            const uint32_t kd = p >> g.logB;
                            const uint32_t b = (kd >= k0) ? tab[kd - k0] : cbt_block(g.left, g.right, rec.x, kd);
                            const size_t at = ((size_t)b << g.logB) + (p & (g.B - 1));
                            g.pool[at] = ev[t][j];
                            if (g.weighted) g.wpool[at] = wv[t][j];
                        }
                        ++p;
                    }
                wpos += tot;
                __syncthreads();
            }
        }
        // Free the tail blocks.  Walks only touch surviving ancestors, whose
        // links to other survivors are not modified here.
        const uint32_t nb_new = blocks_for(live, g.logB);
        const uint32_t nfree = nb - nb_new;
        if (threadIdx.x == 0) fbase_s = nfree ? atomicAdd(&g.ctl->free_top, (unsigned long long)nfree) : 0ull;
        __syncthreads();
        const unsigned long long fbase = fbase_s;
        for (uint32_t t = threadIdx.x; t < nfree; t += BIG_THREADS) {
            const uint32_t k = nb_new + t;
            g.free_stack[fbase + t] = cbt_block(g.left, g.right, rec.x, k);
        }
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < nfree; t += BIG_THREADS) {
            const uint32_t k = nb_new + t;
            const uint32_t pk = (k - 1) >> 1;
            if (k > 0 && pk < nb_new) {
                const uint32_t pb = cbt_block(g.left, g.right, rec.x, pk);
                if (k & 1u) g.left[pb] = GV_NIL; else g.right[pb] = GV_NIL;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t lb = nb_new ? cbt_block(g.left, g.right, rec.x, nb_new - 1) : GV_NIL;
            if (nb_new) g.bcount[lb] = live - ((nb_new - 1) << g.logB);
            g.vtx[u] = make_uint4(nb_new ? rec.x : GV_NIL, live, live, lb);
            g.dirty[u] = 0;
        }
        __syncthreads();
    }
}

__global__ void k_compact_done(Ctl *ctl) {
    ctl->ndirty = 0;
    ctl->nbig = 0;
}

// --------------------------------------------------------- vertex delete
// Every entry of a flagged vertex, and every entry pointing at one, becomes
// a tombstone; live counts, the control block and the dirty list change as a
// batch delete changes them, so gv_compact reclaims the blocks.
template <int TPV>
__global__ void __launch_bounds__(UPD_THREADS) k_vertex_delete(DevGraph g, const uint8_t *__restrict__ del) {
    Group<TPV> G;
    constexpr int GPC = UPD_THREADS / TPV;
    const uint32_t ngroups = gridDim.x * GPC;
    for (uint32_t u = blockIdx.x * GPC + threadIdx.x / TPV; u < g.n; u += ngroups) {
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, nb = blocks_for(fill, g.logB);
        if (rec.z == 0) continue;
        const bool all = del[u] != 0;
        uint32_t cnt = 0;
        for (uint32_t k = 0; k < nb; ++k) {
            const uint32_t b = (k == 0) ? rec.x : cbt_block(g.left, g.right, rec.x, k);
            const uint32_t slots = min(g.B, fill - (k << g.logB));
            uint32_t *blk = g.pool + ((size_t)b << g.logB);
            for (uint32_t i = G.gl; i < slots; i += TPV) {
                const uint32_t v = blk[i];
                if (v != GV_TOMB && (all || del[v])) {
                    blk[i] = GV_TOMB;
                    g.affected[v] = 1;
                    ++cnt;
                }
            }
        }
        cnt = G.sum(cnt);
        if (G.gl == 0 && cnt) {
            g.vtx[u].z = rec.z - cnt;
            g.affected[u] = 1;
            atomicAdd(&g.ctl->live_edges, (unsigned long long)(-(long long)cnt));
            if (!g.dirty[u]) {
                g.dirty[u] = 1;
                g.dirty_list[atomicAdd(&g.ctl->ndirty, 1ull)] = u;
            }
        }
    }
}

// ------------------------------------------------------------------ export
// The live adjacency as CSR, each vertex's entries in storage order.  Bound
// by memory: 4 bytes read and 4 written per entry, plus the weights.
//
//   k_export: vertices and entries laid end to end (a vertex takes EXP_ROW
//   units for its record and one per entry) are cut into equal shares, one
//   per warp, so that neither a hub of thousands of blocks nor a long run of
//   isolated vertices is one warp's job.  The warp finds its first vertex
//   with a 32-way search of offset + EXP_ROW * id, then takes 32 vertices at
//   a time: their blocks 32 at a time, a lane each (so the walks to the
//   blocks run side by side), and the blocks' entries as one run, 32 a step,
//   in which a lane finds its block by bisecting the warp's prefix sums and
//   the writes are contiguous.  In a vertex with tombstones each entry's place
//   depends on those before it: the warp whose share holds the vertex's record
//   packs the whole vertex (export_rows; not where nothing of it is live), or
//   lists it for k_export_holes above EXP_HEAVY blocks, for a share may hold 32
//   vertices of few live entries and as many slots each.
//   k_export_holes: a CTA per listed vertex.
//
// 133 M entries (R-MAT scale 22, 1.1 GB moved): 11.9 ms with a lane group per
// vertex, 0.6 ms with a warp per 512 units (the search and the walks of so
// small a piece are latency), 0.35 ms so (2.9 TB/s; a quarter of the warps or 16
// times as many are slower); 31 M: 0.10 ms; 0.4 M: 167 -> 6 us.  The ten shuffles
// per 32 entries, not memory, bound it now.
// With tombstones: a clique of 1,500 whose first vertices are deleted 710 us a call
// with the vertices' slots read 32 at a time, 61 so; R-MAT scale 22, a tenth deleted,
// 1.72 ms and 1.31.
constexpr uint32_t EXP_SHARE = 256;
constexpr uint32_t EXP_ROW = 8;
constexpr uint32_t EXP_HEAVY = 8;

__device__ __forceinline__ uint32_t export_block(const DevGraph &g, uint32_t root, uint32_t k) {
    return k == 0 ? root : cbt_block(g.left, g.right, root, k);
}

__device__ __forceinline__ uint32_t export_scan(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(GV_FULL_MASK, v, d);
        if (lane >= (uint32_t)d) v += t;
    }
    return v;
}

// The lane whose inclusive sum first exceeds p (31 if none does).
__device__ __forceinline__ uint32_t export_find(uint32_t incl, uint32_t p) {
    uint32_t j = 0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        if (__shfl_sync(GV_FULL_MASK, incl, j + d - 1) <= p) j += d;
    return j;
}

// A warp's vertices with tombstones (v, in the lanes where mine): listed, or cut into
// rows of 32 slots, which lie in one block each, B being a multiple of 32.  A lane walks
// to the block of one row, then the rows are packed in order, four in flight.  Not
// inlined: its registers would cost k_export the warps that hide its loads.
template <bool W>
__device__ __noinline__ void export_rows(const DevGraph &g, bool mine, uint32_t v, uint32_t my_root, uint32_t my_fill,
                                         uint32_t room, unsigned long long o, uint32_t *__restrict__ out,
                                         float *__restrict__ wout, uint32_t *__restrict__ list) {
    const uint32_t lane = threadIdx.x & 31u;
    if (mine && blocks_for(my_fill, g.logB) > EXP_HEAVY) {
        const uint32_t at = atomicAdd(&list[0], 1u);
        if (at + 1 < g.n) {  // one the list has no room for stays here
            list[at + 1] = v;
            mine = false;
        }
    }
    const uint32_t rows = mine ? (my_fill + 31) >> 5 : 0u;
    const uint32_t rincl = export_scan(rows, lane);
    const uint32_t nrow = __shfl_sync(GV_FULL_MASK, rincl, 31);
    uint32_t done = 0;  // entries of the row's vertex before it
    for (uint32_t q0 = 0; q0 < nrow; q0 += 32) {
        const uint32_t q = q0 + lane;
        const uint32_t j = export_find(rincl, q);
        const uint32_t i0 = (q - __shfl_sync(GV_FULL_MASK, rincl - rows, j)) * 32;
        const uint32_t root = __shfl_sync(GV_FULL_MASK, my_root, j), fill = __shfl_sync(GV_FULL_MASK, my_fill, j);
        const uint32_t lim = __shfl_sync(GV_FULL_MASK, room, j);
        const unsigned long long oj = __shfl_sync(GV_FULL_MASK, o, j);
        const bool has = q < nrow;
        const uint32_t b = has ? export_block(g, root, i0 >> g.logB) : 0u;
        const unsigned long long src = ((unsigned long long)b << g.logB) + (i0 & (g.B - 1));
        const uint32_t cnt = has ? min(32u, fill - i0) : 0u;
        const uint32_t first = __ballot_sync(GV_FULL_MASK, i0 == 0);
        for (uint32_t t0 = 0; t0 < min(32u, nrow - q0); t0 += 4) {
            uint32_t e[4];
            float w[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const unsigned long long at = __shfl_sync(GV_FULL_MASK, src, t0 + t) + lane;
                e[t] = GV_TOMB;
                if (lane < __shfl_sync(GV_FULL_MASK, cnt, t0 + t)) {
                    e[t] = g.pool[at];
                    if (W) w[t] = g.wpool[at];
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if ((first >> (t0 + t)) & 1u) done = 0;
                const uint32_t live = __ballot_sync(GV_FULL_MASK, e[t] != GV_TOMB);
                const uint32_t pos = done + __popc(live & ((1u << lane) - 1u));
                const unsigned long long to = __shfl_sync(GV_FULL_MASK, oj, t0 + t) + pos;
                if (pos < __shfl_sync(GV_FULL_MASK, lim, t0 + t) && e[t] != GV_TOMB) {
                    out[to] = e[t];
                    if (W) wout[to] = w[t];
                }
                done += __popc(live);
            }
        }
    }
}

template <bool W>
__global__ void __launch_bounds__(UPD_THREADS) k_export(const __grid_constant__ DevGraph g, const unsigned long long *__restrict__ off,
                                                        uint32_t *__restrict__ out, float *__restrict__ wout,
                                                        uint32_t *__restrict__ list) {
    constexpr int U = W ? 4 : 8;  // entries in flight per lane
    const uint32_t lane = threadIdx.x & 31u, n = g.n;
    const uint64_t units = off[n] + (uint64_t)n * EXP_ROW;
    const uint64_t nw = (uint64_t)gridDim.x * (UPD_THREADS / 32);
    const uint64_t share = max((uint64_t)EXP_SHARE, (units + nw - 1) / nw);
    const uint64_t u0 = ((uint64_t)blockIdx.x * (UPD_THREADS / 32) + (threadIdx.x >> 5)) * share;
    const uint64_t u1 = min(units, u0 + share);
    if (u0 >= units) return;
    // the last vertex whose record, at unit off[v] + EXP_ROW * v, starts at or before u0
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t probe = (uint64_t)lo + (uint64_t)(lane + 1) * step;
        const bool below = probe < hi && off[probe] + probe * EXP_ROW <= u0;
        const uint32_t c = __popc(__ballot_sync(GV_FULL_MASK, below));
        const uint32_t nlo = lo + c * step;
        hi = (uint32_t)min((uint64_t)hi, (uint64_t)nlo + step);
        lo = nlo;
    }
    // record and offset of a window's vertices, loaded one window ahead
    auto load = [&](uint64_t v, uint4 &r, unsigned long long &o) {
        r = v < n ? g.vtx[v] : make_uint4(GV_NIL, 0u, 0u, GV_NIL);
        o = off[min(v, (uint64_t)n)];
    };
    uint4 rec_n;
    unsigned long long o_n;
    load((uint64_t)lo + lane, rec_n, o_n);
    for (uint64_t v0 = lo; v0 < n; v0 += 32) {
        const uint4 rec = rec_n;
        const unsigned long long o = o_n;
        const uint32_t v = (uint32_t)v0 + lane;
        const bool ok = v0 + lane < n;
        const uint64_t unit = ok ? o + (uint64_t)v * EXP_ROW : ~0ull;
        if (__shfl_sync(GV_FULL_MASK, unit, 0) >= u1) break;  // this vertex belongs to a later warp
        load(v0 + 32 + lane, rec_n, o_n);
        unsigned long long oe = __shfl_down_sync(GV_FULL_MASK, o, 1);
        const unsigned long long o32 = __shfl_sync(GV_FULL_MASK, o_n, 0);
        if (lane == 31) oe = o32;
        const uint32_t room = (uint32_t)(oe - o);  // bounds every write of this vertex
        const bool holes = rec.z != rec.y;
        const uint32_t len = holes ? 0u : min(rec.y, room);
        // entries [first, last) of the vertex lie in the share: entry i is unit + EXP_ROW + i
        uint32_t first = 0, last = 0;
        if (ok && unit < u1) {
            if (u0 > unit + EXP_ROW) first = (uint32_t)min((uint64_t)len, u0 - unit - EXP_ROW);
            if (u1 > unit + EXP_ROW) last = (uint32_t)min((uint64_t)len, u1 - unit - EXP_ROW);
        }
        // the blocks that hold them, 32 at a time: a lane walks to one block
        const uint32_t k0 = first >> g.logB;
        const uint32_t nk = last > first ? ((last - 1) >> g.logB) - k0 + 1u : 0u;
        const uint32_t kincl = export_scan(nk, lane);
        const uint32_t nblk = __shfl_sync(GV_FULL_MASK, kincl, 31);
        for (uint32_t q0 = 0; q0 < nblk; q0 += 32) {
            const uint32_t q = q0 + lane;
            const uint32_t j = export_find(kincl, q);
            const uint32_t k = q - __shfl_sync(GV_FULL_MASK, kincl - nk, j) + __shfl_sync(GV_FULL_MASK, k0, j);
            const uint32_t root = __shfl_sync(GV_FULL_MASK, rec.x, j);
            const uint32_t lo_e = max(__shfl_sync(GV_FULL_MASK, first, j), k << g.logB);
            const uint32_t hi_e = min(__shfl_sync(GV_FULL_MASK, last, j), (k + 1) << g.logB);
            const unsigned long long oj = __shfl_sync(GV_FULL_MASK, o, j);
            const bool has = q < nblk;
            const uint32_t cnt = has ? hi_e - lo_e : 0u;
            const uint32_t incl = export_scan(cnt, lane);
            const uint32_t total = __shfl_sync(GV_FULL_MASK, incl, 31);
            // place p of the run is entry src + p of the pool and goes to dst + p
            const uint32_t b = has ? export_block(g, root, k) : 0u;
            const unsigned long long src = ((unsigned long long)b << g.logB) + (lo_e & (g.B - 1)) - (incl - cnt);
            const unsigned long long dst = oj + lo_e - (incl - cnt);
            for (uint32_t p0 = 0; p0 < total; p0 += 32 * U) {
                unsigned long long to[U];
                uint32_t e[U];
                float w[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t p = p0 + 32 * u + lane;
                    const uint32_t f = export_find(incl, p);
                    const unsigned long long at = __shfl_sync(GV_FULL_MASK, src, f) + p;
                    to[u] = __shfl_sync(GV_FULL_MASK, dst, f) + p;
                    if (p < total) {
                        e[u] = g.pool[at];
                        if (W) w[u] = g.wpool[at];
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (p0 + 32 * u + lane < total) {
                        out[to[u]] = e[u];
                        if (W) wout[to[u]] = w[u];
                    }
            }
        }
        // vertices with tombstones whose own unit lies here, and that keep an entry
        const bool mine = ok && holes && room && unit >= u0 && unit < u1;
        if (__any_sync(GV_FULL_MASK, mine)) export_rows<W>(g, mine, v, rec.x, rec.y, room, o, out, wout, list);
    }
}

template <bool W>
__global__ void __launch_bounds__(UPD_THREADS) k_export_holes(DevGraph g, const unsigned long long *__restrict__ off,
                                                              uint32_t *__restrict__ out, float *__restrict__ wout,
                                                              const uint32_t *__restrict__ list) {
    __shared__ uint32_t tab[BIG_TAB];
    __shared__ uint32_t wt[33];
    const uint32_t nl = min(list[0], g.n - 1);
    for (uint32_t it = blockIdx.x; it < nl; it += gridDim.x) {
        const uint32_t v = list[it + 1];
        const uint4 rec = g.vtx[v];
        const uint32_t nb = blocks_for(rec.y, g.logB);
        const unsigned long long o = off[v];
        const uint32_t room = (uint32_t)(off[v + 1] - o);
        uint32_t done = 0;
        for (uint32_t k0 = 0; k0 < nb; k0 += BIG_TAB) {
            const uint32_t kc = min((uint32_t)BIG_TAB, nb - k0);
            __syncthreads();
            fill_block_table(g, rec.x, k0, kc, tab, threadIdx.x, UPD_THREADS);
            __syncthreads();
            const uint32_t cnt = min(rec.y - (k0 << g.logB), kc << g.logB);
            for (uint32_t i0 = 0; i0 < cnt; i0 += UPD_THREADS) {
                const uint32_t i = i0 + threadIdx.x;
                size_t at = 0;
                uint32_t e = GV_TOMB;
                if (i < cnt) {
                    at = ((size_t)tab[i >> g.logB] << g.logB) + (i & (g.B - 1));
                    e = g.pool[at];
                }
                uint32_t tot;
                const uint32_t pos = done + cta_excl_scan<uint32_t, UPD_THREADS>(e != GV_TOMB ? 1u : 0u, wt, tot);
                if (e != GV_TOMB && pos < room) {
                    out[o + pos] = e;
                    if (W) wout[o + pos] = g.wpool[at];
                }
                done += tot;
            }
        }
        __syncthreads();
    }
}

__global__ void k_live_degrees(DevGraph g, uint32_t *__restrict__ deg) {
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < g.n; u += gridDim.x * blockDim.x)
        deg[u] = g.vtx[u].z;
}

// ------------------------------------------------------------------- check
// Codes: 1 root/fill mismatch, 2 live > fill, 3 bad block index, 4 owner,
// 5 block count, 6 predecessor, 7 left child, 8 right child, 9 last block,
// 10 live count, 11 block used twice or lost, 12 bad free entry, 13 totals.
__device__ void report(unsigned long long *viol, uint32_t *first, uint32_t code, uint32_t u) {
    if (atomicAdd(viol, 1ull) == 0) {
        first[0] = code;
        first[1] = u;
    }
}

__global__ void k_check_vertices(DevGraph g, uint32_t *__restrict__ mark, unsigned long long *viol,
                                 uint32_t *first, unsigned long long *used_blocks) {
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < g.n; u += gridDim.x * blockDim.x) {
        const uint4 rec = g.vtx[u];
        const uint32_t fill = rec.y, live = rec.z, nb = blocks_for(fill, g.logB);
        if ((fill == 0) != (rec.x == GV_NIL)) { report(viol, first, 1, u); continue; }
        if (live > fill) report(viol, first, 2, u);
        if (nb == 0) continue;
        atomicAdd(used_blocks, (unsigned long long)nb);
        uint32_t prev = GV_NIL, cnt = 0;
        bool ok = true;
        for (uint32_t k = 0; k < nb && ok; ++k) {
            // walk with bounds checks
            uint32_t p = k + 1, b = rec.x;
            int d = 31 - __clz(p);
            for (int i = d - 1; i >= 0; --i) {
                if (b >= g.P) break;
                b = ((p >> i) & 1u) ? g.right[b] : g.left[b];
            }
            if (b >= g.P) { report(viol, first, 3, u); ok = false; break; }
            atomicAdd(&mark[b], 1u);
            if (g.owner[b] != u) report(viol, first, 4, u);
            const uint32_t want = (k + 1 < nb) ? g.B : fill - ((nb - 1) << g.logB);
            if (g.bcount[b] != want) report(viol, first, 5, u);
            if (k > 0 && g.pred[b] != prev) report(viol, first, 6, u);
            const bool hl = 2 * k + 1 < nb, hr = 2 * k + 2 < nb;
            if (hl != (g.left[b] != GV_NIL)) report(viol, first, 7, u);
            if (hr != (g.right[b] != GV_NIL)) report(viol, first, 8, u);
            const uint32_t slots = min(g.B, fill - (k << g.logB));
            for (uint32_t i = 0; i < slots; ++i) cnt += (g.pool[((size_t)b << g.logB) + i] != GV_TOMB);
            prev = b;
        }
        if (ok && prev != rec.w) report(viol, first, 9, u);
        if (ok && cnt != live) report(viol, first, 10, u);
    }
}

__global__ void k_check_free(DevGraph g, uint32_t *__restrict__ mark, unsigned long long *viol, uint32_t *first) {
    unsigned long long top = g.ctl->free_top;
    if (top > g.P) {
        if (blockIdx.x == 0 && threadIdx.x == 0) report(viol, first, 13, 0);
        top = g.P;
    }
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < top;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t b = g.free_stack[i];
        if (b >= g.P) { report(viol, first, 12, 0); continue; }
        atomicAdd(&mark[b], 1u);
    }
}

__global__ void k_check_marks(DevGraph g, const uint32_t *__restrict__ mark, unsigned long long *viol,
                              uint32_t *first, const unsigned long long *used_blocks) {
    for (unsigned long long b = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b < g.P;
         b += (unsigned long long)gridDim.x * blockDim.x)
        if (mark[b] != 1u) report(viol, first, 11, (uint32_t)b);
    if (blockIdx.x == 0 && threadIdx.x == 0 && *used_blocks + g.ctl->free_top != g.P)
        report(viol, first, 13, 0);
}

}  // namespace

// ====================================================================== host
static gv_status apply_segments(gv_graph *g, uint64_t E, bool vals, bool is_delete, bool finish, cudaStream_t s);

gv_status run_update(gv_graph *g, const uint32_t *dsrc, const uint32_t *ddst, const float *dw,
                     uint64_t k, bool symmetric, bool is_delete, cudaStream_t s) {
    BatchScratch &bs = g->bs;
    const uint64_t E = symmetric ? 2 * k : k;
    const bool vals = (dw != nullptr) && !is_delete;
    int which = 0;
    if (E <= SB_KEYS) {  // one CTA's batch
        ProfScope ps(PROF_RADIX, s);
        auto launch = [&](auto weighted) {
            constexpr bool W = decltype(weighted)::value;
            cudaFuncSetAttribute(k_small_batch<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SbSmem<W>));
            GV_LAUNCH(k_small_batch<W>, 1, SB_THREADS, sizeof(SbSmem<W>), s, dsrc, ddst, dw, (uint32_t)k,
                      symmetric ? 1 : 0, g->d.n, g->bitsn, bs.bdst, bs.bw, bs.found, bs.seg_vertex, bs.seg_start,
                      g->d.affected, g->d.ctl);
        };
        if (vals) launch(std::true_type{});
        else launch(std::false_type{});
        return apply_segments(g, E, vals, is_delete, true, s);
    }
    {
        ProfScope ps(PROF_RADIX, s);
        GV_LAUNCH(k_expand, grid_for(k, 256), 256, 0, s, dsrc, ddst, k, symmetric ? 1 : 0, g->d.n,
                  g->bitsn, bs.keys, vals ? bs.vals : nullptr, g->d.ctl);
        which = radix_sort_u64(bs.keys, bs.keys_alt, vals ? bs.vals : nullptr, vals ? bs.vals_alt : nullptr,
                               E, 2 * (int)g->bitsn, bs.rs_counts, bs.scan_tmp, s);
    }
    const unsigned long long *K = which ? bs.keys_alt : bs.keys;
    const uint32_t *V = which ? bs.vals_alt : bs.vals;
    return apply_sorted(g, K, vals ? V : nullptr, E, symmetric, dw, is_delete, true, s);
}

void launch_commit_keep_abort(gv_graph *g, cudaStream_t s) {
    GV_LAUNCH(k_commit_keep_abort, 1, 1, 0, s, g->d.ctl);
}

void launch_finish(gv_graph *g, cudaStream_t s) { GV_LAUNCH(k_finish, 1, 1, 0, s, g->d.ctl); }

gv_status launch_window_apply(gv_graph *g, const uint32_t *seg_vertex, const uint32_t *seg_start,
                              const uint32_t *bdst, const uint32_t *btype, uint8_t *found, uint32_t *big_list,
                              unsigned long long *queue, cudaStream_t s) {
    DevGraph d = g->d;
    WinSegs w{seg_vertex, seg_start, bdst, btype, found, big_list, queue};
    {
        ProfScope ps(PROF_MEMBER, s);
        GV_LAUNCH(k_window_classify, 148 * 4, 256, 0, s, d, w);
    }
    {
        ProfScope ps(PROF_APPLY, s);
        dispatch_tpv(g->cfg.threads_per_vertex, [&](auto t) {
            constexpr int T = decltype(t)::value;
            GV_LAUNCH((k_window_apply<T>), 148 * WIN_CTAS, BIG_THREADS, 0, s, d, w);
        });
    }
    GV_LAUNCH(k_finish, 1, 1, 0, s, d.ctl);
    return cuda_status(cudaGetLastError(), "window apply launch");
}

gv_status apply_sorted(gv_graph *g, const unsigned long long *K, const uint32_t *V, uint64_t E, bool symmetric,
                       const float *dw, bool is_delete, bool finish, cudaStream_t s) {
    BatchScratch &bs = g->bs;
    const bool vals = (V != nullptr) && (dw != nullptr) && !is_delete;
    const unsigned long long sent = (g->bitsn >= 32) ? ~0ull : ((1ull << (2 * g->bitsn)) - 1ull);
    const unsigned ntiles = (unsigned)((E + SEG_TILE - 1) / SEG_TILE);
    {
        ProfScope ps(PROF_SEGMENT, s);
        GV_LAUNCH(k_seg_count, ntiles, SEG_THREADS, 0, s, K, E, sent, g->bitsn, bs.tile_cnt);
        scan_exclusive_u64(bs.tile_cnt, bs.tile_cnt, ntiles, &g->d.ctl->scratch0, bs.scan_tmp, s);
        GV_LAUNCH(k_seg_write, ntiles, SEG_THREADS, 0, s, K, V, E, sent, g->bitsn, symmetric ? 1 : 0,
                  (const unsigned long long *)bs.tile_cnt, dw, bs.bdst, vals ? bs.bw : nullptr, bs.found,
                  bs.seg_vertex, bs.seg_start, g->d.affected, g->d.ctl);
    }
    return apply_segments(g, E, vals, is_delete, finish, s);
}

// Membership and apply of the segments in the batch scratch (at most E).
static gv_status apply_segments(gv_graph *g, uint64_t E, bool vals, bool is_delete, bool finish, cudaStream_t s) {
    BatchScratch &bs = g->bs;
    // Segments <= unique entries <= E.
    const unsigned gsmall = grid_for(E, 64);
    const unsigned gbig = 148 * 4;
    const uint32_t tpv = g->cfg.threads_per_vertex;
    // a small batch leaves most of the chip idle: whole warps per vertex, so
    // that the longest list is scanned sooner (1,000 pairs on 16 K vertices,
    // lists of up to 1,024: 24 us with 8 lanes, 16 with 32)
    const uint32_t mtpv = E <= SB_KEYS ? 32 : tpv;
    DevGraph d = g->d;
    {
        ProfScope ps(PROF_MEMBER, s);
        dispatch_tpv(mtpv, [&](auto t) {
            constexpr int T = decltype(t)::value;
            if (is_delete)
                GV_LAUNCH((k_member<T, true>), gsmall, UPD_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start,
                          bs.bdst, bs.found, bs.seg_found, bs.big_list);
            else
                GV_LAUNCH((k_member<T, false>), gsmall, UPD_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start,
                          bs.bdst, bs.found, bs.seg_found, bs.big_list);
        });
        if (is_delete)
            GV_LAUNCH(k_member_big<true>, gbig, BIG_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start, bs.bdst,
                      bs.found, bs.seg_found, bs.big_list);
        else
            GV_LAUNCH(k_member_big<false>, gbig, BIG_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start, bs.bdst,
                      bs.found, bs.seg_found, bs.big_list);
    }
    if (!is_delete) {
        ProfScope ps(PROF_APPLY, s);
        GV_LAUNCH(k_plan, grid_for(E, UPD_THREADS), UPD_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start,
                  bs.seg_found, bs.seg_newblocks, bs.seg_blkbase);
        GV_LAUNCH(k_admit, 1, 1, 0, s, d.ctl);
        dispatch_tpv(tpv, [&](auto t) {
            constexpr int T = decltype(t)::value;
            GV_LAUNCH((k_apply<T>), gsmall, UPD_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start, bs.bdst,
                      vals ? bs.bw : nullptr, bs.found, bs.seg_found, bs.seg_newblocks, bs.seg_blkbase);
        });
        GV_LAUNCH(k_apply_big, gbig, BIG_THREADS, 0, s, d, bs.seg_vertex, bs.seg_start, bs.bdst,
                  vals ? bs.bw : nullptr, bs.found, bs.seg_found, bs.seg_newblocks, bs.seg_blkbase,
                  bs.big_list);
    }
    if (finish) GV_LAUNCH(k_finish, 1, 1, 0, s, d.ctl);
    else GV_LAUNCH(k_commit_keep_abort, 1, 1, 0, s, d.ctl);
    return cuda_status(cudaGetLastError(), "update launch");
}

gv_status run_compact(gv_graph *g, cudaStream_t s) {
    DevGraph d = g->d;
    ProfScope ps(PROF_COMPACT, s);
    // The dirty list holds at most n vertices; size the grid for it.  Few vertices:
    // whole warps each (as for small batches; R-MAT of 64 K: 27 us, 36 with eight
    // lanes), and CTAs for all of them, for they may all be dirty (uniform, 16 K
    // vertices: 28 us with CTAs for an eighth, 20 so).
    const bool few = g->d.n <= (1u << 16);
    dispatch_tpv(few ? 32 : g->cfg.threads_per_vertex, [&](auto t) {
        constexpr int T = decltype(t)::value;
        const unsigned grid = few ? grid_for(g->d.n, UPD_THREADS / T, 148 * 32) : grid_for(g->d.n, 64);
        GV_LAUNCH((k_compact<T>), grid, UPD_THREADS, 0, s, d, d.vbig_list);
    });
    GV_LAUNCH(k_compact_big, 148 * 4, BIG_THREADS, 0, s, d, (const uint32_t *)d.vbig_list);
    GV_LAUNCH(k_compact_done, 1, 1, 0, s, d.ctl);
    return cuda_status(cudaGetLastError(), "compact launch");
}

gv_status run_export(gv_graph *g, unsigned long long *offsets, uint32_t *dst, float *w, uint64_t entries, uint32_t *list,
                     cudaStream_t s) {
    DevGraph d = g->d;
    cudaMemsetAsync(list, 0, 4, s);
    const unsigned grid = grid_for(entries + (uint64_t)d.n * EXP_ROW, (UPD_THREADS / 32) * EXP_SHARE, 148 * 16);
    auto launch = [&](auto weighted) {
        constexpr bool W = decltype(weighted)::value;
        GV_LAUNCH(k_export<W>, grid, UPD_THREADS, 0, s, d, offsets, dst, w, list);
        GV_LAUNCH(k_export_holes<W>, 148 * 4, UPD_THREADS, 0, s, d, offsets, dst, w, (const uint32_t *)list);
    };
    if (w) launch(std::true_type{});
    else launch(std::false_type{});
    return cuda_status(cudaGetLastError(), "export launch");
}

gv_status run_vertex_delete(gv_graph *g, const uint8_t *del, cudaStream_t s) {
    DevGraph d = g->d;
    dispatch_tpv(g->cfg.threads_per_vertex, [&](auto t) {
        constexpr int T = decltype(t)::value;
        GV_LAUNCH((k_vertex_delete<T>), grid_for(g->d.n, UPD_THREADS / T), UPD_THREADS, 0, s, d, del);
    });
    return cuda_status(cudaGetLastError(), "vertex delete launch");
}

void launch_degrees(gv_graph *g, uint32_t *deg, cudaStream_t s) {
    GV_LAUNCH(k_live_degrees, grid_for(g->d.n, 256), 256, 0, s, g->d, deg);
}

gv_status run_check(gv_graph *g, uint64_t *violations, uint32_t *code, uint32_t *vertex) {
    DevGraph d = g->d;
    uint32_t *mark = nullptr;
    unsigned long long *cnt = nullptr;
    cudaError_t e = cudaMalloc(&mark, d.P * sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_status(e, "check alloc");
    e = cudaMalloc(&cnt, 4 * sizeof(unsigned long long));
    if (e != cudaSuccess) {
        cudaFree(mark);
        return cuda_status(e, "check alloc");
    }
    cudaMemset(mark, 0, d.P * sizeof(uint32_t));
    cudaMemset(cnt, 0, 4 * sizeof(unsigned long long));
    unsigned long long *viol = cnt, *used = cnt + 1;
    uint32_t *first = reinterpret_cast<uint32_t *>(cnt + 2);
    GV_LAUNCH(k_check_vertices, grid_for(d.n, 256), 256, 0, 0, d, mark, viol, first, used);
    GV_LAUNCH(k_check_free, grid_for(d.P, 256), 256, 0, 0, d, mark, viol, first);
    GV_LAUNCH(k_check_marks, grid_for(d.P, 256), 256, 0, 0, d, (const uint32_t *)mark, viol, first,
              (const unsigned long long *)used);
    unsigned long long h[4] = {0, 0, 0, 0};
    e = cudaMemcpy(h, cnt, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(mark);
    cudaFree(cnt);
    if (e != cudaSuccess) return cuda_status(e, "check");
    *violations = h[0];
    const uint32_t *f = reinterpret_cast<const uint32_t *>(&h[2]);
    if (code) *code = f[0];
    if (vertex) *vertex = f[1];
    return GV_OK;
}

}  // namespace gv
