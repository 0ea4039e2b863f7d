// PageRank over a sweep plan: the undirected store compiled, once per call,
// into a degree-ordered padded CSR that the sweeps read instead of walking
// the edge-block trees.
//
// Why: a pull sweep is bound by its gathers of the neighbours'
// contributions, not by the adjacency stream.  On R-MAT graphs those gathers
// concentrate on a few vertices (at scale 22 the 16 K highest-degree
// vertices receive 40% of them, the top 256 K 85%), but vertex ids scatter
// the hot values over the whole contribution vector, so every 32-byte sector
// the L1 keeps holds one hot value and seven cold ones.  The plan renumbers
// the vertices by descending degree class (stable in id order inside a
// class), so the hot contributions are contiguous: the top 16 K fit in 64 KB
// and stay in L1, the top 256 K in 1 MB of L2.  A row is the vertex's used
// slots in block order, tombstones and the padding to whole 16-byte quads
// written as a sentinel neighbour whose contribution is 0, so every load is
// an aligned uint4 and no tombstone or fill test remains; slot e of block k
// lands at k*B + e, so the blocks of a hub are copied in parallel.
//
// The plan: perm (new row -> vertex), inv (vertex -> new row), off[n+1]
// (uint32 row starts), col (neighbour rows, padded), the degree-class tier
// boundaries and the hub items.  Sweeps keep x and the contributions in plan
// order; the result is permuted back at the end.  Tiers by degree (rows are
// contiguous per tier): hubs of at least HUB_DEG entries are cut into items
// of ITEM_ENTRIES for one warp each (partials combined in item order), rows
// of WARP_DEG or more take a warp, rows of GROUP_DEG or more 8 lanes, the
// rest one thread; isolated rows take their value once and are not swept.
// One launch runs the four tiers, CTAs interleaved in proportion to their
// work; a second one combines the hub items, and its CTA that finishes last
// sums the residuals, all in fixed orders (deterministic).
//
// plan_csr_solve runs the same sweeps over a plan of a CSR with weights: the
// in-edge transpose (weighted PageRank, PageRank on directed stores) and the
// out-edges (the adjoint).
//
// Same iteration as the store sweep (x0 = 1/n or the caller's start, L1 step
// < epsilon or max_iter, contributions x/deg, no dangling redistribution:
// src/algorithm/pagerank/pagerank.cu:3-68, pr_kernel.cu:3-48).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include "store.cuh"
#include "group.cuh"
#include "prims.cuh"
#include "launch.hpp"
#include "prof.hpp"

namespace gv {
namespace {

constexpr int PL_THREADS = 256;
constexpr uint32_t NCLASS = 34;        // degree classes: 0 (isolated), 1 + floor(log2 deg)
constexpr uint32_t PL_TILE = 512;      // vertices per counting-sort tile (a warp places them in turn)
constexpr uint32_t HUB_DEG = 2048;     // rows with at least this many entries are cut into items
constexpr uint32_t ITEM_ENTRIES = 2048;
constexpr uint32_t WARP_DEG = 64;
constexpr uint32_t GROUP_DEG = 8;
constexpr unsigned PL_PERIOD = 16;
constexpr unsigned PL_WAVES_MAX = 148 * 128 / PL_PERIOD;
constexpr unsigned PL_GRID = PL_PERIOD * PL_WAVES_MAX;  // residual slots (the most CTAs a sweep launches)
constexpr unsigned PL_FIN = 148;      // CTAs that end a batched sweep
constexpr unsigned PL_FIN_MAX = 592;  // CTAs that end a single sweep

// Row lengths of what is planned: a vertex's live entries in the store, or a
// CSR row.
struct DegOfStore {
    const uint4 *vtx;
    __device__ __forceinline__ uint32_t operator()(uint32_t v) const { return vtx[v].z; }
};
struct DegOfCsr {
    const unsigned long long *off;
    __device__ __forceinline__ uint32_t operator()(uint32_t v) const { return (uint32_t)(off[v + 1] - off[v]); }
};

__device__ __forceinline__ uint32_t deg_class(uint32_t d) { return d ? 32u - __clz(d) : 0u; }

// ---------------------------------------------------------------- plan build
// Counting sort of the vertices by descending class, stable in id order:
// tile counts (class-major), a scan, then one warp per tile places its
// vertices in order.
template <typename Deg>
__global__ void k_pl_count(Deg deg, uint32_t n, uint32_t ntiles, uint32_t *__restrict__ cnt) {
    __shared__ uint32_t h[NCLASS];
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        for (uint32_t i = threadIdx.x; i < NCLASS; i += blockDim.x) h[i] = 0;
        __syncthreads();
        const uint32_t v0 = t * PL_TILE, v1 = min(n, v0 + PL_TILE);
        for (uint32_t v = v0 + threadIdx.x; v < v1; v += blockDim.x)
            atomicAdd(&h[NCLASS - 1 - deg_class(deg(v))], 1u);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < NCLASS; i += blockDim.x) cnt[(size_t)i * ntiles + t] = h[i];
        __syncthreads();
    }
}

template <typename Deg>
__global__ void k_pl_place(Deg deg, uint32_t n, uint32_t ntiles, const uint32_t *__restrict__ start,
                           uint32_t *__restrict__ perm, uint32_t *__restrict__ inv) {
    __shared__ uint32_t base[PL_THREADS / 32][NCLASS];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t t = blockIdx.x * (PL_THREADS / 32) + warp;
    if (t >= ntiles) return;
    for (uint32_t i = lane; i < NCLASS; i += 32) base[warp][i] = start[(size_t)i * ntiles + t];
    __syncwarp();
    const uint32_t v0 = t * PL_TILE, v1 = min(n, v0 + PL_TILE);
    for (uint32_t r = v0; r < v1; r += 32) {
        const uint32_t v = r + lane;
        const bool ok = v < v1;
        const uint32_t c = ok ? NCLASS - 1 - deg_class(deg(v)) : NCLASS;  // NCLASS: no vertex
        const uint32_t peers = __match_any_sync(GV_FULL_MASK, c);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        const uint32_t leader = __ffs(peers) - 1;
        uint32_t pos = 0;
        if (ok) pos = base[warp][c] + rank;
        __syncwarp();
        if (ok && lane == leader) base[warp][c] += __popc(peers);
        __syncwarp();
        if (ok) {
            perm[pos] = v;
            inv[v] = pos;
        }
    }
}

// What the host reads of a plan, gathered so that it is one copy: the class
// starts (first row of each class) from the scanned counts, the padded entries
// and the copy items; then the hub items and the row starts of the tiers.
struct PlanFacts {
    uint32_t cls[NCLASS], total, nfill;
};
__global__ void k_pl_facts(const uint32_t *__restrict__ start, uint32_t ntiles, const uint32_t *__restrict__ total,
                           const uint32_t *__restrict__ nfill, PlanFacts *__restrict__ out) {
    const uint32_t i = threadIdx.x;
    if (i < NCLASS) out->cls[i] = start[(size_t)i * ntiles];
    if (i == NCLASS) out->total = *total;
    if (i == NCLASS + 1) out->nfill = nfill ? *nfill : 0u;
}

struct PlanTiers {
    uint32_t hoff[4], nitems;
};
__global__ void k_pl_tier_facts(const uint32_t *__restrict__ off, uint4 rows, const uint32_t *__restrict__ nitems,
                                PlanTiers *__restrict__ out) {
    const uint32_t r[4] = {rows.x, rows.y, rows.z, rows.w};
    if (threadIdx.x < 4) out->hoff[threadIdx.x] = off[r[threadIdx.x]];
    if (threadIdx.x == 4) out->nitems = rows.x ? *nitems : 0u;
}

// Padded row lengths in plan order: a row holds the vertex's used slots
// (tombstones included, as the sentinel) rounded up to whole quads, so slot e
// of block k lands at k*B + e of the row and blocks are copied independently.
// Also the inverse live degrees and, per row of two or more blocks, its
// number of 32-block copy items.
__global__ void k_pl_rowlen(DevGraph g, const uint32_t *__restrict__ perm, uint32_t *__restrict__ plen,
                            float *__restrict__ rdeg, uint32_t *__restrict__ fitems) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
        const uint4 rec = g.vtx[perm[i]];
        plen[i] = (rec.y + 3u) & ~3u;
        rdeg[i] = rec.z ? 1.0f / (float)rec.z : 0.f;
        const uint32_t nb = blocks_for(rec.y, g.logB);
        fitems[i] = nb > 1 ? (nb + 31u) >> 5 : 0u;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) rdeg[g.n] = 0.f;
}

__device__ __forceinline__ uint32_t pl_map(uint32_t e, uint32_t slot, uint32_t fill, const uint32_t *__restrict__ inv,
                                           uint32_t n) {
    return (slot < fill && e != GV_TOMB) ? inv[e] : n;
}

// Rows of at most one block: 8 lanes per row copy its quads, neighbours
// renumbered, tombstones and the padding as the sentinel n.
__global__ void k_pl_fill_small(DevGraph g, const uint32_t *__restrict__ perm, const uint32_t *__restrict__ inv,
                                const uint32_t *__restrict__ off, uint32_t *__restrict__ col) {
    Group<8> G;
    const uint32_t ng = gridDim.x * (blockDim.x / 8);
    for (uint32_t i = blockIdx.x * (blockDim.x / 8) + threadIdx.x / 8; i < g.n; i += ng) {
        const uint4 rec = g.vtx[perm[i]];
        if (rec.y > g.B) continue;  // the copy items take it
        const uint32_t o = off[i], nq = (off[i + 1] - o) >> 2;
        const uint4 *src = reinterpret_cast<const uint4 *>(g.pool + ((size_t)rec.x << g.logB));
        uint4 *dst = reinterpret_cast<uint4 *>(col + o);
        for (uint32_t q = G.gl; q < nq; q += 8) {
            const uint4 v = src[q];
            const uint32_t e = q << 2;
            dst[q] = make_uint4(pl_map(v.x, e, rec.y, inv, g.n), pl_map(v.y, e + 1, rec.y, inv, g.n),
                                pl_map(v.z, e + 2, rec.y, inv, g.n), pl_map(v.w, e + 3, rec.y, inv, g.n));
        }
    }
}

// Rows of two or more blocks: a warp per item of 32 blocks, the lanes walk
// the tree to one block each, then copy the blocks quad by quad.
__global__ void k_pl_fill_items(DevGraph g, const uint32_t *__restrict__ perm, const uint32_t *__restrict__ inv,
                                const uint32_t *__restrict__ off, const uint32_t *__restrict__ frow,
                                const uint32_t *__restrict__ ffirst, uint32_t nitems, uint32_t *__restrict__ col) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    const uint32_t qpb = g.B >> 2;  // quads per block
    for (uint32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < nitems; it += nw) {
        const uint32_t r = frow[it];
        const uint4 rec = g.vtx[perm[r]];
        const uint32_t nb = blocks_for(rec.y, g.logB);
        const uint32_t kb0 = (it - ffirst[r]) << 5;
        const uint32_t k = kb0 + lane;
        const uint32_t myb = k < nb ? (k == 0 ? rec.x : cbt_block(g.left, g.right, rec.x, k)) : GV_NIL;
        const uint32_t o = off[r];
        const uint32_t nk = min(32u, nb - kb0);
        for (uint32_t j = 0; j < nk; ++j) {
            const uint32_t b = __shfl_sync(GV_FULL_MASK, myb, j);
            const uint32_t kk = kb0 + j;
            const uint32_t e0 = kk << g.logB;
            const uint32_t quads = (min(g.B, rec.y - e0) + 3u) >> 2;
            const uint4 *src = reinterpret_cast<const uint4 *>(g.pool + ((size_t)b << g.logB));
            uint4 *dst = reinterpret_cast<uint4 *>(col + o + e0);
            for (uint32_t q = lane; q < quads; q += 32) {
                const uint4 v = src[q];
                const uint32_t e = e0 + (q << 2);
                dst[q] = make_uint4(pl_map(v.x, e, rec.y, inv, g.n), pl_map(v.y, e + 1, rec.y, inv, g.n),
                                    pl_map(v.z, e + 2, rec.y, inv, g.n), pl_map(v.w, e + 3, rec.y, inv, g.n));
            }
        }
        (void)qpb;
    }
}

// CSR rows: padded lengths, then the columns, renumbered, with their weights.
// A warp takes 128 quads of the output in turn; their rows are bisected
// between those of the first and the last one (most often the same).
__global__ void k_pl_rowlen_csr(DegOfCsr deg, uint32_t n, const uint32_t *__restrict__ perm,
                                uint32_t *__restrict__ plen) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        plen[i] = (deg(perm[i]) + 3u) & ~3u;
}

// last row of off[0, n] whose start is at most e (e below the total)
__device__ __forceinline__ uint32_t pl_row_of(const uint32_t *__restrict__ off, uint32_t lo, uint32_t hi, uint32_t e) {
    while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (off[mid] <= e) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <bool W>
__global__ void k_pl_fill_csr(DegOfCsr deg, uint32_t n, const uint32_t *__restrict__ dst, const float *__restrict__ w,
                              const uint32_t *__restrict__ perm, const uint32_t *__restrict__ inv,
                              const uint32_t *__restrict__ off, uint32_t quads, uint32_t *__restrict__ col,
                              float *__restrict__ pw) {
    constexpr uint32_t RUN = 128;
    const uint32_t lane = threadIdx.x & 31u, nw = gridDim.x * (blockDim.x >> 5);
    for (uint32_t q0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * RUN; q0 < quads; q0 += nw * RUN) {
        const uint32_t q1 = min(quads, q0 + RUN);
        uint32_t r = 0;
        if (lane < 2) r = pl_row_of(off, 0, n, (lane ? q1 - 1 : q0) << 2);
        const uint32_t ra = __shfl_sync(GV_FULL_MASK, r, 0), rb = __shfl_sync(GV_FULL_MASK, r, 1);
        for (uint32_t q = q0 + lane; q < q1; q += 32) {
            const uint32_t row = pl_row_of(off, ra, rb + 1, q << 2);
            const uint32_t k = (q << 2) - off[row], v = perm[row];
            const uint32_t len = deg(v);
            const unsigned long long at = deg.off[v] + k;
            uint32_t c[4];
            float x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool in = k + j < len;
                c[j] = in ? dst[at + j] : 0u;
                x[j] = in && W ? w[at + j] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) c[j] = k + j < len ? inv[c[j]] : n;
            reinterpret_cast<uint4 *>(col)[q] = make_uint4(c[0], c[1], c[2], c[3]);
            if (W) reinterpret_cast<float4 *>(pw)[q] = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
}

// a vector of vertex order in plan order
__global__ void k_pl_gather(uint32_t n, const uint32_t *__restrict__ perm, const float *__restrict__ x,
                            float *__restrict__ y) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = x[perm[i]];
}

// hub items: per hub row its item count, then item -> row
__global__ void k_pl_item_count(const uint32_t *__restrict__ off, uint32_t nhub, uint32_t *__restrict__ icnt) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nhub; i += gridDim.x * blockDim.x)
        icnt[i] = (off[i + 1] - off[i] + ITEM_ENTRIES - 1) / ITEM_ENTRIES;
}

__global__ void k_pl_item_fill(const uint32_t *__restrict__ ifirst, uint32_t nhub, uint32_t *__restrict__ irow) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nhub; i += gridDim.x * blockDim.x)
        for (uint32_t k = ifirst[i]; k < ifirst[i + 1]; ++k) irow[k] = i;
}

// x0 in plan order (from the caller's start, or 1/n, or the source), its
// contributions; x_out in vertex order at the end
// Isolated rows [rz, n) take their final value (the base, plus the source
// term) in both iterate buffers here and are left out of the sweeps.
__global__ void k_pl_init(uint32_t n, const uint32_t *__restrict__ perm, const float *__restrict__ xin,
                          float fill, uint32_t src_row, float src_val, const float *__restrict__ rdeg,
                          uint32_t rz, float base, float src_base, float *__restrict__ x, float *__restrict__ c,
                          float *__restrict__ x_other, float *__restrict__ c_other) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        if (i == n) {
            x[n] = 0.f;
            c[n] = 0.f;
            x_other[n] = 0.f;
            c_other[n] = 0.f;
            continue;
        }
        if (i >= rz) {
            const float v = base + (i == src_row ? src_base : 0.f);
            x[i] = v;
            x_other[i] = v;
            c[i] = 0.f;
            c_other[i] = 0.f;
            continue;
        }
        const float v = xin ? xin[perm[i]] : (i == src_row ? src_val : fill);
        x[i] = v;
        c[i] = rdeg ? v * rdeg[i] : v;
    }
}

__global__ void k_pl_out(uint32_t n, const uint32_t *__restrict__ inv, const float *__restrict__ x,
                         float *__restrict__ out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) out[v] = x[inv[v]];
}

// ------------------------------------------------------------------- sweeps
struct PlanSweep {
    const uint32_t *off, *col, *irow, *ifirst;
    const float *w;       // weights beside col (weighted sweeps)
    const float *rdeg;    // contribution of a row: its value times rdeg (null: the value itself)
    const float *cvec;    // additive term of a row (null: base and the source's term)
    const float *rscale;  // multiplier of a row's sum (null: 1)
    const float *gather;  // contributions, plan order, [n] = 0
    const float *xold;
    float *xnew, *cnew;   // cnew null: the next sweep gathers xnew
    float *ipart;         // per hub item
    double *partial;      // residual per CTA of the sweep, then of the finish launch
    int *state;           // [0] converged, [1] sweeps done, [2] CTAs of the finish launch done
    float alpha, base, eps;
    uint32_t src_row;     // personalised source (plan order) or GV_NIL
    float src_val;
    uint32_t rH, rW, rG, rZ, n, nitems;  // tier row boundaries; rows past rZ are not swept
    uint32_t split;       // CTAs per period: items | warp << 8 | group << 16 | thread << 24
};

// The gathers of one quad; weights are 0 in the padding.
// LOOP: the values were written by this same launch, so not the read-only path.
template <bool W, bool LOOP>
__device__ __forceinline__ float pl_quad(const float *c, uint4 q, float4 w) {
    auto at = [&](uint32_t i) { return LOOP ? __ldca(c + i) : __ldg(c + i); };
    if (W) return (w.x * at(q.x) + w.y * at(q.y)) + (w.z * at(q.z) + w.w * at(q.w));
    return (at(q.x) + at(q.y)) + (at(q.z) + at(q.w));
}

// QF quads of a row of nq, j, j + stride, ...: all loads first, then their
// gathers (4 QF in flight).
template <int QF, bool W>
struct PlQuads {
    uint4 v[QF];
    float4 w[W ? QF : 1];
    __device__ __forceinline__ void load(const PlanSweep &a, uint32_t o, uint32_t j, uint32_t nq, uint32_t stride) {
        const uint4 *q = reinterpret_cast<const uint4 *>(a.col + o);
        const float4 *qw = reinterpret_cast<const float4 *>(a.w + o);
#pragma unroll
        for (int t = 0; t < QF; ++t) {
            const bool in = j + t * stride < nq;
            v[t] = in ? __ldcs(q + j + t * stride) : make_uint4(a.n, a.n, a.n, a.n);
            if (W) w[t] = in ? __ldcs(qw + j + t * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    template <bool LOOP>
    __device__ __forceinline__ float sum(const PlanSweep &a) const {
        float part = 0.f;
#pragma unroll
        for (int t = 0; t < QF; ++t) part += pl_quad<W, LOOP>(a.gather, v[t], w[W ? t : 0]);
        return part;
    }
};

// Row i's new value from its sum; returns its step.
__device__ __forceinline__ double pl_finish(const PlanSweep &a, uint32_t i, float sum) {
    const float b = a.cvec ? a.cvec[i] : a.base + (i == a.src_row ? a.src_val : 0.f);
    const float xv = b + a.alpha * (a.rscale ? a.rscale[i] * sum : sum);
    a.xnew[i] = xv;
    if (a.cnew) a.cnew[i] = a.rdeg ? xv * a.rdeg[i] : xv;
    return (double)fabsf(xv - a.xold[i]);
}

// Hub items: a warp per item of ITEM_ENTRIES entries, four quads per lane in
// flight; k_pl_fin combines a row's items.
template <bool W>
__device__ __forceinline__ void pl_items(const PlanSweep &a, uint32_t vb, uint32_t vg) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = vg * (PL_THREADS / 32);
    for (uint32_t it = vb * (PL_THREADS / 32) + (threadIdx.x >> 5); it < a.nitems; it += nw) {
        const uint32_t r = a.irow[it];
        const uint32_t e0 = a.off[r] + (it - a.ifirst[r]) * ITEM_ENTRIES;
        const uint32_t nq = (min(a.off[r + 1], e0 + ITEM_ENTRIES) - e0) >> 2;
        float sum = 0.f;
        for (uint32_t j = lane; j < nq; j += 128) {
            PlQuads<4, W> q;
            q.load(a, e0, j, nq, 32);
            sum += q.template sum<false>(a);
        }
        sum = warp_sum(sum);
        if (lane == 0) a.ipart[it] = sum;
    }
}

// Hub rows inside the one-launch loop: a CTA per row, so that a sweep needs no
// second round for the items.
template <bool W>
__device__ __forceinline__ void pl_hub_rows(const PlanSweep &a, uint32_t vb, uint32_t vg, double &res) {
    __shared__ float part[PL_THREADS / 32];
    for (uint32_t r = vb; r < a.rH; r += vg) {
        const uint32_t o = a.off[r], nq = (a.off[r + 1] - o) >> 2;
        float sum = 0.f;
        for (uint32_t j = threadIdx.x; j < nq; j += 4 * PL_THREADS) {
            PlQuads<4, W> q;
            q.load(a, o, j, nq, PL_THREADS);
            sum += q.template sum<true>(a);
        }
        sum = warp_sum(sum);
        if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.f;
            for (int i = 0; i < PL_THREADS / 32; ++i) t += part[i];
            res += pl_finish(a, r, t);
        }
        __syncthreads();
    }
}

// rows of TPV lanes each over [r0, r1): quads strided by TPV, QF of them
// (4 QF gathers) in flight per lane.  Rows of a group or a thread (TPV < 32)
// are short, so a row's dependent loads (bounds, quads, gathers, finish)
// would each wait in turn: the next row's bounds and first quads are loaded
// while this row's gathers are in flight.  Sums are formed in the same order
// either way.
template <int TPV, int QF, bool W, bool LOOP>
__device__ __forceinline__ void pl_rows(const PlanSweep &a, uint32_t r0, uint32_t r1, uint32_t vb, uint32_t vg,
                                        double &res) {
    Group<TPV> G;
    constexpr uint32_t GPC = PL_THREADS / TPV;
    const uint32_t ng = vg * GPC;
    uint32_t i = r0 + vb * GPC + threadIdx.x / TPV;
    if constexpr (TPV == 32) {
        for (; i < r1; i += ng) {
            const uint32_t o = a.off[i];
            const uint32_t nq = (a.off[i + 1] - o) >> 2;
            float sum = 0.f;
            for (uint32_t j = G.gl; j < nq; j += QF * TPV) {
                PlQuads<QF, W> q;
                q.load(a, o, j, nq, TPV);
                sum += q.template sum<LOOP>(a);
            }
            sum = G.sum(sum);
            if (G.gl == 0) res += pl_finish(a, i, sum);
        }
    } else {
        uint32_t o = 0, nq = 0;
        if (i < r1) {
            o = a.off[i];
            nq = (a.off[i + 1] - o) >> 2;
        }
        PlQuads<QF, W> q;
        q.load(a, o, G.gl, nq, TPV);
        while (i < r1) {
            const uint32_t in = i + ng;
            uint32_t on = 0, nqn = 0;
            if (in < r1) {
                on = a.off[in];
                nqn = (a.off[in + 1] - on) >> 2;
            }
            float sum = 0.f;
            sum += q.template sum<LOOP>(a);
            for (uint32_t j = G.gl + QF * TPV; j < nq; j += QF * TPV) {
                PlQuads<QF, W> t;
                t.load(a, o, j, nq, TPV);
                sum += t.template sum<LOOP>(a);
            }
            q.load(a, on, G.gl, nqn, TPV);
            if (TPV > 1) sum = G.sum(sum);
            if (G.gl == 0) res += pl_finish(a, i, sum);
            i = in;
            o = on;
            nq = nqn;
        }
    }
}

// The tiers of one sweep, as CTA vb of vg (a multiple of PL_PERIOD); returns
// the thread's residual.
template <bool W, bool LOOP>
__device__ __forceinline__ double pl_tiers(const PlanSweep &a, uint32_t vb, uint32_t vg) {
    const uint32_t t0 = a.split & 0xFFu, t1 = (a.split >> 8) & 0xFFu, t2 = (a.split >> 16) & 0xFFu,
                   t3 = (a.split >> 24) & 0xFFu;
    const uint32_t r = vb % PL_PERIOD, w = vb / PL_PERIOD, waves = vg / PL_PERIOD;
    double res = 0.0;
    if (r < t0) {
        if (LOOP) pl_hub_rows<W>(a, w * t0 + r, waves * t0, res);
        else pl_items<W>(a, w * t0 + r, waves * t0);
    }
    else if (r < t0 + t1) pl_rows<32, 4, W, LOOP>(a, a.rH, a.rW, w * t1 + (r - t0), waves * t1, res);
    else if (r < t0 + t1 + t2) pl_rows<8, 2, W, LOOP>(a, a.rW, a.rG, w * t2 + (r - t0 - t1), waves * t2, res);
    else pl_rows<1, 2, W, LOOP>(a, a.rG, a.rZ, w * t3 + (r - t0 - t1 - t2), waves * t3, res);
    return res;
}

// Hub rows of one sweep: a warp each, the row's item partials in a fixed order.
__device__ __forceinline__ double pl_hubs(const PlanSweep &a, uint32_t vb, uint32_t vg) {
    const uint32_t lane = threadIdx.x & 31u;
    double res = 0.0;
    for (uint32_t i = vb * (PL_THREADS / 32) + (threadIdx.x >> 5); i < a.rH; i += vg * (PL_THREADS / 32)) {
        const uint32_t k0 = a.ifirst[i], k1 = a.ifirst[i + 1];
        float t = 0.f;
        for (uint32_t k = k0 + lane; k < k1; k += 32) t += a.ipart[k];
        t = warp_sum(t);
        if (lane == 0) res += pl_finish(a, i, t);
    }
    return res;
}

// Sum over the CTA in a fixed order; every thread gets it.
__device__ __forceinline__ double pl_cta_total(double v, double *red) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int i = 0; i < PL_THREADS / 32; ++i) s += red[i];
    return s;
}

template <bool W>
__global__ void __launch_bounds__(PL_THREADS, W ? 6 : 8) k_pl_sweep(PlanSweep a) {
    __shared__ double red[PL_THREADS / 32];
    if (a.state[0]) return;
    const double s = pl_cta_total(pl_tiers<W, false>(a, blockIdx.x, gridDim.x), red);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = s;
}

// Thread 0: whether this CTA is the last of the launch to come here; what the
// others wrote before is visible to it.
__device__ __forceinline__ bool pl_last(int *arrived) {
    __threadfence();
    const bool last = atomicAdd(arrived, 1) == (int)gridDim.x - 1;
    __threadfence();
    return last;
}

// Ends a sweep: hub rows (a warp each, the row's item partials in a fixed
// order), a share of the sweep's residual slots per CTA, and in the CTA that
// finishes last the whole residual (slots in a fixed order) and the
// convergence flag.  One CTA summing 9,472 slots took 12 us of every sweep on
// top of a hub launch of 6; the two together take 8 (4 with one CTA, without
// hubs).  Inside the sweep itself the same steps cost it a quarter (0.36 -> 0.46
// ms at R-MAT scale 22): the fence of every finishing CTA empties its SM's L1,
// where the hot contributions live.
__global__ void __launch_bounds__(PL_THREADS) k_pl_fin(PlanSweep a, uint32_t nslots) {
    __shared__ double red[PL_THREADS / 32];
    __shared__ bool last;
    if (a.state[0]) return;
    double res = pl_hubs(a, blockIdx.x, gridDim.x);
    for (uint32_t i = blockIdx.x * PL_THREADS + threadIdx.x; i < nslots; i += gridDim.x * PL_THREADS)
        res += a.partial[i];
    double s = pl_cta_total(res, red);
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) {
            a.partial[nslots + blockIdx.x] = s;
            last = pl_last(&a.state[2]);
        }
        __syncthreads();
        if (!last) return;
        res = 0.0;
        for (uint32_t i = threadIdx.x; i < gridDim.x; i += PL_THREADS) res += __ldcg(a.partial + nslots + i);
        s = pl_cta_total(res, red);
    }
    if (threadIdx.x == 0) {
        a.state[1] += 1;
        a.state[2] = 0;
        if (s < (double)a.eps) a.state[0] = 1;
    }
}

// Waits until every CTA of a cooperative launch has come here `round` times
// (from 1), as seen in at most `tries` looks.  Past them state[3] is set, which
// ends every other wait too, and the sweeps are done again launch by launch.
// The count of arrivals may wrap around: no CTA is two rounds ahead of another.
constexpr uint32_t PL_WAIT_LIMIT = 1u << 24;
__device__ __forceinline__ bool pl_grid_wait(int *state, uint32_t round, uint32_t tries) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&state[2], 1);
        const uint32_t want = round * gridDim.x;
        const volatile int *seen = state;
        ok = tries != 0;
        for (uint32_t i = 1; ok && (int)(want - (uint32_t)seen[2]) > 0; ++i)
            if (seen[3] || i >= tries) ok = 0;
        if (!ok) atomicExch(&state[3], 1);
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// All the sweeps of a small graph in one cooperative launch: with launches per
// sweep and a read-back every eight, 14 sweeps over 16 K vertices took 371 us of
// a call, 279 so.
// Every CTA sums the residual slots itself, in the same order, so all see the
// same end.  gather, xold, xnew and cnew are those of the first sweep and
// swap after each; rows [rG, rz_first) are swept by the first two.
template <bool W>
__global__ void __launch_bounds__(PL_THREADS, 4) k_pl_loop(PlanSweep a, uint32_t rz_first, uint32_t rz, int max_iter,
                                                           uint32_t tries) {
    __shared__ double red[PL_THREADS / 32];
    const bool contrib = a.cnew != nullptr;
    float *xa = const_cast<float *>(a.xold), *xb = a.xnew, *ca = const_cast<float *>(a.gather), *cb = a.cnew;
    int done = 0;
    for (int it = 0; it < max_iter; ++it) {
        a.gather = contrib ? ca : xa;
        a.xold = xa;
        a.xnew = xb;
        a.cnew = contrib ? cb : nullptr;
        a.rZ = it < 2 ? rz_first : rz;
        // two sets of slots, so that a CTA ahead does not overwrite what one behind still sums
        double *slots = a.partial + (it & 1) * gridDim.x;
        double s = pl_cta_total(pl_tiers<W, true>(a, blockIdx.x, gridDim.x), red);
        if (threadIdx.x == 0) slots[blockIdx.x] = s;
        if (!pl_grid_wait(a.state, it + 1, tries)) return;
        double res = 0.0;
        for (uint32_t i = threadIdx.x; i < gridDim.x; i += PL_THREADS) res += __ldcg(slots + i);
        s = pl_cta_total(res, red);
        ++done;
        if (s < (double)a.eps) break;
        float *t = xa;
        xa = xb;
        xb = t;
        t = ca;
        ca = cb;
        cb = t;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.state[1] = done;
}

// CTAs per period for the four tiers in proportion to their work (entries
// plus a per-row cost of 16 entries); a tier with work gets at least one.
uint32_t plan_split(const double w[4]) {
    double tot = w[0] + w[1] + w[2] + w[3];
    uint32_t t[4] = {0, 0, 0, 0}, sum = 0;
    if (tot <= 0) return 1u | (1u << 8) | (1u << 16) | (13u << 24);
    for (int i = 0; i < 4; ++i) {
        t[i] = w[i] > 0 ? std::max<uint32_t>(1, (uint32_t)(PL_PERIOD * w[i] / tot + 0.5)) : 0;
        sum += t[i];
    }
    int big = 0;
    for (int i = 1; i < 4; ++i)
        if (t[i] > t[big]) big = i;
    while (sum > PL_PERIOD) { --t[big]; --sum; }
    while (sum < PL_PERIOD) { ++t[big]; ++sum; }
    return t[0] | (t[1] << 8) | (t[2] << 16) | (t[3] << 24);
}

// CTAs of a sweep over `work` (entries plus 16 per row): rounds of PL_PERIOD,
// PL_CTA_WORK per CTA, at most eight waves of 8 resident CTAs per SM.  At
// R-MAT scale 22 a sweep takes 0.309 ms with eight waves, 0.314 with six,
// 0.325 with four, 0.359 with two and 0.406 with one (smaller CTA shares even
// out the tiers' tails); on 16 K vertices 9,472 CTAs with hardly a row each
// took 10.5 us, 672 take 6.  GV_PL_WAVES overrides the number of rounds.
constexpr double PL_CTA_WORK = 1024;
unsigned plan_waves(double work, const char *env_name) {
    if (const char *env = std::getenv(env_name)) {
        const unsigned w = (unsigned)std::strtoul(env, nullptr, 10);
        if (w >= 1 && w <= PL_WAVES_MAX) return w;
    }
    return (unsigned)std::min<double>(148 * 64 / PL_PERIOD, std::max(1.0, std::ceil(work / (PL_CTA_WORK * PL_PERIOD))));
}

template <typename T>
T *carve(char *&p, size_t count) {
    T *r = reinterpret_cast<T *>(p);
    p += ((count * sizeof(T)) + 255) & ~(size_t)255;
    return r;
}

// ------------------------------------------------ batched PPR over the plan
// k personalised queries (2 <= k <= 32) share every adjacency read of a
// sweep.  Values are row-major in plan order with a power-of-two stride K >= k
// (x[row * K + q]), so the k contributions of one neighbour are one aligned
// load of at most 128 bytes.  A group of K lanes owns a row (lane q = query
// q); 32 / K groups share a warp.  Rows of WARP_DEG or more entries take the
// whole warp (groups interleave over the entries, then combine), hub rows are
// cut into the single sweep's items.  Entries are summed in row order inside a
// group and the groups combine in a fixed butterfly, so results repeat bit
// for bit.  Same iteration as the store's batched sweep (one lane per query,
// residual per query, every query under epsilon to stop).
struct PlanBatch {
    const uint32_t *off, *col, *irow, *ifirst;
    const float *rdeg;
    const float *gather;  // contributions [(n + 1) K], plan order
    const float *xold;
    float *xnew, *cnew;
    float *ipart;         // [nitems][K]
    double *partial;      // [CTA][32]
    int *state;           // [0] converged, [1] sweeps done, [2] CTAs of the finish launch done
    const uint32_t *srow; // [32]: query q's source row, GV_NIL past k
    float alpha, src_val, eps;
    uint32_t k, rH, rW, rZ, n, nitems;
    uint32_t split;       // CTAs per period: items | warp rows << 8 (the rest: group rows)
};

// Entries [e0, e1) by the whole warp: group g takes the entries at g K + t of
// each run of 32 (U runs in flight); returns, in every lane, the sum for its
// query over all the entries.
template <int K>
__device__ __forceinline__ float plk_warp_segment(const PlanBatch &a, uint32_t e0, uint32_t e1) {
    constexpr int U = K >= 8 ? 1 : 8 / K;
    const uint32_t lane = threadIdx.x & 31u, q = lane % K, grp = lane / K;
    const bool live = q < a.k;
    float acc = 0.f;
    for (uint32_t b = e0; b < e1; b += 32 * U) {
        uint32_t c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t e = b + 32 * u + lane;
            c[u] = e < e1 ? __ldcs(a.col + e) : a.n;
        }
        float v[U][K];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int t = 0; t < K; ++t) {
                const uint32_t ct = __shfl_sync(GV_FULL_MASK, c[u], grp * K + t);
                v[u][t] = (ct < a.n && live) ? __ldg(a.gather + (size_t)ct * K + q) : 0.f;
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int t = 0; t < K; ++t) acc += v[u][t];
    }
#pragma unroll
    for (int o = K; o < 32; o <<= 1) acc += __shfl_xor_sync(GV_FULL_MASK, acc, o);
    return acc;
}

template <int K>
__device__ __forceinline__ void plk_finish(const PlanBatch &a, uint32_t r, uint32_t q, uint32_t my_src, float acc,
                                           double &res) {
    const float b = my_src == r ? a.src_val : 0.f;
    const float xv = b + a.alpha * acc;
    const size_t at = (size_t)r * K + q;
    a.xnew[at] = xv;
    a.cnew[at] = xv * a.rdeg[r];
    res += (double)fabsf(xv - a.xold[at]);
}

template <int K>
__device__ __forceinline__ void plk_items(const PlanBatch &a, uint32_t vb, uint32_t vg) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = vg * (PL_THREADS / 32);
    for (uint32_t it = vb * (PL_THREADS / 32) + (threadIdx.x >> 5); it < a.nitems; it += nw) {
        const uint32_t r = a.irow[it];
        const uint32_t e0 = a.off[r] + (it - a.ifirst[r]) * ITEM_ENTRIES;
        const uint32_t e1 = min(a.off[r + 1], e0 + ITEM_ENTRIES);
        const float acc = plk_warp_segment<K>(a, e0, e1);
        if (lane < K) a.ipart[(size_t)it * K + lane] = acc;
    }
}

template <int K>
__device__ __forceinline__ void plk_warp_rows(const PlanBatch &a, uint32_t my_src, uint32_t vb, uint32_t vg,
                                              double &res) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = vg * (PL_THREADS / 32);
    for (uint32_t r = a.rH + vb * (PL_THREADS / 32) + (threadIdx.x >> 5); r < a.rW; r += nw) {
        const float acc = plk_warp_segment<K>(a, a.off[r], a.off[r + 1]);
        if (lane < a.k) plk_finish<K>(a, r, lane, my_src, acc, res);
    }
}

// Rows [rW, rZ): a group of K lanes per row, 32 / K rows per warp; lane q
// loads entry j + u K + q of its row, the group's lanes take turns as the
// neighbour.
template <int K>
__device__ __forceinline__ void plk_group_rows(const PlanBatch &a, uint32_t my_src, uint32_t vb, uint32_t vg,
                                               double &res) {
    constexpr int U = K >= 8 ? 1 : 8 / K;
    constexpr uint32_t G = 32 / K;
    const uint32_t lane = threadIdx.x & 31u, q = lane % K, grp = lane / K;
    const bool live = q < a.k;
    const uint32_t nw = vg * (PL_THREADS / 32);
    for (uint32_t rb = a.rW + (vb * (PL_THREADS / 32) + (threadIdx.x >> 5)) * G; rb < a.rZ; rb += nw * G) {
        const uint32_t r = rb + grp;
        const bool ok = r < a.rZ;
        const uint32_t o = ok ? a.off[r] : 0u, len = ok ? a.off[r + 1] - o : 0u;
        const uint32_t most = __reduce_max_sync(GV_FULL_MASK, len);
        float acc = 0.f;
        for (uint32_t j = 0; j < most; j += K * U) {
            uint32_t c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t e = j + u * K + q;
                c[u] = e < len ? __ldcs(a.col + o + e) : a.n;
            }
            float v[U][K];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int t = 0; t < K; ++t) {
                    const uint32_t ct = __shfl_sync(GV_FULL_MASK, c[u], grp * K + t);
                    v[u][t] = (ct < a.n && live) ? __ldg(a.gather + (size_t)ct * K + q) : 0.f;
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int t = 0; t < K; ++t) acc += v[u][t];
        }
        if (ok && live) plk_finish<K>(a, r, q, my_src, acc, res);
    }
}

// Per-query residual of a CTA into partial[slot][0, K): lanes of one query
// are combined across warps, then across the groups of a warp (fixed orders).
template <int K>
__device__ __forceinline__ void plk_residual(double res, double *__restrict__ partial, uint32_t slot) {
    __shared__ double red[PL_THREADS / 32][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    red[warp][lane] = res;
    __syncthreads();
    if (warp == 0) {
        double t = 0.0;
        for (int w = 0; w < PL_THREADS / 32; ++w) t += red[w][lane];
#pragma unroll
        for (int o = K; o < 32; o <<= 1) t += __shfl_xor_sync(GV_FULL_MASK, t, o);
        if (lane < K) partial[(size_t)slot * 32 + lane] = t;
    }
}

template <int K>
__device__ __forceinline__ void plk_sweep_body(const PlanBatch &a) {
    if (a.state[0]) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t my_src = a.srow[lane % K];
    const uint32_t t0 = a.split & 0xFFu, t1 = (a.split >> 8) & 0xFFu, t2 = PL_PERIOD - t0 - t1;
    const uint32_t r = blockIdx.x % PL_PERIOD, w = blockIdx.x / PL_PERIOD, waves = gridDim.x / PL_PERIOD;
    double res = 0.0;
    if (r < t0) plk_items<K>(a, w * t0 + r, waves * t0);
    else if (r < t0 + t1) plk_warp_rows<K>(a, my_src, w * t1 + (r - t0), waves * t1, res);
    else plk_group_rows<K>(a, my_src, w * t2 + (r - t0 - t1), waves * t2, res);
    plk_residual<K>(res, a.partial, blockIdx.x);
}

// One sweep.  16 and 32 queries are compiled for six resident CTAs (40
// registers, a few spilled): at R-MAT scale 25 that took their sweeps from
// 17.4 to 14.9 ms and from 31.6 to 26.4 ms; fewer queries keep the
// compiler's choice (32-40 registers; capped at 40, 4 queries went from 4.9
// to 5.4 ms).
template <int K>
__global__ void __launch_bounds__(PL_THREADS) k_plk_sweep(PlanBatch a) {
    plk_sweep_body<K>(a);
}

template <int K>
__global__ void __launch_bounds__(PL_THREADS, 6) k_plk_sweep_wide(PlanBatch a) {
    plk_sweep_body<K>(a);
}

// Ends a sweep: hub rows (a thread per row and query, the row's item partials
// in item order), a share of the sweep's residual slots per CTA, and in the CTA
// that finishes last the residual of every query and the convergence flag; all
// sums in fixed orders.  (One CTA summing all 9,472 slots of 32 queries took
// 150 us of every sweep.)
template <int K>
__global__ void __launch_bounds__(PL_THREADS) k_plk_fin(PlanBatch a, uint32_t nslots) {
    __shared__ double red[PL_THREADS / 32][32];
    __shared__ bool last;
    if (a.state[0]) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t q = threadIdx.x % K;  // the stride is a multiple of K
    const uint32_t my_src = a.srow[q];
    double res = 0.0;
    const uint32_t total = a.rH * K;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const uint32_t r = i / K;
        if (q >= a.k) continue;
        float t = 0.f;
        for (uint32_t it = a.ifirst[r]; it < a.ifirst[r + 1]; ++it) t += a.ipart[(size_t)it * K + q];
        plk_finish<K>(a, r, q, my_src, t, res);
    }
    if (lane < K)
#pragma unroll 4
        for (uint32_t p = blockIdx.x + PL_FIN * warp; p < nslots; p += PL_FIN * (PL_THREADS / 32))
            res += a.partial[(size_t)p * 32 + lane];
    plk_residual<K>(res, a.partial, nslots + blockIdx.x);
    if (warp == 0) {  // it wrote the CTA's slot
        __threadfence();
        __syncwarp();
        if (lane == 0) last = pl_last(&a.state[2]);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    if (lane < K)
#pragma unroll 4
        for (uint32_t p = warp; p < PL_FIN; p += PL_THREADS / 32) t += __ldcg(a.partial + (size_t)(nslots + p) * 32 + lane);
    red[warp][lane] = t;
    __syncthreads();
    if (warp == 0) {
        double sum = 0.0;
        for (int w = 0; w < PL_THREADS / 32; ++w) sum += red[w][lane];
        const bool ok = __all_sync(GV_FULL_MASK, lane >= a.k || sum < (double)a.eps);
        if (lane == 0) {
            a.state[1] += 1;
            a.state[2] = 0;
            if (ok) a.state[0] = 1;
        }
    }
}

// source rows of the k queries; GV_NIL in the unused slots
__global__ void k_plk_sources(const uint32_t *__restrict__ sources, uint32_t k, uint32_t n,
                              const uint32_t *__restrict__ inv, uint32_t *__restrict__ srow) {
    const uint32_t q = threadIdx.x;
    if (q >= 32) return;
    const uint32_t v = q < k ? sources[q] : GV_NIL;
    srow[q] = v < n ? inv[v] : GV_NIL;  // a source out of range matches no row
}

// x0 = the source indicator per query and its contributions; isolated rows
// [rz, n) take their final value in both iterate buffers; row n (the
// sentinel) is zero.  Lanes past k are never read.
template <int K>
__global__ void k_plk_init(uint32_t n, const uint32_t *__restrict__ srow, const float *__restrict__ rdeg, uint32_t rz,
                           float src_base, float *__restrict__ x, float *__restrict__ c, float *__restrict__ x_other,
                           float *__restrict__ c_other) {
    const size_t total = ((size_t)n + 1) * K;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / K), q = (uint32_t)(i % K);
        const bool src = srow[q] == r;
        if (r == n) {
            x[i] = c[i] = x_other[i] = c_other[i] = 0.f;
        } else if (r >= rz) {
            const float v = src ? src_base : 0.f;
            x[i] = x_other[i] = v;
            c[i] = c_other[i] = 0.f;
        } else {  // both buffers: lanes past k are read (and never used) by the vector loads
            const float v = src ? 1.f : 0.f;
            x[i] = x_other[i] = v;
            c[i] = c_other[i] = v * rdeg[r];
        }
    }
}

// x_out[v][q] (stride k, vertex order) from the plan-order rows
template <int K>
__global__ void k_plk_out(uint32_t n, uint32_t k, const uint32_t *__restrict__ inv, const float *__restrict__ x,
                          float *__restrict__ out) {
    const size_t total = (size_t)n * k;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)(i / k), q = (uint32_t)(i % k);
        out[i] = x[(size_t)inv[v] * K + q];
    }
}

}  // namespace

namespace {

bool plan_enabled() {
    const char *env = std::getenv("GV_PR_PLAN");
    return !(env && env[0] == '0');
}

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

bool plan_pagerank_enabled(gv_graph *g) { return !g->cfg.directed && !g->cfg.weighted && plan_enabled(); }

namespace {

// The plan of the store's current adjacency (see the top of this file).
struct Plan {
    uint32_t *perm, *inv, *off, *ifirst, *col, *irow;
    float *w;          // weights beside col (plans of a weighted CSR)
    float *rdeg;
    float *ipart;      // nitems x the caller's width
    uint32_t *cnt;     // class counts per tile, scanned
    PlanFacts *facts;
    PlanTiers *tiers;
    char *extra;       // the caller's bytes at the end of the plan scratch
    uint32_t nitems, rH, rW, rG, rZ;
    uint32_t hoff[4];  // row starts of rows rH, rW, rG, rZ
};

// Plan arrays in auxiliary slot 12, with extra_bytes of the caller's behind
// them, then the class order of the rows.
template <typename Deg>
gv_status plan_order(gv_graph *g, Deg deg, size_t extra_bytes, cudaStream_t s, Plan &P) {
    const uint32_t n = g->d.n;
    const uint32_t ntiles = (n + PL_TILE - 1) / PL_TILE;
    // seven arrays, each carved to a 256-byte boundary, then the caller's bytes
    const size_t plan_bytes = (size_t)8 * 256 + ((size_t)NCLASS * ntiles + 1) * 4 + (size_t)n * 4 * 2 +
                              ((size_t)n + 1) * 4 * 3 + sizeof(PlanFacts) + sizeof(PlanTiers) + 256 + extra_bytes;
    char *p = (char *)aux_scratch(g, 12, plan_bytes);
    if (!p) return GV_ERR_NOMEM;
    P.cnt = carve<uint32_t>(p, (size_t)NCLASS * ntiles + 1);
    P.perm = carve<uint32_t>(p, n);
    P.inv = carve<uint32_t>(p, n);
    P.off = carve<uint32_t>(p, (size_t)n + 1);
    P.ifirst = carve<uint32_t>(p, (size_t)n + 1);
    P.rdeg = carve<float>(p, (size_t)n + 1);
    P.facts = carve<PlanFacts>(p, 1);
    P.tiers = carve<PlanTiers>(p, 1);
    P.extra = p;
    uint32_t *cnt = P.cnt;
    GV_LAUNCH((k_pl_count<Deg>), std::min<uint32_t>(ntiles, 148 * 8), PL_THREADS, 0, s, deg, n, ntiles, cnt);
    scan_exclusive_u32(cnt, cnt, (uint64_t)NCLASS * ntiles, cnt + (size_t)NCLASS * ntiles, g->bs.scan_tmp, s);
    GV_LAUNCH((k_pl_place<Deg>), (ntiles + PL_THREADS / 32 - 1) / (PL_THREADS / 32), PL_THREADS, 0, s, deg, n, ntiles,
              (const uint32_t *)cnt, P.perm, P.inv);
    return GV_OK;
}

// The class starts, the padded entries and the copy items, on the host.
gv_status plan_facts(const Plan &P, uint32_t n, const uint32_t *nfill, cudaStream_t s, PlanFacts &h) {
    GV_LAUNCH(k_pl_facts, 1, 64, 0, s, (const uint32_t *)P.cnt, (n + PL_TILE - 1) / PL_TILE,
              (const uint32_t *)(P.off + n), nfill, P.facts);
    cudaError_t e = cudaMemcpyAsync(&h, P.facts, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return cuda_status(e, "plan classes");
}

// Row boundaries of the tiers from the class starts.
void plan_tiers(const uint32_t *hcls, Plan &P) {
    // rows of class c hold degrees [2^(c-1), 2^c); classes run in descending order
    auto first_row_below = [&](uint32_t deg) {  // first row whose degree is < deg (deg a power of two)
        const uint32_t c = 32u - (uint32_t)__builtin_clz(deg);  // class of deg itself
        return hcls[NCLASS - c];                                  // start of class c - 1
    };
    P.rH = first_row_below(HUB_DEG);
    P.rW = first_row_below(WARP_DEG);
    P.rG = first_row_below(GROUP_DEG);
    P.rZ = hcls[NCLASS - 1];  // first isolated row (class 0 comes last)
}

// Hub items (auxiliary slot 15, with ipart_width floats each), and the entry
// offsets of the tier boundaries.
gv_status plan_items(gv_graph *g, uint32_t ipart_width, cudaStream_t s, Plan &P) {
    P.nitems = 0;
    P.irow = nullptr;
    P.ipart = nullptr;
    if (P.rH) {
        GV_LAUNCH(k_pl_item_count, grid_for(P.rH, 256), 256, 0, s, (const uint32_t *)P.off, P.rH, P.ifirst);
        scan_exclusive_u32(P.ifirst, P.ifirst, P.rH, P.ifirst + P.rH, g->bs.scan_tmp, s);
    }
    GV_LAUNCH(k_pl_tier_facts, 1, 32, 0, s, (const uint32_t *)P.off, make_uint4(P.rH, P.rW, P.rG, P.rZ),
              (const uint32_t *)(P.ifirst + P.rH), P.tiers);
    PlanTiers h;
    cudaError_t e = cudaMemcpyAsync(&h, P.tiers, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "plan items");
    std::copy(h.hoff, h.hoff + 4, P.hoff);
    P.nitems = h.nitems;
    if (P.rH) {
        char *q = (char *)aux_scratch(g, 15, (size_t)P.nitems * 4 * (1 + ipart_width) + 512);
        if (!q) return GV_ERR_NOMEM;
        P.irow = carve<uint32_t>(q, P.nitems);
        P.ipart = carve<float>(q, (size_t)P.nitems * ipart_width);
        GV_LAUNCH(k_pl_item_fill, grid_for(P.rH, 256), 256, 0, s, (const uint32_t *)P.ifirst, P.rH, P.irow);
    }
    return GV_OK;
}

// Builds the store's plan into auxiliary slots 12-15 (plan arrays and
// extra_bytes, padded columns, copy items, hub items with ipart_width floats
// each).  *ok is false, with nothing built, when the padded rows would not
// fit uint32 row starts.
gv_status plan_build(gv_graph *g, size_t extra_bytes, uint32_t ipart_width, cudaStream_t s, Plan &P, bool *ok) {
    *ok = false;
    DevGraph d = g->d;
    const uint32_t n = d.n;
    Ctl cc;
    gv_status st = read_ctl(g, &cc, s);
    if (st != GV_OK) return st;
    // rows hold the used slots (at most the used blocks' slots) plus padding
    const uint64_t padded_max = (d.P - cc.free_top) * (uint64_t)d.B + 3ull * n;
    if (padded_max >= 0xFFFFFFF0ull || n == 0) return GV_OK;  // uint32 row starts: the store sweep serves it
    st = plan_order(g, DegOfStore{d.vtx}, extra_bytes, s, P);
    if (st != GV_OK) return st;
    uint32_t *perm = P.perm, *inv = P.inv, *off = P.off, *ifirst = P.ifirst;
    // row lengths, starts, inverse degrees, copy items of the multi-block rows
    uint32_t *ffirst = ifirst;  // free until the hub items are built
    GV_LAUNCH(k_pl_rowlen, grid_for(n, 256), 256, 0, s, d, (const uint32_t *)perm, off, P.rdeg, ffirst);
    scan_exclusive_u32(off, off, n, off + n, g->bs.scan_tmp, s);
    scan_exclusive_u32(ffirst, ffirst, n, ffirst + n, g->bs.scan_tmp, s);
    PlanFacts h;
    st = plan_facts(P, n, ffirst + n, s, h);
    if (st != GV_OK) return st;
    const uint32_t total = h.total, nfill = h.nfill;
    plan_tiers(h.cls, P);
    // the padded, renumbered columns, straight from the store's blocks
    P.col = (uint32_t *)aux_scratch(g, 13, ((size_t)total + 4) * 4 + 256);
    uint32_t *frow = (uint32_t *)aux_scratch(g, 14, ((size_t)nfill + 1) * 4 + 256);
    if (!P.col || !frow) return GV_ERR_NOMEM;
    GV_LAUNCH(k_pl_fill_small, 148 * 16, PL_THREADS, 0, s, d, (const uint32_t *)perm, (const uint32_t *)inv,
              (const uint32_t *)off, P.col);
    if (nfill) {
        GV_LAUNCH(k_pl_item_fill, grid_for(n, 256), 256, 0, s, (const uint32_t *)ffirst, n, frow);
        GV_LAUNCH(k_pl_fill_items, 148 * 16, PL_THREADS, 0, s, d, (const uint32_t *)perm, (const uint32_t *)inv,
                  (const uint32_t *)off, (const uint32_t *)frow, (const uint32_t *)ffirst, nfill, P.col);
    }
    st = plan_items(g, ipart_width, s, P);
    *ok = st == GV_OK;
    return st;
}

// Builds the plan of a CSR (in_ as plan_csr_solve takes it), weights in slot
// 18.  *ok is false when it does not fit uint32 row starts or the scratch
// could not be had.
gv_status plan_build_csr(gv_graph *g, const PlanCsr &in, size_t extra_bytes, cudaStream_t s, Plan &P, bool *ok) {
    *ok = false;
    const uint32_t n = g->d.n;
    if (in.entries + 3ull * n >= 0xFFFFFFF0ull || n == 0) return GV_OK;
    const DegOfCsr deg{in.off};
    P.col = (uint32_t *)aux_scratch(g, 13, (in.entries + 3ull * n + 4) * 4 + 256);
    P.w = (in.w && P.col) ? (float *)aux_scratch(g, 18, (in.entries + 3ull * n + 4) * 4 + 256) : nullptr;
    if (!P.col || (in.w && !P.w)) return GV_OK;
    if (plan_order(g, deg, extra_bytes, s, P) != GV_OK) return GV_OK;
    GV_LAUNCH(k_pl_rowlen_csr, grid_for(n, 256), 256, 0, s, deg, n, (const uint32_t *)P.perm, P.off);
    scan_exclusive_u32(P.off, P.off, n, P.off + n, g->bs.scan_tmp, s);
    PlanFacts h;
    gv_status st = plan_facts(P, n, nullptr, s, h);
    if (st != GV_OK) return st;
    plan_tiers(h.cls, P);
    const uint32_t quads = h.total >> 2;
    if (quads) {
        const unsigned grid = grid_for(quads, 8 * 128, 148 * 32);
        if (in.w)
            GV_LAUNCH(k_pl_fill_csr<true>, grid, PL_THREADS, 0, s, deg, n, in.dst, in.w, (const uint32_t *)P.perm,
                      (const uint32_t *)P.inv, (const uint32_t *)P.off, quads, P.col, P.w);
        else
            GV_LAUNCH(k_pl_fill_csr<false>, grid, PL_THREADS, 0, s, deg, n, in.dst, in.w, (const uint32_t *)P.perm,
                      (const uint32_t *)P.inv, (const uint32_t *)P.off, quads, P.col, P.w);
    }
    st = plan_items(g, 1, s, P);
    if (st == GV_ERR_NOMEM) return GV_OK;
    *ok = st == GV_OK;
    return st;
}

// Iterates, contributions, residual slots and flags of a single-vector solve,
// behind the plan arrays.
struct PlanVecs {
    float *x0, *x1, *c0, *c1, *stage;
    double *partial;
    int *state;
};

size_t plan_vecs_bytes(uint32_t n) {
    return ((size_t)n + 1) * 4 * 4 + 4 * 256 + ((size_t)PL_GRID + PL_FIN_MAX) * 8 + 256 + 64 + 256 + (size_t)n * 4 + 256;
}

PlanVecs plan_vecs(const Plan &P, uint32_t n) {
    char *p = P.extra;
    PlanVecs v;
    v.x0 = carve<float>(p, (size_t)n + 1);
    v.x1 = carve<float>(p, (size_t)n + 1);
    v.c0 = carve<float>(p, (size_t)n + 1);
    v.c1 = carve<float>(p, (size_t)n + 1);
    v.partial = carve<double>(p, PL_GRID + PL_FIN_MAX);
    v.state = carve<int>(p, 16);
    v.stage = carve<float>(p, n);
    return v;
}

// Work (entries plus 16 per row) up to which all sweeps run in one launch
// (GV_PL_LOOP overrides it).  A call, sweep by sweep against one launch, R-MAT
// and uniform graphs of edge factor 16: 16 K vertices 371 / 279 and 288 / 211
// us, 128 K 527 / 454 and 516 / 367, 256 K (work 12e6) 701 / 626 and 739 / 575,
// 512 K (25e6) 988 / 1066 and 1130 / 999: many CTAs per SM even out larger
// sweeps better than the resident ones do.
double plan_loop_max() {
    if (const char *env = std::getenv("GV_PL_LOOP")) return std::strtod(env, nullptr);
    return 16e6;
}

// CTAs of k_pl_loop that can be resident together.
template <bool W>
unsigned plan_loop_ctas() {
    int dev = 0, sms = 0, coop = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pl_loop<W>, PL_THREADS, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (unsigned)(sms * std::min(per, 4));
}

// Sweeps from v.x0 (and v.c0) until the step is below eps or max_iter; rows
// [a.rZ, n) are swept in the first two sweeps only (they gather nothing, so
// they keep the value those leave in both iterates) when last_row is n, never
// when it is a.rZ.  *result is the iterate that holds the last one.  init()
// launches what sets the iterates to their start.
template <bool W, typename Init>
gv_status plan_run(PlanSweep a, const Plan &P, const PlanVecs &v, uint32_t last_row, float eps, int max_iter,
                   int prof_slot, cudaStream_t s, int *sweeps, float **result, Init init) {
    init();
    // tier work (entries + 16 per row) from the row starts read back by the build
    const uint32_t *hoff = P.hoff;
    const double w[4] = {(double)hoff[0], (double)(hoff[1] - hoff[0]) + 16.0 * (P.rW - P.rH),
                         (double)(hoff[2] - hoff[1]) + 16.0 * (P.rG - P.rW),
                         (double)(hoff[3] - hoff[2]) + 16.0 * (P.rZ - P.rG) + (last_row > P.rZ ? 16.0 : 0.0)};
    cudaMemsetAsync(v.state, 0, 16, s);
    // the sweep uses little shared memory: give the SM's on-chip memory to L1,
    // where the hot contributions live
    cudaFuncSetAttribute(k_pl_sweep<W>, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
    cudaGetLastError();
    a.off = P.off;
    a.col = P.col;
    a.w = P.w;
    a.irow = P.irow;
    a.ifirst = P.ifirst;
    a.ipart = P.ipart;
    a.partial = v.partial;
    a.state = v.state;
    a.eps = eps;
    a.rH = P.rH;
    a.rW = P.rW;
    a.rG = P.rG;
    a.nitems = P.nitems;
    a.split = plan_split(w);
    const unsigned grid = PL_PERIOD * plan_waves(w[0] + w[1] + w[2] + w[3], "GV_PL_WAVES");
    float *xa = v.x0, *xb = v.x1, *ca = v.c0, *cb = v.c1;
    const bool contrib = a.cnew != nullptr;
    const double work = w[0] + w[1] + w[2] + w[3];
    if (work <= plan_loop_max() && max_iter > 0) {
        a.gather = contrib ? ca : xa;
        a.xold = xa;
        a.xnew = xb;
        unsigned loop_grid = std::min(grid, plan_loop_ctas<W>());
        loop_grid -= loop_grid % PL_PERIOD;
        uint32_t rz = P.rZ;
        uint32_t tries = PL_WAIT_LIMIT;  // GV_PL_WAIT: looks for the other CTAs before the loop is given up
        if (const char *env = std::getenv("GV_PL_WAIT")) tries = (uint32_t)std::strtoul(env, nullptr, 10);
        void *args[] = {&a, &last_row, &rz, &max_iter, &tries};
        cudaError_t e = loop_grid ? cudaErrorUnknown : cudaErrorCooperativeLaunchTooLarge;
        if (loop_grid) {
            ProfScope ps(prof_slot, s);
            e = cudaLaunchCooperativeKernel((const void *)k_pl_loop<W>, dim3(loop_grid), dim3(PL_THREADS), args, 0, s);
            if (e == cudaSuccess) g_launches.fetch_add(1, std::memory_order_relaxed);
        }
        if (e == cudaSuccess) {
            int h[4] = {0, 0, 0, 0};
            e = cudaMemcpyAsync(h, v.state, 16, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return cuda_status(e, "plan loop");
            if (!h[3]) {
                *sweeps = h[1];
                *result = (h[1] & 1) ? v.x1 : v.x0;
                return GV_OK;
            }
            cudaMemsetAsync(v.state, 0, 16, s);  // a wait ran out: sweep by sweep, from the start
            init();
        } else {
            cudaGetLastError();  // no cooperative launch to be had: sweep by sweep
        }
    }
    // finish: a warp per hub row, 512 slots a CTA, one CTA where that is all it takes
    const unsigned fin = (P.rH <= 64 && grid <= 4096) ? 1u : grid_for((uint64_t)P.rH * 64 + grid, 512, PL_FIN_MAX);
    int h_state[2] = {0, 0};
    int launched = 0;
    while (launched < max_iter) {
        const int chunk = std::min(8, max_iter - launched);
        for (int i = 0; i < chunk; ++i) {
            a.gather = contrib ? ca : xa;
            a.xold = xa;
            a.xnew = xb;
            a.cnew = contrib ? cb : nullptr;
            a.rZ = launched + i < 2 ? last_row : P.rZ;
            {
                ProfScope ps(prof_slot, s);
                GV_LAUNCH(k_pl_sweep<W>, grid, PL_THREADS, 0, s, a);
                GV_LAUNCH(k_pl_fin, fin, PL_THREADS, 0, s, a, grid);
            }
            std::swap(xa, xb);
            std::swap(ca, cb);
        }
        launched += chunk;
        cudaError_t e = cudaMemcpyAsync(h_state, v.state, 8, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "plan sweeps");
        if (h_state[0]) break;
    }
    *sweeps = h_state[1];
    *result = (h_state[1] & 1) ? v.x1 : v.x0;  // sweep i (1-based) wrote x1 when i is odd
    return GV_OK;
}

}  // namespace

gv_status plan_pagerank(gv_graph *g, float alpha, float eps, int max_iter, const float *x_init, int init_mem,
                        uint32_t source, float *x_out, int32_t *sweeps, int mem, cudaStream_t s,
                        bool *planned) {
    *planned = false;
    const uint32_t n = g->d.n;
    Plan P{};
    bool ok = false;
    gv_status st = plan_build(g, plan_vecs_bytes(n), 1, s, P, &ok);
    if (st != GV_OK || !ok) return st;
    const PlanVecs v = plan_vecs(P, n);
    cudaError_t e = cudaSuccess;
    // start vector
    uint32_t src_row = GV_NIL;
    if (source != GV_NIL) {
        e = cudaMemcpyAsync(&src_row, P.inv + source, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "plan source");
    }
    const float *xin = nullptr;
    if (x_init) {
        if (init_mem == GV_MEM_DEVICE) xin = x_init;
        else {
            e = cudaMemcpyAsync(v.stage, x_init, (size_t)n * 4, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return cuda_status(e, "pagerank init");
            xin = v.stage;
        }
    }
    // x0 and its contributions in plan order; the isolated rows, which the
    // sweeps never reach, get their value in x1 too
    const float fill = source == GV_NIL ? 1.0f / (float)n : 0.f;
    const float base = source == GV_NIL ? (1.0f - alpha) / (float)n : 0.f;
    const float src_val = source == GV_NIL ? 0.f : 1.0f - alpha;
    auto init = [&] {
        GV_LAUNCH(k_pl_init, grid_for((uint64_t)n + 1, 256), 256, 0, s, n, (const uint32_t *)P.perm, xin, fill, src_row,
                  1.f, (const float *)P.rdeg, P.rZ, base, src_val, v.x0, v.c0, v.x1, v.c1);
    };
    PlanSweep a{};
    a.rdeg = P.rdeg;
    a.cnew = v.c1;
    a.alpha = alpha;
    a.base = base;
    a.src_row = src_row;
    a.src_val = src_val;
    a.n = n;
    int sw = 0;
    float *res = nullptr;
    st = plan_run<false>(a, P, v, P.rZ, eps, max_iter, PROF_PULL, s, &sw, &res, init);
    if (st != GV_OK) return st;
    float *dst = mem == GV_MEM_DEVICE ? x_out : res == v.x1 ? v.x0 : v.x1;  // the other buffer is free
    GV_LAUNCH(k_pl_out, grid_for(n, 256), 256, 0, s, n, (const uint32_t *)P.inv, (const float *)res, dst);
    if (mem != GV_MEM_DEVICE) e = cudaMemcpyAsync(x_out, dst, (size_t)n * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "plan out");
    g->last_sweeps = sw;
    if (sweeps) *sweeps = sw;
    *planned = true;
    return cuda_status(cudaGetLastError(), "plan pagerank");
}

gv_status plan_csr_solve(gv_graph *g, const PlanCsr &in, const PlanSolve &q, float *x_dev, int *sweeps, cudaStream_t s,
                         bool *planned) {
    *planned = false;
    if (!plan_enabled()) return GV_OK;
    const uint32_t n = g->d.n;
    Plan P{};
    bool ok = false;
    const size_t vec = al256(((size_t)n + 1) * 4);
    gv_status st = plan_build_csr(g, in, plan_vecs_bytes(n) + 3 * vec, s, P, &ok);
    if (st != GV_OK || !ok) return st;
    const PlanVecs v = plan_vecs(P, n);
    // the row terms in plan order
    char *p = P.extra + plan_vecs_bytes(n);
    p = (char *)(((uintptr_t)p + 255) & ~(uintptr_t)255);
    auto permuted = [&](const float *x) -> float * {
        if (!x) return nullptr;
        float *y = carve<float>(p, (size_t)n);
        GV_LAUNCH(k_pl_gather, grid_for(n, 256), 256, 0, s, n, (const uint32_t *)P.perm, x, y);
        return y;
    };
    PlanSweep a{};
    a.rdeg = permuted(q.oscale);
    a.cvec = permuted(q.cvec);
    a.rscale = permuted(q.rscale);
    a.cnew = a.rdeg ? v.c1 : nullptr;
    a.alpha = q.alpha;
    a.base = q.base;
    a.src_row = GV_NIL;
    a.src_val = q.src_val;
    a.n = n;
    if (q.source != GV_NIL) {
        cudaError_t e = cudaMemcpyAsync(&a.src_row, P.inv + q.source, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "plan source");
    }
    // the sentinel row n is 0 in every buffer that a sweep gathers from
    auto init = [&] {
        GV_LAUNCH(k_pl_init, grid_for((uint64_t)n + 1, 256), 256, 0, s, n, (const uint32_t *)P.perm, q.x0, 0.f, GV_NIL,
                  0.f, (const float *)a.rdeg, n, 0.f, 0.f, v.x0, v.c0, v.x1, v.c1);
    };
    int sw = 0;
    float *res = nullptr;
    st = in.w ? plan_run<true>(a, P, v, n, q.eps, q.max_iter, q.prof_slot, s, &sw, &res, init)
              : plan_run<false>(a, P, v, n, q.eps, q.max_iter, q.prof_slot, s, &sw, &res, init);
    if (st != GV_OK) return st;
    GV_LAUNCH(k_pl_out, grid_for(n, 256), 256, 0, s, n, (const uint32_t *)P.inv, (const float *)res, x_dev);
    *sweeps = sw;
    *planned = true;
    return cuda_status(cudaGetLastError(), "plan solve");
}

namespace {

template <int K>
gv_status plan_ppr_batch_k(gv_graph *g, const Plan &P, const uint32_t *sources, int src_mem, uint32_t k, float alpha,
                           float eps, int max_iter, float *x_out, int32_t *sweeps, int mem, cudaStream_t s) {
    const uint32_t n = g->d.n;
    const size_t vec = ((size_t)n + 1) * K * sizeof(float);
    // tier work: entries, plus 16 per row of a warp and 16 per group of rows
    constexpr uint32_t G = 32 / K;
    const double w[4] = {(double)P.hoff[0], (double)(P.hoff[1] - P.hoff[0]) + 16.0 * (P.rW - P.rH),
                         (double)(P.hoff[3] - P.hoff[1]) + 16.0 * ((P.rZ - P.rW + G - 1) / G), 0.0};
    const unsigned grid = PL_PERIOD * plan_waves(w[0] + w[1] + w[2], "GV_PLK_WAVES");
    const uint32_t nparts = grid + PL_FIN;
    // iterates and contributions (4 vectors of n + 1 rows), residual slots,
    // state, sources and their rows; a host result is staged in a free iterate
    const size_t bytes = 4 * vec + (size_t)nparts * 32 * 8 + 3 * 256;
    char *p = (char *)analytics_scratch(g, bytes + 4 * 256);
    if (!p) return GV_ERR_NOMEM;
    float *x0 = carve<float>(p, vec / 4), *x1 = carve<float>(p, vec / 4);
    float *c0 = carve<float>(p, vec / 4), *c1 = carve<float>(p, vec / 4);
    double *partial = carve<double>(p, (size_t)nparts * 32);
    int *state = carve<int>(p, 16);
    uint32_t *srow = carve<uint32_t>(p, 32);
    uint32_t *dsrc = carve<uint32_t>(p, 32);
    cudaError_t e = cudaMemcpyAsync(dsrc, sources, (size_t)k * 4,
                                    src_mem == GV_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_status(e, "plan ppr sources");
    GV_LAUNCH(k_plk_sources, 1, 32, 0, s, (const uint32_t *)dsrc, k, n, (const uint32_t *)P.inv, srow);
    GV_LAUNCH(k_plk_init<K>, grid_for(((uint64_t)n + 1) * K, 256, 148 * 16), 256, 0, s, n, (const uint32_t *)srow,
              (const float *)P.rdeg, P.rZ, 1.0f - alpha, x0, c0, x1, c1);
    cudaMemsetAsync(state, 0, 16, s);
    // most of the SM's on-chip memory to L1, but room for the residual
    // tables (2 KB, plus 1 KB the system keeps per CTA) of 8 resident CTAs: a
    // zero carveout held the SM to two CTAs (25% of its warps)
    void (*sweep)(PlanBatch) = nullptr;
    if constexpr (K >= 16) sweep = k_plk_sweep_wide<K>;
    else sweep = k_plk_sweep<K>;
    cudaFuncSetAttribute(sweep, cudaFuncAttributePreferredSharedMemoryCarveout, 12);
    cudaGetLastError();
    PlanBatch a{};
    a.off = P.off;
    a.col = P.col;
    a.irow = P.irow;
    a.ifirst = P.ifirst;
    a.rdeg = P.rdeg;
    a.ipart = P.ipart;
    a.partial = partial;
    a.state = state;
    a.srow = srow;
    a.alpha = alpha;
    a.src_val = 1.0f - alpha;
    a.eps = eps;
    a.k = k;
    a.rH = P.rH;
    a.rW = P.rW;
    a.rZ = P.rZ;
    a.n = n;
    a.nitems = P.nitems;
    a.split = plan_split(w) & 0xFFFFu;  // items | warp rows; the group rows take the rest
    float *xa = x0, *xb = x1, *ca = c0, *cb = c1;
    int h_state[2] = {0, 0};
    int launched = 0;
    while (launched < max_iter) {
        const int chunk = std::min(8, max_iter - launched);
        for (int i = 0; i < chunk; ++i) {
            a.gather = ca;
            a.xold = xa;
            a.xnew = xb;
            a.cnew = cb;
            {
                ProfScope ps(PROF_PULL, s);
                GV_LAUNCH(sweep, grid, PL_THREADS, 0, s, a);
                GV_LAUNCH(k_plk_fin<K>, PL_FIN, PL_THREADS, 0, s, a, grid);
            }
            std::swap(xa, xb);
            std::swap(ca, cb);
        }
        launched += chunk;
        e = cudaMemcpyAsync(h_state, state, 8, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_status(e, "plan ppr sweeps");
        if (h_state[0]) break;
    }
    const float *res = (h_state[1] & 1) ? x1 : x0;
    float *dst = mem == GV_MEM_DEVICE ? x_out : (h_state[1] & 1) ? x0 : x1;  // n k floats fit an iterate
    GV_LAUNCH(k_plk_out<K>, grid_for((uint64_t)n * k, 256, 148 * 16), 256, 0, s, n, k, (const uint32_t *)P.inv, res,
              dst);
    if (mem != GV_MEM_DEVICE) e = cudaMemcpyAsync(x_out, dst, (size_t)n * k * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "plan ppr out");
    g->last_sweeps = h_state[1];
    if (sweeps) *sweeps = h_state[1];
    return cuda_status(cudaGetLastError(), "plan ppr batch");
}

}  // namespace

gv_status plan_ppr_batch(gv_graph *g, const uint32_t *sources, int src_mem, uint32_t k, float alpha, float eps,
                         int max_iter, float *x_out, int32_t *sweeps, int mem, cudaStream_t s, bool *planned) {
    *planned = false;
    // Per sweep at R-MAT scale 25 (1.05 G entries): 3.9 ms for 2 queries,
    // 9.6 for 8, 15.0 for 16 and 26.0 for 32, against 31-43 ms for the
    // store's batched sweep and 3.3 ms for one query's plan sweep.
    if (k < 2 || k > 32) return GV_OK;
    const uint32_t K = k <= 2 ? 2 : k <= 4 ? 4 : k <= 8 ? 8 : k <= 16 ? 16 : 32;
    Plan P{};
    bool ok = false;
    gv_status st = plan_build(g, 0, K, s, P, &ok);
    if (st != GV_OK || !ok) return st;
    *planned = true;
    switch (K) {
        case 2: return plan_ppr_batch_k<2>(g, P, sources, src_mem, k, alpha, eps, max_iter, x_out, sweeps, mem, s);
        case 4: return plan_ppr_batch_k<4>(g, P, sources, src_mem, k, alpha, eps, max_iter, x_out, sweeps, mem, s);
        case 8: return plan_ppr_batch_k<8>(g, P, sources, src_mem, k, alpha, eps, max_iter, x_out, sweeps, mem, s);
        case 16: return plan_ppr_batch_k<16>(g, P, sources, src_mem, k, alpha, eps, max_iter, x_out, sweeps, mem, s);
        default: return plan_ppr_batch_k<32>(g, P, sources, src_mem, k, alpha, eps, max_iter, x_out, sweeps, mem, s);
    }
}

}  // namespace gv
