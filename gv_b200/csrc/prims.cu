// Exclusive scan (reduce-then-scan) and stable LSD radix sort, hand-written
// for sm_100a.  The radix sort ranks each tile of keys in shared memory and
// stages it in digit order so that the global scatter writes contiguous runs;
// a pass is one launch whose tiles look back on one another (k_os_pass), or,
// above 2^30 keys, a count, a scan and a scatter (k_rs_*).
#include "prims.cuh"
#include <algorithm>
#include <cstdlib>
#include "common.cuh"
#include "launch.hpp"

namespace gv {

std::atomic<unsigned long long> g_launches{0};

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int SCAN_TOP_THREADS = 1024;
constexpr int SCAN_TOP_ITEMS = 4;

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total_out (all threads see it).
template <typename T, int NT>
__device__ __forceinline__ T block_exclusive_scan(T v, T *warp_tot, T &total_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(GV_FULL_MASK, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        constexpr int NW = NT / 32;
        T w = (lane < NW) ? warp_tot[lane] : T(0);
        T wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T t = __shfl_up_sync(GV_FULL_MASK, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < NW) warp_tot[lane] = wi - w;  // exclusive warp offsets
        if (lane == 31) warp_tot[32] = wi;       // block total
    }
    __syncthreads();
    T res = warp_tot[warp] + incl - v;
    total_out = warp_tot[32];
    __syncthreads();
    return res;
}

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const Tin *__restrict__ in, uint64_t n,
                                                              Tout *__restrict__ tile_sums) {
    __shared__ Tout wt[33];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    Tout s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        uint64_t i = base + (uint64_t)j * SCAN_THREADS + threadIdx.x;
        if (i < n) s += (Tout)in[i];
    }
    Tout tot;
    block_exclusive_scan<Tout, SCAN_THREADS>(s, wt, tot);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

template <typename Tout>
__global__ void __launch_bounds__(SCAN_TOP_THREADS) k_scan_top(Tout *__restrict__ sums, uint64_t ntiles,
                                                               Tout *__restrict__ total) {
    __shared__ Tout wt[33];
    Tout carry = 0;
    for (uint64_t cb = 0; cb < ntiles; cb += (uint64_t)SCAN_TOP_THREADS * SCAN_TOP_ITEMS) {
        Tout v[SCAN_TOP_ITEMS];
        Tout ts = 0;
#pragma unroll
        for (int j = 0; j < SCAN_TOP_ITEMS; ++j) {
            uint64_t i = cb + (uint64_t)threadIdx.x * SCAN_TOP_ITEMS + j;
            v[j] = (i < ntiles) ? sums[i] : Tout(0);
            ts += v[j];
        }
        Tout tot;
        Tout ex = block_exclusive_scan<Tout, SCAN_TOP_THREADS>(ts, wt, tot);
        Tout run = carry + ex;
#pragma unroll
        for (int j = 0; j < SCAN_TOP_ITEMS; ++j) {
            uint64_t i = cb + (uint64_t)threadIdx.x * SCAN_TOP_ITEMS + j;
            if (i < ntiles) sums[i] = run;
            run += v[j];
        }
        carry += tot;
    }
    if (total && threadIdx.x == 0) *total = carry;
}

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const Tin *in, Tout *out, uint64_t n,
                                                            const Tout *__restrict__ tile_off) {
    __shared__ Tout buf[SCAN_TILE];
    __shared__ Tout wt[33];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        uint64_t i = base + (uint64_t)j * SCAN_THREADS + threadIdx.x;
        buf[j * SCAN_THREADS + threadIdx.x] = (i < n) ? (Tout)in[i] : Tout(0);
    }
    __syncthreads();
    Tout v[SCAN_ITEMS];
    Tout ts = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        v[j] = buf[threadIdx.x * SCAN_ITEMS + j];
        ts += v[j];
    }
    Tout tot;
    Tout run = block_exclusive_scan<Tout, SCAN_THREADS>(ts, wt, tot) + tile_off[blockIdx.x];
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        buf[threadIdx.x * SCAN_ITEMS + j] = run;
        run += v[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        uint64_t i = base + (uint64_t)j * SCAN_THREADS + threadIdx.x;
        if (i < n) out[i] = buf[j * SCAN_THREADS + threadIdx.x];
    }
}

// Short arrays in one launch: a CTA takes SCAN_ONE_TILE elements at a time, a
// warp SCAN_ONE_ROWS rows of 32 of them, and carries its sum on.  Three launches
// cost 7 us whatever the size (and three trips through the driver); this takes
// 5 to 10 us.
constexpr int SCAN_ONE_ROWS = 16;
constexpr uint64_t SCAN_ONE_TILE = SCAN_TOP_THREADS * SCAN_ONE_ROWS;
constexpr uint64_t SCAN_ONE = 2 * SCAN_ONE_TILE;
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(SCAN_TOP_THREADS) k_scan_one(const Tin *in, Tout *out, uint64_t n, Tout *total) {
    __shared__ Tout wt[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Tout carry = 0;
    for (uint64_t cb = 0; cb < n; cb += SCAN_ONE_TILE) {
        const uint64_t at = cb + (uint64_t)warp * (32 * SCAN_ONE_ROWS) + lane;
        Tout v[SCAN_ONE_ROWS];
#pragma unroll
        for (int j = 0; j < SCAN_ONE_ROWS; ++j) v[j] = at + 32 * j < n ? (Tout)in[at + 32 * j] : Tout(0);
        Tout sum = 0;
#pragma unroll
        for (int j = 0; j < SCAN_ONE_ROWS; ++j) {
            Tout incl = v[j];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const Tout t = __shfl_up_sync(GV_FULL_MASK, incl, o);
                if (lane >= o) incl += t;
            }
            v[j] = sum + incl - v[j];
            sum += __shfl_sync(GV_FULL_MASK, incl, 31);
        }
        Tout tot;  // every lane holds its warp's sum; lane 31's stands for it
        const Tout before = carry + block_exclusive_scan<Tout, SCAN_TOP_THREADS>(lane == 31 ? sum : Tout(0), wt, tot);
        const Tout base = __shfl_sync(GV_FULL_MASK, before, 0);
#pragma unroll
        for (int j = 0; j < SCAN_ONE_ROWS; ++j)
            if (at + 32 * j < n) out[at + 32 * j] = base + v[j];
        carry += tot;
    }
    if (total && threadIdx.x == 0) *total = carry;
}

template <typename Tin, typename Tout>
void scan_exclusive_impl(const Tin *in, Tout *out, uint64_t n, Tout *total, void *scratch,
                         cudaStream_t s) {
    if (n == 0) {
        if (total) cudaMemsetAsync(total, 0, sizeof(Tout), s);
        return;
    }
    if (n <= SCAN_ONE) {
        GV_LAUNCH((k_scan_one<Tin, Tout>), 1, SCAN_TOP_THREADS, 0, s, in, out, n, total);
        return;
    }
    uint64_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    Tout *sums = static_cast<Tout *>(scratch);
    GV_LAUNCH((k_scan_reduce<Tin, Tout>), (unsigned)ntiles, SCAN_THREADS, 0, s, in, n, sums);
    GV_LAUNCH((k_scan_top<Tout>), 1, SCAN_TOP_THREADS, 0, s, sums, ntiles, total);
    GV_LAUNCH((k_scan_down<Tin, Tout>), (unsigned)ntiles, SCAN_THREADS, 0, s, in, out, n,
              (const Tout *)sums);
}

// ---------------------------------------------------------------- radix sort
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 4096 keys
constexpr int RS_RADIX = 256;

__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const unsigned long long *__restrict__ keys,
                                                           uint64_t n, int shift, uint32_t mask,
                                                           uint32_t *__restrict__ counts,
                                                           uint32_t ntiles) {
    __shared__ uint32_t hist[RS_RADIX];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * RS_TILE;
#pragma unroll 4
    for (int j = 0; j < RS_ITEMS; ++j) {
        uint64_t i = base + (uint64_t)j * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&hist[(uint32_t)(keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    counts[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

struct RsSmem {
    unsigned long long keys[RS_TILE];
    uint32_t vals[RS_TILE];
    uint32_t wcount[RS_WARPS][RS_RADIX];
    uint32_t run[RS_RADIX];
    uint32_t tstart[RS_RADIX];
    uint32_t gstart[RS_RADIX];
    uint32_t wt[33];
};

template <bool VALS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_downsweep(const unsigned long long *__restrict__ kin,
                                                             unsigned long long *__restrict__ kout,
                                                             const uint32_t *__restrict__ vin,
                                                             uint32_t *__restrict__ vout, uint64_t n,
                                                             int shift, uint32_t mask,
                                                             const uint32_t *__restrict__ offsets,
                                                             uint32_t ntiles) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RsSmem &S = *reinterpret_cast<RsSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * RS_TILE;
    const uint64_t rem = n - base;
    const uint32_t tile_n = rem < (uint64_t)RS_TILE ? (uint32_t)rem : (uint32_t)RS_TILE;

    unsigned long long k[RS_ITEMS];
    uint32_t v[RS_ITEMS];
    uint32_t rank[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        uint32_t li = (uint32_t)j * RS_THREADS + tid;
        k[j] = (li < tile_n) ? kin[base + li] : 0ull;
        if (VALS) v[j] = (li < tile_n) ? vin[base + li] : 0u;
    }
    S.run[tid] = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) S.wcount[w][tid] = 0;
    __syncthreads();

    const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        uint32_t li = (uint32_t)j * RS_THREADS + tid;
        bool valid = li < tile_n;
        uint32_t d = valid ? ((uint32_t)(k[j] >> shift) & mask) : 0x100u;
        uint32_t peers = __match_any_sync(GV_FULL_MASK, d);
        uint32_t r = __popc(peers & lt_mask);
        if (valid && r == 0) S.wcount[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t acc = S.run[d] + r;
            for (int w = 0; w < warp; ++w) acc += S.wcount[w][d];
            rank[j] = acc;
        }
        __syncthreads();
        {
            uint32_t sum = 0;
#pragma unroll
            for (int w = 0; w < RS_WARPS; ++w) {
                sum += S.wcount[w][tid];
                S.wcount[w][tid] = 0;
            }
            S.run[tid] += sum;
        }
        __syncthreads();
    }
    // Tile-local digit starts and global digit starts for this tile.
    uint32_t tot;
    uint32_t ex = block_exclusive_scan<uint32_t, RS_THREADS>(S.run[tid], S.wt, tot);
    S.tstart[tid] = ex;
    S.gstart[tid] = offsets[(uint64_t)tid * ntiles + blockIdx.x];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        uint32_t li = (uint32_t)j * RS_THREADS + tid;
        if (li < tile_n) {
            uint32_t d = (uint32_t)(k[j] >> shift) & mask;
            uint32_t pos = S.tstart[d] + rank[j];
            S.keys[pos] = k[j];
            if (VALS) S.vals[pos] = v[j];
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < tile_n; i += RS_THREADS) {
        unsigned long long key = S.keys[i];
        uint32_t d = (uint32_t)(key >> shift) & mask;
        uint64_t pos = (uint64_t)S.gstart[d] + (i - S.tstart[d]);
        kout[pos] = key;
        if (VALS) vout[pos] = S.vals[i];
    }
}

// ------------------------------------------------- radix sort, one sweep
// A pass in one launch: each tile ranks its keys, publishes its digit counts
// and finds its place by looking back over the tiles before it, so a pass reads
// and writes every key once and needs no counting launch or scan of its own
// (those read every key again and were four of a pass's five launches).  The
// digit totals of all passes come from one launch ahead of the first.
//
// A tile is numbered by the order in which its CTA starts, so the tiles a CTA
// looks back on are running or done.  It still waits for none without a
// limit: past OS_WAIT tries it counts the other tile's digits itself, from keys
// that this pass only reads.
//
// Status of (tile, digit): a count in 30 bits and a two-bit code, for the
// tile alone (OS_ALONE) or for all tiles up to it (OS_UPTO).  The codes of even
// and odd passes differ, so that one clearing serves all passes: even passes
// find 0 (cleared, or an odd pass's end) in words not yet written, odd ones 2.
//
// A warp owns ITEMS runs of 32 consecutive keys and ranks them against
// counters of its own, in order, so the sort is stable and the
// ranking has no barrier.  A pass: 1 M keys 29 -> 18 us, 8.4 M with values 123 ->
// 97, 16.7 M with values 240 -> 178 (the counting launch ahead of the first:
// 13, 43 and 57).  Its instructions (150 per 32 keys at 37% of the warps, ncu)
// and, up to a few million keys, the walk back over tiles that started together
// (8 us of 18) bound it, not memory.
constexpr int OS_THREADS = 256;
constexpr int OS_WARPS = OS_THREADS / 32;
constexpr int OS_PASSES = 8;
constexpr uint32_t OS_TILE_MIN = OS_THREADS * 8;
constexpr uint32_t OS_COUNT = (1u << 30) - 1u;
constexpr uint64_t OS_MAX = OS_COUNT;  // keys; more take the passes above
constexpr uint32_t OS_WAIT = 1u << 16;

template <int ITEMS, bool VALS>
struct OsSmem {
    unsigned long long keys[OS_THREADS * ITEMS];
    uint32_t vals[VALS ? OS_THREADS * ITEMS : 1];
    uint32_t cnt[OS_WARPS][RS_RADIX];
    uint32_t tstart[RS_RADIX], gstart[RS_RADIX];
    uint32_t wt[33];
    uint32_t tile;
};

// Digit `pass` of a key, without the key's bits past nbits.
struct OsDigit {
    uint32_t shift, mask;
    bool high;
    __device__ __forceinline__ OsDigit(int pass, int nbits)
        : shift(8u * ((uint32_t)pass & 3u)), mask(nbits - 8 * pass >= 8 ? 0xFFu : (1u << (nbits - 8 * pass)) - 1u),
          high(pass > 3) {}
    __device__ __forceinline__ uint32_t operator()(unsigned long long key) const {
        const uint32_t word = high ? (uint32_t)(key >> 32) : (uint32_t)key;
        return (word >> shift) & mask;
    }
};

// The keys there are: n of them, or fewer by a count on the device.
struct OsCount {
    uint64_t n;
    const unsigned long long *units;  // null: n
    uint32_t per;                     // keys per unit
    __device__ __forceinline__ uint64_t operator()() const { return units && *units * per < n ? *units * per : n; }
};

__global__ void __launch_bounds__(OS_THREADS) k_os_hist(const unsigned long long *__restrict__ keys, OsCount count,
                                                        int passes, int nbits, uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[OS_PASSES][RS_RADIX];
    const uint64_t n = count();
    for (int p = 0; p < passes; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t stride = (uint64_t)gridDim.x * OS_THREADS * 4;
    for (uint64_t base = (uint64_t)blockIdx.x * OS_THREADS * 4; base < n; base += stride) {
        unsigned long long k[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint64_t i = base + t * OS_THREADS + threadIdx.x;
            k[t] = i < n ? keys[i] : 0ull;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const bool in = base + t * OS_THREADS + threadIdx.x < n;
            const uint32_t live = __ballot_sync(GV_FULL_MASK, in);
            for (int p = 0; p < passes; ++p) {
                const uint32_t d = OsDigit(p, nbits)(k[t]);
                int same;  // runs of one digit (sentinels, high bits) in one add
                __match_all_sync(GV_FULL_MASK, in ? d : RS_RADIX, &same);
                if (same) {
                    if (lane == 0 && live) atomicAdd(&h[p][d], 32u);
                } else if (in) {
                    atomicAdd(&h[p][d], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p)
        if (h[p][threadIdx.x]) atomicAdd(&hist[p * RS_RADIX + threadIdx.x], h[p][threadIdx.x]);
}

// Keys of tile `tile` whose digit is d (the way out of a wait).
__device__ __noinline__ uint32_t os_recount(const unsigned long long *kin, uint64_t n, uint64_t base, uint32_t tile_keys,
                                            int pass, int nbits, uint32_t d) {
    const OsDigit digit(pass, nbits);
    uint32_t c = 0;
    for (uint64_t i = base; i < base + tile_keys && i < n; ++i) c += digit(kin[i]) == d ? 1u : 0u;
    return c;
}

template <int ITEMS, bool VALS>
__global__ void __launch_bounds__(OS_THREADS, ITEMS == 8 ? 4 : 3) k_os_pass(const unsigned long long *__restrict__ kin,
                                                        unsigned long long *__restrict__ kout,
                                                        const uint32_t *__restrict__ vin, uint32_t *__restrict__ vout,
                                                        OsCount count, int pass, int nbits,
                                                        const uint32_t *__restrict__ hist, uint32_t *ticket,
                                                        uint32_t *status, uint32_t wait) {
    constexpr uint32_t TILE = OS_THREADS * ITEMS;
    extern __shared__ __align__(16) unsigned char os_raw[];
    OsSmem<ITEMS, VALS> &S = *reinterpret_cast<OsSmem<ITEMS, VALS> *>(os_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t alone = pass & 1 ? 3u : 1u, upto = pass & 1 ? 0u : 2u, unset = pass & 1 ? 2u : 0u;
    const OsDigit digit(pass, nbits);
    if (tid == 0) S.tile = atomicAdd(&ticket[pass], 1u);
#pragma unroll
    for (int w = 0; w < OS_WARPS; ++w) S.cnt[w][tid] = 0;
    __syncthreads();
    const uint32_t tile = S.tile;
    const uint64_t base = (uint64_t)tile * TILE, n = count();
    if (base >= n) return;  // tiles behind the keys, and no tile looks back to them
    const uint32_t tile_n = n - base < (uint64_t)TILE ? (uint32_t)(n - base) : TILE;
    const uint32_t first = warp * (32 * ITEMS) + lane;
    unsigned long long key[ITEMS];
    uint32_t val[VALS ? ITEMS : 1], rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t li = first + 32 * j;
        key[j] = li < tile_n ? kin[base + li] : 0ull;
        if (VALS) val[j] = li < tile_n ? vin[base + li] : 0u;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const bool in = first + 32 * j < tile_n;
        const uint32_t d = digit(key[j]);
        const uint32_t peers = digit_peers(d, in);
        const uint32_t below = __popc(peers & ((1u << lane) - 1u));
        const uint32_t before = in ? S.cnt[warp][d] : 0u;
        rank[j] = before + below;
        __syncwarp();
        if (in && below == 0) S.cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread d: the tile's count of digit d, and the warps' starts in it
    uint32_t mine = 0;
#pragma unroll
    for (int w = 0; w < OS_WARPS; ++w) {
        const uint32_t c = S.cnt[w][tid];
        S.cnt[w][tid] = mine;
        mine += c;
    }
    volatile uint32_t *st = status;
    if (tile) st[(uint64_t)tile * RS_RADIX + tid] = (alone << 30) | mine;
    uint32_t tot;
    const uint32_t ts = block_exclusive_scan<uint32_t, OS_THREADS>(mine, S.wt, tot);
    S.tstart[tid] = ts;
#pragma unroll
    for (int w = 0; w < OS_WARPS; ++w) S.cnt[w][tid] += ts;  // places in the staged tile
    uint32_t at;  // place of the tile's first key of digit d
    if (tile == 0) {
        at = block_exclusive_scan<uint32_t, OS_THREADS>(hist[pass * RS_RADIX + tid], S.wt, tot);
    } else {
        // the tiles before it, two at a time (eight or 32 in flight crowd L2
        // with repeats: 20 and 26 us a pass of 1 M keys against 17)
        constexpr int OS_BACK = 2;
        at = 0;
        bool found = false;
        uint32_t tries = 0;
        for (uint32_t t = tile; !found;) {  // tiles [t, tile) are in `at`
            uint32_t w[OS_BACK];
#pragma unroll
            for (int i = 0; i < OS_BACK; ++i)
                w[i] = (uint32_t)i < t ? st[(uint64_t)(t - 1 - i) * RS_RADIX + tid] : unset << 30;
            uint32_t used = 0;
#pragma unroll
            for (int i = 0; i < OS_BACK; ++i) {
                if (found || (uint32_t)i != used || (w[i] >> 30) == unset) continue;
                at += w[i] & OS_COUNT;
                found = (w[i] >> 30) == upto;
                ++used;
            }
            t -= used;
            if (found || used) {
                tries = 0;
                continue;
            }
            if (tries++ < wait) continue;
            at += os_recount(kin, n, (uint64_t)(t - 1) * TILE, TILE, pass, nbits, tid);
            if (--t == 0) {  // all keys of smaller digits come first
                for (uint32_t d = 0; d < tid; ++d) at += hist[pass * RS_RADIX + d];
                found = true;
            }
        }
    }
    st[(uint64_t)tile * RS_RADIX + tid] = (upto << 30) | (at + mine);
    S.gstart[tid] = at - S.tstart[tid];  // place of staged key i of digit d: gstart[d] + i
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
        if (first + 32 * j < tile_n) {
            const uint32_t d = digit(key[j]);
            const uint32_t p = S.cnt[warp][d] + rank[j];
            S.keys[p] = key[j];
            if (VALS) S.vals[p] = val[j];
        }
    __syncthreads();
    for (uint32_t i = tid; i < tile_n; i += OS_THREADS) {
        const unsigned long long k = S.keys[i];
        const uint32_t d = digit(k);
        const uint32_t p = S.gstart[d] + i;
        kout[p] = k;
        if (VALS) vout[p] = S.vals[i];
    }
}

template <int ITEMS, bool VALS>
void os_launch(const unsigned long long *kin, unsigned long long *kout, const uint32_t *vin, uint32_t *vout, OsCount n,
               int pass, int nbits, const uint32_t *hist, uint32_t *ticket, uint32_t *status, uint32_t wait,
               cudaStream_t s) {
    const int smem = (int)sizeof(OsSmem<ITEMS, VALS>);
    cudaFuncSetAttribute(k_os_pass<ITEMS, VALS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const unsigned ntiles = (unsigned)((n.n + OS_THREADS * ITEMS - 1) / (OS_THREADS * ITEMS));
    GV_LAUNCH((k_os_pass<ITEMS, VALS>), ntiles, OS_THREADS, smem, s, kin, kout, vin, vout, n, pass, nbits, hist, ticket,
              status, wait);
}

}  // namespace

size_t scan_scratch_bytes(uint64_t n) {
    uint64_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    return (size_t)(ntiles + 1) * sizeof(unsigned long long);
}

void scan_exclusive_u32(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total,
                        void *scratch, cudaStream_t s) {
    scan_exclusive_impl<uint32_t, uint32_t>(in, out, n, total, scratch, s);
}

void scan_exclusive_u32_to_u64(const uint32_t *in, unsigned long long *out, uint64_t n,
                               unsigned long long *total, void *scratch, cudaStream_t s) {
    scan_exclusive_impl<uint32_t, unsigned long long>(in, out, n, total, scratch, s);
}

void scan_exclusive_u64(const unsigned long long *in, unsigned long long *out, uint64_t n,
                        unsigned long long *total, void *scratch, cudaStream_t s) {
    scan_exclusive_impl<unsigned long long, unsigned long long>(in, out, n, total, scratch, s);
}

bool radix_takes_count(uint64_t n) { return n <= OS_MAX; }

uint64_t radix_counts_elems(uint64_t n) {
    // one sweep: status words, digit totals, tickets; else counts per tile
    const uint64_t tile = n <= OS_MAX ? OS_TILE_MIN : RS_TILE;
    return ((n + tile - 1) / tile) * RS_RADIX + OS_PASSES * (RS_RADIX + 1);
}

int radix_sort_u64(unsigned long long *keys, unsigned long long *keys_alt, uint32_t *vals,
                   uint32_t *vals_alt, uint64_t n, int nbits, uint32_t *counts, void *scratch,
                   cudaStream_t s, const unsigned long long *units, uint32_t per) {
    if (n <= 1 || nbits <= 0) return 0;
    if (n <= OS_MAX) {
        const int passes = (nbits + 7) / 8;
        // small tiles keep the chip full up to a few million keys
        const bool small = n <= (1u << 22);
        const uint64_t tile = OS_THREADS * (small ? 8 : 16), words = ((n + tile - 1) / tile) * RS_RADIX;
        const OsCount count{n, units, per};
        uint32_t *status = counts, *hist = counts + words, *ticket = hist + OS_PASSES * RS_RADIX;
        cudaMemsetAsync(counts, 0, (words + OS_PASSES * (RS_RADIX + 1)) * 4, s);
        GV_LAUNCH(k_os_hist, (unsigned)std::min<uint64_t>(148 * 8, (n + 4 * OS_THREADS - 1) / (4 * OS_THREADS)),
                  OS_THREADS, 0, s, keys, count, passes, nbits, hist);
        uint32_t wait = OS_WAIT;  // GV_RS_WAIT: tries before a tile counts another's digits itself
        if (const char *env = std::getenv("GV_RS_WAIT")) wait = (uint32_t)std::strtoul(env, nullptr, 10);
        for (int p = 0; p < passes; ++p) {
            const unsigned long long *ki = p & 1 ? keys_alt : keys;
            unsigned long long *ko = p & 1 ? keys : keys_alt;
            const uint32_t *vi = p & 1 ? vals_alt : vals;
            uint32_t *vo = p & 1 ? vals : vals_alt;
            if (small && vals) os_launch<8, true>(ki, ko, vi, vo, count, p, nbits, hist, ticket, status, wait, s);
            else if (small) os_launch<8, false>(ki, ko, vi, vo, count, p, nbits, hist, ticket, status, wait, s);
            else if (vals) os_launch<16, true>(ki, ko, vi, vo, count, p, nbits, hist, ticket, status, wait, s);
            else os_launch<16, false>(ki, ko, vi, vo, count, p, nbits, hist, ticket, status, wait, s);
        }
        return passes & 1;
    }
    static bool attr_set = false;
    const size_t smem = sizeof(RsSmem);
    if (!attr_set) {
        cudaFuncSetAttribute(k_rs_downsweep<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
        cudaFuncSetAttribute(k_rs_downsweep<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
        attr_set = true;
    }
    const uint32_t ntiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
    const uint64_t ncounts = (uint64_t)ntiles * RS_RADIX;
    unsigned long long *kin = keys, *kout = keys_alt;
    uint32_t *vin = vals, *vout = vals_alt;
    int cur = 0;
    for (int shift = 0; shift < nbits; shift += 8) {
        const uint32_t mask = nbits - shift >= 8 ? 0xFFu : (1u << (nbits - shift)) - 1u;  // bits past nbits stay out
        GV_LAUNCH(k_rs_upsweep, ntiles, RS_THREADS, 0, s, kin, n, shift, mask, counts, ntiles);
        scan_exclusive_u32(counts, counts, ncounts, nullptr, scratch, s);
        if (vals)
            GV_LAUNCH(k_rs_downsweep<true>, ntiles, RS_THREADS, smem, s, kin, kout, vin, vout, n,
                      shift, mask, counts, ntiles);
        else
            GV_LAUNCH(k_rs_downsweep<false>, ntiles, RS_THREADS, smem, s, kin, kout, nullptr,
                      nullptr, n, shift, mask, counts, ntiles);
        std::swap(kin, kout);
        std::swap(vin, vout);
        cur ^= 1;
    }
    return cur;
}

}  // namespace gv
