// Matrix-Market ingest on the device and binary snapshots of a graph.
//
// gv_mtx_parse replaces the reference's host reader readFile
// (src/reader/marketReader.cu:3-121) and CSR::readGraph / initializeCSR
// (src/dynamicStructure/csr.cu:55-78): the header (first line not starting
// with '%') gives rows, cols and entries; every later line gives "src dst
// [value]", 1-based.  Here the text is copied to the device once; the lines
// that hold an entry are counted per 4 KB tile, the tile counts scanned, and
// each tile parses its lines, staged in shared memory, straight to their
// places, a thread per line, with no host loop over the data.  Lines that
// start with '%' or are blank are skipped, as the reference skips '%' lines.
//
// Bound by the text (read twice) and the outputs: 83 MB of weighted lines,
// 4.2 M entries, in device memory: 0.17 ms of kernels (0.40 with a newline
// list and per-line arrays between passes), 0.25 ms a call (5.1 with ten
// allocations per call).
//
// gv_snapshot_save / gv_snapshot_load write and read a graph as a checksummed
// CSR file (offsets, destinations, weights), the checkpoint and epoch
// snapshot of a store; loading builds the store with gv_bulk_build_csr.
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include <cuda.h>
#include "store.cuh"
#include "group.cuh"
#include "prims.cuh"
#include "launch.hpp"
#include "../../include/gv_ingest.h"

namespace gv {
namespace {

constexpr int MTX_THREADS = 256;
constexpr uint32_t MTX_TILE = MTX_THREADS * 16;  // bytes per tile, 16 per thread
constexpr uint32_t MTX_AHEAD = 256;              // bytes staged past the tile, for the line that leaves it

// Data bytes [begin, len) of the text, cut into tiles from `origin`, the last
// 16-byte boundary of memory at or before begin.
struct MtxText {
    const char *text;
    uint64_t begin, len;
    int64_t origin;
    // past the end a line ends
    __device__ __forceinline__ char operator[](uint64_t p) const { return p < len ? text[p] : '\n'; }
};

__device__ __forceinline__ bool mtx_space(char ch) { return ch == ' ' || ch == '\t' || ch == '\r'; }

// The 16 bytes at g (a multiple of 16 from origin); bytes that are not data
// come back as 0.  One aligned load where all 16 lie inside the text.
__device__ __forceinline__ uint4 mtx_load16(const MtxText &t, int64_t g) {
    if (g >= (int64_t)t.begin && g + 16 <= (int64_t)t.len) return *reinterpret_cast<const uint4 *>(t.text + g);
    union {
        uint4 v;
        char c[16];
    } r;
    r.v = make_uint4(0u, 0u, 0u, 0u);
    for (int j = 0; j < 16; ++j)
        if (g + j >= (int64_t)t.begin && g + j < (int64_t)t.len) r.c[j] = t.text[g + j];
    return r.v;
}

// Bit j: byte j is a newline.
__device__ __forceinline__ uint32_t mtx_newlines(uint4 v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t eq = __vcmpeq4(w[i], 0x0A0A0A0Au) & 0x08040201u;  // byte k keeps its bit k
        m |= ((eq | eq >> 8 | eq >> 16 | eq >> 24) & 0xFu) << (4 * i);
    }
    return m;
}

// Whether the line that starts at p holds an entry (not blank, no comment).
__device__ __forceinline__ bool mtx_entry(const MtxText &t, uint64_t p) {
    while (mtx_space(t[p])) ++p;
    const char ch = t[p];
    return ch != '\n' && ch != '%';
}

// Bit j: an entry's line starts after byte j of the 16 at g; bit 16: the first
// line does, before them.
__device__ __forceinline__ uint32_t mtx_starts(const MtxText &t, int64_t g, uint4 v, bool first) {
    uint32_t out = 0;
    for (uint32_t m = mtx_newlines(v); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        if (mtx_entry(t, (uint64_t)(g + j + 1))) out |= 1u << j;
    }
    if (first && mtx_entry(t, t.begin)) out |= 1u << 16;
    return out;
}

__global__ void __launch_bounds__(MTX_THREADS) k_mtx_count(MtxText t, uint32_t *__restrict__ tile_cnt) {
    __shared__ uint32_t red[33];
    const int64_t g = t.origin + (int64_t)blockIdx.x * MTX_TILE + threadIdx.x * 16;
    const uint32_t c = __popc(mtx_starts(t, g, mtx_load16(t, g), blockIdx.x == 0 && threadIdx.x == 0));
    const uint32_t total = cta_sum<uint32_t, MTX_THREADS>(c, red);
    if (threadIdx.x == 0) tile_cnt[blockIdx.x] = total;
}

// Unsigned decimal at p (after blanks); returns false without digits.  The
// newline that ends every line ends the scans.
template <typename Text, typename Pos>
__device__ __forceinline__ bool mtx_uint(const Text &text, Pos &p, unsigned long long &out) {
    while (mtx_space(text[p])) ++p;
    uint32_t w = 0;  // the first nine digits fit 32 bits
    Pos q = p;
    char ch = text[q];
    while (ch >= '0' && ch <= '9' && q - p < 9) {
        w = w * 10 + (uint32_t)(ch - '0');
        ch = text[++q];
    }
    unsigned long long v = w;
    while (text[q] >= '0' && text[q] <= '9' && q - p < 20) v = v * 10 + (unsigned long long)(text[q++] - '0');
    if (q == p) return false;
    p = q;
    out = v;
    return true;
}

// Decimal real (sign, digits, fraction, exponent), accumulated in fp64.
template <typename Text, typename Pos>
__device__ __forceinline__ bool mtx_real(const Text &text, Pos &p, double &out) {
    while (mtx_space(text[p])) ++p;
    Pos q = p;
    double sign = 1.0;
    if ((text[q] == '-' || text[q] == '+')) sign = text[q++] == '-' ? -1.0 : 1.0;
    double v = 0.0;
    int digits = 0, frac = 0;
    while (text[q] >= '0' && text[q] <= '9') { v = v * 10.0 + (text[q++] - '0'); ++digits; }
    if (text[q] == '.') {
        ++q;
        while (text[q] >= '0' && text[q] <= '9') { v = v * 10.0 + (text[q++] - '0'); ++digits; ++frac; }
    }
    if (!digits) return false;
    int ex = 0;
    if ((text[q] == 'e' || text[q] == 'E')) {
        Pos r = q + 1;
        int es = 1;
        if ((text[r] == '-' || text[r] == '+')) es = text[r++] == '-' ? -1 : 1;
        int ev = 0, ed = 0;
        while (text[r] >= '0' && text[r] <= '9' && ed < 6) { ev = ev * 10 + (text[r++] - '0'); ++ed; }
        if (ed) { ex = es * ev; q = r; }
    }
    const int p10 = ex - frac;
    double scale = 1.0;
    for (int i = 0; i < (p10 < 0 ? -p10 : p10) && i < 400; ++i) scale *= 10.0;
    out = sign * (p10 < 0 ? v / scale : v * scale);
    p = q;
    return true;
}

// Staged text in shared memory, for lines that end inside it.
struct MtxStaged {
    const char *s;
    __device__ __forceinline__ char operator[](uint32_t p) const { return s[p]; }
};

// One entry line from p on: ids and value; returns the error bits.
template <typename Text, typename Pos>
__device__ __forceinline__ uint32_t mtx_line(const Text &x, Pos p, uint64_t rows, uint64_t cols, int with_value,
                                             uint32_t &src, uint32_t &dst, float &val) {
    unsigned long long a = 0, b = 0;
    if (!mtx_uint(x, p, a) || !mtx_uint(x, p, b)) return 1u;  // a data line without two ids
    if (a < 1 || b < 1 || a > rows || b > cols || a > 0xFFFFFFFFull || b > 0xFFFFFFFFull) return 2u;
    src = (uint32_t)(a - 1);
    dst = (uint32_t)(b - 1);
    double w = 1.0;
    const bool bad = with_value && !mtx_real(x, p, w);
    val = (float)w;
    return bad ? 4u : 0u;
}

// The entries whose lines start in the tile, a thread per line; entry k of the
// text goes to place k.  Nothing is stored when the entries exceed cap; bad
// lines raise err all the same.  Lines are read from the staged text, byte by
// byte but from shared memory; the few that do not end in it, where they lie.
__global__ void __launch_bounds__(MTX_THREADS) k_mtx_parse(MtxText t, const unsigned long long *__restrict__ tile_off,
                                                           uint32_t ntiles, uint64_t cap, uint64_t rows, uint64_t cols,
                                                           int with_value, uint32_t *__restrict__ src,
                                                           uint32_t *__restrict__ dst, float *__restrict__ val,
                                                           uint32_t *err) {
    __shared__ __align__(16) char buf[MTX_TILE + MTX_AHEAD];
    __shared__ uint16_t start[MTX_TILE / 2 + 2];  // a line takes two bytes at least
    __shared__ uint32_t wt[33];
    __shared__ uint32_t closed;                   // one past the last newline staged
    if (threadIdx.x == 0) closed = 0;
    const int64_t g0 = t.origin + (int64_t)blockIdx.x * MTX_TILE, g = g0 + threadIdx.x * 16;
    const uint4 v = mtx_load16(t, g);
    const bool ahead = threadIdx.x < MTX_AHEAD / 16;
    const uint4 va = ahead ? mtx_load16(t, g + MTX_TILE) : make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4 *>(buf)[threadIdx.x] = v;
    if (ahead) reinterpret_cast<uint4 *>(buf)[MTX_THREADS + threadIdx.x] = va;
    const uint32_t m = mtx_starts(t, g, v, blockIdx.x == 0 && threadIdx.x == 0);
    uint32_t cnt;
    uint32_t at = cta_excl_scan<uint32_t, MTX_THREADS>(__popc(m), wt, cnt);
    if (m >> 16) start[at++] = (uint16_t)((int64_t)t.begin - g0);
    for (uint32_t r = m & 0xFFFFu; r; r &= r - 1) start[at++] = (uint16_t)(threadIdx.x * 16 + __ffs(r));
    const uint32_t nl = mtx_newlines(v), nla = mtx_newlines(va);
    uint32_t end = nl ? threadIdx.x * 16 + 32 - __clz(nl) : 0u;
    if (nla) end = MTX_TILE + threadIdx.x * 16 + 32 - __clz(nla);
    end = __reduce_max_sync(GV_FULL_MASK, end);
    if ((threadIdx.x & 31u) == 0) atomicMax(&closed, end);
    __syncthreads();
    const uint32_t staged = closed;
    const unsigned long long base = tile_off[blockIdx.x];
    const bool store = tile_off[ntiles] <= cap;
    uint32_t bad = 0;
    for (uint32_t i = threadIdx.x; i < cnt; i += MTX_THREADS) {
        uint32_t a = 0, b = 0;
        float w = 0.f;
        const uint32_t p = start[i];
        const uint32_t e = p < staged ? mtx_line(MtxStaged{buf}, p, rows, cols, with_value, a, b, w)
                                      : mtx_line(t, (uint64_t)(g0 + p), rows, cols, with_value, a, b, w);
        bad |= e;
        if (e || !store) continue;
        src[base + i] = a;
        dst[base + i] = b;
        if (val) val[base + i] = w;
    }
    if (bad) atomicOr(err, bad);
}

__global__ void k_mtx_ones(float *__restrict__ v, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) v[i] = 1.0f;
}

// The id of the allocation that holds p, which no other allocation of the
// process ever has; 0 when there is none (its context is gone).
uint64_t buffer_id(void *p) {
    using Query = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const Query query = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (Query)f;
    }();
    unsigned long long id = 0;
    return query && query(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, (CUdeviceptr)p) == CUDA_SUCCESS ? id : 0;
}

// Scratch of gv_mtx_parse, which has no graph to keep it: a cudaMalloc and
// cudaFree cost 0.6 ms a call, more than the parse.  Each host thread keeps
// one block of at most MTX_KEEP bytes (3 bytes per KB of text) and gives it
// back when it ends; the call ends with a synchronize, so the block is idle
// between calls whatever stream they name.  A device reset takes the block with
// it, and the address may come back as someone else's, so the block is used and
// freed only while its allocation has the id that it got (under 1 us a call).
constexpr size_t MTX_KEEP = 4u << 20;
struct MtxScratch {
    void *p = nullptr;
    size_t bytes = 0;
    uint64_t id = 0;
    int device = -1;
    void *get(size_t want) {
        int dev = -1;
        if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
        if (p && (bytes < want || device != dev || buffer_id(p) != id)) drop();
        if (!p) {
            if (cudaMalloc(&p, want) != cudaSuccess) {
                cudaGetLastError();
                p = nullptr;
                return nullptr;
            }
            bytes = want;
            device = dev;
            id = buffer_id(p);
        }
        return p;
    }
    void done() {
        if (bytes > MTX_KEEP || !id) drop();  // without an id nothing is kept
    }
    void drop() {
        if (p && buffer_id(p) == id) cudaFree(p);
        p = nullptr;
        bytes = 0;
        id = 0;
    }
    ~MtxScratch() { drop(); }
};
thread_local MtxScratch t_mtx;

// Header parse on the host: banner (field, symmetry), then the size line.
bool mtx_header(const char *t, uint64_t len, gv_mtx_info *info, uint64_t *data_begin) {
    std::memset(info, 0, sizeof(*info));
    uint64_t p = 0;
    bool have_banner = false;
    while (p < len) {
        uint64_t e = p;
        while (e < len && t[e] != '\n') ++e;
        std::string line(t + p, t + e);
        if (!line.empty() && line[0] == '%') {
            if (!have_banner && line.rfind("%%MatrixMarket", 0) == 0) {
                have_banner = true;
                info->pattern = line.find("pattern") != std::string::npos;
                info->symmetric = line.find("symmetric") != std::string::npos ||
                                  line.find("hermitian") != std::string::npos;
            }
        } else {
            unsigned long long r = 0, c = 0, z = 0;
            if (std::sscanf(line.c_str(), "%llu %llu %llu", &r, &c, &z) == 3) {
                info->rows = r;
                info->cols = c;
                info->entries = z;
                *data_begin = e < len ? e + 1 : len;
                return true;
            }
            bool blank = true;
            for (char ch : line) blank = blank && (ch == ' ' || ch == '\t' || ch == '\r');
            if (!blank) return false;
        }
        p = e + 1;
    }
    return false;
}

}  // namespace
}  // namespace gv

using namespace gv;

extern "C" gv_status gv_mtx_parse(const char *text, uint64_t len, int mem, gv_mtx_info *info, uint32_t *src,
                                  uint32_t *dst, float *values, uint64_t cap, uint64_t *count, void *stream) {
    if (!text || !info || !count) { set_error("null argument"); return GV_ERR_INVALID; }
    if (mem != GV_MEM_HOST && mem != GV_MEM_DEVICE) { set_error("bad mem flag"); return GV_ERR_INVALID; }
    cudaStream_t s = (cudaStream_t)stream;
    // header from the first bytes (host copy when the text is on the device):
    // 4 KB, and 1 MB when the size line does not end in them
    std::vector<char> head;
    uint64_t begin = 0;
    bool found = false;
    if (mem == GV_MEM_DEVICE) {
        for (uint64_t most : {1ull << 12, 1ull << 20}) {
            const uint64_t hlen = std::min<uint64_t>(len, most);
            head.resize(hlen);
            cudaError_t e = cudaMemcpyAsync(head.data(), text, hlen, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return cuda_status(e, "mtx header");
            found = mtx_header(head.data(), hlen, info, &begin);
            if (hlen == len || (found && begin > 0 && head[begin - 1] == '\n')) break;
        }
    } else {
        found = mtx_header(text, len, info, &begin);
    }
    if (!found) { set_error("no Matrix-Market size line"); return GV_ERR_INVALID; }
    if (info->rows == 0 || info->rows > 0xFFFFFFF0ull) { set_error("row count out of range"); return GV_ERR_INVALID; }
    *count = 0;
    if (!src) return GV_OK;  // header only
    if (!dst) { set_error("null argument"); return GV_ERR_INVALID; }
    if (begin >= len) return GV_OK;
    // device copy of the text (pinned staging is the caller's choice; pageable works)
    const char *dtext = text;
    std::vector<void *> owned;
    auto dalloc = [&](size_t bytes) -> void * {
        void *p = nullptr;
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        owned.push_back(p);
        return p;
    };
    auto release = [&]() {
        for (void *p : owned) cudaFree(p);
        owned.clear();
        t_mtx.done();
    };
    gv_status st = GV_OK;
    if (mem == GV_MEM_HOST) {
        char *t = (char *)dalloc(len);
        if (!t) { set_error("mtx text allocation failed"); return GV_ERR_NOMEM; }
        cudaError_t e = cudaMemcpyAsync(t, text, len, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) { release(); return cuda_status(e, "mtx text"); }
        dtext = t;
    }
    // Entry lines counted per tile, the counts scanned, then each tile parses
    // its lines to their places: the text is read twice and the outputs
    // written once, with no arrays per line in between.
    MtxText t{dtext, begin, len, (int64_t)begin - (int64_t)((uintptr_t)(dtext + begin) & 15u)};
    const uint64_t ntiles = ((uint64_t)((int64_t)len - t.origin) + MTX_TILE - 1) / MTX_TILE;
    if (ntiles >= 0x7FFFFFFFull) { release(); set_error("mtx text too long"); return GV_ERR_INVALID; }
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t o_off = al(ntiles * 4), o_tmp = o_off + al((ntiles + 1) * 8);
    const size_t o_err = o_tmp + al(scan_scratch_bytes(ntiles + 1));
    char *scratch = (char *)t_mtx.get(o_err + 256);
    if (!scratch) { release(); set_error("mtx scratch allocation failed"); return GV_ERR_NOMEM; }
    uint32_t *tile_cnt = (uint32_t *)scratch, *err = (uint32_t *)(scratch + o_err);
    unsigned long long *tile_off = (unsigned long long *)(scratch + o_off);
    const bool want_val = values && !info->pattern;
    cudaMemsetAsync(err, 0, 4, s);
    GV_LAUNCH(k_mtx_count, (unsigned)ntiles, MTX_THREADS, 0, s, t, tile_cnt);
    scan_exclusive_u32_to_u64(tile_cnt, tile_off, ntiles, tile_off + ntiles, scratch + o_tmp, s);
    unsigned long long nent = 0;
    cudaError_t e = cudaSuccess;
    // device arrays are written in place, host arrays through device staging
    uint32_t *osrc = src, *odst = dst;
    float *oval = want_val ? values : nullptr;
    if (mem == GV_MEM_HOST) {
        e = cudaMemcpyAsync(&nent, tile_off + ntiles, 8, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { release(); return cuda_status(e, "mtx lines"); }
        const size_t each = al(std::min<uint64_t>(nent, cap) * 4 + 16);
        char *o = (char *)dalloc(each * (want_val ? 3 : 2));
        if (!o) { release(); set_error("mtx output allocation failed"); return GV_ERR_NOMEM; }
        osrc = (uint32_t *)o;
        odst = (uint32_t *)(o + each);
        if (want_val) oval = (float *)(o + 2 * each);
    }
    GV_LAUNCH(k_mtx_parse, (unsigned)ntiles, MTX_THREADS, 0, s, t, (const unsigned long long *)tile_off,
              (uint32_t)ntiles, cap, info->rows, info->cols, want_val ? 1 : 0, osrc, odst, oval, err);
    uint32_t herr = 0;
    e = cudaMemcpyAsync(&nent, tile_off + ntiles, 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { release(); return cuda_status(e, "mtx parse"); }
    if (herr) {
        release();
        set_error(herr & 2u ? "mtx entry id out of range" : herr & 1u ? "mtx data line without two ids"
                                                                       : "mtx entry without a value");
        return GV_ERR_INVALID;
    }
    *count = nent;
    if (nent > cap) {
        release();
        set_error("mtx entries exceed the output capacity");
        return GV_ERR_CAPACITY;
    }
    if (mem == GV_MEM_HOST) {
        e = cudaMemcpyAsync(src, osrc, nent * 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, odst, nent * 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && want_val) e = cudaMemcpyAsync(values, oval, nent * 4, cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess && values && info->pattern) {  // pattern files: every value is 1
        if (mem == GV_MEM_HOST) {
            for (uint64_t i = 0; i < nent; ++i) values[i] = 1.0f;
        } else {
            GV_LAUNCH(k_mtx_ones, grid_for(nent, 256, 148 * 16), 256, 0, s, values, nent);
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    release();
    return cuda_status(e, "mtx out");
}

// ------------------------------------------------------------- snapshots
namespace {

struct SnapHeader {
    char magic[8];        // "GVSNAP\0\1"
    uint32_t version;     // 1
    uint32_t flags;       // bit 0 directed, bit 1 weighted
    uint32_t n;
    uint32_t block_size;
    uint64_t m;           // stored entries
    uint64_t checksum;    // FNV-1a 64 of the payload
    uint64_t reserved[3];
};
static_assert(sizeof(SnapHeader) == 64, "snapshot header is 64 bytes");
const char kSnapMagic[8] = {'G', 'V', 'S', 'N', 'A', 'P', 0, 1};

uint64_t fnv1a(uint64_t h, const void *data, size_t bytes) {
    const unsigned char *p = (const unsigned char *)data;
    for (size_t i = 0; i < bytes; ++i) {
        h ^= p[i];
        h *= 1099511628211ull;
    }
    return h;
}

}  // namespace

extern "C" gv_status gv_snapshot_save(gv_graph *g, const char *path) {
    if (!g || !path) { set_error("null argument"); return GV_ERR_INVALID; }
    uint32_t n = 0;
    uint64_t m = 0;
    gv_status st = gv_num_vertices(g, &n);
    if (st == GV_OK) st = gv_num_edges(g, &m);
    if (st != GV_OK) return st;
    const bool weighted = g->cfg.weighted != 0;
    std::vector<uint64_t> off((size_t)n + 1);
    std::vector<uint32_t> dst(std::max<uint64_t>(m, 1));
    std::vector<float> w(weighted ? std::max<uint64_t>(m, 1) : 0);
    st = gv_export_csr(g, off.data(), dst.data(), weighted ? w.data() : nullptr, m, GV_MEM_HOST, nullptr);
    if (st != GV_OK) return st;
    SnapHeader h{};
    std::memcpy(h.magic, kSnapMagic, 8);
    h.version = 1;
    h.flags = (g->cfg.directed ? 1u : 0u) | (weighted ? 2u : 0u);
    h.n = n;
    h.block_size = g->cfg.block_size;
    h.m = m;
    uint64_t c = 1469598103934665603ull;
    c = fnv1a(c, off.data(), off.size() * 8);
    c = fnv1a(c, dst.data(), m * 4);
    if (weighted) c = fnv1a(c, w.data(), m * 4);
    h.checksum = c;
    FILE *f = std::fopen(path, "wb");
    if (!f) { set_error(std::string("cannot open ") + path); return GV_ERR_INVALID; }
    bool ok = std::fwrite(&h, sizeof(h), 1, f) == 1;
    ok = ok && std::fwrite(off.data(), 8, off.size(), f) == off.size();
    ok = ok && (m == 0 || std::fwrite(dst.data(), 4, m, f) == m);
    ok = ok && (!weighted || m == 0 || std::fwrite(w.data(), 4, m, f) == m);
    ok = (std::fclose(f) == 0) && ok;
    if (!ok) { set_error(std::string("write failed: ") + path); return GV_ERR_INVALID; }
    return GV_OK;
}

extern "C" gv_status gv_snapshot_load(const char *path, const gv_config *base, gv_graph **out) {
    if (!path || !out) { set_error("null argument"); return GV_ERR_INVALID; }
    *out = nullptr;
    FILE *f = std::fopen(path, "rb");
    if (!f) { set_error(std::string("cannot open ") + path); return GV_ERR_INVALID; }
    SnapHeader h{};
    bool ok = std::fread(&h, sizeof(h), 1, f) == 1 && std::memcmp(h.magic, kSnapMagic, 8) == 0 && h.version == 1 &&
              h.n > 0;
    std::vector<uint64_t> off;
    std::vector<uint32_t> dst;
    std::vector<float> w;
    const bool weighted = (h.flags & 2u) != 0;
    if (ok) {
        off.resize((size_t)h.n + 1);
        dst.resize(std::max<uint64_t>(h.m, 1));
        if (weighted) w.resize(std::max<uint64_t>(h.m, 1));
        ok = std::fread(off.data(), 8, off.size(), f) == off.size();
        ok = ok && (h.m == 0 || std::fread(dst.data(), 4, h.m, f) == h.m);
        ok = ok && (!weighted || h.m == 0 || std::fread(w.data(), 4, h.m, f) == h.m);
    }
    std::fclose(f);
    if (!ok) { set_error(std::string("not a readable snapshot: ") + path); return GV_ERR_INVALID; }
    uint64_t c = 1469598103934665603ull;
    c = fnv1a(c, off.data(), off.size() * 8);
    c = fnv1a(c, dst.data(), h.m * 4);
    if (weighted) c = fnv1a(c, w.data(), h.m * 4);
    if (c != h.checksum || off[h.n] != h.m) { set_error("snapshot checksum mismatch"); return GV_ERR_INVALID; }
    for (uint64_t i = 0; i < h.m; ++i)
        if (dst[i] >= h.n) { set_error("snapshot entry out of range"); return GV_ERR_INVALID; }
    gv_config cfg;
    if (base) cfg = *base;
    else gv_config_init(&cfg, h.n);
    cfg.num_vertices = h.n;
    cfg.directed = h.flags & 1u;
    cfg.weighted = weighted ? 1 : 0;
    if (!base) cfg.block_size = h.block_size;
    if (cfg.max_batch_pairs < h.m) cfg.max_batch_pairs = h.m;
    gv_graph *g = nullptr;
    gv_status st = gv_create(&cfg, &g);
    if (st != GV_OK) return st;
    st = gv_bulk_build_csr(g, off.data(), dst.data(), weighted ? w.data() : nullptr, GV_MEM_HOST, nullptr);
    if (st == GV_OK) st = gv_synchronize(g, nullptr);
    if (st != GV_OK) {
        gv_destroy(g);
        return st;
    }
    *out = g;
    return GV_OK;
}

extern "C" gv_status gv_graph_from_mtx(const char *path, const gv_config *base, gv_graph **out) {
    if (!path || !out) { set_error("null argument"); return GV_ERR_INVALID; }
    *out = nullptr;
    FILE *f = std::fopen(path, "rb");
    if (!f) { set_error(std::string("cannot open ") + path); return GV_ERR_INVALID; }
    std::fseek(f, 0, SEEK_END);
    const long len = std::ftell(f);
    std::fseek(f, 0, SEEK_SET);
    std::vector<char> text(len > 0 ? (size_t)len : 1);
    const bool ok = len > 0 && std::fread(text.data(), 1, (size_t)len, f) == (size_t)len;
    std::fclose(f);
    if (!ok) { set_error(std::string("cannot read ") + path); return GV_ERR_INVALID; }
    gv_mtx_info info;
    uint64_t cnt = 0;
    gv_status st = gv_mtx_parse(text.data(), (uint64_t)len, GV_MEM_HOST, &info, nullptr, nullptr, nullptr, 0, &cnt, nullptr);
    if (st != GV_OK) return st;
    gv_config cfg;
    if (base) cfg = *base;
    else gv_config_init(&cfg, (uint32_t)info.rows);
    cfg.num_vertices = (uint32_t)info.rows;
    const uint64_t cap = std::max<uint64_t>(info.entries, 1) + 16;
    std::vector<uint32_t> src(cap), dst(cap);
    std::vector<float> val(cfg.weighted ? cap : 0);
    st = gv_mtx_parse(text.data(), (uint64_t)len, GV_MEM_HOST, &info, src.data(), dst.data(),
                      cfg.weighted ? val.data() : nullptr, cap, &cnt, nullptr);
    if (st != GV_OK) return st;
    if (cfg.max_batch_pairs < cnt) cfg.max_batch_pairs = cnt;
    gv_graph *g = nullptr;
    st = gv_create(&cfg, &g);
    if (st != GV_OK) return st;
    // an undirected store keeps both directions, as the reader symmetrises
    // for !DIRECTED (marketReader.cu:55-62)
    st = gv_insert_edges(g, src.data(), dst.data(), cfg.weighted ? val.data() : nullptr, cnt, GV_MEM_HOST, nullptr);
    if (st == GV_OK) st = gv_synchronize(g, nullptr);
    if (st != GV_OK) {
        gv_destroy(g);
        return st;
    }
    *out = g;
    return GV_OK;
}
