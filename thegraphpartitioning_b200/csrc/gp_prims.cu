// gp_prims.cu -- arena, prefix scans and the LSD radix sort.
//
// Scans reduce tiles of 256 threads x 8 items, then scan every tile from the
// sums of the tiles before it; few tiles are summed by each tile's own block
// (two launches), many by a kernel in between (three), and short arrays take
// one block and one launch.  The radix sort is a stable LSD sort of 64-bit keys
// with 32-bit payloads, 8-bit digits: per pass a tile histogram kernel, a
// kernel that scans each digit's tile counts (one block per digit), and a
// scatter kernel that adds the digits' bases and ranks items stably inside the
// tile with warp match/ballot and per-warp digit counters in shared memory.
// Sorts and weight scans take their length from device memory when the caller
// has it only there.
#define GP_TU_ID 1   // site ids of the bounds-checked build
#include "gp_common.cuh"

#include <algorithm>
#include <cstring>

namespace gp {

// ================================================================ arena
void* Arena::alloc(size_t bytes) {
    bytes = (bytes + 255) & ~(size_t)255;
    if (!chunks_.empty()) {
        for (size_t i = cur_; i < chunks_.size(); ++i) {
            Chunk& ch = chunks_[i];
            if (i > cur_) ch.off = 0;
            if (ch.off + bytes <= ch.size) {
                cur_ = i;
                void* p = ch.p + ch.off;
                ch.off += bytes;
                used_total_ += bytes;
                peak_total_ = std::max(peak_total_, used_total_);
                return p;
            }
        }
    }
    size_t last = chunks_.empty() ? 0 : chunks_.back().size;
    size_t sz = std::max<size_t>(bytes, std::max<size_t>(last * 2, (size_t)64 << 20));
    char* p = nullptr;
    cudaError_t e = cudaMalloc(&p, sz);
    if (e != cudaSuccess) {
        cudaGetLastError();
        sz = bytes;
        e = cudaMalloc(&p, sz);
        if (e != cudaSuccess) {
            cudaGetLastError();
            throw GpError(GP_ENOMEM, "device allocation of " + std::to_string(bytes) + " bytes failed");
        }
    }
    chunks_.push_back(Chunk{p, sz, bytes});
    cur_ = chunks_.size() - 1;
    used_total_ += bytes;
    peak_total_ = std::max(peak_total_, used_total_);
    return p;
}

void Arena::restore(const Mark& m) {
    if (chunks_.empty()) return;
    for (size_t i = m.chunk + 1; i < chunks_.size(); ++i) chunks_[i].off = 0;
    cur_ = m.chunk;
    chunks_[cur_].off = m.off;
    used_total_ = m.total;
}

void Arena::reset() {
    for (auto& ch : chunks_) ch.off = 0;
    cur_ = 0;
    used_total_ = 0;
}

void Arena::consolidate() {
    if (chunks_.size() <= 1) { reset(); peak_total_ = 0; return; }
    size_t want = 0;
    for (auto& ch : chunks_) want += ch.size;
    want = std::max(want, peak_total_);
    release();
    char* p = nullptr;
    if (cudaMalloc(&p, want) == cudaSuccess) chunks_.push_back(Chunk{p, want, 0});
    else cudaGetLastError();
    cur_ = 0; used_total_ = 0; peak_total_ = 0;
}

void Arena::release() {
    for (auto& ch : chunks_) cudaFree(ch.p);
    chunks_.clear();
    cur_ = 0; used_total_ = 0;
}

size_t Arena::capacity() const {
    size_t s = 0;
    for (auto& ch : chunks_) s += ch.size;
    return s;
}

// ================================================================ helpers
int64_t read_i64(Ctx& c, const int64_t* d) {
    GP_CUDA(cudaMemcpyAsync(c.h_pinned, d, sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
    c.sync();
    return c.h_pinned[0];
}

void memset_async(Ctx& c, void* p, int value, size_t bytes) {
    if (bytes) GP_CUDA(cudaMemsetAsync(p, value, bytes, c.s));
}

// ================================================================ scan
constexpr int SCAN_T = 256;
constexpr int SCAN_I = 8;
constexpr int SCAN_TILE = SCAN_T * SCAN_I;

// scan inputs: an array; the vertex weights of a list of vertices (1 without weights)
template <class T>
struct InArray {
    const T* p;
    __device__ __forceinline__ int64_t operator()(int64_t i) const { return (int64_t)p[i]; }
};
struct InRep {                 // 1 for the representative of a matched pair and for unmatched vertices
    const int32_t* match;
    __device__ __forceinline__ int64_t operator()(int64_t i) const {
        const int32_t u = match[i];
        return u < 0 || i < u ? 1 : 0;
    }
};
struct InListWeight {
    const int32_t* list;
    const int32_t* vw;
    __device__ __forceinline__ int64_t operator()(int64_t i) const { return vw ? (int64_t)vw[list[i]] : 1; }
};

template <class In>
__global__ void k_tile_reduce(In in, int64_t n, const int64_t* __restrict__ n_dev, int64_t* __restrict__ tile_sums) {
    __shared__ int64_t sh[33];
    if (n_dev) n = *n_dev;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_I; ++i) {
        int64_t idx = base + (int64_t)i * SCAN_T + threadIdx.x;
        if (idx < n) s += in(idx);
    }
    int64_t tot;
    block_excl_scan<int64_t>(s, sh, tot);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

// single block: exclusive scan of the tile sums, in place
__global__ void k_scan_small(int64_t* __restrict__ a, int64_t n) {
    __shared__ int64_t sh[33];
    int64_t carry = 0;
    for (int64_t base = 0; base < n; base += blockDim.x) {
        int64_t idx = base + threadIdx.x;
        int64_t x = idx < n ? a[idx] : 0;
        int64_t tot;
        int64_t e = block_excl_scan<int64_t>(x, sh, tot);
        if (idx < n) a[idx] = carry + e;
        carry += tot;
    }
}

// SUMMED: tile_offs holds the tiles' exclusive offsets; else their sums, and
// each block adds up those before it.  The last tile writes the total.
template <class In, bool SUMMED>
__global__ void k_tile_scan(In in, int64_t* __restrict__ out, int64_t n, const int64_t* __restrict__ n_dev,
                            const int64_t* __restrict__ tile_offs, int64_t* __restrict__ total) {
    __shared__ int64_t sh[33];
    if (n_dev) n = *n_dev;
    int64_t off;
    if (SUMMED) off = tile_offs[blockIdx.x];
    else {
        int64_t s = 0;
        for (int64_t t = threadIdx.x; t < blockIdx.x; t += SCAN_T) s += tile_offs[t];
        block_excl_scan<int64_t>(s, sh, off);
    }
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_I;
    int64_t v[SCAN_I];
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_I; ++i) {
        int64_t idx = base + i;
        v[i] = idx < n ? in(idx) : 0;
        s += v[i];
    }
    int64_t tot;
    int64_t e = block_excl_scan<int64_t>(s, sh, tot) + off;
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = off + tot;
#pragma unroll
    for (int i = 0; i < SCAN_I; ++i) {
        int64_t idx = base + i;
        if (idx < n) out[idx] = e;
        e += v[i];
    }
}

// short arrays: one block, one launch
constexpr int SCAN_ONE_T = 1024;
template <class In>
__global__ void __launch_bounds__(SCAN_ONE_T) k_scan_one(In in, int64_t* __restrict__ out, int64_t n,
                                                         const int64_t* __restrict__ n_dev, int64_t* __restrict__ total) {
    __shared__ int64_t sh[33];
    if (n_dev) n = *n_dev;
    int64_t carry = 0;
    for (int64_t base = 0; base < n; base += SCAN_ONE_T * SCAN_I) {
        const int64_t b = base + (int64_t)threadIdx.x * SCAN_I;
        int64_t v[SCAN_I];
        int64_t s = 0;
#pragma unroll
        for (int i = 0; i < SCAN_I; ++i) {
            v[i] = b + i < n ? in(b + i) : 0;
            s += v[i];
        }
        int64_t tot;
        int64_t e = carry + block_excl_scan<int64_t>(s, sh, tot);
#pragma unroll
        for (int i = 0; i < SCAN_I; ++i) {
            if (b + i < n) out[b + i] = e;
            e += v[i];
        }
        carry += tot;
    }
    if (total && threadIdx.x == 0) *total = carry;
}

// n: the length, or a bound on *n_dev
constexpr int64_t SCAN_ONE = 16384;      // one block up to here: two passes of 8192
constexpr int64_t SCAN_TWO_TILES = 2048; // a block adds up at most 8 sums per thread
template <class In>
static void scan_excl(Ctx& c, In in, int64_t* out, int64_t n, const int64_t* n_dev, int64_t* d_total) {
    if (n <= 0) {
        if (d_total) GP_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int64_t), c.s));
        return;
    }
    c.bytes += (int64_t)(2 * sizeof(int32_t) + sizeof(int64_t)) * n;
    if (n <= SCAN_ONE) {
        k_scan_one<In><<<1, SCAN_ONE_T, 0, c.s>>>(in, out, n, n_dev, d_total);
        GP_LAUNCHED(c);
        return;
    }
    auto m = c.tmp->save();
    const int64_t nt = (n + SCAN_TILE - 1) / SCAN_TILE;
    int64_t* sums = c.tmp_alloc<int64_t>(nt);
    k_tile_reduce<In><<<(unsigned)nt, SCAN_T, 0, c.s>>>(in, n, n_dev, sums);
    GP_LAUNCHED(c);
    if (nt <= SCAN_TWO_TILES) {
        k_tile_scan<In, false><<<(unsigned)nt, SCAN_T, 0, c.s>>>(in, out, n, n_dev, sums, d_total);
        GP_LAUNCHED(c);
    } else {
        k_scan_small<<<1, 1024, 0, c.s>>>(sums, nt);
        GP_LAUNCHED(c);
        k_tile_scan<In, true><<<(unsigned)nt, SCAN_T, 0, c.s>>>(in, out, n, n_dev, sums, d_total);
        GP_LAUNCHED(c);
    }
    c.tmp->restore(m);
}

void scan_excl_i32_to_i64(Ctx& c, const int32_t* in, int64_t* out, int64_t n, int64_t* d_total) {
    scan_excl(c, InArray<int32_t>{in}, out, n, nullptr, d_total);
}
void scan_excl_i64(Ctx& c, const int64_t* in, int64_t* out, int64_t n, int64_t* d_total) {
    scan_excl(c, InArray<int64_t>{in}, out, n, nullptr, d_total);
}
void scan_representatives(Ctx& c, const int32_t* match, int64_t* out, int64_t n) {
    scan_excl(c, InRep{match}, out, n, nullptr, nullptr);
}
void scan_list_weights(Ctx& c, const int32_t* list, const int32_t* vw, int64_t* out, int64_t n, const int64_t* n_dev,
                       int64_t* d_total) {
    scan_excl(c, InListWeight{list, vw}, out, n, n_dev, d_total);
}

// ================================================================ radix sort
constexpr int RS_T = 256;                 // threads per tile
constexpr int RS_I = 8;                   // items per thread
constexpr int RS_TILE = RS_T * RS_I;      // 2048 items
constexpr int RS_W = RS_T / 32;           // warps per tile
constexpr int RS_WITEMS = 32 * RS_I;      // items per warp (contiguous)

// digit-major counts: counts[d * ntiles + tile]
__global__ void k_rs_hist(const uint64_t* __restrict__ keys, int64_t n, const int64_t* __restrict__ n_dev, int shift,
                          int32_t* __restrict__ counts, int64_t ntiles) {
    __shared__ int32_t h[256];
    if (n_dev) n = *n_dev;
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RS_TILE;
#pragma unroll
    for (int i = 0; i < RS_I; ++i) {
        int64_t idx = base + (int64_t)i * RS_T + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 0xFF], 1);
    }
    __syncthreads();
    counts[(int64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// one block per digit: exclusive scan of its tile counts in place, its total apart
__global__ void __launch_bounds__(RS_T) k_rs_scan(int32_t* __restrict__ counts, int64_t ntiles,
                                                  int32_t* __restrict__ totals) {
    __shared__ int32_t sh[33];
    int32_t* row = counts + (int64_t)blockIdx.x * ntiles;
    int32_t carry = 0;
    for (int64_t base = 0; base < ntiles; base += RS_T) {
        const int64_t i = base + threadIdx.x;
        const int32_t x = i < ntiles ? row[i] : 0;
        int32_t tot;
        const int32_t e = block_excl_scan<int32_t>(x, sh, tot);
        if (i < ntiles) row[i] = carry + e;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(RS_T) k_rs_scatter(const uint64_t* __restrict__ kin, const int32_t* __restrict__ vin,
                             uint64_t* __restrict__ kout, int32_t* __restrict__ vout,
                             int64_t n, const int64_t* __restrict__ n_dev, int shift,
                             const int32_t* __restrict__ offs, const int32_t* __restrict__ totals, int64_t ntiles) {
    __shared__ int32_t wcnt[RS_W][256];
    __shared__ int32_t dbase[256];
    __shared__ int32_t sh[33];
    if (n_dev) n = *n_dev;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RS_W * 256; i += RS_T) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t wbase = (int64_t)blockIdx.x * RS_TILE + (int64_t)w * RS_WITEMS;
    uint64_t k[RS_I];
    int32_t v[RS_I];
    uint32_t dg[RS_I];
    const uint32_t lt = (1u << lane) - 1u;
    // pass A: per-warp digit counts
#pragma unroll
    for (int i = 0; i < RS_I; ++i) {
        int64_t idx = wbase + i * 32 + lane;
        bool ok = idx < n;
        k[i] = ok ? kin[idx] : 0;
        v[i] = ok ? vin[idx] : 0;
        dg[i] = ok ? (uint32_t)((k[i] >> shift) & 0xFF) : 256u;
        uint32_t peers = __match_any_sync(0xffffffffu, dg[i]);
        int leader = __ffs(peers) - 1;
        if (ok && lane == leader) wcnt[w][dg[i]] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // exclusive prefix over warps per digit, plus the global tile offset
    {
        int d = threadIdx.x;  // RS_T == 256 digits
        int32_t all;
        const int32_t first = block_excl_scan<int32_t>(totals[d], sh, all);   // the digit's base
        const int32_t off = first + offs[(int64_t)d * ntiles + blockIdx.x];
        int32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < RS_W; ++ww) {
            int32_t cnt = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += cnt;
        }
        dbase[d] = off;
        __syncthreads();
        // pass B: positions
#pragma unroll
        for (int i = 0; i < RS_I; ++i) {
            int64_t idx = wbase + i * 32 + lane;
            bool ok = idx < n;
            uint32_t peers = __match_any_sync(0xffffffffu, dg[i]);
            int leader = __ffs(peers) - 1;
            int32_t basecnt = ok ? wcnt[w][dg[i]] : 0;
            __syncwarp();
            if (ok) {
                const int64_t pos = (int64_t)dbase[dg[i]] + basecnt + __popc(peers & lt);
                if (GP_IN(pos, n)) {
                    kout[pos] = k[i];
                    vout[pos] = v[i];
                }
                if (lane == leader) wcnt[w][dg[i]] = basecnt + __popc(peers);
            }
            __syncwarp();
        }
    }
}

void radix_sort_pairs(Ctx& c, uint64_t* keys, int32_t* vals, uint64_t* keys_tmp, int32_t* vals_tmp,
                      int64_t n, int bits, const int64_t* n_dev) {
    if (n <= 1 || bits <= 0) return;
    if (n > INT32_MAX) throw GpError(GP_EINTERNAL, "radix sort of more than 2^31 - 1 items");
    auto m = c.tmp->save();
    const int64_t ntiles = (n + RS_TILE - 1) / RS_TILE;
    int32_t* counts = c.tmp_alloc<int32_t>(256 * ntiles);
    int32_t* totals = c.tmp_alloc<int32_t>(256);
    int passes = (bits + 7) / 8;
    uint64_t* ka = keys; int32_t* va = vals;
    uint64_t* kb = keys_tmp; int32_t* vb = vals_tmp;
    for (int p = 0; p < passes; ++p) {
        int shift = 8 * p;
        k_rs_hist<<<(unsigned)ntiles, RS_T, 0, c.s>>>(ka, n, n_dev, shift, counts, ntiles);
        GP_LAUNCHED(c);
        k_rs_scan<<<256, RS_T, 0, c.s>>>(counts, ntiles, totals);
        GP_LAUNCHED(c);
        k_rs_scatter<<<(unsigned)ntiles, RS_T, 0, c.s>>>(ka, va, kb, vb, n, n_dev, shift, counts, totals, ntiles);
        GP_LAUNCHED(c);
        c.bytes += n * (8 + 2 * 12);
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys) {
        GP_CUDA(cudaMemcpyAsync(keys, ka, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(vals, va, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, c.s));
    }
    c.tmp->restore(m);
}

}  // namespace gp
