// gp_coarsen.cu -- matching and contraction kernels of one coarsening level.
//
// Replaces matchVertices / rematchVertices / resetMatch / mapVertices /
// relabel_coarse_vertices_kernel / countUniqueEdges / prefix_sum /
// fillEdgeArrays / updateRowPtr (src/gpu_part.cu:55-250) and the host loop
// around them (src/gpu_part.cu:1003-1152).
//
// Layout: CSR with int64 row pointers, int32 column ids and int32 weights;
// a NULL weight array means unit weights (the input level only).  The matching
// takes rows by degree bucket: rows longer than heavy_deg in pieces of a CTA each
// (blocks [0, nitems) of a launch), rows of 17 entries and more a warp each, shorter
// ones a thread each (16 lanes each where they are few).  The contraction takes
// coarse rows by the length of their walk, in the tiers listed there.
#define GP_TU_ID 2   // site ids of the bounds-checked build
#include "gp_internal.cuh"

namespace gp {

// ---------------------------------------------------------------- degree buckets
// Control block of one level (device): what the host reads of it comes in one
// copy at the end of the level's contraction.
enum LevelCtl { C_BUCKETS = 0 /* 4: bucket and heavy counts */, C_MAXDEG = 4, C_MAXVW = 5, C_MC = 6, C_ERR = 7,
                C_LONG = 8 /* 6: long-row tiers */, C_NCTL = 16 };

// raise *out to the warp's largest x (the plain read keeps most warps from the atomic)
__device__ __forceinline__ void warp_max_to(int64_t x, int64_t* out) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { const int64_t y = __shfl_xor_sync(0xffffffffu, x, o); x = y > x ? y : x; }
    if ((threadIdx.x & 31) == 0 && x > *(volatile int64_t*)out)
        atomicMax((unsigned long long*)out, (unsigned long long)x);
}

// Lists in any order (each row is processed on its own).  Appends are
// aggregated per block (block_append), 4 rows per thread at a time on lists
// long enough for that to matter.
// Lists of under 256 K rows are appended one row per thread: there latency
// counts (9 us against 4 us a launch), not the counter.
constexpr int64_t kAppendMany = 262144;
__device__ __forceinline__ int degree_bucket(int64_t d, int32_t heavy_deg) {
    return d <= kShortDeg ? 0 : (d <= kTile32 ? 1 : (d <= heavy_deg ? 2 : 3));
}

template <int kAppendRows>
__global__ void k_buckets(const int64_t* __restrict__ rp, int64_t n, int32_t heavy_deg, int64_t heavy_cap,
                          int32_t* __restrict__ heavy,
                          int32_t* __restrict__ b0, int32_t* __restrict__ b1, int32_t* __restrict__ b2,
                          int64_t* __restrict__ count) {
    int32_t* const lists[4] = {b0, b1, b2, heavy};
    const int64_t caps[4] = {n, n, n, heavy_cap};
    const int64_t per = (int64_t)blockDim.x * kAppendRows;
    int64_t most = 0;
    for (int64_t base = blockIdx.x * per; base < n; base += gridDim.x * per) {
        int b[kAppendRows];
        int32_t vs[kAppendRows];
#pragma unroll
        for (int r = 0; r < kAppendRows; ++r) {
            const int64_t v = base + (int64_t)r * blockDim.x + threadIdx.x;
            vs[r] = (int32_t)v;
            const int64_t d = v < n ? rp[v + 1] - rp[v] : -1;
            b[r] = v < n ? degree_bucket(d, heavy_deg) : -1;
            most = d > most ? d : most;
        }
        block_append<4, kAppendRows>(b, vs, lists, caps, count);
    }
    warp_max_to(most, &count[C_MAXDEG]);
}

__global__ void k_heavy_bounds(const int64_t* __restrict__ rp, const int32_t* __restrict__ heavy, int64_t nh,
                               int64_t* __restrict__ out) {
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x) {
        out[2 * h] = rp[heavy[h]];
        out[2 * h + 1] = rp[heavy[h] + 1];
    }
}

// cost of light unit u (order: bucket 2, bucket 1, groups of 4 of bucket 0)
__global__ void k_unit_cost(const int64_t* __restrict__ rp, const int32_t* __restrict__ b0, int64_t n0,
                            const int32_t* __restrict__ b1, int64_t n1, const int32_t* __restrict__ b2, int64_t n2,
                            int64_t* __restrict__ cost) {
    const int64_t U0 = (n0 + 3) / 4, U = n2 + n1 + U0;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < U; u += (int64_t)gridDim.x * blockDim.x) {
        int64_t cst = u < n2 + n1 ? 32 : 8;
        if (u < n2) cst += rp[b2[u] + 1] - rp[b2[u]];
        else if (u < n2 + n1) cst += rp[b1[u - n2] + 1] - rp[b1[u - n2]];
        else {
            const int64_t g = u - n2 - n1;
            for (int i = 0; i < 4 && 4 * g + i < n0; ++i) cst += rp[b0[4 * g + i] + 1] - rp[b0[4 * g + i]];
        }
        cost[u] = cst;
    }
}

// enqueue the bucket lists of L (counts and the longest row into ctl), then take
// what the host read of ctl into L
static void buckets_begin(Ctx& c, Level& L, int64_t heavy_cap, int64_t* ctl) {
    L.heavy = c.keep_alloc<int32_t>(heavy_cap);
    for (int b = 0; b < 3; ++b) L.bucket[b] = c.keep_alloc<int32_t>(L.g.n);
    const int per = L.g.n >= kAppendMany ? 4 : 1;
    (per == 4 ? k_buckets<4> : k_buckets<1>)<<<grid_for(L.g.n, 256 * per), 256, 0, c.s>>>(
        L.g.rp, L.g.n, L.heavy_deg, heavy_cap, L.heavy, L.bucket[0], L.bucket[1], L.bucket[2], ctl);
    GP_LAUNCHED(c);
    c.bytes += 8 * (L.g.n + 1) + 4 * L.g.n;
}
static void buckets_end(Ctx& c, Level& L, const int64_t* h, bool units) {
    for (int b = 0; b < 3; ++b) L.nbucket[b] = h[C_BUCKETS + b];
    L.nheavy = h[C_BUCKETS + 3];
    L.max_deg = h[C_MAXDEG];
    auto mk = c.tmp->save();
    // items: heavy row h covers [rp[v], rp[v+1]) in pieces of at most item_len
    std::vector<int64_t> rb((size_t)std::max<int64_t>(L.nheavy, 1)), re((size_t)std::max<int64_t>(L.nheavy, 1));
    if (L.nheavy > 0) {
        // row bounds of the heavy rows
        int64_t* d_rb = c.tmp_alloc<int64_t>(2 * L.nheavy);
        k_heavy_bounds<<<grid_for(L.nheavy, 256), 256, 0, c.s>>>(L.g.rp, L.heavy, L.nheavy, d_rb);
        GP_LAUNCHED(c);
        std::vector<int64_t> hb((size_t)(2 * L.nheavy));
        GP_CUDA(cudaMemcpyAsync(hb.data(), d_rb, sizeof(int64_t) * 2 * L.nheavy, cudaMemcpyDeviceToHost, c.s));
        c.sync();
        c.tmp->restore(mk);
        for (int64_t h = 0; h < L.nheavy; ++h) { rb[h] = hb[2 * h]; re[h] = hb[2 * h + 1]; }
    }
    std::vector<int32_t> irow, rows_items((size_t)std::max<int64_t>(L.nheavy, 1)), rows_first((size_t)std::max<int64_t>(L.nheavy, 1));
    std::vector<int64_t> ib, ie;
    for (int64_t h = 0; h < L.nheavy; ++h) {
        rows_first[h] = (int32_t)irow.size();
        int32_t cnt = 0;
        for (int64_t b = rb[h]; b < re[h]; b += L.item_len) {
            irow.push_back((int32_t)h);
            ib.push_back(b);
            ie.push_back(std::min<int64_t>(b + L.item_len, re[h]));
            ++cnt;
        }
        rows_items[h] = cnt;
    }
    L.nitems = (int64_t)irow.size();
    if (units) {
        L.nunits = L.nbucket[2] + L.nbucket[1] + (L.nbucket[0] + 3) / 4;
        int64_t* cost = c.tmp_alloc<int64_t>(L.nunits + 1);
        L.unit_cost = c.keep_alloc<int64_t>(L.nunits + 1);
        k_unit_cost<<<grid_for(L.nunits, 256), 256, 0, c.s>>>(L.g.rp, L.bucket[0], L.nbucket[0], L.bucket[1],
                                                              L.nbucket[1], L.bucket[2], L.nbucket[2], cost);
        GP_LAUNCHED(c);
        scan_excl_i64(c, cost, L.unit_cost, L.nunits, L.unit_cost + L.nunits);
        c.tmp->restore(mk);
    }
    L.item_row = c.keep_alloc<int32_t>(L.nitems);
    L.item_beg = c.keep_alloc<int64_t>(L.nitems);
    L.item_end = c.keep_alloc<int64_t>(L.nitems);
    L.row_items = c.keep_alloc<int32_t>(L.nheavy);
    L.row_first = c.keep_alloc<int32_t>(L.nheavy);
    if (L.nitems > 0) {
        GP_CUDA(cudaMemcpyAsync(L.item_row, irow.data(), sizeof(int32_t) * L.nitems, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(L.item_beg, ib.data(), sizeof(int64_t) * L.nitems, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(L.item_end, ie.data(), sizeof(int64_t) * L.nitems, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(L.row_items, rows_items.data(), sizeof(int32_t) * L.nheavy, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(L.row_first, rows_first.data(), sizeof(int32_t) * L.nheavy, cudaMemcpyHostToDevice, c.s));
        c.sync();  // host vectors go out of scope
    }
}

__global__ void k_max_vw(int64_t n, const int32_t* __restrict__ vw, int64_t* __restrict__ out) {
    int64_t mx = 0;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        mx = vw[v] > mx ? vw[v] : mx;
    warp_max_to(mx, out);
}

void build_heavy(Ctx& c, Level& L, bool units) {
    auto mk = c.tmp->save();
    int64_t* ctl = c.tmp_alloc<int64_t>(C_NCTL);
    memset_async(c, ctl, 0, C_NCTL * sizeof(int64_t));
    buckets_begin(c, L, std::max<int64_t>(1, L.g.m / L.heavy_deg + 1), ctl);
    if (L.g.vw) {
        k_max_vw<<<grid_for(L.g.n, 256, c.sm_count * 4), 256, 0, c.s>>>(L.g.n, L.g.vw, ctl + C_MAXVW);
        GP_LAUNCHED(c);
    }
    GP_CUDA(cudaMemcpyAsync(c.h_pinned, ctl, C_NCTL * sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
    c.sync();
    int64_t h[C_NCTL];
    std::copy(c.h_pinned, c.h_pinned + C_NCTL, h);
    c.tmp->restore(mk);
    L.max_vw = L.g.vw ? h[C_MAXVW] : 1;
    buckets_end(c, L, h, units);
}

// ---------------------------------------------------------------- argmax helpers
// Larger key wins; equal keys: smaller id wins (ids compared unsigned so that
// -1, meaning "none", loses every tie).
__device__ __forceinline__ void argmax_merge(uint64_t& k, int32_t& id, uint64_t k2, int32_t i2) {
    if (k2 > k || (k2 == k && (uint32_t)i2 < (uint32_t)id)) { k = k2; id = i2; }
}
__device__ __forceinline__ void warp_argmax(uint64_t& k, int32_t& id) { group_argmax64(0xffffffffu, k, id); }
// the two best distinct neighbours (by argmax_merge's order; a neighbour
// listed twice counts with its larger key) among those offered so far
__device__ __forceinline__ bool key_before(uint64_t k2, int32_t i2, uint64_t k, int32_t i) {
    return k2 > k || (k2 == k && (uint32_t)i2 < (uint32_t)i);
}
__device__ __forceinline__ void top2_insert(uint64_t& k1, int32_t& i1, uint64_t& k2, int32_t& i2, uint64_t k,
                                            int32_t i) {
    if (i == i1) { if (k > k1) k1 = k; return; }
    if (i == i2) {
        if (k > k2) k2 = k;
        if (key_before(k2, i2, k1, i1)) { const uint64_t tk = k1; const int32_t ti = i1; k1 = k2; i1 = i2; k2 = tk; i2 = ti; }
        return;
    }
    if (key_before(k, i, k1, i1)) { k2 = k1; i2 = i1; k1 = k; i1 = i; }
    else if (key_before(k, i, k2, i2)) { k2 = k; i2 = i; }
}
// block-wide; result valid in thread 0
__device__ __forceinline__ void block_argmax(uint64_t& k, int32_t& id, uint64_t* sk, int32_t* sid) {
    warp_argmax(k, id);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) { sk[w] = k; sid[w] = id; }
    __syncthreads();
    if (w == 0) {
        k = lane < nw ? sk[lane] : 0;
        id = lane < nw ? sid[lane] : -1;
        warp_argmax(k, id);
    }
    __syncthreads();
}

// ---------------------------------------------------------------- matching
// MODE 0: proposal to the best eligible unmatched neighbour (handshake round).
// MODE 1: anchor = best neighbour over all neighbours (two-hop pairing).
// Work units: one row of buckets 1 and 2 per warp, two rows of bucket 0 per
// warp (k_match_short takes them when there are many), heavy rows one per CTA
// in blocks [0, nheavy).
struct MatchArgs {
    DGraph g;
    const int32_t* heavy;
    int64_t nheavy;
    const int32_t* item_row;   // heavy rows split into items (one CTA each)
    const int64_t* item_beg;
    const int64_t* item_end;
    const int32_t* row_items;
    const int32_t* row_first;
    int64_t nitems;
    uint64_t* ikey;            // per-item partial best
    int32_t* iid;
    int32_t* hdone;            // per heavy row: items finished (reset by the last)
    const int32_t* list[3];   // rows to process, by degree bucket
    int64_t nlist[3];         // their counts, or bounds on them when
    const int64_t* dlist;     // the counts are in device memory (nullptr: they are not)
    int split;                // list[0] is k_match_short's
    __device__ __forceinline__ int64_t count(int b) const { return dlist ? dlist[b] : nlist[b]; }
    const int32_t* match;
    int32_t* out;             // MODE 0: proposals
    uint32_t salt;
    int64_t maxvw;
    uint64_t* keys;           // MODE 1: (anchor << nbits | v)
    int64_t* nkeys;
    int nbits;
    const int32_t* prio;      // learned priorities per entry (nullptr: edge weights)
    int2* cand;               // MODE 0, rows of 33+ entries (one piece): the best eligible
    uint8_t* cmore;           // neighbours of the row's last scan (warp rows: the best; CTA rows:
                              // the two best) and whether it had more (nullptr: no cache)
    int32_t* anchor0;         // the same rows' best neighbour in round 0; with no weight check
                              // that is the two-hop anchor (MODE 1 reads it instead of scanning)
    const uint8_t* hdead;     // MODE 0: heavy rows left without an eligible neighbour (nullptr: none)
    int any_matched;          // MODE 0: 0 in the first round (no neighbour to look up in match[])
    int check_vw;             // MODE 0: 0 when no two vertices of the level can exceed maxvw
};

// high word of an entry's matching priority: learned score or edge weight
__device__ __forceinline__ int32_t key_word(const MatchArgs& A, int64_t e) {
    return A.prio ? A.prio[e] : (A.g.ew ? __ldcs(&A.g.ew[e]) : 1);
}

template <int MODE>
__device__ __forceinline__ bool match_ok(const MatchArgs& A, int64_t v, int32_t u, int64_t vwv) {
    if (u == (int32_t)v || !GP_IN(u, A.g.n)) return false;
    if (MODE == 0) {
        if (A.any_matched && A.match[u] != -1) return false;
        if (A.check_vw && vwv + (A.g.vw ? A.g.vw[u] : 1) > A.maxvw) return false;
    }
    return true;
}

template <int MODE>
__device__ __forceinline__ void match_emit(const MatchArgs& A, bool valid, int64_t v, int32_t best) {
    if (MODE == 0) {
        if (valid) A.out[v] = best;
        return;
    }
    const bool take = valid && best >= 0;
    const uint32_t m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd((unsigned long long*)A.nkeys, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    const int64_t idx = (int64_t)base + __popc(m & ((1u << lane) - 1u));
    if (take && GP_IN(idx, A.g.n)) A.keys[idx] = ((uint64_t)(uint32_t)best << A.nbits) | (uint64_t)v;
}

// bucket-1 rows: one warp, an entry per lane
template <int MODE>
__device__ __forceinline__ void match_lane(const MatchArgs& A, int64_t v) {
    const int lane = threadIdx.x & 31;
    const bool valid = A.match[v] == -1;  // else matched already (round 0 / anchors)
    uint64_t bk = 0;
    int32_t bid = -1;
    if (valid) {
        const int64_t e = A.g.rp[v] + lane;
        if (e < A.g.rp[v + 1]) {
            const int32_t u = __ldcs(&A.g.ci[e]);
            const int64_t vwv = A.g.vw ? A.g.vw[v] : 1;
            if (match_ok<MODE>(A, v, u, vwv)) {
                bk = edge_key(key_word(A, e), edge_hash(A.salt, (int32_t)v, u));
                bid = u;
            }
        }
    }
    warp_argmax(bk, bid);
    if (MODE == 0) {
        if (lane == 0) A.out[v] = valid ? bid : -1;
    } else {
        match_emit<MODE>(A, lane == 0 && valid, v, bid);
    }
}

// bucket-0 rows (at most 16 entries), few of them: 16 lanes per row, two rows
// per warp (v < 0: none), the best by butterfly shuffles
template <int MODE>
__device__ __forceinline__ void match_half(const MatchArgs& A, int64_t v) {
    const int tl = threadIdx.x & 15;
    const bool valid = v >= 0 && A.match[v] == -1;
    uint64_t bk = 0;
    int32_t bid = -1;
    if (valid) {
        const int64_t e = A.g.rp[v] + tl;
        if (e < A.g.rp[v + 1]) {
            const int32_t u = __ldcs(&A.g.ci[e]);
            const int64_t vwv = A.g.vw ? A.g.vw[v] : 1;
            if (match_ok<MODE>(A, v, u, vwv)) {
                bk = edge_key(key_word(A, e), edge_hash(A.salt, (int32_t)v, u));
                bid = u;
            }
        }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const uint64_t k2 = __shfl_xor_sync(0xffffffffu, bk, o);
        const int32_t i2 = __shfl_xor_sync(0xffffffffu, bid, o);
        argmax_merge(bk, bid, k2, i2);
    }
    if (MODE == 0) {
        if (tl == 0 && v >= 0) A.out[v] = valid ? bid : -1;
    } else {
        match_emit<MODE>(A, tl == 0 && valid, v, bid);
    }
}

// bucket-0 rows, many of them: one row per lane, every lane of the warp calls
// it; entries 4 at a time while any lane of the warp has some left, their
// match[] and weight gathers in flight together, the best kept in registers (no
// shuffles).  (All 16 at a time takes 80 registers: 351 -> 450 us for round 0 of
// the 256^3 grid's level 0.)
template <int MODE>
__device__ __forceinline__ int32_t match_short(const MatchArgs& A, int32_t v, int64_t beg, int len, int64_t vwv) {
    const int32_t* __restrict__ row = A.g.ci + beg;
    const int32_t* __restrict__ kw = A.prio ? A.prio + beg : (A.g.ew ? A.g.ew + beg : nullptr);
    uint64_t bk = 0;
    int32_t bid = -1;
#pragma unroll
    for (int c = 0; c < kShortDeg; c += 4) {
        if (!__any_sync(0xffffffffu, len > c)) break;
        int32_t u[4], w[4], mm[4], vv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) u[i] = c + i < len ? __ldg(row + c + i) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (u[i] == v || !GP_IN(u[i] < 0 ? 0 : u[i], A.g.n)) u[i] = -1;
            w[i] = (kw && u[i] >= 0) ? __ldg(kw + c + i) : 1;
            mm[i] = (MODE == 0 && A.any_matched && u[i] >= 0) ? A.match[u[i]] : -1;
            vv[i] = (MODE == 0 && A.check_vw && A.g.vw && u[i] >= 0) ? A.g.vw[u[i]] : 1;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (u[i] < 0) continue;
            if (MODE == 0 && (mm[i] != -1 || (A.check_vw && vwv + vv[i] > A.maxvw))) continue;
            argmax_merge(bk, bid, edge_key(w[i], edge_hash(A.salt, v, u[i])), u[i]);
        }
    }
    return bid;
}
// the rows of list[0], in their own launch (k_match_scan's longer rows run
// best at 40 registers): from kMatchSplit rows on.  256^3 grid, round 0:
// level 0 (16.8 M rows of 6 entries; 8 lanes each in one launch with the rest)
// 1317 -> 350 us, level 1 (9.1 M rows, two thirds of 9-10 entries; a warp each) 2111 -> 293 us
constexpr int64_t kMatchSplit = 24576;
template <int MODE>
__global__ void __launch_bounds__(256) k_match_short(MatchArgs A) {
    const int64_t n0 = A.count(0);
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n0;
         i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + (threadIdx.x & 31);
        const int32_t v = i < n0 ? A.list[0][i] : -1;
        const bool valid = v >= 0 && A.match[v] == -1;
        int64_t beg = 0, vwv = 1;
        int len = 0;
        if (valid) {
            beg = A.g.rp[v];
            len = (int)(A.g.rp[v + 1] - beg);
            if (MODE == 0 && A.check_vw && A.g.vw) vwv = A.g.vw[v];
        }
        const int32_t best = match_short<MODE>(A, v, beg, len, vwv);
        if (MODE == 0) {
            if (v >= 0) A.out[v] = valid ? best : -1;
        } else {
            match_emit<MODE>(A, valid, v, best);
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(256, 6) k_match_scan(MatchArgs A) {
    __shared__ uint64_t sk[32];
    __shared__ int32_t sid[32];
    const int lane = threadIdx.x & 31;
    if ((int64_t)blockIdx.x < A.nitems) {
        // one piece of a long row per CTA; the last piece of a row reduces
        // the partial bests of all its pieces in item order
        const int32_t h = A.item_row[blockIdx.x];
        const int64_t v = A.heavy[h];
        if (A.match[v] != -1 || (A.hdead && A.hdead[h])) { if (MODE == 0 && threadIdx.x == 0) A.out[v] = -1; return; }
        const int nit = A.row_items[h];
        if (MODE == 1 && A.anchor0 && nit == 1) {
            if (threadIdx.x < 32) match_emit<MODE>(A, threadIdx.x == 0, v, A.anchor0[v]);
            return;
        }
        // a row in one piece keeps its two best eligible neighbours (as the warp rows do)
        const bool cached = MODE == 0 && A.cand && nit == 1;
        if (cached && A.any_matched) {
            const int2 cc = A.cand[v];
            const int32_t m1 = cc.x >= 0 ? A.match[cc.x] : 0, m2 = cc.y >= 0 ? A.match[cc.y] : 0;
            int32_t r = -2;
            if (cc.x >= 0 && m1 == -1) r = cc.x;
            else if (cc.y >= 0 && m2 == -1) r = cc.y;
            else if (!A.cmore[v]) r = -1;
            if (r != -2) { if (threadIdx.x == 0) A.out[v] = r; return; }
        }
        const int64_t vwv = A.g.vw ? A.g.vw[v] : 1;
        uint64_t bk = 0; int32_t bid = -1;
        uint64_t k2 = 0; int32_t i2 = -1, cnt = 0;
        const int64_t beg = A.item_beg[blockIdx.x], end = A.item_end[blockIdx.x];
        const int32_t* kw = A.prio ? A.prio : A.g.ew;
        const bool v4 = aligned16(A.g.ci) && aligned16(kw);
        for (int64_t base = beg & ~(int64_t)3; base < end; base += 4 * (int64_t)blockDim.x) {
            int32_t uu[4], ww[4];
            const int64_t e4 = base + 4 * threadIdx.x;
            ld4_row(A.g.ci, e4, beg, end, v4, -1, uu);
            if (kw) ld4_row(kw, e4, beg, end, v4, 0, ww);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (uu[c] < 0 || !match_ok<MODE>(A, v, uu[c], vwv)) continue;
                const uint64_t key = edge_key(kw ? ww[c] : 1, edge_hash(A.salt, (int32_t)v, uu[c]));
                if (cached) { top2_insert(bk, bid, k2, i2, key, uu[c]); ++cnt; }
                else argmax_merge(bk, bid, key, uu[c]);
            }
        }
        if (cached) {
            __shared__ int32_t s_best, s_cnt;
            const uint64_t k1 = bk;
            const int32_t i1 = bid;
            block_argmax(bk, bid, sk, sid);
            if (threadIdx.x == 0) { s_best = bid; s_cnt = 0; }
            __syncthreads();
            uint64_t ks = i1 == s_best ? k2 : k1;
            int32_t is = i1 == s_best ? i2 : i1;
            block_argmax(ks, is, sk, sid);
            const int32_t wc = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)cnt);
            if (lane == 0 && wc) atomicAdd(&s_cnt, wc);
            __syncthreads();
            if (threadIdx.x == 0) {
                A.cand[v] = make_int2(s_best, ks ? is : -1);
                A.cmore[v] = s_cnt > 2 ? 1 : 0;
                if (!A.any_matched && A.anchor0) A.anchor0[v] = s_best;
                A.out[v] = s_best;
            }
            return;
        }
        block_argmax(bk, bid, sk, sid);
        __shared__ int s_last;
        if (threadIdx.x == 0) {
            s_last = 1;
            if (nit > 1) {
                A.ikey[blockIdx.x] = bk;
                A.iid[blockIdx.x] = bid;
                __threadfence();
                s_last = atomicAdd(&A.hdone[h], 1) == nit - 1;
                if (s_last) {
                    __threadfence();
                    bk = 0; bid = -1;
                    const int32_t f = A.row_first[h];
                    for (int i = 0; i < nit; ++i)
                        argmax_merge(bk, bid, __ldcg((const unsigned long long*)&A.ikey[f + i]), __ldcg(&A.iid[f + i]));
                    A.hdone[h] = 0;
                }
            }
        }
        __syncthreads();
        if (s_last && threadIdx.x < 32) match_emit<MODE>(A, threadIdx.x == 0, v, bid);
        return;
    }
    const int64_t wid = ((int64_t)(blockIdx.x - A.nitems) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)(gridDim.x - A.nitems) * blockDim.x) >> 5;
    const int64_t n0 = A.split ? 0 : A.count(0);
    const int64_t U0 = (n0 + 1) / 2, U1 = A.count(1), U2 = A.count(2);
    for (int64_t u = wid; u < U0 + U1 + U2; u += nw) {
        if (u < U0) {
            const int64_t i = u * 2 + (lane >> 4);
            match_half<MODE>(A, i < n0 ? A.list[0][i] : -1);
        } else if (u < U0 + U1) {
            match_lane<MODE>(A, A.list[1][u - U0]);
        } else {
            const int64_t v = A.list[2][u - U0 - U1];
            const bool valid = A.match[v] == -1;
            uint64_t bk = 0; int32_t bid = -1;
            bool scan = valid;
            if (MODE == 1 && valid && A.anchor0) { bid = A.anchor0[v]; scan = false; }
            if (MODE == 0 && valid && A.cand && A.any_matched) {
                // neighbours only ever become matched, so the row's cached best
                // eligible neighbour, if still unmatched, is its best eligible
                // neighbour; with it matched and no other eligible entry, none
                const int2 cc = A.cand[v];
                const int32_t m1 = cc.x >= 0 ? A.match[cc.x] : 0, m2 = cc.y >= 0 ? A.match[cc.y] : 0;
                if (cc.x >= 0 && m1 == -1) { bid = cc.x; scan = false; }
                else if (cc.y >= 0 && m2 == -1) { bid = cc.y; scan = false; }
                else if (!A.cmore[v]) { bid = -1; scan = false; }
            }
            int32_t cnt = 0;   // eligible entries
            if (scan) {
                const int64_t vwv = A.g.vw ? A.g.vw[v] : 1;
                const int64_t beg = A.g.rp[v], end = A.g.rp[v + 1];
                // 128 entries per sweep, four consecutive ones per lane (16-byte loads)
                const int32_t* kw = A.prio ? A.prio : A.g.ew;
                const bool v4 = aligned16(A.g.ci) && aligned16(kw);
                for (int64_t base = beg & ~(int64_t)3; base < end; base += 128) {
                    int32_t uu[4], ww[4], mm[4], vv[4];
                    const int64_t e4 = base + 4 * lane;
                    ld4_row(A.g.ci, e4, beg, end, v4, -1, uu);
                    if (kw) ld4_row(kw, e4, beg, end, v4, 0, ww);
                    else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) ww[c] = 1;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const bool ok = uu[c] >= 0 && GP_IN(uu[c], A.g.n);
                        if (!ok) uu[c] = -1;
                        mm[c] = (MODE == 0 && A.any_matched && ok) ? A.match[uu[c]] : -1;
                        vv[c] = (MODE == 0 && A.check_vw && ok && A.g.vw) ? A.g.vw[uu[c]] : 1;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int32_t x = uu[c];
                        if (x < 0 || x == (int32_t)v) continue;
                        if (MODE == 0 && (mm[c] != -1 || (A.check_vw && vwv + vv[c] > A.maxvw))) continue;
                        const uint64_t key = edge_key(ww[c], edge_hash(A.salt, (int32_t)v, x));
                        argmax_merge(bk, bid, key, x);
                        if (MODE == 0 && A.cand) ++cnt;
                    }
                }
                warp_argmax(bk, bid);
                if (MODE == 0 && A.cand) {
                    // warp rows keep the best only (a second candidate costs more in
                    // round 0 than the rescans it saves)
                    const int32_t tot = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)cnt);
                    if (lane == 0) {
                        A.cand[v] = make_int2(bid, -1);
                        A.cmore[v] = tot > 1 ? 1 : 0;
                        if (!A.any_matched && A.anchor0) A.anchor0[v] = bid;
                    }
                }
            }
            if (MODE == 0) { if (lane == 0) A.out[v] = valid ? bid : -1; }
            else match_emit<MODE>(A, lane == 0 && valid, v, bid);
        }
    }
}

// Mutual proposals become pairs; vertices left unmatched go to the next
// round's worklists, bucketed by degree (any order: each vertex's proposal is
// its own).  A vertex that proposed nobody has no unmatched neighbour within
// the weight cap, and never will (vertices only become matched), so it leaves
// the worklists; a heavy one is flagged in hdead instead (heavy vertices are
// not listed: their CTAs check match[] and hdead[] directly).  next_n[3]
// counts the heavy vertices still live.
template <int kAppendRows>
__global__ void k_handshake(const int64_t* __restrict__ rp, int64_t n, int32_t heavy_deg, const int32_t* l0,
                            const int32_t* l1,
                            const int32_t* l2, int64_t n0, int64_t n1, int64_t n2,
                            const int64_t* __restrict__ dlist, const int32_t* __restrict__ heavy,
                            int64_t nheavy,
                            const int32_t* __restrict__ prop, int32_t* __restrict__ match, int64_t* __restrict__ pairs,
                            int32_t* nl0, int32_t* nl1, int32_t* nl2, int64_t* next_n, uint8_t* __restrict__ hdead) {
    if (dlist) { n0 = dlist[0]; n1 = dlist[1]; n2 = dlist[2]; }
    int64_t local = 0, live = 0;
    const int64_t total = n0 + n1 + n2 + nheavy;
    int32_t* const lists[3] = {nl0, nl1, nl2};
    const int64_t caps[3] = {n, n, n};
    const int64_t per = (int64_t)blockDim.x * kAppendRows;
    for (int64_t base = blockIdx.x * per; base < total; base += gridDim.x * per) {
        int b[kAppendRows];
        int32_t vs[kAppendRows];
#pragma unroll
        for (int r = 0; r < kAppendRows; ++r) {
            const int64_t i = base + (int64_t)r * blockDim.x + threadIdx.x;
            int64_t v = -1;
            if (i < n0) v = l0[i];
            else if (i < n0 + n1) v = l1[i - n0];
            else if (i < n0 + n1 + n2) v = l2[i - n0 - n1];
            else if (i < total) v = heavy[i - n0 - n1 - n2];
            const bool is_heavy = i >= n0 + n1 + n2;
            b[r] = -1;
            vs[r] = (int32_t)v;
            if (v >= 0 && match[v] == -1 && !(is_heavy && hdead[i - n0 - n1 - n2])) {
                const int32_t u = prop[v];
                if (u >= 0 && GP_IN(u, n) && prop[u] == (int32_t)v) {
                    match[v] = u;
                    if (v < u) ++local;
                } else if (u < 0) {
                    if (is_heavy) hdead[i - n0 - n1 - n2] = 1;
                } else if (is_heavy) {
                    ++live;
                } else {
                    b[r] = degree_bucket(rp[v + 1] - rp[v], heavy_deg);
                }
            }
        }
        block_append<3, kAppendRows>(b, vs, lists, caps, next_n);
    }
    if (live) atomicAdd((unsigned long long*)&next_n[3], (unsigned long long)live);
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd((unsigned long long*)pairs, (unsigned long long)local);
}

// sorted (anchor << nbits | v) keys: pair ranks (0,1), (2,3), ... of each anchor group
__global__ void k_twohop_pair(const uint64_t* __restrict__ keys, const int64_t* __restrict__ cnt_dev, int64_t n, int nbits,
                              const int32_t* __restrict__ vw,
                              int64_t maxvw, int32_t* __restrict__ match, int64_t* __restrict__ pairs) {
    int64_t local = 0;
    const int64_t cnt = *cnt_dev;
    const uint64_t lowmask = (1ull << nbits) - 1;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t a = keys[i] >> nbits;
        // first index of this anchor group (lower bound)
        int64_t lo = 0, hi = i;
        while (lo < hi) {
            int64_t mid = (lo + hi) >> 1;
            if ((keys[mid] >> nbits) < a) lo = mid + 1; else hi = mid;
        }
        if (((i - lo) & 1) || i + 1 >= cnt || (keys[i + 1] >> nbits) != a) continue;
        const int32_t x = (int32_t)(keys[i] & lowmask), y = (int32_t)(keys[i + 1] & lowmask);
        if (!GP_IN(x, n) || !GP_IN(y, n)) continue;
        const int64_t wx = vw ? vw[x] : 1, wy = vw ? vw[y] : 1;
        if (wx + wy <= maxvw) { match[x] = y; match[y] = x; ++local; }
    }
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd((unsigned long long*)pairs, (unsigned long long)local);
}

static int bits_for(int64_t x) {  // bits to represent values in [0, x)
    int b = 1;
    while ((1ll << b) < x) ++b;
    return b;
}

// one matching scan over A's lists: the short rows apart when there are many
template <int MODE>
static void match_scan(Ctx& c, const MatchArgs& A) {
    const int64_t units = (A.split ? 0 : (A.nlist[0] + 1) / 2) + A.nlist[1] + A.nlist[2];
    if (A.split) {
        k_match_short<MODE><<<grid_for(A.nlist[0], 256, c.sm_count * c.ctas_per_sm), 256, 0, c.s>>>(A);
        GP_LAUNCHED(c);
    }
    if (!A.split || units + A.nitems > 0) {
        const int grid = (int)A.nitems + grid_for(units * 32, 256, c.sm_count * c.ctas_per_sm);
        k_match_scan<MODE><<<grid, 256, 0, c.s>>>(A);
        GP_LAUNCHED(c);
    }
}

int64_t match_level(Ctx& c, const Level& L, int level, const Params& P, int32_t* match, int* rounds_out,
                    const int32_t* prio) {
    const DGraph& g = L.g;
    const uint32_t salt = edge_salt(P.seed, level);
    auto mk = c.tmp->save();
    int32_t* prop = c.tmp_alloc<int32_t>(g.n);
    int32_t* wl[2][3];
    for (int s2 = 0; s2 < 2; ++s2)
        for (int b = 0; b < 3; ++b) wl[s2][b] = c.tmp_alloc<int32_t>(std::max<int64_t>(L.nbucket[b], 1));
    // counters of a batch of rounds: pairs, the next lists' three counts, live heavy rows
    constexpr int kBatch = 4, kCnt = 8;
    int64_t* d_cnt = c.tmp_alloc<int64_t>(kBatch * kCnt);
    GP_CUDA(cudaMemsetAsync(match, 0xff, sizeof(int32_t) * g.n, c.s));
    MatchArgs A;
    A.g = g; A.heavy = L.heavy; A.nheavy = L.nheavy; A.match = match; A.out = prop; A.salt = salt;
    A.item_row = L.item_row; A.item_beg = L.item_beg; A.item_end = L.item_end; A.row_items = L.row_items;
    A.row_first = L.row_first; A.nitems = L.nitems;
    A.ikey = c.tmp_alloc<uint64_t>(std::max<int64_t>(L.nitems, 1));
    A.iid = c.tmp_alloc<int32_t>(std::max<int64_t>(L.nitems, 1));
    A.hdone = c.tmp_alloc<int32_t>(std::max<int64_t>(L.nheavy, 1));
    memset_async(c, A.hdone, 0, sizeof(int32_t) * std::max<int64_t>(L.nheavy, 1));
    A.maxvw = P.maxvw; A.keys = nullptr; A.nkeys = nullptr; A.nbits = 0; A.prio = prio;
    // rows of 33+ entries keep their two best eligible neighbours between rounds (written by round 0)
    A.cand = c.tmp_alloc<int2>(g.n);
    A.cmore = c.tmp_alloc<uint8_t>(g.n);
    A.anchor0 = c.tmp_alloc<int32_t>(g.n);
    // weight cap: skip the per-neighbour weight check when the two heaviest
    // vertices of the level together stay within maxvw
    A.check_vw = 2 * L.max_vw > P.maxvw ? 1 : 0;
    uint8_t* hdead = c.tmp_alloc<uint8_t>(std::max<int64_t>(L.nheavy, 1));
    memset_async(c, hdead, 0, std::max<int64_t>(L.nheavy, 1));
    A.hdead = hdead;
    for (int b = 0; b < 3; ++b) { A.list[b] = L.bucket[b]; A.nlist[b] = L.nbucket[b]; }
    A.dlist = nullptr;
    A.split = L.nbucket[0] >= kMatchSplit ? 1 : 0;
    int64_t pairs = 0;
    int rounds = 0;
    bool anchors_ready = false;   // round 0 ran and wrote anchor0
    const int64_t tot0 = A.nlist[0] + A.nlist[1] + A.nlist[2] + L.nheavy;
    // Rounds are enqueued four at a time, each taking its lists' counts from
    // device memory (the level's counts bound them), and read together.  A round
    // that adds no pair ends the matching: the rounds after it add none either,
    // since nothing they look at has changed.
    bool done = tot0 == 0;
    if (done && P.o.match_rounds > 0) rounds = 1;
    int64_t left = tot0;
    for (int r0 = 0; r0 < P.o.match_rounds && !done; r0 += kBatch) {
        const int nr = std::min(kBatch, P.o.match_rounds - r0);
        memset_async(c, d_cnt, 0, kBatch * kCnt * sizeof(int64_t));
        for (int i = 0; i < nr; ++i) {
            const int r = r0 + i;
            int64_t* cnt = d_cnt + i * kCnt;
            A.any_matched = r > 0 ? 1 : 0;
            match_scan<0>(c, A);
            anchors_ready = true;
            int32_t** nxt = wl[r & 1];
            const int per = tot0 >= kAppendMany ? 4 : 1;
            (per == 4 ? k_handshake<4> : k_handshake<1>)<<<grid_for(tot0, 256 * per), 256, 0, c.s>>>(
                g.rp, g.n, L.heavy_deg, A.list[0], A.list[1], A.list[2], A.nlist[0], A.nlist[1], A.nlist[2], A.dlist,
                L.heavy, L.nheavy, prop, match, cnt, nxt[0], nxt[1], nxt[2], cnt + 1, hdead);
            GP_LAUNCHED(c);
            for (int b = 0; b < 3; ++b) A.list[b] = nxt[b];
            A.dlist = cnt + 1;
        }
        GP_CUDA(cudaMemcpyAsync(c.h_pinned, d_cnt, kBatch * kCnt * sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
        c.sync();
        for (int i = 0; i < nr && !done; ++i) {
            const int64_t* h = c.h_pinned + i * kCnt;
            const int64_t share = g.n ? (left * 1000) / g.n : 0;
            c.bytes += (L.scan_bytes() + 4 * g.m) * share / 1000 + 16 * left;
            rounds = r0 + i + 1;
            pairs += h[0];
            left = h[1] + h[2] + h[3] + L.nheavy;
            if (h[0] == 0) done = true;
        }
        if (r0 + kBatch < P.o.match_rounds) {   // the counters are cleared: the counts move to the host
            for (int b = 0; b < 3; ++b) A.nlist[b] = c.h_pinned[(nr - 1) * kCnt + 1 + b];
            A.dlist = nullptr;
            A.split = A.nlist[0] >= kMatchSplit ? 1 : 0;
        }
    }
    if (P.o.two_hop > 0 && 4 * (g.n - pairs) > 3 * g.n) {
        const int nb = bits_for(g.n);
        uint64_t* keys = c.tmp_alloc<uint64_t>(g.n);
        uint64_t* keys2 = c.tmp_alloc<uint64_t>(g.n);
        int32_t* vals = c.tmp_alloc<int32_t>(g.n);
        int32_t* vals2 = c.tmp_alloc<int32_t>(g.n);
        memset_async(c, d_cnt, 0, 2 * sizeof(int64_t));
        MatchArgs B2 = A;
        B2.dlist = nullptr;
        B2.split = L.nbucket[0] >= kMatchSplit ? 1 : 0;
        B2.hdead = nullptr;   // anchors: the top neighbour over all neighbours
        B2.cand = nullptr; B2.cmore = nullptr;
        // round 0 saw every neighbour but v itself when no pair can exceed the weight cap
        if (A.check_vw || !anchors_ready) B2.anchor0 = nullptr;
        B2.any_matched = 1;
        for (int b = 0; b < 3; ++b) { B2.list[b] = L.bucket[b]; B2.nlist[b] = L.nbucket[b]; }
        B2.out = nullptr; B2.keys = keys; B2.nkeys = d_cnt + 1; B2.nbits = nb;
        match_scan<1>(c, B2);
        c.bytes += L.scan_bytes() + 4 * g.n;
        // at most the unmatched vertices have an anchor; vals is payload nobody reads
        const int64_t most = g.n - 2 * pairs;
        if (most > 1) {
            radix_sort_pairs(c, keys, vals, keys2, vals2, most, 2 * nb, d_cnt + 1);
            k_twohop_pair<<<grid_for(most, 256), 256, 0, c.s>>>(keys, d_cnt + 1, g.n, nb, g.vw, P.maxvw, match, d_cnt);
            GP_LAUNCHED(c);
            c.bytes += 24 * most;
            pairs += read_i64(c, d_cnt);
        }
    }
    c.tmp->restore(mk);
    if (rounds_out) *rounds_out = rounds;
    return pairs;
}

// ---------------------------------------------------------------- contraction
// cmap for every fine vertex; members, weight and row-length bound per coarse vertex
__global__ void k_cmap(DGraph g, const int32_t* __restrict__ match, const int64_t* __restrict__ cid,
                       int32_t* __restrict__ cmap, int32_t* __restrict__ mem, int32_t* __restrict__ cvw,
                       int64_t* __restrict__ cdeg, int64_t* __restrict__ max_vw) {
    int64_t most = 0;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = match[v];
        const bool rep = (u < 0 || v < u);
        const int64_t r = rep ? v : u;
        if (!GP_IN(r, g.n)) continue;
        const int32_t cc = (int32_t)cid[r];
        cmap[v] = cc;
        if (rep) {
            mem[2 * (int64_t)cc] = (int32_t)v;
            mem[2 * (int64_t)cc + 1] = u;
            int64_t w = g.vw ? g.vw[v] : 1;
            int64_t d = g.rp[v + 1] - g.rp[v];
            if (u >= 0) { w += g.vw ? g.vw[u] : 1; d += g.rp[u + 1] - g.rp[u]; }
            cvw[cc] = (int32_t)w;
            cdeg[cc] = d;
            most = w > most ? w : most;
        }
    }
    warp_max_to(most, max_vw);
}

// ---- row dedup in first-occurrence order
// Coarse row c walks N(a) then N(b) (a = representative, b = partner) in CSR
// order; position j in that walk.  Every coarse neighbour is kept once, at
// the rank of its first position, with the weights of all its positions
// summed; c itself is dropped.
//
// Tiers S to C2 read the walk straight from the fine CSR, mapping each
// column id through cmap as they go, and read it once.  Tier D reads its rows
// three times, so k_fill_walk_d first writes those rows, mapped, into a walk
// layout (row c at off[c]).  Every tier writes its unique entries at off[c]
// (a bound on the row) and k_contract_copy packs them.  Tiers by row length d:
//   S  d <= 32         one thread, 16 or 32 entries in registers
//   A  d <= 128        one warp, 256-slot table in shared memory
//   A2 d <= 256        one warp, 512-slot table
//   B  d <= 512        one warp, 1024-slot table (11 KB per warp: 20 warps per SM)
//   C1 d <= 2048       one CTA of 256 threads, two-phase (first position kept by
//                      an atomic minimum), 4096-slot table on chip (36 KB, 52 with
//                      64-bit slots: four CTAs per SM)
//   C  d <= 4096       the same with 512 threads and an 8192-slot table (72 KB, 104
//                      with 64-bit slots: two CTAs per SM)
//   C2 d <= 12288      the same with 1024 threads and a 16384-slot table (152 KB, 216
//                      with 64-bit slots: one CTA per SM; load factor at most 3/4)
//   C3 d <= 65536      one 1024-thread CTA, the C2 table in P = 2..8 passes: pass p
//                      dedups the keys whose pass hash is p, first positions are
//                      marked in a shared-memory bitmap of the whole walk
//   D  longer          pieces of 16K entries, one CTA each, table in global memory
// A and B insert 32 entries at a time in walk order (match_any leaders), so
// new neighbours get consecutive ranks; C and D rank first positions with one
// block scan over per-thread contiguous segments.  The on-chip tables are
// cleared once per CTA and afterwards only in the slots a row used.
constexpr int TA_ROW = 128, TA_SLOTS = 256;
constexpr int TA2_ROW = 256, TA2_SLOTS = 512;
constexpr int TB_ROW = 512, TB_SLOTS = 1024, TB_WARPS = 4;
constexpr int TC1_ROW = 2048, TC1_SLOTS = 4096, TC1_T = 256;
constexpr int TC_ROW = 4096, TC_SLOTS = 8192, TC_T = 512;
constexpr int TC2_ROW = 12288, TC2_SLOTS = 16384, TC2_T = 1024;
constexpr int TC3_ROW = 65536, TC3_KEYS = 12288;   // at most TC3_KEYS walk entries per pass on average
constexpr int TD_T = 1024;
constexpr int32_t EMPTY_KEY = -1;

__device__ __forceinline__ uint32_t slot_hash(int32_t key, int lg) {
    return ((uint32_t)key * 0x9E3779B1u) >> (32 - lg);
}

// The walk of coarse row c in the fine CSR: positions [0, da) are a's row,
// [da, deg) b's row (a = representative, b = partner or none).
struct Walk {
    int64_t ea, da, eb;
    __device__ __forceinline__ int64_t entry(int64_t j) const { return j < da ? ea + j : eb + (j - da); }
};
__device__ __forceinline__ Walk walk_of(const DGraph& g, const int32_t* __restrict__ mem, int64_t c) {
    const int32_t a = mem[2 * c], b = mem[2 * c + 1];
    Walk W;
    W.ea = g.rp[a];
    W.da = g.rp[a + 1] - W.ea;
    W.eb = b >= 0 ? g.rp[b] : 0;
    return W;
}
// mapped id and weight of walk position j
__device__ __forceinline__ void walk_load(const DGraph& g, const int32_t* __restrict__ cmap, const Walk& W, int64_t j,
                                          int32_t& cu, int32_t& w) {
    const int64_t e = W.entry(j);
    const int32_t u = __ldcs(&g.ci[e]);
    cu = GP_IN(u, g.n) ? cmap[u] : 0;
    w = g.ew ? __ldcs(&g.ew[e]) : 1;
}

// tier-D rows in walk layout, by the pieces the tier-D kernels use
struct TierD;
__global__ void k_fill_walk_d(TierD D, DGraph g, const int32_t* __restrict__ cmap, const int32_t* __restrict__ mem,
                              const int64_t* __restrict__ off, int32_t* __restrict__ mapped, int32_t* __restrict__ mw);

// Ordered insertion of one walk by one warp into a shared-memory table.
// okey/wacc: output ids and weights by rank (shared), oslot: the slot of each
// rank (the row's used slots, cleared afterwards); returns the row length.
template <int SLOTS, class IdxT>
__device__ __forceinline__ int32_t warp_dedup(const DGraph& g, const int32_t* __restrict__ cmap, const Walk& W,
                                              int64_t deg, int32_t self, int32_t* key, IdxT* tidx, IdxT* oslot,
                                              int32_t* okey, int32_t* wacc, int lg) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    int32_t count = 0;
    int32_t cu_next = -1, w_next = 0;
    if (lane < deg) walk_load(g, cmap, W, lane, cu_next, w_next);
    for (int64_t base = 0; base < deg; base += 32) {
        const int64_t j = base + lane;
        const int32_t cu = cu_next, wt = w_next;
        // prefetch the next chunk
        if (j + 32 < deg) walk_load(g, cmap, W, j + 32, cu_next, w_next);
        const bool act = (j < deg) && cu != self;
        const uint32_t peers = __match_any_sync(0xffffffffu, act ? (uint32_t)cu : (0x80000000u | (uint32_t)lane));
        const int leader = __ffs(peers) - 1;
        bool isnew = false;
        int32_t h = -1;
        if (act && lane == leader) {
            h = (int32_t)slot_hash(cu, lg);
            for (int probe = 0; probe < SLOTS; ++probe) {
                const int32_t old = atomicCAS(&key[h], EMPTY_KEY, cu);
                if (old == EMPTY_KEY) { isnew = true; break; }
                if (old == cu) break;
                h = (h + 1) & (SLOTS - 1);
            }
        }
        const uint32_t newmask = __ballot_sync(0xffffffffu, isnew);
        int32_t idx = -1;
        if (isnew) {
            idx = count + __popc(newmask & lt);
            tidx[h] = (IdxT)idx;
            oslot[idx] = (IdxT)h;
            okey[idx] = cu;
        }
        __syncwarp();
        if (act && lane == leader && !isnew) idx = tidx[h];
        idx = __shfl_sync(0xffffffffu, idx, leader);
        if (act) atomicAdd(&wacc[idx], wt);
        count += __popc(newmask);
        __syncwarp();
    }
    return count;
}

// Tier S: a row of at most N walk entries by one thread.  The entries' loads,
// then their cmap gathers, are in flight together; a later copy of a key adds
// its weight to the first one's register and drops out, so the keys that remain
// are in first-occurrence order.  A warp per row spent most of its issue slots
// on rows of a dozen entries (256^3 grid, level 0: 9.1 M coarse rows of at most
// 12 walk entries, 3.3 -> 0.9 ms).
template <int N>
__device__ __forceinline__ int32_t thread_dedup(const DGraph& g, const int32_t* __restrict__ cmap, const Walk& W,
                                                int32_t deg, int32_t self, int32_t* __restrict__ tci,
                                                int32_t* __restrict__ tew) {
    int32_t key[N], w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) key[i] = i < deg ? __ldg(&g.ci[W.entry(i)]) : -1;
    if (g.ew) {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = i < deg ? __ldg(&g.ew[W.entry(i)]) : 0;
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = 1;
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (key[i] >= 0) key[i] = GP_IN(key[i], g.n) ? cmap[key[i]] : -1;
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (key[i] == self) key[i] = -1;
#pragma unroll
    for (int j = 1; j < N; ++j)
#pragma unroll
        for (int i = 0; i < j; ++i)
            if (key[j] >= 0 && key[i] == key[j]) { w[i] += w[j]; key[j] = -1; }
    int32_t r = 0;
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (key[i] >= 0) { tci[r] = key[i]; tew[r] = w[i]; ++r; }
    return r;
}
constexpr int TS_ROW = 32;
template <int N>
__global__ void __launch_bounds__(128) k_dedup_thread(DGraph g, const int32_t* __restrict__ cmap,
                                                      const int32_t* __restrict__ mem, int64_t nc, int64_t minrow,
                                                      const int64_t* __restrict__ off, const int64_t* __restrict__ cdeg,
                                                      int32_t* __restrict__ tci, int32_t* __restrict__ tew,
                                                      int32_t* __restrict__ cnt) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t deg = cdeg[c];
        if (deg > N || deg < minrow) continue;
        const int64_t o = off[c];
        cnt[c] = thread_dedup<N>(g, cmap, walk_of(g, mem, c), (int32_t)deg, (int32_t)c, tci + o, tew + o);
    }
}

template <int MAXROW, int SLOTS, class IdxT>
__host__ __device__ constexpr size_t warp_dedup_smem() {
    return ((sizeof(int32_t) * (SLOTS + 2 * MAXROW) + sizeof(IdxT) * (SLOTS + MAXROW)) + 15) & ~(size_t)15;
}

// tiers A (MAXROW 128) and B (MAXROW 1024): one warp per row
template <int MAXROW, int SLOTS, int WARPS, class IdxT>
__global__ void __launch_bounds__(WARPS * 32) k_dedup_warp(DGraph g, const int32_t* __restrict__ cmap,
                                                           const int32_t* __restrict__ mem, int64_t nc, int64_t minrow,
                                                           const int64_t* __restrict__ off,
                                                           const int64_t* __restrict__ cdeg, int32_t* __restrict__ tci,
                                                           int32_t* __restrict__ tew, int32_t* __restrict__ cnt) {
    // dynamic shared memory per warp: key[SLOTS] okey[MAXROW] wacc[MAXROW] idx[SLOTS] oslot[MAXROW]
    extern __shared__ int32_t dsm[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t per_warp = warp_dedup_smem<MAXROW, SLOTS, IdxT>() / sizeof(int32_t);
    int32_t* key = dsm + w * per_warp;
    int32_t* okey = key + SLOTS;
    int32_t* wacc = okey + MAXROW;
    IdxT* tidx = (IdxT*)(wacc + MAXROW);
    IdxT* oslot = tidx + SLOTS;
    for (int i = lane; i < SLOTS; i += 32) key[i] = EMPTY_KEY;
    for (int i = lane; i < MAXROW; i += 32) wacc[i] = 0;
    __syncwarp();
    int lg = 0;
    while ((1 << lg) < SLOTS) ++lg;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = wid; c < nc; c += nw) {
        const int64_t deg = cdeg[c];
        if (deg > MAXROW || deg < minrow) continue;
        const int64_t o = off[c];
        const int32_t count = warp_dedup<SLOTS, IdxT>(g, cmap, walk_of(g, mem, c), deg, (int32_t)c, key, tidx, oslot,
                                                      okey, wacc, lg);
        for (int i = lane; i < count; i += 32) {
            tci[o + i] = okey[i];
            tew[o + i] = wacc[i];
            wacc[i] = 0;
            key[oslot[i]] = EMPTY_KEY;
        }
        if (lane == 0) cnt[c] = count;
        __syncwarp();
    }
}

__device__ __forceinline__ int32_t block_scan_excl(int32_t x, int32_t* sh, int32_t& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { int32_t y = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += y; }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        int32_t s2 = lane < nw ? sh[lane] : 0, i2 = s2;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int32_t y = __shfl_up_sync(0xffffffffu, i2, o); if (lane >= o) i2 += y; }
        if (lane < nw) sh[lane] = i2 - s2;
        if (lane == nw - 1) sh[32] = i2;
    }
    __syncthreads();
    const int32_t r = inc - x + sh[w];
    total = sh[32];
    __syncthreads();
    return r;
}

// rows longer than TB_ROW: lists of the on-chip tiers C1 (<= TC1_ROW), C
// (<= TC_ROW), C2 (<= TC2_ROW), C3 (<= TC3_ROW) and of tier D.  count[0] =
// rows of tier C, count[1] = rows of tier D, count[2] = longest tier-D row,
// count[3] = rows of tier C2, count[4] = rows of tier C3, count[5] = rows of
// tier C1
__global__ void k_long_rows(int64_t nc, const int64_t* __restrict__ cdeg, int32_t* __restrict__ listC1,
                            int32_t* __restrict__ listC, int32_t* __restrict__ listC2, int32_t* __restrict__ listC3,
                            int32_t* __restrict__ listD, int64_t* __restrict__ count) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t d = cdeg[c];
        if (d <= TB_ROW) continue;
        if (d <= TC1_ROW) {
            unsigned long long slot = atomicAdd((unsigned long long*)&count[5], 1ull);
            listC1[slot] = (int32_t)c;
        } else if (d <= TC_ROW) {
            unsigned long long slot = atomicAdd((unsigned long long*)&count[0], 1ull);
            listC[slot] = (int32_t)c;
        } else if (d <= TC2_ROW) {
            unsigned long long slot = atomicAdd((unsigned long long*)&count[3], 1ull);
            listC2[slot] = (int32_t)c;
        } else if (d <= TC3_ROW) {
            unsigned long long slot = atomicAdd((unsigned long long*)&count[4], 1ull);
            listC3[slot] = (int32_t)c;
        } else {
            unsigned long long slot = atomicAdd((unsigned long long*)&count[1], 1ull);
            listD[slot] = (int32_t)c;
            atomicMax((unsigned long long*)&count[2], (unsigned long long)d);
        }
    }
}

// A slot of the one-block tiers' tables: a key and its first walk position.
// PB > 0: 32 bits, key << PB | position (position < 2^PB, key < 2^(32 - PB) - 1),
// all ones meaning empty: native compare-and-swap and minimum, 8 bytes a slot
// with the weight.  PB = 0: 64 bits, (key + 1) << 32 | (deg - position), zero
// meaning empty, the first position being the maximum.
template <int PB>
struct Slot {
    using T = uint32_t;
    static constexpr T EMPTY = 0xFFFFFFFFu;
    static __device__ __forceinline__ T make(int32_t key, int32_t j, int32_t) { return ((uint32_t)key << PB) | (uint32_t)j; }
    static __device__ __forceinline__ bool same(T a, T b) { return ((a ^ b) >> PB) == 0u; }
    static __device__ __forceinline__ T cas(T* s, T v) { return atomicCAS(s, EMPTY, v); }
    static __device__ __forceinline__ void first(T* s, T old, T v) { if (v < old) atomicMin(s, v); }
    static __device__ __forceinline__ int32_t pos(T v, int32_t) { return (int32_t)(v & ((1u << PB) - 1u)); }
    static __device__ __forceinline__ int32_t key(T v) { return (int32_t)(v >> PB); }
};
template <>
struct Slot<0> {
    using T = unsigned long long;
    static constexpr T EMPTY = 0ull;
    static __device__ __forceinline__ T make(int32_t key, int32_t j, int32_t deg) {
        return ((unsigned long long)((uint32_t)key + 1u) << 32) | (uint32_t)(deg - j);
    }
    static __device__ __forceinline__ bool same(T a, T b) { return (uint32_t)((a ^ b) >> 32) == 0u; }
    static __device__ __forceinline__ T cas(T* s, T v) { return atomicCAS(s, EMPTY, v); }
    static __device__ __forceinline__ void first(T* s, T old, T v) { if (v > old) atomicMax(s, v); }
    static __device__ __forceinline__ int32_t pos(T v, int32_t deg) { return deg - (int32_t)(uint32_t)v; }
    static __device__ __forceinline__ int32_t key(T v) { return (int32_t)((uint32_t)(v >> 32) - 1u); }
};
// Inserts up to four entries of this thread (cu == self: none) into a table of
// 2^lg slots and adds their weights; h: their slots.  The probes of the four go
// on together, so that their shared-memory round trips overlap, in odd steps of
// the key's own (full cycles; unit steps pile up in tables three quarters full).
// R-MAT 24, rows of 4097-12288 / 2049-4096 / 513-2048 / 12289-65536 entries, in all:
// 31.1 / 15.3 / 13.8 / 46.0 ms one entry after the other, 22.7 / 13.1 / 12.8 / 41.2
// together, 20.9 / 12.5 / 12.0 / 39.6 with the steps.
template <int PB>
__device__ __forceinline__ void slots_insert(typename Slot<PB>::T* slot, int32_t* wsum, int lg, int32_t self,
                                             const int32_t (&cu)[4], const int32_t (&wt)[4],
                                             const typename Slot<PB>::T (&val)[4], uint32_t (&h)[4], int32_t* err) {
    using S = Slot<PB>;
    const uint32_t mask = (1u << lg) - 1u;
    typename S::T old[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        h[c] = slot_hash(cu[c], lg);
        old[c] = cu[c] != self ? S::cas(&slot[h[c]], val[c]) : S::EMPTY;
    }
    for (uint32_t probe = 1; probe <= mask; ++probe) {
        bool any = false;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (old[c] != S::EMPTY && !S::same(old[c], val[c])) {
                any = true;
                h[c] = (h[c] + (((uint32_t)cu[c] * 0x85EBCA77u) >> 24 | 1u)) & mask;
                old[c] = S::cas(&slot[h[c]], val[c]);
            }
        }
        if (!any) break;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (cu[c] == self) continue;
        if (old[c] != S::EMPTY && !S::same(old[c], val[c])) { atomicExch(err, 1); continue; }
        if (old[c] != S::EMPTY) S::first(&slot[h[c]], old[c], val[c]);
        atomicAdd(&wsum[h[c]], wt[c]);
    }
}

// tiers C1, C and C2: one CTA per row, table in shared memory, two phases.
// Phase 1 reads the walk once (straight from the fine CSR) and inserts every
// entry (Slot): the claiming compare-and-swap stores the first position seen, an
// earlier one replaces it; weights add up in wsum, and position j keeps its slot
// in hj[j].  Phase 2: every warp takes a contiguous range of 32-position words,
// ballots their first-occurrence flags (lane i keeps word i's), and scans their
// counts by shuffles; the warps' totals meet in shared memory, and the warps
// write the first occurrences at their ranks, emptying their slots (each used
// slot has exactly one), so the table is clear for the CTA's next row.
// What bounds a row of a few thousand entries is its chain of latencies: three
// barriers, and the loads list -> members -> row pointers -> ids -> cmap.  The
// headers are taken two rows ahead, the ids and weights one sweep ahead (the
// first sweep of the next row before this row's barriers).
// C2 / C / C1 on R-MAT 24, in all: 37.9 / 18.5 / 17.2 ms with seven barriers,
// bitmap and ranks in shared memory and every chain in the open, 35.2 / 16.8 /
// 15.2 with headers one row ahead, 20.9 / 12.5 / 12.0 with ids ahead, 32-bit slots
// and the probes of a thread's four entries together.
constexpr uint16_t NO_SLOT = 0xFFFF;
constexpr int TC1_PB = 11, TC_PB = 12, TC2_PB = 14, TC3_PB = 16;   // position bits of each tier's 32-bit slots
template <int PB>
static bool slot_fits(int64_t nc) { return nc < ((int64_t)1 << (32 - PB)); }

// shared memory of an on-chip tier: SLOTS slots and int32 weight sums, a slot id
// per walk position
template <int SLOTS, int MAXROW, int PB>
constexpr size_t cta_dedup_smem() {
    return (sizeof(typename Slot<PB>::T) + sizeof(int32_t)) * SLOTS + sizeof(uint16_t) * MAXROW;
}

// table of at least twice the row length, at most SLOTS
template <int T, int SLOTS, int MAXROW, int PB>
__global__ void __launch_bounds__(T, 1024 / T)
    k_dedup_cta_smem(DGraph g, const int32_t* __restrict__ cmap, const int32_t* __restrict__ mem,
                     const int32_t* __restrict__ list, int64_t nlist, const int64_t* __restrict__ off,
                     const int64_t* __restrict__ cdeg, int32_t* __restrict__ tci, int32_t* __restrict__ tew,
                     int32_t* __restrict__ cnt, int32_t* __restrict__ err) {
    static_assert(SLOTS <= 65535, "slot ids are 16-bit");
    static_assert(PB == 0 || (1 << PB) >= MAXROW, "positions fit");
    constexpr int NW = T / 32;
    static_assert((MAXROW + 32 * NW - 1) / (32 * NW) <= 32, "a warp's words fit in its lanes");
    using S = Slot<PB>;
    using ST = typename S::T;
    extern __shared__ __align__(16) unsigned char stab_raw[];
    ST* slot = (ST*)stab_raw;                                          // SLOTS
    int32_t* wsum = (int32_t*)(slot + SLOTS);                          // SLOTS
    uint16_t* hj = (uint16_t*)(wsum + SLOTS);                          // MAXROW
    __shared__ int32_t s_tot[NW];
    for (int i = threadIdx.x; i < SLOTS; i += T) { slot[i] = S::EMPTY; wsum[i] = 0; }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    int64_t li = blockIdx.x;
    if (li >= nlist) return;
    int32_t self = list[li], deg = (int32_t)cdeg[self];
    Walk W = walk_of(g, mem, self);
    int32_t u[4], wt[4];   // ids and weights of the sweep to come
    auto ahead = [&](const Walk& X, int32_t base, int32_t d) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int32_t j = base + c * T + threadIdx.x;
            u[c] = -1; wt[c] = 0;
            if (j < d) {
                const int64_t e = X.entry(j);
                u[c] = __ldcs(&g.ci[e]);
                wt[c] = g.ew ? __ldcs(&g.ew[e]) : 1;
            }
        }
    };
    ahead(W, 0, deg);
    int64_t ln = li + gridDim.x;
    int32_t cn = ln < nlist ? list[ln] : -1;   // the next row: its header complete,
    int32_t ndeg = 0;
    Walk nW{0, 0, 0};
    if (cn >= 0) { ndeg = (int32_t)cdeg[cn]; nW = walk_of(g, mem, cn); }
    __syncthreads();
    for (;;) {
        const int64_t l2 = ln + gridDim.x;
        const int32_t c2 = l2 < nlist ? list[l2] : -1;   // the one after it, its loads one phase ahead of their use
        const int64_t o = off[self];
        int lg = 0;
        while ((1 << lg) < 2 * deg && (1 << lg) < SLOTS) ++lg;
        for (int32_t base = 0; base < deg; base += 4 * T) {
            int32_t cu[4], cw[4];
            ST val[4];
            uint32_t h[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                cu[c] = u[c] < 0 ? self : (GP_IN(u[c], g.n) ? cmap[u[c]] : 0);
                cw[c] = wt[c];
            }
            if (base + 4 * T < deg) ahead(W, base + 4 * T, deg);
            else if (cn >= 0) ahead(nW, 0, ndeg);
#pragma unroll
            for (int c = 0; c < 4; ++c) val[c] = S::make(cu[c], base + c * T + (int32_t)threadIdx.x, deg);
            slots_insert<PB>(slot, wsum, lg, self, cu, cw, val, h, err);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int32_t j = base + c * T + threadIdx.x;
                if (j < deg) hj[j] = cu[c] == self ? NO_SLOT : (uint16_t)h[c];
            }
        }
        int32_t a = 0, b = -1, d2 = 0;
        if (c2 >= 0) { a = mem[2 * (int64_t)c2]; b = mem[2 * (int64_t)c2 + 1]; d2 = (int32_t)cdeg[c2]; }
        __syncthreads();
        const int32_t nwords = (deg + 31) / 32, wpw = (nwords + NW - 1) / NW, wbeg = wid * wpw;
        uint32_t mine = 0;   // lane i: first-occurrence flags of word wbeg + i
        for (int32_t i = 0; i < wpw && wbeg + i < nwords; ++i) {
            const int32_t j = (wbeg + i) * 32 + lane;
            bool first = false;
            if (j < deg) {
                const uint16_t hh = hj[j];
                first = hh != NO_SLOT && S::pos(slot[hh], deg) == j;
            }
            const uint32_t word = __ballot_sync(0xffffffffu, first);
            if (lane == i) mine = word;
        }
        const int32_t pop = __popc(mine), inc = warp_incl_scan<int32_t>(pop);
        if (lane == 31) s_tot[wid] = inc;
        Walk W2{0, 0, 0};
        if (c2 >= 0) {
            W2.ea = g.rp[a];
            W2.da = g.rp[a + 1] - W2.ea;
            if (b >= 0) W2.eb = g.rp[b];
        }
        __syncthreads();
        const int32_t wtot = lane < NW ? s_tot[lane] : 0;
        const int32_t before = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)(lane < wid ? wtot : 0));
        if (wid == 0) {
            const int32_t tot = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)wtot);
            if (lane == 0) cnt[self] = tot;
        }
        const int32_t at = before + inc - pop;
        for (int32_t i = 0; i < wpw && wbeg + i < nwords; ++i) {
            const uint32_t word = __shfl_sync(0xffffffffu, mine, i);
            const int32_t r = __shfl_sync(0xffffffffu, at, i) + __popc(word & lt);
            if (!((word >> lane) & 1u)) continue;
            const uint16_t hh = hj[(wbeg + i) * 32 + lane];
            if (!GP_IN(r, deg) || !GP_IN(hh, SLOTS)) continue;
            tci[o + r] = S::key(slot[hh]);
            tew[o + r] = wsum[hh];
            slot[hh] = S::EMPTY;   // nobody else looks at this slot any more
            wsum[hh] = 0;
        }
        if (cn < 0) break;
        __syncthreads();
        ln = l2; self = cn; deg = ndeg; W = nW; cn = c2; ndeg = d2; nW = W2;
    }
}

// rows of a one-CTA-per-row tier, longest walk first: the block scheduler
// starts CTAs in list order, so the long rows no longer trail the launch
__global__ void k_len_keys(const int32_t* __restrict__ list, int64_t nlist, const int64_t* __restrict__ cdeg,
                           int64_t maxrow, uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nlist; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = list[i];
        const int64_t d = cdeg[c];
        keys[i] = (uint64_t)(d < maxrow ? maxrow - d : 0);
        vals[i] = c;
    }
}
static int32_t* longest_first(Ctx& c, const int32_t* list, int64_t nlist, const int64_t* cdeg, int64_t maxrow) {
    uint64_t* keys = c.tmp_alloc<uint64_t>(nlist);
    uint64_t* keys2 = c.tmp_alloc<uint64_t>(nlist);
    int32_t* vals = c.tmp_alloc<int32_t>(nlist);
    int32_t* vals2 = c.tmp_alloc<int32_t>(nlist);
    k_len_keys<<<grid_for(nlist, 256), 256, 0, c.s>>>(list, nlist, cdeg, maxrow, keys, vals);
    GP_LAUNCHED(c);
    radix_sort_pairs(c, keys, vals, keys2, vals2, nlist, bits_for(maxrow + 1));
    return vals;
}

// tier C3: one 1024-thread CTA per row of TC2_ROW < d <= TC3_ROW walk entries.
// Pass 0 gathers the walk through cmap once and leaves the mapped ids and
// weights in the row's range of the scratch arrays (key_at, w_at); passes
// 1..P-1 read them from there (P = the power of two with min(d, nc) / P <=
// TC3_KEYS: there are at most nc keys).
// Pass p inserts only the keys whose pass hash is p into the 16384-slot table
// (Slot, weights summed), then every used slot marks its first
// position in a bitmap of the walk, leaves its weight sum at that position of
// w_at (later passes never read the weights of another pass's keys), and is
// cleared.  After the passes one block scan ranks
// the marked positions and the keys are written in first-occurrence order, as
// every other tier writes them.  Each sweep's ids are loaded a sweep ahead (39.6
// -> 38.7 ms on R-MAT 24; 46.8 with the entries' probes one after the other).
template <int PB>
constexpr size_t tc3_smem() {
    return (sizeof(typename Slot<PB>::T) + sizeof(int32_t)) * TC2_SLOTS + sizeof(uint32_t) * 2 * (TC3_ROW / 32);
}
__device__ __forceinline__ uint32_t pass_of(int32_t key, int lgp) {
    return lgp ? ((uint32_t)key * 0x85EBCA77u) >> (32 - lgp) : 0u;
}
template <int PB>
__global__ void __launch_bounds__(TC2_T) k_dedup_multipass(DGraph g, int64_t nc, const int32_t* __restrict__ cmap,
                                                           const int32_t* __restrict__ mem,
                                                           const int32_t* __restrict__ list, int64_t nlist,
                                                           const int64_t* __restrict__ off,
                                                           const int64_t* __restrict__ cdeg,
                                                           int32_t* __restrict__ key_at, int32_t* __restrict__ w_at,
                                                           int32_t* __restrict__ tci, int32_t* __restrict__ tew,
                                                           int32_t* __restrict__ cnt, int32_t* __restrict__ err) {
    constexpr int T = TC2_T, S = TC2_SLOTS, LG = 14;
    static_assert((1 << LG) == S, "table size");
    extern __shared__ __align__(16) unsigned char mp_raw[];
    using SL = Slot<PB>;
    using ST = typename SL::T;
    ST* slot = (ST*)mp_raw;                                            // S
    int32_t* wsum = (int32_t*)(slot + S);                              // S
    uint32_t* bits = (uint32_t*)(wsum + S);                            // TC3_ROW / 32
    int32_t* wpre = (int32_t*)(bits + TC3_ROW / 32);                   // TC3_ROW / 32
    __shared__ int32_t sh[33];
    for (int i = threadIdx.x; i < S; i += T) { slot[i] = SL::EMPTY; wsum[i] = 0; }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = T / 32;
    for (int64_t li = blockIdx.x; li < nlist; li += gridDim.x) {
        const int64_t c = list[li];
        const int64_t deg = cdeg[c], o = off[c];
        const int32_t self = (int32_t)c;
        const Walk W = walk_of(g, mem, c);
        const int64_t nwords = (deg + 31) / 32;
        int lgp = 0;
        const int64_t most = deg < nc ? deg : nc;
        while ((most >> lgp) > TC3_KEYS) ++lgp;
        for (int64_t i = threadIdx.x; i < nwords; i += T) bits[i] = 0u;
        __syncthreads();
        int32_t u[4], uw[4];   // the sweep to come: ids and weights (pass 0) or mapped ids
        auto ahead = [&](uint32_t pass, int64_t base) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t j = base + q * T + threadIdx.x;
                u[q] = pass ? self : -1; uw[q] = 0;
                if (j >= deg) continue;
                if (pass) { u[q] = __ldcg(&key_at[o + j]); continue; }   // this thread's own store
                const int64_t e = W.entry(j);
                u[q] = __ldcs(&g.ci[e]);
                uw[q] = g.ew ? __ldcs(&g.ew[e]) : 1;
            }
        };
        ahead(0, 0);
        for (uint32_t pass = 0; pass < (1u << lgp); ++pass) {
            for (int64_t base = 0; base < deg; base += 4 * T) {
                int32_t cu[4], wt[4];
                if (pass == 0) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        cu[q] = u[q] < 0 ? self : (GP_IN(u[q], g.n) ? cmap[u[q]] : 0);
                        wt[q] = uw[q];
                    }
                    if (base + 4 * T < deg) ahead(0, base + 4 * T);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int64_t j = base + q * T + threadIdx.x;
                        if (j < deg) { key_at[o + j] = cu[q]; w_at[o + j] = wt[q]; }
                        if (cu[q] != self && pass_of(cu[q], lgp) != pass) cu[q] = self;
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int64_t j = base + q * T + threadIdx.x;
                        cu[q] = u[q] != self && pass_of(u[q], lgp) == pass ? u[q] : self;
                        wt[q] = cu[q] != self ? __ldcg(&w_at[o + j]) : 0;
                    }
                    if (base + 4 * T < deg) ahead(pass, base + 4 * T);
                }
                if (base + 4 * T >= deg && pass + 1 < (1u << lgp)) ahead(pass + 1, 0);
                ST val[4];
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    val[q] = SL::make(cu[q], (int32_t)base + q * T + (int32_t)threadIdx.x, (int32_t)deg);
                slots_insert<PB>(slot, wsum, LG, self, cu, wt, val, h, err);
            }
            __syncthreads();
            // the pass's keys: mark first positions, park key and weight there, clear
            for (int i = threadIdx.x; i < S; i += T) {
                const ST v = slot[i];
                if (v == SL::EMPTY) continue;
                const int64_t j = SL::pos(v, (int32_t)deg);
                if (GP_IN(j, deg)) {
                    atomicOr(&bits[j >> 5], 1u << (j & 31));
                    w_at[o + j] = wsum[i];
                }
                slot[i] = SL::EMPTY;
                wsum[i] = 0;
            }
            __syncthreads();
        }
        // ranks of the marked positions: contiguous word ranges per thread
        const int64_t per = (nwords + T - 1) / T;
        const int64_t w0 = (int64_t)threadIdx.x * per, w1 = w0 + per < nwords ? w0 + per : nwords;
        int32_t mine = 0;
        for (int64_t wi = w0; wi < w1; ++wi) mine += __popc(bits[wi]);
        int32_t tot;
        int32_t run = block_scan_excl(mine, sh, tot);
        for (int64_t wi = w0; wi < w1; ++wi) { wpre[wi] = run; run += __popc(bits[wi]); }
        __syncthreads();
        const uint32_t lt = (1u << lane) - 1u;
        for (int64_t wi = wid; wi < nwords; wi += nwarp) {
            const uint32_t word = bits[wi];
            if (!((word >> lane) & 1u)) continue;
            const int64_t j = wi * 32 + lane;
            const int32_t r = wpre[wi] + __popc(word & lt);
            if (!GP_IN(r, deg)) continue;
            tci[o + r] = key_at[o + j];
            tew[o + r] = w_at[o + j];
        }
        if (threadIdx.x == 0) cnt[c] = tot;
        __syncthreads();
    }
}

// tier D split over CTAs: rows longer than TC_ROW are cut into pieces of
// TD_PIECE entries, one CTA each, all pieces of a row sharing that row's
// global table.  D1 inserts: a 64-bit slot holds (key + 1) << 32 | (deg - j),
// zero meaning empty; the claiming compare-and-swap stores the first
// position seen, later copies of the key raise it by atomicMax (the largest
// deg - j is the first occurrence), weights add up in a 32-bit array.  D2 ballots the
// first-occurrence flags of each 32-entry word, a device-wide scan of the word
// popcounts ranks the words of every row, D3 writes the first occurrences at
// their ranks.  Same output as one CTA per row: unique neighbours in order of
// first occurrence with summed weights.
constexpr int64_t TD_PIECE = 16384;   // multiple of 32
struct TierD {
    const int32_t* rc;      // coarse row of each tier-D row
    const int32_t* rlg;     // log2 of its table size
    const int64_t* rtab;    // table offset
    const int64_t* rword;   // first word of the row in the word arrays
    const int32_t* prow;    // row of each piece
    const int64_t* pbeg;    // entry range of the piece within the row
    const int64_t* pend;
    unsigned long long* slot;   // tables: (key + 1) << 32 | (deg - first position), 0 = empty
    int32_t* wsum;              // weight sums
    uint32_t* bits;         // first-occurrence flags, one word per 32 entries
    int32_t* wcnt;          // their popcounts
    const int64_t* wpre;    // exclusive prefix of wcnt (+ total)
};

// mapped ids and weights of the tier-D rows in walk layout, one CTA per piece
__global__ void __launch_bounds__(TD_T) k_fill_walk_d(TierD D, DGraph g, const int32_t* __restrict__ cmap,
                                                      const int32_t* __restrict__ mem, const int64_t* __restrict__ off,
                                                      int32_t* __restrict__ mapped, int32_t* __restrict__ mw) {
    const int32_t c = D.rc[D.prow[blockIdx.x]];
    const Walk W = walk_of(g, mem, c);
    const int64_t o = off[c];
    for (int64_t j = D.pbeg[blockIdx.x] + threadIdx.x; j < D.pend[blockIdx.x]; j += TD_T)
        walk_load(g, cmap, W, j, mapped[o + j], mw[o + j]);
}

__device__ __forceinline__ uint32_t td_lookup(const unsigned long long* slot, int32_t cu, int lg) {
    const uint32_t mask = (1u << lg) - 1u;
    const uint32_t tag = (uint32_t)cu + 1u;
    uint32_t h = slot_hash(cu, lg);
    for (uint32_t probe = 0; probe <= mask && (uint32_t)(slot[h] >> 32) != tag; ++probe) h = (h + 1) & mask;
    return h;
}

__global__ void __launch_bounds__(TD_T) k_td_insert(TierD D, const int64_t* __restrict__ off,
                                                    const int64_t* __restrict__ cdeg,
                                                    const int32_t* __restrict__ mapped, const int32_t* __restrict__ mw,
                                                    int32_t* __restrict__ err) {
    const int32_t r = D.prow[blockIdx.x];
    const int32_t self = D.rc[r];
    const int lg = D.rlg[r];
    const uint32_t mask = (1u << lg) - 1u;
    unsigned long long* slot = D.slot + D.rtab[r];
    int32_t* wsum = D.wsum + D.rtab[r];
    const int64_t o = off[self], deg = cdeg[self], end = D.pend[blockIdx.x];
    for (int64_t base = D.pbeg[blockIdx.x]; base < end; base += 4 * TD_T) {
        int32_t cu[4], wt[4];
        unsigned long long val[4], old[4];
        uint32_t h[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int64_t j = base + c * TD_T + threadIdx.x;
            cu[c] = j < end ? __ldcs(&mapped[o + j]) : self;
            wt[c] = j < end ? __ldcs(&mw[o + j]) : 0;
            val[c] = ((unsigned long long)((uint32_t)cu[c] + 1u) << 32) | (uint32_t)(deg - j);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            h[c] = slot_hash(cu[c], lg);
            old[c] = cu[c] != self ? atomicCAS(&slot[h[c]], 0ull, val[c]) : 0ull;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (cu[c] == self) continue;
            const uint32_t tag = (uint32_t)cu[c] + 1u;
            uint32_t probe = 1;
            while (old[c] != 0ull && (uint32_t)(old[c] >> 32) != tag && probe <= mask) {
                h[c] = (h[c] + 1) & mask;
                old[c] = atomicCAS(&slot[h[c]], 0ull, val[c]);
                ++probe;
            }
            if (old[c] != 0ull && (uint32_t)(old[c] >> 32) != tag) { atomicExch(err, 1); continue; }
            // claimed with this position, or the key was there: keep the earliest position
            if (old[c] != 0ull && old[c] < val[c]) atomicMax(&slot[h[c]], val[c]);
            atomicAdd(&wsum[h[c]], wt[c]);
        }
    }
}

__global__ void __launch_bounds__(TD_T) k_td_flags(TierD D, const int64_t* __restrict__ off,
                                                   const int64_t* __restrict__ cdeg,
                                                   const int32_t* __restrict__ mapped) {
    const int32_t r = D.prow[blockIdx.x];
    const int32_t self = D.rc[r];
    const int lg = D.rlg[r];
    const unsigned long long* slot = D.slot + D.rtab[r];
    const int64_t o = off[self], deg = cdeg[self];
    const int lane = threadIdx.x & 31;
    const int64_t w0 = D.pbeg[blockIdx.x] / 32, w1 = (D.pend[blockIdx.x] + 31) / 32;
    for (int64_t wi = w0 + (threadIdx.x >> 5); wi < w1; wi += TD_T / 32) {
        const int64_t j = wi * 32 + lane;
        bool first = false;
        if (j < deg) {
            const int32_t cu = mapped[o + j];
            if (cu != self) first = (uint32_t)slot[td_lookup(slot, cu, lg)] == (uint32_t)(deg - j);
        }
        const uint32_t word = __ballot_sync(0xffffffffu, first);
        if (lane == 0) {
            D.bits[D.rword[r] + wi] = word;
            D.wcnt[D.rword[r] + wi] = __popc(word);
        }
    }
}

__global__ void __launch_bounds__(TD_T) k_td_write(TierD D, const int64_t* __restrict__ off,
                                                   const int64_t* __restrict__ cdeg,
                                                   const int32_t* __restrict__ mapped, int32_t* __restrict__ tci,
                                                   int32_t* __restrict__ tew, int32_t* __restrict__ rowcnt) {
    const int32_t r = D.prow[blockIdx.x];
    const int32_t self = D.rc[r];
    const int lg = D.rlg[r];
    const unsigned long long* slot = D.slot + D.rtab[r];
    const int32_t* wsum = D.wsum + D.rtab[r];
    const int64_t o = off[self], deg = cdeg[self];
    const int64_t rw = D.rword[r], nwords = (deg + 31) / 32;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t w0 = D.pbeg[blockIdx.x] / 32, w1 = (D.pend[blockIdx.x] + 31) / 32;
    for (int64_t wi = w0 + (threadIdx.x >> 5); wi < w1; wi += TD_T / 32) {
        const uint32_t word = D.bits[rw + wi];
        if (!((word >> lane) & 1u)) continue;
        const int32_t cu = mapped[o + wi * 32 + lane];
        const int64_t rank = D.wpre[rw + wi] - D.wpre[rw] + __popc(word & lt);
        if (!GP_IN(rank, deg)) continue;
        tci[o + rank] = cu;
        tew[o + rank] = wsum[td_lookup(slot, cu, lg)];
    }
    if (D.pbeg[blockIdx.x] == 0 && threadIdx.x == 0) rowcnt[self] = (int32_t)(D.wpre[rw + nwords] - D.wpre[rw]);
}

__global__ void k_td_rows(const int32_t* __restrict__ list, int64_t n, const int64_t* __restrict__ cdeg,
                          int64_t* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = cdeg[list[i]];
}

// warp per coarse row: temporary (walk-bound offsets) -> final CSR
// Packs every row's deduplicated entries (crp[c + 1] - crp[c] of them at
// walk offset off[c] of tci / tew) into the coarse CSR, entry-sliced (csr_sweep);
// up to eight groups of 32 entries are loaded before any is stored.
__global__ void __launch_bounds__(256) k_contract_copy(int64_t nc, int64_t cm, int64_t slice,
                                                       const int64_t* __restrict__ off,
                                                       const int64_t* __restrict__ crp, const int32_t* __restrict__ tci,
                                                       const int32_t* __restrict__ tew, int32_t* __restrict__ ci,
                                                       int32_t* __restrict__ ew) {
    const int lane = threadIdx.x & 31;
    // payload: source of output entry 0 as seen from the row
    csr_sweep<8, int64_t>(crp, nc, cm, slice, [&](int64_t r, int64_t start) { return r < nc ? off[r] - start : 0; },
                       [&](auto full, int64_t o, int64_t lim, int64_t o0, int64_t, int32_t s, int64_t src) {
        int32_t a[8], b[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (!full && o + 32 * q >= lim) break;
            const int64_t oi = o + 32 * q + lane;
            const int64_t p = __shfl_sync(0xffffffffu, src, csr_lane(s, (int32_t)(oi - o0))) + oi;
            if (full || oi < lim) { a[q] = __ldcs(&tci[p]); b[q] = __ldcs(&tew[p]); }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int64_t oi = o + 32 * q + lane;
            if (full || oi < lim) { ci[oi] = a[q]; ew[oi] = b[q]; }
        }
    });
}

void contract_level(Ctx& c, Level& fine, Level& coarse, const int32_t* match, int64_t pairs) {
    const DGraph& g = fine.g;
    const int64_t nc = g.n - pairs;
    fine.cmap = c.keep_alloc<int32_t>(g.n);
    int32_t* cvw = c.keep_alloc<int32_t>(nc);
    int64_t* crp = c.keep_alloc<int64_t>(nc + 1);
    coarse.g.n = nc;
    coarse.g.rp = crp;
    coarse.g.vw = cvw;
    auto mk = c.tmp->save();
    int64_t* cid = c.tmp_alloc<int64_t>(g.n);
    int64_t* ctl = c.tmp_alloc<int64_t>(C_NCTL);
    memset_async(c, ctl, 0, C_NCTL * sizeof(int64_t));
    scan_representatives(c, match, cid, g.n);
    int32_t* mem = c.tmp_alloc<int32_t>(2 * nc);
    int64_t* cdeg = c.tmp_alloc<int64_t>(nc);
    k_cmap<<<grid_for(g.n, 256), 256, 0, c.s>>>(g, match, cid, fine.cmap, mem, cvw, cdeg, ctl + C_MAXVW);
    GP_LAUNCHED(c);
    int64_t* off = c.tmp_alloc<int64_t>(nc + 1);
    scan_excl_i64(c, cdeg, off, nc, nullptr);
    const int64_t T = g.m;
    int32_t* mapped = c.tmp_alloc<int32_t>(T);
    int32_t* mw = c.tmp_alloc<int32_t>(T);
    int32_t* tci = c.tmp_alloc<int32_t>(T);
    int32_t* tew = c.tmp_alloc<int32_t>(T);
    int32_t* rowcnt = c.tmp_alloc<int32_t>(nc);
    int32_t* listC1 = c.tmp_alloc<int32_t>(nc);
    int32_t* listC = c.tmp_alloc<int32_t>(nc);
    int32_t* listC2 = c.tmp_alloc<int32_t>(nc);
    int32_t* listC3 = c.tmp_alloc<int32_t>(nc);
    int32_t* listD = c.tmp_alloc<int32_t>(nc);
    int64_t* lcount = ctl + C_LONG;
    int32_t* err = (int32_t*)(ctl + C_ERR);
    const int64_t most = 2 * fine.max_deg;   // no coarse row has a longer walk
    {
        constexpr size_t smA = 8 * warp_dedup_smem<TA_ROW, TA_SLOTS, int32_t>();
        constexpr size_t smA2 = 8 * warp_dedup_smem<TA2_ROW, TA2_SLOTS, int16_t>();
        constexpr size_t smB = TB_WARPS * warp_dedup_smem<TB_ROW, TB_SLOTS, int16_t>();
        auto kA = k_dedup_warp<TA_ROW, TA_SLOTS, 8, int32_t>;
        auto kA2 = k_dedup_warp<TA2_ROW, TA2_SLOTS, 8, int16_t>;
        auto kB = k_dedup_warp<TB_ROW, TB_SLOTS, TB_WARPS, int16_t>;
        k_dedup_thread<16><<<grid_for(nc, 128, c.sm_count * c.ctas_per_sm), 128, 0, c.s>>>(g, fine.cmap, mem, nc, 0, off,
                                                                                         cdeg, tci, tew, rowcnt);
        GP_LAUNCHED(c);
        if (most > 16) {
            k_dedup_thread<TS_ROW><<<grid_for(nc, 128, c.sm_count * c.ctas_per_sm), 128, 0, c.s>>>(
                g, fine.cmap, mem, nc, 17, off, cdeg, tci, tew, rowcnt);
            GP_LAUNCHED(c);
        }
        if (most > TS_ROW) {
            kA<<<grid_for(nc * 32, 256, c.sm_count * c.ctas_per_sm), 256, smA, c.s>>>(g, fine.cmap, mem, nc, TS_ROW + 1, off,
                                                                                      cdeg, tci, tew, rowcnt);
            GP_LAUNCHED(c);
        }
        if (most > TA_ROW) {
            kA2<<<grid_for(nc * 32, 256, c.sm_count * c.ctas_per_sm), 256, smA2, c.s>>>(
                g, fine.cmap, mem, nc, TA_ROW + 1, off, cdeg, tci, tew, rowcnt);
            GP_LAUNCHED(c);
        }
        if (most > TA2_ROW) {
            kB<<<grid_for(nc * 32, TB_WARPS * 32, c.sm_count * c.ctas_per_sm), TB_WARPS * 32, smB, c.s>>>(
                g, fine.cmap, mem, nc, TA2_ROW + 1, off, cdeg, tci, tew, rowcnt);
            GP_LAUNCHED(c);
        }
    }
    int64_t nC = 0, nD = 0, nC2 = 0, nC3 = 0, nC1 = 0;
    if (most > TB_ROW) {
        k_long_rows<<<grid_for(nc, 256), 256, 0, c.s>>>(nc, cdeg, listC1, listC, listC2, listC3, listD, lcount);
        GP_LAUNCHED(c);
        GP_CUDA(cudaMemcpyAsync(c.h_pinned, lcount, 6 * sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
        c.sync();
        nC = c.h_pinned[0]; nD = c.h_pinned[1]; nC2 = c.h_pinned[3]; nC3 = c.h_pinned[4]; nC1 = c.h_pinned[5];
    }
    // one CTA per row: the block scheduler balances rows of unequal length
    if (nC2 > c.sm_count) listC2 = longest_first(c, listC2, nC2, cdeg, TC2_ROW);
    if (nC3 > c.sm_count) listC3 = longest_first(c, listC3, nC3, cdeg, TC3_ROW);
    auto cta_tier = [&](auto kernel, const int32_t* list, int64_t nl, int T, size_t smem) {
        kernel<<<(unsigned)std::min<int64_t>(nl, (int64_t)c.sm_count * c.ctas_per_sm), T, smem, c.s>>>(
            g, fine.cmap, mem, list, nl, off, cdeg, tci, tew, rowcnt, err);
        GP_LAUNCHED(c);
    };
    if (nC1 > 0) {
        if (slot_fits<TC1_PB>(nc)) cta_tier(k_dedup_cta_smem<TC1_T, TC1_SLOTS, TC1_ROW, TC1_PB>, listC1, nC1, TC1_T, cta_dedup_smem<TC1_SLOTS, TC1_ROW, TC1_PB>());
        else cta_tier(k_dedup_cta_smem<TC1_T, TC1_SLOTS, TC1_ROW, 0>, listC1, nC1, TC1_T, cta_dedup_smem<TC1_SLOTS, TC1_ROW, 0>());
    }
    if (nC > 0) {
        if (slot_fits<TC_PB>(nc)) cta_tier(k_dedup_cta_smem<TC_T, TC_SLOTS, TC_ROW, TC_PB>, listC, nC, TC_T, cta_dedup_smem<TC_SLOTS, TC_ROW, TC_PB>());
        else cta_tier(k_dedup_cta_smem<TC_T, TC_SLOTS, TC_ROW, 0>, listC, nC, TC_T, cta_dedup_smem<TC_SLOTS, TC_ROW, 0>());
    }
    if (nC2 > 0) {
        if (slot_fits<TC2_PB>(nc)) cta_tier(k_dedup_cta_smem<TC2_T, TC2_SLOTS, TC2_ROW, TC2_PB>, listC2, nC2, TC2_T, cta_dedup_smem<TC2_SLOTS, TC2_ROW, TC2_PB>());
        else cta_tier(k_dedup_cta_smem<TC2_T, TC2_SLOTS, TC2_ROW, 0>, listC2, nC2, TC2_T, cta_dedup_smem<TC2_SLOTS, TC2_ROW, 0>());
    }
    if (nC3 > 0) {
        // key and weight of each first occurrence are parked at its walk position
        // in mapped / mw (free at these rows: only tier-D rows use them otherwise)
        const bool fits = slot_fits<TC3_PB>(nc);
        (fits ? k_dedup_multipass<TC3_PB> : k_dedup_multipass<0>)<<<
            (unsigned)std::min<int64_t>(nC3, (int64_t)c.sm_count * c.ctas_per_sm), TC2_T,
            fits ? tc3_smem<TC3_PB>() : tc3_smem<0>(), c.s>>>(g, nc, fine.cmap, mem, listC3, nC3, off, cdeg, mapped, mw,
                                                              tci, tew, rowcnt, err);
        GP_LAUNCHED(c);
    }
    if (nD > 0) {
        // row lengths to the host: tables, word ranges and pieces
        int64_t* d_deg = c.tmp_alloc<int64_t>(nD);
        k_td_rows<<<grid_for(nD, 256), 256, 0, c.s>>>(listD, nD, cdeg, d_deg);
        GP_LAUNCHED(c);
        std::vector<int64_t> hdeg((size_t)nD);
        std::vector<int32_t> hlist((size_t)nD);
        GP_CUDA(cudaMemcpyAsync(hdeg.data(), d_deg, sizeof(int64_t) * nD, cudaMemcpyDeviceToHost, c.s));
        GP_CUDA(cudaMemcpyAsync(hlist.data(), listD, sizeof(int32_t) * nD, cudaMemcpyDeviceToHost, c.s));
        c.sync();
        std::vector<int32_t> rlg((size_t)nD), prow;
        std::vector<int64_t> rtab((size_t)nD), rword((size_t)nD), pbeg, pend;
        int64_t tab = 0, words = 0;
        for (int64_t r = 0; r < nD; ++r) {
            int64_t S = 2;
            int lg = 1;
            while (S < 2 * hdeg[r]) { S <<= 1; ++lg; }
            rlg[r] = lg; rtab[r] = tab; rword[r] = words;
            tab += S;
            words += (hdeg[r] + 31) / 32;
            for (int64_t b = 0; b < hdeg[r]; b += TD_PIECE) {
                prow.push_back((int32_t)r);
                pbeg.push_back(b);
                pend.push_back(std::min<int64_t>(b + TD_PIECE, hdeg[r]));
            }
        }
        const int64_t np = (int64_t)prow.size();
        TierD D;
        int32_t* d_rc = c.tmp_alloc<int32_t>(nD);
        int32_t* d_rlg = c.tmp_alloc<int32_t>(nD);
        int64_t* d_rtab = c.tmp_alloc<int64_t>(nD);
        int64_t* d_rword = c.tmp_alloc<int64_t>(nD);
        int32_t* d_prow = c.tmp_alloc<int32_t>(np);
        int64_t* d_pbeg = c.tmp_alloc<int64_t>(np);
        int64_t* d_pend = c.tmp_alloc<int64_t>(np);
        GP_CUDA(cudaMemcpyAsync(d_rc, hlist.data(), sizeof(int32_t) * nD, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_rlg, rlg.data(), sizeof(int32_t) * nD, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_rtab, rtab.data(), sizeof(int64_t) * nD, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_rword, rword.data(), sizeof(int64_t) * nD, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_prow, prow.data(), sizeof(int32_t) * np, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_pbeg, pbeg.data(), sizeof(int64_t) * np, cudaMemcpyHostToDevice, c.s));
        GP_CUDA(cudaMemcpyAsync(d_pend, pend.data(), sizeof(int64_t) * np, cudaMemcpyHostToDevice, c.s));
        D.rc = d_rc; D.rlg = d_rlg; D.rtab = d_rtab; D.rword = d_rword;
        D.prow = d_prow; D.pbeg = d_pbeg; D.pend = d_pend;
        D.slot = c.tmp_alloc<unsigned long long>(tab);
        D.wsum = c.tmp_alloc<int32_t>(tab);
        D.bits = (uint32_t*)c.tmp_alloc<int32_t>(words);
        D.wcnt = c.tmp_alloc<int32_t>(words);
        int64_t* wpre = c.tmp_alloc<int64_t>(words + 1);
        D.wpre = wpre;
        GP_CUDA(cudaMemsetAsync(D.slot, 0, sizeof(unsigned long long) * tab, c.s));
        GP_CUDA(cudaMemsetAsync(D.wsum, 0, sizeof(int32_t) * tab, c.s));
        k_fill_walk_d<<<(unsigned)np, TD_T, 0, c.s>>>(D, g, fine.cmap, mem, off, mapped, mw);
        GP_LAUNCHED(c);
        k_td_insert<<<(unsigned)np, TD_T, 0, c.s>>>(D, off, cdeg, mapped, mw, err);
        GP_LAUNCHED(c);
        k_td_flags<<<(unsigned)np, TD_T, 0, c.s>>>(D, off, cdeg, mapped);
        GP_LAUNCHED(c);
        scan_excl_i32_to_i64(c, D.wcnt, wpre, words, wpre + words);
        k_td_write<<<(unsigned)np, TD_T, 0, c.s>>>(D, off, cdeg, mapped, tci, tew, rowcnt);
        GP_LAUNCHED(c);
    }
    scan_excl_i32_to_i64(c, rowcnt, crp, nc, crp + nc);
    GP_CUDA(cudaMemcpyAsync(ctl + C_MC, crp + nc, sizeof(int64_t), cudaMemcpyDeviceToDevice, c.s));
    // the coarse rows' buckets, then everything the host needs in one read
    buckets_begin(c, coarse, std::max<int64_t>(1, g.m / coarse.heavy_deg + 1), ctl);
    GP_CUDA(cudaMemcpyAsync(c.h_pinned, ctl, C_NCTL * sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
    c.sync();
    int64_t h[C_NCTL];
    std::copy(c.h_pinned, c.h_pinned + C_NCTL, h);
    const int64_t mc = h[C_MC];
    if ((int32_t)h[C_ERR] != 0) throw GpError(GP_EINTERNAL, "contraction hash table overflow");
    int32_t* cci = c.keep_alloc<int32_t>(mc);
    int32_t* cew = c.keep_alloc<int32_t>(mc);
    const int64_t cslice = csr_slice(mc, c.sm_count);
    k_contract_copy<<<grid_for((mc + cslice - 1) / cslice * 32, 256, c.sm_count * c.ctas_per_sm), 256, 0, c.s>>>(
        nc, mc, cslice, off, crp, tci, tew, cci, cew);
    GP_LAUNCHED(c);
    // rows read twice (count and rank for long rows), cmap gathered per entry,
    // unique entries written to the temporary and copied once
    c.bytes += 2 * (8 * (g.n + 1) + 8 * g.m) + 4 * g.m + 8 * (nc + 1) + 4 * nc + 24 * mc + 24 * nc;
    coarse.g.m = mc;
    coarse.g.ci = cci;
    coarse.g.ew = cew;
    coarse.max_vw = h[C_MAXVW];
    c.tmp->restore(mk);
    buckets_end(c, coarse, h, true);
}

// shared-memory caps of the contraction kernels above 48 KB; set once per
// device (the cap is per kernel and shared by every thread of the process)
void coarsen_smem_caps() {
    constexpr size_t smA = 8 * warp_dedup_smem<TA_ROW, TA_SLOTS, int32_t>();
    constexpr size_t smA2 = 8 * warp_dedup_smem<TA2_ROW, TA2_SLOTS, int16_t>();
    constexpr size_t smB = TB_WARPS * warp_dedup_smem<TB_ROW, TB_SLOTS, int16_t>();
    GP_CUDA(cudaFuncSetAttribute(k_dedup_warp<TA_ROW, TA_SLOTS, 8, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smA));
    GP_CUDA(cudaFuncSetAttribute(k_dedup_warp<TA2_ROW, TA2_SLOTS, 8, int16_t>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smA2));
    GP_CUDA(cudaFuncSetAttribute(k_dedup_warp<TB_ROW, TB_SLOTS, TB_WARPS, int16_t>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smB));
    auto big_smem = [](auto kernel, size_t bytes) {
        GP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    };
    big_smem(k_dedup_cta_smem<TC1_T, TC1_SLOTS, TC1_ROW, TC1_PB>, cta_dedup_smem<TC1_SLOTS, TC1_ROW, TC1_PB>());
    big_smem(k_dedup_cta_smem<TC1_T, TC1_SLOTS, TC1_ROW, 0>, cta_dedup_smem<TC1_SLOTS, TC1_ROW, 0>());
    big_smem(k_dedup_cta_smem<TC_T, TC_SLOTS, TC_ROW, TC_PB>, cta_dedup_smem<TC_SLOTS, TC_ROW, TC_PB>());
    big_smem(k_dedup_cta_smem<TC_T, TC_SLOTS, TC_ROW, 0>, cta_dedup_smem<TC_SLOTS, TC_ROW, 0>());
    big_smem(k_dedup_cta_smem<TC2_T, TC2_SLOTS, TC2_ROW, TC2_PB>, cta_dedup_smem<TC2_SLOTS, TC2_ROW, TC2_PB>());
    big_smem(k_dedup_cta_smem<TC2_T, TC2_SLOTS, TC2_ROW, 0>, cta_dedup_smem<TC2_SLOTS, TC2_ROW, 0>());
    big_smem(k_dedup_multipass<TC3_PB>, tc3_smem<TC3_PB>());
    big_smem(k_dedup_multipass<0>, tc3_smem<0>());
}

}  // namespace gp
