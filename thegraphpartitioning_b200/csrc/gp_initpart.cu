// gp_initpart.cu -- GPU initial partition of the coarsest graph.
//
// Replaces convertCSRtoMETISandRun + the `gpmetis -ptype=rb` subprocess and the
// partition-file read-back (src/gpu_part.cu:803-864, 1157-1185).  One CTA runs
// one seeded trial of recursive bisection entirely on chip-resident control
// state: at each depth every label with more than one part is split by
//   1. seed = vertex of the label with the smallest (top-32 hash bits, id),
//   2. BFS inside the label from the seed; the farthest vertex (smallest id on
//      ties) becomes the pseudo-peripheral start,
//   3. BFS from the start; vertices are ordered by (distance, id), unreached
//      ones last,
//   4. the left side is the longest prefix of that order whose weight is at
//      most target = W_label * left_parts / parts, plus the next vertex when
//      that lands strictly closer to the target.
// The prefix is found without sorting: a per-label binary search over the key
// domain (distance * n + id) with shared-memory weight sums.  Labels are part
// ranges identified by their first part.  Trials run in parallel, one per CTA;
// the kept trial is the balanced one with the lowest cut (lowest trial id on
// ties), else the one with the smallest heaviest part.
#define GP_TU_ID 3   // site ids of the bounds-checked build
#include "gp_internal.cuh"

namespace gp {

constexpr int IP_T = 1024;
constexpr int32_t IP_INF = 0x7fffffff;

struct IpShared {
    int32_t* cnt;     // parts per label (label = first part)
    int32_t* cnt_d;   // snapshot at the start of a depth
    int32_t* incl;
    int64_t* WL;
    int64_t* target;
    uint64_t* s0;
    uint64_t* pk;
    int64_t* lo;
    int64_t* hi;
    int64_t* flo;
    int64_t* fsum;
    int64_t* xw;
};

// Adds w to sum[L] for every lane of the warp, one shared-memory atomic per
// distinct label in the warp (lanes of one label are combined by match_any +
// reduce).  L < 0: the lane adds nothing.  Exact: a label's weights total at
// most the graph's vertex weight, which fits in 32 bits.
__device__ __forceinline__ void ip_label_add(int64_t* sum, int32_t L, uint32_t w) {
    const uint32_t peers = __match_any_sync(0xffffffffu, (uint32_t)L);
    const uint32_t tot = __reduce_add_sync(peers, L >= 0 ? w : 0u);
    const int lane = threadIdx.x & 31;
    if (L >= 0 && lane == __ffs(peers) - 1 && tot) atomicAdd((unsigned long long*)&sum[L], (unsigned long long)tot);
}

// atomicMin (MAX = false) or atomicMax (MAX = true) of 64-bit keys into
// slot[L], one shared-memory atomic per distinct label in the warp.  L < 0:
// the lane takes no part.
template <bool MAX>
__device__ __forceinline__ void ip_label_ext(uint64_t* slot, int32_t L, uint64_t key) {
    const uint32_t peers = __match_any_sync(0xffffffffu, (uint32_t)L);
    const uint32_t hi = (uint32_t)(key >> 32), lo = (uint32_t)key;
    const uint32_t ident = MAX ? 0u : 0xffffffffu;
    const uint32_t bh = MAX ? __reduce_max_sync(peers, L >= 0 ? hi : ident) : __reduce_min_sync(peers, L >= 0 ? hi : ident);
    const uint32_t cand = (L >= 0 && hi == bh) ? lo : ident;
    const uint32_t bl = MAX ? __reduce_max_sync(peers, cand) : __reduce_min_sync(peers, cand);
    const int lane = threadIdx.x & 31;
    if (L >= 0 && lane == __ffs(peers) - 1) {
        const unsigned long long best = ((unsigned long long)bh << 32) | bl;
        if (MAX) atomicMax((unsigned long long*)&slot[L], best);
        else atomicMin((unsigned long long*)&slot[L], best);
    }
}

__device__ __forceinline__ int64_t ip_key(int32_t d, int64_t v, int64_t n) {
    return (int64_t)(d == IP_INF ? n : d) * n + v;
}

// BFS inside each splitting label from src (stored as vertex id in srcs[label]);
// dist[] must be IP_INF for all vertices of splitting labels except sources.
__device__ void ip_bfs(const DGraph& g, const int32_t* lab, int32_t* dist, const IpShared& S, int* flags) {
    const int64_t n = g.n;
    if (threadIdx.x == 0) { flags[0] = 0; flags[1] = 0; flags[2] = 0; }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int32_t r = 0;; ++r) {
        // one warp per frontier vertex: rows of the coarsest graph can be long
        for (int64_t v = wid; v < n; v += nw) {
            const int32_t L = lab[v];
            if (S.cnt_d[L] <= 1 || dist[v] != r) continue;
            for (int64_t e = g.rp[v] + lane; e < g.rp[v + 1]; e += 32) {
                const int32_t u = g.ci[e];
                if (lab[u] == L && dist[u] == IP_INF) { dist[u] = r + 1; flags[r % 3] = 1; }
            }
        }
        if (threadIdx.x == 0) flags[(r + 1) % 3] = 0;
        __syncthreads();
        if (!flags[r % 3]) break;
    }
    __syncthreads();
}

// Trials of graphs too large for k_initpart_chip (coarsening that stalled
// above 65,534 vertices, or no room for its shared-memory state): labels and
// distances in the trial's slices of the global arrays.  What bounds it is the
// latency of its sweeps over all vertices, so two blocks per SM (32 registers) pay
// when there are more trials than SMs: 256 trials of a Chung-Lu graph of 30,700
// vertices, k = 1000, 284 ms against 441 with one block of 58 registers.
__global__ void __launch_bounds__(IP_T) k_initpart(DGraph g, int32_t k, uint64_t seed, int32_t* __restrict__ labels,
                                                    int32_t* __restrict__ dists, int64_t* __restrict__ tcut,
                                                    int64_t* __restrict__ tmaxpw, int key_iters) {
    extern __shared__ int64_t ipsm[];
    __shared__ int flags[3];
    __shared__ int any;
    __shared__ int64_t red[IP_T / 32];
    const int64_t n = g.n;
    const int t = blockIdx.x;
    IpShared S;
    {
        int64_t* p = ipsm;
        S.WL = p; p += k; S.target = p; p += k; S.lo = p; p += k; S.hi = p; p += k;
        S.flo = p; p += k; S.fsum = p; p += k; S.xw = p; p += k;
        S.s0 = (uint64_t*)p; p += k; S.pk = (uint64_t*)p; p += k;
        int32_t* q = (int32_t*)p;
        S.cnt = q; q += k; S.cnt_d = q; q += k; S.incl = q; q += k;
    }
    int32_t* lab = labels + (int64_t)t * n;
    int32_t* dist = dists + (int64_t)t * n;
    // two opaque pointers: the compiler otherwise keeps addresses derived from both
    // arrays per loop and spills 100 bytes at 32 registers (the trial above, 64 times:
    // 250 ms instead of 233; random geometric, 68,672 vertices, k = 8: 1375
    // instead of 1250)
    asm volatile("" : "+l"(lab), "+l"(dist));
    const uint64_t ts = trial_salt(seed, t);
    for (int64_t v = threadIdx.x; v < n; v += blockDim.x) lab[v] = 0;
    for (int q = threadIdx.x; q < k; q += blockDim.x) S.cnt[q] = (q == 0) ? k : 0;
    __syncthreads();
    for (int d = 0;; ++d) {
        if (threadIdx.x == 0) any = 0;
        __syncthreads();
        for (int q = threadIdx.x; q < k; q += blockDim.x) {
            S.cnt_d[q] = S.cnt[q];
            if (S.cnt[q] > 1) any = 1;
            S.WL[q] = 0; S.s0[q] = ~0ull; S.pk[q] = 0;
        }
        __syncthreads();
        if (!any) break;
        const uint64_t ds = depth_salt(ts, d);
        // label weights and seeds (warp-uniform trip count for the label sums)
        for (int64_t v0 = threadIdx.x & ~31; v0 < n; v0 += blockDim.x) {
            const int64_t v = v0 + (threadIdx.x & 31);
            int32_t L = v < n ? lab[v] : -1;
            if (L >= 0 && S.cnt_d[L] <= 1) L = -1;
            ip_label_add(S.WL, L, L >= 0 ? (uint32_t)(g.vw ? g.vw[v] : 1) : 0u);
            const uint64_t h = L >= 0 ? (((mix64(ds ^ (uint64_t)(uint32_t)v) >> 32) << 32) | (uint32_t)v) : ~0ull;
            ip_label_ext<false>(S.s0, L, h);
        }
        __syncthreads();
        // BFS 1 from the seed
        for (int64_t v = threadIdx.x; v < n; v += blockDim.x) {
            const int32_t L = lab[v];
            if (S.cnt_d[L] <= 1) continue;
            dist[v] = ((S.s0[L] & 0xffffffffull) == (uint64_t)v) ? 0 : IP_INF;
        }
        __syncthreads();
        ip_bfs(g, lab, dist, S, flags);
        // pseudo-peripheral vertex: max distance, smallest id
        for (int64_t v0 = threadIdx.x & ~31; v0 < n; v0 += blockDim.x) {
            const int64_t v = v0 + (threadIdx.x & 31);
            int32_t L = v < n ? lab[v] : -1;
            if (L >= 0 && (S.cnt_d[L] <= 1 || dist[v] == IP_INF)) L = -1;
            const uint64_t key = L >= 0 ? (((uint64_t)(uint32_t)dist[v] << 32) | (uint64_t)(0xffffffffu - (uint32_t)v)) : 0ull;
            ip_label_ext<true>(S.pk, L, key);
        }
        __syncthreads();
        for (int64_t v = threadIdx.x; v < n; v += blockDim.x) {
            const int32_t L = lab[v];
            if (S.cnt_d[L] <= 1) continue;
            const uint32_t src = 0xffffffffu - (uint32_t)(S.pk[L] & 0xffffffffull);
            dist[v] = ((uint32_t)v == src) ? 0 : IP_INF;
        }
        __syncthreads();
        ip_bfs(g, lab, dist, S, flags);
        // binary search of the split key per label
        for (int q = threadIdx.x; q < k; q += blockDim.x) {
            const int32_t c = S.cnt_d[q];
            if (c > 1) {
                S.target[q] = S.WL[q] * (c / 2) / c;
                S.lo[q] = 0; S.hi[q] = n * (n + 1); S.flo[q] = 0; S.xw[q] = 0;
            }
        }
        __syncthreads();
        for (int it = 0; it < key_iters; ++it) {
            for (int q = threadIdx.x; q < k; q += blockDim.x) S.fsum[q] = 0;
            __syncthreads();
            for (int64_t v0 = threadIdx.x & ~31; v0 < n; v0 += blockDim.x) {
                const int64_t v = v0 + (threadIdx.x & 31);
                int32_t L = v < n ? lab[v] : -1;
                if (L >= 0 && S.cnt_d[L] <= 1) L = -1;
                bool below = false;
                if (L >= 0) below = ip_key(dist[v], v, n) < ((S.lo[L] + S.hi[L]) >> 1);
                ip_label_add(S.fsum, below ? L : -1, below ? (uint32_t)(g.vw ? g.vw[v] : 1) : 0u);
            }
            __syncthreads();
            for (int q = threadIdx.x; q < k; q += blockDim.x) {
                if (S.cnt_d[q] <= 1 || S.hi[q] - S.lo[q] <= 1) continue;
                const int64_t mid = (S.lo[q] + S.hi[q]) >> 1;
                if (S.fsum[q] <= S.target[q]) { S.lo[q] = mid; S.flo[q] = S.fsum[q]; }
                else S.hi[q] = mid;
            }
            __syncthreads();
        }
        for (int64_t v = threadIdx.x; v < n; v += blockDim.x) {
            const int32_t L = lab[v];
            if (S.cnt_d[L] <= 1) continue;
            if (ip_key(dist[v], v, n) == S.lo[L]) S.xw[L] = g.vw ? g.vw[v] : 1;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < k; q += blockDim.x) {
            const int32_t c = S.cnt_d[q];
            if (c > 1) {
                S.incl[q] = (S.xw[q] > 0 && 2 * S.target[q] > 2 * S.flo[q] + S.xw[q]) ? 1 : 0;
                S.cnt[q] = c / 2;
                S.cnt[q + c / 2] = c - c / 2;
            }
        }
        __syncthreads();
        for (int64_t v = threadIdx.x; v < n; v += blockDim.x) {
            const int32_t L = lab[v];
            const int32_t c = S.cnt_d[L];
            if (c <= 1) continue;
            const int64_t key = ip_key(dist[v], v, n);
            const bool left = key < S.lo[L] || (key == S.lo[L] && S.incl[L]);
            if (!left) lab[v] = L + c / 2;
        }
        __syncthreads();
    }
    // evaluate the trial: cut and heaviest part
    for (int q = threadIdx.x; q < k; q += blockDim.x) S.WL[q] = 0;
    __syncthreads();
    int64_t cross = 0;
    {
        const int lane = threadIdx.x & 31;
        for (int64_t v = threadIdx.x >> 5; v < n; v += blockDim.x >> 5) {
            const int32_t p = lab[v];
            if (lane == 0) atomicAdd((unsigned long long*)&S.WL[p], (unsigned long long)(g.vw ? g.vw[v] : 1));
            for (int64_t e = g.rp[v] + lane; e < g.rp[v + 1]; e += 32)
                if (lab[g.ci[e]] != p) cross += g.ew ? g.ew[e] : 1;
        }
    }
    for (int o = 16; o > 0; o >>= 1) cross += __shfl_xor_sync(0xffffffffu, cross, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cross;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int i = 0; i < IP_T / 32; ++i) s += red[i];
        int64_t mp = 0;
        for (int q = 0; q < k; ++q) mp = S.WL[q] > mp ? S.WL[q] : mp;
        tcut[t] = s;
        tmaxpw[t] = mp;
    }
}

// ------------------------------------------------------------------ on-chip trials
// The same trial with its whole state in shared memory (k_initpart_chip):
// one 32-bit word per vertex (label << 16 | BFS distance, 0xFFFF: unreached),
// a BFS queue and a work list of 16-bit ids.  What bounds it is the chain of
// BFS levels (two barriers and the row loads of one frontier each), so the
// work per level is the frontier's rows only, not a sweep over all vertices:
//  - top-down levels expand the queue's frontier, a group of `tile` lanes per
//    vertex (8, 16 or 32 by the mean degree); on graphs of a mean degree of
//    32 and more a level whose frontier F is large runs bottom-up instead
//    (every unreached vertex scans its row until it meets the frontier): about
//    n / F entries per unreached vertex against F whole rows, so bottom-up
//    when unreached * n < F * F * degree.  Its rows are the frontier's mirrored,
//    so only on graphs that pass the symmetry fingerprint;
//  - the second BFS sums each label's frontier weight level by level, which
//    gives the distance at which the label's target weight is crossed, and
//    stops there; the crossing vertex among that distance's vertices (in id
//    order) is found by a 16-way search over ids, at most four rounds;
//  - label weights are carried from split to split instead of summed anew.
// CSR_SM: rows (32-bit starts, 16-bit ids) are copied to shared memory first,
// which takes the L2 latency out of every level; taken when they fit.
// 64 trials on a B200, this kernel against one whose BFS levels sweep every
// vertex and whose split key takes a binary search over (distance, id):
// 823 vertices k = 8 893 -> 143 us, random geometric 8,864 vertices k = 300
// 44.0 -> 1.5 ms, Chung-Lu 1,789 vertices k = 64 5.4 -> 1.7 ms, R-MAT (dense)
// 1,999 vertices k = 64 11.2 -> 3.5 ms; the last two 0.91 and 1.38 ms with the cuts
// in k_trial_cuts and NB = 4 entries of a lane in flight.  NB = 4 from a mean
// degree of 32 on rows in L2; on the random geometric graph (degree 12) it takes
// 1.8 ms.
constexpr int32_t IPC_FAR = 0xFFFF;    // unreached / no crossing distance below it
constexpr int IPC_BINS = 16;

struct IpcLabels {
    int32_t* cnt;      // parts of the label
    int32_t* cnt_d;    // snapshot at the start of a depth
    int32_t* W;        // weight
    int32_t* target;   // weight wanted on the left
    int32_t* cum;      // weight below the current distance / below the crossing vertex
    int32_t* wlev;     // weight at the current distance
    int32_t* crit;     // crossing distance (-1: not found yet, IPC_FAR: among the unreached)
    int32_t* lo;       // id search range [lo, hi); lo ends as the crossing vertex
    int32_t* hi;
    int32_t* incl;     // crossing vertex goes left
    uint32_t* pk;      // farthest vertex: distance << 16 | 0xFFFF - id
    int32_t* hist;     // IPC_BINS weights
    uint64_t* s0;      // seed: top-32 hash << 32 | id
};
constexpr size_t ipc_label_bytes() { return sizeof(int32_t) * (11 + IPC_BINS) + sizeof(uint64_t); }

// shared counters of one trial
struct IpcShared {
    int32_t tail, nlist, nact, any;
    int64_t red[32];
};

template <bool CSR_SM>
struct IpcRows {
    const int64_t* rp;
    const int32_t* ci;
    const uint32_t* srp;
    const uint16_t* sci;
    __device__ __forceinline__ int64_t beg(int32_t v) const { return CSR_SM ? (int64_t)srp[v] : rp[v]; }
    __device__ __forceinline__ int32_t id(int64_t e) const { return CSR_SM ? (int32_t)sci[e] : ci[e]; }
};

// appends of the calling lanes (any subset of a warp): one shared atomic per warp
__device__ __forceinline__ int32_t ipc_slot(int32_t* counter) {
    const uint32_t m = __activemask();
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    int32_t base = 0;
    if (lane == lead) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(m, base, lead);
    return base + __popc(m & ((1u << lane) - 1u));
}

// BFS inside every splitting label from the sources queued at [0, tail) with
// distance 0.  CROSS: track the crossing distances and stop once every
// splitting label has one.  nv: vertices of splitting labels.
template <bool CSR_SM, bool CROSS, int NB>
__device__ void ipc_bfs(const DGraph& g, const IpcRows<CSR_SM>& R, uint32_t* state, uint16_t* queue, uint16_t* list,
                        const IpcLabels& S, IpcShared& sh, int32_t k, int32_t nv, int tile, int64_t davg) {
    const int32_t n = (int32_t)g.n;
    const int lane = threadIdx.x & 31;
    const int tl = threadIdx.x & (tile - 1);
    const int32_t grp = threadIdx.x / tile, ngrp = blockDim.x / tile;
    int32_t h = 0, t = sh.tail;
    __syncthreads();
    for (int32_t r = 0; h < t; ++r) {
        const int64_t F = t - h, U = nv - t;
        const bool up = davg >= 32 && U * n < F * F * davg;
        if (up) {
            // unreached vertices of labels still searching
            for (int32_t v = threadIdx.x; v < n; v += blockDim.x) {
                const uint32_t s = state[v];
                const int32_t L = (int32_t)(s >> 16);
                if ((s & 0xFFFFu) == (uint32_t)IPC_FAR && S.cnt_d[L] > 1 && (!CROSS || S.crit[L] < 0))
                    list[ipc_slot(&sh.nlist)] = (uint16_t)v;
            }
            if (CROSS)
                for (int32_t i = h + threadIdx.x; i < t; i += blockDim.x) {
                    const int32_t v = queue[i];
                    const int32_t L = (int32_t)(state[v] >> 16);
                    if (S.crit[L] < 0) atomicAdd(&S.wlev[L], g.vw ? g.vw[v] : 1);
                }
            __syncthreads();
            const int32_t nl = sh.nlist;
            for (int32_t i = threadIdx.x >> 5; i < nl; i += blockDim.x >> 5) {
                const int32_t v = list[i];
                const uint32_t want = (state[v] & 0xFFFF0000u) | (uint32_t)r;
                const int64_t end = R.beg(v + 1);
                bool hit = false;
                for (int64_t e0 = R.beg(v); e0 < end && !hit; e0 += 32 * NB) {
                    int32_t u[NB];
#pragma unroll
                    for (int b = 0; b < NB; ++b) { const int64_t e = e0 + 32 * b + lane; u[b] = e < end ? R.id(e) : -1; }
                    bool f = false;
#pragma unroll
                    for (int b = 0; b < NB; ++b) f = f || (u[b] >= 0 && GP_IN(u[b], n) && state[u[b]] == want);
                    hit = __any_sync(0xffffffffu, f);
                }
                if (hit && lane == 0) {
                    state[v] = want + 1u;
                    queue[atomicAdd(&sh.tail, 1)] = (uint16_t)v;
                }
            }
        } else {
            for (int32_t i = h + grp; i < t; i += ngrp) {
                const int32_t v = queue[i];
                const uint32_t lab = state[v] & 0xFFFF0000u;
                if (CROSS) {
                    const int32_t L = (int32_t)(lab >> 16);
                    if (S.crit[L] >= 0) continue;
                    if (tl == 0) atomicAdd(&S.wlev[L], g.vw ? g.vw[v] : 1);
                }
                const uint32_t open = lab | (uint32_t)IPC_FAR;
                const int64_t end = R.beg(v + 1);
                for (int64_t e0 = R.beg(v) + tl; e0 < end; e0 += (int64_t)NB * tile) {
                    int32_t u[NB];
#pragma unroll
                    for (int b = 0; b < NB; ++b) { const int64_t e = e0 + b * tile; u[b] = e < end ? R.id(e) : -1; }
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        if (u[b] >= 0 && GP_IN(u[b], n) && state[u[b]] == open &&
                            atomicCAS(&state[u[b]], open, lab | (uint32_t)(r + 1)) == open)
                            queue[ipc_slot(&sh.tail)] = (uint16_t)u[b];
                }
            }
        }
        __syncthreads();
        h = t;
        t = sh.tail;
        if (threadIdx.x == 0) sh.nlist = 0;
        if (CROSS) {
            for (int32_t q = threadIdx.x; q < k; q += blockDim.x) {
                const int32_t w = S.wlev[q];
                if (w == 0) continue;
                S.wlev[q] = 0;
                if (S.cum[q] + w > S.target[q]) { S.crit[q] = r; atomicSub(&sh.nact, 1); }
                else S.cum[q] += w;
            }
        }
        __syncthreads();
        if (CROSS && sh.nact == 0) break;
    }
}

// one trial per CTA; shared memory: ipc_smem(n, m, k, CSR_SM, lists on chip)
template <bool CSR_SM, int NB>
__global__ void __launch_bounds__(IP_T) k_initpart_chip(DGraph g, int32_t k, uint64_t seed, int32_t* __restrict__ labels,
                                                        uint16_t* __restrict__ lists, int64_t* __restrict__ tcut,
                                                        int64_t* __restrict__ tmaxpw, int tile, int cut,
                                                        const int64_t* __restrict__ asym) {
    extern __shared__ __align__(16) unsigned char ipc_raw[];
    __shared__ IpcShared sh;
    const int32_t n = (int32_t)g.n;
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    IpcLabels S;
    S.s0 = (uint64_t*)ipc_raw;
    int32_t* p = (int32_t*)(S.s0 + k);
    S.cnt = p; p += k; S.cnt_d = p; p += k; S.W = p; p += k; S.target = p; p += k; S.cum = p; p += k;
    S.wlev = p; p += k; S.crit = p; p += k; S.lo = p; p += k; S.hi = p; p += k; S.incl = p; p += k;
    S.pk = (uint32_t*)p; p += k;
    S.hist = p; p += (int64_t)IPC_BINS * k;
    uint32_t* state = (uint32_t*)p;
    uint32_t* after = state + n;
    IpcRows<CSR_SM> R{g.rp, g.ci, nullptr, nullptr};
    if (CSR_SM) {
        uint32_t* srp = after;
        after += n + 1;
        uint16_t* sci = (uint16_t*)after;
        after += (g.m + 1) / 2;
        for (int32_t v = threadIdx.x; v <= n; v += blockDim.x) srp[v] = (uint32_t)g.rp[v];
        for (int32_t e = threadIdx.x; e < (int32_t)g.m; e += blockDim.x) sci[e] = (uint16_t)g.ci[e];
        R.srp = srp; R.sci = sci;
    }
    // queue and list: n ids each, on chip unless the caller brings them
    uint16_t* queue = lists ? lists + 2 * (int64_t)t * n : (uint16_t*)after;
    uint16_t* list = queue + n;
    // asym: the level's symmetry_sums (nullptr: known to be symmetric); 0: no level runs bottom-up
    const int64_t davg = !asym || (asym[2] == 0 && asym[3] == 0) ? g.m / (n > 0 ? n : 1) : 0;
    const uint64_t ts = trial_salt(seed, t);
    int64_t wsum = 0;
    for (int32_t v = threadIdx.x; v < n; v += blockDim.x) { state[v] = 0; wsum += g.vw ? g.vw[v] : 1; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if (lane == 0) sh.red[warp] = wsum;
    for (int32_t q = threadIdx.x; q < k; q += blockDim.x) {
        S.cnt[q] = q == 0 ? k : 0;
        S.W[q] = 0; S.wlev[q] = 0;
    }
    for (int32_t i = threadIdx.x; i < IPC_BINS * k; i += blockDim.x) S.hist[i] = 0;
    if (threadIdx.x == 0) sh.nlist = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int i = 0; i < nwarp; ++i) s += sh.red[i];
        S.W[0] = (int32_t)s;   // the total fits in int32 (checked on input)
    }
    int32_t vbits = 1;   // 16-way rounds of the id search: 4 bits each
    while ((1 << vbits) < n) ++vbits;
    for (int d = 0;; ++d) {
        if (threadIdx.x == 0) { sh.any = 0; sh.tail = 0; sh.nact = 0; }
        __syncthreads();
        int32_t mine = 0;
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x) {
            const int32_t c = S.cnt[q];
            S.cnt_d[q] = c;
            S.s0[q] = ~0ull; S.pk[q] = 0;
            if (c > 1) {
                ++mine;
                S.target[q] = (int32_t)((int64_t)S.W[q] * (c / 2) / c);
                S.cum[q] = 0; S.crit[q] = -1; S.lo[q] = 0; S.hi[q] = n;
            }
        }
        if (mine) atomicAdd(&sh.any, mine);
        __syncthreads();
        const int32_t nsplit = sh.any;
        if (nsplit == 0) break;
        const uint64_t ds = depth_salt(ts, d);
        // seeds, and every vertex of a splitting label unreached.  Few labels:
        // one 64-bit atomic per label and warp; many: a plain check keeps most
        // lanes from the atomic
        int32_t myv = 0;
        for (int32_t v0 = threadIdx.x & ~31; v0 < n; v0 += blockDim.x) {
            const int32_t v = v0 + lane;
            int32_t L = v < n ? (int32_t)(state[v] >> 16) : -1;
            if (L >= 0 && S.cnt_d[L] <= 1) L = -1;
            uint64_t key = ~0ull;
            if (L >= 0) {
                state[v] = ((uint32_t)L << 16) | (uint32_t)IPC_FAR;
                key = ((mix64(ds ^ (uint64_t)(uint32_t)v) >> 32) << 32) | (uint32_t)v;
                ++myv;
            }
            if (nsplit <= 4) ip_label_ext<false>(S.s0, L, key);
            else if (L >= 0 && key < S.s0[L]) atomicMin((unsigned long long*)&S.s0[L], (unsigned long long)key);
        }
        myv = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)myv);
        if (lane == 0) sh.red[warp] = myv;
        __syncthreads();
        int32_t nv = 0;
        for (int i = 0; i < nwarp; ++i) nv += (int32_t)sh.red[i];
        // BFS 1 from the seeds
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x)
            if (S.cnt_d[q] > 1 && S.s0[q] != ~0ull) {
                const int32_t v = (int32_t)(uint32_t)S.s0[q];
                state[v] = (uint32_t)q << 16;
                queue[atomicAdd(&sh.tail, 1)] = (uint16_t)v;
            }
        __syncthreads();
        ipc_bfs<CSR_SM, false, NB>(g, R, state, queue, list, S, sh, k, nv, tile, davg);
        // pseudo-peripheral vertex: largest distance, smallest id
        const int32_t reached = sh.tail;
        for (int32_t i0 = threadIdx.x & ~31; i0 < reached; i0 += blockDim.x) {
            const int32_t i = i0 + lane;
            const int32_t v = i < reached ? (int32_t)queue[i] : 0;
            const uint32_t s = state[v];
            const int32_t L = i < reached ? (int32_t)(s >> 16) : -1;
            const uint32_t key = L >= 0 ? ((s & 0xFFFFu) << 16 | (0xFFFFu - (uint32_t)v)) : 0u;
            if (L >= 0 && key > S.pk[L]) atomicMax(&S.pk[L], key);
        }
        __syncthreads();
        for (int32_t v = threadIdx.x; v < n; v += blockDim.x) state[v] |= (uint32_t)IPC_FAR;
        if (threadIdx.x == 0) sh.tail = 0;
        __syncthreads();
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x)
            if (S.cnt_d[q] > 1 && S.s0[q] != ~0ull) {
                const int32_t v = (int32_t)(0xFFFFu - (S.pk[q] & 0xFFFFu));
                state[v] = (uint32_t)q << 16;
                queue[atomicAdd(&sh.tail, 1)] = (uint16_t)v;
                atomicAdd(&sh.nact, 1);
            }
        __syncthreads();
        ipc_bfs<CSR_SM, true, NB>(g, R, state, queue, list, S, sh, k, nv, tile, davg);
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x)
            if (S.cnt_d[q] > 1 && S.crit[q] < 0) S.crit[q] = IPC_FAR;   // its component ended below the target
        __syncthreads();
        // crossing vertex: the first, in id order, of the crossing distance's
        // vertices that takes the label's weight above the target
        for (int32_t v = threadIdx.x; v < n; v += blockDim.x) {
            const uint32_t s = state[v];
            const int32_t L = (int32_t)(s >> 16);
            if (S.cnt_d[L] > 1 && (int32_t)(s & 0xFFFFu) == S.crit[L]) list[ipc_slot(&sh.nlist)] = (uint16_t)v;
        }
        __syncthreads();
        const int32_t nl = sh.nlist;
        for (int32_t b = vbits; b > 0; b -= 4) {
            for (int32_t i = threadIdx.x; i < nl; i += blockDim.x) {
                const int32_t v = list[i];
                const int32_t L = (int32_t)(state[v] >> 16), lo = S.lo[L], hi = S.hi[L];
                if (v < lo || v >= hi) continue;
                const int32_t width = (hi - lo + IPC_BINS - 1) / IPC_BINS;
                atomicAdd(&S.hist[IPC_BINS * L + (v - lo) / width], g.vw ? g.vw[v] : 1);
            }
            __syncthreads();
            if (threadIdx.x == 0) sh.nlist = 0;
            for (int32_t q = threadIdx.x; q < k; q += blockDim.x) {
                if (S.cnt_d[q] <= 1) continue;
                const int32_t lo = S.lo[q], hi = S.hi[q];
                const int32_t width = (hi - lo + IPC_BINS - 1) / IPC_BINS;
                int32_t sum = S.cum[q], at = -1;
                for (int i = 0; i < IPC_BINS; ++i) {
                    const int32_t w = S.hist[IPC_BINS * q + i];
                    S.hist[IPC_BINS * q + i] = 0;
                    if (at < 0) { if (sum + w > S.target[q]) at = i; else sum += w; }
                }
                if (at >= 0) {   // always, unless the label is empty
                    S.cum[q] = sum;
                    S.lo[q] = lo + at * width;
                    S.hi[q] = lo + (at + 1) * width < hi ? lo + (at + 1) * width : hi;
                }
            }
            __syncthreads();
        }
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x) {
            const int32_t c = S.cnt_d[q];
            if (c <= 1) continue;
            const int32_t W = S.W[q], flo = S.cum[q];
            const int32_t xw = W > 0 ? (g.vw ? g.vw[S.lo[q]] : 1) : 0;
            const int32_t in = (xw > 0 && 2 * (int64_t)S.target[q] > 2 * (int64_t)flo + xw) ? 1 : 0;
            S.incl[q] = in;
            const int32_t left = W > 0 ? flo + (in ? xw : 0) : 0;
            S.cnt[q] = c / 2;
            S.cnt[q + c / 2] = c - c / 2;
            S.W[q] = left;
            S.W[q + c / 2] = W - left;
        }
        __syncthreads();
        for (int32_t v = threadIdx.x; v < n; v += blockDim.x) {
            const uint32_t s = state[v];
            const int32_t L = (int32_t)(s >> 16), c = S.cnt_d[L];
            if (c <= 1) continue;
            const int32_t dv = (int32_t)(s & 0xFFFFu), cd = S.crit[L], x = S.lo[L];
            const bool left = dv < cd || (dv == cd && (v < x || (v == x && S.incl[L])));
            if (!left) state[v] = (uint32_t)(L + c / 2) << 16;
        }
        __syncthreads();
    }
    // the trial's cut (cut: 0: k_trial_cuts adds it up) and heaviest part
    int64_t cross = 0;
    const int tl = threadIdx.x & (tile - 1);
    for (int32_t v = cut ? threadIdx.x / tile : n; v < n; v += blockDim.x / tile) {
        const uint32_t pv = state[v] >> 16;
        const int64_t end = R.beg(v + 1);
        for (int64_t e = R.beg(v) + tl; e < end; e += tile) {
            const int32_t u = R.id(e);
            if (GP_IN(u, n) && (state[u] >> 16) != pv) cross += g.ew ? g.ew[e] : 1;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cross += __shfl_xor_sync(0xffffffffu, cross, o);
    int32_t mp = 0;
    for (int32_t q = threadIdx.x; q < k; q += blockDim.x) mp = S.W[q] > mp ? S.W[q] : mp;
    mp = (int32_t)__reduce_max_sync(0xffffffffu, (uint32_t)mp);
    __shared__ int32_t s_mp[32];
    if (lane == 0) { sh.red[warp] = cross; s_mp[warp] = mp; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int i = 0; i < nwarp; ++i) { s += sh.red[i]; mp = s_mp[i] > mp ? s_mp[i] : mp; }
        tcut[t] = s;
        tmaxpw[t] = mp;
    }
    for (int32_t v = threadIdx.x; v < n; v += blockDim.x) labels[(int64_t)t * n + v] = (int32_t)(state[v] >> 16);
}

// Directed cross weights of 16 trials (blockIdx.y) over the rows of blockIdx.x's
// warps: the trials' labels lie in shared memory 16 to a vertex (LT: uint8 for k
// <= 256, else uint16), so an entry and its weight are read once for all of them
// and its neighbour's labels are one or two 16-byte loads.  Inside the trial's own
// block the sweep read every entry per trial, one in flight per lane, on 64 of 148
// SMs: 0.99 of the 2.28 ms of 64 trials on R-MAT's coarsest graph (1,999
// vertices, 2.7 M entries), here 87 us.
constexpr int TC_G = 16;
template <class LT>
__global__ void __launch_bounds__(512) k_trial_cuts(DGraph g, int32_t T, const int32_t* __restrict__ labels,
                                                    unsigned long long* __restrict__ tcut) {
    extern __shared__ __align__(16) unsigned char tc_raw[];
    constexpr int NV = TC_G * sizeof(LT) / 16;   // 16-byte words per vertex
    constexpr int PW = 4 / sizeof(LT);           // labels per 32-bit word
    __shared__ uint32_t s_sum[TC_G];
    LT* lab = (LT*)tc_raw;
    const int32_t n = (int32_t)g.n, t0 = blockIdx.y * TC_G;
    if (threadIdx.x < TC_G) s_sum[threadIdx.x] = 0;
    for (int t = 0; t < TC_G; ++t)
        for (int32_t v = threadIdx.x; v < n; v += blockDim.x)
            lab[(int64_t)v * TC_G + t] = t0 + t < T ? (LT)labels[(int64_t)(t0 + t) * n + v] : (LT)0;
    __syncthreads();
    const uint4* lv = (const uint4*)lab;
    const int lane = threadIdx.x & 31;
    uint32_t acc[TC_G];   // the weights of all entries add up to less than 2^32
#pragma unroll
    for (int t = 0; t < TC_G; ++t) acc[t] = 0;
    const int32_t nw = (int32_t)(gridDim.x * blockDim.x) >> 5;
    for (int32_t v = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        uint4 mine[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) mine[i] = lv[(int64_t)v * NV + i];
        const int64_t end = g.rp[v + 1];
        for (int64_t e0 = g.rp[v] + lane; e0 < end; e0 += 128) {
            int32_t u[4];
            uint32_t w[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int64_t e = e0 + 32 * c;
                u[c] = e < end ? __ldg(&g.ci[e]) : -1;
                w[c] = e < end ? (g.ew ? (uint32_t)__ldg(&g.ew[e]) : 1u) : 0u;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (u[c] < 0 || !GP_IN(u[c], n)) continue;
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    const uint4 o = lv[(int64_t)u[c] * NV + i];
                    const uint32_t x[4] = {o.x ^ mine[i].x, o.y ^ mine[i].y, o.z ^ mine[i].z, o.w ^ mine[i].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int b = 0; b < PW; ++b)
                            acc[(i * 4 + q) * PW + b] += ((x[q] >> (8 * sizeof(LT) * b)) & (LT)~(LT)0) ? w[c] : 0u;
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < TC_G; ++t) {
        const uint32_t x = __reduce_add_sync(0xffffffffu, acc[t]);
        if (lane == 0 && x) atomicAdd(&s_sum[t], x);
    }
    __syncthreads();
    if (threadIdx.x < TC_G && t0 + (int)threadIdx.x < T && s_sum[threadIdx.x])
        atomicAdd(&tcut[t0 + threadIdx.x], (unsigned long long)s_sum[threadIdx.x]);
}

// the kept trial: balanced before not, then (not balanced) the smaller heaviest
// part, then the lower cut, then the lower trial; one warp.  tcut: directed cross
// weights
__global__ void k_pick_trial(int T, const int64_t* __restrict__ tcut, const int64_t* __restrict__ tmaxpw, int64_t Lmax,
                             int64_t* __restrict__ best) {
    const int lane = threadIdx.x & 31;
    int64_t a = INT64_MAX, b = INT64_MAX;   // (max(heaviest, Lmax), cut)
    int bt = INT32_MAX;
    auto take = [&](int64_t a2, int64_t b2, int t2) {
        if (a2 < a || (a2 == a && (b2 < b || (b2 == b && t2 < bt)))) { a = a2; b = b2; bt = t2; }
    };
    for (int t = lane; t < T; t += 32) take(tmaxpw[t] > Lmax ? tmaxpw[t] : Lmax, tcut[t] / 2, t);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int64_t a2 = __shfl_xor_sync(0xffffffffu, a, o), b2 = __shfl_xor_sync(0xffffffffu, b, o);
        const int t2 = __shfl_xor_sync(0xffffffffu, bt, o);
        take(a2, b2, t2);
    }
    if (threadIdx.x == 0) best[0] = bt;
}

static int bits_for64(int64_t x) {
    int b = 1;
    while (b < 63 && (1ll << b) < x) ++b;
    return b;
}

size_t initpart_smem_max();

// entries from which the trials' cuts are added up by k_trial_cuts (a launch of
// 5 us and more; a trial's own sweep takes 0.36 us per 1000 entries)
constexpr int64_t kTrialCuts = 65536;

int initial_partition(Ctx& c, const Level& L, const Params& P, int32_t* part_out) {
    const int64_t n = L.g.n, m = L.g.m;
    const int T = P.o.init_trials;
    auto mk = c.tmp->save();
    int32_t* labels = c.tmp_alloc<int32_t>((int64_t)T * n);
    int64_t* tcut = c.tmp_alloc<int64_t>(T);
    int64_t* tmaxpw = c.tmp_alloc<int64_t>(T);
    int64_t* best = c.tmp_alloc<int64_t>(1);
    const size_t cap = initpart_smem_max();
    // 16-bit ids and distances, state of every vertex on chip: k_initpart_chip
    const size_t chip = (size_t)P.k * ipc_label_bytes() + sizeof(uint32_t) * (size_t)n;
    if (n < IPC_FAR && chip <= cap) {
        const size_t lists = sizeof(uint16_t) * 2 * (size_t)n;
        const size_t csr = sizeof(uint32_t) * (size_t)(n + 1) + sizeof(uint32_t) * (size_t)((m + 1) / 2);
        const bool lists_on = chip + lists <= cap;
        // at most half the block's shared memory for a copy of the rows: two trials stay resident per SM
        const bool csr_on = chip + lists + csr <= cap / 2;
        uint16_t* glists = lists_on ? nullptr : c.tmp_alloc<uint16_t>(2 * (int64_t)T * n);
        const int64_t davg = m / std::max<int64_t>(n, 1);
        const int tile = davg <= 8 ? 8 : (davg <= 16 ? 16 : 32);
        const int threads = (n <= 4096 && m <= 65536) ? IP_T / 2 : IP_T;
        const size_t smem = chip + (lists_on ? lists : 0) + (csr_on ? csr : 0);
        // cuts of all trials together: rows in L2, labels of 16 trials on chip
        const size_t lab = (size_t)n * TC_G * (P.k <= 256 ? 1 : 2);
        // (16 trials per row of the grid, which has at most 65,535 rows)
        const bool cuts = !csr_on && m >= kTrialCuts && lab <= cap && T <= 65535 * TC_G;
        auto kernel = csr_on ? k_initpart_chip<true, 1> : (davg >= 32 ? k_initpart_chip<false, 4> : k_initpart_chip<false, 1>);
        // an input that was not checked, or is not symmetric: look at this level (21 us on
        // 2.7 M entries, where searches without bottom-up levels take 2.9 ms more)
        int64_t* asym = nullptr;
        if (davg >= 32 && !P.symmetric) {
            asym = c.tmp_alloc<int64_t>(5);
            symmetry_sums(c, L.g, asym);
        }
        kernel<<<T, threads, smem, c.s>>>(L.g, P.k, P.seed, labels, glists, tcut, tmaxpw, tile, cuts ? 0 : 1, asym);
        GP_LAUNCHED(c);
        if (cuts) {
            const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(c.sm_count * TC_G / T + 1, (n + 15) / 16)),
                            (unsigned)((T + TC_G - 1) / TC_G));
            (P.k <= 256 ? k_trial_cuts<uint8_t> : k_trial_cuts<uint16_t>)<<<grid, 512, lab, c.s>>>(
                L.g, T, labels, (unsigned long long*)tcut);
            GP_LAUNCHED(c);
        }
    } else {
        int32_t* dists = c.tmp_alloc<int32_t>((int64_t)T * n);
        const size_t base = (size_t)P.k * (9 * sizeof(int64_t) + 3 * sizeof(int32_t));
        const int key_iters = bits_for64(n * (n + 1)) + 1;
        k_initpart<<<T, IP_T, base, c.s>>>(L.g, P.k, P.seed, labels, dists, tcut, tmaxpw, key_iters);
        GP_LAUNCHED(c);
    }
    k_pick_trial<<<1, 32, 0, c.s>>>(T, tcut, tmaxpw, P.Lmax, best);
    GP_LAUNCHED(c);
    const int bt = (int)read_i64(c, best);
    GP_CUDA(cudaMemcpyAsync(part_out, labels + (int64_t)bt * n, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, c.s));
    c.bytes += (int64_t)T * (L.scan_bytes() * 4 + 8 * n);
    c.tmp->restore(mk);
    return bt;
}

// the trials' kernels may use the whole opt-in shared memory of a block (per-label
// arrays; in k_initpart_chip also the vertices' state, lists and rows that fit); set
// once per device (the cap is per kernel, shared by every thread of the process)
static size_t g_ip_smem_max = 0;

size_t initpart_smem_max() { return g_ip_smem_max; }

void initpart_smem_caps() {
    int dev = 0, optin = 0;
    GP_CUDA(cudaGetDevice(&dev));
    GP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t need = (size_t)GP_MAX_K * (9 * sizeof(int64_t) + 3 * sizeof(int32_t));
    // static shared memory of the kernel (flags, reductions) stays outside the cap
    const size_t cap = std::max(need, (size_t)optin > 4096 ? (size_t)optin - 4096 : need);
    GP_CUDA(cudaFuncSetAttribute(k_initpart, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    GP_CUDA(cudaFuncSetAttribute(k_trial_cuts<uint8_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    GP_CUDA(cudaFuncSetAttribute(k_trial_cuts<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    GP_CUDA(cudaFuncSetAttribute(k_initpart_chip<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    GP_CUDA(cudaFuncSetAttribute(k_initpart_chip<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    GP_CUDA(cudaFuncSetAttribute(k_initpart_chip<false, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    g_ip_smem_max = cap;
}

}  // namespace gp
