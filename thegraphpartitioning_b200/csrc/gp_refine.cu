// gp_refine.cu -- gain refinement, rebalancing and projection.
//
// Replaces deterministicRefinement (src/gpu_part.cu:509-759) with its kernels
// computeGainsAndDestinations, markCandidates, tokenPassing,
// bufferCandidateMoves, computeAvailableCapacity, bitonicSortStep/customSortMoves,
// selectMoves, commitMoves (src/gpu_part.cu:258-397, 472-506), the edge-cut
// kernel (src/gpu_part.cu:400-423) and kwayMapCoarseToFine (src/gpu_part.cu:763-772).
//
// One refinement iteration:
//   k_conn      one pass over every row: exact int32 part-connectivity histogram
//               in shared memory (warp-private for rows <= kHeavyDeg, CTA-wide
//               for longer rows), cut contribution of every vertex (so the cut
//               of the current state costs no extra pass), and the move proposal
//               of the mode the device derives from the part weights
//               (label propagation when no part exceeds Lmax, else rebalancing).
//   LP:         k_lp_apply (the connectivity pass already copied part/lock into
//               the next buffers): each candidate re-evaluates its gain
//               against the proposals of higher-priority neighbours
//               ((gain desc, id asc)) and moves when that gain is >= 0;
//               double-buffered part/lock arrays, part-weight deltas aggregated
//               per CTA in shared memory.
//   rebalance:  candidates (keys = source | loss bucket | id) are radix sorted,
//               exclusive prefix sums of vertex weight select the moves that
//               cover each source's excess and fit each destination's capacity
//               (weak) or the concatenated free capacities (strong).
#define GP_TU_ID 4   // site ids of the bounds-checked build
#include "gp_internal.cuh"

#include <cstring>
#include <mutex>

namespace gp {

constexpr int RT = 256;              // threads per CTA
constexpr int RW = RT / 32;          // warps per CTA
enum { MODE_LP = 0, MODE_RB = 1, MODE_EVAL = 2 };

__device__ __forceinline__ void argmax_q(uint64_t& bk, int32_t& bq, uint64_t k2, int32_t q2) {
    if (k2 > bk || (k2 == bk && (uint32_t)q2 < (uint32_t)bq)) { bk = k2; bq = q2; }
}
__device__ __forceinline__ void warp_argmax_q(uint64_t& bk, int32_t& bq) { group_argmax64(0xffffffffu, bk, bq); }
template <class T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Argmax over a lane group of (connectivity h > 0, part q): largest h, ties
// to the smaller q; h = 0 means "no candidate" and yields (0, -1).  Two
// redux.sync steps replace the shuffle tree (connectivities fit in 32 bits).
__device__ __forceinline__ void group_argmax_u32(uint32_t mask, uint64_t& bk, int32_t& bq, uint32_t h, int32_t q) {
    const uint32_t mh = __reduce_max_sync(mask, h);
    const uint32_t mq = __reduce_min_sync(mask, (h != 0u && h == mh) ? (uint32_t)q : 0xffffffffu);
    bk = mh;
    bq = mh ? (int32_t)mq : -1;
}
__device__ __forceinline__ void argmax_u32(uint32_t& bh, int32_t& bq, uint32_t h, int32_t q) {
    if (h > bh || (h == bh && (uint32_t)q < (uint32_t)bq)) { bh = h; bq = q; }
}

// LP candidate rule: gain >= 0, or -gain < own/den (integer division; for
// x = 1 - gain, x <= own/den exactly when x * den <= own: one wide multiply)
__device__ __forceinline__ bool lp_candidate(int32_t g, int32_t own, int32_t den) {
    return g >= 0 || (int64_t)(1 - (int64_t)g) * den <= own;
}

// ------------------------------------------------------------------ k_conn
// Light rows are taken 8 units (4 bucket-0 rows, 1 bucket-1 row or 1 bucket-2
// row each) per warp at a time (conn_group); rows longer than kHeavyDeg take
// CTAs [0, nheavy).  Bucket-0 rows take one thread each, bucket-1 and bucket-2
// rows the warp; bucket 2 and heavy rows build the whole shared-memory
// histogram.
// status: [S_CROSS] += directed cross weight; [S_MAXPW], [S_MODE], [S_LIGHT]
// written by CTA 0; LP candidates are appended to clist[bucket] (any order:
// each is evaluated on its own), with [S_NL0..S_NL2] their counts and
// [S_CDEG] the sum of their degrees.  Rebalance candidates are the vertices of
// overweight parts, [S_CDEG] their number; they are collected in vertex order
// afterwards.  A rebalancing pass stores dest and gain of those only (of every
// vertex when traced): the others' are left from the pass before.

// What decides whether a pass is the level's last (the host loop's rule, from
// its state before the pass): such a pass sweeps nothing when the cut's change
// is known.
struct ConnStop {
    int64_t cross2, best_cut, best_mp;   // cross weight before the step; best state so far
    int may;        // 0: the level goes on in any case, or the step's change is not tracked
    int patience;   // one more state without a significant improvement ends the level
    int idle;       // a step without moves ends the level
};
// state (cut, heaviest part) against the best one: better, and by how much
__device__ __host__ __forceinline__ bool state_better(int64_t cut, int64_t mp, int64_t best_cut, int64_t best_mp,
                                                      int64_t Lmax, bool& signif) {
    const bool cb = mp <= Lmax, bb = best_mp <= Lmax;
    signif = false;
    if (cb && !bb) { signif = true; return true; }
    if (cb && bb) { signif = 1000 * cut < 999 * best_cut; return cut < best_cut; }
    if (!cb && !bb) { signif = mp < best_mp; return mp < best_mp || (mp == best_mp && cut < best_cut); }
    return false;
}
struct ConnArgs {
    DGraph g;
    int32_t k;
    int64_t Lmax;
    int32_t den;
    int force_eval;
    const uint8_t* lock;
    const int64_t* pw;
    const int32_t* heavy;
    const int32_t* item_row;
    const int64_t* item_beg;
    const int64_t* item_end;
    const int32_t* row_items;
    int64_t nitems;
    const int32_t* bucket[3];
    int64_t nbucket[3];
    const int64_t* wfirst;      // first light unit of each range, and the end (nranges + 1)
    int64_t nranges;
    int32_t* dest;
    int32_t* gain;
    const void* pc;             // the partition: PT[n], uint8 (k <= 256), uint16 (k <= 1024) or int32
    void* pc_next;              // label propagation: partition and cleared lock copied here for the
    uint8_t* lock_next;         // move step (nullptr: not needed)
    int64_t* status;
    int32_t* clist[3];          // nullptr: no candidate lists (the one-block loop rescans dest)
    int32_t* hhist;
    int64_t* hsum;
    int32_t* hdone;
    uint64_t* pdg;              // label propagation: pdg_pack(part, dest, gain) per row (nullptr: none)
    const int64_t* prev;        // status block of the iteration before (nullptr: none)
    int64_t track_deg;          // its step's cross-weight change is known (k_track) when the moved rows
                                // had at most this many entries (-1: never)
    ConnStop stop;
    int rb_all;                 // rebalancing passes store proposals of every row (trace)
    int64_t* host;              // host-resident copy of the status block, written by the pass's last
    int nblocks;                // block out of nblocks (over all its launches)
    int lp_dg;                  // label propagation also writes dest and gain (no pdg, or someone
                                // else reads them)
};

// one word per vertex for the move step: part (bits 44-53), dest + 1 (bits
// 32-43; 0: no proposal) and gain (bits 0-31); k <= 1024
__device__ __forceinline__ uint64_t pdg_pack(int32_t p, int32_t d, int32_t g) {
    return ((uint64_t)(uint32_t)p << 44) | ((uint64_t)(uint32_t)(d + 1) << 32) | (uint64_t)(uint32_t)g;
}
__device__ __forceinline__ int32_t pdg_part(uint64_t x) { return (int32_t)((x >> 44) & 0x3FFu); }
__device__ __forceinline__ int32_t pdg_dest(uint64_t x) { return (int32_t)((x >> 32) & 0xFFFu) - 1; }
__device__ __forceinline__ int32_t pdg_gain(uint64_t x) { return (int32_t)(uint32_t)x; }

// part id of neighbour u (uint8 / uint16: read-only in the kernel; the int32
// partition of the one-block loop changes within its kernel: plain loads)
template <class PT>
__device__ __forceinline__ int32_t gpart(const void* pc, int32_t u, int64_t n) {
    if (!GP_IN(u, n)) return 0;
    if constexpr (sizeof(PT) == 4) return ((const PT*)pc)[u];
    else return (int32_t)__ldg((const PT*)pc + u);
}

// one part id of a partition stored in pcb bytes per vertex (1, 2 or 4)
__device__ __forceinline__ void store_pc(void* pc, int pcb, int64_t v, int32_t d) {
    if (pcb == 1) ((uint8_t*)pc)[v] = (uint8_t)d;
    else if (pcb == 2) ((uint16_t*)pc)[v] = (uint16_t)d;
    else ((int32_t*)pc)[v] = d;
}
__device__ __forceinline__ int32_t load_pc(const void* pc, int pcb, int64_t v) {
    return pcb == 1 ? (int32_t)((const uint8_t*)pc)[v]
                    : (pcb == 2 ? (int32_t)((const uint16_t*)pc)[v] : ((const int32_t*)pc)[v]);
}

__device__ __forceinline__ void hist_add(int32_t* hist, int32_t q, int32_t w, bool valid, int32_t k) {
    if (valid && GP_IN(q, k)) atomicAdd(&hist[q], w);
}

// warp-aggregated append of the lanes with take set
__device__ __forceinline__ void warp_push(bool take, int32_t v, int32_t* list, int64_t* count, int64_t cap) {
    const uint32_t m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd((unsigned long long*)count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    const int64_t idx = (int64_t)base + __popc(m & ((1u << lane) - 1u));
    if (take && GP_IN(idx, cap)) list[idx] = v;
}

// decision of one row from its best other part (bq, bk), its cross weight and
// its total weighted degree; returns true when an LP candidate is recorded
template <class PT>
__device__ __forceinline__ bool conn_decide(const ConnArgs& A, int mode, bool active, int32_t v, int32_t p,
                                            int32_t tot, int32_t cross, uint32_t bk, int32_t bq, int32_t light) {
    const int32_t own = tot - cross;
    int32_t d = -1, gn = 0;
    bool cand = false;
    if (mode == MODE_EVAL || (mode == MODE_RB && !active && !A.rb_all)) return false;
    if (mode == MODE_LP) {
        if (A.pc_next) { ((PT*)A.pc_next)[v] = (PT)p; A.lock_next[v] = 0; }
        if (active && bq >= 0) {
            const int32_t gg = (int32_t)bk - own;
            if (lp_candidate(gg, own, A.den)) { d = bq; gn = gg; cand = true; }
        }
        if (A.pdg) A.pdg[v] = pdg_pack(p, d, gn);
        if (!A.lp_dg) return cand;
    } else if (mode == MODE_RB && active) {
        d = bq >= 0 ? bq : light;
        gn = bq >= 0 ? (int32_t)bk - own : -own;
    }
    A.dest[v] = d;
    A.gain[v] = gn;
    return cand;
}

// one row of the connectivity pass: id (-1: none), entry range, part, and
// whether it looks for a move in this mode
struct ConnRow {
    int64_t beg, end;
    int32_t v, p;
    bool active;
};
// full: the pass sums the cross weight over every row; else only active rows
// are swept (the others read as empty)
template <class PT>
__device__ __forceinline__ ConnRow conn_row(const ConnArgs& A, int32_t v, int mode, bool full, const uint8_t* over) {
    ConnRow r;
    r.v = v; r.beg = 0; r.end = 0; r.p = -1; r.active = false;
    if (v >= 0) {
        r.p = gpart<PT>(A.pc, v, A.g.n);
        r.active = (mode == MODE_LP && !A.lock[v]) || (mode == MODE_RB && over[r.p]);
        if (full || r.active) { r.beg = A.g.rp[v]; r.end = A.g.rp[v + 1]; }
    }
    return r;
}
// shared-memory copy of a ConnRow (pa: part, bit 31 = active)
struct ConnRowS {
    int64_t beg, end;
    int32_t v, pa;
};
__device__ __forceinline__ ConnRowS conn_stage(const ConnRow& r) {
    ConnRowS s;
    s.beg = r.beg; s.end = r.end; s.v = r.v;
    s.pa = (int32_t)((uint32_t)r.p | (r.active ? 0x80000000u : 0u));
    return s;
}
__device__ __forceinline__ ConnRow conn_unstage(const ConnRowS& s) {
    ConnRow r;
    r.beg = s.beg; r.end = s.end; r.v = s.v;
    r.p = s.v >= 0 ? (int32_t)((uint32_t)s.pa & 0x7fffffffu) : -1;
    r.active = s.v >= 0 && s.pa < 0;
    return r;
}
// the LP candidate list and its count slot of bucket b
__device__ __forceinline__ int64_t* conn_list_count(const ConnArgs& A, int b) {
    return &A.status[b == 0 ? S_NL0 : (b == 1 ? S_NL1 : S_NL2)];
}

// what one row contributes and its best other part (bk = 0, bq = -1: none);
// a row's weights add up to less than 2^31
struct ConnRes {
    int32_t tot, cross;
    uint32_t bk;
    int32_t bq;
};

// bucket 0 (at most 16 entries): one row per thread; every lane of the warp
// calls it (rows of no vertex: no entries).  What bounds these rows is the
// instruction count, not the loads: a warp's 32 rows are mostly consecutive
// (the entry loads hit the lines the first of them brought in), and all of a
// row's loads, then all its gathers, are in flight together (8 or 16 of them,
// by the longest row of the warp).  The part sums are compares among the
// thread's own registers, part by part in ascending order (so ties keep the
// smaller part), done only in warps with a row that has a neighbour in another
// part and looks for a move.
template <int N, class PT>
__device__ __forceinline__ ConnRes conn_thread_n(const ConnArgs& A, const ConnRow& R, int mode, const uint8_t* over) {
    ConnRes x{0, 0, 0u, -1};
    const int len = (int)(R.end - R.beg);
    const int32_t* __restrict__ row = A.g.ci + R.beg;
    int32_t q[N], w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = i < len ? __ldg(row + i) : -1;
    if (A.g.ew) {
        const int32_t* __restrict__ wrow = A.g.ew + R.beg;
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = i < len ? __ldg(wrow + i) : 0;
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = i < len ? 1 : 0;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = q[i] >= 0 ? gpart<PT>(A.pc, q[i], A.g.n) : -1;
#pragma unroll
    for (int i = 0; i < N; ++i) { x.tot += w[i]; x.cross += q[i] != R.p ? w[i] : 0; }
    bool go = R.active && x.cross > 0;
    int32_t cur = -1;
    while (__any_sync(0xffffffffu, go)) {
        int32_t nx = INT32_MAX;   // the next part above cur
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (q[i] > cur && q[i] != R.p && q[i] < nx) nx = q[i];
        go = go && nx != INT32_MAX;
        if (go) {
            int32_t h = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) h += q[i] == nx ? w[i] : 0;
            if ((uint32_t)h > x.bk && (mode != MODE_RB || !over[nx])) { x.bk = (uint32_t)h; x.bq = nx; }
            cur = nx;
        }
    }
    return x;
}
template <class PT>
__device__ __forceinline__ ConnRes conn_thread(const ConnArgs& A, const ConnRow& R, int mode, const uint8_t* over) {
    const uint32_t most = __reduce_max_sync(0xffffffffu, (uint32_t)(R.end - R.beg));
    return most <= 8 ? conn_thread_n<8, PT>(A, R, mode, over) : conn_thread_n<kShortDeg, PT>(A, R, mode, over);
}

// bucket 1 (17 to 32 entries): one row per warp, one entry per lane; the
// entries are added into the warp's shared-memory histogram and each lane
// reads its own part's bin back (lanes of the same part hold the same value,
// which the argmax, ties to the smaller part, does not mind).  hist: the
// warp's k zeroed bins, left zeroed.
template <class PT>
__device__ __forceinline__ ConnRes conn_lane(const ConnArgs& A, const ConnRow& R, int mode, const uint8_t* over,
                                             int32_t* hist) {
    const int lane = threadIdx.x & 31;
    const int64_t e = R.beg + lane;
    const bool has = e < R.end;
    int32_t q = -1, w = 0;
    if (has) { q = gpart<PT>(A.pc, __ldcs(&A.g.ci[e]), A.g.n); w = A.g.ew ? __ldcs(&A.g.ew[e]) : 1; }
    const bool in = has && q != R.p && GP_IN(q, A.k);   // the own part's bin is not needed
    ConnRes x;
    x.cross = (int32_t)__reduce_add_sync(0xffffffffu, (has && q != R.p) ? (uint32_t)w : 0u);
    x.tot = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)w);
    x.bk = 0; x.bq = -1;
    if (R.active && x.cross > 0) {   // one row per warp: uniform
        uint32_t h = 0;
        if (in) atomicAdd(&hist[q], w);
        __syncwarp();
        if (in) h = (uint32_t)hist[q];
        __syncwarp();
        if (in) hist[q] = 0;
        __syncwarp();
        uint64_t bk;
        group_argmax_u32(0xffffffffu, bk, x.bq, (in && (mode != MODE_RB || !over[q])) ? h : 0u, q);
        x.bk = (uint32_t)bk;
    }
    return x;
}

// bucket 2: one row per warp, shared-memory histogram.  The row is swept
// 128 entries at a time (4 independent loads per lane in flight).  The own
// part is never added (its connectivity is tot - cross), which keeps the
// most contended bin out of the shared-memory atomics.  For rows at least as
// long as k, or k <= kBinsK, the best part is taken over the k histogram bins,
// otherwise over the row's entries again (same candidates: parts with a
// non-zero connection).
constexpr int kBinsK = 256;
template <class PT>
__device__ __forceinline__ ConnRes conn_warp(const ConnArgs& A, const ConnRow& R, int mode, const uint8_t* over,
                                             int32_t* hist) {
    const int lane = threadIdx.x & 31;
    const int64_t beg = R.beg, end = R.end;
    const int32_t p = R.p;
    const bool active = R.active;
    int32_t cross = 0, tot = 0;
    // 128 entries per sweep, four consecutive ones per lane (16-byte loads)
    const bool v4 = aligned16(A.g.ci) && aligned16(A.g.ew);
    for (int64_t base = beg & ~(int64_t)3; base < end; base += 128) {
        int32_t u[4], w[4], q[4];
        const int64_t e4 = base + 4 * lane;
        ld4_row(A.g.ci, e4, beg, end, v4, -1, u);
        if (A.g.ew) ld4_row(A.g.ew, e4, beg, end, v4, 0, w);
        else {
#pragma unroll
            for (int c = 0; c < 4; ++c) w[c] = u[c] >= 0 ? 1 : 0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) q[c] = u[c] >= 0 ? gpart<PT>(A.pc, u[c], A.g.n) : -1;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            tot += w[c];
            if (q[c] >= 0 && q[c] != p) cross += w[c];
            if (active) hist_add(hist, q[c], w[c], q[c] >= 0 && q[c] != p, A.k);
        }
    }
    cross = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)cross);
    tot = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)tot);
    uint64_t bk = 0;
    int32_t bq = -1;
    if (active) {
        __syncwarp();
        uint32_t lh = 0;
        int32_t lq = -1;
        if (end - beg >= A.k || A.k <= kBinsK) {
            for (int q = lane; q < A.k; q += 32) {
                const int32_t h = hist[q];
                if (h > 0 && q != p && (mode != MODE_RB || !over[q])) argmax_u32(lh, lq, (uint32_t)h, q);
            }
            group_argmax_u32(0xffffffffu, bk, bq, lh, lq);
            __syncwarp();
            for (int q = lane; q < A.k; q += 32) hist[q] = 0;
        } else {
            for (int64_t e = beg + lane; e < end; e += 32) {
                const int32_t q = gpart<PT>(A.pc, __ldcs(&A.g.ci[e]), A.g.n);
                if (!GP_IN(q, A.k)) continue;
                if (q != p && (mode != MODE_RB || !over[q])) argmax_u32(lh, lq, (uint32_t)hist[q], q);
            }
            group_argmax_u32(0xffffffffu, bk, bq, lh, lq);
            __syncwarp();
            for (int64_t e = beg + lane; e < end; e += 32) {
                const int32_t q = gpart<PT>(A.pc, __ldcs(&A.g.ci[e]), A.g.n);
                if (GP_IN(q, A.k)) hist[q] = 0;
            }
        }
        __syncwarp();
    }
    return ConnRes{tot, cross, (uint32_t)bk, bq};
}

// Up to 8 light units [ub, ub + nu) by one warp (unit order: bucket 2 rows,
// bucket 1 rows, groups of 4 bucket-0 rows).  Lane l first fetches row slot l
// (unit l / 4; its row, or the (l % 4)-th row of a group of 4), so the list and
// row-header loads of 8 units are in flight together; the rows' results land
// in the lane of their slot, and the decisions of all of them are taken and
// stored together (a warp's stores of consecutive rows coalesce), their
// candidates appended together (one atomic per list present).  rows: the
// warp's 32 slots in shared memory.  SHORT: there may be bucket-0 units.
template <class PT, bool SHORT>
__device__ __forceinline__ void conn_group(const ConnArgs& A, int64_t ub, int nu, int mode, bool full, const uint8_t* over,
                                           int32_t light, int32_t* hist, ConnRowS* rows, int64_t& acc, int64_t& cdeg) {
    const int lane = threadIdx.x & 31;
    const int64_t U2 = A.nbucket[2], U21 = U2 + A.nbucket[1];
    const int64_t u = ub + (lane >> 2);
    const int sub = lane & 3;
    const int lb = u < U2 ? 2 : (!SHORT || u < U21 ? 1 : 0);
    int32_t v = -1;
    if (u < ub + nu) {
        if (lb == 2) { if (sub == 0) v = A.bucket[2][u]; }
        else if (lb == 1) { if (sub == 0) v = A.bucket[1][u - U2]; }
        else {
            const int64_t i = (u - U21) * 4 + sub;
            if (i < A.nbucket[0]) v = A.bucket[0][i];
        }
    }
    const ConnRow r = conn_row<PT>(A, v, mode, full, over);
    ConnRes x{0, 0, 0u, -1};
    if (SHORT && ub + nu > U21 && __any_sync(0xffffffffu, r.end > r.beg)) {
        ConnRow tr = r;
        if (lb != 0) { tr.end = tr.beg; tr.active = false; }
        x = conn_thread<PT>(A, tr, mode, over);
    }
    if (ub < U21) {   // warp rows among the units
        rows[lane] = conn_stage(r);
        __syncwarp();
        const int nlong = U21 - ub < nu ? (int)(U21 - ub) : nu;
        const uint32_t todo = __ballot_sync(0xffffffffu, r.end > r.beg);   // rows to sweep
        for (int j = 0; j < nlong; ++j) {
            if (!((todo >> (4 * j)) & 1u)) continue;
            const ConnRow wr = conn_unstage(rows[4 * j]);
            const ConnRes y = ub + j < U2 ? conn_warp<PT>(A, wr, mode, over, hist)
                                          : conn_lane<PT>(A, wr, mode, over, hist);
            if (lane == 4 * j) x = y;
        }
        __syncwarp();
    }
    bool take = false;
    if (r.v >= 0) {
        acc += x.cross;
        take = conn_decide<PT>(A, mode, r.active, r.v, r.p, x.tot, x.cross, x.bk, x.bq, light);
        if (take) cdeg += r.end - r.beg;
        else if (mode == MODE_RB && r.active) ++cdeg;
    }
    if (A.clist[0] == nullptr || !__any_sync(0xffffffffu, take)) return;
#pragma unroll
    for (int b = SHORT ? 0 : 1; b < 3; ++b) warp_push(take && lb == b, r.v, A.clist[b], conn_list_count(A, b), A.g.n);
}

// part-weight summary every block of a connectivity pass starts from: over
// flags, the heaviest part, the lightest part within Lmax (ties: lower id) and
// the mode they imply; block 0 writes the summary to the status block
struct ConnHead {
    int64_t red[RW];
    uint64_t k[RW];
    int32_t q[RW];
    int64_t maxpw;
    int32_t light;
};
__device__ __forceinline__ int conn_head(const ConnArgs& A, uint8_t* over, ConnHead& sh, int32_t& light, bool& full) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t Lmax = A.Lmax;
    int64_t mx = 0;
    uint64_t lk = 0; int32_t lq = -1;  // argmax of (~pw) == argmin pw
    for (int q = threadIdx.x; q < A.k; q += RT) {
        const int64_t x = A.pw[q];
        over[q] = x > Lmax;
        mx = x > mx ? x : mx;
        if (x <= Lmax) argmax_q(lk, lq, ~(uint64_t)x, q);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { int64_t y = __shfl_xor_sync(0xffffffffu, mx, o); mx = y > mx ? y : mx; }
    warp_argmax_q(lk, lq);
    if (lane == 0) { sh.red[w] = mx; sh.k[w] = lk; sh.q[w] = lq; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t m2 = 0; uint64_t k2 = 0; int32_t q2 = -1;
        for (int i = 0; i < RW; ++i) { m2 = sh.red[i] > m2 ? sh.red[i] : m2; argmax_q(k2, q2, sh.k[i], sh.q[i]); }
        sh.maxpw = m2; sh.light = q2;
    }
    __syncthreads();
    const int64_t maxpw = sh.maxpw;
    light = sh.light;
    int mode = A.force_eval ? MODE_EVAL : (maxpw > Lmax ? MODE_RB : MODE_LP);
    // a rebalancing pass sweeps only the rows of overweight parts when k_track
    // has the last step's change of the cut (the same test there), the level's
    // last pass nothing
    const bool known = A.prev && A.prev[S_MVDEG] <= A.track_deg;
    full = mode != MODE_RB || !known;
    if (known && A.stop.may) {
        bool signif;
        state_better((A.stop.cross2 + A.prev[S_DELTA]) / 2, maxpw, A.stop.best_cut, A.stop.best_mp, Lmax, signif);
        if (A.force_eval || (!signif && A.stop.patience) || (A.stop.idle && A.prev[S_STEP_MOVES] == 0)) {
            mode = MODE_EVAL;
            full = false;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.status[S_MAXPW] = maxpw; A.status[S_MODE] = mode; A.status[S_LIGHT] = light;
    }
    return mode;
}
// adds every thread's cross weight to the status block, one atomic per block;
// the pass's last block then writes the block to the host (pinned, mapped
// memory: no copy operation between the pass and the host's wait)
__device__ __forceinline__ void conn_tail(const ConnArgs& A, int64_t acc, int64_t* s_red, bool full) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    acc = warp_sum(acc);
    __syncthreads();
    if (lane == 0) s_red[w] = acc;
    __syncthreads();
    if (w != 0) return;
    uint32_t last = 0;
    if (lane == 0) {
        int64_t s = 0;
        for (int i = 0; i < RW; ++i) s += s_red[i];
        if (s) atomicAdd((unsigned long long*)&A.status[S_CROSS], (unsigned long long)s);
        __threadfence();
        last = atomicAdd((unsigned long long*)&A.status[S_DONE], 1ull) == (unsigned long long)A.nblocks - 1ull;
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    // one store of the warp (HostSlot)
    if (lane < H_NSLOTS) {
        const int64_t* from = lane < S_NRESET ? A.status + lane : nullptr;
        if (A.prev && lane == H_MOVES) from = A.prev + S_STEP_MOVES;
        if (A.prev && lane == H_DELTA) from = A.prev + S_DELTA;
        const int64_t x = from ? (int64_t)__ldcg((const unsigned long long*)from) : 0;
        A.host[lane] = lane == H_FULL ? (full ? 1 : 0) : x;
    }
}

// Bucket-0 rows of a large level: one row per lane, 32 listed rows per warp at
// a time, grid-stride.  Its own kernel because a thread's 16 entries, weights
// and gathers take 64 registers, while the longer rows (k_conn) run best at
// 48: with them in k_conn its R-MAT 24 passes took 138 ms in all (spills),
// apart 125.  256^3 grid, k = 32, one pass, against 8 lanes per row of up to 8
// entries and a warp per row above: level 0 (16.8 M rows of 6 entries) 1860 ->
// 330 us; all 270 passes of its V-cycle 182 -> 44 ms.
template <class PT>
__global__ void __launch_bounds__(RT, 4) k_conn_short(ConnArgs A) {
    extern __shared__ int32_t csm[];
    uint8_t* over = (uint8_t*)csm;
    __shared__ ConnHead sh;
    int32_t light;
    bool full;
    const int mode = conn_head(A, over, sh, light, full);
    const int lane = threadIdx.x & 31;
    int64_t acc = 0, cdeg = 0;
    const int64_t n0 = mode == MODE_EVAL && !full ? 0 : A.nbucket[0];
    for (int64_t i0 = (int64_t)blockIdx.x * RT + (threadIdx.x & ~31); i0 < n0; i0 += (int64_t)gridDim.x * RT) {
        const int64_t i = i0 + lane;
        const ConnRow r = conn_row<PT>(A, i < n0 ? A.bucket[0][i] : -1, mode, full, over);
        if (!full && !A.rb_all && !__any_sync(0xffffffffu, r.active)) continue;
        const ConnRes x = conn_thread<PT>(A, r, mode, over);
        bool take = false;
        if (r.v >= 0) {
            acc += x.cross;
            take = conn_decide<PT>(A, mode, r.active, r.v, r.p, x.tot, x.cross, x.bk, x.bq, light);
            if (take) cdeg += r.end - r.beg;
            else if (mode == MODE_RB && r.active) ++cdeg;
        }
        warp_push(take, r.v, A.clist[0], conn_list_count(A, 0), A.g.n);
    }
    cdeg = warp_sum(cdeg);
    if (lane == 0 && cdeg) atomicAdd((unsigned long long*)&A.status[S_CDEG], (unsigned long long)cdeg);
    conn_tail(A, acc, sh.red, full);
}

// SHORT: the light units include the bucket-0 rows (small levels: one launch);
// else they are left to k_conn_short
template <class PT, bool SHORT>
__global__ void __launch_bounds__(RT, SHORT ? 4 : 5) k_conn(ConnArgs A) {
    extern __shared__ int32_t csm[];
    const int32_t k = A.k;
    const int kpad = (k + 15) & ~15;
    uint8_t* over = (uint8_t*)csm;
    int32_t* hist_all = csm + kpad / 4;
    __shared__ ConnHead sh;
    __shared__ ConnRowS s_rows[RT];   // light warps: 32 staged rows each
    int64_t* s_red = sh.red;
    uint64_t* s_k = sh.k;
    int32_t* s_q = sh.q;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ uint32_t s_next;   // light blocks: ranges taken so far
    if (threadIdx.x == 0) s_next = 0;
    for (int i = threadIdx.x; i < RW * k; i += RT) hist_all[i] = 0;
    int32_t light;
    bool full;
    const int mode = conn_head(A, over, sh, light, full);
    int64_t acc = 0;  // directed cross weight (this thread)

    if (mode == MODE_EVAL && !full) {
        // nothing to sweep
    } else if ((int64_t)blockIdx.x < A.nitems) {
        // ---- one piece of a long row per CTA; pieces of the same row are
        // combined in global accumulators and the last CTA decides
        int32_t* hist = hist_all;
        const int32_t h = A.item_row[blockIdx.x];
        const int64_t v = A.heavy[h];
        const int nit = A.row_items[h];
        const int32_t p = gpart<PT>(A.pc, (int32_t)v, A.g.n);
        const bool active = (mode == MODE_LP && !A.lock[v]) || (mode == MODE_RB && over[p]);
        const bool sweep = full || active;   // the same for every piece of the row
        if (!sweep && A.rb_all && threadIdx.x == 0) { A.dest[v] = -1; A.gain[v] = 0; }
        const int64_t beg = sweep ? A.item_beg[blockIdx.x] : 0, end = sweep ? A.item_end[blockIdx.x] : 0;
        int64_t cross = 0, tot = 0;
        const bool v4 = aligned16(A.g.ci) && aligned16(A.g.ew);
        for (int64_t base = beg & ~(int64_t)3; base < end; base += 4 * RT) {
            int32_t uu[4], ww[4], qq[4];
            const int64_t e4 = base + 4 * threadIdx.x;
            ld4_row(A.g.ci, e4, beg, end, v4, -1, uu);
            if (A.g.ew) ld4_row(A.g.ew, e4, beg, end, v4, 0, ww);
            else {
#pragma unroll
                for (int c = 0; c < 4; ++c) ww[c] = uu[c] >= 0 ? 1 : 0;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) qq[c] = uu[c] >= 0 ? gpart<PT>(A.pc, uu[c], A.g.n) : -1;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tot += ww[c];
                if (qq[c] >= 0 && qq[c] != p) cross += ww[c];
                if (active) hist_add(hist, qq[c], ww[c], qq[c] >= 0 && qq[c] != p, k);
            }
        }
        cross = warp_sum(cross); tot = warp_sum(tot);
        acc += (lane == 0) ? cross : 0;  // the cut adds every piece
        __syncthreads();
        if (lane == 0) { s_red[w] = cross; s_k[w] = (uint64_t)tot; }
        __syncthreads();
        __shared__ int s_last;
        if (threadIdx.x == 0) {
            int64_t c2 = 0, t2 = 0;
            for (int i = 0; i < RW; ++i) { c2 += s_red[i]; t2 += (int64_t)s_k[i]; }
            s_red[0] = c2; s_k[0] = (uint64_t)t2;
            s_last = sweep ? 1 : 0;
        }
        __syncthreads();
        if (sweep && nit > 1) {
            if (active)
                for (int q = threadIdx.x; q < k; q += RT)
                    if (hist[q]) atomicAdd(&A.hhist[(int64_t)h * k + q], hist[q]);
            if (threadIdx.x == 0) {
                atomicAdd((unsigned long long*)&A.hsum[2 * h], (unsigned long long)s_red[0]);
                atomicAdd((unsigned long long*)&A.hsum[2 * h + 1], (unsigned long long)s_k[0]);
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) s_last = (atomicAdd(&A.hdone[h], 1) == nit - 1) ? 1 : 0;
            __syncthreads();
            if (s_last) {
                __threadfence();
                for (int q = threadIdx.x; q < k; q += RT) {
                    hist[q] = active ? __ldcg(&A.hhist[(int64_t)h * k + q]) : 0;
                    A.hhist[(int64_t)h * k + q] = 0;
                }
                if (threadIdx.x == 0) {
                    s_red[0] = (int64_t)__ldcg((const unsigned long long*)&A.hsum[2 * h]);
                    s_k[0] = (uint64_t)__ldcg((const unsigned long long*)&A.hsum[2 * h + 1]);
                    A.hsum[2 * h] = 0; A.hsum[2 * h + 1] = 0; A.hdone[h] = 0;
                }
                __syncthreads();
            }
        }
        if (s_last) {
            cross = s_red[0]; tot = (int64_t)s_k[0];
            __syncthreads();
            uint64_t bk = 0; int32_t bq = -1;
            if (active)
                for (int q = threadIdx.x; q < k; q += RT)
                    if (q != p && hist[q] > 0 && (mode != MODE_RB || !over[q])) argmax_q(bk, bq, (uint64_t)hist[q], q);
            warp_argmax_q(bk, bq);
            if (lane == 0) { s_k[w] = bk; s_q[w] = bq; }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int i = 1; i < RW; ++i) argmax_q(bk, bq, s_k[i], s_q[i]);
                const int64_t rdeg = A.g.rp[v + 1] - A.g.rp[v];
                if (conn_decide<PT>(A, mode, active, (int32_t)v, p, (int32_t)tot, (int32_t)cross, (uint32_t)bk, bq, light))
                    atomicAdd((unsigned long long*)&A.status[S_CDEG], (unsigned long long)rdeg);
                else if (mode == MODE_RB && active) atomicAdd((unsigned long long*)&A.status[S_CDEG], 1ull);
            }
        }
    } else {
        int32_t* hist = hist_all + w * k;
        ConnRowS* rows = s_rows + w * 32;
        int64_t cdeg = 0;   // degree sum of this lane's candidates
        for (;;) {
            const int64_t r = block_unit(&s_next, blockIdx.x - A.nitems, gridDim.x - A.nitems);
            if (r >= A.nranges) break;
            const int64_t u0 = A.wfirst[r], u1 = A.wfirst[r + 1];
            for (int64_t ub = u0; ub < u1; ub += 8)
                conn_group<PT, SHORT>(A, ub, (int)(u1 - ub < 8 ? u1 - ub : 8), mode, full, over, light, hist, rows, acc,
                                      cdeg);
        }
        cdeg = warp_sum(cdeg);
        if (lane == 0 && cdeg) atomicAdd((unsigned long long*)&A.status[S_CDEG], (unsigned long long)cdeg);
    }
    conn_tail(A, acc, s_red, full);
}

// ------------------------------------------------------------------ LP apply
template <class PT>
__device__ __forceinline__ int32_t ab_term(const DGraph& g, int64_t e, int64_t v, int32_t p, int32_t d, int32_t gv,
                                           const void* pc, const int32_t* __restrict__ dest,
                                           const int32_t* __restrict__ gain, const uint64_t* __restrict__ pdg) {
    const int32_t u = __ldcs(&g.ci[e]);
    if (!GP_IN(u, g.n)) return 0;
    int32_t pu, du, gu = 0;
    if (pdg) {
        const uint64_t x = pdg[u];
        pu = pdg_part(x); du = pdg_dest(x); gu = pdg_gain(x);
    } else {
        pu = gpart<PT>(pc, u, g.n);
        du = dest[u];
        if (du >= 0) gu = gain[u];
    }
    if (du >= 0 && (gu > gv || (gu == gv && u < (int32_t)v))) pu = du;
    const int32_t wt = g.ew ? __ldcs(&g.ew[e]) : 1;
    return pu == d ? wt : (pu == p ? -wt : 0);
}

struct ApplyArgs {
    DGraph g;
    int32_t k;
    const int32_t* dest;
    const int32_t* gain;
    const int32_t* heavy;
    const int32_t* item_row;
    const int64_t* item_beg;
    const int64_t* item_end;
    const int32_t* row_items;
    int64_t nitems;
    const int32_t* clist[3];
    const int64_t* status;
    uint8_t* lock_next;
    const void* pc;             // the partition (as in ConnArgs)
    void* pc_next;              // the partition after the step
    int64_t* pw;
    int64_t* step;              // status block the step's moves and moved entries are added to
    int64_t* hsum;
    int32_t* hdone;
    const uint64_t* pdg;        // packed part / dest / gain of every vertex (nullptr: gather them apart)
};

// a thread's moves and the entries of their rows
struct AbCount {
    int64_t moves = 0, deg = 0;
};
template <class PT>
__device__ __forceinline__ void ab_commit(const ApplyArgs& A, int64_t v, int32_t p, int32_t d, int64_t deg,
                                          int32_t* delta, AbCount& cnt) {
    if (!GP_IN(d, A.k) || !GP_IN(p, A.k)) return;
    ((PT*)A.pc_next)[v] = (PT)d;
    A.lock_next[v] = 1;
    const int32_t wv = A.g.vw ? A.g.vw[v] : 1;
    atomicAdd(&delta[d], wv);
    atomicAdd(&delta[p], -wv);
    ++cnt.moves;
    cnt.deg += deg;
}

// part, destination (-1: no candidate) and gain of row v
template <class PT>
__device__ __forceinline__ void ab_row(const ApplyArgs& A, int64_t v, int32_t& p, int32_t& d, int32_t& gv) {
    if (A.pdg) {
        const uint64_t x = A.pdg[v];
        p = pdg_part(x); d = pdg_dest(x); gv = pdg_gain(x);
    } else {
        p = gpart<PT>(A.pc, (int32_t)v, A.g.n); d = A.dest[v]; gv = A.gain[v];
    }
}

// candidate rows of bucket 0, many of them: one row per lane (v < 0: none),
// every lane of the warp calls it; all of a row's entries are in flight
// together (8 or 16 of them, by the longest row of the warp)
template <int N, class PT>
__device__ __forceinline__ int32_t ab_short_n(const ApplyArgs& A, int64_t v, int32_t p, int32_t d, int32_t gv,
                                              int64_t beg, int len) {
    const int32_t* __restrict__ row = A.g.ci + beg;
    int32_t u[N], t = 0;
    uint64_t x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) u[i] = i < len ? __ldg(row + i) : -1;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = 0;
        if (u[i] < 0 || !GP_IN(u[i], A.g.n)) { u[i] = -1; continue; }
        if (A.pdg) x[i] = A.pdg[u[i]];
        else x[i] = pdg_pack(gpart<PT>(A.pc, u[i], A.g.n), A.dest[u[i]], A.dest[u[i]] >= 0 ? A.gain[u[i]] : 0);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (u[i] < 0) continue;
        int32_t q = pdg_part(x[i]);
        const int32_t du = pdg_dest(x[i]), gu = pdg_gain(x[i]);
        if (du >= 0 && (gu > gv || (gu == gv && u[i] < (int32_t)v))) q = du;
        const int32_t w = A.g.ew ? __ldg(A.g.ew + beg + i) : 1;
        t += q == d ? w : (q == p ? -w : 0);
    }
    return t;
}
template <class PT>
__device__ __forceinline__ void ab_short(const ApplyArgs& A, int64_t v, int32_t* delta, AbCount& cnt) {
    int32_t p = -1, d = -1, gv = 0;
    int64_t beg = 0;
    int len = 0;
    if (v >= 0) {
        ab_row<PT>(A, v, p, d, gv);
        beg = A.g.rp[v];
        len = (int)(A.g.rp[v + 1] - beg);
    }
    const uint32_t most = __reduce_max_sync(0xffffffffu, (uint32_t)len);
    const int32_t t = most <= 8 ? ab_short_n<8, PT>(A, v, p, d, gv, beg, len)
                                : ab_short_n<kShortDeg, PT>(A, v, p, d, gv, beg, len);
    if (v >= 0 && t >= 0) ab_commit<PT>(A, v, p, d, len, delta, cnt);
}

// candidate rows of at most TILE entries, TILE lanes each (v < 0: none)
template <int TILE, class PT>
__device__ __forceinline__ void ab_tile(const ApplyArgs& A, int64_t v, int32_t* delta, AbCount& cnt) {
    const int lane = threadIdx.x & 31, tl = lane & (TILE - 1);
    int32_t t = 0, p = -1, d = -1;
    int64_t beg = 0, end = 0;
    if (v >= 0) {
        int32_t gv;
        ab_row<PT>(A, v, p, d, gv);
        beg = A.g.rp[v]; end = A.g.rp[v + 1];
        if (beg + tl < end) t = ab_term<PT>(A.g, beg + tl, v, p, d, gv, A.pc, A.dest, A.gain, A.pdg);
    }
#pragma unroll
    for (int o = TILE / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (tl == 0 && v >= 0 && t >= 0) ab_commit<PT>(A, v, p, d, end - beg, delta, cnt);
}

// this thread's part (thread t of nt) of the ab_term sum over entries
// [beg, end) of row v: four consecutive entries at a time (16-byte loads),
// the four neighbours' part and destination gathers in flight together
template <class PT>
__device__ __forceinline__ int32_t ab_sum(const ApplyArgs& A, int64_t beg, int64_t end, int t, int nt, int64_t v,
                                          int32_t p, int32_t d, int32_t gv) {
    int32_t g2 = 0;
    const bool v4 = aligned16(A.g.ci) && aligned16(A.g.ew);
    for (int64_t base = beg & ~(int64_t)3; base < end; base += 4 * (int64_t)nt) {
        int32_t uu[4], ww[4], pu[4], du[4];
        const int64_t e4 = base + 4 * t;
        ld4_row(A.g.ci, e4, beg, end, v4, -1, uu);
        if (A.g.ew) ld4_row(A.g.ew, e4, beg, end, v4, 0, ww);
        else {
#pragma unroll
            for (int c = 0; c < 4; ++c) ww[c] = uu[c] >= 0 ? 1 : 0;
        }
        int32_t gu[4];
        if (A.pdg) {   // one gather per entry: part, dest and gain in one word
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool ok = uu[c] >= 0 && GP_IN(uu[c], A.g.n);
                const uint64_t x = ok ? A.pdg[uu[c]] : 0ull;
                pu[c] = ok ? pdg_part(x) : -1; du[c] = pdg_dest(x); gu[c] = pdg_gain(x);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool ok = uu[c] >= 0 && GP_IN(uu[c], A.g.n);
                pu[c] = ok ? gpart<PT>(A.pc, uu[c], A.g.n) : -1;
                du[c] = ok ? A.dest[uu[c]] : -1;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) gu[c] = du[c] >= 0 ? A.gain[uu[c]] : 0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (uu[c] < 0 || pu[c] < 0) continue;
            int32_t q = pu[c];
            if (du[c] >= 0 && (gu[c] > gv || (gu[c] == gv && uu[c] < (int32_t)v))) q = du[c];
            g2 += q == d ? ww[c] : (q == p ? -ww[c] : 0);
        }
    }
    return g2;
}

// one candidate row of 33..heavy_deg entries per warp, 128 entries per sweep
template <class PT>
__device__ __forceinline__ void ab_warp(const ApplyArgs& A, int64_t v, int32_t* delta, AbCount& cnt) {
    const int lane = threadIdx.x & 31;
    int32_t p, d, gv;
    ab_row<PT>(A, v, p, d, gv);
    const int64_t beg = A.g.rp[v], end = A.g.rp[v + 1];
    const int32_t g2 = warp_sum(ab_sum<PT>(A, beg, end, lane, 32, v, p, d, gv));
    if (lane == 0 && g2 >= 0) ab_commit<PT>(A, v, p, d, end - beg, delta, cnt);
}

// a block's part-weight changes (32-bit shared atomics, see rb_delta_begin) and
// moves, added to the totals
__device__ __forceinline__ void ab_begin(const ApplyArgs& A, int32_t* delta) {
    for (int q = threadIdx.x; q < A.k; q += RT) delta[q] = 0;
    __syncthreads();
}
__device__ __forceinline__ void ab_end(const ApplyArgs& A, const int32_t* delta, AbCount cnt) {
    cnt.moves = warp_sum(cnt.moves);
    cnt.deg = warp_sum(cnt.deg);
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && cnt.moves) {
        atomicAdd((unsigned long long*)&A.step[S_STEP_MOVES], (unsigned long long)cnt.moves);
        atomicAdd((unsigned long long*)&A.step[S_MVDEG], (unsigned long long)cnt.deg);
    }
    for (int q = threadIdx.x; q < A.k; q += RT)
        if (delta[q]) atomicAdd((unsigned long long*)&A.pw[q], (unsigned long long)(int64_t)delta[q]);
}

// the candidates of bucket 0 on large levels, one per lane (their registers
// apart from k_lp_apply's, as k_conn_short)
template <class PT>
__global__ void __launch_bounds__(RT) k_lp_short(ApplyArgs A) {
    extern __shared__ int32_t delta[];
    ab_begin(A, delta);
    AbCount cnt;
    const int64_t n0 = A.status[S_NL0];
    for (int64_t i0 = (int64_t)blockIdx.x * RT + (threadIdx.x & ~31); i0 < n0; i0 += (int64_t)gridDim.x * RT) {
        const int64_t i = i0 + (threadIdx.x & 31);
        ab_short<PT>(A, i < n0 ? A.clist[0][i] : -1, delta, cnt);
    }
    ab_end(A, delta, cnt);
}

// every other candidate row (split: bucket 0 is k_lp_short's)
template <class PT>
__global__ void __launch_bounds__(RT) k_lp_apply(ApplyArgs A, int split) {
    extern __shared__ int32_t delta[];
    __shared__ int64_t s_red[RW];
    __shared__ uint32_t s_next;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_next = 0;
    ab_begin(A, delta);
    AbCount cnt;
    if ((int64_t)blockIdx.x < A.nitems) {
        const int32_t h = A.item_row[blockIdx.x];
        const int64_t v = A.heavy[h];
        int32_t p, d, gv;
        ab_row<PT>(A, v, p, d, gv);
        if (d >= 0) {
            const int nit = A.row_items[h];
            int32_t g2 = ab_sum<PT>(A, A.item_beg[blockIdx.x], A.item_end[blockIdx.x], threadIdx.x, RT, v, p, d, gv);
            g2 = warp_sum(g2);
            if (lane == 0) s_red[w] = g2;
            __syncthreads();
            if (threadIdx.x == 0) {
                int64_t sum = 0;
                for (int i = 0; i < RW; ++i) sum += s_red[i];
                bool last = true;
                if (nit > 1) {
                    atomicAdd((unsigned long long*)&A.hsum[2 * h], (unsigned long long)sum);
                    __threadfence();
                    last = atomicAdd(&A.hdone[h], 1) == nit - 1;
                    if (last) {
                        __threadfence();
                        sum = (int64_t)__ldcg((const unsigned long long*)&A.hsum[2 * h]);
                        A.hsum[2 * h] = 0;
                        A.hdone[h] = 0;
                    }
                }
                if (last && sum >= 0) ab_commit<PT>(A, v, p, d, A.g.rp[v + 1] - A.g.rp[v], delta, cnt);
            }
        }
    } else {
        const int64_t n0 = split ? 0 : A.status[S_NL0], n1 = A.status[S_NL1], n2 = A.status[S_NL2];
        // longest rows first
        const int64_t U2 = n2, U21 = n2 + n1, U = U21 + (n0 + 1) / 2;
        for (;;) {
            const int64_t u = block_unit(&s_next, blockIdx.x - A.nitems, gridDim.x - A.nitems);
            if (u >= U) break;
            if (u >= U21) {
                const int64_t i = (u - U21) * 2 + (lane >> 4);
                ab_tile<16, PT>(A, i < n0 ? A.clist[0][i] : -1, delta, cnt);
            } else if (u >= U2) {
                ab_tile<kTile32, PT>(A, A.clist[1][u - U2], delta, cnt);
            } else {
                ab_warp<PT>(A, A.clist[2][u], delta, cnt);
            }
        }
    }
    ab_end(A, delta, cnt);
}

// ------------------------------------------------------------------ rebalance
constexpr int RB_SHIFT = 10;   // key = segment << 10 | loss bucket

// Candidates (vertices of overweight parts) in vertex order with key (source <<
// 10 | bucket(loss)): k_rb_count counts those of every tile of PER * 256
// vertices, k_rb_collect adds up the counts of the tiles before its own and
// writes them, clearing the locks and copying the partition (the state before
// the step) on the way.  From kRbWide vertices on a thread takes 32 consecutive
// ones in 16-byte loads and stores (256^3 grid, level 0, one overweight part in
// 32: 8 + 48 us against 200 us for flags, a scan of them and a gather); below, one
// (a warp's 32 rounds of writes are a chain of load latencies: 26 us on 250 K
// vertices).
constexpr int64_t kRbWide = 1 << 20;
constexpr int RB_PER = 32;             // vertices per thread on large levels
// over flags of the parts in dynamic shared memory (k bytes)
__device__ __forceinline__ void rb_over(const int64_t* __restrict__ pw, int64_t Lmax, int32_t k, uint8_t* over) {
    for (int q = threadIdx.x; q < k; q += blockDim.x) over[q] = pw[q] > Lmax;
    __syncthreads();
}
// a thread's 32 vertices from v0 on (v0 a multiple of 32): bit i of the result
// says whether vertex v0 + i lies in an overweight part; copy (may be nullptr)
// and lock receive the parts and zeros
template <class PT>
__device__ __forceinline__ uint32_t rb_mask(int64_t v0, int64_t n, const PT* __restrict__ pc, const uint8_t* over,
                                            PT* __restrict__ copy, uint8_t* __restrict__ lock) {
    constexpr int V = 16 / sizeof(PT), NV = RB_PER / V;
    uint32_t m = 0;
    if (v0 + RB_PER <= n) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint4 x = *reinterpret_cast<const uint4*>(pc + v0 + i * V);
            if (copy) *reinterpret_cast<uint4*>(copy + v0 + i * V) = x;
            const uint32_t word[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const uint32_t p = (word[j * sizeof(PT) / 4] >> (8 * (j * sizeof(PT) % 4))) & (uint32_t)(PT)~(PT)0;
                m |= (over[p] ? 1u : 0u) << (i * V + j);
            }
        }
        if (lock) {
            reinterpret_cast<uint4*>(lock + v0)[0] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4*>(lock + v0)[1] = make_uint4(0, 0, 0, 0);
        }
    } else {
        for (int i = 0; i < RB_PER && v0 + i < n; ++i) {
            const PT p = pc[v0 + i];
            if (copy) copy[v0 + i] = p;
            if (lock) lock[v0 + i] = 0;
            m |= (over[p] ? 1u : 0u) << i;
        }
    }
    return m;
}
template <class PT, int PER>
__global__ void __launch_bounds__(RT) k_rb_count(int64_t n, const PT* __restrict__ pc, const int64_t* __restrict__ pw,
                                                 int64_t Lmax, int32_t k, int32_t* __restrict__ cnt) {
    extern __shared__ uint8_t rb_ov[];
    __shared__ int32_t s_cnt[RW];
    rb_over(pw, Lmax, k, rb_ov);
    const int64_t v0 = ((int64_t)blockIdx.x * RT + threadIdx.x) * PER;
    int32_t c;
    if (PER == 1) c = v0 < n && rb_ov[pc[v0]] ? 1 : 0;
    else c = __popc(rb_mask<PT>(v0, n, pc, rb_ov, nullptr, nullptr));
    c = (int32_t)__reduce_add_sync(0xffffffffu, (uint32_t)c);
    if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t t = 0;
        for (int i = 0; i < RW; ++i) t += s_cnt[i];
        cnt[blockIdx.x] = t;
    }
}
template <class PT, int PER>
__global__ void __launch_bounds__(RT) k_rb_collect(int64_t n, const PT* __restrict__ pc, const int64_t* __restrict__ pw,
                                                   int64_t Lmax, int32_t k, const int32_t* __restrict__ cnt,
                                                   int64_t ncand, const int32_t* __restrict__ gain,
                                                   PT* __restrict__ pc_old, uint8_t* __restrict__ lock,
                                                   uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    extern __shared__ uint8_t rb_ov[];
    __shared__ int64_t sh[33];
    rb_over(pw, Lmax, k, rb_ov);
    const int lane = threadIdx.x & 31;
    int64_t before = 0, s = 0, all;
    for (int64_t t = threadIdx.x; t < blockIdx.x; t += RT) s += cnt[t];
    block_excl_scan<int64_t>(s, sh, before);
    const int64_t v0 = ((int64_t)blockIdx.x * RT + threadIdx.x) * PER;
    if (PER == 1) {
        const int32_t p = v0 < n ? (int32_t)pc[v0] : -1;
        const bool take = p >= 0 && rb_ov[p];
        if (p >= 0) { pc_old[v0] = (PT)p; lock[v0] = 0; }
        const int64_t at = before + block_excl_scan<int64_t>(take ? 1 : 0, sh, all);
        if (take && GP_IN(at, ncand)) {
            keys[at] = ((uint64_t)(uint32_t)p << RB_SHIFT) | loss_bucket(-gain[v0]);
            vals[at] = (int32_t)v0;
        }
        return;
    }
    const uint32_t mine = rb_mask<PT>(v0, n, pc, rb_ov, pc_old, lock);
    const int64_t at0 = before + block_excl_scan<int64_t>(__popc(mine), sh, all);
    // the warp writes the 32 vertices of each lane together
    for (int i = 0; i < 32; ++i) {
        const uint32_t m = __shfl_sync(0xffffffffu, mine, i);
        if (!m) continue;
        const int64_t at = __shfl_sync(0xffffffffu, at0, i) + __popc(m & ((1u << lane) - 1u));
        if (((m >> lane) & 1u) && GP_IN(at, ncand)) {
            const int64_t v = v0 + (int64_t)(i - lane) * RB_PER + lane;
            keys[at] = ((uint64_t)(uint32_t)pc[v] << RB_SHIFT) | loss_bucket(-gain[v]);
            vals[at] = (int32_t)v;
        }
    }
}

// first index of every key segment (key >> RB_SHIFT = d, d = 0..k) of a
// sorted candidate list: k + 1 searches instead of one per candidate
// (a warp per segment, 32 probes at a time)
template <class F>
__device__ __forceinline__ int64_t warp_first(int64_t lo, int64_t hi, F below);
__global__ void k_seg_first(const int64_t* __restrict__ cnt, const uint64_t* __restrict__ keys, int32_t k,
                            int64_t* __restrict__ first) {
    const int64_t n = *cnt;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int d = w; d <= k; d += nw) {
        const int64_t f = warp_first(0, n, [&](int64_t i) { return (int64_t)(keys[i] >> RB_SHIFT) < d; });
        if ((threadIdx.x & 31) == 0) first[d] = f;
    }
}

// What the sorted candidates let each source part give up, in one block: a
// source keeps the prefix of its candidates whose weight before the candidate
// is below its excess.  Also the part weights before the step and the
// concatenated free capacities (strong).  pre: exclusive weight prefix of the
// list (pre[ncand] = total).
struct RbPlan {
    int64_t* seg;      // first candidate of the source
    int64_t* acc;      // candidates it keeps
    int64_t* off;      // kept candidates of the sources before it
    int64_t* woff;     // and their weight
    int64_t* cum;      // k + 1: free capacity of the parts before
    int64_t* snap;     // part weights before the step
    int64_t* n2;       // kept candidates in all
};
// First index in [lo, hi) where below(i) turns false (below is true up to
// there), by a warp: 32 probes at a time.
template <class F>
__device__ __forceinline__ int64_t warp_first(int64_t lo, int64_t hi, F below) {
    const int lane = threadIdx.x & 31;
    while (lo < hi) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t i = lo + (int64_t)lane * step;
        const uint32_t m = __ballot_sync(0xffffffffu, i < hi && below(i));   // a run of low lanes
        const int t = __popc(m);
        if (t == 0) return lo;
        hi = lo + (int64_t)t * step < hi ? lo + (int64_t)t * step : hi;   // probe t (if any) is not below
        lo = lo + (int64_t)(t - 1) * step + 1;                             // probe t - 1 is
    }
    return lo;
}
__global__ void __launch_bounds__(GP_MAX_K) k_rb_plan(int64_t ncand, const uint64_t* __restrict__ keys,
                                                      const int64_t* __restrict__ pre, const int64_t* __restrict__ pw,
                                                      int64_t Lmax, int32_t k, RbPlan P) {
    __shared__ int64_t sh[33];
    __shared__ int64_t s_a[GP_MAX_K], s_w[GP_MAX_K];
    // a warp per part: its segment, and the prefix that covers its excess
    for (int q = threadIdx.x >> 5; q < k; q += blockDim.x >> 5) {
        const int64_t x = pw[q];
        int64_t s = 0, a = 0, wa = 0;
        if (x > Lmax) {
            s = warp_first(0, ncand, [&](int64_t i) { return (int64_t)(keys[i] >> RB_SHIFT) < q; });
            const int64_t e = warp_first(s, ncand, [&](int64_t i) { return (int64_t)(keys[i] >> RB_SHIFT) <= q; });
            const int64_t p0 = s < ncand ? pre[s] : 0;
            const int64_t f = warp_first(s, e, [&](int64_t i) { return pre[i] - p0 < x - Lmax; });
            a = f - s;
            wa = a > 0 ? pre[f] - p0 : 0;
        }
        if ((threadIdx.x & 31) == 0) {
            s_a[q] = a; s_w[q] = wa;
            P.seg[q] = s; P.acc[q] = a; P.snap[q] = x;
        }
    }
    __syncthreads();
    const int q = threadIdx.x;
    const int64_t x = q < k ? pw[q] : 0;
    int64_t tot;
    int64_t e = block_excl_scan<int64_t>(q < k ? s_a[q] : 0, sh, tot);
    if (q < k) P.off[q] = e;
    if (q == 0) *P.n2 = tot;
    e = block_excl_scan<int64_t>(q < k ? s_w[q] : 0, sh, tot);
    if (q < k) P.woff[q] = e;
    e = block_excl_scan<int64_t>(q < k && x <= Lmax ? Lmax - x : 0, sh, tot);
    if (q < k) P.cum[q] = e;
    if (q == 0) P.cum[k] = tot;
}

// weak: kept candidates, in list order, re-keyed by (dest << 10 | bucket)
__global__ void k_rb_rekey(int64_t cnt, const uint64_t* __restrict__ keys, const int32_t* __restrict__ vals, RbPlan P,
                           const int32_t* __restrict__ dest, uint64_t* __restrict__ keys2, int32_t* __restrict__ vals2) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t key = keys[i];
        const int64_t q = (int64_t)(key >> RB_SHIFT), r = i - P.seg[q];
        if (r >= P.acc[q]) continue;
        const int32_t v = vals[i];
        const int64_t j = P.off[q] + r;
        if (!GP_IN(j, cnt)) continue;
        keys2[j] = ((uint64_t)(uint32_t)dest[v] << RB_SHIFT) | (key & ((1ull << RB_SHIFT) - 1));
        vals2[j] = v;
    }
}

// part-weight changes and moves of a block, added to the global totals once
// per part (dynamic shared memory: k int32).  The vertex weights add up to less
// than 2^31, so every partial sum fits in 32 bits; a 64-bit shared add is a
// compare-and-swap loop, which a rebalance step (most moves leave one part)
// drives into full contention: k_rb_step_cta on R-MAT 20 (k = 64), longest launch 757 -> 123 us
__device__ __forceinline__ void rb_delta_begin(int32_t* delta, int32_t k) {
    for (int q = threadIdx.x; q < k; q += blockDim.x) delta[q] = 0;
    __syncthreads();
}
__device__ __forceinline__ void rb_delta_end(int32_t* delta, int32_t k, AbCount cnt, int64_t* __restrict__ pw,
                                             int64_t* __restrict__ step) {
    cnt.moves = warp_sum(cnt.moves);
    cnt.deg = warp_sum(cnt.deg);
    if ((threadIdx.x & 31) == 0 && cnt.moves) {
        atomicAdd((unsigned long long*)&step[S_STEP_MOVES], (unsigned long long)cnt.moves);
        atomicAdd((unsigned long long*)&step[S_MVDEG], (unsigned long long)cnt.deg);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < k; q += blockDim.x)
        if (delta[q]) atomicAdd((unsigned long long*)&pw[q], (unsigned long long)(int64_t)delta[q]);
}

// weak: keep moves whose destination prefix fits the capacity; apply
__global__ void k_rb_weak_apply(const int64_t* __restrict__ cnt_dev, const uint64_t* __restrict__ keys,
                                const int64_t* __restrict__ segf,
                                const int32_t* __restrict__ vals, const int64_t* __restrict__ pre,
                                const int32_t* __restrict__ vw, const int64_t* __restrict__ pw_snap, int64_t Lmax,
                                int32_t k, void* __restrict__ pc, int pcb, uint8_t* __restrict__ lock,
                                int64_t* __restrict__ pw, const int64_t* __restrict__ rp, int64_t* __restrict__ step) {
    extern __shared__ int32_t rb_delta[];
    rb_delta_begin(rb_delta, k);
    AbCount nm;
    const int64_t cnt = *cnt_dev;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t d = keys[i] >> RB_SHIFT;
        const int64_t s = segf[d];
        const int32_t v = vals[i];
        const int64_t wv = vw ? vw[v] : 1;
        if ((pre[i] - pre[s]) + wv <= Lmax - pw_snap[d]) {
            const int32_t p = load_pc(pc, pcb, v);
            store_pc(pc, pcb, v, (int32_t)d);
            lock[v] = 1;
            if (GP_IN(d, k) && GP_IN(p, k)) {
                atomicAdd(&rb_delta[d], (int32_t)wv);
                atomicAdd(&rb_delta[p], -(int32_t)wv);
            }
            ++nm.moves;
            nm.deg += rp[v + 1] - rp[v];
        }
    }
    rb_delta_end(rb_delta, k, nm, pw, step);
}

// strong: kept candidates laid over the concatenated free capacities
__global__ void k_rb_strong_apply(int64_t cnt, const uint64_t* __restrict__ keys, const int32_t* __restrict__ vals,
                                  const int64_t* __restrict__ P, RbPlan plan, const int32_t* __restrict__ vw,
                                  int32_t k, void* __restrict__ pc, int pcb,
                                  uint8_t* __restrict__ lock, int64_t* __restrict__ pw,
                                  const int64_t* __restrict__ rp, int64_t* __restrict__ step) {
    const int64_t* __restrict__ cum = plan.cum;
    extern __shared__ int32_t rb_delta[];
    rb_delta_begin(rb_delta, k);
    AbCount nm;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t src = (int64_t)(keys[i] >> RB_SHIFT), s = plan.seg[src];
        if (i - s >= plan.acc[src]) continue;
        const int64_t pre = plan.woff[src] + (P[i] - P[s]);
        if (pre >= cum[k]) continue;
        // q with cum[q] <= pre < cum[q+1]: last index with cum <= pre
        int lo = 0, hi = k;  // search in cum[0..k]
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (cum[mid] <= pre) lo = mid; else hi = mid - 1;
        }
        const int q = lo;
        const int32_t v = vals[i];
        const int64_t wv = vw ? vw[v] : 1;
        if (q < k && pre + wv <= cum[q + 1]) {
            const int32_t p = load_pc(pc, pcb, v);
            store_pc(pc, pcb, v, q);
            lock[v] = 1;
            if (GP_IN(p, k)) {
                atomicAdd(&rb_delta[q], (int32_t)wv);
                atomicAdd(&rb_delta[p], -(int32_t)wv);
            }
            ++nm.moves;
            nm.deg += rp[v + 1] - rp[v];
        }
    }
    rb_delta_end(rb_delta, k, nm, pw, step);
}

// ------------------------------------------------------------------ cut change of a step
// After a move step whose next pass will rebalance: the change of the directed
// cross weight, from the rows of the moved vertices alone (those whose part
// differs between the partition before and after).  An entry (v, u) of a moved
// v changes by w ([new v != new u] - [old v != old u]); its mirror (u, v), the
// same weight on a symmetric graph, is counted with it when u did not move.
// Exact integers, so that the pass after it need not sweep the rows it looks
// for no move in, and a pass that would end the level sweeps nothing: on the
// 256^3 grid (k = 32) the rebalancing passes, two thirds of all, sweep one part in
// 32 instead of every row: all its passes take 42 -> 30 ms, k_track 3.2 ms; on
// R-MAT 24 they take 131 -> 102 ms, k_track 13.  Left out when the next pass sweeps
// every row anyway: no overweight part and a level that may go on, or moved rows
// of more than track_deg entries.  Blocks [0, nitems) take the pieces of the heavy
// rows, range_blocks the warp rows by the connectivity pass's ranges (block_unit:
// moved rows' lengths differ widely; one range of vertices per block, short and
// long rows alike, took 49 ms on R-MAT 24 instead of 13), the others compare the
// partitions over a range of vertices each, 4 bytes per lane, and queue the moved
// short rows, which then get a thread each.
struct TrackArgs {
    DGraph g;
    int32_t k;
    int64_t Lmax;
    const int64_t* pw;
    const void* pc;             // after the step
    const void* pc_old;         // before it
    int64_t* step;              // its status block
    int64_t track_deg;
    const int32_t* bucket[3];
    int64_t nbucket[3];
    const int64_t* wfirst;      // the connectivity pass's ranges of longer rows
    int64_t nranges, range_blocks;
    int32_t range;              // vertices per block, a multiple of 4 * RT up to kTrackRange
    int always;                 // also when no part is overweight (the next pass may be the level's last)
    const int32_t* heavy;
    const int32_t* item_row;
    const int64_t* item_beg;
    const int64_t* item_end;
    int64_t nitems;
};
constexpr int kTrackRange = 8192;
// part of u before and after the step (both in one word per vertex, filled by a
// kernel of its own, measured the same on R-MAT 24: 13.2 + 0.4 ms against 12.7)
template <class PT>
__device__ __forceinline__ uint32_t track_pair(const TrackArgs& T, int32_t u) {
    return (uint32_t)__ldg((const PT*)T.pc_old + u) | ((uint32_t)__ldg((const PT*)T.pc + u) << (8 * sizeof(PT)));
}
__device__ __forceinline__ bool track_runs(const TrackArgs& T) {
    if (T.step[S_STEP_MOVES] == 0 || T.step[S_MVDEG] > T.track_deg) return false;   // uniform
    int over = 0;
    for (int q = threadIdx.x; q < T.k; q += RT) over |= T.pw[q] > T.Lmax ? 1 : 0;
    return __syncthreads_or(over) || T.always;
}
template <class PT>
__device__ __forceinline__ int32_t track_change(uint32_t x, int32_t po, int32_t pn, int32_t w) {
    const int32_t uo = (int32_t)(x & (PT)~(PT)0), un = (int32_t)(x >> (8 * sizeof(PT)));
    const int32_t c = (pn != un ? 1 : 0) - (po != uo ? 1 : 0);
    return uo == un ? 2 * c * w : c * w;
}
// this thread's part (t of nt) of entries [beg, end), four consecutive ones at a time
template <class PT>
__device__ __forceinline__ int64_t track_sum(const TrackArgs& T, int64_t beg, int64_t end, int t, int nt,
                                             int32_t po, int32_t pn) {
    const bool v4 = aligned16(T.g.ci) && aligned16(T.g.ew);
    int64_t sum = 0;
    for (int64_t base = beg & ~(int64_t)3; base < end; base += 4 * (int64_t)nt) {
        int32_t u[4], w[4];
        uint32_t x[4];
        const int64_t e4 = base + 4 * t;
        ld4_row(T.g.ci, e4, beg, end, v4, -1, u);
        if (T.g.ew) ld4_row(T.g.ew, e4, beg, end, v4, 0, w);
        else {
#pragma unroll
            for (int c = 0; c < 4; ++c) w[c] = 1;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = u[c] >= 0 && GP_IN(u[c], T.g.n) ? track_pair<PT>(T, u[c]) : 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (u[c] >= 0 && GP_IN(u[c], T.g.n)) sum += track_change<PT>(x[c], po, pn, w[c]);
    }
    return sum;
}
template <class PT>
__global__ void __launch_bounds__(RT) k_track(TrackArgs T) {
    __shared__ int32_t s_queue[kTrackRange];
    __shared__ int32_t s_cnt;
    __shared__ uint32_t s_next;
    __shared__ int64_t s_red[RW];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) { s_cnt = 0; s_next = 0; }
    if (!track_runs(T)) return;
    constexpr int PB = 8 * sizeof(PT);
    int64_t acc = 0;
    if ((int64_t)blockIdx.x < T.nitems) {
        const uint32_t x = track_pair<PT>(T, T.heavy[T.item_row[blockIdx.x]]);
        const int32_t po = (int32_t)(x & (PT)~(PT)0), pn = (int32_t)(x >> PB);
        if (po != pn) acc = track_sum<PT>(T, T.item_beg[blockIdx.x], T.item_end[blockIdx.x], threadIdx.x, RT, po, pn);
    } else if ((int64_t)blockIdx.x < T.nitems + T.range_blocks) {
        const int64_t U2 = T.nbucket[2], U21 = U2 + T.nbucket[1];
        for (;;) {
            const int64_t r = block_unit(&s_next, blockIdx.x - T.nitems, T.range_blocks);
            if (r >= T.nranges) break;
            const int64_t u0 = T.wfirst[r], u1 = T.wfirst[r + 1] < U21 ? T.wfirst[r + 1] : U21;
            for (int64_t ub = u0; ub < u1; ub += 32) {
                const int64_t u = ub + lane;
                int32_t po = 0, pn = 0;
                int64_t beg = 0, end = 0;
                if (u < u1) {
                    const int32_t v = u < U2 ? T.bucket[2][u] : T.bucket[1][u - U2];
                    const uint32_t x = track_pair<PT>(T, v);
                    po = (int32_t)(x & (PT)~(PT)0); pn = (int32_t)(x >> PB);
                    if (po != pn) { beg = T.g.rp[v]; end = T.g.rp[v + 1]; }
                }
                uint32_t todo = __ballot_sync(0xffffffffu, po != pn);
                while (todo) {
                    const int j = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int64_t b = __shfl_sync(0xffffffffu, beg, j), e = __shfl_sync(0xffffffffu, end, j);
                    acc += track_sum<PT>(T, b, e, lane, 32, __shfl_sync(0xffffffffu, po, j), __shfl_sync(0xffffffffu, pn, j));
                }
            }
        }
    } else {
        constexpr int per = 4 / sizeof(PT);   // ids per 4-byte word
        const int64_t v0 = ((int64_t)blockIdx.x - T.nitems - T.range_blocks) * T.range;
        for (int32_t i = threadIdx.x * per; i < T.range; i += RT * per) {
            const int64_t v = v0 + i;
            uint32_t a = 0, b = 0;
            if (v + per <= T.g.n) {
                a = ((const uint32_t*)T.pc_old)[v / per];
                b = ((const uint32_t*)T.pc)[v / per];
            } else {
                for (int j = 0; j < per && v + j < T.g.n; ++j) {
                    a |= (uint32_t)((const PT*)T.pc_old)[v + j] << (8 * sizeof(PT) * j);
                    b |= (uint32_t)((const PT*)T.pc)[v + j] << (8 * sizeof(PT) * j);
                }
            }
            const uint32_t x = a ^ b;
            if (!__any_sync(0xffffffffu, x != 0)) continue;
#pragma unroll
            for (int j = 0; j < per; ++j) {
                const bool mv = ((x >> (8 * sizeof(PT) * j)) & (PT)~(PT)0) != 0;
                const uint32_t m = __ballot_sync(0xffffffffu, mv);
                if (!m) continue;
                int32_t at = 0;
                if (lane == __ffs(m) - 1) at = atomicAdd(&s_cnt, __popc(m));
                at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
                if (mv && GP_IN(at, kTrackRange)) s_queue[at] = (int32_t)(v + j);
            }
        }
        __syncthreads();
        const int32_t cnt = s_cnt;
        for (int32_t i = threadIdx.x; i < cnt; i += RT) {
            const int32_t v = s_queue[i];
            const int64_t beg = T.g.rp[v], end = T.g.rp[v + 1];
            if (end - beg > kShortDeg) continue;
            const uint32_t x = track_pair<PT>(T, v);
            const int32_t po = (int32_t)(x & (PT)~(PT)0), pn = (int32_t)(x >> PB);
            for (int64_t e = beg; e < end; ++e) {
                const int32_t u = __ldcs(&T.g.ci[e]);
                if (GP_IN(u, T.g.n))
                    acc += track_change<PT>(track_pair<PT>(T, u), po, pn, T.g.ew ? __ldcs(&T.g.ew[e]) : 1);
            }
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) s_red[w] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int i = 0; i < RW; ++i) s += s_red[i];
        if (s) atomicAdd((unsigned long long*)&T.step[S_DELTA], (unsigned long long)s);
    }
}

// ------------------------------------------------------------------ projection, weights, cut
__global__ void k_project(int64_t n, const int32_t* __restrict__ cmap, const int32_t* __restrict__ pc,
                          int32_t* __restrict__ pf) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        pf[v] = pc[cmap[v]];
}

// unit weights: 32-bit shared counts; given weights: 64-bit sums (an edge-cut
// call takes weights whose total is not checked against 2^31)
__global__ void k_part_weights(int64_t n, const int32_t* __restrict__ part, const int32_t* __restrict__ vw, int32_t k,
                               int64_t* __restrict__ pw) {
    extern __shared__ int64_t spw[];
    int32_t* cnt = (int32_t*)spw;
    for (int q = threadIdx.x; q < k; q += blockDim.x) spw[q] = 0;
    __syncthreads();
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        if (vw) atomicAdd((unsigned long long*)&spw[part[v]], (unsigned long long)vw[v]);
        else atomicAdd(&cnt[part[v]], 1);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < k; q += blockDim.x) {
        const int64_t x = vw ? spw[q] : (int64_t)cnt[q];
        if (x) atomicAdd((unsigned long long*)&pw[q], (unsigned long long)x);
    }
}

// directed cross weight, entry-sliced (csr_sweep): each lane of a window also
// holds its row's part; up to kCutG groups of 32 entries have their column ids
// loaded, then their neighbours' parts gathered, together.  PT: part ids of 1
// byte where a compacted copy pays (kCutCompact), else the caller's int32
constexpr int kCutG = 4;
template <class PT>
__global__ void __launch_bounds__(RT, 6) k_cut(DGraph g, int64_t slice, const PT* __restrict__ part,
                                            int64_t* __restrict__ cross2) {
    __shared__ int64_t s_red[RW];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t n = g.n;
    int64_t acc = 0;
    csr_sweep<kCutG, int32_t>(g.rp, n, g.m, slice, [&](int64_t r, int64_t) { return r < n ? (int32_t)part[r] : 0; },
                       [&](auto full, int64_t o, int64_t lim, int64_t o0, int64_t, int32_t s, int32_t pv) {
        int32_t u[kCutG], pr[kCutG], wt[kCutG];
#pragma unroll
        for (int q = 0; q < kCutG; ++q) {
            u[q] = -1; pr[q] = 0; wt[q] = 0;
            if (!full && o + 32 * q >= lim) continue;
            const int64_t oi = o + 32 * q + lane;
            pr[q] = __shfl_sync(0xffffffffu, pv, csr_lane(s, (int32_t)(oi - o0)));
            if (full || oi < lim) {
                u[q] = __ldcs(&g.ci[oi]);
                wt[q] = g.ew ? __ldcs(&g.ew[oi]) : 1;
            }
        }
#pragma unroll
        for (int q = 0; q < kCutG; ++q) u[q] = u[q] >= 0 && GP_IN(u[q], n) ? (int32_t)__ldg(&part[u[q]]) : pr[q];
#pragma unroll
        for (int q = 0; q < kCutG; ++q) acc += u[q] != pr[q] ? wt[q] : 0;
    });
    acc = warp_sum(acc);
    if (lane == 0) s_red[w] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int i = 0; i < RW; ++i) s += s_red[i];
        if (s) atomicAdd((unsigned long long*)cross2, (unsigned long long)s);
    }
}

void project(Ctx& c, const Level& fine, const int32_t* part_coarse, int32_t* part_fine) {
    k_project<<<grid_for(fine.g.n, 256), 256, 0, c.s>>>(fine.g.n, fine.cmap, part_coarse, part_fine);
    GP_LAUNCHED(c);
    c.bytes += 12 * fine.g.n;
}

void part_weights(Ctx& c, const DGraph& g, const int32_t* part, int32_t k, int64_t* pw) {
    memset_async(c, pw, 0, sizeof(int64_t) * k);
    k_part_weights<<<grid_for(g.n, 256, c.sm_count * 4), 256, sizeof(int64_t) * k, c.s>>>(g.n, part, g.vw, k, pw);
    GP_LAUNCHED(c);
    c.bytes += 4 * g.n + (g.vw ? 4 * g.n : 0);
}

// entries from which the cut gathers from a copy of the parts in bytes, on graphs
// of a mean degree of 8 and more (the copy costs 5 bytes a vertex and a launch).  Whole
// calls from int32 and from bytes, the copy included: R-MAT 16 / 17 (1.8 and 3.7 M
// entries) 68 / 78 us and 70 / 80, Erdos-Renyi of 2.6 M with weights 82 and 84; R-MAT 18 /
// 19 / 20 / 21 / 22 (7.6 to 128 M) 101 / 126 / 189 / 315 / 650 and 93 / 118 / 180 / 304 / 626;
// Erdos-Renyi, whose parts are met evenly, of 10 / 60 M 127 / 378 and 130 / 386
constexpr int64_t kCutCompact = 1 << 22;
__global__ void k_compact_part(int64_t n, const int32_t* __restrict__ part, void* pc, int pcb);
void cut_and_weights(Ctx& c, const DGraph& g, const int32_t* part, int32_t k, int64_t* d_cross2, int64_t* d_pw) {
    memset_async(c, d_cross2, 0, sizeof(int64_t));
    const int64_t slice = csr_slice(g.m, c.sm_count);
    const int grid = grid_for((g.m + slice - 1) / slice * 32, RT, c.sm_count * c.ctas_per_sm);
    uint8_t* pc = nullptr;
    auto mk = c.tmp->save();
    if (k <= 256 && g.m >= kCutCompact && g.m >= 8 * g.n) {
        try {
            pc = c.tmp_alloc<uint8_t>(g.n);
        } catch (const GpError&) {   // no memory for it: the caller's array serves
            cudaGetLastError();
        }
    }
    if (pc) {
        k_compact_part<<<grid_for(g.n, 256), 256, 0, c.s>>>(g.n, part, pc, 1);
        GP_LAUNCHED(c);
        k_cut<uint8_t><<<grid, RT, 0, c.s>>>(g, slice, pc, d_cross2);
    } else {
        k_cut<int32_t><<<grid, RT, 0, c.s>>>(g, slice, part, d_cross2);
    }
    GP_LAUNCHED(c);
    c.tmp->restore(mk);
    c.bytes += 8 * (g.n + 1) + 8 * g.m + (g.ew ? 4 * g.m : 0) + 4 * g.n;
    if (d_pw) part_weights(c, g, part, k, d_pw);
}

// ------------------------------------------------------------------ one-CTA refinement
// A level with at most small_level_n (<= kCtaMaxN) vertices and no row longer
// than kHeavyDeg is refined by one thread block in one launch: the whole
// iteration loop of refine_level (connectivity pass, label propagation with
// afterburner, weak/strong rebalancing, best-state tracking and the stop
// rules) runs on the device, with the same per-row helpers as the
// multi-kernel path and the same integer results.  Rebalance candidates are
// sorted by a bitonic network in shared memory on unique 64-bit keys
// (source, loss bucket, id), then (destination, loss bucket, source, id).
// The block's 64 registers per thread hold the short rows' thread-per-row form only
// with spills (364 and 336 bytes); it still takes a random geometric graph of 8,000
// vertices, k = 16, 3.7 -> 1.5 ms against a lane group per row, and 128 graphs of 1,000
// vertices in one batch 3.1 -> 2.4.
constexpr int CT = 1024, CW = CT / 32;
constexpr int64_t kCtaMaxN = 16384;                 // candidates sorted in shared memory (8 B each)
// A rebalance step of at most this many candidates is taken by one block
// (k_rb_step_cta), of more by about 20 launches over the whole chip.  1024, 2048,
// 4096, 16384: weighted RGG 150k k = 300 7.8 / 7.2 / 7.0 / 7.0 ms, R-MAT 20 k = 64
// 44.8 / 44.1 / 44.2 / 45.5 ms, Chung-Lu 262k k = 64 17.4 / 16.8 / 16.6 / 17.3 ms.
constexpr int64_t kRbCta = 4096;

struct CtaRefineArgs {
    DGraph g;
    int32_t k;
    int64_t Lmax;
    int32_t den, max_iters, patience, strong_after;
    const int32_t* bucket[3];
    int64_t nbucket[3];
    int32_t* part;
    int32_t* part_next;
    uint8_t* lock;
    uint8_t* lock_next;
    int32_t* best;
    int64_t* pw;          // in: part weights of part; out: those of the kept state
    int32_t* dest;
    int32_t* gain;
    int64_t* status;      // counters of the per-row helpers
    int32_t* clist[3];
    int64_t* pre;         // n scratch
    int32_t* flag;        // n scratch
    uint64_t* gkeys;      // n scratch
    int32_t* tr_arrays;   // optional: per step dest[n], gain[n], part[n]
    int64_t* tr_scalars;  // optional: per step mode, cut before, max part weight before, moves
    int64_t* out;         // [0] steps
};

__device__ __forceinline__ int64_t cta_sum(int64_t x, int64_t* sh) {
    int64_t tot;
    block_excl_scan<int64_t>(x, sh, tot);
    return tot;
}

// exclusive prefix sums of val(i), i < cnt, in index order into out; returns the total
template <class F>
__device__ int64_t cta_scan(int64_t cnt, F val, int64_t* out, int64_t* sh) {
    const int64_t per = (cnt + CT - 1) / CT;
    const int64_t b = (int64_t)threadIdx.x * per, e = b + per < cnt ? b + per : cnt;
    int64_t s = 0;
    for (int64_t i = b; i < e; ++i) s += val(i);
    int64_t tot;
    int64_t base = block_excl_scan<int64_t>(s, sh, tot);
    for (int64_t i = b; i < e; ++i) { const int64_t x = val(i); out[i] = base; base += x; }
    __syncthreads();
    return tot;
}

// ascending bitonic sort of N (a power of two) unique keys in shared memory.
// Compare-exchange steps whose partner is within 16 positions run on
// registers with warp shuffles (element i sits in lane i % 32 of its warp,
// partner i ^ stride in the same warp); wider steps go through shared memory,
// one block barrier each.
__device__ void cta_bitonic(uint64_t* a, int N) {
    const int tid = threadIdx.x;
    const int E = N > CT ? N / CT : 1;
    // strides top, top/2, ..., 1 of merge size `size` (size 0: every size 2..top*2)
    auto warp_steps = [&](int size, int top) {
        for (int e = 0; e < E; ++e) {
            const int i = e * CT + tid;
            const bool valid = i < N;
            uint64_t x = valid ? a[i] : ~0ull;
            const int s0 = size ? size : 2, s1 = size ? size : 2 * top;
            for (int sz = s0; sz <= s1; sz <<= 1) {
                for (int stride = size ? top : (sz >> 1); stride > 0; stride >>= 1) {
                    const uint64_t y = __shfl_xor_sync(0xffffffffu, x, stride);
                    const bool up = (i & sz) == 0, lower = (i & stride) == 0;
                    x = (lower == up) ? (x < y ? x : y) : (x < y ? y : x);
                }
            }
            if (valid) a[i] = x;
        }
        __syncthreads();
    };
    // merge sizes up to 32: within warps
    warp_steps(0, (N < 32 ? N : 32) >> 1);
    for (int size = 64; size <= N; size <<= 1) {
        for (int stride = size >> 1; stride >= 32; stride >>= 1) {
            for (int i = tid; i < N; i += CT) {
                const int j = i ^ stride;
                if (j > i) {
                    const uint64_t x = a[i], y = a[j];
                    const bool up = (i & size) == 0;
                    if ((x > y) == up) { a[i] = y; a[j] = x; }
                }
            }
            __syncthreads();
        }
        warp_steps(size, 16);
    }
}

// first index in [0, i] whose key has the same segment (key >> shift) as key i
__device__ __forceinline__ int cta_seg_start(const uint64_t* a, int i, int shift) {
    const uint64_t seg = a[i] >> shift;
    int lo = 0, hi = i;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((a[mid] >> shift) < seg) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// One rebalance step by one thread block (the rules of the multi-kernel path
// below: candidates ordered (source, loss bucket, id); a source keeps the
// prefix before the vertex below its excess; weak: per destination, ordered
// (destination, loss bucket, source, id), moves that fit the remaining
// capacity; strong: kept moves laid over the concatenated free capacities).
// cand: the candidates in vertex order (ncand of them), or nullptr to take
// every v < n of an overweight part.  s_pw (shared) is updated; returns this
// thread's moves.  Needs ncand <= kCtaMaxN.
struct RbCta {
    const int32_t* vw;
    void* pc;                   // the partition
    int pcb;                    // its bytes per id
    void* pc_old;               // receives the partition before the step (nullptr, or a candidate list:
                                // not wanted / copied already)
    const int64_t* rp;          // row pointers (nullptr: entries of moved rows not wanted)
    uint8_t* lock;
    const int32_t* dest;
    const int32_t* gain;
    int64_t* pre;
    int32_t* flag;
    uint64_t* gkeys;
    int32_t k;
    int64_t Lmax;
};

__device__ AbCount cta_rebalance(const RbCta& R, int mode, int64_t n, const int32_t* cand, int64_t ncand_in,
                                 int32_t* s_pw, int32_t* s_snap, int64_t* s_cum, uint64_t* s_keys, int64_t* sh) {
    const int32_t k = R.k;
    const int64_t Lmax = R.Lmax;
    uint8_t* lock = R.lock;
    AbCount cnt;
    auto moved = [&](uint32_t v) {
        ++cnt.moves;
        if (R.rp) cnt.deg += R.rp[v + 1] - R.rp[v];
    };
    for (int q = threadIdx.x; q < k; q += CT) s_snap[q] = s_pw[q];
    __syncthreads();
    int64_t ncand = ncand_in;
    auto key1 = [&](uint32_t v) -> uint64_t {
        const uint64_t key = ((uint64_t)(uint32_t)load_pc(R.pc, R.pcb, v) << RB_SHIFT) | loss_bucket(-R.gain[v]);
        return (key << 32) | v;
    };
    if (cand == nullptr) {
        // candidates in vertex order, then sorted by (source, loss bucket, id)
        auto over = [&](int64_t v) -> int64_t { return s_snap[load_pc(R.pc, R.pcb, v)] > Lmax ? 1 : 0; };
        ncand = cta_scan(n, over, R.pre, sh);
        for (int64_t v = threadIdx.x; v < n; v += CT)
            if (over(v)) s_keys[R.pre[v]] = key1((uint32_t)v);
    } else {
        for (int64_t i = threadIdx.x; i < ncand; i += CT) s_keys[i] = key1((uint32_t)cand[i]);
    }
    int N = 1;
    while (N < ncand) N <<= 1;
    for (int64_t i = ncand + threadIdx.x; i < N; i += CT) s_keys[i] = ~0ull;
    __syncthreads();
    cta_bitonic(s_keys, N);
    auto vwt = [&](uint32_t v) -> int64_t { return R.vw ? R.vw[v] : 1; };
    cta_scan(ncand, [&](int64_t i) -> int64_t { return vwt((uint32_t)s_keys[i]); }, R.pre, sh);
    // kept: the source's prefix before the vertex is below its excess
    for (int64_t i = threadIdx.x; i < ncand; i += CT) {
        const uint32_t src = (uint32_t)(s_keys[i] >> (32 + RB_SHIFT));
        const int s0 = cta_seg_start(s_keys, (int)i, 32 + RB_SHIFT);
        R.flag[i] = (R.pre[i] - R.pre[s0]) < (s_snap[src] - Lmax) ? 1 : 0;
    }
    __syncthreads();
    if (mode == 1) {
        // kept moves re-keyed (dest, loss bucket, source, id): 10 + 10 + 10 + 32 bits
        const int64_t n2 = cta_scan(ncand, [&](int64_t i) -> int64_t { return R.flag[i]; }, R.pre, sh);
        for (int64_t i = threadIdx.x; i < ncand; i += CT)
            if (R.flag[i]) {
                const uint64_t key = s_keys[i];
                const uint32_t v = (uint32_t)key, b = (uint32_t)(key >> 32) & ((1u << RB_SHIFT) - 1);
                const uint32_t src = (uint32_t)(key >> (32 + RB_SHIFT));
                R.gkeys[R.pre[i]] = ((((uint64_t)(uint32_t)R.dest[v] << RB_SHIFT | b) << RB_SHIFT | src) << 32) | v;
            }
        __syncthreads();
        int N2 = 1;
        while (N2 < n2) N2 <<= 1;
        for (int64_t i = threadIdx.x; i < N2; i += CT) s_keys[i] = i < n2 ? R.gkeys[i] : ~0ull;
        __syncthreads();
        cta_bitonic(s_keys, N2);
        cta_scan(n2, [&](int64_t i) -> int64_t { return vwt((uint32_t)s_keys[i]); }, R.pre, sh);
        for (int64_t i = threadIdx.x; i < n2; i += CT) {
            const uint32_t v = (uint32_t)s_keys[i];
            const int32_t d = (int32_t)(s_keys[i] >> (32 + 2 * RB_SHIFT));
            const int s0 = cta_seg_start(s_keys, (int)i, 32 + 2 * RB_SHIFT);
            const int64_t wv = vwt(v);
            if ((R.pre[i] - R.pre[s0]) + wv <= Lmax - s_snap[d]) {
                const int32_t p = load_pc(R.pc, R.pcb, v);
                store_pc(R.pc, R.pcb, v, d);
                lock[v] = 1;
                atomicAdd(&s_pw[d], (int32_t)wv);
                atomicAdd(&s_pw[p], -(int32_t)wv);
                moved(v);
            }
        }
    } else {
        // free capacities of the parts within Lmax, concatenated (k <= CT)
        {
            const int64_t f = (threadIdx.x < k && s_snap[threadIdx.x] <= Lmax) ? Lmax - s_snap[threadIdx.x] : 0;
            int64_t tot;
            const int64_t ex = block_excl_scan<int64_t>(f, sh, tot);
            if (threadIdx.x < k) s_cum[threadIdx.x] = ex;
            if (threadIdx.x == 0) s_cum[k] = tot;
            __syncthreads();
        }
        cta_scan(ncand, [&](int64_t i) -> int64_t { return R.flag[i] ? vwt((uint32_t)s_keys[i]) : 0; }, R.pre, sh);
        for (int64_t i = threadIdx.x; i < ncand; i += CT) {
            if (!R.flag[i]) continue;
            const int64_t pre = R.pre[i];
            if (pre >= s_cum[k]) continue;
            int lo = 0, hi = k;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_cum[mid] <= pre) lo = mid; else hi = mid - 1;
            }
            const uint32_t v = (uint32_t)s_keys[i];
            const int64_t wv = vwt(v);
            if (lo < k && pre + wv <= s_cum[lo + 1]) {
                const int32_t p = load_pc(R.pc, R.pcb, v);
                store_pc(R.pc, R.pcb, v, lo);
                lock[v] = 1;
                atomicAdd(&s_pw[lo], (int32_t)wv);
                atomicAdd(&s_pw[p], -(int32_t)wv);
                moved(v);
            }
        }
    }
    __syncthreads();
    return cnt;
}

// one rebalance step of the multi-kernel loop in one launch: candidates are every
// vertex of an overweight part (cand == nullptr, n <= kCtaMaxN; locks cleared and the
// partition copied here) or a compacted list of them; part weights in and out of
// global memory; the step's moves and their entries added to its status block
__global__ void __launch_bounds__(CT, 1) k_rb_step_cta(RbCta R, int mode, int64_t n, const int32_t* cand,
                                                        int64_t ncand, int64_t* pw, int64_t* step) {
    extern __shared__ __align__(16) unsigned char rsm[];
    const int32_t k = R.k;
    int32_t* s_pw = (int32_t*)rsm;               // part weights fit in 32 bits (rb_delta_begin)
    int32_t* s_snap = s_pw + 2 * k;
    int64_t* s_cum = (int64_t*)rsm + 3 * k;
    uint64_t* s_keys = (uint64_t*)(rsm + (((size_t)(4 * k + 1) * 8 + k + 15) & ~(size_t)15));
    __shared__ int64_t sh[33];
    for (int q = threadIdx.x; q < k; q += CT) s_pw[q] = (int32_t)pw[q];
    if (cand == nullptr)
        for (int64_t v = threadIdx.x; v < n; v += CT) {
            R.lock[v] = 0;
            store_pc(R.pc_old, R.pcb, v, load_pc(R.pc, R.pcb, v));
        }
    __syncthreads();
    const AbCount cnt = cta_rebalance(R, mode, n, cand, ncand, s_pw, s_snap, s_cum, s_keys, sh);
    const int64_t moves = cta_sum(cnt.moves, sh), deg = cta_sum(cnt.deg, sh);
    for (int q = threadIdx.x; q < k; q += CT) pw[q] = s_pw[q];
    if (threadIdx.x == 0) { step[S_STEP_MOVES] += moves; step[S_MVDEG] += deg; }
}

// the whole refinement loop of one level by one block of CT threads; rsm:
// cta_refine_smem(k) bytes of dynamic shared memory
__device__ void cta_refine_level(const CtaRefineArgs& R, unsigned char* rsm) {
    const int32_t k = R.k;
    const int64_t Lmax = R.Lmax, n = R.g.n;
    int32_t* s_pw = (int32_t*)rsm;               // k: current part weights (32 bits: rb_delta_begin)
    int32_t* s_snap = s_pw + 2 * k;              // k: weights at the start of a rebalance step
    int32_t* s_best = s_snap + 2 * k;            // k: weights of the kept state
    int64_t* s_cum = (int64_t*)rsm + 3 * k;      // k + 1: free capacity prefix (strong)
    uint8_t* s_over = (uint8_t*)(s_cum + k + 1); // k
    unsigned char* big = rsm + (((size_t)(4 * k + 1) * 8 + k + 15) & ~(size_t)15);
    int32_t* s_hist = (int32_t*)big;             // CW * k connectivity histograms, or
    uint64_t* s_keys = (uint64_t*)big;           // up to kCtaMaxN sort keys
    __shared__ int64_t sh[33];
    __shared__ uint64_t s_lk[CW];
    __shared__ int32_t s_lq[CW];
    __shared__ int64_t s_mx[CW];
    __shared__ ConnRowS s_rows[CT];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t* part = R.part;
    int32_t* part_next = R.part_next;
    uint8_t* lock = R.lock;
    uint8_t* lock_next = R.lock_next;
    for (int q = threadIdx.x; q < k; q += CT) s_pw[q] = (int32_t)R.pw[q];
    for (int64_t v = threadIdx.x; v < n; v += CT) lock[v] = 0;
    __syncthreads();
    int64_t best_cut = 0, best_mp = 0, prev_moves = -1, nmoves = 0;
    int stall = 0, rb_streak = 0, steps = 0, last_mode = 0;
    const int64_t U2 = R.nbucket[2], U1 = R.nbucket[1], U0 = (R.nbucket[0] + 3) / 4;
    for (int it = 0;; ++it) {
        const bool final_eval = it == R.max_iters;
        // ---- part-weight summary (as k_conn's prologue)
        int64_t mx = 0;
        uint64_t lk = 0; int32_t lq = -1;
        for (int q = threadIdx.x; q < k; q += CT) {
            const int64_t x = s_pw[q];
            s_over[q] = x > Lmax;
            mx = x > mx ? x : mx;
            if (x <= Lmax) argmax_q(lk, lq, ~(uint64_t)x, q);
        }
        for (int i = threadIdx.x; i < CW * k; i += CT) s_hist[i] = 0;
        if (threadIdx.x < S_NRESET) R.status[threadIdx.x] = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { const int64_t y = __shfl_xor_sync(0xffffffffu, mx, o); mx = y > mx ? y : mx; }
        warp_argmax_q(lk, lq);
        if (lane == 0) { s_mx[w] = mx; s_lk[w] = lk; s_lq[w] = lq; }
        __syncthreads();
        int64_t maxpw = 0; uint64_t lk2 = 0; int32_t light = -1;
        for (int i = 0; i < CW; ++i) { maxpw = s_mx[i] > maxpw ? s_mx[i] : maxpw; argmax_q(lk2, light, s_lk[i], s_lq[i]); }
        const int dmode = final_eval ? MODE_EVAL : (maxpw > Lmax ? MODE_RB : MODE_LP);
        // ---- connectivity pass
        ConnArgs CA;
        CA.g = R.g; CA.k = k; CA.Lmax = Lmax; CA.den = R.den; CA.force_eval = final_eval ? 1 : 0;
        CA.lock = lock; CA.pw = nullptr; CA.heavy = nullptr; CA.item_row = nullptr;
        CA.item_beg = nullptr; CA.item_end = nullptr; CA.row_items = nullptr; CA.nitems = 0;
        for (int b = 0; b < 3; ++b) { CA.bucket[b] = R.bucket[b]; CA.nbucket[b] = R.nbucket[b]; CA.clist[b] = nullptr; }
        CA.wfirst = nullptr;
        CA.nranges = 0;
        CA.dest = R.dest; CA.gain = R.gain; CA.status = R.status;
        CA.lock_next = nullptr; CA.prev = nullptr; CA.track_deg = -1; CA.host = nullptr; CA.nblocks = 0;
        CA.rb_all = R.tr_arrays ? 1 : 0;
        CA.pc = part; CA.pc_next = nullptr; CA.pdg = nullptr; CA.lp_dg = 1;
        CA.hhist = nullptr; CA.hsum = nullptr; CA.hdone = nullptr;
        int64_t acc = 0, cdeg = 0;
        int32_t* hist = s_hist + w * k;
        for (int64_t ub = 8 * w; ub < U2 + U1 + U0; ub += 8 * CW)
            conn_group<int32_t, true>(CA, ub, (int)(U2 + U1 + U0 - ub < 8 ? U2 + U1 + U0 - ub : 8), dmode, true, s_over, light, hist,
                                s_rows + 32 * w, acc, cdeg);
        acc = warp_sum(acc);
        const int64_t cur_cut = cta_sum(lane == 0 ? acc : 0, sh) / 2;   // also orders the pass
        const int64_t cur_mp = maxpw;
        // ---- best state and stop rules (every thread holds the same values)
        if (it == 0) {
            best_cut = cur_cut; best_mp = cur_mp;
            for (int64_t v = threadIdx.x; v < n; v += CT) R.best[v] = part[v];
            for (int q = threadIdx.x; q < k; q += CT) s_best[q] = s_pw[q];
        } else {
            const bool cb = cur_mp <= Lmax, bb = best_mp <= Lmax;
            bool better = false, signif = false;
            if (cb && !bb) { better = true; signif = true; }
            else if (cb && bb) { better = cur_cut < best_cut; signif = 1000 * cur_cut < 999 * best_cut; }
            else if (!cb && !bb) { better = cur_mp < best_mp || (cur_mp == best_mp && cur_cut < best_cut); signif = cur_mp < best_mp; }
            if (better) {
                best_cut = cur_cut; best_mp = cur_mp;
                for (int64_t v = threadIdx.x; v < n; v += CT) R.best[v] = part[v];
                for (int q = threadIdx.x; q < k; q += CT) s_best[q] = s_pw[q];
            }
            stall = signif ? 0 : stall + 1;
            const bool lp_idle = (last_mode == 0 && nmoves == 0 && prev_moves == 0);
            prev_moves = nmoves;
            bool rb_stuck = false;
            if (last_mode != 0 && nmoves == 0) {
                if (last_mode == 1) rb_streak = R.strong_after; else rb_stuck = true;
            }
            if (stall >= R.patience || lp_idle || rb_stuck) break;
        }
        if (final_eval) break;
        int mode;
        if (dmode == MODE_RB) { mode = (rb_streak >= R.strong_after) ? 2 : 1; ++rb_streak; }
        else { mode = 0; rb_streak = 0; }
        last_mode = mode;
        __syncthreads();
        if (mode == 0) {
            for (int64_t v = threadIdx.x; v < n; v += CT) { part_next[v] = part[v]; lock_next[v] = 0; }
            __syncthreads();
            ApplyArgs AA;
            AA.g = R.g; AA.k = k; AA.dest = R.dest; AA.gain = R.gain; AA.heavy = nullptr;
            AA.item_row = nullptr; AA.item_beg = nullptr; AA.item_end = nullptr; AA.row_items = nullptr; AA.nitems = 0;
            for (int b = 0; b < 3; ++b) AA.clist[b] = R.clist[b];
            AA.status = R.status; AA.lock_next = lock_next; AA.pw = nullptr;
            AA.pc = part; AA.pc_next = part_next;
            AA.step = nullptr; AA.hsum = nullptr; AA.hdone = nullptr; AA.pdg = nullptr;
            AbCount cnt;
            for (int64_t u = w; u < U2 + U1; u += CW) {
                const int64_t v = u < U2 ? R.bucket[2][u] : R.bucket[1][u - U2];
                if (R.dest[v] < 0) continue;
                if (u < U2) ab_warp<int32_t>(AA, v, s_pw, cnt);
                else ab_tile<kTile32, int32_t>(AA, v, s_pw, cnt);
            }
            for (int64_t i0 = 32 * w; i0 < R.nbucket[0]; i0 += 32 * CW) {
                const int64_t v = i0 + lane < R.nbucket[0] ? R.bucket[0][i0 + lane] : -1;
                ab_short<int32_t>(AA, v >= 0 && R.dest[v] >= 0 ? v : -1, s_pw, cnt);
            }
            nmoves = cta_sum(cnt.moves, sh);
            int32_t* tp = part; part = part_next; part_next = tp;
            uint8_t* tl = lock; lock = lock_next; lock_next = tl;
        } else {
            for (int64_t v = threadIdx.x; v < n; v += CT) lock[v] = 0;
            __syncthreads();
            RbCta RA;
            RA.vw = R.g.vw; RA.pc = part; RA.pcb = 4; RA.pc_old = nullptr; RA.rp = nullptr; RA.lock = lock; RA.dest = R.dest;
            RA.gain = R.gain; RA.pre = R.pre;
            RA.flag = R.flag; RA.gkeys = R.gkeys; RA.k = k; RA.Lmax = Lmax;
            nmoves = cta_sum(cta_rebalance(RA, mode, n, nullptr, 0, s_pw, s_snap, s_cum, s_keys, sh).moves, sh);
        }
        if (R.tr_arrays) {
            int32_t* t = R.tr_arrays + (int64_t)steps * 3 * n;
            for (int64_t v = threadIdx.x; v < n; v += CT) { t[v] = R.dest[v]; t[n + v] = R.gain[v]; t[2 * n + v] = part[v]; }
            if (threadIdx.x == 0) {
                int64_t* sc = R.tr_scalars + 4 * steps;
                sc[0] = mode; sc[1] = cur_cut; sc[2] = cur_mp; sc[3] = nmoves;
            }
        }
        ++steps;
        __syncthreads();
    }
    __syncthreads();
    // the kept state
    for (int64_t v = threadIdx.x; v < n; v += CT) R.part[v] = R.best[v];
    for (int q = threadIdx.x; q < k; q += CT) R.pw[q] = s_best[q];
    if (threadIdx.x == 0) R.out[0] = steps;
}

__global__ void __launch_bounds__(CT, 1) k_refine_cta(CtaRefineArgs R) {
    extern __shared__ __align__(16) unsigned char rsm[];
    cta_refine_level(R, rsm);
}

// ------------------------------------------------------------------ batched one-block levels
// A chain is the run of one graph's levels, coarsest first, that one block
// refines (at most kCtaMaxN vertices, no row longer than kHeavyDeg).  The
// persistent kernel k_refine_chains takes chains from a device work queue (an
// atomic ticket over the chains, ordered by cost, largest first) and, for
// each level of the chain, projects the coarser level's partition and runs
// the level's whole refinement loop, with no host round trip between
// levels or iterations.  Chains are independent, so no block ever waits for
// another.
struct ChainItem {
    CtaRefineArgs R;          // R.part receives the projected partition
    const int32_t* cmap;      // fine -> coarse map of this level (nullptr: coarsest level, no projection)
    const int32_t* pcoarse;   // refined partition of the next coarser level
};

__global__ void __launch_bounds__(CT, 1) k_refine_chains(const int32_t* __restrict__ chain_first,
                                                         const int32_t* __restrict__ chain_len, int32_t nchains,
                                                         const ChainItem* __restrict__ items, int32_t* ticket) {
    extern __shared__ __align__(16) unsigned char rsm[];
    __shared__ int32_t s_chain;
    for (;;) {
        if (threadIdx.x == 0) s_chain = atomicAdd(ticket, 1);
        __syncthreads();
        const int32_t ch = s_chain;
        __syncthreads();
        if (ch >= nchains) return;
        for (int32_t t = 0; t < chain_len[ch]; ++t) {
            const ChainItem& it = items[chain_first[ch] + t];
            if (it.cmap)
                for (int64_t v = threadIdx.x; v < it.R.g.n; v += CT) it.R.part[v] = it.pcoarse[it.cmap[v]];
            __syncthreads();
            cta_refine_level(it.R, rsm);
            __syncthreads();
        }
    }
}

static size_t cta_refine_smem(int32_t k) {
    const size_t head = (((size_t)(4 * k + 1) * 8 + k + 15) & ~(size_t)15);
    const size_t hist = sizeof(int32_t) * CW * (size_t)k, keys = sizeof(uint64_t) * kCtaMaxN;
    return head + (hist > keys ? hist : keys);
}

void refine_smem_caps() {
    GP_CUDA(cudaFuncSetAttribute(k_refine_cta, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cta_refine_smem(GP_MAX_K)));
    GP_CUDA(cudaFuncSetAttribute(k_rb_step_cta, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cta_refine_smem(GP_MAX_K)));
    GP_CUDA(cudaFuncSetAttribute(k_refine_chains, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cta_refine_smem(GP_MAX_K)));
}

static bool cta_refine_ok(const Level& L, const Params& P) {
    const int64_t lim = std::min<int64_t>(P.o.small_level_n, kCtaMaxN);
    return P.o.small_level_n > 0 && L.nheavy == 0 && L.g.n <= lim && P.k <= GP_MAX_K;
}

static int refine_level_cta(Ctx& c, const Level& L, const Params& P, RefineBufs& B, int level, const Tracer& tr) {
    const DGraph& g = L.g;
    const int64_t n = g.n;
    auto mk = c.tmp->save();
    CtaRefineArgs R;
    R.g = g; R.k = P.k; R.Lmax = P.Lmax; R.den = P.o.lp_filter_den; R.max_iters = P.o.refine_max_iters;
    R.patience = P.o.refine_patience; R.strong_after = P.o.strong_after;
    for (int b = 0; b < 3; ++b) { R.bucket[b] = L.bucket[b]; R.nbucket[b] = L.nbucket[b]; R.clist[b] = B.clist[b]; }
    R.part = B.part; R.part_next = B.part_next; R.lock = B.lock; R.lock_next = B.lock_next; R.best = B.best;
    R.pw = B.pw; R.dest = B.dest; R.gain = B.gain; R.status = B.status;
    R.pre = c.tmp_alloc<int64_t>(n);
    R.flag = c.tmp_alloc<int32_t>(n);
    R.gkeys = c.tmp_alloc<uint64_t>(n);
    R.tr_arrays = nullptr; R.tr_scalars = nullptr;
    if (tr.on()) {
        R.tr_arrays = c.tmp_alloc<int32_t>((int64_t)P.o.refine_max_iters * 3 * n);
        R.tr_scalars = c.tmp_alloc<int64_t>((int64_t)P.o.refine_max_iters * 4);
    }
    R.out = c.tmp_alloc<int64_t>(1);
    k_refine_cta<<<1, CT, cta_refine_smem(P.k), c.s>>>(R);
    GP_LAUNCHED(c);
    const int steps = (int)read_i64(c, R.out);
    // each step: one connectivity pass plus its move step; one closing pass
    c.bytes += (int64_t)(steps + 1) * (L.scan_bytes() + 13 * n) + (int64_t)steps * (9 * n + 16 * n);
    if (tr.on() && steps > 0) {
        std::vector<int32_t> arr((size_t)steps * 3 * n);
        std::vector<int64_t> sc((size_t)steps * 4);
        GP_CUDA(cudaMemcpyAsync(arr.data(), R.tr_arrays, sizeof(int32_t) * arr.size(), cudaMemcpyDeviceToHost, c.s));
        GP_CUDA(cudaMemcpyAsync(sc.data(), R.tr_scalars, sizeof(int64_t) * sc.size(), cudaMemcpyDeviceToHost, c.s));
        c.sync();
        for (int it = 0; it < steps; ++it) {
            gp_trace_event ev;
            memset(&ev, 0, sizeof ev);
            ev.kind = GP_TR_REFINE_ITER; ev.level = level; ev.iter = it; ev.mode = (int32_t)sc[4 * it];
            ev.n = n; ev.m = g.m; ev.cut = sc[4 * it + 1]; ev.maxpw = sc[4 * it + 2]; ev.count = sc[4 * it + 3];
            int32_t* base = arr.data() + (size_t)it * 3 * n;
            ev.a0 = base; ev.a1 = base + n; ev.a2 = base + 2 * n;
            tr.emit(ev);
        }
    }
    c.tmp->restore(mk);
    return steps;
}

// One block refines a level as long as its passes are latency, not entries: with
// levels of any number of entries the longest chain of a batch of 128 graphs (1,000
// to 200,000 vertices, 16 workers) ran 36.6 ms and the batch 116.5 ms; up to
// 262,144 / 131,072 / 65,536 / 32,768 entries 30.9 / 22.0 / 9.1 / 4.5 and 114.2 /
// 110.7 / 107.6 / 109.5 (the workers' launches for the larger levels grow).
constexpr int64_t kChainM = 65536;
static bool chain_level_ok(const Level& L, const Params& P) {
    return L.nheavy == 0 && L.g.n <= kCtaMaxN && L.g.m <= kChainM && P.k <= GP_MAX_K;
}

struct ChainBatch {
    std::mutex mu;
    std::vector<ChainItem> items;
    struct Rec { VState* S; int32_t first, len; int64_t cost; };
    std::vector<Rec> chains;
    int32_t kmax = 2;
};

ChainBatch* chain_batch_new() { return new ChainBatch(); }
void chain_batch_delete(ChainBatch* cb) { delete cb; }

int chain_add(Ctx& c, ChainBatch* cb, VState& S) {
    const Params& P = S.P;
    if (P.k <= 1 || S.refined_to != S.L + 1) return 0;
    int s = S.L + 1;
    while (s > 0 && chain_level_ok(S.lv[s - 1], P)) --s;
    const int len = S.L + 1 - s;
    if (len == 0) return 0;
    int64_t nmax = 1, cost = 0;
    for (int l = s; l <= S.L; ++l) { nmax = std::max(nmax, S.lv[l].g.n); cost += S.lv[l].g.n + S.lv[l].g.m; }
    RefineBufs& B = S.B;
    int64_t* pre = c.keep_alloc<int64_t>(nmax);
    int32_t* flag = c.keep_alloc<int32_t>(nmax);
    uint64_t* gkeys = c.keep_alloc<uint64_t>(nmax);
    std::vector<ChainItem> mine((size_t)len);
    for (int t = 0; t < len; ++t) {
        const int l = S.L - t;
        const Level& L = S.lv[l];
        ChainItem& it = mine[t];
        CtaRefineArgs& R = it.R;
        R.g = L.g; R.k = P.k; R.Lmax = P.Lmax; R.den = P.o.lp_filter_den; R.max_iters = P.o.refine_max_iters;
        R.patience = P.o.refine_patience; R.strong_after = P.o.strong_after;
        for (int b = 0; b < 3; ++b) { R.bucket[b] = L.bucket[b]; R.nbucket[b] = L.nbucket[b]; R.clist[b] = B.clist[b]; }
        // the partition alternates between the two part buffers level by level
        int32_t* cur = (t & 1) ? B.part_next : B.part;
        int32_t* other = (t & 1) ? B.part : B.part_next;
        R.part = cur; R.part_next = other; R.lock = B.lock; R.lock_next = B.lock_next; R.best = B.best;
        R.pw = B.pw; R.dest = B.dest; R.gain = B.gain; R.status = B.status;
        R.pre = pre; R.flag = flag; R.gkeys = gkeys;
        R.tr_arrays = nullptr; R.tr_scalars = nullptr;
        R.out = nullptr;   // set by chain_run
        it.cmap = t == 0 ? nullptr : L.cmap;
        it.pcoarse = other;
    }
    std::lock_guard<std::mutex> lk(cb->mu);
    cb->chains.push_back({&S, (int32_t)cb->items.size(), (int32_t)len, cost});
    cb->items.insert(cb->items.end(), mine.begin(), mine.end());
    cb->kmax = std::max(cb->kmax, P.k);
    return len;
}

void chain_run(Ctx& c, ChainBatch* cb) {
    const int32_t nch = (int32_t)cb->chains.size();
    if (nch == 0) return;
    // largest chains first
    std::vector<int32_t> order((size_t)nch);
    for (int32_t i = 0; i < nch; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        return cb->chains[a].cost > cb->chains[b].cost; });
    std::vector<int32_t> hfirst((size_t)nch), hlen((size_t)nch);
    for (int32_t i = 0; i < nch; ++i) { hfirst[i] = cb->chains[order[i]].first; hlen[i] = cb->chains[order[i]].len; }
    auto mk = c.tmp->save();
    const int64_t ni = (int64_t)cb->items.size();
    ChainItem* d_items = (ChainItem*)c.tmp->alloc(sizeof(ChainItem) * (size_t)ni);
    int32_t* d_first = c.tmp_alloc<int32_t>(nch);
    int32_t* d_len = c.tmp_alloc<int32_t>(nch);
    int32_t* d_ticket = c.tmp_alloc<int32_t>(1);
    int64_t* d_steps = c.tmp_alloc<int64_t>(ni);
    for (int64_t i = 0; i < ni; ++i) cb->items[i].R.out = d_steps + i;
    GP_CUDA(cudaMemcpyAsync(d_items, cb->items.data(), sizeof(ChainItem) * (size_t)ni, cudaMemcpyHostToDevice, c.s));
    GP_CUDA(cudaMemcpyAsync(d_first, hfirst.data(), sizeof(int32_t) * nch, cudaMemcpyHostToDevice, c.s));
    GP_CUDA(cudaMemcpyAsync(d_len, hlen.data(), sizeof(int32_t) * nch, cudaMemcpyHostToDevice, c.s));
    memset_async(c, d_ticket, 0, sizeof(int32_t));
    const size_t smem = cta_refine_smem(cb->kmax);
    int per_sm = 1;
    GP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine_chains, CT, smem));
    const int grid = (int)std::min<int64_t>(nch, (int64_t)std::max(per_sm, 1) * c.sm_count);
    k_refine_chains<<<grid, CT, smem, c.s>>>(d_first, d_len, nch, d_items, d_ticket);
    GP_LAUNCHED(c);
    // steps of every level; the partition ends in the buffer of the last level
    std::vector<int64_t> steps((size_t)ni);
    GP_CUDA(cudaMemcpyAsync(steps.data(), d_steps, sizeof(int64_t) * (size_t)ni, cudaMemcpyDeviceToHost, c.s));
    c.sync();
    c.tmp->restore(mk);
    for (auto& rec : cb->chains) {
        VState& S = *rec.S;
        for (int t = 0; t < rec.len; ++t) {
            const Level& L = S.lv[S.L - t];
            const int64_t n = L.g.n;
            const int64_t st = steps[rec.first + t];
            S.iters += (int)st;
            S.bytes += (st + 1) * (L.scan_bytes() + 13 * n) + st * (9 * n + 16 * n) + (t ? 12 * n : 0);
        }
        if ((rec.len - 1) & 1) std::swap(S.B.part, S.B.part_next);
        S.refined_to = S.L + 1 - rec.len;
    }
}

// ------------------------------------------------------------------ level controller
static int bits_for(int64_t x) {
    int b = 1;
    while ((1ll << b) < x) ++b;
    return b;
}

// the partition in 1 or 2 bytes per vertex, as a level's refinement holds it
// (B.part is int32 between levels), and back
__global__ void k_compact_part(int64_t n, const int32_t* __restrict__ part, void* pc, int pcb) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        store_pc(pc, pcb, v, part[v]);
}
__global__ void k_expand_part(int64_t n, const void* __restrict__ pc, int pcb, int32_t* __restrict__ part) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        part[v] = load_pc(pc, pcb, v);
}

static void trace_iter(Ctx& c, const RefineBufs& B, const int64_t* step_d, int64_t n, int64_t m, int level, int it, int mode,
                       int64_t cut_before, int64_t mp_before, const Tracer& tr) {
    std::vector<int32_t> d(n), gn(n), p(n);
    k_expand_part<<<grid_for(n, 256), 256, 0, c.s>>>(n, B.pc, B.pcb, B.part);
    GP_LAUNCHED(c);
    GP_CUDA(cudaMemcpyAsync(d.data(), B.dest, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c.s));
    GP_CUDA(cudaMemcpyAsync(gn.data(), B.gain, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c.s));
    GP_CUDA(cudaMemcpyAsync(p.data(), B.part, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c.s));
    GP_CUDA(cudaMemcpyAsync(c.h_pinned, step_d + S_STEP_MOVES, sizeof(int64_t), cudaMemcpyDeviceToHost, c.s));
    c.sync();
    gp_trace_event ev;
    memset(&ev, 0, sizeof ev);
    ev.kind = GP_TR_REFINE_ITER; ev.level = level; ev.iter = it; ev.mode = mode;
    ev.n = n; ev.m = m; ev.cut = cut_before; ev.maxpw = mp_before; ev.count = c.h_pinned[0];
    ev.a0 = d.data(); ev.a1 = gn.data(); ev.a2 = p.data();
    tr.emit(ev);
}

constexpr int64_t kConnWarpCost = 8 * (8 + 28);
// light blocks of a pass: one range per warp up to two resident waves, then
// ranges of kConnRangeCost that a block's warps share, and more blocks only where
// theirs would cost more than kConnBlockCost.  With one range per warp on every
// level R-MAT 20 spent 53% of its warps' time at the end of their blocks, behind
// the warp with a row of thousands of entries: its 73 passes took 11.1 ms in all
// against 8.5, its move steps 1.85 against 1.24 (passes, the last of each level
// skipped: 6.75 ms with 20,000 per block, 7.33 with 10,000, 6.91 with 42,000).  R-MAT 24's take 114 ms with 700,000 per block, 101 with 340,000,
// 96 with 170,000, 94 with 85,000.
constexpr int64_t kConnWave = 10;            // blocks per SM, 5 resident
constexpr int64_t kConnRangeCost = 768;
constexpr int64_t kConnBlockCost = 98304;
// bucket-0 rows from which they take their own launch: below, a second launch
// (about 3 us a pass) costs more than the registers
constexpr int64_t kConnSplit = 32768;
// or entries.  Refinement with 1 M / 2 M / 4 M entries: R-MAT 16 4.3 / 4.0 / 4.0 ms, R-MAT 17
// 6.8 / 6.6 / 6.4, Erdos-Renyi of 2.6 M entries 8.9 / 8.9 / 9.1, R-MAT 20 15.7 / 15.7 / 15.6
constexpr int64_t kConnSplitM = 1 << 21;
// moved rows' share of the entries up to which the cut's change is tracked: before
// a pass that looks for moves in the overweight parts (an eighth to a half of the
// rows) and before one that may be the level's last (R-MAT 24, passes and k_track:
// 1/16 and 1/4 117 ms, 1/8 and 1/3 115, 1/4 and 1/2 116; the whole refinement of R-MAT 22
// 40.4 / 40.4 / 41.0, of a 200^3 grid 43.1 with each)
constexpr int64_t kTrackShare = 8;
constexpr int64_t kTrackLast = 3;
// entries from which the cut's change is tracked.  Refinement with 2 M / 4 M / 8 M / never:
// Erdos-Renyi of 2.5 M entries 14.8 / 14.3 / 14.2 / 14.3 ms, 100^3 grid (5.9 M) 21.7 / 21.7 /
// 21.3 / 21.4, random geometric of 8 M 10.5 / 10.5 / 10.7 / 10.7, 200^3 grid (48 M) 43.2 /
// 43.1 / 43.2 / 45.4, R-MAT 22 (128 M) 40.4 / 40.4 / 40.5 / 42.5
constexpr int64_t kTrackMin = 1 << 22;
// How a level's connectivity passes are cut: bucket-0 rows in their own launches
// when they are many, and on levels whose longer rows are the work (k_conn without
// them runs at 48 registers); the rest in contiguous ranges of light units.  A range
// costs as much as a group of 8 units of short rows, so that a warp's lanes have
// rows to work on; on levels too small for 16 such ranges per SM latency counts and
// units are spread thinner
struct ConnPlan {
    bool split, long_rows;
    int64_t nunits, cost, wave, nranges;
};
static ConnPlan conn_plan(const Ctx& c, const Level& L) {
    ConnPlan p;
    p.split = L.nbucket[0] >= kConnSplit || L.g.m >= kConnSplitM;
    p.long_rows = !p.split || L.nitems + L.nbucket[1] + L.nbucket[2] > 0;
    p.nunits = p.split ? L.nbucket[2] + L.nbucket[1] : L.nunits;
    p.cost = L.g.m + 32 * (L.nbucket[2] + L.nbucket[1]) + (p.split ? 0 : 2 * L.nbucket[0]);
    p.wave = (int64_t)c.sm_count * kConnWave;
    const int64_t most = (int64_t)c.sm_count * c.ctas_per_sm * RW * 4;
    const int64_t want = std::max<int64_t>(std::max(std::min(p.cost / kConnWarpCost, p.wave * RW), p.cost / kConnRangeCost),
                                           (int64_t)c.sm_count * 16);
    p.nranges = std::max<int64_t>(std::min(std::min(p.nunits, want), most), 1);
    return p;
}
int64_t conn_ranges(const Ctx& c, const Level& L) { return conn_plan(c, L).nranges; }

// range t of the nw of a connectivity pass holds the units [first unit with cost
// prefix >= T * t / nw, the same for t + 1), T the total cost: contiguous ranges
// of equal cost, the same for every pass of a level
__global__ void k_warp_bounds(const int64_t* __restrict__ cost, int64_t nunits, int64_t nw,
                              int64_t* __restrict__ out) {
    const int64_t T = cost[nunits];
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t <= nw; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t target = (T * t) / nw;
        int64_t lo = 0, hi = nunits;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (cost[mid] < target) lo = mid + 1; else hi = mid;
        }
        out[t] = lo;
    }
}

int refine_level(Ctx& c, const Level& L, const Params& P, RefineBufs& B, int level, const Tracer& tr) {
    if (cta_refine_ok(L, P)) return refine_level_cta(c, L, P, B, level, tr);
    const DGraph& g = L.g;
    const int64_t n = g.n;
    const int32_t k = P.k;
    const int64_t Lmax = P.Lmax;
    memset_async(c, B.lock, 0, n);
    // the level's partition is held in uint8 (k <= 256) or uint16: a quarter or
    // half of the bytes per gather, of the array that has to stay in L2, and of
    // every copy of it
    B.pcb = k <= 256 ? 1 : 2;
    k_compact_part<<<grid_for(n, 256), 256, 0, c.s>>>(n, B.part, B.pc, B.pcb);
    GP_LAUNCHED(c);
    c.bytes += 4 * n + B.pcb * n;
    const int kpad = (k + 15) & ~15;
    const size_t conn_smem = kpad + sizeof(int32_t) * RW * k;
    // at most 1024 + 32 * GP_MAX_K bytes: below the 48 KB default, no attribute needed
    const ConnPlan cut = conn_plan(c, L);
    const bool split = cut.split, long_rows = cut.long_rows;
    const int64_t nunits = cut.nunits, cost = cut.cost, wave = cut.wave, nranges = cut.nranges;
    if (nranges >= B.wfirst_cap) throw GpError(GP_EINTERNAL, "connectivity ranges exceed their array");
    const int light_blocks = (int)std::min<int64_t>(grid_for(nranges, RW, c.sm_count * c.ctas_per_sm),
                                                    std::max(wave, cost / kConnBlockCost));
    const int grid = (int)L.nitems + light_blocks;
    const int short_grid = grid_for(L.nbucket[0], RT, c.sm_count * std::min(c.ctas_per_sm, 8));
    const int lp_grid = grid_for(L.nbucket[0], 4 * RT, c.sm_count * 8);
    if (long_rows) {
        k_warp_bounds<<<grid_for(nranges + 1, 256), 256, 0, c.s>>>(L.unit_cost, nunits, nranges, B.wfirst);
        GP_LAUNCHED(c);
    }
    int64_t best_cut = 0, best_mp = 0;
    int stall = 0, rb_streak = 0, steps = 0, last_mode = 0;
    int64_t prev_moves = -1;
    const int nb_k = bits_for(k);
    int64_t* step_d = nullptr;   // status block of the last step
    int64_t cross2 = 0;          // directed cross weight of the current state
    // the cut's change over a step is taken from the moved rows when they hold
    // few of the entries, on levels whose passes cost more than k_track's launches;
    // an input that is not symmetric has no mirror entries
    const bool track = P.symmetric && g.m >= kTrackMin;
    int64_t track_deg = -1;         // of the step before this pass
    ConnStop stop;
    memset(&stop, 0, sizeof stop);
    int32_t track_range = 4 * RT;   // about 8 blocks per SM
    while (track_range < kTrackRange && n > (int64_t)track_range * c.sm_count * 8) track_range *= 2;
    const bool move_head = B.mp && P.gnn && gnn_has_move_head(P.gnn);
    // with pdg, proposals and gains of a label-propagation pass are stored apart
    // only for the move head and the trace
    const int lp_dg = (!B.pdg || move_head || tr.on()) ? 1 : 0;
    for (int it = 0;; ++it) {
        const bool final_eval = (it == P.o.refine_max_iters);
        // this iteration's status block; the half of the ring that is not in use
        // is cleared ahead
        constexpr int half = kStatusRing / 2;
        int64_t* status = B.status + (int64_t)(it % kStatusRing) * S_NSLOTS;
        if (it == 0) memset_async(c, B.status, 0, sizeof(int64_t) * S_NSLOTS * kStatusRing);
        else if (it % kStatusRing == half / 2) memset_async(c, B.status + half * S_NSLOTS, 0, sizeof(int64_t) * S_NSLOTS * half);
        else if (it % kStatusRing == half + half / 2) memset_async(c, B.status, 0, sizeof(int64_t) * S_NSLOTS * half);
        if (c.profile) GP_CUDA(cudaEventRecord(c.ev_a, c.s));
        ConnArgs CA;
        CA.g = g; CA.k = k; CA.Lmax = Lmax; CA.den = P.o.lp_filter_den; CA.force_eval = final_eval ? 1 : 0;
        CA.lock = B.lock; CA.pw = B.pw; CA.heavy = L.heavy;
        CA.item_row = L.item_row; CA.item_beg = L.item_beg; CA.item_end = L.item_end; CA.row_items = L.row_items;
        CA.nitems = L.nitems; CA.hhist = B.hhist; CA.hsum = B.hsum; CA.hdone = B.hdone;
        for (int b = 0; b < 3; ++b) { CA.bucket[b] = L.bucket[b]; CA.nbucket[b] = L.nbucket[b]; CA.clist[b] = B.clist[b]; }
        CA.wfirst = B.wfirst;
        CA.nranges = nranges;
        CA.dest = B.dest; CA.gain = B.gain; CA.status = status;
        CA.prev = step_d; CA.track_deg = track_deg; CA.stop = stop; CA.rb_all = tr.on() ? 1 : 0; CA.host = c.h_pinned; CA.nblocks = (long_rows ? grid : 0) + (split && L.nbucket[0] > 0 ? short_grid : 0);
        CA.pc = B.pc; CA.pc_next = B.pc_next; CA.lock_next = B.lock_next;   // the LP step's starting copy
        CA.pdg = B.pdg; CA.lp_dg = lp_dg;
        if (long_rows) {
            auto kc = B.pcb == 1 ? (split ? k_conn<uint8_t, false> : k_conn<uint8_t, true>)
                                 : (split ? k_conn<uint16_t, false> : k_conn<uint16_t, true>);
            kc<<<grid, RT, conn_smem, c.s>>>(CA);
            GP_LAUNCHED(c);
        }
        if (split && L.nbucket[0] > 0) {
            auto ks = B.pcb == 1 ? k_conn_short<uint8_t> : k_conn_short<uint16_t>;
            ks<<<short_grid, RT, kpad, c.s>>>(CA);
            GP_LAUNCHED(c);
        }
        if (c.profile) GP_CUDA(cudaEventRecord(c.ev_b, c.s));
        // rowptr, colidx, weights, gathered part[u] (pcb bytes); part[v], lock[v] read; proposal and gain written
        c.sync();   // the pass wrote its status block to c.h_pinned
        // a rebalancing pass that sweeps the rows of overweight parts only: their share
        // is not known here, the lists and parts of all rows are counted; a pass that
        // ends the level reads nothing
        const bool swept = c.h_pinned[H_FULL] != 0;
        const int64_t conn_bytes = swept ? L.scan_bytes() - (4 - B.pcb) * g.m + B.pcb * n + n + 8 * n
                                         : (c.h_pinned[S_MODE] == MODE_EVAL ? 0 : (4 + B.pcb) * n);
        c.bytes += conn_bytes;
        if (c.profile) {
            float t = 0;
            GP_CUDA(cudaEventElapsedTime(&t, c.ev_a, c.ev_b));
            c.ms_conn += t;
            c.conn_launches += 1;
            c.conn_bytes += conn_bytes;
        }
        cross2 = c.h_pinned[H_FULL] ? c.h_pinned[S_CROSS] : cross2 + c.h_pinned[H_DELTA];
        const int64_t cur_cut = cross2 / 2;
        const int64_t cur_mp = c.h_pinned[S_MAXPW];
        const int dev_mode = (int)c.h_pinned[S_MODE];
        const int64_t nlist = c.h_pinned[S_NL0] + c.h_pinned[S_NL1] + c.h_pinned[S_NL2];
        const int64_t cdeg = c.h_pinned[S_CDEG];
        if (it == 0) {
            best_cut = cur_cut; best_mp = cur_mp;
            GP_CUDA(cudaMemcpyAsync(B.best, B.pc, (size_t)B.pcb * n, cudaMemcpyDeviceToDevice, c.s));
            GP_CUDA(cudaMemcpyAsync(B.best_pw, B.pw, sizeof(int64_t) * k, cudaMemcpyDeviceToDevice, c.s));
        } else {
            const int64_t nmoves = c.h_pinned[H_MOVES];
            bool signif;
            const bool better = state_better(cur_cut, cur_mp, best_cut, best_mp, Lmax, signif);
            if (better) {
                best_cut = cur_cut; best_mp = cur_mp;
                GP_CUDA(cudaMemcpyAsync(B.best, B.pc, (size_t)B.pcb * n, cudaMemcpyDeviceToDevice, c.s));
                GP_CUDA(cudaMemcpyAsync(B.best_pw, B.pw, sizeof(int64_t) * k, cudaMemcpyDeviceToDevice, c.s));
            }
            stall = signif ? 0 : stall + 1;
            const bool lp_idle = (last_mode == 0 && nmoves == 0 && prev_moves == 0);
            prev_moves = nmoves;
            // a rebalance step that moved nothing: weak escalates to strong, strong ends the level
            bool rb_stuck = false;
            if (last_mode != 0 && nmoves == 0) {
                if (last_mode == 1) rb_streak = P.o.strong_after; else rb_stuck = true;
            }
            if (stall >= P.o.refine_patience || lp_idle || rb_stuck) break;
        }
        if (final_eval) break;
        if (dev_mode == MODE_EVAL) throw GpError(GP_EINTERNAL, "refinement pass ended a level that goes on");
        int mode;
        if (dev_mode == MODE_RB) { mode = (rb_streak >= P.o.strong_after) ? 2 : 1; ++rb_streak; }
        else { mode = 0; rb_streak = 0; }
        last_mode = mode;
        step_d = status;   // moves of this step, read at the next sync
        if (mode == 0) {
            // pc_next / lock_next were filled by the connectivity pass
            ApplyArgs AA;
            AA.g = g; AA.k = k; AA.dest = B.dest; AA.gain = B.gain; AA.heavy = L.heavy;
            AA.item_row = L.item_row; AA.item_beg = L.item_beg; AA.item_end = L.item_end; AA.row_items = L.row_items;
            AA.nitems = L.nitems; AA.hsum = B.hsum; AA.hdone = B.hdone;
            for (int b = 0; b < 3; ++b) AA.clist[b] = B.clist[b];
            AA.status = status; AA.lock_next = B.lock_next; AA.pw = B.pw;
            AA.step = step_d;
            AA.pc = B.pc; AA.pc_next = B.pc_next; AA.pdg = B.pdg;
            if (move_head) {
                // learned order of the afterburner: (move priority, id) instead of (gain, id)
                gnn_move_priorities(c, P.gnn, g, level, B.dest, B.gain, B.mp);
                AA.gain = B.mp;
                AA.pdg = nullptr;   // the packed words hold the gains
                if (tr.on()) {
                    std::vector<int32_t> hm((size_t)n);
                    GP_CUDA(cudaMemcpyAsync(hm.data(), B.mp, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c.s));
                    c.sync();
                    gp_trace_event ev;
                    memset(&ev, 0, sizeof ev);
                    ev.kind = GP_TR_MOVE_PRIO; ev.level = level; ev.iter = it; ev.n = n; ev.m = g.m;
                    ev.a0 = hm.data();
                    tr.emit(ev);
                }
            }
            const size_t ksm = sizeof(int32_t) * k;
            if (long_rows) {
                (B.pcb == 1 ? k_lp_apply<uint8_t> : k_lp_apply<uint16_t>)<<<grid, RT, ksm, c.s>>>(AA, split ? 1 : 0);
                GP_LAUNCHED(c);
            }
            if (split && L.nbucket[0] > 0) {
                (B.pcb == 1 ? k_lp_short<uint8_t> : k_lp_short<uint16_t>)<<<lp_grid, RT, ksm, c.s>>>(AA);
                GP_LAUNCHED(c);
            }
            // copy pass + afterburner: candidate rows with gathered part (pcb bytes), dest and gain per entry
            c.bytes += (9 + B.pcb) * n + 16 * nlist + cdeg * (4 + (g.ew ? 4 : 0) + 8 + B.pcb);
            std::swap(B.lock, B.lock_next);
            std::swap(B.pc, B.pc_next);
            // label propagation leaves the state before the step in pc_next (swapped)
        } else if (n <= kCtaMaxN && cdeg <= kRbCta) {
            // the whole step in one thread block
            auto mk = c.tmp->save();
            RbCta RA;
            RA.vw = g.vw; RA.pc = B.pc; RA.pcb = B.pcb; RA.pc_old = B.pc_next; RA.rp = g.rp; RA.lock = B.lock; RA.dest = B.dest;
            RA.gain = B.gain;
            RA.pre = c.tmp_alloc<int64_t>(n); RA.flag = c.tmp_alloc<int32_t>(n);
            RA.gkeys = c.tmp_alloc<uint64_t>(n); RA.k = k; RA.Lmax = Lmax;
            k_rb_step_cta<<<1, CT, cta_refine_smem(k), c.s>>>(RA, mode, n, nullptr, 0, B.pw, step_d);
            GP_LAUNCHED(c);
            c.bytes += 4 * n + 12 * n + 80 * n;
            c.tmp->restore(mk);
        } else {
            // candidates in vertex order; stable sort -> (source, bucket, id)
            const int64_t ncand = cdeg;
            auto mk = c.tmp->save();
            const int per = n >= kRbWide ? RB_PER : 1;
            const int64_t ntile = (n + (int64_t)per * RT - 1) / ((int64_t)per * RT);
            int32_t* tcnt = c.tmp_alloc<int32_t>(ntile);
            auto collect = [&](auto* pc, auto* pc_old, auto kcount, auto kcollect) {
                kcount<<<(unsigned)ntile, RT, kpad, c.s>>>(n, pc, B.pw, Lmax, k, tcnt);
                GP_LAUNCHED(c);
                kcollect<<<(unsigned)ntile, RT, kpad, c.s>>>(n, pc, B.pw, Lmax, k, tcnt, ncand, B.gain, pc_old, B.lock,
                                                             B.ckeys, B.cvals);
                GP_LAUNCHED(c);
            };
            if (B.pcb == 1 && per > 1)
                collect((uint8_t*)B.pc, (uint8_t*)B.pc_next, k_rb_count<uint8_t, RB_PER>, k_rb_collect<uint8_t, RB_PER>);
            else if (B.pcb == 1)
                collect((uint8_t*)B.pc, (uint8_t*)B.pc_next, k_rb_count<uint8_t, 1>, k_rb_collect<uint8_t, 1>);
            else if (per > 1)
                collect((uint16_t*)B.pc, (uint16_t*)B.pc_next, k_rb_count<uint16_t, RB_PER>, k_rb_collect<uint16_t, RB_PER>);
            else
                collect((uint16_t*)B.pc, (uint16_t*)B.pc_next, k_rb_count<uint16_t, 1>, k_rb_collect<uint16_t, 1>);
            c.bytes += 9 * n;
            if (ncand > 0 && ncand <= kRbCta) {
                // few candidates: sort, select and apply in one thread block
                RbCta RA;
                RA.vw = g.vw; RA.pc = B.pc; RA.pcb = B.pcb; RA.pc_old = B.pc_next; RA.rp = g.rp; RA.lock = B.lock; RA.dest = B.dest;
                RA.gain = B.gain;
                RA.pre = c.tmp_alloc<int64_t>(ncand); RA.flag = c.tmp_alloc<int32_t>(ncand);
                RA.gkeys = c.tmp_alloc<uint64_t>(ncand); RA.k = k; RA.Lmax = Lmax;
                k_rb_step_cta<<<1, CT, cta_refine_smem(k), c.s>>>(RA, mode, n, B.cvals, ncand, B.pw, step_d);
                GP_LAUNCHED(c);
                c.bytes += 80 * ncand;
            } else if (ncand > 0) {
                const int bits = RB_SHIFT + nb_k;
                radix_sort_pairs(c, B.ckeys, B.cvals, B.ckeys2, B.cvals2, ncand, bits);
                int64_t* pre = c.tmp_alloc<int64_t>(ncand + 1);
                scan_list_weights(c, B.cvals, g.vw, pre, ncand, nullptr, pre + ncand);
                RbPlan plan;
                int64_t* pl = c.tmp_alloc<int64_t>(6 * (int64_t)k + 2);
                plan.seg = pl; plan.acc = pl + k; plan.off = pl + 2 * k; plan.woff = pl + 3 * k; plan.snap = pl + 4 * k;
                plan.cum = pl + 5 * k; plan.n2 = pl + 6 * k + 1;
                k_rb_plan<<<1, GP_MAX_K, 0, c.s>>>(ncand, B.ckeys, pre, B.pw, Lmax, k, plan);
                GP_LAUNCHED(c);
                if (mode == 1) {
                    k_rb_rekey<<<grid_for(ncand, 256), 256, 0, c.s>>>(ncand, B.ckeys, B.cvals, plan, B.dest, B.ckeys2,
                                                                      B.cvals2);
                    GP_LAUNCHED(c);
                    radix_sort_pairs(c, B.ckeys2, B.cvals2, B.ckeys, B.cvals, ncand, bits, plan.n2);
                    scan_list_weights(c, B.cvals2, g.vw, pre, ncand, plan.n2, nullptr);
                    int64_t* segf = c.tmp_alloc<int64_t>(k + 1);
                    k_seg_first<<<grid_for(k + 1, 8), 256, 0, c.s>>>(plan.n2, B.ckeys2, k, segf);
                    GP_LAUNCHED(c);
                    k_rb_weak_apply<<<grid_for(ncand, 256, c.sm_count * 8), 256, sizeof(int32_t) * k, c.s>>>(
                        plan.n2, B.ckeys2, segf, B.cvals2, pre, g.vw, plan.snap, Lmax, k, B.pc, B.pcb, B.lock, B.pw,
                        g.rp, step_d);
                    GP_LAUNCHED(c);
                } else {
                    k_rb_strong_apply<<<grid_for(ncand, 256, c.sm_count * 8), 256, sizeof(int32_t) * k, c.s>>>(
                        ncand, B.ckeys, B.cvals, pre, plan, g.vw, k, B.pc, B.pcb, B.lock, B.pw, g.rp, step_d);
                    GP_LAUNCHED(c);
                }
                c.bytes += 80 * ncand;
            }
            c.tmp->restore(mk);
        }
        if (track) {
            // the next pass is the level's last when it does not improve on the best
            // state (or in any case): all it would compute is the cut
            stop.may = stall + 1 >= P.o.refine_patience || it + 1 == P.o.refine_max_iters ? 1 : 0;
            stop.cross2 = cross2; stop.best_cut = best_cut; stop.best_mp = best_mp;
            stop.patience = stall + 1 >= P.o.refine_patience ? 1 : 0;
            stop.idle = mode == 2 || (mode == 0 && prev_moves == 0) ? 1 : 0;
            track_deg = stop.may ? g.m / kTrackLast : g.m / kTrackShare;
            TrackArgs T;
            T.g = g; T.k = k; T.Lmax = Lmax; T.pw = B.pw; T.pc = B.pc; T.pc_old = B.pc_next; T.step = step_d;
            T.track_deg = track_deg; T.heavy = L.heavy; T.item_row = L.item_row;
            T.item_beg = L.item_beg; T.item_end = L.item_end; T.nitems = L.nitems;
            T.range = track_range;
            T.always = stop.may;
            for (int b = 0; b < 3; ++b) { T.bucket[b] = L.bucket[b]; T.nbucket[b] = L.nbucket[b]; }
            T.wfirst = B.wfirst;
            T.nranges = long_rows && L.nbucket[1] + L.nbucket[2] > 0 ? nranges : 0;
            T.range_blocks = T.nranges > 0 ? light_blocks : 0;
            const int tg = (int)(L.nitems + T.range_blocks + (n + track_range - 1) / track_range);
            (B.pcb == 1 ? k_track<uint8_t> : k_track<uint16_t>)<<<tg, RT, 0, c.s>>>(T);
            GP_LAUNCHED(c);
        }
        ++steps;
        if (tr.on()) trace_iter(c, B, step_d, n, g.m, level, it, mode, cur_cut, cur_mp, tr);
    }
    k_expand_part<<<grid_for(n, 256), 256, 0, c.s>>>(n, B.best, B.pcb, B.part);
    GP_LAUNCHED(c);
    c.bytes += 4 * n + B.pcb * n;
    GP_CUDA(cudaMemcpyAsync(B.pw, B.best_pw, sizeof(int64_t) * k, cudaMemcpyDeviceToDevice, c.s));
    return steps;
}

}  // namespace gp
