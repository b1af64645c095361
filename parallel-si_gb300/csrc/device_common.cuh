// device_common.cuh -- shared constants and helpers of the sm_103a kernels.
#ifndef PSI_DEVICE_COMMON_CUH
#define PSI_DEVICE_COMMON_CUH

#include <climits>
#include <cstdint>
#include <cooperative_groups.h>

#include "kernels.h"
#include <cuda_runtime.h>

namespace psi {

// Per-vertex status word written by an evaluation (and frozen for solved
// vertices):  >= 1  finite valuation, the value is the length of the strategy
// path from the vertex to the sink (its depth in the sink tree);
//             -1    valuation -inf (the path ends in a cycle won by Odd);
//             -2    valuation +inf (the path ends in a cycle won by Even);
//              0    the sink itself (never stored for a vertex).
constexpr int32_t ST_NEG_INF = -1;
constexpr int32_t ST_POS_INF = -2;
constexpr int32_t ST_UNRESOLVED = INT32_MIN;

constexpr int kBlock = 256;   // threads per block of most kernels

__host__ __device__ __forceinline__ int32_t st_infinite(int32_t st)
{
    return st == ST_POS_INF ? 1 : (st == ST_NEG_INF ? -1 : 0);
}

// Path record of a vertex, written by an evaluation: its successor in the
// strategy (-1 = the sink), its priority, and a summary of its path to the
// sink: the highest priority on it (rmax) and one word with the path's length
// and how many of its vertices carry rmax (path_word).  rmax == RM_UNKNOWN
// until the vertex is evaluated, RM_POS_INF / RM_NEG_INF where its valuation
// is infinite.  16-byte aligned so one load fetches it all and the
// (rmax, word) pair is published as one 8-byte store.
struct __align__(16) PathNode {
    int32_t parent, pri, rmax, word;
};
constexpr int32_t RM_UNKNOWN = INT32_MIN;
constexpr int32_t RM_POS_INF = INT32_MIN + 1;
constexpr int32_t RM_NEG_INF = INT32_MIN + 2;

// Depth (path length) and count in one word, 16 bits each: a walk that meets
// a finished ancestor takes both from the record it has loaded anyway, where
// a separate depth array cost one more random access per vertex.  A path of
// kDeepPath vertices or more has the word's depth at kDeepPath: its depth is
// then in the status word and its count in the array rdeep.
constexpr int32_t kDeepPath = 0xffff;
__host__ __device__ __forceinline__ int32_t path_word(int32_t depth, int32_t count)
{
    return depth < kDeepPath ? (int32_t)((uint32_t)depth << 16 | (uint32_t)count) : (int32_t)((uint32_t)kDeepPath << 16);
}
__host__ __device__ __forceinline__ int32_t path_word_depth(int32_t w) { return (int32_t)((uint32_t)w >> 16); }
__host__ __device__ __forceinline__ int32_t path_word_count(int32_t w) { return w & 0xffff; }

// Comparison key of a vertex after an evaluation: 4 bytes, what the switch
// step gathers per compared edge (n = 2^24 keys take 64 MiB and stay in L2).
// With (M, c) the root-path summary of a finite vertex (the highest priority
// on its path to the sink and its count), let
//   q = M < KEY_MCAP ? (M << 7 | min(c, 126)) : KEY_MCAP << 7
// and key = +q if M is even, -q if M is odd; +inf -> KEY_POS_INF, -inf ->
// KEY_NEG_INF; the sink (empty path) -> 0.  The key is a monotone function of
// the valuation order: between distinct summaries the highest priority whose
// counts differ is max(M_u, M_w), so a higher even M is better and a higher
// odd M worse, and at equal M a larger count is better if M is even, worse if
// odd -- clamping c, or M together with c, only merges neighbours.  Hence
// key_u > key_w implies u better than w, and equal keys of distinct finite
// vertices are decided by their exact summaries, then by a walk.
constexpr int32_t KEY_POS_INF = INT32_MAX;
constexpr int32_t KEY_NEG_INF = -INT32_MAX;
constexpr int32_t KEY_MCAP = (1 << 24) - 1;
__host__ __device__ __forceinline__ int32_t finite_key(int32_t m, int32_t c)
{
    int32_t q = (m < KEY_MCAP) ? ((m << 7) | (c < 126 ? c : 126)) : (KEY_MCAP << 7);
    return (m & 1) ? -q : q;
}
__host__ __device__ __forceinline__ int key_infinite(int32_t k)
{
    return k == KEY_POS_INF ? 1 : (k == KEY_NEG_INF ? -1 : 0);
}

// Change tracking (kernels.h: ChangeTrack), warp-collective: every lane of a
// converged warp calls it.  mode 2 (a changed key): every in-neighbour of the
// lane's vertex v gets need = 1; mode 1 (v re-evaluated, key unchanged):
// those with tie set; 0: none.  The in-edges of the lanes with a mode are
// spread over the warp's lanes (their rev_off spans laid end to end), so one
// round of rev_src loads usually covers them all, instead of one dependent
// load per in-edge on those lanes while the rest of the warp waits.
// With rev (b, d) given, the lane's in-edges are rev_src[b, b + d) and
// rev_off is not read.
__device__ __forceinline__ void flag_in_neighbours(const ChangeTrack &t, int mode, int32_t v,
                                                   const int2 *rev = nullptr)
{
    if (!t.need || (t.quiet && *t.quiet)) return;
    if (!t.tie && mode == 1) mode = 0;
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned lanes = __ballot_sync(kAll, mode != 0);
    if (!lanes) return;
    const int lane = threadIdx.x & 31;
    int32_t b = 0, d = 0;
    if (mode) {
        if (rev) {
            b = rev->x;
            d = rev->y;
        } else {
            b = t.rev_off[v];
            d = t.rev_off[v + 1] - b;
        }
    }
    int32_t incl = d;   // inclusive prefix of d over the lanes
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t x = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += x;
    }
    const int32_t total = __shfl_sync(kAll, incl, 31);   // <= m: distinct vertices' in-edges
    const int32_t excl = incl - d;
    for (int32_t j0 = 0; j0 < total; j0 += 32) {
        const int32_t j = j0 + lane;
        // owner lane of edge j: the number of lanes whose inclusive count is
        // <= j (a binary search over the non-decreasing prefix, five rounds of
        // shuffles; lanes without in-edges own none)
        int l = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const int32_t y = __shfl_sync(kAll, incl, l + step - 1);
            if (y <= j) l += step;
        }
        const int32_t el = __shfl_sync(kAll, excl, l), bl = __shfl_sync(kAll, b, l);
        const int ml = __shfl_sync(kAll, mode, l);
        if (j < total) {
            const int32_t u = t.rev_src[bl + (j - el)];
            if (ml == 2 || t.tie[u]) t.need[u] = 1;
        }
    }
}
__device__ __forceinline__ void flag_in_neighbours(const ChangeTrack &t, bool changed, int32_t v)
{
    flag_in_neighbours(t, changed ? 2 : 0, v);
}

// (max, count of max) of the union of two priority multisets
__device__ __forceinline__ void top1_merge(int32_t &m, int32_t &c, int32_t m2, int32_t c2)
{
    if (m2 > m) {
        m = m2;
        c = c2;
    } else if (m2 == m) {
        c += c2;
    }
}

struct Top2 {
    int32_t m1, c1, m2, c2;
};

__device__ __forceinline__ void top2_add(Top2 &t, int32_t p)
{
    if (p > t.m1) {
        t.m2 = t.m1;
        t.c2 = t.c1;
        t.m1 = p;
        t.c1 = 1;
    } else if (p == t.m1) {
        t.c1++;
    } else if (p > t.m2) {
        t.m2 = p;
        t.c2 = 1;
    } else if (p == t.m2) {
        t.c2++;
    }
}

// adds count occurrences of priority p
__device__ __forceinline__ void top2_add_n(Top2 &t, int32_t p, int32_t count)
{
    if (count <= 0) return;
    if (p > t.m1) {
        t.m2 = t.m1;
        t.c2 = t.c1;
        t.m1 = p;
        t.c1 = count;
    } else if (p == t.m1) {
        t.c1 += count;
    } else if (p > t.m2) {
        t.m2 = p;
        t.c2 = count;
    } else if (p == t.m2) {
        t.c2 += count;
    }
}

// Landmark skips for the comparison walks.  A finite vertex at depth d has
// its landmark at depth L = SKIP_K * floor((d - 1) / SKIP_K): the ancestor
// there (the sink at L = 0).  skip[v] = (landmark, top two priorities of the
// segment from v up to the landmark, exclusive, one word: their counts, a
// segment holds at most SKIP_K vertices, and the number of the evaluation that
// wrote it).  Written by the walks of a full evaluation (root_kernels.cu) as
// one 16-byte word, where want_landmarks asks for them; a patch marks its
// vertices' records unknown (the paths of all other vertices are unchanged).  SKIP_K
// measured on GB300 (graph solve of the 2^24 random game, long-path 2^23):
// 64: 63.8, 57.8 ms; 32: 62.8, 57.8; 16: 62.0, 57.0; 8: 61.6, 55.5; 4: 61.8,
// 55.5 ms: shorter segments shorten the steps after the last jump more than
// they add jumps.
constexpr int32_t SKIP_K = 8;
constexpr int32_t SKIP_UNKNOWN = INT32_MIN;
__host__ __device__ __forceinline__ int32_t skip_landmark_depth(int32_t d) { return ((d - 1) / SKIP_K) * SKIP_K; }
// the record's word: c1 - 1 (3 bits), c2 (4 bits), evaluation number (25 bits)
constexpr uint32_t kEpochMask = (1u << 25) - 1;
__device__ __forceinline__ int32_t skip_c1(int32_t w) { return (w & 7) + 1; }
__device__ __forceinline__ int32_t skip_c2(int32_t w) { return (w >> 3) & 15; }
__device__ __forceinline__ uint32_t skip_epoch(int32_t w) { return (uint32_t)w >> 7; }
__device__ __forceinline__ int4 skip_pack(int32_t anc, const Top2 &t, uint32_t epoch = 0)
{
    return make_int4(anc, t.m1, t.m2, (int32_t)(epoch << 7 | (uint32_t)t.c2 << 3 | (uint32_t)(t.c1 - 1)));
}
__device__ __forceinline__ void skip_merge(Top2 &t, const int4 s)
{
    top2_add_n(t, s.y, skip_c1(s.w));
    top2_add_n(t, s.z, skip_c2(s.w));
}

// 16-byte records read and written whole while other threads do the same.
__device__ __forceinline__ int4 load_whole(const int4 *p)
{
    int4 r;
    asm volatile("{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
                 "ld.relaxed.gpu.global.b128 t, [%4];\n\t"
                 "mov.b128 {lo, hi}, t;\n\t"
                 "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p)
                 : "memory");
    return r;
}
__device__ __forceinline__ void store_whole(int4 *p, const int4 r)
{
    asm volatile("{\n\t.reg .b128 t;\n\t.reg .b64 lo, hi;\n\t"
                 "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\t"
                 "mov.b128 t, {lo, hi};\n\t"
                 "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w)
                 : "memory");
}

// Publishes a summary (rmax, word) as one 8-byte word.  deep: what was written
// before it (status, rdeep) is visible to any thread that acquires it; the
// release costs a wait for all of the thread's stores, so others do without.
__device__ __forceinline__ void publish_summary(PathNode *p, int32_t m, int32_t word, bool deep = false)
{
    const unsigned long long w = (unsigned long long)(uint32_t)m | ((unsigned long long)(uint32_t)word << 32);
    if (deep) asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(&p->rmax), "l"(w) : "memory");
    else asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(&p->rmax), "l"(w) : "memory");
}
__device__ __forceinline__ int32_t acquire_rmax(const PathNode *p)
{
    int32_t x;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(x) : "l"(&p->rmax) : "memory");
    return x;
}

// Warps in the largest block (1,024 threads): the block-aggregated appends
// keep one count per warp, for any block size the kernels use.
constexpr int kMaxBlockWarps = 32;

// Block-aggregated append: every thread of the block calls it (no early
// return before); one atomic on the shared counter per block instead of one
// per warp, which serialises when most warps append (the sink's children,
// the unreached vertices).
__device__ __forceinline__ void block_append(bool flag, int32_t value, int32_t *__restrict__ list,
                                             int32_t *__restrict__ count)
{
    __shared__ int32_t warp_base[kMaxBlockWarps];
    __shared__ int32_t block_base;
    const unsigned mask = __ballot_sync(0xffffffffu, flag);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) warp_base[w] = __popc(mask);
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t sum = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            int32_t t = warp_base[i];
            warp_base[i] = sum;
            sum += t;
        }
        block_base = sum ? atomicAdd(count, sum) : 0;
    }
    __syncthreads();
    if (flag) list[block_base + warp_base[w] + __popc(mask & ((1u << lane) - 1))] = value;
}

// Block-aggregated append of up to K values per thread (v[k] < 0: none):
// every thread of the block calls it; one atomic per block and three block
// barriers per call (the last one frees the shared words for the next call).
// Scans give each thread K items per pass, so K loads are in flight before
// the barriers instead of one.
template <int K>
__device__ __forceinline__ void block_append_k(const int32_t (&v)[K], int32_t *__restrict__ list,
                                               int32_t *__restrict__ count)
{
    __shared__ int32_t warp_base[kMaxBlockWarps];
    __shared__ int32_t block_base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t mine = 0;
#pragma unroll
    for (int k = 0; k < K; k++) mine += v[k] >= 0;
    int32_t incl = mine;   // inclusive prefix over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_base[w] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t sum = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            const int32_t t = warp_base[i];
            warp_base[i] = sum;
            sum += t;
        }
        block_base = sum ? atomicAdd(count, sum) : 0;
    }
    __syncthreads();
    int32_t at = block_base + warp_base[w] + incl - mine;
#pragma unroll
    for (int k = 0; k < K; k++)
        if (v[k] >= 0) list[at++] = v[k];
    __syncthreads();
}

// Sixteen byte flags as one 16-byte word (vector loads of flag arrays).
union Bytes16 {
    int4 q;
    uint8_t b[16];
};

__device__ __forceinline__ bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

// Warp-aggregated slot reservation: every lane of a converged warp calls it;
// a lane with flag set gets base + its rank among the flagged lanes, where
// base = atomicAdd(count, flagged lanes) (one atomic per warp); -1 otherwise.
__device__ __forceinline__ int32_t warp_reserve(bool flag, int32_t *count, int32_t base_offset = 0)
{
    const unsigned m = __ballot_sync(0xffffffffu, flag);
    if (!m) return -1;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int32_t base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    return flag ? base_offset + base + __popc(m & ((1u << lane) - 1)) : -1;
}

// Appends a changed vertex to the change list, one atomic per group of lanes
// that changed together; nothing once the list has overflowed (its count
// then stays above the capacity, which marks it incomplete).
__device__ __forceinline__ void note_change(const ChangeList &c, int32_t v)
{
    if (*(volatile int32_t *)c.count > c.cap) return;
    cooperative_groups::coalesced_group grp = cooperative_groups::coalesced_threads();
    int32_t base = 0;
    if (grp.thread_rank() == 0) base = atomicAdd(c.count, (int32_t)grp.size());
    base = grp.shfl(base, 0);
    const int32_t p = base + (int32_t)grp.thread_rank();
    if (p < c.cap) c.list[p] = v;
}

// What a solver keeps of its count of grid barriers between launches
// (SolveSync): phase k votes in word k % 3, so the remainder.  The count itself
// would wrap around at 2^32, no multiple of 3, and two phases in a row, one of
// which clears the other's votes, would share a word.
__host__ __device__ __forceinline__ uint32_t kept_phase(uint32_t phase) { return phase % 3; }

// Whether the coming full evaluation writes landmark records: a sixth to a
// quarter of its time (2^24: 0.86 -> 0.64 ms), which pays where the comparisons
// walk much (one switch step of 2^24 vertices with 5*10^7 jumps and steps 1.9
// ms, without them over 5).  So it does when the last switch step took more
// than n / 2 steps, or with records n / 8 jumps and steps, or a single vertex
// had far to walk.  ms per solve, always -> so: 2^24 random games 32.9, 40.2,
// 41.3, 37.5 -> 30.9, 38.8, 38.9, 35.7 (never: 31.5, 48.5, 38.7, 35.9), long-path
// 2^23 17.6 -> 15.3, 256 games 16.9 -> 16.1; n and n / 8, n / 2 and n / 4, n / 8 and
// n / 16 are within 2% of it.
__host__ __device__ __forceinline__ bool want_landmarks(const EvalGates *g, const unsigned long long *sw, int32_t n)
{
    return g->lm_far || sw[1] > (unsigned long long)(g->lm_have ? n / 8 : n / 2);
}

// Before an evaluation (one thread): decides between a patch and the full
// evaluation (patch_kernels.cu) and resets what either starts from.
__host__ __device__ __forceinline__ void patch_begin(const PatchArgs &a)
{
    EvalGates *g = a.g;
    ++*a.epoch;
    const bool fresh = *a.quiet > 0;   // after a reset: the statistics are of another solve
    if (fresh) --*a.quiet;
    g->lm_want = !fresh && want_landmarks(g, a.sw, a.n);
    g->lm_far = 0;
    const int32_t cc = g->ccount;
    g->ccount = 0;   // the next switch steps list their changes afresh
    g->csnap = cc;
    g->acount = 0;
    g->lcnt[0] = g->lcnt[1] = g->lcnt[2] = 0;
    bool ok = g->try_patch && cc <= a.ccap && (int64_t)*a.ucount + a.acap <= a.ucap;
    // the evaluation numbered 0 clears the landmark records of the last round
    // (k_root_init), so it is a full one
    if ((*a.epoch & kEpochMask) == 0) ok = false;
    if (ok && g->skip > 0) {
        g->skip--;
        ok = false;
    }
    g->patch = ok ? 1 : 0;
    g->eval = ok ? 0 : 1;
    if (!ok) {
        *a.ucount = 0;      // the full evaluation collects the unreached vertices afresh
        g->mfrom[0] = g->mfrom[1] = 0;
    }
}

// One event of a batch's per-game accounting (switch_kernels.cu says what
// state and events are).
__device__ __forceinline__ void batch_event(int32_t event, int4 &state, unsigned long long &gcount)
{
    int4 s = state;
    if (event == 0) {
        if (!s.w && !s.z) s.x++;
    } else if (event == 1) {
        if (!s.w && !s.z && gcount == 0) s.z = 1;
        gcount = 0;
    } else if (event == 2) {
        if (!s.w) s.y++;
    } else {
        if (!s.w) {
            if (gcount == 0) s.w = 1;
            else s.z = 0;
        }
        gcount = 0;
    }
    state = s;
}

// mark_solved restricted to the last evaluation's unreached vertices: every
// other non-solved vertex is finite.  Every thread of the grid calls it.
// With game_of/gmask (served games), only vertices of games whose mask is set.
__device__ __forceinline__ void mark_solved_pass(const MarkArgs &m)
{
    const int32_t nu = *m.ucount;
    const int32_t i0 = m.from ? *m.from : 0;
    const int32_t target = (m.player == 0) ? ST_POS_INF : ST_NEG_INF;
    for (int64_t i = i0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nu; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = m.ulist[i];
        if (m.gmask) {
            const int32_t g = m.game_of[u];
            if (g < 0 || !m.gmask[g]) continue;
        }
        if (m.st[u] == target) m.solved[u] = 1;
    }
    if (!m.from) return;
    // the last block to finish (every block has read *from by then) moves
    // the start past the entries scanned
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicInc(m.done, gridDim.x - 1) == gridDim.x - 1) *m.from = nu;
    }
}

// Tour node ids (an Euler tour of the strategy forest, two nodes per vertex):
// node 2v is v's "down" node (leaving v's subtree toward the sink), 2v+1 its
// "up" node (entering it); 2n / 2n+1 are the sink's down / up nodes.  The list
// starts at the sink's up node and ends at the sink's down node (successor -1).
constexpr int32_t TOUR_END = -1;

// Device-side error bits (a word the host reads back at sync points).
constexpr uint32_t DERR_SUBLIST_CAP = 1u << 0;   // a sublist walk exceeded the list length
constexpr uint32_t DERR_WALK_CAP = 1u << 1;      // a valuation walk exceeded its step cap
constexpr uint32_t DERR_PASS_CAP = 1u << 2;      // a comparison exceeded its pass cap
constexpr uint32_t DERR_BAD_INPUT = 1u << 3;     // malformed strategy (target out of range)


__host__ __device__ __forceinline__ int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace psi

#define PSI_CUDA_TRY(expr)                                                            \
    do {                                                                              \
        cudaError_t e__ = (expr);                                                     \
        if (e__ != cudaSuccess)                                                       \
            return ::psi::fail(PSI_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e__)); \
    } while (0)

#endif
