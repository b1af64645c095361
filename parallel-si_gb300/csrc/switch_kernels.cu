// switch_kernels.cu -- the all-switches step and valuation export on sm_103a.
//
// Valuation order (cpu_parity.cpp:154-236, valuation.cpp:70-115): +inf > every
// finite valuation > -inf.  Two finite valuations are count vectors over the
// priorities on the strategy paths to the sink; the higher one has the larger
// count at the highest priority where the counts differ if that priority is
// even, the smaller count if it is odd.
//
// A comparison of two finite valuations u, w is settled in three tiers, each
// exact:
//  1. u == w: equal.
//  2. Root-path summaries (highest priority M on the path, its count c), made
//     by the evaluation: if (M_u, c_u) != (M_w, c_w), the highest priority
//     whose counts differ is max(M_u, M_w) -- every higher priority is absent
//     from both paths -- and its two counts are known.
//  3. Otherwise walk both paths up to their lowest common ancestor (the counts
//     on the common part cancel), keeping the highest priority and its count
//     per side; if both sides agree, walk again below it (compare.cuh).  Every
//     pass removes a distinct priority, so the passes are bounded by the path
//     lengths.
//
// The switch rule is the reference's (cpu_parity.cpp:239-263,
// gpu_parity.cu:264-300): scan the successors in CSR order, move to a
// successor only on a strict improvement for the owner, count the moves.
#include <climits>
#include <cooperative_groups.h>
#include <cub/block/block_reduce.cuh>

#include "compare.cuh"
#include "device_common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace psi {

namespace {

inline unsigned grid_for(int64_t items, int block = kBlock)
{
    int64_t g = ceil_div(items, block);
    return (unsigned)(g < 1 ? 1 : g);
}

constexpr int32_t kFarWalk = 4096;   // steps after which landmarks are asked for (want_landmarks)

// Even's view of finite u against finite w (u != w) when their keys are
// equal: the exact summaries decide, else a walk to the lowest common
// ancestor (w = -1 is the sink).
__device__ int compare_equal_keys(const PathNode *__restrict__ node, const Landmarks &marks,
                                  const int32_t *__restrict__ st, const int32_t *__restrict__ rdeep, int32_t u, int32_t w, int32_t &loads,
                                  uint32_t *__restrict__ err)
{
    const int2 ru = *reinterpret_cast<const int2 *>(&node[u].rmax);
    const int2 rw = (w >= 0) ? *reinterpret_cast<const int2 *>(&node[w].rmax) : make_int2(-1, 0);
    int32_t du = path_word_depth(ru.y), cu = path_word_count(ru.y);
    int32_t dw = path_word_depth(rw.y), cw = path_word_count(rw.y);   // the sink: depth 0, count 0
    if (du == kDeepPath) {
        du = st[u];
        cu = rdeep[u];
    }
    if (dw == kDeepPath) {
        dw = st[w];
        cw = rdeep[w];
    }
    if (ru.x != rw.x) return ru.x > rw.x ? decide(ru.x, cu, 0) : decide(rw.x, 0, cw);
    if (cu != cw) return decide(ru.x, cu, cw);
    const int32_t before = loads;
    const int c = marks.skip ? lean_compare<true>(node, marks.skip, u, du, w, dw, loads, INT_MAX, err)
                             : lean_compare<false>(node, nullptr, u, du, w, dw, loads, INT_MAX, err);
    if (loads - before > kFarWalk) *marks.far = 1;
    return c;
}

// The vertices of plist whose need flag is set (and, with gmask, whose game
// takes this step), appended to list with one atomic per block.  A block
// pass covers kNeedPer * blockDim entries (each thread kNeedPer of them,
// blockDim apart, so every load is coalesced; plist + offset may not be
// 16-byte aligned, so no vector loads): block_append_k per pass.
constexpr int kNeedPer = 4;

// What a step needs done before its switch kernel, in the launch that collects
// its list: the work counter and the statistics cleared, and mark_solved
// (launches of their own cost 2 us each and more where steps are small).
__device__ __forceinline__ void need_prelude(uint32_t *claim, unsigned long long *stats, const MarkArgs &mark)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (claim) *claim = 0;
        stats[0] = stats[1] = stats[2] = stats[3] = 0;
    }
    if (mark.ucount) mark_solved_pass(mark);
}

// The same for a player without vertices, gated as its list would be: in the
// solve graph Even's mark_solved waits for Odd's best response also where no
// vertex is Even's.
__global__ void k_need_none(const int32_t *__restrict__ gate, unsigned long long *__restrict__ stats, MarkArgs mark)
{
    if (gate && !*gate) return;
    need_prelude(nullptr, stats, mark);
}

// The switch kernels' last block clears the list's counter for the next step:
// every block calls it at its end, all its threads having read the counter.
__device__ __forceinline__ void list_used(int32_t *count, uint32_t *done)
{
    if (!done) return;
    __syncthreads();
    if (threadIdx.x == 0 && atomicInc(done, gridDim.x - 1) == gridDim.x - 1) *count = 0;
}
__global__ void k_need_list(int32_t np, const int32_t *__restrict__ plist, const uint8_t *__restrict__ need,
                            const int32_t *__restrict__ game_of, const int32_t *__restrict__ gmask,
                            const int32_t *__restrict__ gate, int32_t *__restrict__ list, int32_t *__restrict__ count,
                            uint32_t *__restrict__ claim, unsigned long long *__restrict__ stats, MarkArgs mark)
{
    if (gate && !*gate) return;
    need_prelude(claim, stats, mark);
    const int64_t pass = (int64_t)kNeedPer * blockDim.x;
    for (int64_t b0 = (int64_t)blockIdx.x * pass; b0 < np; b0 += (int64_t)gridDim.x * pass) {
        int32_t v[kNeedPer];
#pragma unroll
        for (int k = 0; k < kNeedPer; k++) {
            const int64_t i = b0 + (int64_t)k * blockDim.x + threadIdx.x;
            v[k] = (i < np) ? plist[i] : -1;
        }
#pragma unroll
        for (int k = 0; k < kNeedPer; k++)
            if (v[k] >= 0 && !(need[v[k]] && (!gmask || gmask[game_of[v[k]]]))) v[k] = -1;
        block_append_k(v, list, count);
    }
}

// The same list from the vertex arrays themselves, for a single game or a
// batch (every vertex of `player` is on plist): kVec consecutive vertices per
// thread and pass, their need and owner bytes in one 16-byte load each, so the
// scan streams 2n bytes instead of plist and a gather of need through it.
// The list is in vertex order within a block pass, which is all the switch
// kernel needs (each vertex is examined on its own).
constexpr int kVec = 16;
__global__ void k_need_ids(int32_t n, int32_t player, const int8_t *__restrict__ owner,
                           const uint8_t *__restrict__ need, const int32_t *__restrict__ gate,
                           int32_t *__restrict__ list, int32_t *__restrict__ count, uint32_t *__restrict__ claim,
                           unsigned long long *__restrict__ stats, MarkArgs mark)
{
    if (gate && !*gate) return;
    need_prelude(claim, stats, mark);
    const bool vec = aligned16(owner) && aligned16(need);
    const int64_t pass = (int64_t)kVec * blockDim.x;
    for (int64_t b0 = (int64_t)blockIdx.x * pass; b0 < n; b0 += (int64_t)gridDim.x * pass) {
        const int64_t v0 = b0 + (int64_t)kVec * threadIdx.x;
        int32_t v[kVec];
        if (vec && v0 + kVec <= n) {
            Bytes16 nd, ow;
            nd.q = *reinterpret_cast<const int4 *>(need + v0);
            ow.q = *reinterpret_cast<const int4 *>(owner + v0);
#pragma unroll
            for (int k = 0; k < kVec; k++) v[k] = (nd.b[k] && ow.b[k] == player) ? (int32_t)(v0 + k) : -1;
        } else {
#pragma unroll
            for (int k = 0; k < kVec; k++) {
                const int64_t i = v0 + k;
                v[k] = (i < n && need[i] && owner[i] == player) ? (int32_t)i : -1;
            }
        }
        block_append_k(v, list, count);
    }
}

// One thread per vertex of the list (all owned by `player`; the list is plist
// itself, np entries, or -- with count != nullptr -- the *count vertices
// k_need_list selected).  Per compared edge the common case is one 4-byte
// gather (the successor's comparison key) and one integer comparison; equal
// keys of distinct finite vertices fall back to the exact summaries and,
// rarely, a walk.  stats[0] += compared edges, stats[1] += parent/priority
// loads of the walks, stats[2] += vertices whose strategy changed, stats[3]
// += strict improvements.  For a batch of games (game_of != nullptr) the
// strict improvements are also added to gcount[game of the vertex]; with
// gmask only vertices of games whose mask is set switch.  With need, an
// examined vertex is sticky if its best key is shared by two distinct
// finite vertices (start or successors): its choice then rests on a walk,
// which depends on more than the keys tracked between steps.  With tie_out
// the examined vertex gets need = 0 and tie_out = sticky (ChangeTrack says
// when it is looked at again), and the successors a sticky vertex's choice
// rests on (those at its best key) get watch = 1; without it, need = sticky.
// The choice the scan ends with is the first of the best vertices, so exact
// comparisons are wanted only among those at the best key.  Only COUNT, where
// the caller wants the number of strict improvements the scan makes, compares
// equal keys on the way there too; otherwise a changed vertex counts as one.
// With that and lean_compare for the walks, switch steps of the 2^24 random
// game 12.0 -> 10.5 ms per solve (long-path 7.05 -> 6.85).  Blocks per SM: four
// (64 registers) without COUNT, ms per solve against the five of 48 registers
// and spills that the compiler chose: 2^24 30.8, 38.3, 38.6 -> 30.2, 37.5, 38.2,
// long-path 2^23 14.7 -> 14.45; three (79 registers) with COUNT: 2^18 to 4*10^5
// vertices step by step 2% faster than four.
// COUNT's comparisons go from tie to tie too (a mask, as without): what the
// scan's choice is at a tie follows from the places that set the best key
// before it.  Step by step at 2*10^4, 5*10^4, 4*10^5 vertices and 5*10^4 with 8
// priorities 2110, 2430, 5660, 4200 -> 1990, 2270, 5300, 3770 us against redoing
// such a vertex successor by successor (kept past 32 successors).
template <bool COUNT>
__global__ void __launch_bounds__(kBlock) k_switch(int32_t np, const int32_t *__restrict__ plist,
                                                   int32_t *__restrict__ count, int32_t player,
                                                   const int32_t *__restrict__ off, const int32_t *__restrict__ tgt,
                                                   int32_t *__restrict__ strat, const int32_t *__restrict__ st,
                                                   const int32_t *__restrict__ key,
                                                   const PathNode *__restrict__ node,
                                                   const int32_t *__restrict__ rdeep,
                                                   unsigned long long *__restrict__ stats,
                                                   const int32_t *__restrict__ game_of,
                                                   unsigned long long *__restrict__ gcount,
                                                   const int32_t *__restrict__ gmask,
                                                   uint32_t *__restrict__ err,
                                                   const int32_t *__restrict__ gate, uint8_t *__restrict__ need,
                                                   ChangeList changes, uint8_t *__restrict__ tie_out,
                                                   uint8_t *__restrict__ watch, Landmarks marks,
                                                   uint32_t *__restrict__ claim, uint32_t *__restrict__ list_done)
{
    if (gate && !*gate) return;
    if (!*marks.have) marks.skip = nullptr;
    if (count) np = *(volatile int32_t *)count;
    // a block past the list's end has nothing to count either (uniform per
    // block: the block reduction below is never left waiting)
    if ((int64_t)blockIdx.x * blockDim.x >= np) {
        list_used(count, list_done);
        return;
    }
    // A bounded grid, so the work counters are reduced once per block (a few
    // thousand atomics per launch instead of a set per 256 vertices).  The
    // list is dealt out to warps in chunks of 32 entries: every warp takes
    // the chunk at its own index first, then -- with claim, a device word
    // zeroed by k_need_list -- from a counter, one atomic per claim, else the
    // next chunk one grid's worth of warps further on.  Claims keep a warp
    // that meets a long comparison walk from holding up chunks that a fixed
    // stride would have dealt to it as well (2^24 random game: 16.0 -> 14.8 ms
    // of switch steps per solve); the first chunk at the warp's own index
    // keeps short lists spread over the whole grid.  All warps of the GPU
    // claim from one address, so a claim takes half of what would be the
    // warp's share of the rest, 2 to 16 chunks: large while there is much
    // left, small at the end, where a walk would hold up the launch (2^24
    // random games, ms per solve with 2, 4, 8, 16 chunks always: 12.6, 11.9,
    // 11.5, 11.8 with few ties, 21.2, 20.7, 21.0, 22.5 with many, 2^22 vertices
    // with 8 priorities 6.5, 6.8, 7.5, 9.2; so: 11.1, 19.8, 6.5).  In a batch
    // chunks in a row belong to one game, whose walks may all be long: one at
    // a time (256 games of 100 to 200,000 vertices, ms per solve: 17.3, with
    // up to 16 18.1; 150 games up to 50,000: 4.43 and 4.59).  The next
    // entry's vertex, choice and edge range are read before the present one's
    // successors and keys, which wait for theirs (11.1 -> 10.9, 8 priorities
    // 6.5 -> 6.4, long-path 5.23 -> 5.10; its successors ahead as well: 11.3,
    // 21.7, 6.9, for the registers).  A thread's edge count is at most m (< 2^31).
    constexpr int kMinClaim = 2, kMaxClaim = 16;
    const int lane = threadIdx.x & 31;
    const int64_t nchunk = (np + 31) >> 5;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    int64_t base = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int per = 1;
    int32_t t_edges = 0, t_loads = 0, t_changed = 0, t_moves = 0;
    while (base < nchunk) {
        int32_t vn = -1, curn = 0, e0n = 0, e1n = 0;   // the next entry (-1: none)
        auto ahead = [&](int k) {
            const int64_t i = (base + k) * 32 + lane;
            vn = (k < per && i < np) ? __ldcs(&plist[i]) : -1;   // one-use streams are evict-first: L2 keeps the keys
            if (vn < 0) return;
            curn = strat[vn];
            e0n = __ldcs(&off[vn]);
            e1n = __ldcs(&off[vn + 1]);
        };
        ahead(0);
        for (int k = 0; k < per; k++) {
            const int32_t v = vn;
            int32_t cur = curn;
            const int32_t e0 = e0n, e1 = e1n;
            ahead(k + 1);
            if (v < 0) continue;
            if (gmask && !gmask[game_of[v]]) continue;
            int32_t kc = (cur >= 0) ? key[cur] : 0;
            t_edges += e1 - e0;
            int32_t moves = 0;
            // best key over the start and all successors, and whether a second
            // distinct vertex attains it (a tie)
            int32_t ext = kc, ext_v = cur;
            bool tie = false;
            // which of the first 32 successors attain it, besides the first that
            // does; with COUNT, which attain the best key up to their place, and
            // which set it
            uint32_t ties = 0, sets = 0;
            // Key pass: successors in batches of kBatch -- all ids, then all
            // keys, before the comparisons (independent gathers in flight per
            // thread).  Five per batch (one batch for out-degrees up to 5): switch
            // steps 12.6 -> 12.1 ms per 2^24 solve against four; six the same as five.
            constexpr int kBatch = 5;
            const int32_t cur0 = cur, kc0 = kc;
            bool exact = false;
            for (int32_t eb = e0; eb < e1; eb += kBatch) {
                const int32_t cnt = min(kBatch, e1 - eb);
                int32_t us[kBatch], ks[kBatch];
    #pragma unroll
                for (int j = 0; j < kBatch; j++) us[j] = (j < cnt) ? __ldcs(&tgt[eb + j]) : 0;
    #pragma unroll
                for (int j = 0; j < kBatch; j++) ks[j] = (j < cnt) ? key[us[j]] : 0;
    #pragma unroll
                for (int j = 0; j < kBatch; j++) {
                    if (j >= cnt) break;
                    const int32_t u = us[j], ku = ks[j], at = eb - e0 + j;
                    if ((player == 0) ? ku > ext : ku < ext) {
                        ext = ku;
                        ext_v = u;
                        tie = false;
                        if (!COUNT) ties = 0;
                        else if (at < 32) sets |= 1u << at;
                        moves++;
                    } else if (ku == ext && u != ext_v) {
                        tie = true;
                        if (at < 32) ties |= 1u << at;
                        if (COUNT && !key_infinite(ku)) exact = true;
                    }
                }
            }
            // the first vertex at the best key, then exact comparisons with the
            // others that share it (none for an infinity)
            cur = ext_v;
            const uint32_t tied = ties;
            if (!COUNT) {
                if (tie && !key_infinite(ext)) {
                    for (int32_t j = 0;; j++) {
                        if (next_tied(ties, j) >= e1 - e0) break;
                        const int32_t u = tgt[e0 + j];
                        if (u == cur || (j >= 32 && key[u] != ext)) continue;
                        const int c = compare_equal_keys(node, marks, st, rdeep, u, cur, t_loads, err);
                        if ((player == 0) ? c > 0 : c < 0) cur = u;
                    }
                }
                moves = cur != cur0 ? 1 : 0;
            } else if (exact && e1 - e0 <= 32) {
                // the scan again, from tie to tie: each against the choice up to
                // there, the last vertex that set the best key or one that won since
                int32_t set = -1;
                cur = cur0;
                for (; ties; ties &= ties - 1) {
                    const int32_t j = __ffs(ties) - 1, before = 31 - __clz(sets & ((1u << j) - 1));   // -1: none
                    if (before != set) {
                        set = before;
                        cur = tgt[e0 + set];
                    }
                    const int32_t u = tgt[e0 + j];
                    if (u == cur || key_infinite(key[u])) continue;
                    const int c = compare_equal_keys(node, marks, st, rdeep, u, cur, t_loads, err);
                    if ((player == 0) ? c > 0 : c < 0) {
                        cur = u;
                        moves++;
                    }
                }
                if (31 - __clz(sets) != set) cur = ext_v;   // set after the last tie
            } else if (exact) {
                cur = cur0;
                kc = kc0;
                moves = 0;
                for (int32_t e = e0; e < e1; e++) {
                    const int32_t u = tgt[e], ku = key[u];
                    int c;
                    if (ku != kc) c = ku > kc ? 1 : -1;
                    else if (u == cur || key_infinite(ku)) c = 0;
                    else c = compare_equal_keys(node, marks, st, rdeep, u, cur, t_loads, err);
                    if ((player == 0 && c > 0) || (player == 1 && c < 0)) {
                        cur = u;
                        kc = ku;
                        moves++;
                    }
                }
            }
            const bool sticky = tie && ext != 0 && !key_infinite(ext);
            if (tie_out) {
                need[v] = 0;
                tie_out[v] = sticky ? 1 : 0;
                // the successors the tie rests on, from the mask (2^20 vertices 5.02 ->
                // 4.92 ms per solve, 2^22 8.51 -> 8.37, long-path 2^23 15.3 -> 15.1)
                if (sticky && watch && !COUNT && e1 - e0 <= 32) {
                    if (ext_v >= 0) watch[ext_v] = 1;
                    for (uint32_t t = tied; t; t &= t - 1) watch[tgt[e0 + __ffs(t) - 1]] = 1;
                } else if (sticky && watch) {
                    for (int32_t e = e0; e < e1; e++) {
                        const int32_t u = tgt[e];
                        if (key[u] == ext) watch[u] = 1;
                    }
                }
            } else if (need) {
                need[v] = sticky ? 1 : 0;
            }
            if (moves) {   // strict improvements never return to cur0: cur != cur0
                strat[v] = cur;
                if (game_of) atomicAdd(&gcount[game_of[v]], (unsigned long long)moves);
                t_changed++;
                t_moves += moves;
                if (changes.list) note_change(changes, v);
            }
        }
        if (claim) {
            const int64_t share = (nchunk - base) / (2 * warps);
            per = game_of ? 1 : (int)(share < kMinClaim ? kMinClaim : (share < kMaxClaim ? share : kMaxClaim));
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(claim, (uint32_t)per);
            base = warps + __shfl_sync(0xffffffffu, b, 0);
        } else {
            base += warps;
        }
    }
    typedef cub::BlockReduce<longlong4, kBlock> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    longlong4 mine = make_longlong4(t_edges, t_loads, t_changed, t_moves);
    longlong4 tot = Reduce(tmp).Reduce(mine, [](const longlong4 &x, const longlong4 &y) {
        return make_longlong4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
    });
    if (threadIdx.x == 0) {
        if (tot.x) atomicAdd(&stats[0], (unsigned long long)tot.x);
        if (tot.y) atomicAdd(&stats[1], (unsigned long long)tot.y);
        if (tot.z) atomicAdd(&stats[2], (unsigned long long)tot.z);
        if (tot.w) atomicAdd(&stats[3], (unsigned long long)tot.w);
    }
    list_used(count, list_done);
}

// ---- warp-cooperative all-switches
// A warp takes 32 entries of the list at a time (one vertex per lane) and
// lays their successor lists end to end; every lane then gathers one
// successor and its key per round of 32 edges, whatever the degrees.  The
// switch rule is a prefix maximum: with score = key for Even and -key for Odd
// (a strict improvement for the owner is a strictly larger score), the running
// choice before successor j is the first vertex attaining the maximum score
// over the incumbent and the successors before j; j is a strict improvement
// (a move) iff its score exceeds that maximum.  A segmented warp scan (one
// segment per vertex, max with the earlier element winning ties, the
// incumbent as the carry into the first round) gives every lane that running
// choice, so the moves of a vertex are the improving lanes of its segment and
// its final choice is the scan's last value.  Equal scores of distinct finite
// vertices mean that the keys cannot tell: such a vertex is redone by its
// lane with the exact comparisons (summaries, then walks), as in k_switch.
struct ScoreArg {
    int32_t sc, u;
};

// the earlier element wins ties (first strict maximum)
__device__ __forceinline__ ScoreArg first_max(ScoreArg a, ScoreArg b) { return (a.sc >= b.sc) ? a : b; }

__global__ void __launch_bounds__(kBlock) k_switch_warp(int32_t np, const int32_t *__restrict__ plist,
                                                        int32_t *__restrict__ count, int32_t player,
                                                        const int32_t *__restrict__ off,
                                                        const int32_t *__restrict__ tgt, int32_t *__restrict__ strat,
                                                        const int32_t *__restrict__ st,
                                                        const int32_t *__restrict__ key,
                                                        const PathNode *__restrict__ node,
                                                        const int32_t *__restrict__ rdeep,
                                                        unsigned long long *__restrict__ stats,
                                                        const int32_t *__restrict__ game_of,
                                                        unsigned long long *__restrict__ gcount,
                                                        const int32_t *__restrict__ gmask,
                                                        uint32_t *__restrict__ err,
                                                        const int32_t *__restrict__ gate, uint8_t *__restrict__ need,
                                                        ChangeList changes, uint8_t *__restrict__ tie_out,
                                                        uint8_t *__restrict__ watch, Landmarks marks,
                                                        uint32_t *__restrict__ list_done)
{
    if (gate && !*gate) return;
    if (!*marks.have) marks.skip = nullptr;
    if (count) np = *(volatile int32_t *)count;
    // a block past the list's end has nothing to count either (uniform per block)
    if ((int64_t)blockIdx.x * blockDim.x >= np) {
        list_used(count, list_done);
        return;
    }
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int32_t sgn = (player == 0) ? 1 : -1;   // score = sgn * key
    int32_t t_edges = 0, t_loads = 0, t_changed = 0, t_moves = 0;
    for (int64_t g0 = warp * 32; g0 < np; g0 += nwarps * 32) {
        // this lane's vertex
        const int64_t i = g0 + lane;
        int32_t v = -1, cur0 = -1, e0 = 0, deg = 0;
        if (i < np) {
            v = __ldcs(&plist[i]);
            if (gmask && !gmask[game_of[v]]) v = -1;
        }
        if (v >= 0) {
            cur0 = strat[v];
            e0 = __ldcs(&off[v]);
            deg = __ldcs(&off[v + 1]) - e0;
        }
        const int32_t kc0 = (cur0 >= 0) ? key[cur0] : 0;
        // successor lists end to end: base = exclusive prefix of the degrees
        int32_t incl = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(kAll, incl, o);
            if (lane >= o) incl += y;
        }
        const int32_t base = incl - deg;
        const int32_t total = __shfl_sync(kAll, incl, 31);
        // per vertex (held by its lane): running choice, moves, tie, exact
        ScoreArg run = {sgn * kc0, cur0};
        int32_t moves = 0;
        bool tie = false, exact = false;
        // kRounds rounds of 32 edges at a time: every round's successor ids,
        // then every round's keys, are loaded before any of them is used, so
        // a warp has up to 32 * kRounds gathers in flight
        constexpr int kRounds = 4;
        for (int32_t c0 = 0; c0 < total; c0 += 32 * kRounds) {
            int32_t us[kRounds], ks[kRounds], segs[kRounds];
#pragma unroll
            for (int r = 0; r < kRounds; r++) {
                const int32_t t = c0 + 32 * r + lane;
                // the lane whose segment holds edge t: the last lane with base <= t
                int32_t seg = 0;
#pragma unroll
                for (int step = 16; step; step >>= 1) {
                    const int32_t b = __shfl_sync(kAll, base, seg + step);
                    if (b <= t) seg += step;
                }
                const int32_t sb = __shfl_sync(kAll, base, seg), se0 = __shfl_sync(kAll, e0, seg);
                segs[r] = seg;
                us[r] = (t < total) ? __ldcs(&tgt[se0 + (t - sb)]) : -1;
            }
#pragma unroll
            for (int r = 0; r < kRounds; r++) ks[r] = (us[r] >= 0) ? __ldg(&key[us[r]]) : 0;
#pragma unroll
            for (int r = 0; r < kRounds; r++) {
                const int32_t c = c0 + 32 * r;
                if (c >= total) break;   // warp-uniform
                const int32_t seg = segs[r], u = us[r], k = ks[r];
                const bool valid = u >= 0;
                ScoreArg x = {valid ? sgn * k : INT_MIN, u};
                // segmented inclusive scan (segments are runs of equal seg)
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t osc = __shfl_up_sync(kAll, x.sc, o), ou = __shfl_up_sync(kAll, x.u, o);
                    const int32_t oseg = __shfl_up_sync(kAll, seg, o);
                    if (lane >= o && oseg == seg && osc >= x.sc) {
                        x.sc = osc;
                        x.u = ou;
                    }
                }
                // the running choice before this edge: the segment's carry, then
                // the inclusive value of the previous lane of the same segment
                const ScoreArg carry = {__shfl_sync(kAll, run.sc, seg), __shfl_sync(kAll, run.u, seg)};
                const int32_t psc = __shfl_up_sync(kAll, x.sc, 1), pu = __shfl_up_sync(kAll, x.u, 1);
                const int32_t pseg = __shfl_up_sync(kAll, seg, 1);
                const bool first = (lane == 0) || (pseg != seg);
                const ScoreArg excl = first ? carry : first_max(carry, ScoreArg{psc, pu});
                const int32_t sc = valid ? sgn * k : INT_MIN;
                const bool rec = valid && sc > excl.sc;
                const bool eqd = valid && sc == excl.sc && u != excl.u;
                const bool exd = eqd && !key_infinite(k);
                const unsigned recm = __ballot_sync(kAll, rec), eqm = __ballot_sync(kAll, eqd);
                const unsigned exm = __ballot_sync(kAll, exd);
                const ScoreArg last = first_max(carry, x);   // inclusive, with the carry
                // each vertex lane collects its segment's lanes of this round
                const int32_t lo = base - c, hi = base + deg - c;   // [lo, hi) of this round's lanes
                int32_t lastlane = 0;
                unsigned segm = 0;
                if (deg > 0 && hi > 0 && lo < 32) {
                    const int32_t a = lo > 0 ? lo : 0, b = hi < 32 ? hi : 32;
                    segm = (b - a == 32) ? kAll : (((1u << (b - a)) - 1u) << a);
                    lastlane = b - 1;
                }
                const int32_t lsc = __shfl_sync(kAll, last.sc, lastlane), lu = __shfl_sync(kAll, last.u, lastlane);
                if (segm) {
                    const unsigned rm = recm & segm;
                    moves += __popc(rm);
                    if (rm) {
                        const int top = 31 - __clz(rm);
                        tie = (top < 31) && ((eqm & segm) >> (top + 1)) != 0;
                    } else {
                        tie = tie || (eqm & segm) != 0;
                    }
                    exact = exact || (exm & segm) != 0;
                    run.sc = lsc;
                    run.u = lu;
                }
            }
        }
        int32_t cur = run.u;
        int32_t ext = sgn * run.sc;   // the best key (the owner's view), as a key
        if (v >= 0 && exact) {
            // the keys cannot order two distinct finite vertices: redo this
            // vertex with the exact comparisons, successor by successor
            cur = cur0;
            int32_t kc = kc0;
            moves = 0;
            ext = kc0;
            int32_t ext_v = cur0;
            tie = false;
            for (int32_t e = e0; e < e0 + deg; e++) {
                const int32_t uu = tgt[e], ku = key[uu];
                if ((player == 0) ? ku > ext : ku < ext) {
                    ext = ku;
                    ext_v = uu;
                    tie = false;
                } else if (ku == ext && uu != ext_v) {
                    tie = true;
                }
                int cmp;
                if (ku != kc) cmp = ku > kc ? 1 : -1;
                else if (uu == cur || key_infinite(ku)) cmp = 0;
                else cmp = compare_equal_keys(node, marks, st, rdeep, uu, cur, t_loads, err);
                if ((player == 0 && cmp > 0) || (player == 1 && cmp < 0)) {
                    cur = uu;
                    kc = ku;
                    moves++;
                }
            }
        }
        if (v >= 0) {
            t_edges += deg;
            const bool sticky = tie && ext != 0 && !key_infinite(ext);
            if (tie_out) {
                need[v] = 0;
                tie_out[v] = sticky ? 1 : 0;
                if (sticky && watch)   // the successors the tie rests on
                    for (int32_t e = e0; e < e0 + deg; e++) {
                        const int32_t uu = tgt[e];
                        if (key[uu] == ext) watch[uu] = 1;
                    }
            } else if (need) {
                need[v] = sticky ? 1 : 0;
            }
            if (moves) {   // strict improvements never return to cur0: cur != cur0
                strat[v] = cur;
                if (game_of) atomicAdd(&gcount[game_of[v]], (unsigned long long)moves);
                t_changed++;
                t_moves += moves;
            }
        }
        if (changes.list) {   // warp-collective (coalesced lanes)
            if (v >= 0 && moves) note_change(changes, v);
        }
    }
    typedef cub::BlockReduce<longlong4, kBlock> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    longlong4 mine = make_longlong4(t_edges, t_loads, t_changed, t_moves);
    longlong4 tot = Reduce(tmp).Reduce(mine, [](const longlong4 &x, const longlong4 &y) {
        return make_longlong4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
    });
    if (threadIdx.x == 0) {
        if (tot.x) atomicAdd(&stats[0], (unsigned long long)tot.x);
        if (tot.y) atomicAdd(&stats[1], (unsigned long long)tot.y);
        if (tot.z) atomicAdd(&stats[2], (unsigned long long)tot.z);
        if (tot.w) atomicAdd(&stats[3], (unsigned long long)tot.w);
    }
    list_used(count, list_done);
}

// Per-game accounting of the solve_si loop (main.cpp:20-55) run over a batch
// of games packed as one disjoint union.  Paths never leave their game, so a
// game's strategies and valuations evolve exactly as in a solo solve; a game
// whose loop has already converged only sees steps that change nothing.  The
// counters below therefore reproduce each game's solo iteration and
// evaluation counts.  state[g] = (evaluations, iterations, Odd's best response
// reached, game done); gcount[g] = strict improvements of game g in the last
// switch step (read and cleared here).
//   event 0: an evaluation      -> evaluations++ for games inside their best-response loop
//   event 1: after switch(Odd)  -> a game whose Odd made no improvement has its best response
//   event 2: before switch(Even)-> iterations++ for games not done
//   event 3: after switch(Even) -> a game whose Even made no improvement is done; the others
//                                  re-enter their best-response loop
__global__ void k_batch_account(int32_t games, int32_t event, int4 *__restrict__ state,
                                unsigned long long *__restrict__ gcount)
{
    int32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < games) batch_event(event, state[g], gcount[g]);
}

// Dense row of v: counts of the priorities on its strategy path (the reference
// layout, vals[v][p]); rows of infinite vertices are left zero.
__global__ void k_materialize(int32_t v0, int32_t count, int32_t d, const int32_t *__restrict__ st,
                              const PathNode *__restrict__ node, int32_t *__restrict__ rows,
                              uint32_t *__restrict__ err)
{
    int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    int32_t *row = rows + (int64_t)i * d;
    for (int32_t p = 0; p < d; p++) row[p] = 0;
    int32_t v = v0 + i;
    int32_t depth = st[v];
    int32_t x = v;
    for (int32_t k = 0; k < depth; k++) {
        if (x < 0) {
            atomicOr(err, DERR_WALK_CAP);
            return;
        }
        int2 q = *reinterpret_cast<const int2 *>(&node[x]);
        row[q.y] += 1;
        x = q.x;
    }
}

std::atomic<int> g_switch_blocks[2][kMaxCachedDevices];   // COUNT

template <bool COUNT>
int switch_grid()
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_switch<COUNT>, kBlock, 0);
    // one wave of resident blocks: the chunk claims balance the work, and
    // fewer blocks reduce fewer counters (switch steps 13.2 -> 12.6 ms per
    // 2^24 solve against four waves)
    int b = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
    return b > 0 ? b : 1;
}

}  // namespace

void launch_switch(cudaStream_t s, int32_t np, const int32_t *plist, int32_t player, const int32_t *off,
                   const int32_t *tgt, int32_t *strat, const int32_t *st, const int32_t *key, const PathNode *node,
                   const int32_t *rdeep, unsigned long long *stats, const int32_t *game_of, unsigned long long *gcount,
                   const int32_t *gmask, uint32_t *err, const int32_t *gate, uint8_t *need,
                   int32_t *list, int32_t *list_count, ChangeList changes, uint8_t *tie, uint8_t *watch,
                   Landmarks marks, bool warp, uint32_t *claim, const int8_t *owner, int32_t n_all, bool count_moves,
                   uint32_t *list_done, const MarkArgs *mark)
{
    const MarkArgs m = mark ? *mark : MarkArgs();
    if (np <= 0) {
        count_launch();
        k_need_none<<<mark ? kMarkBlocks : 1, kBlock, 0, s>>>(gate, stats, m);
        return;
    }
    // one wave of resident blocks
    const int blocks = count_moves ? per_device(g_switch_blocks[1], switch_grid<true>)
                                   : per_device(g_switch_blocks[0], switch_grid<false>);
    unsigned g = grid_for(np);
    g = g < (unsigned)blocks ? g : (unsigned)blocks;
    // only the vertices whose need flag is set (ChangeTrack)
    {
        count_launch();
        if (owner && !gmask) {
            // its own cap (four times the switch's one wave): the scan is one
            // pass of streaming loads per block
            unsigned gn = grid_for(ceil_div(n_all, kVec));
            gn = gn < 4u * (unsigned)blocks ? gn : 4u * (unsigned)blocks;
            k_need_ids<<<gn, kBlock, 0, s>>>(n_all, player, owner, need, gate, list, list_count,
                                             warp ? nullptr : claim, stats, m);
        } else {
            unsigned gn = grid_for(ceil_div(np, kNeedPer));
            gn = gn < (unsigned)blocks ? gn : (unsigned)blocks;
            k_need_list<<<gn, kBlock, 0, s>>>(np, plist, need, game_of, gmask, gate, list, list_count,
                                              warp ? nullptr : claim, stats, m);
        }
    }
    count_launch();
    if (warp)
        k_switch_warp<<<g, kBlock, 0, s>>>(np, list, list_count, player, off, tgt, strat, st, key, node, rdeep, stats,
                                           game_of, gcount, gmask, err, gate, need, changes, tie, watch, marks,
                                           list_done);
    else
        (count_moves ? k_switch<true> : k_switch<false>)<<<g, kBlock, 0, s>>>(
            np, list, list_count, player, off, tgt, strat, st, key, node, rdeep, stats, game_of, gcount, gmask, err,
            gate, need, changes, tie, watch, marks, claim, list_done);
}

void launch_batch_account(cudaStream_t s, int32_t games, int32_t event, int4 *state, unsigned long long *gcount)
{
    if (games <= 0) return;
    count_launch();
    k_batch_account<<<grid_for(games), kBlock, 0, s>>>(games, event, state, gcount);
}

void launch_materialize(cudaStream_t s, int32_t v0, int32_t count, int32_t d, const int32_t *st,
                        const PathNode *node, int32_t *rows, uint32_t *err)
{
    if (count > 0) {
        count_launch();
        k_materialize<<<grid_for(count, 128), 128, 0, s>>>(v0, count, d, st, node, rows, err);
    }
}

}  // namespace psi
