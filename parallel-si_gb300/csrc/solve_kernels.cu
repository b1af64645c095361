// solve_kernels.cu -- solve_si (main.cpp:20-55) of one game in one persistent
// kernel on sm_103a, for games whose state stays in L2.
//
// What bounds such a solve is latency: a step of the loop touches a few MB,
// but as a sequence of launches (about 18 per step, each with its own ramp)
// it took 80 us whatever the size.  Here the whole loop is one cooperative
// launch; a step is two phases with a grid barrier after each, three when
// Even moves, and every evaluation is a full one.
//
//  - Jump phase.  Every vertex v has a record jump[v] = (target, top priority
//    of the window from v up to the target, how many of the window's vertices
//    carry it, the window's length), one 16-byte word that is read and
//    written whole.  It starts as (successor, own priority, 1, 1).  v's
//    thread reads its target's record, appends that window to its own and
//    stores the result, until the target is the sink (the record is then v's
//    summary) or a vertex known to be infinite.  All threads do so at once
//    without barriers: whichever state of the target's record a reader
//    finds, it is a window of the same path.  So a vertex at depth d is done
//    after about log2 d reads, where a walk would take d (all vertices start
//    together here: no ancestor is finished yet).  A window of n vertices or
//    a return to a vertex seen before (Brent's marker) means that the target
//    lies on a cycle; its top priority is collected along the records from
//    there on, until they return to it or cover n vertices.
//    A vertex makes at most kJumps reads per pass; should one be left, the
//    pass is repeated (its windows are kept, so a few passes reach any depth).
//  - Switch phase of one player.  mark_solved and the all-switches step touch
//    different words, so they share a phase, and each vertex's thread also
//    writes the next evaluation's initial records, into the other of two
//    buffers (comparisons still read the current ones).  The paths that
//    comparisons walk change at the start of the jump phase.
//  - Comparisons that walk far (equal summaries, paths that meet late) hold
//    up a whole phase.  A vertex whose walks pass their budget of steps is left
//    over; only if there are any, all threads write landmark records
//    (device_common.cuh) and those vertices are done again with them.
//
// A thread owns the same vertices in every phase (plist[tid], plist[tid +
// threads], ...), so what a vertex's phases start from -- its id, CSR range,
// choice and first successors -- stays in shared memory, 32 bytes
// per vertex; the first dependent load of a phase is then a key or a record.
//
// Every vertex of the player is examined in every switch phase: with all keys
// in L2 that costs less than tracking which have changed.  What would cost is
// to repeat the walks of ties that nothing has touched, so a record also says
// whether a strategy on the vertex's path has changed since the last
// evaluation (Odd's last examination) and since Even's last one.
#include <climits>
#include <cooperative_groups.h>

#include "compare.cuh"
#include "device_common.cuh"
#include "jump.cuh"
#include "kernels.h"
#include "solver.h"
#include "spread.h"

namespace cg = cooperative_groups;

namespace psi {

namespace {

// Steps of comparison walks per vertex before it is left over: a step is a
// dependent read from L2, the second round costs the landmark records of all
// vertices and two barriers, and a warp's lanes walk together.  Solve in us
// with 16, 64, 256, 1,024, 4,096 steps where a thread has more than two vertices:
// 3640, 3622, 3448, 3248, 3250 (10^6), 6210, 5212, 5160, 5090, 4830 (9*10^5, 100
// priorities), 3737, 3339, 2528, 2527, 2515 (10^6, long paths); with 256, 512, 1,024,
// 4,096 where not: 669, 654, 653, 653 (10^5), 1600, 1542, 1433, 1424 (2^18, 8
// priorities).  More is the same: few ties are that far apart.
constexpr int32_t kWalkBudget = 4096;

// Even's view of finite u against finite w (distinct, equal keys; -1: the sink).
__device__ __forceinline__ int compare_tied(const int4 *jump, const int2 *path, const int4 *skip, int32_t u, int32_t w,
                                         int32_t &loads, int32_t budget, uint32_t *err)
{
    const int4 ru = jump[u];
    const int4 rw = (w >= 0) ? jump[w] : make_int4(kSink, -1, 0, 0);   // w's length: 0
    if (ru.y != rw.y) return ru.y > rw.y ? decide(ru.y, ru.z, 0) : decide(rw.y, 0, rw.z);
    if (ru.z != rw.z) return decide(ru.y, ru.z, rw.z);
    return skip ? lean_compare<true>(path, skip, u, ru.w & kLen, w, rw.w & kLen, loads, budget, err)
                : lean_compare<false>(path, skip, u, ru.w & kLen, w, rw.w & kLen, loads, budget, err);
}

// A vertex's choice word: (choice + 1) << kChoiceShift and bits.  Solved; its
// path touched since Even's last examination, since the last evaluation; the
// infinity its record ended in; its choice changed since the evaluation.  With
// them a switch phase reads no record but those it compares: a phase is bound
// by L2 sectors once a thread has several vertices (n = 7*10^5: own records,
// paths and priorities were 0.3 of 0.85 million per 155,648 vertices; 62 -> 51
// us per evaluation).
constexpr int32_t kSolved = 1, kTouched = 2, kFresh = 4, kNeg = 8, kPos = 16, kChanged = 32;
constexpr int kChoiceShift = 6;
constexpr int32_t kChoiceBits = (1 << kChoiceShift) - 1;
__device__ __forceinline__ int32_t chosen(int32_t t) { return (t >> kChoiceShift) - 1; }
constexpr int kFirst = 5;       // successors kept per vertex
constexpr int kWords = 3 + kFirst;
constexpr int32_t kIdBits = 20, kManySuccessors = (1 << (32 - kIdBits)) - 1;
constexpr int kSmallBytes = 227 * 1024;   // all a block can have
// Games below this size are solved there.  Solve in us, k_solve -> here: n = 100
// 96 -> 62, 300 145 -> 91, 1,024 189 -> 152, 1,537 295 -> 263, 2,048 235 -> 241,
// 4,000 308 -> 454 (one SM's issue slots).
constexpr int32_t kSmall = 2000;
constexpr int kMaxWaves = 32;   // vertices per thread (a bit mask)
constexpr int kMaxCached = 7;   // vertices per thread kept (224 KB); further ones are read anew
constexpr int kSharedBytes = 4 * kWords * kSolveThreads * kMaxCached;   // 224 KB

__global__ void __launch_bounds__(kSolveThreads, 1) k_solve(SolveArgs a)
{
    extern __shared__ int32_t own[];   // [wave][word][thread]
    const int32_t n = a.n;
    const int32_t tid = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    const int32_t nth = (int32_t)(gridDim.x * blockDim.x);
    // Barrier with two votes: whether any thread passed true.  Phase k uses the
    // words k % 3, which thread 0 clears in phase k - 1, when everyone has
    // read their last use (phase k - 3); the count goes on from launch to
    // launch (kept_phase).  err: the error bits thread 0 saw on its way into the barrier
    // (the same for all threads, as the loop's control has to be).
    uint32_t phase = a.sync->phase, err = 0;
    bool voted = false, voted2 = false;
    auto barrier = [&](bool mine, bool mine2) {
        const uint32_t k = phase % 3, k1 = (phase + 1) % 3;
        phase++;
        if (tid == 0) {
            a.sync->vote[k1] = a.sync->vote2[k1] = 0;
            a.sync->errs[k] = *(volatile uint32_t *)&a.sync->err;
        }
        if (__syncthreads_or(mine) && threadIdx.x == 0) a.sync->vote[k] = 1;
        if (__syncthreads_or(mine2) && threadIdx.x == 0) a.sync->vote2[k] = 1;
        cg::this_grid().sync();
        err = __ldcg(&a.sync->errs[k]);
        voted = __ldcg(&a.sync->vote[k]) != 0;
        voted2 = __ldcg(&a.sync->vote2[k]) != 0;
    };
    // the thread's vertex in wave w (vertex i of plist): its words
    struct Own {
        int32_t v, e0, deg, t;   // t: choice word (kSolved ...)
    };
    auto word = [&](int32_t w, int k) -> int32_t & { return own[(w * kWords + k) * (int32_t)blockDim.x + threadIdx.x]; };
    auto get = [&](int32_t w, int32_t i) -> Own {
        if (w < kMaxCached) {
            const uint32_t x = (uint32_t)word(w, 0);
            Own o{(int32_t)(x & ((1u << kIdBits) - 1)), word(w, 1), (int32_t)(x >> kIdBits), word(w, 2)};
            if (o.deg == kManySuccessors) o.deg = a.off[o.v + 1] - o.e0;
            return o;
        }
        const int32_t v = a.plist[i], e0 = a.off[v];
        return Own{v, e0, a.off[v + 1] - e0, (a.strat[v] + 1) << kChoiceShift | a.solved[v]};
    };
    auto put = [&](int32_t w, int32_t v, int32_t t) {
        if (w < kMaxCached) {
            word(w, 2) = t;
        } else {
            a.strat[v] = chosen(t);
            a.solved[v] = (uint8_t)(t & kChoiceBits);   // (all the bits until the end)
        }
    };
    auto successor = [&](int32_t w, int32_t e0, int32_t j) -> int32_t {
        return (w < kMaxCached && j < kFirst) ? word(w, 3 + j) : a.tgt[e0 + j];
    };
    // the records of the current evaluation, and those that switch phases prepare
    int4 *jump = a.jump[0], *jump_next = a.jump[1];
    int2 *path = a.path;   // the current evaluation's (choice, priority)
    auto prepare = [&](int4 *j, const Own &o) {
        const bool fresh = o.t & kChanged;
        const int32_t w = 1 | (fresh ? kNew : 0) | (fresh || (o.t & kTouched) ? kNewEven : 0);
        store_whole(&j[o.v], (o.t & kSolved) ? make_int4((o.t & kPos) ? kPosInf : kNegInf, 0, 0, 0)
                                             : make_int4(chosen(o.t), a.pri[o.v], 1, w));
    };
    // The player's choice at a vertex (k_switch's rule): the successors in CSR
    // order, moving only on a strict improvement; that is the first best one,
    // the present choice counting first.  Keys decide; among distinct finite
    // vertices that share the best key, exact comparisons.  The present choice
    // was a best one at the last examination, so where it and the other path
    // are as they were then (newbit; solved vertices' records do not tell), it
    // stands.  False if the walks passed the budget.
    auto choose = [&](int32_t w, const Own &o, int32_t player, const int4 *skip, int32_t budget,
                      int32_t &choice) -> bool {
        const int32_t cur0 = choice;
        int32_t cur = cur0, kc = (cur0 >= 0) ? a.key[cur0] : 0;
        bool tie = false;
        uint32_t ties = 0;   // which of the first 32 successors share the best key with cur
        for (int32_t b = 0; b < o.deg; b += kFirst) {
            int32_t us[kFirst], ks[kFirst];
#pragma unroll
            for (int j = 0; j < kFirst; j++) us[j] = (b + j < o.deg) ? successor(w, o.e0, b + j) : -1;
#pragma unroll
            for (int j = 0; j < kFirst; j++) ks[j] = (us[j] >= 0) ? a.key[us[j]] : 0;
#pragma unroll
            for (int j = 0; j < kFirst; j++) {
                if (us[j] < 0) continue;
                if ((player == 0) ? ks[j] > kc : ks[j] < kc) {
                    cur = us[j];
                    kc = ks[j];
                    tie = false;
                    ties = 0;
                } else if (ks[j] == kc && us[j] != cur) {
                    tie = true;
                    if (b + j < 32) ties |= 1u << (b + j);
                }
            }
        }
        if (tie && !key_infinite(kc)) {
            const int32_t newbit = player == 0 ? kNewEven : kNew;
            const bool settled = cur == cur0 && !(o.t & (kSolved | (player == 0 ? kTouched : kFresh)));
            int32_t loads = 0;
            for (int32_t j = 0;; j++) {
                if (next_tied(ties, j) >= o.deg) break;
                const int32_t u = successor(w, o.e0, j);
                if (u == cur || (j >= 32 && a.key[u] != kc)) continue;
                if (settled && cur == cur0 && !(jump[u].w & newbit)) continue;
                const int c = compare_tied(jump, path, skip, u, cur, loads, budget, &a.sync->err);
                if (c == kUndecided) return false;
                if ((player == 0) ? c > 0 : c < 0) cur = u;
            }
        }
        choice = cur;
        return true;
    };

    // init_strat (cpu_parity.cpp:276-286)
    if (tid == 0) *a.ucount = 0;
    for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
        Own o;
        o.v = a.plist[i];
        o.e0 = a.off[o.v];
        o.deg = a.off[o.v + 1] - o.e0;
        o.t = (i < a.n_even ? 0 : (a.tgt[o.e0] + 1) << kChoiceShift) | kTouched | kChanged;
        if (w < kMaxCached) {
            word(w, 0) = (int32_t)((uint32_t)o.v | (uint32_t)min(o.deg, kManySuccessors) << kIdBits);
            word(w, 1) = o.e0;
#pragma unroll
            for (int j = 0; j < kFirst; j++) word(w, 3 + j) = j < o.deg ? a.tgt[o.e0 + j] : 0;
        }
        put(w, o.v, o.t);
        path[o.v].y = a.pri[o.v];
        prepare(jump, o);
    }
    barrier(false, false);

    int32_t iters = 0, brs = 0, stop = GraphCtl::kRunning;
    while (stop == GraphCtl::kRunning) {
        // evaluation
        voted = true;
        for (int pass = 0; voted; pass++) {
            if (pass == kMaxPasses) {   // cannot happen: windows grow at least kJumps-fold per pass
                if (tid == 0) atomicOr(&a.sync->err, DERR_WALK_CAP);
                break;
            }
            bool left = false;
            for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
                const Own o = get(w, i);
                int32_t t1 = o.t & ~kChanged;
                if (pass == 0 && (o.t & kChanged)) path[o.v].x = chosen(o.t);   // (no phase that reads paths is on)
                if (o.t & kSolved) {   // its record and key stay
                    if (t1 != o.t) put(w, o.v, t1);
                    continue;
                }
                int4 r = load_whole(&jump[o.v]);
                // in the first pass the target is the choice: its record arrives with the own one
                const int32_t t = pass ? r.x : chosen(o.t);
                int4 q = r;
                if (t >= 0) q = load_whole(&jump[t]);
                if (!jump_pass<true>(jump, n, o.v, r, q)) {
                    left = true;
                    if (t1 != o.t) put(w, o.v, t1);
                    continue;
                }
                t1 &= ~(kFresh | kNeg | kPos);
                if (r.w & kNew) t1 |= kFresh | kTouched;
                if (r.x != kSink) t1 |= r.x == kPosInf ? kPos : kNeg;
                if (t1 != o.t) put(w, o.v, t1);
                a.key[o.v] = r.x == kSink ? finite_key(r.y, r.z) : (r.x == kPosInf ? KEY_POS_INF : KEY_NEG_INF);
            }
            barrier(left, false);
        }
        brs++;
        if (tid == 0 && a.inject_at > 0 && brs == a.inject_at) atomicOr(&a.sync->err, a.inject_bits);
        // mark_solved and switch: Odd, and Even when Odd made no move
        int32_t player = 1;
        bool go;
        for (;; player = 0) {
            const int32_t code = player == 0 ? kPos : kNeg;
            uint32_t over = 0;   // the thread's vertices that are left over
            bool moved = false;
            for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
                Own o = get(w, i);
                const int32_t t0 = o.t;
                if (o.t & code) o.t |= kSolved;
                if ((i < a.n_even) == (player == 0)) {
                    int32_t choice = chosen(o.t);
                    if (!choose(w, o, player, nullptr, kWalkBudget, choice)) {
                        over |= 1u << w;
                    } else if (choice != chosen(o.t)) {
                        o.t = (choice + 1) << kChoiceShift | (o.t & kChoiceBits) | kChanged;
                        moved = true;
                    }
                }
                if (player == 0) o.t &= ~kTouched;   // (what changed now is new to the next examination)
                if (o.t != t0) put(w, o.v, o.t);
                prepare(jump_next, o);
            }
            barrier(moved, over != 0);
            go = voted;
            if (voted2) {
                for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
                    const int32_t v = get(w, i).v;
                    const int4 r = jump[v];
                    if (r.x != kSink) continue;
                    Top2 seg = {-1, 0, -1, 0};
                    int32_t anc = v;
                    const int32_t d = r.w & kLen;
                    for (int32_t j = d - skip_landmark_depth(d); j > 0; j--) {
                        const int2 q = path[anc];
                        top2_add(seg, q.y);
                        anc = q.x;
                    }
                    a.skip[v] = skip_pack(anc, seg);
                }
                barrier(false, false);
                moved = false;
                for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
                    if (!(over >> w & 1)) continue;
                    Own o = get(w, i);
                    int32_t choice = chosen(o.t);
                    if (player == 0) o.t |= kTouched;   // (cleared above; the examination is not over)
                    choose(w, o, player, a.skip, INT_MAX, choice);
                    if (player == 0) o.t &= ~kTouched;
                    if (choice != chosen(o.t)) {
                        moved = true;
                        o.t = (choice + 1) << kChoiceShift | (o.t & kChoiceBits) | kChanged;
                        put(w, o.v, o.t);
                        prepare(jump_next, o);
                    }
                }
                barrier(moved, false);
                go |= voted;
            }
            if (go || player == 0) break;
        }
        // the loop's control, as k_ctl_even (solver_graph.cu)
        if (err) {
            stop = GraphCtl::kDeviceError;
        } else if (player == 0) {
            iters++;
            if (!go) stop = GraphCtl::kConverged;
        }
        if (stop == GraphCtl::kRunning && a.max_evals > 0 && brs >= a.max_evals) stop = GraphCtl::kEvalCap;
        if (stop == GraphCtl::kRunning && brs >= a.guard) stop = GraphCtl::kRunaway;
        if (stop != GraphCtl::kRunning) break;
        if (player == 0 && a.reset) {   // cpu_parity.cpp:300-307
            for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
                if (i < a.n_even) continue;
                Own o = get(w, i);
                const int32_t t = successor(w, o.e0, 0);
                if (t != chosen(o.t)) {
                    o.t = (t + 1) << kChoiceShift | (o.t & kChoiceBits) | kChanged;
                    put(w, o.v, o.t);
                    prepare(jump_next, o);
                }
            }
            barrier(false, false);
        }
        int4 *j = jump;
        jump = jump_next;
        jump_next = j;
    }

    // the last evaluation as a solver leaves it (device_common.cuh); the
    // landmark records are unknown, so later comparisons step
    for (int32_t w = 0, i = tid; i < n; w++, i += nth) {
        const Own o = get(w, i);
        const int32_t v = o.v;
        const int4 r = jump[v];
        const int2 q = path[v];
        const bool fin = r.x == kSink;
        if (w < kMaxCached) a.strat[v] = chosen(o.t);
        a.solved[v] = o.t & kSolved;
        const int32_t d = r.w & kLen;
        if (!fin && !(o.t & kSolved)) a.ulist[atomicAdd(a.ucount, 1)] = v;   // (none once the loop has converged)
        a.st[v] = fin ? d : (r.x == kPosInf ? ST_POS_INF : ST_NEG_INF);
        if (fin && d >= kDeepPath) a.rdeep[v] = r.z;
        *reinterpret_cast<int4 *>(&a.node[v]) =
            fin ? make_int4(q.x, q.y, r.y, path_word(d, r.z))
                : make_int4(q.x, q.y, r.x == kPosInf ? RM_POS_INF : RM_NEG_INF, 0);
    }
    if (tid == 0) {
        a.ctl->iters = iters;
        a.ctl->brs = brs;
        a.ctl->stop = stop;
        a.ctl->mfrom[0] = a.ctl->mfrom[1] = 0;
        a.ctl->lm_have = a.ctl->lm_far = 0;
        *a.err = *(volatile uint32_t *)&a.sync->err;
        a.sync->err = 0;
        a.sync->phase = kept_phase(phase);
    }
}

// ---- the smallest games: one block, everything a phase reads in shared memory
// (its latency is a tenth of L2's, a block barrier's a fortieth of a grid's).
// Evaluations are plain pointer doubling between two buffers: in round r every
// record is a window of 2^r vertices or finished, and once 2^r >= n what is
// left is on or into a cycle that its target's window covers.  Vertices in id
// order, v = thread, thread + threads, ...

// low bits of the choice word: kSolved, kTouched, and the owner
constexpr int32_t kOddBit = 4;

struct SmallLayout {   // byte offsets in shared memory
    int32_t jump[2], path, key, off, choice, tgt, total;
};
__host__ __device__ inline SmallLayout small_layout(int32_t n, int64_t m)
{
    SmallLayout l;
    int32_t at = 0;
    auto take = [&](int64_t bytes) {
        const int32_t x = at;
        at += (int32_t)((bytes + 15) & ~15ll);
        return x;
    };
    l.jump[0] = take(16ll * n);
    l.jump[1] = take(16ll * n);
    l.path = take(8ll * n);
    l.key = take(4ll * n);
    l.off = take(4ll * (n + 1));
    l.choice = take(4ll * n);
    l.tgt = at;
    l.total = at;
    if (4 * m + at <= kSmallBytes) l.total = at + (int32_t)(4 * m);   // the successors too, if they fit
    return l;
}

__global__ void __launch_bounds__(kSolveThreads, 1) k_solve_small(SolveArgs a)
{
    extern __shared__ __align__(16) unsigned char mem[];
    const int32_t n = a.n, tid = threadIdx.x, nth = blockDim.x;
    const SmallLayout l = small_layout(n, a.m);
    int4 *jump[2] = {reinterpret_cast<int4 *>(mem + l.jump[0]), reinterpret_cast<int4 *>(mem + l.jump[1])};
    int2 *path = reinterpret_cast<int2 *>(mem + l.path);
    int32_t *key = reinterpret_cast<int32_t *>(mem + l.key), *off = reinterpret_cast<int32_t *>(mem + l.off);
    int32_t *choice = reinterpret_cast<int32_t *>(mem + l.choice);
    const bool held = l.total > l.tgt;
    int32_t *held_tgt = reinterpret_cast<int32_t *>(mem + l.tgt);
    const int32_t *tgt = held ? held_tgt : a.tgt;
    int rounds = 0;
    while ((1 << rounds) < n) rounds++;

    for (int32_t v = tid; v <= n; v += nth) off[v] = a.off[v];
    if (held)
        for (int32_t e = tid; e < (int32_t)a.m; e += nth) held_tgt[e] = a.tgt[e];
    for (int32_t v = tid; v < n; v += nth) {   // init_strat (cpu_parity.cpp:276-286)
        const bool odd = a.owner[v] != 0;
        const int32_t t = odd ? a.tgt[a.off[v]] : kSink;
        choice[v] = (t + 1) * 8 + (odd ? kOddBit : 0) + kTouched;
        path[v] = make_int2(t, a.pri[v]);
    }
    if (tid == 0) *a.ucount = 0;
    bool all_new = true;   // every vertex counts as changed in the first evaluation
    int32_t iters = 0, brs = 0, stop = GraphCtl::kRunning;
    int4 *in = jump[0];
    while (stop == GraphCtl::kRunning) {
        // evaluation; bit w: the thread's vertex v = tid + w nth
        in = jump[0];
        int4 *out = jump[1];
        uint32_t active = 0, fresh_done = 0;   // unfinished; finished in the last round (one buffer has it)
        for (int32_t w = 0, v = tid; v < n; w++, v += nth) {
            const int32_t c = choice[v], t = (c >> 3) - 1;
            int2 p = path[v];
            const bool fresh = all_new || p.x != t;
            p.x = t;
            path[v] = p;
            const int32_t wd = 1 | (fresh ? kNew | kNewEven : 0) | ((c & kTouched) ? kNewEven : 0);
            int4 x = make_int4(t, p.y, 1, wd);
            if (c & kSolved) x = make_int4(key[v] == KEY_POS_INF ? kPosInf : kNegInf, 0, 0, 0);
            else if (t == kSink) key[v] = finite_key(p.y, 1);
            if (fresh) choice[v] = c | kTouched;
            in[v] = x;
            if (x.x >= 0) active |= 1u << w;
            else out[v] = x;
        }
        all_new = false;
        __syncthreads();
        for (int r = 0;; r++) {
            uint32_t done = 0;
            for (uint32_t todo = active | fresh_done; todo; todo &= todo - 1) {
                const int w = __ffs(todo) - 1;
                const int32_t v = tid + w * nth;
                int4 x = in[v];
                if (active >> w & 1) {
                    const int4 q = in[x.x];
                    int32_t code = q.x <= kNegInf ? q.x : 0;
                    if (q.x >= 0 && r == rounds) code = (q.y & 1) ? kNegInf : kPosInf;
                    if (code) {
                        x = make_int4(code, 0, 0, 0);
                        key[v] = code == kPosInf ? KEY_POS_INF : KEY_NEG_INF;
                    } else {
                        top1_merge(x.y, x.z, q.y, q.z);
                        x.z = min(x.z, kMaxLen);
                        x.w = min((x.w & kLen) + (q.w & kLen), kMaxLen) | (x.w & kNewEven) | ((x.w | q.w) & kNew);
                        x.x = q.x;
                        if (x.x == kSink) {
                            key[v] = finite_key(x.y, x.z);
                            if (x.w & kNew) {
                                x.w |= kNewEven;
                                choice[v] |= kTouched;
                            }
                        }
                    }
                    if (x.x < 0) done |= 1u << w;
                }
                out[v] = x;
            }
            active &= ~done;
            fresh_done = done;
            int4 *t = in;
            in = out;
            out = t;
            if (!__syncthreads_or(active != 0)) break;
        }
        brs++;
        if (tid == 0 && a.inject_at > 0 && brs == a.inject_at) atomicOr(&a.sync->err, a.inject_bits);
        // mark_solved and switch: Odd, and Even when Odd made no move
        bool go;
        int32_t player = 1;
        for (;; player = 0) {
            const int32_t code = player == 0 ? kPosInf : kNegInf, newbit = player == 0 ? kNewEven : kNew;
            bool moved = false;
            for (int32_t v = tid; v < n; v += nth) {
                int32_t c = choice[v];
                const int4 r = in[v];
                if (r.x == code) c |= kSolved;
                if (player == 0) c &= ~kTouched;
                if (((c & kOddBit) != 0) == (player == 1)) {
                    // the first best successor, the present one counting first (as k_solve)
                    const int32_t e0 = off[v], e1 = off[v + 1], cur0 = (c >> 3) - 1;
                    int32_t cur = cur0, kc = cur0 >= 0 ? key[cur0] : 0;
                    bool tie = false;
                    constexpr int kAt = 4;
                    for (int32_t eb = e0; eb < e1; eb += kAt) {
                        int32_t us[kAt], ks[kAt];
#pragma unroll
                        for (int j = 0; j < kAt; j++) us[j] = tgt[min(eb + j, e1 - 1)];   // (the last one again: no tie)
#pragma unroll
                        for (int j = 0; j < kAt; j++) ks[j] = key[us[j]];
#pragma unroll
                        for (int j = 0; j < kAt; j++) {
                            if ((player == 0) ? ks[j] > kc : ks[j] < kc) {
                                cur = us[j];
                                kc = ks[j];
                                tie = false;
                            } else if (ks[j] == kc && us[j] != cur) {
                                tie = true;
                            }
                        }
                    }
                    if (tie && !key_infinite(kc)) {
                        const bool settled = cur == cur0 && !(c & kSolved) && !(r.w & newbit);
                        int32_t loads = 0;
                        bool after = cur == cur0;
                        for (int32_t e = e0; e < e1; e++) {
                            const int32_t u = tgt[e];
                            if (!after) {
                                after = u == cur;
                                continue;
                            }
                            if (u == cur || key[u] != kc) continue;
                            if (settled && cur == cur0 && !(in[u].w & newbit)) continue;
                            const int x = compare_tied(in, path, nullptr, u, cur, loads, INT_MAX, &a.sync->err);
                            if ((player == 0) ? x > 0 : x < 0) cur = u;
                        }
                    }
                    if (cur != cur0) {
                        moved = true;
                        c = (cur + 1) * 8 + (c & 7);
                    }
                }
                choice[v] = c;
            }
            go = __syncthreads_or(moved);
            if (go || player == 0) break;
        }
        // the loop's control, as k_ctl_even (solver_graph.cu)
        if (__syncthreads_or(tid == 0 && *(volatile uint32_t *)&a.sync->err != 0)) {
            stop = GraphCtl::kDeviceError;
        } else if (player == 0) {
            iters++;
            if (!go) stop = GraphCtl::kConverged;
        }
        if (stop == GraphCtl::kRunning && a.max_evals > 0 && brs >= a.max_evals) stop = GraphCtl::kEvalCap;
        if (stop == GraphCtl::kRunning && brs >= a.guard) stop = GraphCtl::kRunaway;
        if (stop == GraphCtl::kRunning && player == 0 && a.reset)   // cpu_parity.cpp:300-307
            for (int32_t v = tid; v < n; v += nth) {
                const int32_t c = choice[v];
                if (c & kOddBit) choice[v] = (tgt[off[v]] + 1) * 8 + (c & 7);
            }
    }

    for (int32_t v = tid; v < n; v += nth) {   // as k_solve leaves it
        const int4 r = in[v];
        const int2 q = path[v];
        const int32_t c = choice[v];
        const bool fin = r.x == kSink;
        a.strat[v] = (c >> 3) - 1;
        a.solved[v] = c & kSolved;
        a.key[v] = key[v];
        if (!fin && !(c & kSolved)) a.ulist[atomicAdd(a.ucount, 1)] = v;
        a.st[v] = fin ? r.w & kLen : (r.x == kPosInf ? ST_POS_INF : ST_NEG_INF);
        *reinterpret_cast<int4 *>(&a.node[v]) =
            fin ? make_int4(q.x, q.y, r.y, path_word(r.w & kLen, r.z))
                : make_int4(q.x, q.y, r.x == kPosInf ? RM_POS_INF : RM_NEG_INF, 0);
    }
    if (tid == 0) {
        a.ctl->iters = iters;
        a.ctl->brs = brs;
        a.ctl->stop = stop;
        a.ctl->mfrom[0] = a.ctl->mfrom[1] = 0;
        a.ctl->lm_have = a.ctl->lm_far = 0;
        *a.err = *(volatile uint32_t *)&a.sync->err;
        a.sync->err = 0;
    }
}

// ---- one full evaluation by the same jumps, for the step-by-step calls and the
// served arena: init_records, jumps and results in one cooperative launch where
// the walks (root_kernels.cu) take three and each walk its path's length (with
// every vertex in flight at once no ancestor is finished yet).  It leaves what
// they leave: status, path records, keys, landmark records, the unreached
// list, need flags; and does what launch_patch_begin does before them.
__global__ void __launch_bounds__(kSolveThreads, 1) k_eval_jump(EvalArgs a, EvalGates *g, int32_t *quiet)
{
    const int32_t n = a.n, lane = threadIdx.x & 31;
    const int32_t tid = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x), nth = (int32_t)(gridDim.x * blockDim.x);
    SolveSync *sync = a.sync;
    uint32_t phase = sync->phase;
    auto barrier = [&](bool mine) -> bool {   // with a vote, as k_solve's
        const uint32_t k = phase % 3, k1 = (phase + 1) % 3;
        phase++;
        if (tid == 0) sync->vote[k1] = sync->vote2[k1] = 0;
        if (__syncthreads_or(mine) && threadIdx.x == 0) sync->vote[k] = 1;
        cg::this_grid().sync();
        return __ldcg(&sync->vote[k]) != 0;
    };
    if (tid == 0) {
        const bool fresh = *quiet > 0;
        if (fresh) --*quiet;
        g->lm_have = !fresh && want_landmarks(g, a.sw, n);
        g->lm_far = 0;
        g->ccount = g->csnap = 0;
        g->patch = 0;
        g->eval = 1;
        g->mfrom[0] = g->mfrom[1] = 0;
        *a.ucount = 0;
    }
    for (int32_t v = tid; v < n; v += nth) {
        const int32_t t = a.strat[v], p = a.pri[v];
        const bool solved = a.solved[v];
        const int32_t st = solved ? a.st[v] : 0;
        *reinterpret_cast<int4 *>(&a.node[v]) =
            make_int4(solved ? -1 : t, p, !solved ? RM_UNKNOWN : (st == ST_POS_INF ? RM_POS_INF : RM_NEG_INF), 0);
        store_whole(&a.ja[v], solved ? make_int4(st == ST_POS_INF ? kPosInf : kNegInf, 0, 0, 0) : make_int4(t, p, 1, 1));
        if (a.track.tie && a.track.tie[v]) a.track.need[v] = 1;
    }
    bool more = true;
    barrier(false);
    const bool marks = __ldcg(&g->lm_have) != 0;
    for (int pass = 0; more; pass++) {
        if (pass == kMaxPasses) {   // cannot happen: windows grow at least kJumps-fold per pass
            if (tid == 0) atomicOr(a.err, DERR_WALK_CAP);
            break;
        }
        bool left = false;
        for (int32_t b = tid & ~31; b < n; b += nth) {   // whole warps: appends and flags are collective
            const int32_t v = b + lane;
            bool changed = false, infinite = false;
            if (v < n && !a.solved[v]) {
                int4 r = load_whole(&a.ja[v]);
                // in later passes, what is finished has been dealt with
                if (pass == 0 || r.x >= 0) {
                    int4 q = r;
                    if (r.x >= 0) q = load_whole(&a.ja[r.x]);
                    if (jump_pass<true>(a.ja, n, v, r, q)) {
                        const bool fin = r.x == kSink;
                        const int32_t d = r.w & kLen;
                        const int32_t k =
                            fin ? finite_key(r.y, r.z) : (r.x == kPosInf ? KEY_POS_INF : KEY_NEG_INF);
                        a.st[v] = fin ? d : (r.x == kPosInf ? ST_POS_INF : ST_NEG_INF);
                        if (fin && d >= kDeepPath) a.rdeep[v] = r.z;
                        *reinterpret_cast<int2 *>(&a.node[v].rmax) =
                            fin ? make_int2(r.y, path_word(d, r.z))
                                : make_int2(r.x == kPosInf ? RM_POS_INF : RM_NEG_INF, 0);
                        if (fin && marks) {
                            Top2 seg = {-1, 0, -1, 0};
                            int32_t anc = v;
                            for (int32_t j = d - skip_landmark_depth(d); j > 0; j--) {
                                const int2 q = *reinterpret_cast<const int2 *>(&a.node[anc]);
                                top2_add(seg, q.y);
                                anc = q.x;
                            }
                            a.skip[v] = skip_pack(anc, seg);
                        }
                        infinite = !fin;
                        changed = a.key[v] != k;
                        if (changed) a.key[v] = k;
                    } else {
                        left = true;
                    }
                }
            }
            const int32_t p = warp_reserve(infinite, a.ucount);
            if (infinite) a.ulist[p] = v;
            flag_in_neighbours(a.track, changed, v);
        }
        more = barrier(left);
    }
    if (tid == 0) sync->phase = kept_phase(phase);
}

std::atomic<int> g_sms[kMaxCachedDevices];

}  // namespace

static int device_sms()
{
    return per_device(g_sms, [] {
        int dev = 0, x = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&x, cudaDevAttrMultiProcessorCount, dev);
        return x > 0 ? x : 1;
    });
}

int launch_eval_jump(cudaStream_t s, const EvalArgs &a, EvalGates *g, int32_t *quiet)
{
    const int sms = device_sms(), threads = spread_threads(a.n, sms, kSolveThreads);
    const int64_t need = ceil_div(a.n, threads);
    const int grid = (int)(need < 1 ? 1 : (need < sms ? need : sms));
    void *args[] = {(void *)&a, (void *)&g, (void *)&quiet};
    count_launch();
    return (int)cudaLaunchCooperativeKernel((const void *)k_eval_jump, dim3(grid), dim3(threads), args, 0, s);
}

// A switch phase reads every successor of the player's vertices, a thread its
// own lists, so neighbouring reads of a list hit L1 only while the lists of a
// block's 1,024 threads fit there.  With seven vertices per thread (933,889
// vertices on 152 SMs) the kept words leave 32 KB of L1, and dense games lose to
// the graph, whose steps examine what has changed: ms per solve here and there
// at 10^6 vertices of mean degree 9, 12, 15, 24, 40, 100: 2.3, 2.3, 1.5, 2.1, 3.9,
// 8.9 and 3.2, 2.6, 1.6, 1.7, 2.2, 4.7 (at 940,000, degrees 12 and 15: 2.0, 1.5 and
// 1.9, 1.3; degree 200: 17 and 8.7).  With up to six it is the faster one: 930,000
// vertices 1.7, 1.8, 0.8, 1.0, 1.6, 3.5 and 2.8, 3.4, 1.2, 1.5, 1.9, 3.5, 500,000 of
// degree 300 8.8 and 18.5.
constexpr int64_t kDenseDegree = 14;
bool solve_takes(int64_t n, int64_t m)
{
    const int64_t round = (int64_t)kSolveThreads * device_sms();
    return n <= kMaxWaves * round && (n <= (kMaxCached - 1) * round || m <= kDenseDegree * n);
}

int launch_solve(cudaStream_t s, const SolveArgs &a)
{
    const int sms = device_sms();
    if (a.n < kSmall) {
        const SmallLayout l = small_layout(a.n, a.m);
        int threads = 64;
        while (threads < a.n && threads < kSolveThreads) threads *= 2;
        cudaError_t e = cudaFuncSetAttribute(k_solve_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallBytes);
        if (e != cudaSuccess) return (int)e;
        count_launch();
        k_solve_small<<<1, threads, l.total, s>>>(a);
        return (int)cudaGetLastError();
    }
    const int threads = spread_threads(a.n, sms, kOneEach);
    const int64_t need = ceil_div(a.n, threads);
    const int grid = (int)(need < sms ? need : sms);
    const int64_t waves = ceil_div(a.n, (int64_t)grid * threads);
    const size_t smem = 4 * (size_t)kWords * threads * (size_t)(waves < kMaxCached ? waves : kMaxCached);
    cudaError_t e = cudaFuncSetAttribute(k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes);
    if (e != cudaSuccess) return (int)e;
    void *args[] = {(void *)&a};
    count_launch();
    return (int)cudaLaunchCooperativeKernel((const void *)k_solve, dim3(grid), dim3(threads), args, smem, s);
}

}  // namespace psi
