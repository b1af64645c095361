// root_kernels.cu -- full strategy evaluation on sm_103a.
//
// One evaluation turns the current strategy (one successor per vertex, -1 for
// the sink) into every vertex's status word, root-path summary, comparison
// key and landmark skip (device_common.cuh).  The reference ranks an Euler
// tour of the strategy tree for the depths (gpu_list_ranking.cu:52-277); here
// the strategy graph itself is walked, because the summaries need a walk over
// the same paths anyway and a vertex's depth is known as soon as an ancestor's
// is:
//
//  1. k_root_init streams strategies and priorities into the path records.
//     The sink's children get their summary at once, solved vertices their
//     frozen value.
//  2. k_root_walk: one thread per vertex follows the strategy until it meets
//     a vertex whose result is published (by init or by another thread of
//     this launch) and publishes its own: depth, summary, landmark, or an
//     infinity.  A walk on a cycle notices it (Brent's teleporting marker:
//     the marker moves to the current vertex after 1, 2, 4, ... steps, and
//     meeting it again means one round of the cycle, whose top priority was
//     collected since) -- the cycle parity of cpu_parity.cpp:35-52, 80-104.
//     With threads in arbitrary order a walk is short: about two steps on
//     random games, whose paths are 12 vertices long on average (ten for the
//     longest of a warp's walks).  Landmark records only where wanted.
//  3. k_root_settle: walks that did not end within kWalkCap steps (deep
//     chains, long cycles, none on random games) are finished by pointer
//     jumping without barriers (jump.cuh) over those vertices alone.
//
// Against the tour upkeep, sublist walks, reduced-list ranking, depth
// broadcast, summary walks and cycle rounds that this replaces, an evaluation
// of the 2^24 random game reads each record it needs once: the tour and its
// ranking touched two successors, two rank records and the in-neighbours of
// every changed parent, all at random addresses, only for the depths.
#include <climits>
#include <cooperative_groups.h>

#include "device_common.cuh"
#include "jump.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace psi {

namespace {

// Path records of a new evaluation: unknown, except the sink's children
// (depth 1, their own priority) and the solved vertices (their frozen
// infinity; nothing walks past them).  A full evaluation also makes every tied
// vertex be looked at again (ChangeTrack).
__global__ void k_root_init(EvalArgs a)
{
    if (a.gate && !*a.gate) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.lcount = 0;
        a.g->lm_have = a.g->lm_want;
    }
    // the evaluation number wraps around: no record of the last round may look
    // current, those past the arena's present extent among them
    if ((*a.epoch & kEpochMask) == 0)
        for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < a.cap; v += (int64_t)gridDim.x * blockDim.x)
            a.skip[v] = make_int4(SKIP_UNKNOWN, 0, 0, 0);
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < a.n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t t = a.strat[v], p = a.pri[v];
        int4 q = make_int4(t, p, RM_UNKNOWN, 0);
        if (a.solved[v]) q = make_int4(-1, p, a.st[v] == ST_POS_INF ? RM_POS_INF : RM_NEG_INF, 0);
        else if (t < 0) q = make_int4(-1, p, p, path_word(1, 1));
        *reinterpret_cast<int4 *>(&a.node[v]) = q;
        if (a.track.tie && a.track.tie[v]) a.track.need[v] = 1;
    }
}

// Depth and count of a published finite vertex y from its word w; deep ones
// (kDeepPath) keep them in st and rdeep, written before the summary.
__device__ __forceinline__ void path_depth_count(const EvalArgs &a, int32_t y, int32_t w, int32_t &depth,
                                                 int32_t &count)
{
    depth = path_word_depth(w);
    count = path_word_count(w);
    if (depth == kDeepPath) {
        acquire_rmax(&a.node[y]);
        depth = __ldcg(&a.st[y]);
        count = __ldcg(&a.rdeep[y]);
    }
}

// A walk's step cap: longer walks are left to k_root_settle.  So are all of a
// warp's if none of the 32 has ended after kWarpCap steps (the lanes that happen to
// be together then: which walks are left changes no result).  In random games a
// warp has walks that end; where the sink reaches few vertices, 128 steps each were
// most of an evaluation: without, and with 8, 16, 32 steps, ms per solve of one
// cycle of 1.6*10^7 27.5, 5.3, 6.8, 9.8, all Odd 11.1, 4.3, 5.4, 6.8; 2^24 random
// 31.9, 31.8, 31.8, 31.9.  (As a second cap inside one loop: 2^24 random +1%.)
constexpr int32_t kWalkCap = 128, kWarpCap = 8;
constexpr int kWalkThreads = 256;
// unreached vertices buffered per warp before they go to the list with one
// atomic (one atomic per warp and pass on the list's counter would serialise)
constexpr int kUnreachedBuf = 128;

// A warp's buffer; its lanes call both together.
struct Unreached {
    int32_t *buf;
    int held = 0;   // uniform over the warp
    __device__ __forceinline__ void flush(const EvalArgs &a)
    {
        const int lane = threadIdx.x & 31;
        int32_t base = 0;
        if (lane == 0) base = atomicAdd(a.ucount, held);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int i = lane; i < held; i += 32) a.ulist[base + i] = buf[i];
        __syncwarp();
        held = 0;
    }
    __device__ __forceinline__ void add(const EvalArgs &a, bool infinite, int32_t v)
    {
        const unsigned m = __ballot_sync(0xffffffffu, infinite);
        if (!m) return;
        if (infinite) buf[held + __popc(m & ((1u << (threadIdx.x & 31)) - 1))] = v;
        held += __popc(m);
        __syncwarp();
        if (held > kUnreachedBuf - 32) flush(a);
    }
};

// Bound by dependent random reads (2^22 random game: DRAM 40%, L2 36%, issue
// slots 60% busy; 2^24: 2.9 GB in 670 us, 4.1 TB/s), so eight blocks per SM at
// 32 registers; a summary is stored as soon as it is known and without a
// release (which waits for the thread's earlier stores: a third of the stalls),
// the landmark record, where wanted, after it and tagged with the evaluation's
// number.  Walks and init of a 2^24 solve 17.6 -> 14.1 ms (17 full evaluations),
// long-path 11.0 -> 8.9 ms, without landmark records 11.5 and 5.8.  Lanes that
// take the next vertex as soon as their walk ends lose (solve 35.3 -> 35.6,
// long-path 18.3 -> 20.5 ms): a walk's end is 60 instructions that then run at
// almost every step.
__global__ void __launch_bounds__(kWalkThreads, 8) k_root_walk(EvalArgs a)
{
    if (a.gate && !*a.gate) return;
    __shared__ int32_t ubuf[kWalkThreads / 32][kUnreachedBuf];
    const uint32_t epoch = *a.epoch & kEpochMask;
    const bool marks = a.g->lm_want;
    const int lane = threadIdx.x & 31;
    Unreached unreached{ubuf[threadIdx.x >> 5]};
    // every warp takes 32 consecutive vertices at a time
    for (int64_t b0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; b0 < a.n;
         b0 += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)(b0 + lane);
        bool finite = false, infinite = false, left = false;
        int32_t k = 0, old = 0;
        if (v < a.n) {
            const int4 q = *reinterpret_cast<const int4 *>(&a.node[v]);
            old = a.key[v];
            if (q.z != RM_POS_INF && q.z != RM_NEG_INF) {   // not solved
                if (q.x < 0) {   // a child of the sink, published by init: its skip and status are written here
                    a.st[v] = 1;
                    if (marks) store_whole(&a.skip[v], skip_pack(-1, Top2{q.y, 1, -1, 0}, epoch));
                    k = finite_key(q.y, 1);
                    finite = true;
                } else {
                    int32_t m = q.y, c = 1;
                    int32_t y = q.x, s = 1, mark = v;   // s vertices walked, y the next one; the marker
                    int4 r;
                    auto walk = [&](int32_t cap) {
                        while (true) {
                            r = *reinterpret_cast<const int4 *>(&a.node[y]);
                            if (r.z != RM_UNKNOWN || y == mark || s >= cap) break;
                            if ((s & (s - 1)) == 0) mark = y;   // after 1, 2, 4, ... vertices the marker moves here
                            top1_merge(m, c, r.y, 1);
                            y = r.x;
                            s++;
                        }
                    };
                    walk(kWarpCap);
                    if (r.z == RM_UNKNOWN && y != mark && __activemask() != 0xffffffffu) walk(kWalkCap);
                    int32_t code = 0;                       // an infinity, where it is one
                    if (r.z == RM_POS_INF || r.z == RM_NEG_INF) {
                        code = r.z;
                    } else if (r.z == RM_UNKNOWN && y == mark) {   // a cycle of at most s vertices
                        int32_t top = r.y;
                        for (int32_t x = r.x; x != mark;) {
                            const int2 e = *reinterpret_cast<const int2 *>(&a.node[x]);
                            top = max(top, e.y);
                            x = e.x;
                        }
                        code = (top & 1) ? RM_NEG_INF : RM_POS_INF;
                    }
                    if (code) {
                        a.st[v] = (code == RM_POS_INF) ? ST_POS_INF : ST_NEG_INF;
                        publish_summary(&a.node[v], code, 0);
                        k = (code == RM_POS_INF) ? KEY_POS_INF : KEY_NEG_INF;
                        infinite = true;
                    } else if (r.z == RM_UNKNOWN) {
                        left = true;
                    } else {
                        int32_t dy, cy;
                        path_depth_count(a, y, r.w, dy, cy);
                        top1_merge(m, c, r.z, cy);
                        k = finite_key(m, c);
                        finite = true;
                        const int32_t d = s + dy;
                        a.st[v] = d;
                        if (d >= kDeepPath) a.rdeep[v] = c;
                        publish_summary(&a.node[v], m, path_word(d, c), d >= kDeepPath);
                        // the segment from v to its landmark: by steps (the walk has just read
                        // them) up to y, then y's record if the landmark lies beyond and the
                        // record has arrived (its summary may have come first), else by steps
                        if (marks) {
                            const int32_t len = d - skip_landmark_depth(d);
                            Top2 seg = {q.y, 1, -1, 0};
                            int32_t anc = q.x;
                            for (int32_t i = 1; i < len; i++) {
                                if (i == s) {
                                    const int4 sy = load_whole(&a.skip[y]);
                                    if (sy.x != SKIP_UNKNOWN && skip_epoch(sy.w) == epoch) {
                                        skip_merge(seg, sy);
                                        anc = sy.x;
                                        break;
                                    }
                                }
                                const int2 e = *reinterpret_cast<const int2 *>(&a.node[anc]);
                                top2_add(seg, e.y);
                                anc = e.x;
                            }
                            store_whole(&a.skip[v], skip_pack(anc, seg, epoch));
                        }
                    }
                }
            }
        }
        const bool changed = (finite || infinite) && k != old;
        if (changed) a.key[v] = k;
        flag_in_neighbours(a.track, changed, v);
        unreached.add(a, infinite, v);
        const int32_t p = warp_reserve(left, a.lcount);
        if (left) a.la[p] = v;
    }
    if (unreached.held) unreached.flush(a);
}

// The vertices whose walk was cut short (list la, *lcount of them).  Their
// successors are published, and give a finished record at once, or on the list
// too, so from then on only the records (ja, 16 bytes) of vertices on the list
// are read: one random read per jump and no rounds, where the pointer doubling
// that this replaces read the target's path record as well, kept lists of
// what was left and met at a barrier log2 n times.  One cycle of 4*10^6, 1.6*10^7
// vertices (all of them left): 3.3 -> 0.55, 16.8 -> 3.0 ms.
constexpr int kSettleThreads = 1024;   // one block per SM: few blocks at a pass's grid barrier
constexpr int kSmallSettle = 4096;     // up to this many: one block, no grid barrier
__global__ void __launch_bounds__(kSettleThreads, 1) k_root_settle(EvalArgs a)
{
    if (a.gate && !*a.gate) return;   // every block returns: no grid barrier is left waiting
    const int32_t nl = *a.lcount;
    const bool one = nl <= kSmallSettle;
    if (nl == 0 || (one && blockIdx.x)) return;
    __shared__ int32_t ubuf[kSettleThreads / 32][kUnreachedBuf];
    Unreached unreached{ubuf[threadIdx.x >> 5]};
    const int64_t tid = (one ? 0 : (int64_t)blockIdx.x * kSettleThreads) + threadIdx.x;
    const int64_t nth = one ? kSettleThreads : (int64_t)gridDim.x * kSettleThreads;
    // barrier with a vote (k_solve's; one block: its own)
    uint32_t phase = a.sync->phase;
    auto barrier = [&](bool mine) -> bool {
        if (one) return __syncthreads_or(mine);
        const uint32_t k = phase % 3, k1 = (phase + 1) % 3;
        phase++;
        if (tid == 0) a.sync->vote[k1] = a.sync->vote2[k1] = 0;
        if (__syncthreads_or(mine) && threadIdx.x == 0) a.sync->vote[k] = 1;
        cg::this_grid().sync();
        return __ldcg(&a.sync->vote[k]) != 0;
    };
    for (int64_t i = tid; i < nl; i += nth) {
        const int32_t u = a.la[i];
        const int2 p = *reinterpret_cast<const int2 *>(&a.node[u]);   // successor (not the sink), priority
        const int4 q = *reinterpret_cast<const int4 *>(&a.node[p.x]);
        int4 r = make_int4(p.x, p.y, 1, 1);
        if (q.z == RM_POS_INF || q.z == RM_NEG_INF) {
            r = make_int4(q.z == RM_POS_INF ? kPosInf : kNegInf, 0, 0, 0);
        } else if (q.z != RM_UNKNOWN) {
            int32_t d, c;
            path_depth_count(a, p.x, q.w, d, c);
            top1_merge(r.y, r.z, q.z, c);
            r.x = kSink;
            r.w += d;
        }
        store_whole(&a.ja[u], r);
    }
    barrier(false);
    const bool marks = a.g->lm_want;
    const uint32_t epoch = *a.epoch & kEpochMask;
    bool more = true;
    for (int pass = 0; more; pass++) {
        if (pass == kMaxPasses) {   // cannot happen: windows grow at least kJumps-fold per pass
            if (tid == 0) atomicOr(a.err, DERR_WALK_CAP);
            break;
        }
        bool left = false;
        for (int64_t b = tid & ~31ll; b < nl; b += nth) {   // whole warps: flags and appends are collective
            const int64_t i = b + (threadIdx.x & 31);
            bool changed = false, infinite = false;
            int32_t u = -1;
            if (i < nl) {
                u = a.la[i];
                int4 r = load_whole(&a.ja[u]);
                // in later passes, what is finished has been dealt with
                if (pass == 0 || r.x >= 0) {
                    int4 q = r;
                    if (r.x >= 0) q = load_whole(&a.ja[r.x]);
                    if (jump_pass<false>(a.ja, a.n, u, r, q)) {
                        const bool fin = r.x == kSink;
                        const int32_t d = r.w, code = r.x == kPosInf ? RM_POS_INF : RM_NEG_INF;
                        const int32_t k = fin ? finite_key(r.y, r.z) : (r.x == kPosInf ? KEY_POS_INF : KEY_NEG_INF);
                        a.st[u] = fin ? d : (r.x == kPosInf ? ST_POS_INF : ST_NEG_INF);
                        if (fin && d >= kDeepPath) a.rdeep[u] = r.z;
                        *reinterpret_cast<int2 *>(&a.node[u].rmax) =
                            fin ? make_int2(r.y, path_word(d, r.z)) : make_int2(code, 0);
                        if (fin && marks) {
                            Top2 seg = {-1, 0, -1, 0};
                            int32_t anc = u;
                            for (int32_t j = d - skip_landmark_depth(d); j > 0; j--) {
                                const int2 x = *reinterpret_cast<const int2 *>(&a.node[anc]);
                                top2_add(seg, x.y);
                                anc = x.x;
                            }
                            store_whole(&a.skip[u], skip_pack(anc, seg, epoch));
                        }
                        infinite = !fin;
                        changed = a.key[u] != k;
                        if (changed) a.key[u] = k;
                    } else {
                        left = true;
                    }
                }
            }
            flag_in_neighbours(a.track, changed, u);
            unreached.add(a, infinite, u);
        }
        more = barrier(left);
    }
    if (unreached.held) unreached.flush(a);
    if (tid == 0 && !one) a.sync->phase = kept_phase(phase);
}

std::atomic<int> g_sms[kMaxCachedDevices];

int device_sms()
{
    return per_device(g_sms, [] {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return sms > 0 ? sms : 1;
    });
}

// Many more blocks than are resident: walks differ in length, and short blocks
// even that out (2^24 random game, ms per solve with 16, 64, 256 blocks per
// SM: 36.6, 35.3, 35.2, long-path 25.1, 24.1, 23.1).  A gated launch whose
// gate is closed pays for its blocks, 27 us at 256 per SM, so those keep to 64.
unsigned walk_grid(const EvalArgs &a)
{
    const int64_t g = ceil_div(a.n, kBlock), cap = (a.gate ? 64 : 256) * (int64_t)device_sms();
    return (unsigned)(g < 1 ? 1 : (g < cap ? g : cap));
}

}  // namespace

void launch_root_init(cudaStream_t s, const EvalArgs &a)
{
    count_launch();
    k_root_init<<<walk_grid(a), kBlock, 0, s>>>(a);
}

void launch_root_walk(cudaStream_t s, const EvalArgs &a)
{
    count_launch();
    k_root_walk<<<walk_grid(a), kWalkThreads, 0, s>>>(a);
}

int launch_root_settle(cudaStream_t s, const EvalArgs &a)
{
    void *args[] = {(void *)&a};
    count_launch();
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_root_settle, dim3(device_sms()), dim3(kSettleThreads),
                                                args, 0, s);
    return e == cudaSuccess ? 0 : (int)e;
}

}  // namespace psi
