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
//     jumping over those vertices alone.
//
// Against the tour upkeep, sublist walks, reduced-list ranking, depth
// broadcast, summary walks and cycle rounds that this replaces, an evaluation
// of the 2^24 random game reads each record it needs once: the tour and its
// ranking touched two successors, two rank records and the in-neighbours of
// every changed parent, all at random addresses, only for the depths.
#include <climits>
#include <cooperative_groups.h>

#include "device_common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace psi {

namespace {

__device__ __forceinline__ int ceil_log2_dev(int64_t x)
{
    int r = 0;
    while (((int64_t)1 << r) < x) r++;
    return r;
}

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

// Publishes a finite vertex: landmark record, status, summary.
__device__ __forceinline__ void publish_finite(const EvalArgs &a, int32_t v, int32_t d, int32_t m, int32_t c,
                                               int32_t anc, const Top2 &seg, uint32_t epoch, bool marks)
{
    if (marks) store_whole(&a.skip[v], skip_pack(anc, seg, epoch));
    a.st[v] = d;
    if (d >= kDeepPath) a.rdeep[v] = c;
    publish_summary(&a.node[v], m, path_word(d, c), d >= kDeepPath);
}

// A walk's step cap: longer walks are left to k_root_settle.
constexpr int32_t kWalkCap = 128;
constexpr int kWalkThreads = 256;
// unreached vertices buffered per warp before they go to the list with one
// atomic (one atomic per warp and pass on the list's counter would serialise)
constexpr int kUnreachedBuf = 128;

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
    int32_t *buf = ubuf[threadIdx.x >> 5];
    int nbuf = 0;   // uniform over the warp
    auto flush = [&] {
        int32_t base = 0;
        if (lane == 0) base = atomicAdd(a.ucount, nbuf);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int i = lane; i < nbuf; i += 32) a.ulist[base + i] = buf[i];
        __syncwarp();
        nbuf = 0;
    };
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
                    while (true) {
                        r = *reinterpret_cast<const int4 *>(&a.node[y]);
                        if (r.z != RM_UNKNOWN || y == mark || s >= kWalkCap) break;
                        if ((s & (s - 1)) == 0) mark = y;   // after 1, 2, 4, ... vertices the marker moves here
                        top1_merge(m, c, r.y, 1);
                        y = r.x;
                        s++;
                    }
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
        const unsigned um = __ballot_sync(0xffffffffu, infinite);
        if (um) {
            if (infinite) buf[nbuf + __popc(um & ((1u << lane) - 1))] = v;
            nbuf += __popc(um);
            __syncwarp();
            if (nbuf > kUnreachedBuf - 32) flush();
        }
        const int32_t p = warp_reserve(left, a.lcount);
        if (left) a.la[p] = v;
    }
    if (nbuf) flush();
}

// The vertices whose walk was cut short (list la, *lcount of them): pointer
// jumping over them alone.  In round r an entry is (the vertex 2^r steps
// ahead with kFlag possibly set, top priority of the 2^r vertices from u on,
// its count, the largest id among the vertices that carry it).  A target that
// is published settles u: a finite one with the window's summary merged, an
// infinite one with its infinity.  Two windows back to back with the same top
// (priority, id) vertex x mean that the walk meets x twice, so it is on x's
// cycle from the target on, shorter than 2^(r+1): u is flagged, and in the
// next round takes the parity of its target's window, which covers the
// cycle.  After ceil(log2 |la|) + 1 rounds every window is longer than any
// path through unpublished vertices: what is left is on a cycle.  A vertex
// settled in an earlier round is published, so no round reads its entry again.
constexpr int32_t kFlag = 1 << 30;   // vertex ids are below 2^30

constexpr int kSmallSettle = 4096;   // up to this many: one block, no grid barrier

template <bool GRID>
__device__ void settle_body(const EvalArgs &a, int32_t nl)
{
    const int64_t tid = GRID ? (int64_t)blockIdx.x * blockDim.x + threadIdx.x : threadIdx.x;
    const int64_t nth = GRID ? (int64_t)gridDim.x * blockDim.x : blockDim.x;
    auto barrier = [] {
        if (GRID) cg::this_grid().sync();
        else __syncthreads();
    };
    for (int64_t i = tid; i < nl; i += nth) {
        const int32_t u = a.la[i];
        a.ja[u] = make_int4(a.node[u].parent, a.node[u].pri, 1, u);
    }
    if (tid == 0) a.cnt[0] = a.cnt[1] = a.cnt[2] = 0;
    barrier();
    const int32_t *act = a.la;
    int32_t na = nl;
    int4 *in = a.ja, *out = a.jb;
    int32_t *next = a.lb, *spare = a.la;   // la is free after the first round
    const int rounds = ceil_log2_dev(nl) + 2;
    for (int r = 0; r < rounds && na > 0; r++) {
        const bool last = r == rounds - 1;
        int32_t *cnt = &a.cnt[r % 3];
        if (tid == 0) a.cnt[(r + 1) % 3] = 0;    // next round's counter (last read two rounds ago)
        for (int64_t b0 = tid - threadIdx.x; b0 < na; b0 += nth) {   // block-uniform passes
            const int64_t i = b0 + threadIdx.x;
            bool keep = false, changed = false, infinite = false;
            int32_t u = -1;
            if (i < na) {
                u = act[i];
                const int4 e = __ldcg(&in[u]);
                const int32_t t = e.x & ~kFlag;
                const int4 q = __ldcg(reinterpret_cast<const int4 *>(&a.node[t]));
                int32_t code = 0, k = 0;
                bool done = true;
                if (q.z == RM_POS_INF || q.z == RM_NEG_INF) {
                    code = q.z;
                } else if (q.z != RM_UNKNOWN) {
                    int32_t dt, ct, m = e.y, c = e.z;
                    path_depth_count(a, t, q.w, dt, ct);
                    top1_merge(m, c, q.z, ct);
                    const bool marks = a.g->lm_want;
                    const int32_t d = (int32_t)((1u << r) + (uint32_t)dt);
                    const int32_t len = marks ? d - skip_landmark_depth(d) : 0;
                    Top2 seg = {-1, 0, -1, 0};
                    int32_t anc = u;
                    for (int32_t j = 0; j < len; j++) {
                        const int2 x = *reinterpret_cast<const int2 *>(&a.node[anc]);
                        top2_add(seg, x.y);
                        anc = x.x;
                    }
                    publish_finite(a, u, d, m, c, anc, seg, *a.epoch & kEpochMask, marks);
                    k = finite_key(m, c);
                } else {
                    const int4 f = __ldcg(&in[t]);
                    if ((e.x & kFlag) || last) {
                        code = (f.y & 1) ? RM_NEG_INF : RM_POS_INF;
                    } else {
                        int4 o = make_int4(f.x & ~kFlag, e.y, e.z, e.w);
                        if (f.y > e.y) {
                            o.y = f.y;
                            o.z = f.z;
                            o.w = f.w;
                        } else if (f.y == e.y) {
                            o.z = (int32_t)((uint32_t)e.z + (uint32_t)f.z);   // may wrap on a cycle, where no count is used
                            o.w = max(e.w, f.w);
                            if (e.w == f.w) o.x |= kFlag;
                        }
                        out[u] = o;
                        keep = true;
                        done = false;
                    }
                }
                if (code) {
                    a.st[u] = (code == RM_POS_INF) ? ST_POS_INF : ST_NEG_INF;
                    publish_summary(&a.node[u], code, 0);
                    k = (code == RM_POS_INF) ? KEY_POS_INF : KEY_NEG_INF;
                    infinite = true;
                }
                if (done && a.key[u] != k) {
                    a.key[u] = k;
                    changed = true;
                }
            }
            flag_in_neighbours(a.track, changed, u);
            block_append(infinite, u, a.ulist, a.ucount);
            __syncthreads();
            block_append(keep, u, next, cnt);
            __syncthreads();
        }
        barrier();
        na = *(volatile int32_t *)cnt;
        act = next;
        int32_t *l = next;
        next = spare;
        spare = l;
        int4 *t = in;
        in = out;
        out = t;
    }
}

// 1,024-thread blocks, one per SM: few blocks at each round's grid barrier.
constexpr int kSettleThreads = 1024;
__global__ void __launch_bounds__(kSettleThreads, 1) k_root_settle(EvalArgs a)
{
    if (a.gate && !*a.gate) return;   // every block returns: no grid barrier is left waiting
    const int32_t nl = *a.lcount;
    if (nl == 0) return;
    if (nl <= kSmallSettle) {
        if (blockIdx.x == 0) settle_body<false>(a, nl);
        return;
    }
    settle_body<true>(a, nl);
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
