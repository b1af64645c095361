// patch_kernels.cu -- incremental evaluation on sm_103a.
//
// A vertex's valuation depends only on its strategy path: the vertices from
// it to the sink, to a solved vertex (whose value is frozen) or around a
// cycle.  After a switch step that changed few strategies, the path of most
// vertices avoids every changed vertex and their status words, path
// snapshots and keys are still what the last evaluation wrote.  A patch
// re-evaluates only the others -- the set A, the in-forest of the changed
// vertices in the new strategy graph, solved vertices excluded -- and ends
// with exactly the state a full evaluation (compute_valuation,
// gpu_list_ranking.cu:279-326) would leave.  Most evaluations of a solve
// follow such a step: in Odd's best-response loop the number of changed
// strategies falls by about an order of magnitude per step.
//
//  1. patch_begin (one thread; a launch, or part of the graph loop's control) takes the changed vertices the switch steps
//     listed since the last evaluation and opens either the patch's gate or
//     the full evaluation's: a patch needs the list complete, the caller's
//     permission (the list covers every change since the last
//     evaluation) and room in the unreached list.
//  2. k_patch (cooperative) finds A: the changed vertices (the seeds), then
//     the in-neighbours u with strat[u] == x of each vertex x found (reverse
//     CSR), and so on.  Every vertex has one successor, so a vertex other than
//     a seed is found once, by its own successor, with no atomics on the
//     vertex, and its subtree can be searched by whoever found it: every block
//     goes on from its share of the seeds alone, level by level in shared
//     memory, and only after kEpochLevels levels do the blocks meet at a grid
//     barrier and even out what is left.  (With a grid barrier per level and
//     the level's vertices in global memory, a level took 4.1 us.)  On the way
//     down each vertex gets its seed and the summary of its path up to that
//     seed (`rel`: seed index, vertices, top priority, its count), from its
//     successor's, and its in-edge range (`arev`).  If A outgrows its buffer
//     or the levels their cap, the patch gives up: the full evaluation's gates
//     open instead, and the next few evaluations do not try (doubling each
//     time).
//  3. Then the values.  A cycle inside A passes through a seed
//     (a cycle of unchanged vertices has no path to a changed one), so only
//     the seeds need pointer jumping: a seed's successor is the sink, a
//     vertex outside A (an exit with a known value: solved, or its path
//     avoids the changes) or a vertex of A, which leads to its own seed by
//     its rel summary.  The seeds jump without barriers (jump.cuh).  Then every
//     vertex of A takes its
//     seed's value merged with its rel summary, in one parallel pass: depth
//     = its vertices + its seed's depth, or the seed's infinity.  The
//     infinite ones are appended to the unreached list that mark_solved scans
//     (an entry that has since become finite is skipped there, st being
//     finite).  A changed key flags the vertex's in-neighbours as in a full
//     evaluation; an unchanged one only those tied on it (ChangeTrack); the
//     vertex's landmark skip becomes unknown (its path changed).
// A patch of few seeds runs in one block, without grid barriers.
#include <climits>
#include <cooperative_groups.h>

#include "device_common.cuh"
#include "jump.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace psi {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// 1,024 threads: one block per SM (fewer blocks at each grid barrier)
constexpr int kPatchBlock = 1024, kPatchWarps = kPatchBlock / 32;
constexpr int32_t kBackoffMax = 64;
// up to this many changed vertices (an upper bound of the seeds): one block
// (16, 64, 512, 2,048: 9.42, 9.35, 9.26, 9.34 ms per solve of 2*10^6 vertices,
// long-path 2^23 18.6, 18.4, 18.3, 18.6 ms)
constexpr int32_t kSoloSeeds = 512;
// levels between two meetings of the blocks (4, 8, 16, 32: 10.06, 9.35, 8.99,
// 8.95 ms for 2*10^6 vertices, 39.1, 37.9, 37.4, 38.2 ms for 2^24)
constexpr int32_t kEpochLevels = 16;
// vertices of a level a block holds; further ones go to the shared list of
// vertices still to be searched from (a.spill)
constexpr int kQueue = 2048;

// A level in shared memory.
struct Queue {
    int32_t u[kQueue], b[kQueue], d[kQueue], seed[kQueue], len[kQueue], top[kQueue], cnt[kQueue], pos[kQueue];
};

struct PatchShared {
    Queue q[2];
    int32_t count[2];
    int32_t base, bail, total, most;
};

__global__ void k_patch_begin(PatchArgs a, int32_t try_patch)
{
    if (try_patch >= 0) a.g->try_patch = try_patch;
    patch_begin(a);
}

__device__ __forceinline__ void place(const PatchArgs &a, int32_t p, int32_t u, int32_t b, int32_t d, const int4 &rel)
{
    a.alist[p] = u;
    a.apos[u] = p;
    a.arev[p] = make_int2(b, d);
    a.rel[p] = rel;
}

// Puts position p on the shared list; false (and *bail set: the search cannot
// be completed) if there is no room.
__device__ __forceinline__ void spill(const PatchArgs &a, int32_t p, int32_t *bail)
{
    const int32_t i = atomicAdd(&a.g->lcnt[2], 1);
    if (i < 2 * (int64_t)a.acap) a.spill[i] = p;
    else *bail = 1;
}

// Warp-collective: the in-edges of the lanes' vertices (valid ones, entries i
// of cur) laid end to end over the warp's lanes, 32 per round; each lane tests
// its edge's source u for being a child of its x outside A and puts it into
// next with x's seed and the path summary extended by u.  A level is a chain of
// dependent loads, so every load that does not need the test is issued with
// it: u's successor, solved flag, position, priority and in-edge range.
__device__ __forceinline__ void expand(const PatchArgs &a, int32_t ns, const Queue &cur, Queue &next,
                                       int32_t *next_count, int32_t *bail, bool valid, int32_t i)
{
    const int lane = threadIdx.x & 31;
    int32_t d = valid ? cur.d[i] : 0, incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += y;
    }
    const int32_t total = __shfl_sync(kAll, incl, 31);   // distinct vertices' in-edges: <= m
    for (int64_t j0 = 0; j0 < total; j0 += 32) {
        const int64_t j = j0 + lane;
        // owner lane of edge j: the number of lanes whose inclusive count is <= j
        int l = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const int32_t y = __shfl_sync(kAll, incl, l + step - 1);
            if (y <= j) l += step;
        }
        const int32_t il = __shfl_sync(kAll, i, l), el = __shfl_sync(kAll, incl - d, l);
        int32_t u = -1, pu = 0, ub = 0, ue = 0;
        bool child = false;
        if (j < total) {
            u = a.rev_src[cur.b[il] + (j - el)];
            const int32_t su = a.strat[u];
            const uint8_t so = a.solved[u];
            const int32_t ap = a.apos[u];
            pu = a.pri[u];
            ub = a.rev_off[u];
            ue = a.rev_off[u + 1];
            child = su == cur.u[il] && !so && ap == -1;
        }
        const int32_t p = warp_reserve(child, next_count);
        if (!child) continue;
        int32_t m = pu, c = 1;
        top1_merge(m, c, cur.top[il], cur.cnt[il]);
        if (p < kQueue) {
            next.u[p] = u;
            next.b[p] = ub;
            next.d[p] = ue - ub;
            next.seed[p] = cur.seed[il];
            next.len[p] = cur.len[il] + 1;
            next.top[p] = m;
            next.cnt[p] = c;
        } else {   // no room: placed at once and left to whoever has room
            const int32_t at = ns + atomicAdd(&a.g->lcnt[1], 1);
            if (at < a.acap) {
                place(a, at, u, ub, ue - ub, make_int4(cur.seed[il], cur.len[il] + 1, m, c));
                spill(a, at, bail);
            } else {
                *bail = 1;
            }
        }
    }
}

// Entry i of q from position p of A.
__device__ __forceinline__ void take(const PatchArgs &a, Queue &q, int32_t i, int32_t p)
{
    const int2 ev = a.arev[p];
    const int4 r = a.rel[p];
    q.u[i] = a.alist[p];
    q.b[i] = ev.x;
    q.d[i] = ev.y;
    q.seed[i] = r.x;
    q.len[i] = r.y;
    q.top[i] = r.z;
    q.cnt[i] = r.w;
    q.pos[i] = p;
}

__global__ void __launch_bounds__(kPatchBlock, 1) k_patch(PatchArgs a, cudaGraphConditionalHandle full, int32_t in_graph)
{
    extern __shared__ __align__(16) unsigned char patch_mem[];
    PatchShared &sh = *reinterpret_cast<PatchShared *>(patch_mem);
    EvalGates *g = a.g;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    if (!g->patch) {   // read by every block before any grid barrier; written after the last one
        if (leader && in_graph) cudaGraphSetConditional(full, 1);
        return;
    }
    const int32_t nc = g->csnap;
    const bool solo = nc <= kSoloSeeds;
    if (solo && blockIdx.x) return;
    const int32_t nb = solo ? 1 : (int32_t)gridDim.x, tid = blockIdx.x * kPatchBlock + threadIdx.x;
    const int32_t nth = nb * kPatchBlock;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // Barrier with a vote (k_solve's; solo: the block's own).
    uint32_t phase = a.sync->phase;
    auto barrier = [&](bool mine) -> bool {
        if (solo) return __syncthreads_or(mine);
        const uint32_t k = phase % 3, k1 = (phase + 1) % 3;
        phase++;
        if (tid == 0) a.sync->vote[k1] = a.sync->vote2[k1] = 0;
        if (__syncthreads_or(mine) && threadIdx.x == 0) a.sync->vote[k] = 1;
        cg::this_grid().sync();
        return __ldcg(&a.sync->vote[k]) != 0;
    };

    // the seeds: the changed vertices (a vertex listed twice is taken once)
    for (int32_t i0 = tid & ~31; i0 < nc; i0 += nth) {
        const int32_t i = i0 + lane;
        int32_t v = -1;
        bool mine = false;
        if (i < nc) {
            v = a.clist[i];
            mine = !a.solved[v] && atomicCAS(&a.apos[v], -1, -2) == -1;
        }
        const int32_t p = warp_reserve(mine, &g->lcnt[0]);
        if (mine) {
            if (p < a.acap) place(a, p, v, a.rev_off[v], a.rev_off[v + 1] - a.rev_off[v], make_int4(p, 0, -1, 0));
            else a.apos[v] = -1;
        }
    }
    barrier(false);
    const int32_t found = *(volatile int32_t *)&g->lcnt[0];
    const int32_t ns = found < a.acap ? found : a.acap;
    bool bail = found > a.acap;

    // the search, from seeds blockIdx.x, blockIdx.x + nb, ... (as many as the
    // queue takes; the others to the shared list)
    int cur = 0;
    int32_t pending = 0, held = 0;   // thread 0: where the current level's vertices are placed; vertices found
    bool placed = true;       // the current level's vertices have their positions
    int32_t levels = 0, spilled = 0;   // levels gone; entries of the shared list taken
    if (threadIdx.x == 0) {
        const int32_t mine = ns > (int32_t)blockIdx.x ? (ns - (int32_t)blockIdx.x + nb - 1) / nb : 0;
        sh.count[0] = mine < kQueue ? mine : kQueue;
        sh.bail = 0;
    }
    __syncthreads();
    for (int32_t j = threadIdx.x; blockIdx.x + (int64_t)j * nb < ns; j += kPatchBlock) {
        const int32_t p = (int32_t)(blockIdx.x + (int64_t)j * nb);
        if (j < kQueue) take(a, sh.q[0], j, p);
        else spill(a, p, &sh.bail);
    }
    __syncthreads();
    while (!bail) {
        // levels of this block's own; a level's positions are reserved while the
        // next one is being found, so nobody waits for that atomic
        for (int32_t l = 0; l < kEpochLevels || solo; l++) {
            const int32_t c = sh.count[cur];
            if (c == 0 || sh.bail) break;
            if (solo && ++levels > a.max_levels) {
                sh.bail = 1;
                break;
            }
            Queue &q = sh.q[cur], &next = sh.q[cur ^ 1];
            if (threadIdx.x == 0) sh.count[cur ^ 1] = 0;
            __syncthreads();
            // vertices per warp: as few as the level allows, so that a warp's
            // in-edges take one round of dependent loads
            const int32_t k = c >= kPatchBlock ? 32 : (c + kPatchWarps - 1) / kPatchWarps;
            for (int32_t i0 = warp * k; i0 < c; i0 += kPatchWarps * k) {
                const int32_t i = i0 + lane;
                const bool valid = lane < k && i < c;
                expand(a, ns, q, next, &sh.count[cur ^ 1], &sh.bail, valid, i);
            }
            if (threadIdx.x == 0 && !placed) sh.base = pending;
            __syncthreads();
            if (!placed)
                for (int32_t i = threadIdx.x; i < c; i += kPatchBlock) {
                    const int32_t p = sh.base + i;
                    if (p < a.acap) place(a, p, q.u[i], q.b[i], q.d[i], make_int4(q.seed[i], q.len[i], q.top[i], q.cnt[i]));
                    else sh.bail = 1;
                }
            if (threadIdx.x == 0) {
                if (sh.count[cur ^ 1] > kQueue) sh.count[cur ^ 1] = kQueue;
                held += sh.count[cur ^ 1];
                if (solo && held > a.solo_most) sh.bail = 1;
                pending = sh.count[cur ^ 1] ? ns + atomicAdd(&g->lcnt[1], sh.count[cur ^ 1]) : 0;
            }
            placed = false;
            cur ^= 1;
            __syncthreads();
        }
        // the blocks meet: positions of what was found last, and the sizes
        __syncthreads();
        const int32_t c = sh.count[cur];
        if (threadIdx.x == 0 && !placed) sh.base = pending;
        __syncthreads();
        Queue &q = sh.q[cur];
        if (!placed)
            for (int32_t i = threadIdx.x; i < c; i += kPatchBlock) {
                const int32_t p = sh.base + i;
                q.pos[i] = p;
                if (p < a.acap) place(a, p, q.u[i], q.b[i], q.d[i], make_int4(q.seed[i], q.len[i], q.top[i], q.cnt[i]));
                else sh.bail = 1;
            }
        placed = true;
        if (threadIdx.x == 0) a.sizes[blockIdx.x] = c;
        __syncthreads();
        bail = barrier(sh.bail);
        const int32_t reserved = *(volatile int32_t *)&g->lcnt[1], nspill = *(volatile int32_t *)&g->lcnt[2];
        if (!solo) levels += kEpochLevels;
        bail |= ns + (int64_t)reserved > a.acap || levels > a.max_levels;
        if (bail) break;
        if (warp == 0) {
            int32_t sum = 0, most = 0;
            for (int32_t b = lane; b < nb; b += 32) {
                const int32_t x = *(volatile int32_t *)&a.sizes[b];
                sum += x;
                most = max(most, x);
            }
            sum = __reduce_add_sync(kAll, sum);
            most = __reduce_max_sync(kAll, most);
            if (lane == 0) {
                sh.total = sum;
                sh.most = most;
            }
        }
        __syncthreads();
        const int32_t total = sh.total, avg = (total + nb - 1) / nb;
        if (total == 0 && nspill == spilled) break;   // A is complete
        if (nspill == spilled && sh.most <= 2 * avg + 128) {
            if (!solo) barrier(false);   // every block has read the sizes
            continue;
        }
        // uneven: what a block has above the average goes to the shared list,
        // from which each takes its share
        if (c > avg)
            for (int32_t i = avg + threadIdx.x; i < c; i += kPatchBlock) spill(a, q.pos[i], &sh.bail);
        __syncthreads();
        const int32_t kept = c < avg ? c : avg;
        bail = barrier(sh.bail);
        if (bail) break;
        const int32_t end = *(volatile int32_t *)&g->lcnt[2];
        const int32_t room = nb * (kQueue / 2);
        const int32_t some = end - spilled < room ? end - spilled : room;   // the rest: next time
        const int32_t s0 = (int32_t)((int64_t)some * blockIdx.x / nb), s1 = (int32_t)((int64_t)some * (blockIdx.x + 1) / nb);
        int32_t fits = s1 - s0;   // kept <= avg <= kQueue: a share may still not fit
        if (fits > kQueue - kept) fits = kQueue - kept;
        for (int32_t i = threadIdx.x; i < s1 - s0; i += kPatchBlock) {
            const int32_t p = a.spill[spilled + s0 + i];
            if (i < fits) take(a, q, kept + i, p);
            else a.spill2[atomicAdd(&g->acount, 1)] = p;
        }
        spilled += some;
        if (threadIdx.x == 0) sh.count[cur] = kept + fits;
        barrier(false);   // shares read before the list grows again
        const int32_t back = *(volatile int32_t *)&g->acount;
        if (back) {   // what did not fit goes back to the list's end
            for (int32_t i = tid; i < back; i += nth) spill(a, a.spill2[i], &sh.bail);
            __syncthreads();
            bail = barrier(sh.bail);
            if (leader) g->acount = 0;
            barrier(false);
        } else if (spilled == end) {   // the list is used up: from its beginning again
            if (leader) g->lcnt[2] = 0;
            spilled = 0;
            barrier(false);
        }
    }
    const int32_t na = ns + *(volatile int32_t *)&g->lcnt[1];
    if (bail) {   // give up: A's marks cleared, the full evaluation's gates opened
        const int32_t marked = na < a.acap ? na : a.acap;
        barrier(false);   // every block has placed its last vertices
        for (int32_t i = tid; i < marked; i += nth) a.apos[a.alist[i]] = -1;
        if (leader) {
            g->patch = 0;
            g->eval = 1;
            *a.ucount = 0;
            g->mfrom[0] = g->mfrom[1] = 0;
            g->skip = g->backoff;
            g->backoff = g->backoff < kBackoffMax ? 2 * g->backoff : kBackoffMax;
            if (!solo) a.sync->phase = kept_phase(phase);
            if (in_graph) cudaGraphSetConditional(full, 1);
        }
        return;
    }

    // seed records: the next seed its successor leads to, or finished: the sink,
    // or an exit outside A, whose value is current
    for (int32_t s = tid; s < ns; s += nth) {
        const int32_t v = a.alist[s], t = a.strat[v];
        int4 e = make_int4(kSink, a.pri[v], 1, 1);
        if (t >= 0) {
            const int32_t p = a.apos[t];
            if (p >= 0) {
                const int4 r = a.rel[p];
                e.x = r.x;
                e.w += r.y;
                top1_merge(e.y, e.z, r.z, r.w);
            } else {
                const int32_t st = a.st[t];
                if (st >= 1) {
                    const PathNode q = a.node[t];
                    e.w += st;
                    top1_merge(e.y, e.z, q.rmax, st < kDeepPath ? path_word_count(q.word) : a.rdeep[t]);
                } else {
                    e = make_int4(st == ST_POS_INF ? kPosInf : kNegInf, 0, 0, 0);
                }
            }
        }
        store_whole(&a.sja[s], e);
    }
    barrier(false);
    bool left = true;
    for (int pass = 0; left; pass++) {
        if (pass == kMaxPasses) {   // cannot happen: windows grow at least kJumps-fold per pass
            if (tid == 0) atomicOr(a.err, DERR_WALK_CAP);
            break;
        }
        left = false;
        for (int32_t s = tid; s < ns; s += nth) {
            int4 r = load_whole(&a.sja[s]), q = r;
            if (r.x >= 0) q = load_whole(&a.sja[r.x]);
            left |= !jump_pass<false>(a.sja, a.n, s, r, q);
        }
        left = barrier(left);
    }

    // every vertex of A: its seed's value merged with its rel summary, in
    // block-uniform passes (flag_in_neighbours and block_append need every
    // thread of the block)
    for (int32_t b0 = tid - threadIdx.x; b0 < na; b0 += nth) {
        const int32_t i = b0 + threadIdx.x;
        int32_t v = -1;
        bool changed = false, unreached = false;
        int mode = 0;
        int2 ev = make_int2(0, 0);   // v's in-edge range, stored by the search
        if (i < na) {
            v = a.alist[i];
            ev = a.arev[i];
            const int4 r = a.rel[i];
            // v's own words, loaded before any store (which might alias them)
            // so that they travel with the seed's value
            const int32_t sv_strat = a.strat[v], sv_pri = a.pri[v];
            const int32_t oldk = a.key ? a.key[v] : 0;
            const bool watched = a.track.watch && a.track.watch[v];
            const int4 sv = a.sja[r.x];
            int32_t k;
            if (sv.x == kSink) {
                int32_t m = r.z, c = r.w;
                top1_merge(m, c, sv.y, sv.z);
                const int32_t d = r.y + sv.w;
                a.st[v] = d;
                a.node[v] = PathNode{sv_strat, sv_pri, m, path_word(d, c)};
                if (d >= kDeepPath) a.rdeep[v] = c;
                k = finite_key(m, c);
            } else {
                a.st[v] = sv.x == kPosInf ? ST_POS_INF : ST_NEG_INF;
                k = sv.x == kPosInf ? KEY_POS_INF : KEY_NEG_INF;
                unreached = true;
            }
            if (a.key && oldk != k) {
                a.key[v] = k;
                changed = true;
            }
            // re-evaluated: a tied in-neighbour looks again even at an unchanged key
            mode = changed ? 2 : (watched ? 1 : 0);
            if (a.g->lm_have) a.skip[v] = make_int4(SKIP_UNKNOWN, 0, 0, 0);   // its path changed: walks step here
            a.apos[v] = -1;
        }
        flag_in_neighbours(a.track, mode, v, &ev);
        block_append(unreached, v, a.ulist, a.ucount);
    }
    if (leader) {
        g->backoff = 1;
        g->acount = na;
        a.stats[0] += 1;
        a.stats[1] += (unsigned long long)na;
        if (!solo) a.sync->phase = kept_phase(phase);
        if (in_graph) cudaGraphSetConditional(full, 0);
    }
}

int patch_blocks()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_patch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PatchShared));
    return sms > 0 ? (sms < kPatchSizes ? sms : kPatchSizes) : 1;
}

std::atomic<int> g_patch_blocks[kMaxCachedDevices];

}  // namespace

void launch_patch_begin(cudaStream_t s, const PatchArgs &a, int32_t try_patch)
{
    count_launch();
    k_patch_begin<<<1, 1, 0, s>>>(a, try_patch);
}

int launch_patch(cudaStream_t s, const PatchArgs &a, const cudaGraphConditionalHandle *full)
{
    const int blocks = per_device(g_patch_blocks, patch_blocks);
    cudaGraphConditionalHandle h = full ? *full : cudaGraphConditionalHandle();
    int32_t in_graph = full ? 1 : 0;
    void *args[] = {(void *)&a, (void *)&h, (void *)&in_graph};
    count_launch();
    return (int)cudaLaunchCooperativeKernel((const void *)k_patch, dim3(blocks), dim3(kPatchBlock), args,
                                            sizeof(PatchShared), s);
}

}  // namespace psi
