// compare.cuh -- the exact comparison of two finite valuations by walking
// their paths to the lowest common ancestor (the third tier described in
// switch_kernels.cu), for every kernel that switches strategies.
#ifndef PSI_COMPARE_CUH
#define PSI_COMPARE_CUH

#include <climits>

#include "device_common.cuh"

namespace psi {

// Even's view of a difference at priority p: +1 if side a is better.
__device__ __forceinline__ int decide(int32_t p, int32_t ca, int32_t cb)
{
    if ((p & 1) == 0) return ca > cb ? 1 : -1;
    return ca < cb ? 1 : -1;
}

// The next successor to compare exactly: ties holds which of the first 32
// share the best key with the first best one; from the 32nd on all are asked
// for (one that precedes the first best one has another key).  With it the
// lanes of a warp come to their ties together, whatever their places in the
// lists: in a loop over all successors each place was a turn of its own, in
// which the lanes without a tie there waited for a walk (persistent solver,
// 10^4, 10^5, 10^6 vertices and 2^18 with 8 priorities, us per solve: 281, 715,
// 3837, 1928 -> 252, 670, 3648, 1600; graph, 2^24 with many ties, 2^22 with 8
// priorities, ms: 43.4, 13.5 -> 40.2, 12.6).
__device__ __forceinline__ int32_t next_tied(uint32_t &ties, int32_t &j)
{
    if (ties) {
        j = __ffs(ties) - 1;
        ties &= ties - 1;
    } else if (j < 32) {
        j = 32;
    }
    return j;
}

// Tier 3: walks to the lowest common ancestor of u and w (depths du, dw; w may
// be the sink, -1 with depth 0).  Pass k finds the highest priority below the
// last tie on each side's segment below the ancestor, and its count.  With
// skip, whole landmark segments are jumped (device_common.cuh) where their
// record's two priorities tell the one sought: the deeper side jumps while its
// landmark is no shallower than the other side; at equal depths both jump
// while their landmarks differ (the common ancestor is then above both); once
// they share one, the common ancestor lies in that segment and both step one
// vertex at a time.  One priority per pass keeps a step to a few instructions
// without branches on priorities: updating two diverged, about 0.12 us per
// step on top of the loads, where a whole launch or phase waits for its
// longest walk.  path: per vertex a record that begins with (parent,
// priority).  Once loads passes budget: kUndecided.  Without SKIP a step is its
// loads and little else, and they are issued before the checks (persistent
// solver, sizes as above, against a test of skip at run time: 306, 770, 3993,
// 2255 -> 281, 715, 3837, 1928).
constexpr int kUndecided = 2;
__device__ __forceinline__ void top_add(int32_t &m, int32_t &c, int32_t p, int32_t k, int32_t below)
{
    p = p < below ? p : -1;
    c = p > m ? k : (p == m ? c + k : c);
    m = max(m, p);
}
__device__ __forceinline__ bool top_jump(int32_t &m, int32_t &c, const int4 s, int32_t below)
{
    if (s.x == SKIP_UNKNOWN || (s.y >= below && s.z >= below)) return false;
    const bool first = s.y < below;
    top_add(m, c, first ? s.y : s.z, first ? skip_c1(s.w) : skip_c2(s.w), below);
    return true;
}
template <bool SKIP, class Rec>
static __device__ __noinline__ int lean_compare(const Rec *path, const int4 *skip, int32_t u, int32_t du, int32_t w,
                                                int32_t dw, int32_t &loads, int32_t budget, uint32_t *err)
{
    int32_t below = INT_MAX;
    for (int32_t pass = 0; pass <= du + dw; pass++) {
        int32_t a = u, b = w, da = du, db = dw, ma = -1, ca = 0, mb = -1, cb = 0;
        bool swapped = false;
        if (da < db) {   // a is the deeper side
            a = w;
            b = u;
            da = dw;
            db = du;
            swapped = true;
        }
        while (da > db) {
            if (a < 0 || ++loads > budget) break;
            if (SKIP) {
                const int32_t l = skip_landmark_depth(da);
                if (l >= db) {
                    const int4 s = skip[a];
                    if (top_jump(ma, ca, s, below)) {
                        a = s.x;
                        da = l;
                        continue;
                    }
                }
            }
            const int2 q = *reinterpret_cast<const int2 *>(&path[a]);
            top_add(ma, ca, q.y, 1, below);
            a = q.x;
            da--;
        }
        bool jumps = SKIP;
        while (a != b) {
            if (a < 0 || b < 0) break;
            int2 q, r;
            if (!SKIP) {
                q = *reinterpret_cast<const int2 *>(&path[a]);
                r = *reinterpret_cast<const int2 *>(&path[b]);
            }
            loads += 2;
            if (loads > budget) break;
            if (jumps) {
                const int4 s = skip[a], t = skip[b];
                int32_t m2 = ma, c2 = ca, m3 = mb, c3 = cb;
                if (s.x != t.x && top_jump(m2, c2, s, below) && top_jump(m3, c3, t, below)) {
                    ma = m2;
                    ca = c2;
                    mb = m3;
                    cb = c3;
                    a = s.x;
                    b = t.x;
                    da = skip_landmark_depth(da);
                    continue;
                }
                // one landmark: the paths meet in this segment
                jumps = s.x != t.x;
            }
            if (SKIP) {
                q = *reinterpret_cast<const int2 *>(&path[a]);
                r = *reinterpret_cast<const int2 *>(&path[b]);
            }
            top_add(ma, ca, q.y, 1, below);
            top_add(mb, cb, r.y, 1, below);
            a = q.x;
            b = r.x;
            da--;
        }
        if (loads > budget) return kUndecided;
        if (a != b) {   // inconsistent: cannot happen
            atomicOr(err, DERR_WALK_CAP);
            return 0;
        }
        const int32_t m = max(ma, mb);
        if (m < 0) return 0;
        ca = ma == m ? ca : 0;
        cb = mb == m ? cb : 0;
        if (ca != cb) return swapped ? decide(m, cb, ca) : decide(m, ca, cb);
        below = m;
    }
    atomicOr(err, DERR_PASS_CAP);
    return 0;
}

}  // namespace psi

#endif
