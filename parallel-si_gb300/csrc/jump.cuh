// jump.cuh -- pointer jumping without barriers over 16-byte window records
// (described in solve_kernels.cu), for the kernels that evaluate by it.
#ifndef PSI_JUMP_CUH
#define PSI_JUMP_CUH

#include <climits>

#include "device_common.cuh"

namespace psi {

// targets of finished records
constexpr int32_t kSink = -1, kNegInf = -2, kPosInf = -3;
// reads per vertex and pass
constexpr int kJumps = 64;
constexpr int kMaxPasses = 64;
// a record's last word with FLAGS: the window's length (up to kMaxLen: n or
// more only say "a cycle"; n < 2^20), whether a strategy in it has changed
// since the last evaluation, and, once finished, since Even's last examination
constexpr int32_t kMaxLen = 1 << 24, kLen = (1 << 25) - 1;
constexpr int32_t kNew = 1 << 30, kNewEven = 1 << 29;
// without: the length alone (any n)
constexpr int32_t kMaxPlain = 1 << 30;

// One pass of v's record r; true when it is finished.
// q: its target's record, if it has one.
template <bool FLAGS>
__device__ __forceinline__ bool jump_pass(int4 *jump, int32_t n, int32_t v, int4 &r, int4 q)
{
    constexpr int32_t most = FLAGS ? kMaxLen : kMaxPlain, mask = FLAGS ? kLen : INT_MAX;
    if (r.x < 0) return true;
    int32_t mark = v;
    for (int i = 1; i <= kJumps; i++) {
        bool cycle = (r.w & mask) >= n;
        if (!cycle) {
            if (i > 1) q = load_whole(&jump[r.x]);
            if (q.x <= kNegInf) {
                r = make_int4(q.x, 0, 0, 0);
                store_whole(&jump[v], r);
                return true;
            }
            top1_merge(r.y, r.z, q.y, q.z);
            r.z = min(r.z, most);
            const int32_t len = (int32_t)min((uint32_t)(r.w & mask) + (uint32_t)(q.w & mask), (uint32_t)most);
            r.w = FLAGS ? len | (r.w & kNewEven) | ((r.w | q.w) & kNew) : len;
            r.x = q.x;
            cycle = r.x == mark;
            if ((i & (i - 1)) == 0) mark = r.x;
        }
        if (cycle) {
            // the target is on the cycle: the top priority of the windows from
            // it, once around or n vertices
            const int32_t t0 = r.x;
            int32_t t = t0, len = 0, top = -1, code = 0;
            for (int j = 0; j < kJumps; j++) {
                const int4 q = load_whole(&jump[t]);
                if (q.x <= kNegInf) {
                    code = q.x;
                    break;
                }
                top = max(top, q.y);
                len = (int32_t)min((uint32_t)len + (uint32_t)(q.w & mask), (uint32_t)most);
                t = q.x;
                if (t == t0 || len >= n) {
                    code = (top & 1) ? kNegInf : kPosInf;
                    break;
                }
            }
            if (code) {
                r = make_int4(code, 0, 0, 0);
                store_whole(&jump[v], r);
                return true;
            }
            r.w = most | (r.w & ~mask);   // a later pass goes on from the cycle
            store_whole(&jump[v], r);
            return false;
        }
        if (FLAGS && r.x == kSink && (r.w & kNew)) r.w |= kNewEven;
        store_whole(&jump[v], r);
        if (r.x == kSink) return true;
    }
    return false;
}

}  // namespace psi

#endif
