// Rules that the kernels share with the host, run on the host alone.
#include <cstdio>
#include <cstring>

#include "device_common.cuh"

using namespace psi;

// The word a launch's first phase votes in, after launches of p barriers each
// with more than 2^32 barriers in all: one past the last launch's last one.
static int phases()
{
    const uint32_t launches[] = {1, 2, 1u << 31, 5, (1u << 31) - 3, 1, 7, 1u << 31, 1u << 31, 4};
    uint32_t kept = 0;
    unsigned long long all = 0;
    for (uint32_t p : launches) {
        uint32_t phase = kept;
        phase += p;
        kept = kept_phase(phase);
        all += p;
        if (kept % 3 != all % 3) {
            std::printf("after %llu barriers word %u, not %llu\n", all, kept % 3, all % 3);
            return 1;
        }
    }
    return 0;
}

// Whether an evaluation with this number before it, and everything else in
// favour of a patch, is a patch.
static int patch_after(uint32_t epoch)
{
    EvalGates g;
    g.try_patch = 1;
    g.ccount = 3;
    g.mfrom[0] = 7;
    int32_t ucount = 2, quiet = 0;
    unsigned long long sw[4] = {0, 0, 0, 0};
    PatchArgs a;
    a.g = &g;
    a.ucount = &ucount;
    a.quiet = &quiet;
    a.epoch = &epoch;
    a.sw = sw;
    a.n = 100;
    a.acap = a.ccap = 10;
    a.ucap = 110;
    patch_begin(a);
    if (g.eval == g.patch || (g.eval && (ucount != 0 || g.mfrom[0] != 0))) return -1;
    return g.patch;
}

// The evaluation numbered 0 is a full one, whatever the round; others may be
// patches.
static int numbers()
{
    const uint32_t last = kEpochMask;
    const struct { uint32_t before; int patch; } want[] = {
        {0, 1}, {1, 1}, {last - 1, 1}, {last, 0}, {last + 1, 1}, {2 * last + 1, 0}, {UINT32_MAX, 0}, {UINT32_MAX - 1, 1}};
    for (const auto &w : want)
        if (patch_after(w.before) != w.patch) {
            std::printf("after number %u: %d, not %d\n", w.before, patch_after(w.before), w.patch);
            return 1;
        }
    return 0;
}

int main(int argc, char **argv)
{
    if (argc > 1 && !std::strcmp(argv[1], "phases")) return phases();
    if (argc > 1 && !std::strcmp(argv[1], "numbers")) return numbers();
    return 2;
}
