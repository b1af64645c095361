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

int main(int argc, char **argv)
{
    if (argc > 1 && !std::strcmp(argv[1], "phases")) return phases();
    return 2;
}
