// spread.h -- how the cooperative solver kernels (solve_kernels.cu) spread a
// game's vertices over threads.  Host code without CUDA.
#ifndef PSI_SPREAD_H
#define PSI_SPREAD_H

#include <cstdint>

namespace psi {

constexpr int kSolveThreads = 1024;   // the most per block
constexpr int kMinThreads = 128;

// Threads per block that spread n vertices evenly over all SMs, at least
// kMinThreads (n = 10^4: 0.63 ms per solve in ten blocks of 1,024, 0.53 ms in 79
// of 128), and over as few vertices per thread as the SMs hold, evenly too: the
// same for all threads, where blocks of 1,024 left SMs or most threads of the
// last round idle (us per solve at 10^5, 1.8*10^5, 2^18, 3.5*10^5, 10^6 vertices:
// 859, 1256, 1376, 1270, 4030 -> 801, 1123, 1307, 1228, 3990).  one_each: past so
// many vertices per SM two per thread are better than one.  k_solve's are from
// 600 (1.5*10^5: 1080 -> 1023; 10^5: 801 -> 771; 9*10^4 the same; three per thread
// lose: 2^18 1307 -> 1500); a single evaluation's are not (15 to 20 calls at
// 1.2*10^5: 2.58 -> 2.74 ms).
constexpr int kOneEach = 600;
// (no vertices: the least)
inline int spread_threads(int64_t n, int sms, int one_each)
{
    if (n <= 0) return kMinThreads;
    auto parts = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
    int64_t each = parts(n, (int64_t)kSolveThreads * sms);
    if (each == 1 && n > (int64_t)one_each * sms) each = 2;
    const int64_t threads = 32 * parts(parts(n, sms * each), 32);
    return (int)(threads > kMinThreads ? threads : kMinThreads);
}

}  // namespace psi

#endif
