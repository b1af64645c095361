// Prints spread_threads(n, sms, one_each) for every line "n sms one_each" of
// the input.
#include <cstdio>

#include "spread.h"

int main()
{
    long long n;
    int sms, one;
    while (std::scanf("%lld %d %d", &n, &sms, &one) == 3) std::printf("%d\n", psi::spread_threads(n, sms, one));
    return 0;
}
