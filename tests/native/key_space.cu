// Key-space shifts of every side around the powers of two, up to the largest int: exits 1 at a wrong one.
#include "be_api_internal.h"

#include <cstdio>

int main()
{
    for (int k = 0; k <= 30; ++k)
        for (int64_t v = (int64_t(1) << k) - 1; v <= (int64_t(1) << k) + 1; ++v) {
            if (v < 1) continue;
            const int want = v <= 1 ? 0 : 64 - __builtin_clzll(uint64_t(v - 1));
            if (be::ceil_log2(int(v)) != want) {
                std::printf("%lld: %d, not %d\n", (long long)v, be::ceil_log2(int(v)), want);
                return 1;
            }
        }
    return be::ceil_log2(2147483647) == 31 ? 0 : 1;
}
