// Host-side check of half_power (ctd_arith.cuh): reads "p x" lines, prints
// 2^-x mod p by the general product and, below 2^40, by the narrow one.
#include <cinttypes>
#include <cstdio>

#include "../cutrialdive_gb300/csrc/ctd_arith.cuh"

int main()
{
    unsigned long long p, x;
    while (std::scanf("%llu %llu", &p, &x) == 2) {
        const uint64_t pinv = ctd::Mont::neg_inverse(p), r = ctd::half_power<false>(p, pinv, x);
        std::printf("%" PRIu64 " %" PRIu64 "\n", r, p < ctd::MONT_NARROW_LIMIT ? ctd::half_power<true>(p, pinv, x) : r);
    }
    return 0;
}
