// Host-side check of smarandache_fraction (ctd_smarandache.cuh): reads
// "p b s" lines, prints N and Q (plain residues) by the general product and,
// below 2^40, by the narrow one.
#include <cinttypes>
#include <cstdio>

#include "../cutrialdive_gb300/csrc/ctd_smarandache.cuh"

template <class MT>
void print(uint64_t p, uint64_t b, uint64_t s)
{
    MT m;
    m.init(p);
    uint64_t N, Q;
    ctd::smarandache_fraction(m, b, s, N, Q);
    std::printf("%" PRIu64 " %" PRIu64 "\n", m.from(N), m.from(Q));
}

int main()
{
    unsigned long long p, b, s;
    while (std::scanf("%llu %llu %llu", &p, &b, &s) == 3) {
        print<ctd::Mont>(p, b, s);
        if (p < ctd::MONT_NARROW_LIMIT)
            print<ctd::MontN>(p, b, s);
        else
            print<ctd::Mont>(p, b, s);
    }
    return 0;
}
