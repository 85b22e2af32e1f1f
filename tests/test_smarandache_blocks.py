"""Smarandache blocks (smarandache_blocks32, smarandache_blocks64 in
cutrialdive_gb300/csrc/ctd_residue.cu) against the oracle: every block length,
the edges of digit classes and groups, and the primes where the arithmetic
changes."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def check(eng, base, n0, n1, f0, f1):
    job = ctd.CtdJob(O.SMARANDACHE, 32, base, n0, n1, f0, f1)
    buf = ctd.factors_buffer.empty(n0, n1 - n0, 32)
    eng.run_plain(job, buf)
    want = O.trial_factor(O.SMARANDACHE, base, n0, n1, f0, f1, 32, threads=1).format()
    assert str(buf.to_factoring_results()) == want


# multipliers M: 100 (J = 4 below 2^30), 1000 (3), 729, 23 * 10^3 around the
# limit of J = 2 above 2^30, up to 2^20 and past it
@pytest.mark.parametrize("base,n0,n1", [(10, 5, 140), (10, 95, 1100), (9, 90, 800), (2, 1, 300), (16, 4000, 4300),
                                        (13, 2100, 2400), (7, 2390, 2420), (7, 20001, 20101), (2, 9000, 18000),
                                        (10, 99_990, 100_100), (3, 177_000, 177_200)])
@pytest.mark.parametrize("f0,f1", [(3, 2000), ((1 << 30) - 1500, (1 << 30) + 1500), ((1 << 34) - 700, (1 << 34) + 700),
                                   ((1 << 52) - 400, (1 << 52) + 400)])
def test_bases_and_primes(eng, base, n0, n1, f0, f1):
    check(eng, base, n0, n1, f0, f1)


@pytest.mark.parametrize("terms", [1, 2, 3, 7, 8, 9, 12, 13, 16, 17, 31, 32, 33, 34, 40, 41, 65])
@pytest.mark.parametrize("base,n0", [(10, 20), (10, 300), (11, 5000), (5, 20000)])
def test_lengths(eng, base, n0, terms):
    check(eng, base, n0, n0 + terms, 3, 1000)
    check(eng, base, n0, n0 + terms, (1 << 30) - 500, (1 << 30) + 500)


@pytest.mark.parametrize("base", [2, 7, 10, 13])
def test_bases_that_divide(eng, base):
    # primes that divide the base or one less, with the range below them
    check(eng, base, 1, 3, 3, 100)
    check(eng, base, 1, 2200, 3, 50)
