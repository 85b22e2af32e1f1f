"""Mersenne numbers at primes around 2^62, where the orders of 2 are no longer
taken by tiles, and 2^63, where they are taken prime by prime: the factors as the oracle has them, and the route by the number
of kernels launched -- a classified segment launches 13 (screen, eight
classifications, refinement, ninth powers, regroup, walk), the orders 3."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu

TERMS = 20000


@pytest.mark.parametrize("f0,classified", [((1 << 62) - (1 << 14), False), ((1 << 62) - (1 << 13), True),
                                           (1 << 62, True), ((1 << 63) - (1 << 13), True),
                                           ((1 << 63) + 1, False)])
def test_route_and_factors(eng, f0, classified):
    job = ctd.CtdJob(O.MERSENNE, 32, 0, 1, 1 + TERMS, f0, f0 + (1 << 14))
    eng.sieve(job.f0, job.f1)  # the base primes' own launches
    buf = ctd.factors_buffer.empty(1, TERMS, 32)
    before = ctd.load_native().ctd_kernel_launches()
    eng.run_plain(job, buf)
    launches = ctd.load_native().ctd_kernel_launches() - before
    assert (launches >= 13) == classified
    want = O.trial_factor(O.MERSENNE, 0, 1, 1 + TERMS, job.f0, job.f1, 32, threads=1).format()
    assert str(buf.to_factoring_results()) == want
