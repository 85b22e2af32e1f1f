"""Mersenne numbers by the order of 2 (the tiles of ranks in
cutrialdive_gb300/csrc/ctd_rank.cuh) against the oracle and the term-by-term
walk: small primes with many hits, both products around 2^40, the longest index
range of the table, and lengths around the choice."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def run(eng, job, variant):
    t = {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096, "segment_log2": 0,
         "variant": variant}
    eng.set_tuning(job.family, t)
    try:
        buf = ctd.factors_buffer.empty(job.n0, job.n1 - job.n0, job.max_factors)
        eng.run_plain(job, buf)
        return str(buf.to_factoring_results())
    finally:
        eng.set_tuning(job.family, None)


@pytest.mark.parametrize("n0,n1,f0,f1", [
    (1, 9001, 3, 5000),
    (700, 9700, 3, 1 << 16),
    (1, 40001, 1 << 20, (1 << 20) + (1 << 17)),
    (12345, 62345, (1 << 31) + 1, (1 << 31) + (1 << 17)),
    (3, 20003, (1 << 40) - (1 << 15), (1 << 40) + (1 << 15)),
    (1, 30001, (1 << 60) + 1, (1 << 60) + (1 << 14)),
    (2, 1 << 20, 1 << 33, (1 << 33) + (1 << 11)),
])
def test_orders_match_oracle_and_walk(eng, n0, n1, f0, f1):
    job = ctd.CtdJob(O.MERSENNE, 32, 0, n0, n1, f0, f1)
    want = O.trial_factor(O.MERSENNE, 0, n0, n1, f0, f1, 32, threads=1).format()
    assert run(eng, job, 0) == want
    assert run(eng, job, 1) == want


@pytest.mark.parametrize("terms", [1000, 1030, 4000, 5200, 8192, 9000])
@pytest.mark.parametrize("n0", [0, 1])
def test_lengths_around_the_choice(eng, n0, terms):
    job = ctd.CtdJob(O.MERSENNE, 32, 0, n0, n0 + terms, 3, 1 << 18)
    assert run(eng, job, 0) == run(eng, job, 1)
