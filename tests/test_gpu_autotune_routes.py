"""The autotuner times what ctd_run_plain launches: ranks and orders where the run
takes them (three kernels; the power-residue classes take 13), whose launch shape
and index tiles are then not searched, and the short index tiles that an untuned
context gives a list shorter than its threads."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def untune(eng, job):
    eng.set_tuning_for(job.family, max(3, job.f0).bit_length(), None)


def run(eng, job):
    buf = ctd.factors_buffer.empty(job.n0, job.n1 - job.n0, job.max_factors)
    eng.run_plain(job, buf)
    return str(buf.to_factoring_results())


@pytest.mark.parametrize("family", [O.MERSENNE, O.FIBONACCI, O.LUCAS])
def test_ranks_and_orders(eng, family):
    job = ctd.CtdJob(family, 32, 0, 1, 9001, 1 << 31, (1 << 31) + (1 << 22))
    want = run(eng, job)  # and every allocation and base prime that the runs need
    launches = ctd.load_native().ctd_kernel_launches
    try:
        # the starting entry only, timed twice (the second time for a shorter
        # sample) in three passes each, and one sieve of four kernels
        before = launches()
        eng.autotune(job, budget_s=1e-9)
        assert launches() - before == 2 * 3 * 3 + 4
        untune(eng, job)
        best = eng.autotune(job, budget_s=0.5)
        shape = {k: best[k] for k in ("block_size", "ctas_per_sm", "items_per_thread", "min_tile", "classify_min", "refine_q")}
        assert shape == {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096, "classify_min": 0,
                         "refine_q": 0}
        assert run(eng, job) == want
    finally:
        untune(eng, job)


def test_short_list(eng):
    """6500 primes for 155,000 threads, each as long as 2000 terms in a tile of its
    own: 0.7 ms in the short tiles that an untuned context takes, 1.7 in tiles of
    1024 terms and more."""
    job = ctd.CtdJob(O.SMARANDACHE, 32, 7, 1, 2001, 3, 1 << 16)
    want = run(eng, job)
    try:
        assert eng.autotune(job, budget_s=2.0)["min_tile"] == 512
        assert run(eng, job) == want
    finally:
        untune(eng, job)
