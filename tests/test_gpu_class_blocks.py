"""The walk over power-residue classes (run_doubling_class, class_blocks in
cutrialdive_gb300/csrc/ctd_residue.cu) at the lengths where its form changes --
term by term below 64 class terms, blocks of 32 without and with the filter,
blocks of 64 from 2560 -- with every range classified, against the
term-by-term walk."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def run(eng, job, variant):
    t = {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 1 << 20, "segment_log2": 0,
         "variant": variant, "classify_min": 1}
    eng.set_tuning(job.family, t)
    try:
        buf = ctd.factors_buffer.empty(job.n0, job.n1 - job.n0, job.max_factors)
        eng.run_plain(job, buf)
        return str(buf.to_factoring_results())
    finally:
        eng.set_tuning(job.family, None)


@pytest.mark.parametrize("terms", [1, 63, 64, 65, 511, 512, 513, 2559, 2560, 2561, 2689, 9000, 40001])
@pytest.mark.parametrize("family,param", [(O.PROTH, 3), (O.RIESEL, 12345), (O.MERSENNE, 0)])
def test_lengths(eng, family, param, terms):
    for n0, f0, f1 in ((1, 3, 3000), (777, (1 << 20) + 1, (1 << 20) + 20000), (5, (1 << 40) - 30000, (1 << 40) + 30000)):
        job = ctd.CtdJob(family, 32, param, n0, n0 + terms, f0, f1)
        assert run(eng, job, 0) == run(eng, job, 1), (n0, f0)


# class moduli on both sides of 32, where a block's targets change from an M-bit
# reduction to the Shoup product: only lists this long give classes of 2560
# terms and more with such moduli
@pytest.mark.parametrize("family,param", [(O.PROTH, 3), (O.RIESEL, 12345), (O.MERSENNE, 0)])
def test_long_lists(eng, family, param):
    for f0, f1 in (((1 << 33) + 1, (1 << 33) + 8000), ((1 << 62) - 9000, (1 << 62) + 3000)):
        job = ctd.CtdJob(family, 32, param, 11, 400011, f0, f1)
        assert run(eng, job, 0) == run(eng, job, 1), f0
    job = ctd.CtdJob(family, 512, param, 11, 300011, 101, 20000)
    assert run(eng, job, 0) == run(eng, job, 1)
