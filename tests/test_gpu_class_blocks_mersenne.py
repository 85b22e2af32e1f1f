"""The walk over power-residue classes for Mersenne numbers at the lengths where
its form changes (as test_gpu_class_blocks.py has it for Proth and Riesel
numbers).  A plain run takes such ranges by the orders of 2; a list of primes in
the caller's memory goes by classes."""
import numpy as np
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def run(eng, primes, n0, terms, slots, variant):
    torch = pytest.importorskip("torch")
    L = ctd.load_native()
    eng.set_tuning(O.MERSENNE, {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 1 << 20,
                                "segment_log2": 0, "variant": variant, "classify_min": 1})
    try:
        job = ctd.CtdJob(O.MERSENNE, slots, 0, n0, n0 + terms, int(primes.min()), int(primes.max()) + 1)
        d = torch.from_numpy(primes.view(np.int64)).cuda()
        counts = torch.zeros(terms, dtype=torch.int32, device="cuda")
        factors = torch.zeros((terms, slots), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        before = L.ctd_kernel_launches()
        assert L.ctd_residues_device(eng.handle, job, d.data_ptr(), d.numel(), counts.data_ptr(), factors.data_ptr(),
                                     None) == 0
        assert L.ctd_kernel_launches() - before == (1 if variant else 13)  # the walk; the classes
        torch.cuda.synchronize()
        return counts.cpu().numpy(), np.sort(factors.cpu().numpy(), axis=1)
    finally:
        eng.set_tuning(O.MERSENNE, None)


def check(eng, primes, n0, terms, slots=32):
    fast, walk = (run(eng, primes, n0, terms, slots, v) for v in (0, 1))
    assert np.array_equal(fast[0], walk[0]) and np.array_equal(fast[1], walk[1]), (n0, terms, primes[0])


@pytest.mark.parametrize("terms", [1, 63, 64, 65, 511, 512, 513, 2559, 2560, 2561, 2689, 9000, 40001])
def test_lengths(eng, terms):
    for n0, f0, f1 in ((1, 3, 3000), (777, (1 << 20) + 1, (1 << 20) + 20000), (5, (1 << 40) - 30000, (1 << 40) + 30000)):
        check(eng, eng.sieve(f0, f1), n0, terms)


def test_long_lists(eng):
    for f0, f1 in (((1 << 33) + 1, (1 << 33) + 8000), ((1 << 62) - 9000, (1 << 62) + 3000)):
        check(eng, eng.sieve(f0, f1), 11, 400000)
    check(eng, eng.sieve(101, 20000), 11, 300000, 512)
