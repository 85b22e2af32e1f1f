"""Prime lists that ctd_residues_device gets for Fibonacci and Lucas numbers: dense
ones go by tiles of ranks, ones whose tiles are sparse are walked item by item
in a grid of their own.  Lists around the choice (a quarter of the tiles),
against the term-by-term walk; the list is looked over (rank_fit_kernel) and the
walk's kernel launched for every such call."""
import numpy as np
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu

TERMS = 4000
F0 = 1 << 33


def mixed(eng, part):
    """About 8000 primes (tiles of 11), `part` of them 9000 and more apart."""
    near = eng.sieve(F0, F0 + (1 << 18))[:8000]
    far = eng.sieve(F0 + (1 << 18), F0 + (1 << 18) + (1 << 27))[::400]
    n = int(8000 * part)
    return np.concatenate([near[: 8000 - n], far[:n]])


def lists(eng):
    yield from (mixed(eng, part) for part in (0, 0.24, 0.26, 0.5, 1))
    yield np.repeat(mixed(eng, 0)[:4000], 2)
    yield mixed(eng, 0)[:1]
    yield eng.sieve(3, 1 << 16)
    yield eng.sieve((1 << 62) - (1 << 16), (1 << 62) + (1 << 16))
    yield np.random.default_rng(7).permutation(eng.sieve(F0, F0 + (1 << 21)))


@pytest.mark.parametrize("family", [O.FIBONACCI, O.LUCAS])
def test_lists(eng, family):
    torch = pytest.importorskip("torch")
    L = ctd.load_native()
    for primes in lists(eng):
        job = ctd.CtdJob(family, 32, 0, 1, 1 + TERMS, int(primes.min()), int(primes.max()) + 1)
        d = torch.from_numpy(primes.view(np.int64)).cuda()
        got = []
        for variant in (0, 1):
            if variant:
                eng.set_tuning(family, {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096,
                                        "segment_log2": 0, "variant": 1})
            try:
                counts = torch.zeros(TERMS, dtype=torch.int32, device="cuda")
                factors = torch.zeros((TERMS, 32), dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                before = L.ctd_kernel_launches()
                assert L.ctd_residues_device(eng.handle, job, d.data_ptr(), d.numel(), counts.data_ptr(),
                                             factors.data_ptr(), None) == 0
                # look-over, tiles, walk, finish, many hits; or the walk alone
                assert L.ctd_kernel_launches() - before == (1 if variant else 5)
                torch.cuda.synchronize()
                got.append((counts.cpu().numpy(), np.sort(factors.cpu().numpy(), axis=1)))
            finally:
                eng.set_tuning(family, None)
        assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1]), primes[:3]


@pytest.mark.parametrize("block", [64, 512])
@pytest.mark.parametrize("family,f0", [(O.FIBONACCI, 1 << 62), (O.LUCAS, (1 << 62) - (1 << 15)), (O.MERSENNE, 1 << 62),
                                       (O.MERSENNE, (1 << 62) - (1 << 15))])
def test_launch_shapes(family, f0, block):
    """A launch shape has no effect on tiles of ranks; where a range around 2^62 is
    walked instead, one beyond the walk's 256 threads is not an error either."""
    eng = ctd.Engine(0)
    try:
        out = []
        for shape in (0, block):
            eng.set_launch(0, shape)
            buf = ctd.factors_buffer.empty(1, TERMS, 32)
            eng.run_plain(ctd.CtdJob(family, 32, 0, 1, 1 + TERMS, f0, f0 + (1 << 16)), buf)
            out.append(str(buf.to_factoring_results()))
        assert out[0] == out[1]
    finally:
        eng.close()


@pytest.mark.parametrize("block", [64, 512])
@pytest.mark.parametrize("family", [O.FIBONACCI, O.LUCAS])
def test_launch_shapes_of_lists(family, block):
    torch = pytest.importorskip("torch")
    eng = ctd.Engine(0)
    L = ctd.load_native()
    try:
        primes = mixed(eng, 0.5)
        job = ctd.CtdJob(family, 32, 0, 1, 1 + TERMS, int(primes.min()), int(primes.max()) + 1)
        d = torch.from_numpy(primes.view(np.int64)).cuda()
        out = []
        for shape in (0, block):
            eng.set_launch(0, shape)
            counts = torch.zeros(TERMS, dtype=torch.int32, device="cuda")
            factors = torch.zeros((TERMS, 32), dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            assert L.ctd_residues_device(eng.handle, job, d.data_ptr(), d.numel(), counts.data_ptr(),
                                         factors.data_ptr(), None) == 0
            torch.cuda.synchronize()
            out.append((counts.cpu().numpy(), np.sort(factors.cpu().numpy(), axis=1)))
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    finally:
        eng.close()
