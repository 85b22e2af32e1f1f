"""ctd_residues_device for Fibonacci and Lucas numbers (the tiles of ranks) in a
captured CUDA graph: a list longer than any before it, and the graph's replay
after a still longer list made the context's own buffers grow.  Compared with
the term-by-term walk."""
import numpy as np
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu

TERMS = 4000


@pytest.mark.parametrize("family", [O.FIBONACCI, O.LUCAS])
@pytest.mark.parametrize("f0", [3, 1 << 33])
def test_captured_ranks(family, f0):
    torch = pytest.importorskip("torch")
    eng = ctd.Engine(0)
    L = ctd.load_native()
    counts = torch.zeros(TERMS, dtype=torch.int32, device="cuda")
    factors = torch.zeros((TERMS, 32), dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()

    def call(primes):
        job = ctd.CtdJob(family, 32, 0, 1, 1 + TERMS, f0, f0 + (1 << 26))
        return L.ctd_residues_device(eng.handle, job, primes.data_ptr(), primes.numel(), counts.data_ptr(),
                                     factors.data_ptr(), stream.cuda_stream)

    def clear():
        counts.zero_()
        factors.zero_()
        torch.cuda.synchronize()

    def found():
        torch.cuda.synchronize()
        return counts.cpu().numpy(), np.sort(factors.cpu().numpy(), axis=1)

    try:
        lists = [torch.from_numpy(eng.sieve(f0, f0 + (1 << w)).astype(np.int64)).cuda() for w in (12, 18, 22)]
        clear()
        assert call(lists[0]) == 0  # the counters' allocation, and the kernels' loading
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            rc = call(lists[1])
        assert rc == 0, L.ctd_last_error(eng.handle).decode()
        got = []
        for grow in (False, True):
            if grow:
                assert call(lists[2]) == 0
                torch.cuda.synchronize()
            clear()
            graph.replay()
            got.append(found())
        eng.set_tuning(family, {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096,
                                "segment_log2": 0, "variant": 1})
        clear()
        assert call(lists[1]) == 0
        want = found()
        for g in got:
            assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1])
    finally:
        eng.close()
