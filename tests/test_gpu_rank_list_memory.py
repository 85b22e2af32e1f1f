"""The tiles of ranks (Fibonacci, Lucas, Mersenne) hand the primes whose rank is
left to take to a list in device memory.  Where the device has no room for the
list -- or only an earlier, shorter call's list is there -- the tiles finish the
primes themselves: the same factors, no error.  The device's free memory is
filled as in test_gpu_class_memory.py; the comparison with the term-by-term walk
is exact."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu

SEG = 1 << 29
# the segment has 23.8 million primes and more (p / ln p, ln p < 22.5): the list
# for them takes (2^20 + an eighth of them) times 24 bytes, 92 MiB
LIST_BYTES = 24 * ((1 << 20) + SEG * 2 // 45 // 8)
ROOM = 48 << 20


def run(eng, family, variant, f0, f1):
    t = eng.get_tuning(family)
    t["variant"] = variant
    eng.set_tuning(family, t)
    try:
        job = ctd.CtdJob(family, 32, 0, 1, 5001, f0, f1)
        buf = ctd.factors_buffer.empty(1, 5000, 32)
        eng.run_plain(job, buf, segment_length=SEG)
        return buf
    finally:
        eng.set_tuning(family, None)


@pytest.mark.parametrize("family", [O.FIBONACCI, O.LUCAS, O.MERSENNE])
@pytest.mark.parametrize("shorter_first", [False, True])
def test_ranks_without_room_for_their_list(family, shorter_first):
    torch = pytest.importorskip("torch")
    eng = ctd.Engine(0)
    try:
        # the walk first: the engine's other buffers at full size
        walk = run(eng, family, 1, 1 << 32, (1 << 32) + SEG)
        if shorter_first:  # a list for some thousand primes, which stays in use
            run(eng, family, 0, 1 << 32, (1 << 32) + (1 << 16))
        free, _ = torch.cuda.mem_get_info()
        filler = torch.empty(free - ROOM, dtype=torch.uint8, device="cuda")
        try:
            assert torch.cuda.mem_get_info()[0] < LIST_BYTES
            auto = run(eng, family, 0, 1 << 32, (1 << 32) + SEG)
        finally:
            del filler
            torch.cuda.empty_cache()
        assert auto.counts.tolist() == walk.counts.tolist()
        assert str(auto.to_factoring_results()) == str(walk.to_factoring_results())
        assert walk.counts.any()
    finally:
        eng.close()


@pytest.mark.parametrize("family", [O.FIBONACCI, O.LUCAS, O.MERSENNE])
def test_small_primes_without_room_for_their_list(family):
    """Nearly every prime below 2^20 is listed, many with hundreds of hits."""
    torch = pytest.importorskip("torch")
    warm = ctd.Engine(0)  # loads the kernels, which takes device memory too
    run(warm, family, 0, 3, 1 << 20)
    warm.close()
    eng = ctd.Engine(0)
    try:
        walk = run(eng, family, 1, 3, 1 << 20)
        # the list for 82,000 primes and the one for many hits take 3.4 MiB, two
        # pages of 2 MiB; less than that is left
        page = 2 << 20
        filler = torch.empty((torch.cuda.mem_get_info()[0] // page - 1) * page, dtype=torch.uint8, device="cuda")
        try:
            auto = run(eng, family, 0, 3, 1 << 20)
        finally:
            del filler
            torch.cuda.empty_cache()
        assert str(auto.to_factoring_results()) == str(walk.to_factoring_results())
    finally:
        eng.close()
