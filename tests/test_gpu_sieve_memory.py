"""The device sieve keeps 8 bytes a base prime for the primes' first multiples.
Where the device has no room for them the windows find the multiples themselves:
the same primes, no error.  Checked just above 2^60 (54 million base primes, 435
MB of first multiples) with the device's free memory filled but for 512 MiB, which
hold the base primes and the windows; prime lists and factors are integers, the
comparison is exact."""
import numpy as np
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu

LO, HI = (1 << 60) + 1, (1 << 60) + (1 << 21)


def factors(eng, batched):
    job = ctd.CtdJob(O.PROTH, 32, 3, 1, 2001, LO, LO + (1 << 16))
    buf = ctd.factors_buffer.empty(1, 2000, 32)
    if batched:
        eng.batch_run([job], [buf])
    else:
        eng.run_plain(job, buf)
    return str(buf.to_factoring_results())


def test_sieve_without_room_for_the_first_multiples():
    torch = pytest.importorskip("torch")
    room = ctd.Engine(0)
    try:
        want = room.sieve(LO, HI), factors(room, False), factors(room, True)
    finally:
        room.close()
    eng = ctd.Engine(0)
    try:
        free, _ = torch.cuda.mem_get_info()
        filler = torch.empty(free - (512 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = eng.sieve(LO, HI), factors(eng, False), factors(eng, True)
            assert torch.cuda.mem_get_info()[0] < 435 << 20
        finally:
            del filler
            torch.cuda.empty_cache()
        again = eng.sieve(LO, HI), factors(eng, False), factors(eng, True)
    finally:
        eng.close()
    for x in (got, again):
        assert np.array_equal(x[0], want[0]) and x[1:] == want[1:]
