"""Smarandache blocks where test_smarandache_blocks.py does not reach: multipliers
above 2^20 (one term a block below 2^30, the walks above), multipliers that are 0
or 1 modulo the prime with a whole group of blocks, and every block length with
the general product, from 2^40 to 2^44 where the blocks end.  The reference's multi-limb
Sm(n) takes minutes at n = 10^6, so the residues come from Python's integers."""
import pytest

import cutrialdive_gb300 as ctd
import oracle as O

pytestmark = pytest.mark.gpu


def mat(a, b, p):
    return [[sum(a[i][k] * b[k][j] for k in range(3)) % p for j in range(3)] for i in range(3)]


def sm_at(base, n, p):
    """Sm_base(n) mod p: the steps (S, m, 1) -> (M S + m + 1, m + 1, 1) of each digit
    class by a power of their matrix."""
    vec, lo, M = [0, 0, 1], 1, base
    while lo <= n:
        t = min(n, M - 1) - lo + 1
        a, r = [[M % p, 1, 1], [0, 1, 1], [0, 0, 1]], [[1, 0, 0], [0, 1, 0], [0, 0, 1]]
        while t:
            if t & 1:
                r = mat(a, r, p)
            a = mat(a, a, p)
            t >>= 1
        vec = [sum(r[i][k] * vec[k] for k in range(3)) % p for i in range(3)]
        lo, M = M, M * base
    return vec[0]


def zeros(base, n0, n1, p):
    x, M = sm_at(base, n0, p), base
    for n in range(n0, n1):
        if n > n0:
            while M <= n:
                M *= base
            x = (x * M + n) % p
        if x == 0:
            yield n


def check(eng, base, n0, n1, f0, f1):
    job = ctd.CtdJob(O.SMARANDACHE, 32, base, n0, n1, f0, f1)
    buf = ctd.factors_buffer.empty(n0, n1 - n0, 32)
    eng.run_plain(job, buf)
    factors = buf.factors.reshape(-1, 32)
    got = {(n0 + i, int(p)) for i in range(n1 - n0) for p in factors[i] if p}
    want = {(n, int(p)) for p in O.sieve(max(3, f0), f1) for n in zeros(base, n0, n1, int(p))}
    assert got == want and int(buf.counts.sum()) == len(want)


@pytest.mark.parametrize("base", [2, 7, 10, 64])
def test_reference(base):
    p = (1 << 34) + 25
    x, M = 0, base
    for n in range(1, 400):
        M *= base if n == M else 1
        x = (x * M + n) % p
        assert sm_at(base, n, p) == x


def found(eng, base, n0, n1, f0, f1, variant):
    eng.set_tuning(O.SMARANDACHE, {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096,
                                   "segment_log2": 0, "variant": variant})
    try:
        buf = ctd.factors_buffer.empty(n0, n1 - n0, 32)
        eng.run_plain(ctd.CtdJob(O.SMARANDACHE, 32, base, n0, n1, f0, f1), buf)
    finally:
        eng.set_tuning(O.SMARANDACHE, None)
    f = buf.factors.reshape(-1, 32)
    return {(n0 + int(i), int(f[i, j])) for i, j in zip(*f.nonzero())}, int(buf.counts.sum())


# the last class before 2^20 and the first behind it (10^6 and 10^7; 2^20 and
# 2^21; 64^3 and 64^4), from the one into the other and in the second alone,
# against the steps in Montgomery form; each hit against Python's integers
@pytest.mark.parametrize("base,n0,n1", [(10, 999_000, 1_001_000), (10, 1_000_300, 1_002_500), (10, 990_000, 1_000_040),
                                        (2, (1 << 20) - 2500, (1 << 20) + 60), (2, (1 << 20) + 7, (1 << 20) + 3000),
                                        (64, 260_000, 263_000), (64, 300_000, 302_133)])
def test_multipliers_above_2p20(eng, base, n0, n1):
    hits = 0
    for f0, width in (((1 << 21) - (1 << 18), 1 << 19), ((1 << 29) - (1 << 23), 1 << 24), ((1 << 30) - (1 << 24), 1 << 25),
                      ((1 << 34) - (1 << 26), 1 << 27)):
        got = found(eng, base, n0, n1, f0, f0 + width, 0)
        assert got == found(eng, base, n0, n1, f0, f0 + width, 2), f0
        assert all(sm_at(base, n, p) == 0 for n, p in list(got[0])[:40])
        hits += len(got[0])
    assert hits


# bases 0 and 1 modulo the prime, n below it: 24 terms of three a block are a group
@pytest.mark.parametrize("p", [29, 31, 37, 53, 59, 61])
def test_multipliers_0_and_1(eng, p):
    for base in (p, p + 1):
        if base <= 64:
            check(eng, base, 1, p, p, p + 1)
            check(eng, base, 1, p, 3, 200)


# three, two and one term a block: zeros found by the term-by-term walk, at the
# first, some middle and the last term of an index range
@pytest.mark.parametrize("base,n,p", [
    (28, 774, 1130000954573), (27, 69, 1161702652457), (27, 519, 1100869307221), (28, 269, 4477919777921),
    (27, 394, 4508893168163), (28, 636, 17468456298047),
    (10, 3433, 1104934405921), (10, 4167, 4404292986967), (10, 6209, 4404577251083), (10, 4523, 17574024076243),
    (10, 6921, 17560458395699),
    (7, 46349, 1100768151001), (7, 89853, 1100609051357), (7, 18488, 4402512092599), (7, 61487, 4404613326041),
    (7, 110646, 4403717426561), (7, 35731, 17576385561403),
])
def test_general_product(eng, base, n, p):
    low = max(k for k in (base**d for d in range(8)) if k <= n)  # the class's first term
    for before in (0, 1, 2, 3, 7, 24, 40, 101):
        for after in (1, 2, 35, 90):
            check(eng, base, max(low + 1, n - before), n + after, p - 200, p + 200)


# around the ends of the blocks' primes
@pytest.mark.parametrize("base,n0,n1", [(7, 60, 340), (9, 100, 728), (10, 1100, 3007), (10, 5000, 10_060),
                                        (7, 20_001, 20_333), (2, 9000, 17_000)])
@pytest.mark.parametrize("f0", [1 << 30, 1 << 40, 1 << 42, 1 << 44])
def test_ends(eng, base, n0, n1, f0):
    check(eng, base, n0, n1, f0 - 1200, f0 + 1200)
