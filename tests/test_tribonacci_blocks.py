"""The tribonacci blocks around a centre (trib_block, trib_jump, TribShape in
cutrialdive_gb300/csrc/ctd_residue.cu): the bounds and the jump's constants in
the source against the recurrence, and the kernel against the oracle at the
edges of blocks and of the primes they take."""
import os
import re

import pytest

import cutrialdive_gb300 as ctd
import oracle as O

SRC = open(os.path.join(os.path.dirname(__file__), "..", "cutrialdive_gb300", "csrc", "ctd_residue.cu")).read()


@pytest.mark.parametrize("width,ratio", [(40, 1 + 2 ** -8), (36, 1 + 2 ** -4)])
def test_bounds_and_constants(width, ratio):
    back, ahead, behind, most = map(int, re.search(rf"Trib{width} = TribShape<(\d+), (\d+), (\d+), (\d+)>", SRC).groups())
    rows = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]  # T(c + i) in terms of T(c), T(c+1), T(c+2)
    for _ in range(ahead):
        rows.append(tuple(sum(r[i] for r in rows[-3:]) for i in range(3)))
    before = rows[:3]
    for _ in range(back):
        before.insert(0, tuple(before[2][i] - before[1][i] - before[0][i] for i in range(3)))
    terms = rows + before
    # X = k p with 0 <= x_i <= p ratio
    assert -min(sum(min(c, 0) for c in r) for r in terms) * ratio <= behind
    assert max(sum(max(c, 0) for c in r) for r in terms) * ratio < most + 1
    block = back + 3 + ahead
    while len(rows) < 3 + block:
        rows.append(tuple(sum(r[i] for r in rows[-3:]) for i in range(3)))
    t = [0, 0, 1]
    while len(t) < 60:
        t.append(sum(t[-3:]))
    for n in (block, block + 1, block + 2):
        assert rows[n] == (t[n - 1], t[n - 1] + t[n - 2], t[n])  # trib_jump's constants
        # X < 2^64, and X 2^-32 + p is at most p ratio again
        assert sum(rows[n]) * ratio * 2 ** width < 2 ** 64 and sum(rows[n]) * ratio / 2 ** 32 + 1 <= ratio


@pytest.mark.gpu
@pytest.mark.parametrize("terms", [1, 2, 3, 15, 16, 18, 19, 20, 22, 25, 26, 27, 30, 31, 32, 63, 1000])
@pytest.mark.parametrize("n0,f0,f1", [(0, 3, 700), (1, 3, 3000), (77, 1 << 20, (1 << 20) + 3000),
                                      (5, (1 << 36) - 3000, (1 << 36) + 3000), (3, (1 << 40) - 3000, (1 << 40) + 3000)])
def test_block_edges(eng, n0, terms, f0, f1):
    job = ctd.CtdJob(O.TRIBONACCI, 32, 0, n0, n0 + terms, f0, f1)
    want = O.trial_factor(O.TRIBONACCI, 0, n0, n0 + terms, f0, f1, 32, threads=1).format()
    try:
        for variant in (0, 1):  # blocks, and the walk they replace
            eng.set_tuning(O.TRIBONACCI, {"block_size": 256, "ctas_per_sm": 0, "items_per_thread": 8, "min_tile": 4096,
                                          "segment_log2": 0, "variant": variant})
            buf = ctd.factors_buffer.empty(n0, terms, 32)
            eng.run_plain(job, buf)
            assert str(buf.to_factoring_results()) == want
    finally:
        eng.set_tuning(O.TRIBONACCI, None)
