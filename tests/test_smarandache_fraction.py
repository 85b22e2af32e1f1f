"""smarandache_fraction (ctd_smarandache.cuh), Sm_b(s) = N / Q mod p without an
inverse, run on the host against Sm_b(s) from Python's integers."""
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def residues(base, wanted, p):
    out, x, m = {}, 0, base
    for n in range(max(wanted) + 1):
        if n:
            m = m * base if n == m else m
            x = (x * m + n) % p
        if n in wanted:
            out[n] = x
    return out


def test_fraction(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "fraction")
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "-o", exe,
                           os.path.join(HERE, "smarandache_fraction_host_check.cu")])
    rnd = random.Random(3)
    cases, want = [], []
    for p in (2**30 + 3, 2**31 - 1, 2**34 + 25, 2**40 - 87, 2**40 + 15, 2**43 - 57):
        for base in (2, 3, 7, 10, 13, 16, 64):
            ends = [base**d + e for d in range(1, 6) for e in (-1, 0, 1) if base**d < 30000]
            wanted = sorted({0, 1, 2, 20001, rnd.randrange(30000)} | set(ends))
            for s, x in residues(base, set(wanted), p).items():
                cases.append((p, base, s))
                want.append(x)
    out = subprocess.run([exe], input="".join("%d %d %d\n" % c for c in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    got = list(map(int, out))
    for i, ((p, base, s), x) in enumerate(zip(cases, want)):
        for n, q in (got[4 * i: 4 * i + 2], got[4 * i + 2: 4 * i + 4]):
            assert q % p and n * pow(q, -1, p) % p == x, (p, base, s)
