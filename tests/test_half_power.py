"""half_power (ctd_arith.cuh), 2^-x mod p, run on the host against Python's
integers: every x below 200 and the edges of longer ones, primes of every width
including those above 2^63."""
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_half_power(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "half_power")
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "half_power_host_check.cu")])
    rnd = random.Random(8)
    ps = [3, 5, 7, 2**31 - 1, 2**32 + 15, 2**40 - 87, 2**40 + 15, 2**61 - 1, 2**63 - 25, 2**63 + 29, 2**64 - 59]
    ps += [rnd.getrandbits(b) | 1 | 1 << (b - 1) for b in range(3, 65) for _ in range(3)]
    xs = list(range(200)) + [2**k + d for k in (8, 14, 17, 20, 33, 63) for d in (-1, 0, 1)] + [2**64 - 1]
    cs = [(p, x) for p in ps for x in xs]
    out = subprocess.run([exe], input="".join(f"{p} {x}\n" for p, x in cs), capture_output=True, text=True, check=True)
    got = [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    want = [pow(pow(2, -1, p), x, p) for p, x in cs]
    assert got == [(w, w) for w in want]
