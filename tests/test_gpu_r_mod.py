"""r_mod (ctd_arith.cuh), 2^64 mod p by two single-precision quotients, run on the
device against Python's integers: odd p at the bounds of that form, 2^31 and
2^62, around every power of 2, and at random widths."""
import os
import random
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_r_mod(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "r_mod")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-o", exe,
                           os.path.join(HERE, "r_mod_device_check.cu")])
    rnd = random.Random(4)
    ps = [3, 5, 7, 2**64 - 59, 2**64 - 1]
    ps += [2**b + d for b in range(4, 64) for d in range(-15, 16, 2)]
    ps += [2**b + d for b in (31, 62) for d in range(-4001, 4002, 2)]
    ps += [2**b * m // 16 | 1 for b in range(31, 62) for m in range(17, 32)]
    ps += [rnd.getrandbits(b) | 1 | 1 << (b - 1) for b in range(3, 65) for _ in range(3000)]
    out = subprocess.run([exe], input="\n".join(map(str, ps)), capture_output=True, text=True, check=True)
    assert list(map(int, out.stdout.split())) == [2**64 % p for p in ps]
