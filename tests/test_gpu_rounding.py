"""The kernels' quotients, reciprocals and roots where they are hardest.

tests/rounding_check.cu runs tests/division_check.cu with every launch and copy
checked and counts what it compares itself.

* Quotients of the shared reciprocals are the compiled ones bit for bit for
  numerators of 2^-102 and more, for every divisor also the quotients within
  seven of the smallest distances from the midpoint of two floats; x / 6 likewise from 2^-102 (FP32) and 2^-968
  (FP64).
* Smaller numerators lose part of their remainder, so a quotient may be off by
  one unit in its last place: with radii from 2.1 M and sin(theta) above 0.05 the
  divisors are 2^-13 and more, which is 2^-112 for each of six quotients.  Steps
  with momenta down to the subnormals therefore give the same positions, and
  momenta within 2^-100.
* The SFU's 20-bit reciprocal and reciprocal root are within 2^-19 (2^-20 by the
  bits of the operand that they read, 2^-20 by those that they return); one
  cubic step leaves 2^-57, 0.0625 units in the last place, beside the last
  rounding's 0.5, two quadratic ones of the root less: 0.57 in all.
* A root is the library's within one unit in the last place, of subnormals,
  infinity and negative numbers too.
* A difference that is not finite makes the FP64 error norm 1e30, whatever sign a
  NaN has.
"""

from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
HARD, SIXTH_F, SIXTH_D, TINY_KERR, TINY_SCHW, ROOTS, NORM = range(7)


def _build(tmp_path):
    from singularity_gb300 import build as B
    exe = tmp_path / "rounding_check"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "rounding_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


def _hard_numerators():
    """How many numerators one launch of the program's hard() has."""
    u64, n = np.uint64, 0
    for t in range(3):
        odd = np.arange((0x800000 >> t) | 1, 0x1000000 >> t, 2, dtype=u64)
        B, inv = odd << u64(t), odd.copy()
        for _ in range(4):
            inv = (inv * ((u64(2) - odd * inv) & u64(0xffffffff))) & u64(0xffffffff)
        for r in (r for r in range(-7, 8, 2) if abs(r) << t <= 7):
            for k in (24, 25):
                low = (u64(-r % (1 << 32)) * inv) & u64((1 << (k - t)) - 1)
                for j in range(1 << t):
                    M = low + u64(j << (k - t))
                    if k == 24:
                        M |= u64(1 << 24)
                    num = B * M + u64((r << t) % (1 << 64))
                    assert not np.any(num & u64((1 << k) - 1))
                    A = num >> u64(k)
                    n += int(np.sum((M >= 1 << 24) & (A >= 0x800000) & (A <= 0xffffff)))
    return n


def test_no_gpu_is_no_pass(tmp_path):
    """Without a device nothing is compared, and the program says so."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("there is a device")
    assert subprocess.run([str(_build(tmp_path))], capture_output=True).returncode != 0


@pytest.mark.gpu
def test_rounding(tmp_path, sgx):
    run = subprocess.run([str(_build(tmp_path))], capture_output=True, text=True, timeout=240)
    assert run.returncode == 0, run.stderr
    old, new = ([int(x) for x in line.split()] for line in run.stdout.strip().splitlines())
    print(old, new)
    assert old[:7] == [0] * 7 and max(old[7:9]) <= 1 and old[9] <= 8
    miss, done, milli = new[0:14:2], new[1:14:2], new[14:]
    assert done[HARD] == 2 * 16 * _hard_numerators()
    assert done[SIXTH_F] == done[SIXTH_D] == 5 << 23
    assert done[TINY_KERR] == done[TINY_SCHW] == 1 << 22
    assert done[ROOTS] == 14 and done[NORM] == 1 << 20
    assert miss == [0] * 7
    assert 450 < min(milli) and max(milli) <= 570
