"""The kernels' divisions by 6, reciprocals and roots.

tests/rounding_check.cu runs tests/division_check.cu with every launch and copy
checked and counts what it compares itself.

* x / 6 is the compiled quotient bit for bit from 2^-102 (FP32) and 2^-968 (FP64).
* The SFU's 20-bit reciprocal and reciprocal root are within 2^-19 (2^-20 by the
  bits of the operand that they read, 2^-20 by those that they return); one
  cubic step leaves 2^-57, 0.0625 units in the last place, beside the last
  rounding's 0.5, two quadratic ones of the root less: 0.57 in all.
"""

from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SIXTH_F, SIXTH_D = range(2)


def _build(tmp_path):
    from singularity_gb300 import build as B
    exe = tmp_path / "rounding_check"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "rounding_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


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
    miss, done, milli = new[0:4:2], new[1:4:2], new[4:]
    assert done[SIXTH_F] == done[SIXTH_D] == 5 << 23
    assert miss == [0] * 2
    assert 450 < min(milli) and max(milli) <= 570
