"""Divisions, reciprocals and square roots of the kernels against the compiler's.

FP32: the shared-reciprocal quotients, the reciprocal behind them and x / 6
give the correctly rounded result, so they equal the compiled division bit for
bit, for every significand of the divisor, and a fixed step that divides so
equals one with compiled divisions, whatever the state.  The precision form's
norm from one component is the norm over all six, bit for bit.  FP64: the Newton reciprocal is
rounded twice (its correction and the sum), the square root likewise: within
1 ulp of the rounded result.  The FP64 norm takes eight such roundings more than
the definition's four: within 8 ulp.
"""

from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def test_divisions_match_the_compilers(tmp_path, sgx):
    from singularity_gb300 import build as B
    exe = tmp_path / "division_check"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(ROOT / "tests" / "division_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    reciprocal, sixth, quotient, edge, kerr, schwarzschild, norm, rcp_ulp, sqrt_ulp, norm_ulp = map(int, out.split())
    print(out)
    assert reciprocal == sixth == quotient == edge == 0
    assert kerr == schwarzschild == norm == 0
    assert rcp_ulp <= 1 and sqrt_ulp <= 1
    assert norm_ulp <= 8
