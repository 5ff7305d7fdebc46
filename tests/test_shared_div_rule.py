"""Which views take the reference's divisions from shared reciprocals.

The reciprocals hold while Sigma and |Delta| lie in [2^-20, 2^31] (Kerr) or
r^2 |f| in [2^-40, 2^40] (Schwarzschild); a step outside is taken a second time
with compiled divisions.  With escape at 200 M a view of the reference's
default mass lies inside; holes so large or so small that their rays spend most
of their steps outside are not to try.
"""

from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CASES = {  # (metric, log2 M): holds
    ("KERR", 0): True, ("KERR", 7): True, ("KERR", 9): False, ("KERR", -10): True, ("KERR", -16): False,
    ("KERR", -20): False, ("SCHWARZSCHILD", 0): True, ("SCHWARZSCHILD", 10): True, ("SCHWARZSCHILD", 15): False,
    ("SCHWARZSCHILD", -20): True, ("SCHWARZSCHILD", -27): False,
}


def test_rule_covers_both_ends(tmp_path):
    from singularity_gb300 import build as B
    lines = "".join(f"row(SGX_METRIC_{m}, {k});\n" for m, k in CASES)
    src = tmp_path / "rule.cu"
    src.write_text('#include <cmath>\n#include <cstdio>\n#include "sgx_device.cuh"\n'
                   "void row(unsigned metric, int k) {\n"
                   "    const float M = std::ldexp(1.0f, k);\n"
                   "    sgx_uniforms u{};\n"
                   "    u.metric_type = metric; u.mass_M = M; u.spin_a = 0.6f * M; u.rs = 2.0f * M;\n"
                   "    u.cam_pos.x = 30.0f * M; u.escape_r = 200.0f * M; u.horizon_cut = 1.02f * u.rs;\n"
                   '    std::printf("%d ", int(sgxd::shared_div_holds(u)));\n'
                   "}\nint main() {\n" + lines + "}\n")
    exe = tmp_path / "rule"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(src), "-o", str(exe)], check=True, capture_output=True)
    got = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert [bool(int(x)) for x in got] == list(CASES.values())
