"""A batch's view table: every block keeps it in shared memory.

An SM has 228 KB, of which the hardware takes 1 KB a block and the tracer 2,088
bytes beside the table; each view adds three 8-byte offsets and a count to its
row, the set two more offsets and up to 64 sub-pixel offsets.  With 128 threads
a block at 72 (FP32) or 80 registers (precision form), registers allow seven or
six blocks; 100 views are to leave six and 128 views five.
"""

from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_rows_leave_room_for_the_blocks(tmp_path):
    from singularity_gb300 import build as B
    src = tmp_path / "rows.cu"
    src.write_text('#include <cstdio>\n#include "sgx_device.cuh"\n'
                   'int main() { std::printf("%zu %zu\\n", sizeof(sgxd::View<float>), sizeof(sgxd::View<double>)); }\n')
    exe = tmp_path / "rows"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_FLAGS, str(src), "-o", str(exe)], check=True, capture_output=True)
    single, double = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    print(single, double)

    def blocks(views):
        table = views * (single + 28) + 16 + 2 * 64 * 4 + 7 * 15
        return (228 << 10) // (table + 2088 + 1024)

    assert blocks(100) >= 6 and blocks(128) >= 5
    assert double <= 496  # a slot of 512 bytes serves either precision
