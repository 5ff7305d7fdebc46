"""The differentiable form's records at its 16 GiB limit (crossing model).

Every checkpoint slot of 200,000 steps is allocated, few are written, so some
ten thousand rays reach the limit.  The sizes lie just under it: the
records fit, the crossing states behind them do not.  Such a call is served,
within the limit, and its gradient is that of the same rays with 2,000 steps
(all of them end before), whose crossing states are kept: the two form the
same seeds from states that differ by rounding, at most 300 steps of an ulp
each, 2e-5 of the largest component in FP32 and 1e-9 in FP64, where cancelling
sums over the rays lose a few digits more.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 16 << 30


def _bytes(n, steps, ck, size):
    """The records of n rays at one sample a pixel, and their crossing states."""
    def r(x):
        return (x + 255) // 256 * 256
    slots, nx = steps // ck + 1, 8
    need = (r(slots * 9 * n * size) + r(3 * n * size) + 2 * r(n * 4) + r(nx * n * 4) + r(nx * n * size) +
            r(nx * 3 * n * size) + r(4 * n * 8) + r(2 * size) + 256 + r(4 * ((n + 1023) // 1024) * 8) + 256)
    return need, nx * 7 * n * size


@pytest.mark.parametrize("precision,ck", [("fp32", 10), ("fp32", 64), ("fp64", 64)])
def test_crossing_records_stay_within_the_limit(sgx, precision, ck):
    import torch
    from singularity_gb300 import diff as D
    W, N = sgx.workloads, sgx._native
    size, prec = (8, N.PRECISION_FP64) if precision == "fp64" else (4, N.PRECISION_FP32)
    per_ray = _bytes(1 << 20, 200000, ck, size)[0] / (1 << 20)
    w, h = max(((w, int(LIMIT / per_ray) // w) for w in range(120, 520)), key=lambda s: s[0] * s[1])
    need, states = _bytes(w * h, 200000, ck, size)
    print(w, h, need, states)
    assert need <= LIMIT < need + states
    opts = D.DiffOptions(precision=prec, model=0, checkpoint_interval=ck)
    p = W.differentiation_params(W.differentiation_guess())
    out = []
    for steps in (2000, 200000):
        with sgx.Renderer() as r:
            diff = D.DiffRenderer(r)
            diff.forward(W.differentiation_base(1, 1, 1), p, opts)  # a small allocation of its own
            del_me = [torch.ones((h, w, 3), device="cuda") for _ in range(8)]  # so that torch has its blocks
            del del_me
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            img = diff.forward(W.differentiation_base(w, h, 1, max_steps=steps), p, opts)
            taken = free - torch.cuda.mem_get_info()[0]
            out.append((img.clone(), diff.stats()["steps"], diff.backward(torch.ones_like(img)), taken))
    print(out[0][1:], out[1][1:])
    assert out[1][3] <= LIMIT
    assert out[0][1] == out[1][1] and torch.equal(out[0][0], out[1][0])
    g = [o[2] for o in out]
    assert np.any(g[0] != 0.0)
    assert np.max(np.abs(g[0] - g[1])) <= (1e-9 if precision == "fp64" else 2e-5) * np.max(np.abs(g[0]))
