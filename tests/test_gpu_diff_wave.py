"""The FP32 backward on both sides of one wave of 8 warps an SM, on this device.

The 10-step checkpoints run 224-register blocks up to that many rays and
168-register ones above; both replay the steps of the 64-step form in other
kernels, so gradients differ by FP32 rounding alone: about 300 steps of 6e-8 each,
2e-5 of the largest component.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [1, 0])
@pytest.mark.parametrize("more", [0, 1])
def test_dense_matches_sparse_at_one_wave(sgx, renderer, more, model):
    import torch
    from singularity_gb300 import diff as D
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    W, diff, out = sgx.workloads, D.DiffRenderer(renderer), []
    u = W.differentiation_base(256, sms + more, 1)
    p = W.differentiation_params(W.differentiation_guess())
    for ck in (10, 64):
        img = diff.forward(u, p, D.DiffOptions(model=model, checkpoint_interval=ck))
        out.append(diff.backward(torch.ones_like(img)))
    print(sms, more, model, out)
    assert np.max(np.abs(out[0] - out[1])) <= 2e-5 * np.max(np.abs(out[1]))
