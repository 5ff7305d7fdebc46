"""The FP32 backward kernels at the edges of the launch rule.

The sizes are the last rays of a rule and the first of the next: 8 warps on
each of 152 SMs, and the sparse form's change from one-warp to four-warp blocks.  The dense
and the sparse checkpoints replay the same steps in different kernels, so the
gradients differ by FP32 rounding alone: about 300 steps of 6e-8 each, 2e-5 of
the largest component.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [1, 0])
@pytest.mark.parametrize("w,h", [(256, 152), (357, 109), (255, 257), (256, 256)])
def test_dense_matches_sparse_at_the_edges(sgx, renderer, w, h, model):
    import torch
    from singularity_gb300 import diff as D
    W, diff, out = sgx.workloads, D.DiffRenderer(renderer), []
    u = W.differentiation_base(w, h, 1)
    p = W.differentiation_params(W.differentiation_guess())
    for ck in (10, 64):
        img = diff.forward(u, p, D.DiffOptions(model=model, checkpoint_interval=ck))
        out.append(diff.backward(torch.ones_like(img)))
    print(w, h, model, out)
    assert np.max(np.abs(out[0] - out[1])) <= 2e-5 * np.max(np.abs(out[1]))
