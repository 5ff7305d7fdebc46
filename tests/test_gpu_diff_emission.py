"""The hand-derived reverse pass of the disc emission against dual numbers.

In FP64 the two differ by rounding alone: a few hundred operations of 1e-16
each, and sums over at most 2,000 rays whose terms cancel by up to 1e3, so the
bound is 1e-9 of the largest component.  The scenes reach the branches of the
colour: both ends of the temperature range, the join of the blackbody
branches, Doppler and redshift off, the disc's bands moving.  The sizes lie at
the edges of a warp and of a block.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCENES = {
    "cold": dict(t_scale=0.2),
    "join": dict(t_scale=0.75),
    "hot": dict(t_scale=4.5),
    "plain": dict(off=("SGX_FLAG_DOPPLER_ON", "SGX_FLAG_REDSHIFT_ON")),
    "no-redshift": dict(off=("SGX_FLAG_REDSHIFT_ON",)),
    "bands": dict(time_sec=7.3, turbulence=1.0),
}


@pytest.fixture(scope="module")
def diff(sgx, renderer):
    from singularity_gb300 import diff as D
    return D.DiffRenderer(renderer)


def _gradients(sgx, diff, u, params, model, precision):
    import torch
    from singularity_gb300 import diff as D
    N, out = sgx._native, []
    for form in (N.DIFF_ADJOINT_REVERSE, N.DIFF_ADJOINT_DUAL):
        img = diff.forward(u, params, D.DiffOptions(precision=precision, model=model, adjoint_form=form))
        seed = torch.linspace(-1.0, 1.0, img.numel(), device="cuda").reshape(img.shape)
        out.append(diff.backward(seed))
        assert np.array_equal(out[-1], diff.backward(seed))  # the records serve any number of backward passes
    return out


@pytest.mark.parametrize("model", [1, 0])
@pytest.mark.parametrize("scene", list(SCENES))
def test_emission_reverse_matches_duals(diff, sgx, scene, model):
    W, N, s = sgx.workloads, sgx._native, SCENES[scene]
    u = W.differentiation_base(48, 32, 1)
    for flag in s.get("off", ()):
        u.flags &= ~getattr(N, flag)
    u.time_sec, u.disc_turbulence = s.get("time_sec", 0.0), s.get("turbulence", u.disc_turbulence)
    p = list(W.differentiation_params(W.differentiation_guess()))
    p[3] = s.get("t_scale", p[3])
    rev, dual = _gradients(sgx, diff, u, p, model, N.PRECISION_FP64)
    print(scene, model, rev, dual)
    assert np.max(np.abs(rev - dual)) <= 1e-9 * np.max(np.abs(dual))


@pytest.mark.parametrize("model", [1, 0])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (33, 1), (43, 3)])
def test_small_launches(diff, sgx, w, h, model):
    W, N = sgx.workloads, sgx._native
    u = W.differentiation_base(w, h, 1)
    p = W.differentiation_params(W.differentiation_guess())
    rev, dual = _gradients(sgx, diff, u, p, model, N.PRECISION_FP64)
    assert np.max(np.abs(rev - dual)) <= 1e-9 * np.max(np.abs(dual)) + 1e-300
