"""Batches whose views' FP64 constants start at each alignment, and of 128 views.

The precision form reads a view's FP64 constants behind the set's table; the bar
against single-view renders is that of the other batch tests (>= 99.7 % of
values within one level, mean <= 5e-4), since the two kernels contract a few
multiply-adds differently.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["PRECISION_MIXED", "PRECISION_FP32", "PRECISION_FP64"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 128])
def test_views_match_single_renders(sgx, renderer, n, precision):
    rng = np.random.default_rng(n)
    N, views = sgx._native, []
    for _ in range(n):
        sc = sgx.Scene(spin_a_over_M=float(rng.uniform(0, 0.998)), disc_inner_M=6.0, disc_outer_M=30.0,
                       disc_peak_T_K=1e4, render_supersample=1)
        cam = sgx.build_orbital_camera(float(rng.uniform(20, 60)), float(rng.uniform(0.02, 1.4)), 0.0, 30.0)
        views.append(sgx.pack_uniforms(sc, cam, 16 * int(rng.integers(1, 4)), 24))
    opts = sgx.default_opts(integrator=N.INTEGRATOR_ADAPTIVE, precision=getattr(N, precision))
    b = sgx.Batch(renderer, views, opts)
    b.launch()
    b.wait()
    d = [np.abs(b.capture(i).astype(float) - renderer.render_image(v, opts).astype(float)).ravel()
         for i, v in enumerate(views)]
    b.close()
    d = np.concatenate(d)
    print(n, precision, np.mean(d == 0), d.mean() / 255.0)
    assert np.mean(d <= 1.0) >= 0.997 and d.mean() / 255.0 <= 5e-4
