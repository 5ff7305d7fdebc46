"""The fixed-step forms with the reference's divisions at masses on both sides of
the lines between shared reciprocals, the way out of them and the plain divisions.

A single Kerr view outside the lines runs the plain divisions, a batch of it the
way out of the shared reciprocals; both round as the reference's expressions do.
The bar between them is that of the batch tests (>= 99.7 % of values within one
level, mean <= 5e-4): the kernels read their views' constants differently and
contract a few multiply-adds of the camera ray and the shading differently.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,mass", [("KERR", 1.0), ("KERR", 199.0), ("KERR", 201.0), ("KERR", 900.0),
                                         ("KERR", 6e-5), ("KERR", 5e-5), ("KERR", 1e-6), ("SCHWARZSCHILD", 1.0),
                                         ("SCHWARZSCHILD", 1300.0), ("SCHWARZSCHILD", 1400.0),
                                         ("SCHWARZSCHILD", 6e-8), ("SCHWARZSCHILD", 4e-8)])
def test_single_view_matches_batch(sgx, renderer, metric, mass):
    N = sgx._native
    sc = sgx.Scene(spin_a_over_M=0.6 if metric == "KERR" else 0.0, disc_inner_M=6.0, disc_outer_M=20.0,
                   disc_peak_T_K=1e4, render_supersample=2, mass_solar=mass)
    u = sgx.pack_uniforms(sc, sgx.build_orbital_camera(30.0, 0.3, 0.0, 30.0), 93, 61)
    u.h_step = 0.25 * mass
    for c in "xyz":
        setattr(u.cam_pos, c, getattr(u.cam_pos, c) * mass)
    u.metric_type = getattr(N, "SGX_METRIC_" + metric)
    opts = sgx.default_opts(integrator=N.INTEGRATOR_FIXED, precision=N.PRECISION_FP32, rhs_form=1)
    single = renderer.render_image(u, opts).astype(float)
    b = sgx.Batch(renderer, [u], opts)
    b.launch()
    b.wait()
    d = np.abs(b.capture(0) - single)
    b.close()
    print(metric, mass, np.mean(d == 0), d.mean() / 255.0)
    assert np.mean(d <= 1.0) >= 0.997 and d.mean() / 255.0 <= 5e-4
