"""The work this framework is used for, as timed cases over its public entry points.

A case is a dict of plain values.  Four kinds:

* ``frame``    -- frames rendered and captured (``Renderer.render`` / ``capture``), one or several camera positions
* ``hdr``      -- a half-precision HDR frame, bloomed and tone-mapped (``Renderer.render`` / ``bloom``)
* ``batch``    -- many views in one launch, new cameras each time (``Batch.update`` / ``launch`` / ``wait`` / ``capture``)
* ``adjoint``  -- image, loss and gradient of the differentiable form (``diff.render`` and ``backward``)

``exact`` restates the frame and adjoint kinds in 64-bit torch, from the formulas alone.
"""

import math

import numpy as np
import torch

import singularity_gb300 as S
from singularity_gb300 import diff as D

N = S._native

FORMATS = {"rgba8": N.FORMAT_RGBA8_SRGB, "rgba32f": N.FORMAT_RGBA32F}
PRECISIONS = {"fp32": N.PRECISION_FP32, "mixed": N.PRECISION_MIXED, "fp64": N.PRECISION_FP64}
INTEGRATORS = {"fixed": N.INTEGRATOR_FIXED, "adaptive": N.INTEGRATOR_ADAPTIVE}
MODELS = {"slab": N.DIFF_MODEL_SLAB, "crossing": N.DIFF_MODEL_CROSSING}


def _frame(name, w, h, spp, *, kind="frame", metric="kerr", integrator="adaptive", precision="mixed", rhs_form=0,
           format="rgba8", frames=1, spin=0.94, r_obs=40.0, incl=75.0, fov=30.0, r_out=30.0, h_step=0.4, max_steps=2500,
           sigma=0.0):
    return dict(name=name, kind=kind, w=w, h=h, spp=spp, metric=metric, integrator=integrator, precision=precision,
                rhs_form=rhs_form, format=format, frames=frames, spin=spin, r_obs=r_obs, incl=incl, fov=fov, r_out=r_out,
                h_step=h_step, max_steps=max_steps, sigma=sigma)


def _adjoint(name, w, h, spp, *, model="slab", precision="fp32", h_step=0.2, max_steps=2000):
    return dict(name=name, kind="adjoint", w=w, h=h, spp=spp, model=model, precision=precision, h_step=h_step,
                max_steps=max_steps, r_obs=40.0, fov=30.0)


def listed():
    return [
        # the plain method's scene: a Schwarzschild hole at pixel centres, fixed step 0.05, float output
        _frame("schwarzschild-256", 256, 256, 1, metric="schwarzschild", integrator="fixed", precision="fp32",
               format="rgba32f", spin=0.0, r_obs=30.0, incl=80.0, fov=40.0, r_out=20.0, h_step=0.05, max_steps=4000),
        # what the command line renders by default (the reference's fixed step), at 1080p and 16 samples
        _frame("kerr-1080p-fixed", 1920, 1080, 16, integrator="fixed", precision="fp32"),
        # the reference's right-hand side division for division: comparisons with its frames; an odd window size
        _frame("kerr-reference-form", 1279, 719, 4, integrator="fixed", precision="fp32", rhs_form=1),
        # an interactive preview: one sample per pixel, the camera moving from frame to frame
        _frame("kerr-preview", 1280, 720, 1, frames=4),
        # the small window of a preview: launches and host work count most
        _frame("kerr-preview-small", 320, 180, 1, frames=4, precision="fp32"),
        # 1080p with half-float HDR, bloom of 8 px and the tone map
        _frame("kerr-1080p-bloom", 1920, 1080, 16, kind="hdr", sigma=8.0),
        # the headline frame: 4K at 256 samples in the precision form
        _frame("kerr-4k-256spp", 3840, 2160, 256),
        # the FP64 form: ground truth for a window's worth of pixels
        _frame("kerr-fp64", 640, 360, 4, precision="fp64", format="rgba32f"),
        # 64 views of uneven size and samples in one launch
        dict(name="batch-64", kind="batch", views=64, layout=0, side_lo=128, side_hi=1024, spp_hi=64, precision="fp32"),
        # parameter recovery: the gradient of an image loss at 512 x 512 x 4
        _adjoint("adjoint-512", 512, 512, 4),
        # a coarse fit with the reference's equatorial disc crossings, odd size, one sample
        _adjoint("adjoint-crossing", 255, 193, 1, model="crossing"),
        # the FP64 gradient a fit is checked with
        _adjoint("adjoint-fp64", 128, 96, 2, precision="fp64"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["fixed", "fixed", "adaptive", "adaptive", "adaptive", "fp64", "hdr", "batch", "adjoint", "adjoint"])
    if kind == "batch":
        lo = rng.randint(2, 8) * 16
        return dict(kind="batch", views=int(_log(rng, 2, 129)), layout=rng.randint(1, 10 ** 6), side_lo=lo,
                    side_hi=lo * rng.randint(1, 4), spp_hi=int(_log(rng, 1, 33)), precision=rng.choice(["fp32", "fp32", "mixed"]))
    if kind == "adjoint":
        fp64 = rng.random() < 0.25
        rays = _log(rng, 2 ** 9, 2 ** 14.5) if fp64 else _log(rng, 2 ** 12, 2 ** 20)
        spp = rng.choice([1, 1, 2, 3, 4, 7])
        w = max(8, int(math.sqrt(rays / spp * rng.uniform(0.5, 2.0))))
        c = _adjoint("", w, max(8, int(rays / spp / w)), spp, model=rng.choice(["slab", "slab", "crossing"]),
                     precision="fp64" if fp64 else "fp32", h_step=round(rng.uniform(0.15, 0.4), 3))
    else:
        rays = _log(rng, 2 ** 13, 2 ** 26)
        opts = dict(spin=round(rng.uniform(0.0, 0.998), 3), r_obs=round(rng.uniform(20.0, 60.0), 1),
                    incl=round(rng.uniform(10.0, 88.0), 1), fov=round(rng.uniform(20.0, 50.0), 1),
                    r_out=round(rng.uniform(15.0, 35.0), 1))
        if kind == "hdr":
            rays = _log(rng, 2 ** 16, 2 ** 25)
            opts.update(kind="hdr", sigma=rng.choice([0.0, 4.0, 8.0, 13.0]), precision=rng.choice(["fp32", "mixed"]))
        elif kind == "fp64":
            rays = _log(rng, 2 ** 12, 2 ** 20.5)
            opts.update(precision="fp64", format=rng.choice(["rgba32f", "rgba8"]))
        elif kind == "adaptive":
            opts.update(precision=rng.choice(["fp32", "mixed", "mixed"]), format=rng.choice(["rgba8", "rgba8", "rgba32f"]))
        else:
            metric = rng.choice(["kerr", "kerr", "schwarzschild"])
            form = rng.choice([0, 0, 1, 2]) if metric == "kerr" else 0
            rays = _log(rng, 2 ** 13, 2 ** 24 if metric == "kerr" and form != 1 else 2 ** 21)
            opts.update(metric=metric, integrator="fixed", precision="fp32", rhs_form=form,
                        h_step=round(rng.uniform(0.05, 0.4), 3), max_steps=4000,
                        format=rng.choice(["rgba8", "rgba8", "rgba32f"]))
            if metric == "schwarzschild":
                opts["spin"] = 0.0
        spp = min(256, max(1, int(_log(rng, 1, min(257.0, rays / 2048)))))
        w = max(16, int(math.sqrt(rays / spp * rng.uniform(1.0, 2.0))))
        c = _frame("", w, max(16, int(rays / spp / w)), spp, frames=rng.choice([1, 1, 3]) if rays < 2 ** 20 else 1, **opts)
        if c["kind"] == "hdr":
            c["frames"] = 1
    del c["name"]
    return c


# --- inputs -------------------------------------------------------------------------------------------------------

def _isco(a):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - math.sqrt((3 - z1) * (3 + z1 + 2 * z2))


def _views(case, seed):
    """The scenes and cameras of a frame case: the case's own, with the azimuth, the disc's phase and small
    changes of inclination and spin from the seed, and an orbit of 3 degrees a frame."""
    rng = np.random.default_rng([seed, 1])
    azimuth, time = rng.uniform(0, 2 * math.pi), rng.uniform(0, 10)
    incl = math.radians(min(89.0, case["incl"] + rng.uniform(-1, 1)))
    spin = min(0.998, max(0.0, case["spin"] + rng.uniform(-0.01, 0.01))) if case["metric"] == "kerr" else 0.0
    return [dict(azimuth=azimuth + math.radians(3) * k, time=time + k / 30, incl=incl, spin=spin, r_in=_isco(spin))
            for k in range(case["frames"])]


def _uniforms(case, v):
    kerr = case["metric"] == "kerr"
    scene = S.Scene(metric=S.MetricType.Kerr if kerr else S.MetricType.Schwarzschild, spin_a_over_M=v["spin"],
                    disc_inner_M=v["r_in"], disc_outer_M=case["r_out"], disc_peak_T_K=1e4,
                    render_supersample=case["spp"], h_step=case["h_step"], max_steps=case["max_steps"])
    cam = S.build_orbital_camera(case["r_obs"], math.pi / 2 - v["incl"], v["azimuth"], case["fov"])
    return S.pack_uniforms(scene, cam, case["w"], case["h"], v["time"])


def _batch_views(case, seed):
    """Sizes and samples from the case's layout, scenes and cameras from the seed."""
    lay, rng, views = np.random.default_rng([case["layout"], 2]), np.random.default_rng([seed, 2]), []
    for _ in range(case["views"]):
        side = int(lay.integers(case["side_lo"] // 16, case["side_hi"] // 16 + 1)) * 16
        spp, spin = int(lay.integers(1, case["spp_hi"] + 1)), float(rng.uniform(0.0, 0.998))
        scene = S.Scene(spin_a_over_M=spin, disc_inner_M=_isco(spin), disc_outer_M=30.0, disc_peak_T_K=1e4,
                        render_supersample=spp)
        cam = S.build_orbital_camera(float(rng.uniform(20.0, 60.0)),
                                     math.pi / 2 - math.radians(float(rng.uniform(10.0, 89.0))), 0.0, 30.0)
        views.append(S.pack_uniforms(scene, cam, side, side))
    return views


def _batch_rays(case):
    lay, rays, pixels = np.random.default_rng([case["layout"], 2]), 0, 0
    for _ in range(case["views"]):
        side = int(lay.integers(case["side_lo"] // 16, case["side_hi"] // 16 + 1)) * 16
        rays += side * side * int(lay.integers(1, case["spp_hi"] + 1))
        pixels += side * side
    return rays, pixels


def _adjoint_inputs(case, seed):
    """A guess near (spin 0.5, inclination 50 deg, inner radius 1.2 ISCO, temperature scale 0.8) and the image it is
    fitted to: an elliptical ring of light, brighter on its approaching side."""
    rng = np.random.default_rng([seed, 3])
    spin = 0.5 + rng.uniform(-0.1, 0.1)
    params = [spin, math.radians(50 + rng.uniform(-5, 5)), 1.2 * _isco(spin), 0.8 + rng.uniform(-0.1, 0.1)]
    w, h = case["w"], case["h"]
    x = (2 * (np.arange(w) + 0.5) / w - 1)[None, :] * w / h
    y = (2 * (np.arange(h) + 0.5) / h - 1)[:, None]
    rho = np.sqrt(x * x + (y / rng.uniform(0.5, 0.8)) ** 2)
    light = np.exp(-((rho - rng.uniform(0.5, 0.7)) / 0.25) ** 2) * (0.5 - 0.3 * x / np.maximum(rho, 1e-3))
    target = np.stack([0.9 * light, 0.6 * light, 0.4 * light], axis=-1).astype(np.float32)
    return params, target


def prepare(case, seed):
    renderer = S.Renderer()
    if case["kind"] == "batch":
        views = _batch_views(case, seed)
        opts = S.default_opts(integrator=N.INTEGRATOR_ADAPTIVE, precision=PRECISIONS[case["precision"]])
        return dict(kind="batch", views=views, renderer=renderer, batch=S.Batch(renderer, views, opts))
    if case["kind"] == "adjoint":
        params, target = _adjoint_inputs(case, seed)
        scene = S.Scene(spin_a_over_M=0.7, disc_outer_M=30.0, disc_peak_T_K=1e4, render_supersample=case["spp"],
                        h_step=case["h_step"], max_steps=case["max_steps"])
        u = S.pack_uniforms(scene, S.build_orbital_camera(case["r_obs"], 0.3, 0.0, case["fov"]), case["w"], case["h"])
        fp64 = case["precision"] == "fp64"
        return dict(kind="adjoint", dr=D.DiffRenderer(renderer), u=u, target=torch.from_numpy(target).cuda(),
                    params=torch.tensor(params, dtype=torch.float64 if fp64 else torch.float32, requires_grad=True),
                    opts=D.DiffOptions(precision=PRECISIONS[case["precision"]], model=MODELS[case["model"]]))
    renderer.resize(case["w"], case["h"])
    hdr = case["kind"] == "hdr"
    fmt = N.FORMAT_RGBA16F_HDR if hdr else FORMATS[case["format"]]
    opts = S.default_opts(integrator=INTEGRATORS[case["integrator"]], precision=PRECISIONS[case["precision"]],
                          rhs_form=case["rhs_form"], format=fmt)
    return dict(kind=case["kind"], renderer=renderer, frames=[_uniforms(case, v) for v in _views(case, seed)], opts=opts,
                fmt=fmt, sigma=case["sigma"])


def run(state):
    if state["kind"] == "frame":
        return [state["renderer"].render_image(u, state["opts"], state["fmt"]) for u in state["frames"]]
    if state["kind"] == "hdr":
        state["renderer"].render(state["frames"][0], state["opts"])
        return state["renderer"].bloom(sigma_px=state["sigma"])
    if state["kind"] == "batch":
        batch = state["batch"]
        batch.update(state["views"])
        batch.launch()
        batch.wait()
        if batch.n <= 64:
            return [batch.capture(i) for i in range(batch.n)]
        return np.concatenate([batch.capture(i).reshape(-1) for i in range(batch.n)])
    p = state["params"]
    p.grad = None
    image = D.render(p, state["dr"], state["u"], state["opts"])
    loss = torch.mean((image - state["target"]) ** 2)
    loss.backward()
    return dict(image=image.detach(), loss=loss.detach(), grad=p.grad)


# --- work ---------------------------------------------------------------------------------------------------------

# Additions and multiplications (reciprocals, roots, sines as one each) of one integrator step in its leanest form:
# Carter's separated Kerr right-hand side is 41, the Schwarzschild one 45, the stage updates 10 to 14 each.
STEP = {"fixed": 4 * 43 + 3 * 10 + 5 * 7, "schwarzschild": 4 * 45 + 3 * 14 + 7 * 7, "adaptive": 4 * 43 + 3 * 12 + 6 * 7 + 45,
        "forward": 4 * 43 + 3 * 14 + 7 * 7 + 20, "backward": 4 * (43 + 110) + 3 * 14 + 7 * 14}
SHADE = 120


def work(case):
    if case["kind"] == "batch":
        rays, pixels = _batch_rays(case)
        return dict(bytes=4 * pixels + 160 * case["views"], flops=rays * (50 * STEP["adaptive"] + SHADE))
    pixels = case["w"] * case["h"]
    rays = pixels * case["spp"]
    if case["kind"] == "adjoint":
        # a ray's steps to the end, and those the reverse sweep takes from its last emission (two thirds)
        n = 1.6 * case["r_obs"] / case["h_step"]
        return dict(bytes=2 * 12 * pixels + 64, flops=rays * n * (STEP["forward"] + 0.65 * STEP["backward"]))
    if case["integrator"] == "adaptive":
        per_ray = 40 * STEP["adaptive"]
    else:
        per_ray = 1.4 * case["r_obs"] / case["h_step"] * STEP["schwarzschild" if case["metric"] == "schwarzschild" else "fixed"]
    out = 16 if case["format"] == "rgba32f" else 4
    post = 8 + 40 if case["kind"] == "hdr" else 0  # the HDR frame out, and the extract, blur and compose per pixel
    return dict(bytes=case["frames"] * (160 + (out + post) * pixels), flops=case["frames"] * (rays * (per_ray + SHADE) + post * pixels))


# --- the same in 64 bits ------------------------------------------------------------------------------------------

PI = math.pi


class _Dual:
    """A float64 tensor `v` (n) with its derivatives `d` (4, n) by spin, inclination, inner radius, temperature scale."""

    def __init__(self, v, d):
        self.v, self.d = v, d

    def __add__(a, b):
        return _Dual(a.v + b.v, a.d + b.d) if isinstance(b, _Dual) else _Dual(a.v + b, a.d)

    __radd__ = __add__

    def __neg__(a):
        return _Dual(-a.v, -a.d)

    def __sub__(a, b):
        return _Dual(a.v - b.v, a.d - b.d) if isinstance(b, _Dual) else _Dual(a.v - b, a.d)

    def __rsub__(a, b):
        return _Dual(b - a.v, -a.d)

    def __mul__(a, b):
        return _Dual(a.v * b.v, a.d * b.v + a.v * b.d) if isinstance(b, _Dual) else _Dual(a.v * b, a.d * b)

    __rmul__ = __mul__

    def chain(a, f, df):
        return _Dual(f, a.d * df)

    def inv(a):
        i = 1 / a.v
        return a.chain(i, -i * i)

    def __truediv__(a, b):
        return a * b.inv() if isinstance(b, _Dual) else a * (1 / b)

    def __rtruediv__(a, b):
        return a.inv() * b

    def __getitem__(a, k):
        return _Dual(a.v[k], a.d[:, k])


def _v(x):
    return x.v if isinstance(x, _Dual) else x


def _f(x, f, df):
    return x.chain(f(x.v), df(x.v)) if isinstance(x, _Dual) else f(x)


def _sqrt(x):
    return _f(x, torch.sqrt, lambda v: torch.where(v > 0, 0.5 / torch.sqrt(torch.clamp(v, min=1e-300)), torch.zeros_like(v)))


def _exp(x):
    return _f(x, torch.exp, torch.exp)


def _ln(x):
    return _f(x, torch.log, lambda v: 1 / v)


def _cos(x):
    return _f(x, torch.cos, lambda v: -torch.sin(v))


def _pow(x, y):
    return _f(x, lambda v: v ** y, lambda v: y * v ** (y - 1))


def _clip(x, lo, hi):
    return _f(x, lambda v: torch.clamp(v, lo, hi), lambda v: ((v > lo) & (v < hi)).double())


def _where(c, a, b):
    if isinstance(a, _Dual) or isinstance(b, _Dual):
        ad, bd = (x.d if isinstance(x, _Dual) else 0.0 for x in (a, b))
        return _Dual(torch.where(c, _v(a), _v(b)), torch.where(c, ad, bd))
    return torch.where(c, a, b)


def _smooth(x):
    return _f(x, lambda v: torch.clamp(v, 0, 1) ** 2 * (3 - 2 * torch.clamp(v, 0, 1)),
              lambda v: 6 * torch.clamp(v, 0, 1) * (1 - torch.clamp(v, 0, 1)))


def _halton(n, base):
    f, r = 1.0, 0.0
    while n > 0:
        f /= base
        r += f * (n % base)
        n //= base
    return r


def _samples(w, h, spp):
    """Normalised image coordinates of every (pixel, sample), samples innermost."""
    off = [(0.5, 0.5)] if spp == 1 else [(_halton(s + 1, 2), _halton(s + 1, 3)) for s in range(spp)]
    off = torch.tensor(off, dtype=torch.float64, device="cuda")
    x = torch.arange(w, dtype=torch.float64, device="cuda")[None, :, None] + off[None, None, :, 0]
    y = torch.arange(h, dtype=torch.float64, device="cuda")[:, None, None] + off[None, None, :, 1]
    return [t.expand(h, w, spp).reshape(-1).clone() for t in (2 * x / w - 1, -(2 * y / h - 1))]


def _kerr_start(a, s, c, dcam, nr, nt, nph):
    """Canonical state and constants of rays with orthonormal components (nr, nt, nph) at radius dcam."""
    r, s2 = dcam, s * s
    sigma, delta = r * r + a * a * (c * c), r * r - 2 * r + a * a
    g_tt, g_tp, g_rr = -(1 - 2 * r / sigma), -2 * r * a * s2 / sigma, sigma / delta
    g_pp = s2 * ((r * r + a * a) * (r * r + a * a) - a * a * delta * s2) / sigma
    ut, up = nt / r, nph / (r * s)
    B, C = 2 * g_tp * up, g_rr * nr * nr + sigma * ut * ut + g_pp * up * up
    t = (-B - _sqrt(B * B - 4 * g_tt * C)) / (2 * g_tt)
    return -(g_tt * t + g_tp * up), g_tp * t + g_pp * up, g_rr * nr, sigma * ut


def _kerr_rhs(r, s, c, pr, pth, E, L, a):
    a2, s2, r2 = a * a, s * s, r * r
    r2a2 = r2 + a2
    iS, iD = 1 / (r2 + a2 * (c * c)), 1 / (r2a2 - 2 * r)
    P, W, aE = r2a2 * E - a * L, L - a * E * s2, a * E
    Q, U = P * iD, W / _where(_v(s2) < 1e-10, torch.full_like(_v(s2), 1e-10), s2)
    pr2 = pr * pr
    ns = ((r2a2 - 2 * r) * pr2 + pth * pth - P * Q + W * U) * iS
    dth = pth * iS
    return ((r2a2 - 2 * r) * pr * iS, dth, (a * Q + U) * iS, (r * ns + (1 - r) * (Q * Q + pr2) + 2 * E * r * Q) * iS,
            -(s * c) * iS * (a2 * ns - U * (2 * aE + U)))


def _temperature(r, r_in, peak):
    x = r_in / r
    return _where(_v(r) < _v(r_in), torch.zeros_like(_v(r)), peak * _pow(x, 0.75) * _clip(1 - _sqrt(x), 0.0, 1e30) / 0.186)


def _bands(r, ph, r_in, turbulence, time):
    x = r / r_in
    rho = _ln(_clip(x, 0.1, 1e30))
    ph = ph - 0.8 * time * _pow(_clip(x, 0.1, 1e30), -1.5)
    b1 = 0.5 + 0.5 * _cos(10 * rho + 3 * ph + 4 / _clip(_pow(x, 1.5), 0.25, 1e30))
    b2 = 0.5 + 0.5 * _cos(22 * rho - 1.7 * ph)
    return _clip(0.65 + 0.55 * (0.8 + turbulence * (b1 * b1 * b2 - 0.8)), 0.0, 1.3)


def _blackbody(T, blend):
    """Colour of a temperature; its two branches joined over 6500-6700 K where `blend`, at 6600 K otherwise."""
    t = _clip(T, 1000.0, 40000.0) * 0.01
    one = torch.ones_like(_v(t))
    g0 = _clip(0.39008157876901960784 * _ln(t) - 0.63184144378862745098, 0.0, 1.0)
    b0 = _clip(0.54320678911019607843 * _ln(_clip(t - 10, 1.0, 1e30)) - 1.19625408914, 0.0, 1.0)
    b0 = _where(_v(t) <= 19, torch.zeros_like(one), b0)
    t1 = _clip(t - 60, 1.0, 1e30)
    r1 = _clip(1.29293618606274509804 * _pow(t1, -0.1332047592), 0.0, 1.0)
    g1 = _clip(1.12989086089529411765 * _pow(t1, -0.0755148492), 0.0, 1.0)
    if blend:
        k = _smooth((t - 65) * 0.5)
        return [one + k * (r1 - one), g0 + k * (g1 - g0), b0 + k * (one - b0)]
    hot = _v(t) > 66
    return [_where(hot, r1, one), _where(hot, g1, g0), _where(_v(t) >= 66, one, b0)]


def _disc(r, ph, T, r_in, g_grav, om, cos_psi, f_emit, time, blend):
    """Emission of the disc at (r, ph) of local temperature T: redshift, Doppler, bands, g^4."""
    vel = r * om / _sqrt(_clip(f_emit, 1e-6, 1e30))
    g = g_grav * _sqrt(_clip(1 - vel * vel, 0.0, 1e30)) / _clip(1 - vel * _clip(cos_psi, -1.0, 1.0), 1e-4, 1e30)
    k = _clip(_pow(r_in / r, 3.0), 0.05, 1.5) * _bands(r, ph, r_in, 0.5, time) * (g * g) * (g * g)
    return [x * k for x in _blackbody(g * T, blend)]


def _aces(x):
    return _clip(x * (2.51 * x + 0.03) / (x * (2.43 * x + 0.59) + 0.14), 0.0, 1.0)


def _sky(s, c, ph):
    x, y = s * torch.cos(ph), s * torch.sin(ph)
    n = torch.sqrt(x * x + y * y + c * c)
    ix = ((torch.atan2(y, x) + PI) / (2 * PI) * 768).long() % 768
    iy = (torch.acos(torch.clamp(c / n, -1, 1)) / PI * 384).long() % 384
    m = 0xFFFFFFFF
    k = (ix * 0x9E3779B9 + iy) & m
    k = k ^ ((k << 13) & m)
    k = k ^ (k >> 17)
    k = k ^ ((k << 5) & m)
    hue = ((k >> 16) & 255).double() / 255
    b = torch.where((k & 255) < 4, (((k >> 8) & 255).double() / 255) ** 4, torch.zeros_like(hue))
    star = [1 - 0.5 * hue, 0.8 + 0.8 * hue * (1 - hue), 0.4 + 0.6 * hue]
    return [torch.clamp(base + b * x, max=1.0) * 0.6 for base, x in zip((0.0015, 0.002, 0.005), star)]


def _rk4(rhs, y, k1, h):
    """One step from y with k1 = rhs(y): the new state and the last stage's derivative (lists of duals, or one tensor)."""
    if isinstance(y, torch.Tensor):
        k2 = rhs(y + k1 * (0.5 * h))
        k3 = rhs(y + k2 * (0.5 * h))
        k4 = rhs(y + k3 * h)
        return y + (k1 + 2 * (k2 + k3) + k4) * (h / 6), k4
    k2 = rhs([p + k * (0.5 * h) for p, k in zip(y, k1)])
    k3 = rhs([p + k * (0.5 * h) for p, k in zip(y, k2)])
    k4 = rhs([p + k * h for p, k in zip(y, k3)])
    return [p + (a + 2 * b + 2 * c + d) * (h / 6) for p, a, b, c, d in zip(y, k1, k2, k3, k4)], k4


def _exact_frame(case, v):
    """One frame as RGBA floats: rays traced together, those that ended taken out."""
    kerr, adaptive = case["metric"] == "kerr", case["integrator"] == "adaptive"
    X, Y = _samples(case["w"], case["h"], case["spp"])
    a, d, el, az, r_in = v["spin"], case["r_obs"], PI / 2 - v["incl"], math.remainder(v["azimuth"], 2 * PI), v["r_in"]
    tf = math.tan(math.radians(case["fov"]) / 2)
    X, Y = X * tf * case["w"] / case["h"], Y * tf
    # the camera's frame: forward -e_r, right e_phi, up e_theta
    norm = torch.sqrt(1 + X * X + Y * Y)
    s0, c0 = math.cos(el), math.sin(el)
    nr, nt, nph = -1 / norm, Y / norm, X / norm
    th0 = PI / 2 - el
    z = torch.zeros_like(nr)
    hcut = 1.02 * (1 + math.sqrt(1 - a * a)) if kerr else 2.04
    color = [z.clone() for _ in range(3)]
    ids = torch.arange(nr.numel(), device="cuda")
    put = lambda m, col: [c.index_copy_(0, ids[m], x) for c, x in zip(color, col)]  # noqa: E731
    f_obs = 1 - 2 / d

    def emit(m, r, ph, extra):
        om = torch.sqrt(1 / r ** 3)
        om, f = (om / (1 + a * om) if kerr else om), 1 - 2 / r
        cos_psi = extra / r if kerr else -extra * r
        T = _temperature(r, torch.full_like(r, r_in), 1e4)
        col = _disc(r, ph, T, torch.full_like(r, r_in), torch.sqrt(torch.clamp(f, min=1e-6) / f_obs), om, cos_psi, f,
                    v["time"], False)
        put(m, [torch.where(T > 0, x, torch.zeros_like(x)) for x in col])

    if kerr:
        E, L, pr, pth = _kerr_start(a, s0 + z, c0 + z, d, nr, nt, nph)
        Q = pth * pth + c0 * c0 * (L * L / (s0 * s0) - a * a * E * E)
    if adaptive:
        y = torch.stack([d + z, s0 + z, c0 + z, az + z, pr, pth])

        def rhs(y):
            k = _kerr_rhs(y[0], y[1], y[2], y[4], y[5], E, L, a)
            return torch.stack([k[0], y[2] * k[1], -y[1] * k[1], k[2], k[3], k[4]])

        lo, hi = (2 * (1 + math.cos(2 / 3 * math.acos(q * a))) for q in (-1, 1))
        xi = L / E
        g = lambda r: r * r * (3 - r) - a * a * (r + 1) - xi * a * (r - 1)  # noqa: E731
        ok, neg, lo, hi = g(lo + z) * g(hi + z) <= 0, g(lo + z) <= 0, lo + z, hi + z
        for _ in range(12):
            mid = 0.5 * (lo + hi)
            same = (g(mid) <= 0) == neg
            lo, hi = torch.where(same, mid, lo), torch.where(same, hi, mid)
        r_c = 0.5 * (lo + hi) if a > 1e-7 else 3 + z
        r_cap = torch.where((ok | (a <= 1e-7)) & (Q >= 0), torch.clamp(r_c - 0.05, max=r_in), z)
        k1, h = rhs(y), 0.1 * y[0]
    elif kerr:
        y = torch.stack([d + z, th0 + z, az + z, pr, pth])

        def rhs(y):
            return torch.stack(_kerr_rhs(y[0], torch.sin(y[1]), torch.cos(y[1]), y[3], y[4], E, L, a))
    else:
        ut, up = nt / d, nph / (d * s0)
        f = 1 - 2 / d
        y = torch.stack([d + z, th0 + z, az + z, torch.sqrt((nr * nr / f + nt * nt + nph * nph) / f), nr, ut, up])

        def rhs(y):
            r, th, _, ut, ur, uth, uph = y
            f, s, c = 1 - 2 / r, torch.sin(th), torch.cos(th)
            p, q, g = r * r * f, uph * uph, -2 * ur / r
            return torch.stack([ur, uth, uph, -2 * ut * ur / p, (ur * ur - (f * ut) ** 2) / p + r * f * (uth * uth + s * s * q),
                                g * uth + s * c * q, (g - 2 * c / s * uth) * uph])
    prev = y
    for _ in range(case["max_steps"]):
        r = y[0]
        if adaptive:
            fall = ~torch.isfinite(r) | (r < hcut) | ((r < r_cap) & (y[4] < 0))
        else:
            fall = ~torch.isfinite(r) | (r < hcut)
        out = ~fall & (r > 200)
        over = fall | out
        if not adaptive:
            p, q = prev[1] - PI / 2, y[1] - PI / 2
            x = -p / (y[1] - prev[1])
            rc = prev[0] + x * (r - prev[0])
            hit = ~over & (p * q < 0) & (rc >= r_in) & (rc <= case["r_out"])
            if hit.any():
                emit(hit, rc[hit], y[2][hit], L[hit] if kerr else (prev[6] + x * (y[6] - prev[6]))[hit])
            over = over | hit
        if over.any():
            s, c, ph = (t[out] for t in ((y[1], y[2], y[3]) if adaptive else (torch.sin(y[1]), torch.cos(y[1]), y[2])))
            put(out, _sky(s, c, ph))
            keep = ~over
            ids, y, prev = ids[keep], y[:, keep], prev if adaptive else prev[:, keep]
            if kerr:
                E, L = E[keep], L[keep]
            if adaptive:
                Q, r_cap, h, k1 = Q[keep], r_cap[keep], h[keep], k1[:, keep]
            if not ids.numel():
                break
        if not adaptive:
            hs = case["h_step"]
            if kerr:
                hs = hs * torch.clamp(torch.abs(torch.sin(y[1])) * 5, 0.05, 1.0)
            prev, (y, _) = y, _rk4(rhs, y, rhs(y), hs)
            continue
        h = torch.minimum(h, 0.1 * y[0])
        new, k4 = _rk4(rhs, y, k1, h)
        k5 = rhs(new)
        err = (torch.abs(h / 6 * (k4 - k5)) / (1e-6 * (1 + torch.maximum(y.abs(), new.abs())))).amax(0)
        err = torch.where(err <= 1e30, err, torch.full_like(err, 1e30))
        accept = err <= 1
        hit = accept & (y[2] * new[2] < 0) & (new[1] > 0)
        over = torch.zeros_like(hit)
        if hit.any():
            c_0, c_1, d_0, d_1, hh = y[2][hit], new[2][hit], k1[2][hit], k5[2][hit], h[hit]
            cubic = lambda t, p, q, dp, dq: ((2 * t - 3) * t * t + 1) * p + ((t - 2) * t + 1) * t * hh * dp + (3 - 2 * t) * t * t * q + (t - 1) * t * t * hh * dq  # noqa: E731
            t = c_0 / (c_0 - c_1)
            for _ in range(3):
                slope = (6 * t * t - 6 * t) * (c_0 - c_1) + (3 * t * t - 4 * t + 1) * hh * d_0 + (3 * t * t - 2 * t) * hh * d_1
                t = torch.clamp(t - cubic(t, c_0, c_1, d_0, d_1) / slope, 0, 1)
            rc, pc = (cubic(t, y[i][hit], new[i][hit], k1[i][hit], k5[i][hit]) for i in (0, 3))
            on = (rc >= r_in) & (rc <= case["r_out"])
            over[hit] = on
            emit(over, rc[on], pc[on], L[over])
        h = h * torch.where(err <= 1e-30, torch.full_like(err, 4.0), torch.clamp(0.85 / err ** 0.25, 0.2, 4.0))
        n2 = 1.5 - 0.5 * (new[1] ** 2 + new[2] ** 2)
        new[1:3] *= n2
        theta = Q - new[2] ** 2 * (L * L / torch.clamp(new[1] ** 2, min=1e-10) - a * a * E * E)
        new[5] = torch.copysign(torch.sqrt(torch.clamp(theta, min=0)), new[5])
        y, k1 = torch.where(accept, new, y), torch.where(accept, k5, k1)
        if over.any():
            keep = ~over
            ids, y, k1 = ids[keep], y[:, keep], k1[:, keep]
            E, L, Q, r_cap, h = E[keep], L[keep], Q[keep], r_cap[keep], h[keep]
            if not ids.numel():
                break
    rgb = [_aces(c * 1.8).reshape(case["h"], case["w"], case["spp"]).mean(-1) for c in color]
    return torch.stack(rgb + [torch.ones_like(rgb[0])], dim=-1)


def _exact_adjoint(case, params, target):
    """Image, loss and gradient of the differentiable form, its derivatives carried forward with the rays."""
    w, h, spp = case["w"], case["h"], case["spp"]
    slab, d, r_out, fade, width, eps = case["model"] == "slab", case["r_obs"], 30.0, 0.625 * PI, 0.125 * PI, float(np.float32(0.1))
    X, Y = _samples(w, h, spp)
    tf = math.tan(math.radians(case["fov"]) / 2)
    X, Y = X * tf * w / h, Y * tf
    n = X.numel()
    eye = torch.eye(4, dtype=torch.float64, device="cuda")
    a, incl, r_in, scale = (_Dual(torch.full((1,), p, dtype=torch.float64, device="cuda"), eye[:, i:i + 1]) for i, p in enumerate(params))
    s0, c0 = _f(incl, torch.sin, torch.cos), _cos(incl)
    norm = torch.sqrt(1 + X * X + Y * Y)
    flat = lambda x: _Dual(x.v.expand(n).clone(), x.d.expand(4, n).clone()) if isinstance(x, _Dual) else _Dual(x, torch.zeros(4, n, dtype=torch.float64, device="cuda"))  # noqa: E731
    E, L, pr, pth = (flat(x) for x in _kerr_start(a, s0, c0, d, -1 / norm, Y / norm, X / norm))
    zero = flat(torch.zeros_like(X))
    y = [flat(d + 0 * X), flat(incl), zero, pr, pth, flat(s0), flat(c0)]
    psi, tau, psi0 = zero, zero + 1.0, zero
    av = float(a.v)
    hcut = max(2 * (1 + math.cos(2 / 3 * math.acos(-av))) - 0.05, 1.02 * (1 + math.sqrt(1 - av * av)))
    color = [torch.zeros(5, n, dtype=torch.float64, device="cuda") for _ in range(3)]
    ids = torch.arange(n, device="cuda")
    half, kappa = float(np.float32(0.3)), 4.0 / (16 / 15 * float(np.float32(0.3)))
    f_obs = 1 - 2 / d

    def rhs(y):
        k = _kerr_rhs(y[0], y[5], y[6], y[3], y[4], E, L, a)
        return list(k) + [y[6] * k[1], -(y[5] * k[1])]

    def emit(m, r, ph, wgt):
        """Adds tau wgt colour to the rays m (indices among the present) and takes wgt from their transmittance."""
        nonlocal tau
        T = _temperature(r, r_in, 1e4 * scale)
        om, f = _sqrt(1 / (r * r * r)), 1 - 2 / r
        col = _disc(r, ph, T, r_in, _sqrt(_clip(f, 1e-6, 1e30) / f_obs), om / (1 + a * om), L[m] / r, f, 0.0, True)
        k = tau[m] * wgt
        for c, x in zip(color, col):
            x = x * k
            on = _v(T) > 0
            c[:, ids[m]] += torch.cat([x.v[None], x.d]) * on
        left = tau[m] * (1 - wgt)
        tau = _Dual(tau.v.index_copy(0, m, left.v), tau.d.index_copy(1, m, left.d))

    prev = y
    for step in range(case["max_steps"]):
        over = ~torch.isfinite(y[0].v) | (y[0].v < hcut) | (y[0].v > 200)
        if step and slab:
            z = y[0].v * y[6].v
            m = (~over & (z.abs() < half) & (y[0].v > float(r_in.v)) & (y[0].v < r_out) & (psi.v < fade + width)).nonzero()[:, 0]
            if m.numel():
                r, th, ph, s, c = (y[i][m] for i in (0, 1, 2, 5, 6))
                q = r * c / half
                b = 1 - q * q
                dr, dth, dph = r - prev[0][m], th - prev[1][m], ph - prev[2][m]
                ds = _sqrt(dr * dr + r * r * (dth * dth + s * s * (dph * dph)))
                wgt = _smooth((r - r_in) / eps) * _smooth((r_out - r) / eps) * (1 - _smooth((psi[m] - fade) / width))
                emit(m, r, ph, wgt * (1 - _exp(-(kappa * (b * b) * ds))))
        elif step:
            p, q = prev[1].v - PI / 2, y[1].v - PI / 2
            m = (~over & (p * q < 0)).nonzero()[:, 0]
            if m.numel():
                t = (PI / 2 - prev[1][m]) / (y[1][m] - prev[1][m])
                rc = prev[0][m] + t * (y[0][m] - prev[0][m])
                pc = psi0[m] + t * (psi[m] - psi0[m])
                wgt = _smooth((rc - r_in) / eps) * _smooth((r_out - rc) / eps) * (1 - _smooth((pc - fade) / width))
                on = wgt.v > 0
                if on.any():
                    emit(m[on], rc[on], y[2][m][on], wgt[on])
                over = over | (tau.v <= 0)
        over = over | ((y[3].v > 0) & (y[0].v > r_out))
        if step % 8 == 7 or step == 0:
            keep = (~over).nonzero()[:, 0]
            if keep.numel() < over.numel():
                ids, y, E, L, psi, tau = ids[keep], [t[keep] for t in y], E[keep], L[keep], psi[keep], tau[keep]
                over = over[keep]
            if not keep.numel():
                break
        hs = case["h_step"] * _clip(_f(y[5], torch.abs, torch.sign) * 5, 0.05, 1.0)
        new, _ = _rk4(rhs, y, rhs(y), hs)
        n2 = 1.5 - 0.5 * (new[5] * new[5] + new[6] * new[6])
        new[5], new[6] = new[5] * n2, new[6] * n2
        dth, dph = new[1] - y[1], new[2] - y[2]
        ang = _sqrt(dth * dth + new[5] * new[5] * (dph * dph))
        # a ray that has ended stays where it is until it is taken out
        stop = lambda q, p: _where(over, p, q)  # noqa: E731
        prev, psi0 = y, psi
        y, psi = [stop(q, p) for q, p in zip(new, y)], stop(psi + ang, psi)
        if over.any():
            tau = _where(over, tau * 0.0, tau)
    out = []
    for c in color:
        x = _aces(_Dual(c[0], c[1:]) * float(np.float32(1.8)))
        out.append((x.v.reshape(h, w, spp).mean(-1), x.d.reshape(4, h, w, spp).mean(-1)))
    image = torch.stack([x for x, _ in out], dim=-1)
    diff = image - target
    grad = sum((2 * diff[..., k] / diff.numel() * out[k][1]).sum((1, 2)) for k in range(3))
    return dict(image=image, loss=(diff * diff).mean(), grad=grad.cpu())


def exact(case, seed):
    if case["kind"] == "adjoint":
        if case["w"] * case["h"] * case["spp"] * case["r_obs"] / case["h_step"] > 3e8:
            return None
        params, target = _adjoint_inputs(case, seed)
        if case["precision"] == "fp32":
            params = [float(np.float32(p)) for p in params]
        return _exact_adjoint(case, params, torch.from_numpy(target).cuda().double())
    if case["kind"] != "frame" or case["format"] != "rgba32f":
        return None  # bytes
    rays = case["w"] * case["h"] * case["spp"] * case["frames"]
    if rays * (40 if case["integrator"] == "adaptive" else case["r_obs"] / case["h_step"]) > 1e9:
        return None
    return [_exact_frame(case, v) for v in _views(case, seed)]
