"""Fan-beam FBP (recon.fbp_fan_circ) vs an FP64 pipeline built from the oracle pieces.

The oracle pipeline restates the reference's fan-beam path
(src/aprict/scripts/recon_cbfp_cyl_fbp.py:368-701, 1108-1121, 1238): cosine
weight, Ram-Lak convolution at pitch pixwid/L (FP64 numpy), direct-raycast
backprojection with (Z/R)^-2 inside the support cylinder (FP64 oracle), scale
1/(4 pi R M). Gate: rel L2 <= 1e-4 (reconstruction tolerance).
"""

from __future__ import annotations

import numpy as np
import pytest

from aprict_b200 import Volume, phantoms, ramp_kernels
from aprict_b200.cb import flatpanel as fp
from aprict_b200.recon import fan_geometry, fbp_fan_circ
from helpers import circular, rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _fan_problem(n: int = 96, views: int = 180, nu: int = 192, apod: str | None = None):
    pg = circular(views, 120.0, 100.0, 0.5123, nu, 1, theta0=0.0)
    x = phantoms.ellipsoid_volume(31, 8, (n, n, 1), 0.5, semi_axes_vox=(4, 30))
    v = Volume(x, voxwid=0.5)
    ps = fp.ProjectionSet(pg, data=None)
    fp.project(fp.ConfigProject(), v, ps, block=True)
    return pg, x, ps


@pytest.mark.parametrize("apod", [None, "hann"])
def test_fbp_matches_fp64_pipeline(apod: str | None) -> None:
    n = 96
    pg, _, ps = _fan_problem(n=n, apod=apod)
    out = Volume.zeros((n, n, 1), voxwid=0.5)
    fbp_fan_circ(ps, out, apodization=apod)
    got = out.as_numpy()

    R, L, pixwid, nu, nv = fan_geometry(pg)  # noqa: N806
    m = pg.num_projs
    p = ps.data.cpu().numpy().astype(np.float64)
    u = pixwid / L * (np.arange(nu) - (nu - 1) / 2)
    w = 1.0 / np.sqrt(1 + u**2)
    taps = ramp_kernels.ramp_kernel_ramlak(2 * nu - 1, pixwid / L)
    if apod == "hann":
        taps = ramp_kernels.apodize_hann(taps)
    filt = np.empty_like(p)
    for i in range(m):
        filt[i, :, 0] = np.convolve(p[i, :, 0] * w, taps, mode="full")[nu - 1 : 2 * nu - 1]
    filt /= 4 * np.pi * R * m
    cfg = fp.ConfigBackproject(
        fast_approx=True, cyl_mask_rad=R * np.sin(np.arctan(pixwid * nu / 2 / L)), Z_on_val_factor_power=-2,
        Z_on_val_factor_val=R, approx_mode_direct_raycast=True,
    )
    want = O.backproject(pg.to_proj_spec_array(), filt, (n, n, 1), cfg.contents, voxwid=0.5, corner=-np.array((n, n, 1), np.float32) * 0.25)
    assert np.linalg.norm(want) > 0
    assert rel_l2(got, want) <= 1e-4


def test_fbp_reconstructs_phantom() -> None:
    n = 128
    pg, x, ps = _fan_problem(n=n, views=360, nu=256)
    out = Volume.zeros((n, n, 1), voxwid=0.5)
    fbp_fan_circ(ps, out, interpolate=True)
    rec = out.as_numpy()
    inside = np.hypot(*np.meshgrid(np.arange(n) - (n - 1) / 2, np.arange(n) - (n - 1) / 2, indexing="ij"))[..., None] < 0.45 * n
    err = np.linalg.norm((rec - x)[inside]) / np.linalg.norm(x[inside])
    assert err < 0.35, err  # discretised FBP of a piecewise-constant phantom: edges dominate the error
    assert abs(rec[inside].mean() - x[inside].mean()) < 0.05 * x[inside].mean()


def test_batched_slices_equal_single_slice_fbp() -> None:
    from aprict_b200.recon import fbp_fan_circ_batch

    n = 64
    pgs = circular(120, 120.0, 100.0, 0.5123, 128, 1, theta0=0.0)
    projs, singles = [], []
    for k in range(5):
        x = phantoms.ellipsoid_volume(40 + k, 6, (n, n, 1), 0.5, semi_axes_vox=(3, 20))
        ps = fp.ProjectionSet(pgs, data=None)
        fp.project(fp.ConfigProject(), Volume(x, voxwid=0.5), ps, block=True)
        projs.append(ps)
        one = Volume.zeros((n, n, 1), voxwid=0.5)
        fbp_fan_circ(ps, one, apodization="hann")
        singles.append(one.as_numpy())
    outs = [Volume.zeros((n, n, 1), voxwid=0.5) for _ in range(5)]
    fbp_fan_circ_batch(projs, outs, apodization="hann")
    for o, w in zip(outs, singles):
        assert np.linalg.norm(w) > 0
        assert rel_l2(o.as_numpy(), w) <= 1e-6


@pytest.mark.parametrize(("slices", "n", "nu"), [(4, 40, 90), (5, 33, 128), (9, 50, 200), (17, 21, 96), (33, 70, 150),
                                                 (64, 24, 140), (67, 20, 130)])
def test_slice_stack_equals_single_slices(slices: int, n: int, nu: int, monkeypatch: pytest.MonkeyPatch) -> None:
    """Stacks of one scan run through the interleaved kernel: slice counts around its lane groups (4 slices
    a lane, 1 to 16 lanes) and past one call's 64, slices narrower than a tile, rows filtered directly
    (nu < 128) and by FFT. Each slice equals its own reconstruction up to FP32 rounding."""
    from aprict_b200 import recon
    from aprict_b200.recon import fbp_fan_circ_batch

    calls, stack = [], recon._backproject_slices  # noqa: SLF001
    monkeypatch.setattr(recon, "_backproject_slices", lambda *a: (calls.append(len(a[3])), stack(*a)))

    pg = circular(75, 120.0, 100.0, 0.9 * n * 0.5 / nu * 1.2345, nu, 1, theta0=0.21)
    rng = np.random.default_rng(slices)
    projs, vols, want = [], [], []
    for _ in range(slices):
        ps = fp.ProjectionSet(pg, data=rng.random((75, nu, 1)).astype(np.float32))
        one = Volume.zeros((n, n + 3, 1), voxwid=0.5)
        fbp_fan_circ(ps, one)
        projs.append(ps)
        want.append(one.as_numpy())
        vols.append(Volume.zeros((n, n + 3, 1), voxwid=0.5))
        vols[-1].fill(0.25)  # added to
    fbp_fan_circ_batch(projs, vols)
    assert sum(calls) == slices
    for v, w in zip(vols, want):
        assert np.linalg.norm(w) > 0
        assert rel_l2(v.as_numpy() - 0.25, w) <= 2e-6


@pytest.mark.parametrize("case", ["off plane", "other views", "changed geometry", "F order", "other grid", "bilinear"])
def test_slice_stacks_that_do_not_share_a_scan_go_one_by_one(case: str, monkeypatch: pytest.MonkeyPatch) -> None:
    from aprict_b200 import recon
    from aprict_b200.recon import fbp_fan_circ_batch

    def stacked(*_: object) -> None:
        pytest.fail("backprojected as a stack of one scan")

    monkeypatch.setattr(recon, "_backproject_slices", stacked)

    n, nu = 40, 130
    pgs = [circular(60, 120.0, 100.0, 0.21, nu, 1, theta0=0.21) for _ in range(5)]
    order, shapes, z = "C", [(n, n, 1)] * 5, 0.0
    if case == "other views":
        pgs[3] = circular(60, 120.0, 100.0, 0.21, nu, 1, theta0=0.9)
    elif case == "F order":
        order = "F"
    elif case == "other grid":
        shapes = [(n, n, 1), (n, n + 8, 1)] + [(n, n, 1)] * 3
    elif case == "off plane":
        z = 0.05
    rng = np.random.default_rng(3)
    if case == "changed geometry":  # one object, turned by a view after some of the sets were made
        pgs = [pgs[0]] * 5
    projs = []
    for i, g in enumerate(pgs):
        if case == "changed geometry" and i == 3:
            for k in ("source_pos", "det_pos", "det_uvec"):
                a = getattr(g, k)
                a[...] = np.roll(a, 7, axis=0)
        projs.append(fp.ProjectionSet(g, data=rng.random((60, nu, 1)).astype(np.float32)))
    vols = [Volume.zeros(s, voxwid=0.5, order=order, pos_c=(0, 0, z)) for s in shapes]
    fbp_fan_circ_batch(projs, vols, interpolate=case == "bilinear")
    rolled = [fp.ProjGeom(**{k: np.roll(np.broadcast_to(getattr(g, k), (60, 3)), -7, axis=0) for k in
                             ("source_pos", "det_pos", "det_uvec")}, det_vvec=g.det_vvec, nu=g.nu, nv=g.nv)
              if case == "changed geometry" and i < 3 else g for i, g in enumerate(pgs)]
    for p, g, s, v in zip(projs, rolled, shapes, vols):
        one = Volume.zeros(s, voxwid=0.5, order=order, pos_c=(0, 0, z))
        fbp_fan_circ(fp.ProjectionSet(g, data=p.data), one, interpolate=case == "bilinear")
        # (bilinear coordinates are stepped in FP32 from the thread's first voxel, two voxels against four)
        assert rel_l2(v.as_numpy(), one.as_numpy()) <= (2e-5 if case == "bilinear" else 2e-6)
