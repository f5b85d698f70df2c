"""The z-column backprojection of upright views (ab_bpcol.cuh) at the edges of its blocks.

A warp takes a column of 32 XB voxels in blocks of 32, in pairs; a block lies
inside the detector's flat box, across its edge or off the detector; calls
with a view that is not upright take the brick kernel. Against the FP64 oracle:
rel L2 <= 1e-5, the gate of every backprojection mode. Against the brick kernel
(``APRICT_VIEWS_GENERAL``) on the same call: both settle the nearest rows in
FP64 and sum in FP32 (<= 1e-6); bilinear coordinates carry the brick kernel's FP32
error of about 1e-4 pixel (<= 1e-5).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from aprict_b200 import Volume, geometry
from aprict_b200.batch import ScanBatch
from aprict_b200.cb import flatpanel as fp
from helpers import circular, jittered, rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = {
    "nearest": dict(fast_approx=True),
    "nearest-taper": dict(fast_approx=True, cyl_mask_rad=7.0, soften_det_edges_proportion=0.2),
    "bilinear": dict(fast_approx=True, approx_mode_bilinear_interpolate=True),
    "bilinear-taper": dict(fast_approx=True, approx_mode_bilinear_interpolate=True, soften_det_edges_proportion=0.2),
    "raycast": dict(fast_approx=True, approx_mode_direct_raycast=True, Z_on_val_factor_power=-2, Z_on_val_factor_val=100.0),
    "raycast-preset": dict(fast_approx=True, approx_mode_direct_raycast=True, Z_on_val_factor_power=-1,
                           Z_on_val_factor_val=100.0, backproj_weighting_preset=1),
    "raycast-bilinear": dict(fast_approx=True, approx_mode_direct_raycast=True, approx_mode_bilinear_interpolate=True,
                             Z_on_L_factor_power=-1),
    "sub-samples": dict(fast_approx=True, ssx=1, ssy=2, ssz=2),
}


def _run(mode: str, pg: fp.ProjGeom, data: torch.Tensor, shape, order="C", views: int | None = None, vw: float = 1.0) -> np.ndarray:
    v = Volume.zeros(shape, voxwid=vw, order=order)
    ps = fp.ProjectionSet(pg, data=data)
    if views is not None:
        ps._backproject_promise = lambda needs_z: views  # noqa: SLF001
    fp.backproject(fp.ConfigBackproject(**MODES[mode]), v, ps, block=True)
    return v.as_numpy()


def _data(pg: fp.ProjGeom, seed: int = 0) -> torch.Tensor:
    a = np.random.default_rng(seed).random((pg.num_projs, int(pg.nu.flat[0]), int(pg.nv.flat[0]))).astype(np.float32)
    return torch.from_numpy(a).cuda()


def _oracle(mode: str, pg: fp.ProjGeom, data: torch.Tensor, shape, vw: float = 1.0) -> np.ndarray:
    return O.backproject(pg.to_proj_spec_array(), data.cpu().numpy(), shape, fp.ConfigBackproject(**MODES[mode]).contents,
                         voxwid=vw, corner=-np.float32(vw) * np.array(shape, np.float32) / 2)


@pytest.mark.parametrize("nz", [2, 31, 32, 33, 64, 65, 128, 129, 160, 257])
@pytest.mark.parametrize("mode", ["nearest-taper", "bilinear", "raycast"])
def test_heights_match_oracle(nz: int, mode: str) -> None:
    """Heights around the 32-voxel blocks, their pairs and the 2 / 4 / 8 voxels per thread; the detector
    cuts the tall ones off at the top and bottom."""
    shape = (9, 17, nz)
    pg = circular(70, 160, 120, 0.913, 25, 63)  # more than one chunk of 64 views
    data = _data(pg, nz)
    want = _oracle(mode, pg, data, shape)
    assert np.linalg.norm(want) > 0
    got = _run(mode, pg, data, shape)
    assert rel_l2(got, want) <= 1e-5
    assert rel_l2(_run(mode, pg, data, shape, views=0), got) == 0  # no promise: the same kernel after its own look
    assert rel_l2(_run(mode, pg, data, shape, views=2), got) <= (1e-5 if "bilinear" in mode else 1e-6)


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("mode", sorted(MODES))
def test_modes_match_oracle(mode: str, order: str) -> None:
    shape = (20, 13, 70)
    pg = geometry.helical_scan(n_views=40, R=90.0, L_minus_R=70.0, pix_at_iso=0.637, nu=41, nv=38, pitch=1.2, theta_start=0.31)
    data = _data(pg, 5)
    want = _oracle(mode, pg, data, shape)
    assert np.linalg.norm(want) > 0
    assert rel_l2(_run(mode, pg, data, shape, order), want) <= 1e-5


@pytest.mark.parametrize("layout", ["v strided", "u fastest", "views strided"])
@pytest.mark.parametrize("mode", ["nearest", "bilinear", "raycast"])
def test_projection_strides(mode: str, layout: str) -> None:
    """The column address is formed from the strides; bilinear with v not contiguous takes the bricks."""
    shape = (12, 10, 40)
    pg = circular(12, 120, 100, 0.713, 26, 44)
    data = _data(pg, 3)
    if layout == "v strided":
        view = torch.empty((12, 26, 44, 3), device="cuda")[..., 1].copy_(data)
    elif layout == "u fastest":
        view = torch.empty((12, 44, 26), device="cuda").transpose(1, 2).copy_(data)
    else:
        view = torch.empty((12, 2, 26, 44), device="cuda")[:, 1].copy_(data)
    assert rel_l2(_run(mode, pg, view, shape), _run(mode, pg, data, shape)) <= (1e-5 if mode == "bilinear" else 1e-6)


@pytest.mark.parametrize("mode", ["nearest", "bilinear", "raycast"])
def test_tilted_and_mixed_views_take_the_bricks(mode: str) -> None:
    shape = (14, 12, 50)
    pg = circular(20, 120, 100, 0.713, 40, 44)
    tilted = jittered(np.random.default_rng(2), pg)
    vecs = {k: np.broadcast_to(getattr(pg, k), (20, 3)).copy() for k in ("source_pos", "det_pos", "det_uvec", "det_vvec")}
    for k in vecs:
        vecs[k][7] = getattr(tilted, k)[7]  # one view of twenty
    mixed = fp.ProjGeom(**vecs, nu=pg.nu, nv=pg.nv)
    for g in (tilted, mixed):
        data = _data(g, 4)
        want = _oracle(mode, g, data, shape)
        assert rel_l2(_run(mode, g, data, shape), want) <= 1e-5
        assert rel_l2(_run(mode, g, data, shape, views=0), want) <= 1e-5


def test_non_finite_pixels_stay_where_they_project() -> None:
    """An infinite and a NaN pixel reach the voxels that take them and no others."""
    shape = (16, 16, 96)
    pg = circular(6, 200, 150, 0.8137, 40, 140)
    data = _data(pg, 6)
    clean = _run("nearest", pg, data, shape)
    data[2, 20, 70], data[4, 11, 33] = float("inf"), float("nan")
    got, bricks = _run("nearest", pg, data, shape), _run("nearest", pg, data, shape, views=2)
    assert not np.isfinite(got).all()
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(bricks))
    ok = np.isfinite(got)
    assert rel_l2(got[ok], clean[ok]) <= 1e-6


@pytest.mark.parametrize("mode", ["nearest", "bilinear", "raycast"])
def test_batch_of_upright_and_tilted_scans(mode: str) -> None:
    """A batch runs the columns of its upright scans and the bricks of the others; each equals its one-scan call."""
    rng = np.random.default_rng(8)
    shapes = [(20, 18, 24), (10, 30, 150), (33, 9, 70), (12, 12, 40)]
    pgs = [circular(15, 120, 100, 0.713, 50, 52), circular(9, 140, 90, 0.61, 40, 60, theta0=0.4),
           jittered(rng, circular(12, 120, 100, 0.713, 50, 52)), jittered(rng, circular(20, 130, 100, 0.66, 44, 40))]
    cfg = fp.ConfigBackproject(**MODES[mode])
    datas = [_data(g, i) for i, g in enumerate(pgs)]
    vols = [Volume.zeros(s, voxwid=1.0) for s in shapes]
    ScanBatch(vols, [fp.ProjectionSet(g, data=d) for g, d in zip(pgs, datas)]).backproject(cfg, block=True)
    for s, g, d, v in zip(shapes, pgs, datas, vols):
        assert rel_l2(v.as_numpy(), _run(mode, g, d, s)) <= 1e-6


@pytest.mark.parametrize(("shape", "nu", "nv"), [((20, 22, 33), 31, 40), ((21, 19, 64), 30, 41), ((21, 19, 131), 30, 40)])
@pytest.mark.parametrize("mode", ["nearest", "raycast"])
def test_exact_ties_fall_as_in_the_bricks(mode: str, shape: tuple, nu: int, nv: int) -> None:
    """Odd heights on an even detector put the mid plane on the edge between two rows in every view, odd widths the
    axis between two columns: the last bit of the FP64 forms decides, the same one in both kernels. FP32 sums agree to
    1e-6; a voxel-view on the other side changes its voxel by a pixel's difference over 70 views, 1e-3 of the largest."""
    for vw in (1.0, 0.9):
        pg = circular(70, 160, 120, 0.913, nu, nv, theta0=0.3)
        data = _data(pg, 11)
        got, bricks = _run(mode, pg, data, shape, vw=vw), _run(mode, pg, data, shape, views=2, vw=vw)
        assert np.abs(got - bricks).max() <= 1e-5 * np.abs(bricks).max()
        assert rel_l2(got, bricks) <= 1e-6


@pytest.mark.parametrize("pitch", [0.3, 1.0, 3.0])
@pytest.mark.parametrize("mode", ["nearest-taper", "raycast", "bilinear-taper"])
def test_columns_cut_by_the_detector(mode: str, pitch: float) -> None:
    """Helical columns of 2, 4 and 8 blocks, of which each view sees a few: all inside, four inside, pairs, edges."""
    for nz in (60, 120, 250):
        shape = (9, 10, nz)
        pg = geometry.helical_scan(n_views=70, R=300.0, L_minus_R=200.0, pix_at_iso=0.83, nu=21, nv=150, pitch=pitch, theta_start=0.31)
        data = _data(pg, nz)
        want = _oracle(mode, pg, data, shape)
        assert np.linalg.norm(want) > 0
        got = _run(mode, pg, data, shape)
        assert rel_l2(got, want) <= 1e-5
        assert rel_l2(_run(mode, pg, data, shape, views=2), got) <= (1e-5 if "bilinear" in mode else 1e-6)


@pytest.mark.parametrize("mode", ["nearest-taper", "raycast"])
@pytest.mark.parametrize("nz", [33, 65, 97, 161, 257])
def test_many_close_rows(mode: str, nz: int) -> None:
    """More close rows in a group of views than a warp's queue of 32 holds, the rest of a queue at a group's end, and
    the same voxel many times: at magnification 1 on detector rows of half and of a whole voxel nearly all of a
    column's rows are edges between pixels (offset by 2e-6 pixel so that FP64 and the oracle agree on them), or its
    mid plane is in every view. Bit for bit alike in a batch, whose columns take other block counts."""
    for pix, off in ((1.0, 0.5 - 2e-6), (0.5, 0.25 - 1e-6)):
        n, nv = 6, int(nz / pix) + 9
        t = 0.3 + 2 * np.pi * np.arange(70) / 70
        c, s = np.cos(t), np.sin(t)
        L = 4e6  # a source so far that the magnification is 1 to 1e-6 over the volume
        pg = fp.ProjGeom(source_pos=np.stack([L * c, L * s, 0 * t + off], 1), det_pos=np.stack([-40 * c, -40 * s, 0 * t + off], 1),
                         det_uvec=0.913 * np.stack([-s, c, 0 * t], 1), det_vvec=np.tile([0.0, 0.0, -pix], (70, 1)), nu=15, nv=nv)
        data, shape = _data(pg, nz), (n, n, nz)
        got, bricks = _run(mode, pg, data, shape), _run(mode, pg, data, shape, views=2)
        assert np.linalg.norm(bricks) > 0
        assert rel_l2(got, bricks) <= 1e-6
        v = Volume.zeros(shape, voxwid=1.0)
        ScanBatch([v], [fp.ProjectionSet(pg, data=data)]).backproject(fp.ConfigBackproject(**MODES[mode]), block=True)
        np.testing.assert_array_equal(v.as_numpy(), got)


@pytest.fixture
def knob():
    """Sets the z-lane knob (0 = where it pays, 1 = never)."""
    from aprict_b200 import _lib, autotune

    lib = _lib.lib()
    yield lambda value: _lib.check(lib.aprict_b200_set_tuning(autotune.KEY_BP_ZLANES, value), "set_tuning")
    lib.aprict_b200_set_tuning(autotune.KEY_BP_ZLANES, 0)


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("mode", ["nearest-taper", "bilinear", "raycast"])
def test_flat_volumes_on_both_sides_of_the_rule(mode: str, order: str, knob) -> None:  # noqa: ANN001
    """Volumes of more columns than one wave of CTAs: flat ones take the bricks, tall ones the columns; at every
    height the call gives what either kernel gives, alone and in a batch with others of other kinds."""
    shapes = [(90, 71, nz) for nz in (2, 31, 32, 33, 48, 49, 64, 65, 88, 97, 105)]
    pgs = [circular(m, 300, 200, 1.37, 77, max(12, int(0.9 * s[2]))) for s, m in zip(shapes, (17, 16, 17, 16, 17, 17, 8, 17, 9, 17, 17))]
    datas = [_data(g, i) for i, g in enumerate(pgs)]
    tol = 1e-5 if mode == "bilinear" else 1e-6
    auto, bricks = [], []
    for value, out in ((0, auto), (1, bricks)):
        knob(value)
        out.extend(_run(mode, g, d, s, order) for s, g, d in zip(shapes, pgs, datas))
    knob(0)
    vols = [Volume.zeros(s, voxwid=1.0, order=order) for s in shapes]
    ScanBatch(vols, [fp.ProjectionSet(g, data=d) for g, d in zip(pgs, datas)]).backproject(
        fp.ConfigBackproject(**MODES[mode]), block=True)
    for a, b, v in zip(auto, bricks, vols):
        assert np.linalg.norm(b) > 0
        assert rel_l2(a, b) <= tol
        assert rel_l2(v.as_numpy(), b) <= tol


@pytest.mark.parametrize("nz", [64, 130, 260])
@pytest.mark.parametrize("mode", ["nearest-taper", "nearest-z"])
def test_mixed_scans_on_tall_volumes(mode: str, nz: int) -> None:
    """A scan with views of both kinds on a volume of z-lane bricks (4 and 8 voxels per thread, and below them): known
    to be mixed, nothing known, and the form without the table of upright views; alone and in batches."""
    cfg = dict(MODES["nearest-taper"], cyl_mask_rad=5.0) if mode == "nearest-taper" else dict(fast_approx=True, Z_on_val_factor_power=-1, Z_on_val_factor_val=100.0)
    pg = circular(70, 200, 160, 0.913, 25, nz - 20, theta0=0.3)
    tilted = jittered(np.random.default_rng(2), pg)
    vecs = {k: np.broadcast_to(getattr(pg, k), (70, 3)).copy() for k in ("source_pos", "det_pos", "det_uvec", "det_vvec")}
    for k in vecs:
        vecs[k][[3, 40, 41, 69]] = getattr(tilted, k)[[3, 40, 41, 69]]
    g, shape = fp.ProjGeom(**vecs, nu=pg.nu, nv=pg.nv), (9, 11, nz)
    data = _data(g, nz)
    conf = fp.ConfigBackproject(**cfg)
    want = O.backproject(g.to_proj_spec_array(), data.cpu().numpy(), shape, conf.contents, voxwid=1.0,
                         corner=-np.array(shape, np.float32) / 2)
    assert fp.ProjectionSet(g, data=data)._backproject_promise(conf.needs_z) == 3
    out = []
    for views in (3, 0, 2):
        v, ps = Volume.zeros(shape, voxwid=1.0), fp.ProjectionSet(g, data=data)
        ps._backproject_promise = lambda needs_z, views=views: views  # noqa: SLF001
        fp.backproject(conf, v, ps, block=True)
        out.append(v.as_numpy())
        assert rel_l2(out[-1], want) <= 1e-5
    np.testing.assert_array_equal(out[0], out[1])
    geoms = [g, pg, tilted]
    vols = [Volume.zeros(shape, voxwid=1.0) for _ in geoms]
    ScanBatch(vols, [fp.ProjectionSet(k, data=data) for k in geoms]).backproject(conf, block=True)
    for k, v in zip(geoms, vols):
        one = Volume.zeros(shape, voxwid=1.0)
        fp.backproject(conf, one, fp.ProjectionSet(k, data=data), block=True)
        assert rel_l2(v.as_numpy(), one.as_numpy()) <= 1e-6


def test_promise_is_of_the_uploaded_views() -> None:
    """The views' kind is that of the records on the device, whatever became of the host's since."""
    shape = (12, 11, 64)
    pg = jittered(np.random.default_rng(5), circular(9, 120, 100, 0.713, 26, 60))
    data = _data(pg, 1)
    want = _run("nearest", pg, data, shape)
    assert np.linalg.norm(want) > 0
    ps = fp.ProjectionSet(pg, data=data.clone())
    fp.project(fp.ConfigProject(), Volume.zeros(shape, voxwid=1.0), ps)  # uploads the views, adds nothing
    sp = ps.proj_specs
    sp["det_u"]["z"] = sp["det_v"]["x"] = sp["det_v"]["y"] = 0
    for p in (ps, ps._with_data(data), ps.zeroed_copy()):
        assert p._backproject_promise(False) == 2
    v = Volume.zeros(shape, voxwid=1.0)
    fp.backproject(fp.ConfigBackproject(**MODES["nearest"]), v, ps, block=True)
    np.testing.assert_array_equal(v.as_numpy(), want)


@pytest.mark.parametrize("ss", [(1, 1, 3), (3, 1, 1), (2, 2, 3), (1, 3, 2)])
@pytest.mark.parametrize("mode", ["nearest", "raycast"])
def test_sub_samples_on_edges_fall_as_in_the_bricks(mode: str, ss: tuple, knob) -> None:  # noqa: ANN001
    """The middle one of three sub-samples of an odd grid's mid plane or axis lies on the edge between two pixels in
    every view; its offset, rounded as the general kernel's, decides."""
    for shape, nu, nv in (((20, 22, 33), 31, 40), ((21, 19, 33), 30, 41), ((21, 23, 7), 30, 40)):
        pg = circular(40, 160, 120, 0.913, nu, nv, theta0=0.3)
        data, out = _data(pg, 2), []
        for value in (0, 1):
            knob(value)
            v = Volume.zeros(shape, voxwid=0.5)
            fp.backproject(fp.ConfigBackproject(**MODES[mode], ssx=ss[0], ssy=ss[1], ssz=ss[2]), v, fp.ProjectionSet(pg, data=data), block=True)
            out.append(v.as_numpy())
        assert np.abs(out[0] - out[1]).max() <= 1e-5 * np.abs(out[1]).max()
        assert rel_l2(out[0], out[1]) <= 1e-6
