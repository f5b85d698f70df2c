"""FORBILD analytic projection: the FP64 oracle vs the reference, the host shape
compiler, and the GPU kernel vs both.

Gates: GPU vs FP64 oracle rel L2 <= 1e-5 (projections). The reference computes
its intervals in FP32, so GPU vs reference is bounded at 1e-4.
"""

from __future__ import annotations

import numpy as np
import pytest

from aprict_b200 import _structs as S
from aprict_b200 import phantoms
from aprict_b200.cb import forbild
from helpers import circular, random_shapes_all_types, rel_l2
from oracle import oracle as O

TYPES_REF = (1, 2, 3, 4, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16)  # type 5 below


def test_interval_oracle_matches_reference_all_types() -> None:
    if not O.have_ref():
        pytest.skip("reference oracle not built")
    rng = np.random.default_rng(0)
    shapes = random_shapes_all_types(rng, 150, types=TYPES_REF)
    worst = 0.0
    for _ in range(300):
        v1 = rng.uniform(-120, 120, 3)
        v2 = rng.uniform(-120, 120, 3)
        for s in shapes:
            a = O.forbild_interval(v1, v2, s)
            b = O.ref_forbild_interval(v1, v2, s)
            la = 0.0 if a is None else a[1] - a[0]
            lb = max(0.0, b[1] - b[0])
            worst = max(worst, abs(la - lb))
    assert worst <= 2e-5, worst


def test_cone_z_offcentre_reference_quirk_documented() -> None:
    """Cone_z (type 5) away from z = 0: the reference's cull projects the ray
    direction with z = pos.z instead of 0 (FORBILD_volumes.h, FORBILD_Cone_z
    clip), so it can wrongly reject rays; the oracle and the GPU kernel keep the
    exact frustum. Centred at z = 0 both agree."""
    if not O.have_ref():
        pytest.skip("reference oracle not built")
    rng = np.random.default_rng(5)
    shapes = random_shapes_all_types(rng, 40, types=(5,))
    shapes["z"] = 0.0
    for s in shapes:
        s["cas1"]["mode"] = s["cas2"]["mode"] = s["cas3"]["mode"] = 0
    worst = 0.0
    for _ in range(300):
        v1 = rng.uniform(-120, 120, 3)
        v2 = rng.uniform(-120, 120, 3)
        for s in shapes:
            a = O.forbild_interval(v1, v2, s)
            b = O.ref_forbild_interval(v1, v2, s)
            worst = max(worst, abs((0.0 if a is None else a[1] - a[0]) - max(0.0, b[1] - b[0])))
    assert worst <= 2e-5


@pytest.mark.parametrize("overlap_addition", [False, True])
def test_projection_oracle_matches_reference(overlap_addition: bool) -> None:
    if not O.have_ref():
        pytest.skip("reference oracle not built")
    rng = np.random.default_rng(1)
    shapes = random_shapes_all_types(rng, 48, types=TYPES_REF)
    pg = circular(6, 150, 150, 0.5, 40, 36)
    specs = pg.to_proj_spec_array()
    ref, ovf = O.ref_project_forbild(specs, shapes, overlap_addition=overlap_addition)
    ora = O.project_forbild(specs, shapes, mode=1 if overlap_addition else 0)
    assert ovf == 0
    assert np.linalg.norm(ora) > 0
    assert rel_l2(ref, ora) <= 1e-4


def test_compile_shapes() -> None:
    rng = np.random.default_rng(2)
    shapes = random_shapes_all_types(rng, 32)
    q = forbild.compile_shapes(shapes)
    assert q.dtype == S.quadric and len(q) == 32
    kinds = {1: 4, 2: 3, 3: 3, 4: 3, 5: 3, 6: 2, 7: 2, 8: 2, 9: 2, 10: 1, 11: 1, 12: 2, 13: 1, 14: 2, 15: 2, 16: 2}
    assert all(q["kind"][i] == kinds[int(shapes["type"][i])] for i in range(32))
    # bounding boxes contain points sampled from the shapes (oracle in-region test via tiny segments)
    lo, hi = forbild.shape_bboxes(shapes)
    for i in range(32):
        c = np.array([shapes["x"][i], shapes["y"][i], shapes["z"][i]], np.float64)
        assert np.all(lo[i] <= c) and np.all(c <= hi[i])
    bad = shapes[:1].copy()
    bad["type"] = 40
    with pytest.raises(ValueError, match="unknown type"):
        forbild.compile_shapes(bad)
    bad["type"] = 13
    bad["r"] = -1
    with pytest.raises(ValueError, match="invalid parameters"):
        forbild.compile_shapes(bad)


def test_fbvolume_bbox_and_prune() -> None:
    from aprict_b200 import FBVolume

    sh = phantoms.random_quadric_phantom(3, n_ellipsoids=10, n_cylinders=5)
    v = FBVolume(sh)
    lo, hi = v.get_bbox()
    assert np.all(lo < hi)
    assert len(v.prune_to_bbox(lo, hi).shapes) == 15
    assert len(v.prune_to_bbox((1e4, 1e4, 1e4), (2e4, 2e4, 2e4)).shapes) == 0


# ---------------------------------------------------------------- GPU
def _gpu_project(shapes, pg, **cfg):
    from aprict_b200 import FBVolume
    from aprict_b200.cb import flatpanel as fp

    ps = fp.ProjectionSet(pg, data=None)
    fp.project(fp.ConfigProject(**cfg), FBVolume(shapes), ps, block=True)
    return ps.data.cpu().numpy(), ps.out_of_mem_count


@pytest.mark.gpu
@pytest.mark.parametrize(
    ("mode_kw", "mode"),
    [({}, 0), ({"overlap_addition": True}, 1), ({"overlap_addition": True, "additive_line_integral": True}, 2)],
)
def test_gpu_matches_oracle_all_types(mode_kw: dict, mode: int) -> None:
    rng = np.random.default_rng(11)
    shapes = random_shapes_all_types(rng, 64)
    pg = circular(8, 150, 150, 0.5, 64, 48)
    got, ovf = _gpu_project(shapes, pg, **mode_kw)
    want = O.project_forbild(pg.to_proj_spec_array(), shapes, mode=mode)
    assert ovf == 0
    assert np.linalg.norm(want) > 0
    assert rel_l2(got, want) <= 1e-5


@pytest.mark.gpu
def test_gpu_supersampling_multiply_and_chunks() -> None:
    """More shapes than one shared-memory chunk (128), ssu/ssv > 1, mba != 1."""
    rng = np.random.default_rng(12)
    shapes = random_shapes_all_types(rng, 200, radius=60)
    pg = circular(4, 150, 150, 0.5, 48, 40)
    got, _ = _gpu_project(shapes, pg, ssu=2, ssv=3, multiply_before_adding=-1.5)
    want = O.project_forbild(pg.to_proj_spec_array(), shapes, mode=0, ssu=2, ssv=3, mba=-1.5)
    assert rel_l2(got, want) <= 1e-5


@pytest.mark.gpu
def test_gpu_matches_reference_quadric_phantom() -> None:
    if not O.have_ref():
        pytest.skip("reference oracle not built")
    shapes = phantoms.random_quadric_phantom(4, n_ellipsoids=12, n_cylinders=8, radius=60)
    pg = circular(6, 200, 150, 0.4, 64, 64)
    for kw, ovl in (({}, False), ({"overlap_addition": True}, True)):
        got, _ = _gpu_project(shapes, pg, **kw)
        ref, _ = O.ref_project_forbild(pg.to_proj_spec_array(), shapes, overlap_addition=ovl)
        assert rel_l2(got, ref) <= 1e-4


@pytest.mark.gpu
def test_gpu_fan_and_empty() -> None:
    rng = np.random.default_rng(13)
    shapes = random_shapes_all_types(rng, 20)
    pg = circular(10, 150, 150, 0.5, 96, 1)
    got, _ = _gpu_project(shapes, pg)
    want = O.project_forbild(pg.to_proj_spec_array(), shapes, mode=0)
    assert rel_l2(got, want) <= 1e-5
    empty = shapes[:0]
    got0, _ = _gpu_project(empty, pg)
    assert float(np.abs(got0).max()) == 0.0


# ------------------------------------------------- polynomial forms of the ray
_SEED_PROBE = """
#include "ab_common.cuh"
__global__ void k(const double *x, double *r, double *s, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        r[i] = ab_rcp_h3(x[i]);
        s[i] = x[i] > 0.0 ? ab_sqrt_h3(x[i]) : 0.0;
    }
}
extern "C" __attribute__((visibility("default"))) int run(const double *x, double *r, double *s, int n) {
    k<<<(n + 255) / 256, 256>>>(x, r, s, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.gpu
def test_third_order_steps_on_the_device(tmp_path) -> None:  # noqa: ANN001
    """ab_rcp_h3 and ab_sqrt_h3 as the kernels compile them: within one unit in the last place of the rounded 1 / x and
    sqrt(x), over the exponents that the projectors meet (1e-300, the least step along an axis, to 2^300; roots from
    2^-300), powers of two and their neighbours among them."""
    import ctypes
    import subprocess

    import torch

    from aprict_b200 import build

    (tmp_path / "probe.cu").write_text(_SEED_PROBE)
    lib = tmp_path / "probe.so"
    subprocess.run([build._nvcc(), *build.ARCH_FLAGS, *build.NVCC_FLAGS, f"-I{build.INCLUDE}", f"-I{build.CSRC}", "-shared",
                    str(tmp_path / "probe.cu"), "-o", str(lib)], check=True, capture_output=True)
    run = ctypes.CDLL(str(lib)).run
    rng = np.random.default_rng(6)
    two = np.ldexp(1.0, np.arange(-996, 301))
    x = np.concatenate([np.ldexp(rng.uniform(1, 2, 4_000_000), rng.integers(-996, 300, 4_000_000)), two, np.nextafter(two, 0),
                        np.nextafter(two, np.inf), [1e-300, -1e-300, 3.0, -7.0]])
    d, r, s = torch.from_numpy(x).cuda(), *torch.zeros((2, len(x)), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert run(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(r.data_ptr()), ctypes.c_void_p(s.data_ptr()), len(x)) == 0
    want = 1.0 / x
    assert (np.abs(r.cpu().numpy() - want) / np.spacing(np.abs(want))).max() <= 1.0
    k = x > 2.0**-300
    want = np.sqrt(x[k])
    assert (np.abs(s.cpu().numpy()[k] - want) / np.spacing(want)).max() <= 1.0


def test_third_order_steps_bound() -> None:
    """One third-order Householder step from a seed good to 2^-19.9 gives 1 / x and sqrt(x) to the seed's error cubed
    (2^-59.7; for the root, with e twice the seed's, 5/16 of 2^-56.7) and the last steps' rounding: 1.5 and 2 units of 2^-53. Same operations, each
    rounded once, as the device code."""
    from fractions import Fraction as F
    from math import isqrt

    def fma(a: float, b: float, c: float) -> float:
        return float(F(a) * F(b) + F(c))

    rng = np.random.default_rng(5)
    for _ in range(400):
        x = float(np.ldexp(rng.uniform(1.0, 2.0), int(rng.integers(-200, 200))))
        off = float(1.0 + rng.uniform(-1.0, 1.0) * 2.0**-19.9)
        y = (1.0 / x) * off
        e = fma(-x, y, 1.0)
        r = fma(y, fma(e, e, e), y)
        assert abs(F(r) * F(x) - 1) <= F(3, 2) * F(1, 2**53) + F(1, 2**59)
        y = (1.0 / np.sqrt(x)) * off
        h = x * y
        e = fma(-h, y, 1.0)
        s = fma(h, e * fma(0.375, e, 0.5), h)
        root = F(isqrt(int(F(x) * 2**800)), 2**400)  # sqrt(x) to 2^-200 of it
        assert abs(F(s) / root - 1) <= 2 * F(1, 2**53) + F(1, 2**57)


def _edge_shapes() -> np.ndarray:
    """Ellipsoids and cylinders against source (at x = 150) and detector (at x = -150): axis along the central ray,
    source or detector inside, behind either, far larger than the ray, clipped through the middle."""
    rng = np.random.default_rng(21)
    sh = random_shapes_all_types(rng, 12, types=(7, 7, 11, 11, 13, 13, 13, 13, 6, 12, 11, 11))
    for k, (c, r, ln) in enumerate(
        [((0, 0, 0), 6.0, 40.0), ((0, 0.4, 0), 0.3, 200.0), ((150, 0, 0), 9.0, 0), ((-150, 3, 0), 9.0, 0), ((0, 0, 0), 190.0, 0),
         ((175, 0, 0), 11.0, 0), ((-175, 0, 0), 11.0, 0), ((10, 5, -4), 7.0, 0), ((-20, 0, 6), 5.0, 320.0), ((30, 0, -8), 8.0, 15.0),
         ((0, 10, 0), 12.0, 0), ((0, -10, 9), 12.0, 0)]):
        rec = sh[k]
        rec["x"], rec["y"], rec["z"] = c
        rec["r"], rec["l"] = r, ln or rec["l"]
        if k != 4:
            rec["dx"], rec["dy"], rec["dz"] = r, 0.7 * r, 0.4 * r
        if k < 10:
            for f in ("cas1", "cas2", "cas3"):
                rec[f]["mode"] = 0
    return sh


@pytest.mark.gpu
@pytest.mark.parametrize(("mode_kw", "mode"), [({}, 0), ({"overlap_addition": True}, 1),
                                               ({"overlap_addition": True, "additive_line_integral": True}, 2)])
@pytest.mark.parametrize("alone", [True, False])
def test_gpu_ray_forms_at_their_edges(mode_kw: dict, mode: int, alone: bool) -> None:
    """Every pixel, against the FP64 oracle: its roots come from B^2 - A C, which at a tangent keeps
    sqrt(2^-53 (150 / 0.12)^2), about 1e-5 of the smallest solid's chord and 3e-7 of the largest's, and the result is FP32."""
    shapes = _edge_shapes()
    pg = circular(2, 150, 150, 0.5, 65, 49, theta0=0.0)  # odd: the central ray is the x axis
    for sh in (shapes[k : k + 1] for k in range(len(shapes))) if alone else (shapes,):
        got, _ = _gpu_project(sh, pg, **mode_kw)
        want = O.project_forbild(pg.to_proj_spec_array(), sh, mode=mode)
        top = np.abs(want).max()
        assert np.abs(got - want).max() <= 2e-5 * max(top, 1e-30), sh["type"]
        assert rel_l2(got, want) <= 1e-6 if top > 0 else not got.any()


def _end_on(n: int, theta: float, axis: str) -> np.ndarray:
    """Cylinders of radius 6 along the central ray of the view at ``theta``, their axes up to 3 off it: the ray lies
    inside, parallel to the axis."""
    rng = np.random.default_rng(31)
    sh = np.zeros(n, S.forbild_shape)
    for k in range(n):
        rec = sh[k]
        rec["type"], rec["rho"], rec["r"], rec["l"] = {"x": 7, "y": 8, "free": 6}[axis], 0.7, 6.0, 40.0
        rec["x"], rec["y"], rec["z"] = rng.uniform(-3, 3, 3)
        rec["axis"] = (np.cos(theta), np.sin(theta), 0.0)
    return sh


@pytest.mark.gpu
@pytest.mark.parametrize(("theta", "axis"), [(0.0, "x"), (0.5 * np.pi, "y"), (0.0, "free"), (0.7, "free")])
@pytest.mark.parametrize("nu", [65, 64])
def test_gpu_cylinders_seen_end_on(theta: float, axis: str, nu: int) -> None:
    """Rays along a cylinder's axis have A = 0 and a discriminant of 0, either sign by rounding: inside they get the
    whole chord. Every pixel, against the FP64 oracle at the FP32 result's rounding."""
    pg = circular(1, 150, 150, 0.5, nu, 49, theta0=theta)
    for sh in _end_on(60, theta, axis).reshape(-1, 1):
        got, _ = _gpu_project(sh, pg)
        want = O.project_forbild(pg.to_proj_spec_array(), sh, mode=0)
        assert want[0, nu // 2, 24] > 0.7 * 39.0
        assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()


@pytest.mark.gpu
def test_gpu_solids_beside_the_source() -> None:
    """Solids around the source whose centre lies beside it, in front by little more than the records' rounding, project
    to billions of pixels: the forms about that centre have no bits left at the detector's, where the general solver has
    to run."""
    rng = np.random.default_rng(32)
    theta = 0.3
    pg = circular(1, 150, 150, 0.5, 65, 49, theta0=theta)
    sp = pg.to_proj_spec_array()[0]
    sh = np.zeros(4000, S.forbild_shape)
    sh["type"], sh["rho"], sh["r"] = 13, 0.4, rng.uniform(25, 60, len(sh))
    b, e = rng.uniform(-15, 15, len(sh)), 10.0 ** rng.uniform(-9, -5, len(sh))
    sh["x"], sh["y"] = (150 - e) * np.cos(theta) - b * np.sin(theta), (150 - e) * np.sin(theta) + b * np.cos(theta)
    sh["z"] = rng.uniform(-5, 5, len(sh))
    f = lambda v: np.array([v["x"], v["y"], v["z"]], np.float64)  # noqa: E731
    n, s = np.cross(f(sp["det_u"]), f(sp["det_v"])), f(sp["source_pos"])
    ahead = (np.stack([sh["x"], sh["y"], sh["z"]], 1).astype(np.float64) - s) @ n * np.sign((f(sp["det_pos"]) - s) @ n)
    ahead[ahead <= 0] = np.inf
    for k in np.argsort(ahead)[:40]:
        got, _ = _gpu_project(sh[k : k + 1], pg)
        want = O.project_forbild(pg.to_proj_spec_array(), sh[k : k + 1], mode=0)
        assert want.min() > 0
        assert np.abs(got - want).max() <= 2e-6 * want.max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [127, 128, 129])
def test_gpu_around_one_chunk(n: int) -> None:
    """Phantoms of one chunk (kept between the sub-rays of a tile) and of one shape more."""
    shapes = random_shapes_all_types(np.random.default_rng(n), n, radius=60)
    pg = circular(2, 150, 150, 0.5, 48, 40)
    got, _ = _gpu_project(shapes, pg, ssu=2, ssv=2)
    want = O.project_forbild(pg.to_proj_spec_array(), shapes, mode=0, ssu=2, ssv=2)
    assert rel_l2(got, want) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("views", [0, 1, 4, 6])
def test_gpu_projects_when_memory_is_short(views: int, monkeypatch: pytest.MonkeyPatch) -> None:
    """Scratch for all 18 views' records not to be had, only some views' or none: the same projections."""
    import torch

    from aprict_b200 import _lib

    shapes = random_shapes_all_types(np.random.default_rng(4), 30)
    pg = circular(18, 150, 150, 0.5, 40, 33)
    want, _ = _gpu_project(shapes, pg)
    limit, empty, asked = int(_lib.lib().aprict_b200_project_forbild_scratch_bytes(views, 30)), torch.empty, []

    def short(*a: object, **k: object) -> torch.Tensor:
        if k.get("dtype") == torch.uint8:
            asked.append(a[0])
            if a[0] > limit:
                raise torch.cuda.OutOfMemoryError
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", short)
    got, _ = _gpu_project(shapes, pg)
    assert asked and asked[0] > limit
    np.testing.assert_array_equal(got, want)
