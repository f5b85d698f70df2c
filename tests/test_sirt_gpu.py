"""SIRT / Landweber on the GPU vs the same iterations composed from FP64 oracle operators.

Gate: rel L2 <= 1e-4 on the reconstruction (the stated tolerance for
reconstructions). The oracle SIRT restates src/aprict/iterators/sirt_vram.py:62-152
step by step in numpy/FP64.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from aprict_b200 import Volume, phantoms
from aprict_b200.cb import flatpanel as fp
from aprict_b200.iterators import Landweber_flatpanel, SIRT_flatpanel
from helpers import circular, rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPE = (40, 40, 32)


def softmask(a: np.ndarray, r0: float) -> np.ndarray:
    X, Y, _ = a.shape
    ix = np.arange(X)[:, None, None] - (X - 1) / 2
    iy = np.arange(Y)[None, :, None] - (Y - 1) / 2
    rr = np.sqrt(ix**2 + iy**2) / min(X, Y) * 2
    if r0 >= 1:
        m = np.where(rr < 1, 1.0, 0.0)
    else:
        t = np.clip((rr - r0) / (1 - r0), None, 1)
        m = np.where(rr < r0, 1.0, np.clip((1 + np.cos(np.pi * t)) / 2, 0, 1))
    return a * m


class OracleSIRT:
    def __init__(self, pg: fp.ProjGeom, b: np.ndarray) -> None:
        self.specs = pg.to_proj_spec_array()
        self.corner = -np.array(SHAPE, np.float32) / 2
        self.b = b.astype(np.float64)
        cyl = min(SHAPE[:2]) / 2
        self.cfg = fp.ConfigBackproject(fast_approx=True, cyl_mask_rad=cyl, soften_det_edges_proportion=0.05).contents
        s = 1 / float(np.mean(SHAPE))
        M = softmask(np.full(SHAPE, s), 1.0)
        p = self.A(M)
        meanval = p.mean()
        p /= meanval / s
        s /= meanval / s
        M = self.B(p)
        M = np.where(M == 0, 0, 1 / (M + 0.1 * np.exp(-M / 0.1))) * s
        self.M = softmask(M, 0.95)
        self.x = np.zeros(SHAPE)

    def A(self, x: np.ndarray) -> np.ndarray:
        return O.project_siddon(self.specs, x.astype(np.float32), voxwid=1.0, corner=self.corner)[0]

    def B(self, p: np.ndarray) -> np.ndarray:
        return O.backproject(self.specs, p, SHAPE, self.cfg, voxwid=1.0, corner=self.corner)

    def iterate(self) -> None:
        r = self.b - self.A(self.x)
        self.x = self.x + self.M * self.B(r)


def _problem():
    pg = circular(30, 100, 100, 0.537, 56, 48)
    xt = phantoms.ellipsoid_volume(21, 6, SHAPE, 1.0, semi_axes_vox=(3, 12))
    v = Volume(xt, voxwid=1.0)
    ps = fp.ProjectionSet(pg, data=None)
    fp.project(fp.ConfigProject(), v, ps, block=True)
    return pg, xt, ps.data.clone()


def test_sirt_matches_fp64_iterations() -> None:
    pg, _, b = _problem()
    ora = OracleSIRT(pg, b.cpu().numpy())
    x = Volume.zeros(SHAPE, voxwid=1.0)
    sirt = SIRT_flatpanel(SIRT_flatpanel.Config(), x, fp.ProjectionSet(pg, data=b))
    assert rel_l2(sirt.preconditioner.as_numpy(), ora.M) <= 1e-5
    for _ in range(4):
        sirt.iterate()
        ora.iterate()
    torch.cuda.synchronize()
    assert rel_l2(x.as_numpy(), ora.x) <= 1e-4


def test_graph_replay_equals_eager() -> None:
    pg, _, b = _problem()
    xa = Volume.zeros(SHAPE, voxwid=1.0)
    xb = Volume.zeros(SHAPE, voxwid=1.0)
    sa = SIRT_flatpanel(SIRT_flatpanel.Config(), xa, fp.ProjectionSet(pg, data=b.clone()))
    sb = SIRT_flatpanel(SIRT_flatpanel.Config(), xb, fp.ProjectionSet(pg, data=b.clone()))
    for _ in range(6):
        sa.iterate()
    sb.iterate_graph(3)
    sb.iterate_graph(3)
    torch.cuda.synchronize()
    assert sb.iterations == 6
    # the projection uses atomics only in accumulate mode; the residual path is deterministic
    assert rel_l2(xb.as_numpy(), xa.as_numpy()) <= 1e-6


def test_iterate_from_host_equals_eager() -> None:
    # a different measurement every step (as a stream of scans would give) and the
    # volume read back after each: the pipelined transfers change no result
    pg, _, b = _problem()
    xa = Volume.zeros(SHAPE, voxwid=1.0)
    xb = Volume.zeros(SHAPE, voxwid=1.0)
    sa = SIRT_flatpanel(SIRT_flatpanel.Config(), xa, fp.ProjectionSet(pg, data=b.clone()))
    sb = SIRT_flatpanel(SIRT_flatpanel.Config(), xb, fp.ProjectionSet(pg, data=b.clone()))
    bs = [(b * (1.0 + 0.1 * k)).cpu().pin_memory() for k in range(5)]
    outs = [torch.empty(SHAPE, dtype=torch.float32).pin_memory() for _ in range(5)]
    want = []
    for k in range(5):
        sa._meas.data.copy_(bs[k])  # noqa: SLF001
        sa.iterate()
        want.append(xa.as_numpy().copy())
    for k in range(5):
        sb.iterate_from_host(bs[k], outs[k])
    sb.host_sync()
    assert sb.iterations == 5
    for k in range(5):
        assert rel_l2(outs[k].numpy(), want[k]) <= 1e-6
    assert np.abs(want[4] - want[3]).max() > 0
    assert torch.equal(sb._meas.data, b)  # noqa: SLF001  the caller's ProjectionSet is untouched


def test_sirt_converges_and_checkpoints(tmp_path) -> None:
    pg, xt, b = _problem()
    x = Volume.zeros(SHAPE, voxwid=1.0)
    sirt = SIRT_flatpanel(SIRT_flatpanel.Config(), x, fp.ProjectionSet(pg, data=b))
    res = []
    for _ in range(8):
        r = fp.ProjectionSet(pg, data=None)
        fp.project_residual(fp.ConfigProject(multiply_before_adding=-1), x, r, b)
        res.append(float(torch.linalg.vector_norm(r.data)))
        sirt.iterate()
    assert res[-1] < 0.5 * res[0]
    assert all(b2 <= b1 * 1.0001 for b1, b2 in zip(res, res[1:]))
    sd = sirt.state_dict()
    torch.save(sd, tmp_path / "ck.pt")
    x2 = Volume.zeros(SHAPE, voxwid=1.0)
    s2 = SIRT_flatpanel(SIRT_flatpanel.Config(), x2, fp.ProjectionSet(pg, data=b))
    s2.load_state_dict(torch.load(tmp_path / "ck.pt"))
    sirt.iterate()
    s2.iterate()
    torch.cuda.synchronize()
    assert s2.iterations == sirt.iterations
    assert rel_l2(x2.as_numpy(), x.as_numpy()) <= 1e-6


def test_classical_sirt_converges() -> None:
    pg, _, b = _problem()
    x = Volume.zeros(SHAPE, voxwid=1.0)
    sirt = SIRT_flatpanel(SIRT_flatpanel.Config(mode="classical"), x, fp.ProjectionSet(pg, data=b))
    r0 = float(torch.linalg.vector_norm(b))
    for _ in range(10):
        sirt.iterate()
    r = fp.ProjectionSet(pg, data=None)
    fp.project_residual(fp.ConfigProject(multiply_before_adding=-1), x, r, b)
    assert float(torch.linalg.vector_norm(r.data)) < 0.3 * r0


def test_landweber_ordered_subsets() -> None:
    pg, _, b = _problem()
    subsets = [fp.ProjectionSet(pg.sliced(slice(k, None, 2)), data=b[k::2].contiguous()) for k in range(2)]
    x = Volume.zeros(SHAPE, voxwid=1.0)
    lw = Landweber_flatpanel(Landweber_flatpanel.Config(seed=3, exact_adjoint=True), x, subsets)
    assert all(q > 0 for q in lw.rayleigh_quotients)
    r0 = float(torch.linalg.vector_norm(b))
    for _ in range(6):
        lw.iterate()
    r = fp.ProjectionSet(pg, data=None)
    fp.project_residual(fp.ConfigProject(multiply_before_adding=-1), x, r, b)
    assert float(torch.linalg.vector_norm(r.data)) < 0.5 * r0


def test_c_abi_sirt_step_and_graph_equal_the_python_iterator() -> None:
    """aprict_b200_sirt_step / sirt_graph_* (the C entry points) against SIRT_flatpanel."""
    import ctypes

    from aprict_b200 import _lib

    pg, _, b = _problem()
    sa = SIRT_flatpanel(SIRT_flatpanel.Config(), Volume.zeros(SHAPE, voxwid=1.0), fp.ProjectionSet(pg, data=b.clone()))
    sb = SIRT_flatpanel(SIRT_flatpanel.Config(), Volume.zeros(SHAPE, voxwid=1.0), fp.ProjectionSet(pg, data=b.clone()))
    lib = _lib.lib()
    stream = torch.cuda.current_stream().cuda_stream
    meas, r, x, M = sb._meas, sb._scratch, sb.volume, sb.preconditioner  # noqa: SLF001
    pd = _lib.proj_desc(tuple(r.data.shape), tuple(r.data.stride()))
    vd = x._desc()  # noqa: SLF001
    cfg = sb._config_bp.contents  # noqa: SLF001
    args = (meas.specs_device().data_ptr(), _lib.ptr(pd), meas.data.data_ptr(), r.data.data_ptr(), _lib.ptr(vd),
            x.data.data_ptr(), M.data.data_ptr(), _lib.ptr(cfg), None)
    for _ in range(2):
        sa.iterate()
        _lib.check(lib.aprict_b200_sirt_step(*args, stream), "sirt_step")
    torch.cuda.synchronize()
    assert torch.equal(sa.volume.data, x.data)
    g = ctypes.c_void_p()
    _lib.check(lib.aprict_b200_sirt_graph_create(*args, 3, ctypes.byref(g)), "sirt_graph_create")
    try:
        assert lib.aprict_b200_sirt_graph_iterations(g) == 3
        _lib.check(lib.aprict_b200_sirt_graph_launch(g, stream), "sirt_graph_launch")
        for _ in range(3):
            sa.iterate()
        torch.cuda.synchronize()
        assert rel_l2(x.as_numpy(), sa.volume.as_numpy()) <= 1e-6
    finally:
        lib.aprict_b200_sirt_graph_destroy(g)
    with pytest.raises(ValueError):
        _lib.check(lib.aprict_b200_sirt_step(*args[:6], None, _lib.ptr(cfg), None, stream), "sirt_step")


@pytest.mark.parametrize("kind", ["upright", "tilted"])
def test_c_abi_sirt_with_and_without_a_promise(kind: str) -> None:
    """A step and a graph of two, with what is known of the views and without: the same kernel's sums."""
    import ctypes

    from aprict_b200 import _lib
    from helpers import jittered

    pg, _, b = _problem()
    if kind == "tilted":
        pg = jittered(np.random.default_rng(3), pg)
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    ps = fp.ProjectionSet(pg, data=b.clone())
    specs, pd, dptr = fp._view_args(ps, (), 0)  # noqa: SLF001
    cfg = fp.ConfigBackproject(fast_approx=True, apply_summand_multiplier=True).contents
    M = Volume.zeros(SHAPE, voxwid=1.0)  # noqa: N806
    M.fill(1e-5)
    out = []
    for views in (0, ps._backproject_promise(False)):  # noqa: SLF001
        x, r = Volume.zeros(SHAPE, voxwid=1.0), torch.zeros_like(b)
        vd = x._desc()  # noqa: SLF001
        args = (specs, _lib.ptr(pd), dptr, r.data_ptr(), _lib.ptr(vd), x.data.data_ptr(), M.data.data_ptr(), _lib.ptr(cfg), views, None)
        _lib.check(lib.aprict_b200_sirt_step_views(*args, stream), "sirt_step")
        torch.cuda.synchronize()
        g = ctypes.c_void_p()
        _lib.check(lib.aprict_b200_sirt_graph_create_views(*args, 2, ctypes.byref(g)), "sirt_graph_create")
        _lib.check(lib.aprict_b200_sirt_graph_launch(g, stream), "sirt_graph_launch")
        torch.cuda.synchronize()
        lib.aprict_b200_sirt_graph_destroy(g)
        out.append(x.as_numpy())
    assert np.linalg.norm(out[0]) > 0
    np.testing.assert_array_equal(out[0], out[1])
    with pytest.raises(ValueError):
        _lib.check(lib.aprict_b200_sirt_step_views(*args[:8], 4, None, stream), "sirt_step")
