"""What is measured: the calls that a user's reconstruction program makes, over the sizes and options it makes them with.

A case is one pass through a public entry point (``op``):

* ``project``      Siddon forward projection of a voxel volume (``cb.flatpanel.project``);
* ``gradient``     data-fit gradient through autograd: A x, then A^T (A x - b) (``autograd.SiddonProjector``);
* ``backproject``  one backprojection in one of its modes (``cb.flatpanel.backproject``);
* ``sirt``         one SIRT iteration (``iterators.SIRT_flatpanel.iterate``);
* ``sirt_batch``   one SIRT iteration of several uneven scans (``iterators.SIRTBatch.iterate``);
* ``fan_fbp``      fan-beam FBP of a stack of slices (``recon.fbp_fan_circ_batch``);
* ``cone_fbp``     cone-cylinder FBP (``recon.fbp_cone_cyl``);
* ``gbc``          GBC backprojection with its weight sums (``cb.flatpanel.backproject``, preset 7);
* ``gbc_weights``  the GBC expected-weight integral (``gbc.weightinteg``);
* ``quadric``      analytic projection of a quadric phantom (``FBVolume`` through ``project``).

``exact`` restates each of them in 64 bits with torch and numpy alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

PHOTONS = 1e5  # per detector pixel, for the noise of simulated measurements


# ------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    """The listed cases."""
    return [
        # A test-sized scan: a quick look at a geometry, or one call of a small tool, where launches and host work count.
        dict(name="project_small", op="project", nx=40, ny=36, nz=32, views=12, nu=50, nv=42, order="C", half=False,
             helical=0.0, tilt=False, ss=1),
        # The ordinary forward projection: simulation of a scan of a 128^3 volume.
        dict(name="project_128", op="project", nx=128, ny=128, nz=128, views=180, nu=256, nv=256, order="C", half=False,
             helical=0.0, tilt=False, ss=1),
        # One step of gradient descent or of a learned reconstruction: forward and backward.
        dict(name="gradient_128", op="gradient", nx=128, ny=128, nz=128, views=180, nu=256, nv=256, helical=0.0, tilt=False),
        # The matched backprojector, as Landweber with the exact adjoint calls it.
        dict(name="backproject_exact_128", op="backproject", mode="exact", nx=128, ny=128, nz=128, views=180, nu=256,
             nv=256, order="C", taper=0.0, mask=False, mult=False, helical=0.0, tilt=False),
        # Smooth sampling into a ragged volume, with the multiplier and the detector-edge taper of the iterators.
        dict(name="backproject_bilinear", op="backproject", mode="bilinear", nx=210, ny=190, nz=150, views=200, nu=301,
             nv=243, order="C", taper=0.05, mask=True, mult=True, helical=0.0, tilt=False),
        # The iteration that most programs spend their time in, at its ordinary size.
        dict(name="sirt_256", op="sirt", n=256, nz=256, views=360, nu=384, nv=384),
        # Many small, uneven scans with calibrated (jittered) geometries, circular and helical, iterated together.
        dict(name="sirt_batch", op="sirt_batch", scans=12, edge_lo=64, edge_hi=192, views_lo=90, views_hi=360, det_lo=128,
             det_hi=384, layout=5),
        # A stack of fan-beam slices.
        dict(name="fan_fbp_64", op="fan_fbp", slices=64, n=512, views=720, nu=1024, hann=True),
        # A whole cone-cylinder reconstruction: tilted filter, then the direct-raycast backprojection.
        dict(name="cone_fbp_256", op="cone_fbp", n=256, nz=256, views=720, nu=384, nv=384, turn=0.3125, interpolate=False),
        # The backprojection of a GBC reconstruction into its padded volume.
        dict(name="gbc_198", op="gbc", n=198, nz=198, views=360, nu=256, nv=256, interpolate=True),
        # The expected weights of that padded volume's voxel grid.
        dict(name="gbc_weights_198", op="gbc_weights", n=198, z_samps=6000, ang_samps=6000),
        # The analytic projection of a phantom of clipped quadrics onto a large detector.
        dict(name="quadric_1024", op="quadric", ellipsoids=60, cylinders=40, views=240, nu=1024, nv=1024, additive=True),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c: dict) -> float:
    """Rough share of a pass's arithmetic relative to the largest listed case (at most 1 for a drawn one)."""
    op = c["op"]
    if op in ("project", "gradient"):
        steps = c["views"] * c["nu"] * c["nv"] * 1.3 * (c["nx"] + c["ny"] + c["nz"]) / 3 * c.get("ss", 1) ** 2
        return steps * (2.5 if op == "gradient" else 1.0) / 2.5e10
    if op == "backproject":
        return c["nx"] * c["ny"] * c["nz"] * c["views"] * (8 if c["mode"] == "exact" else 2) / 1.2e10
    if op == "sirt":
        return (c["n"] ** 2 * c["nz"] * c["views"] + c["views"] * c["nu"] * c["nv"] * 1.2 * c["n"]) / 2.4e10
    if op == "sirt_batch":
        return c["scans"] * (math.sqrt(c["edge_lo"] * c["edge_hi"])) ** 3 * (c["views_lo"] + c["views_hi"]) / 2.0e10
    if op == "fan_fbp":
        return c["slices"] * c["n"] ** 2 * c["views"] / 1.21e10
    if op == "cone_fbp":
        return c["n"] ** 2 * c["nz"] * c["views"] / 1.21e10
    if op == "gbc":
        return c["n"] ** 2 * c["nz"] * c["views"] / 5e9
    if op == "gbc_weights":
        return 2 * c["n"] * c["z_samps"] * c["ang_samps"] / 2.8e10
    return c["views"] * c["nu"] * c["nv"] * (c["ellipsoids"] + c["cylinders"]) / 2.6e10


def draw(rng) -> dict:
    """One more case of the same ranges."""
    while True:
        op = rng.choice(["project", "gradient", "backproject", "backproject", "sirt", "sirt_batch", "fan_fbp", "cone_fbp",
                         "gbc", "gbc_weights", "quadric"])
        det = lambda: dict(nu=_log_int(rng, 40, 640), nv=_log_int(rng, 40, 480))  # noqa: E731
        vol = lambda: dict(nx=_log_int(rng, 24, 288), ny=_log_int(rng, 24, 288), nz=_log_int(rng, 16, 288))  # noqa: E731
        scan = lambda: dict(helical=rng.choice([0.0, 0.0, round(rng.uniform(0.5, 1.5), 3)]),  # noqa: E731
                            tilt=rng.random() < 0.25)
        if op == "project":
            c = dict(op=op, **vol(), views=_log_int(rng, 8, 400), **det(), order=rng.choice("CCF"), half=rng.random() < 0.2,
                     **scan(), ss=rng.choice([1, 1, 1, 2]))
        elif op == "gradient":
            c = dict(op=op, **vol(), views=_log_int(rng, 8, 300), **det(), **scan())
        elif op == "backproject":
            c = dict(op=op, mode=rng.choice(["exact", "nearest", "bilinear", "raycast"]), **vol(),
                     views=_log_int(rng, 8, 400), **det(), order=rng.choice("CCF"), taper=rng.choice([0.0, 0.05]),
                     mask=rng.random() < 0.5, mult=rng.random() < 0.5, **scan())
        elif op == "sirt":
            n = _log_int(rng, 40, 256)
            c = dict(op=op, n=n, nz=max(16, int(n * rng.uniform(0.4, 1.1))), views=_log_int(rng, 30, 400), **det())
        elif op == "sirt_batch":
            lo = _log_int(rng, 32, 96)
            c = dict(op=op, scans=rng.randint(2, 14), edge_lo=lo, edge_hi=2 * lo, views_lo=30, views_hi=rng.randint(60, 360),
                     det_lo=64, det_hi=rng.randint(96, 384), layout=rng.randint(0, 1 << 20))
        elif op == "fan_fbp":
            c = dict(op=op, slices=_log_int(rng, 1, 64), n=_log_int(rng, 64, 512), views=_log_int(rng, 60, 720),
                     nu=_log_int(rng, 100, 1400), hann=rng.random() < 0.5)
        elif op == "cone_fbp":
            n = _log_int(rng, 48, 256)
            c = dict(op=op, n=n, nz=max(24, int(n * rng.uniform(0.5, 1.2))), views=_log_int(rng, 60, 720),
                     nu=_log_int(rng, 96, 512), nv=_log_int(rng, 96, 384), turn=round(rng.uniform(0.2, 0.6), 4),
                     interpolate=rng.random() < 0.3)
        elif op == "gbc":
            n = _log_int(rng, 40, 198)
            c = dict(op=op, n=n, nz=max(24, int(n * rng.uniform(0.5, 1.1))), views=_log_int(rng, 40, 360),
                     nu=_log_int(rng, 96, 320), nv=_log_int(rng, 96, 320), interpolate=rng.random() < 0.6)
        elif op == "gbc_weights":
            c = dict(op=op, n=_log_int(rng, 20, 198), z_samps=_log_int(rng, 500, 6000), ang_samps=_log_int(rng, 500, 6000))
        else:
            c = dict(op=op, ellipsoids=rng.randint(3, 60), cylinders=rng.randint(0, 40), views=_log_int(rng, 8, 240),
                     nu=_log_int(rng, 100, 1024), nv=_log_int(rng, 100, 1024), additive=rng.random() < 0.5)
        if _cost(c) <= 1.0:
            return c


# ----------------------------------------------------------- inputs, from the seed
VOX = 0.5  # mm
R, LMR = 500.0, 500.0  # source to axis, axis to detector (mm)


def _scan(views: int, nu: int, nv: int, pix: float, theta0: float, *, helical: float = 0.0, rng=None) -> dict:
    """A circular scan, or one helical turn of that pitch (in detector heights), with a gantry start angle; with
    ``rng``, per-view positions and detector orientations as a calibration finds them. Detector pixels of ``pix`` at the axis."""
    t = theta0 + 2 * np.pi * np.arange(views) / views
    z = helical * nv * pix * (np.arange(views) / views - 0.5)
    p = pix * (R + LMR) / R
    src = np.stack([R * np.cos(t), R * np.sin(t), z], 1)
    det = np.stack([-LMR * np.cos(t), -LMR * np.sin(t), z], 1)
    u = p * np.stack([-np.sin(t), np.cos(t), 0 * t], 1)
    v = np.tile(p * np.array([0.0, 0.0, -1.0]), (views, 1))
    if rng is not None:
        src = src + rng.uniform(-2, 2, src.shape)
        det = det + rng.uniform(-2, 2, det.shape)
        ax = rng.standard_normal((views, 3))
        ax /= np.linalg.norm(ax, axis=1, keepdims=True)
        ang = np.deg2rad(rng.uniform(-0.5, 0.5, (views, 1)))
        turn = lambda w: w * np.cos(ang) + np.cross(ax, w) * np.sin(ang) + ax * (ax * w).sum(1, keepdims=True) * (1 - np.cos(ang))  # noqa: E731
        u, v = turn(u), turn(v)
    return dict(src=src.astype(np.float32), det=det.astype(np.float32), u=u.astype(np.float32), v=v.astype(np.float32), nu=nu, nv=nv)


def _cylinder(views: int, nu: int, nv: int, pix: float, height: float, theta0: float) -> dict:
    """Golden-angle sources on a cylinder of that height (the scan of the cone-cylinder methods)."""
    t = theta0 + np.arange(views) * (np.sqrt(5) - 1) * np.pi
    z = np.linspace(-height / 2, height / 2, views + 2)[1:-1]
    p = pix * (R + LMR) / R
    src = np.stack([R * np.cos(t), R * np.sin(t), z], 1)
    det = np.stack([-LMR * np.cos(t), -LMR * np.sin(t), z], 1)
    u = p * np.stack([-np.sin(t), np.cos(t), 0 * t], 1)
    v = np.tile(p * np.array([0.0, 0.0, -1.0]), (views, 1))
    return dict(src=src.astype(np.float32), det=det.astype(np.float32), u=u.astype(np.float32), v=v.astype(np.float32), nu=nu, nv=nv)


def _pix(extent: float, n: int, tall: int | None = None, height: float = 0.0) -> float:
    """A pixel pitch at the axis that lets ``n`` pixels (and ``tall`` ones in height) cover the object with a margin; not a
    round fraction of a voxel."""
    p = 1.2347 * extent / n
    return max(p, 1.1731 * height / tall) if tall else p


def _blobs(rng, count: int, half: np.ndarray, flat: bool = False) -> list[tuple]:
    """Ellipsoids (centre, axes matrix to the unit ball, density) in a box of half extents ``half``."""
    out = []
    for _ in range(count):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        if flat:
            q = np.array([[q[0, 0], -q[1, 0], 0], [q[1, 0], q[0, 0], 0], [0, 0, 1.0]])
            q[:2, :2] /= np.linalg.norm(q[0, :2])
        a = rng.uniform(0.06, 0.5, 3) * half[0]
        c = rng.uniform(-0.6, 0.6, 3) * half
        if flat:
            c[2], a[2] = 0.0, 1e6
        out.append((c, q / a[:, None], rng.uniform(0.01, 0.05)))
    return out


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _phantom(blobs, shape, vw: float, seed: int, noise: float = 5e-4) -> torch.Tensor:
    """The ellipsoids on the voxel grid with a reconstruction's noise (float32, C order)."""
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) * vw - (n - 1) / 2 * vw for n in shape]
    out = torch.randn(shape, device="cuda", generator=_gen(seed)) * noise
    for c, m, rho in blobs:
        s = 0
        for r in range(3):
            s = s + (sum(float(m[r, a]) * (ax[a] - float(c[a])).reshape([-1 if b == a else 1 for b in range(3)]) for a in range(3))) ** 2
        out += rho * (s <= 1)
    return out


def _directions(g: dict, a: int, b: int, dtype) -> tuple[torch.Tensor, torch.Tensor]:
    """Sources (m, 1, 1, 3) and pixel centres (m, nu, nv, 3) of views a..b."""
    t = lambda k: torch.tensor(g[k][a:b], device="cuda", dtype=dtype)[:, None, None, :]  # noqa: E731
    iu = (torch.arange(g["nu"], device="cuda", dtype=dtype) - (g["nu"] - 1) / 2)[None, :, None, None]
    iv = (torch.arange(g["nv"], device="cuda", dtype=dtype) - (g["nv"] - 1) / 2)[None, None, :, None]
    return t("src"), t("det") + t("u") * iu + t("v") * iv


def _measured(blobs, g: dict, seed: int) -> torch.Tensor:
    """-log of photon counts through the ellipsoids (float32, (views, nu, nv))."""
    m = len(g["src"])
    out = torch.empty((m, g["nu"], g["nv"]), device="cuda")
    per = max(1, 4_000_000 // (g["nu"] * g["nv"]))
    for a in range(0, m, per):
        s, p = _directions(g, a, min(m, a + per), torch.float32)
        acc = torch.zeros(p.shape[:-1], device="cuda")
        length = (p - s).norm(dim=-1)
        for c, q, rho in blobs:
            qt, ct = torch.tensor(q, device="cuda", dtype=torch.float32), torch.tensor(c, device="cuda", dtype=torch.float32)
            o, d = (s - ct) @ qt.T, (p - s) @ qt.T
            aa, bb = (d * d).sum(-1), (o * d).sum(-1)
            disc = (bb * bb - aa * ((o * o).sum(-1) - 1)).clamp_(min=0)
            acc += rho * 2 * disc.sqrt() / aa * length
        counts = torch.poisson(PHOTONS * torch.exp(-acc), generator=_gen(seed + 7919 * (a + 1))).clamp_(min=1)
        out[a : a + per] = -torch.log(counts / PHOTONS)
    return out


def _inputs(case: dict, seed: int) -> dict:
    """Geometry arrays, object and measurement of a case: plain numpy and torch, made from the seed alone."""
    rng = np.random.default_rng([seed, 17])
    op, theta0 = case["op"], float(rng.uniform(0, 2 * np.pi))
    if op in ("project", "gradient", "backproject"):
        shape = (case["nx"], case["ny"], case["nz"])
        pix = _pix(VOX * max(shape[:2]), case["nu"], case["nv"], VOX * shape[2])
        g = _scan(case["views"], case["nu"], case["nv"], pix, theta0, helical=case["helical"], rng=rng if case["tilt"] else None)
        blobs = _blobs(rng, 12, VOX * np.array(shape) / 2)
        return dict(g=g, shape=shape, blobs=blobs, rng=rng)
    if op == "sirt":
        shape = (case["n"], case["n"], case["nz"])
        pix = _pix(VOX * case["n"], case["nu"], case["nv"], VOX * case["nz"])
        return dict(g=_scan(case["views"], case["nu"], case["nv"], pix, theta0), shape=shape,
                    blobs=_blobs(rng, 15, VOX * np.array(shape) / 2), rng=rng)
    if op == "sirt_batch":
        lay = np.random.default_rng(case["layout"])
        scans = []
        for _ in range(case["scans"]):
            n = int(round(math.exp(lay.uniform(math.log(case["edge_lo"]), math.log(case["edge_hi"])))))
            views, d = int(lay.integers(case["views_lo"], case["views_hi"] + 1)), int(lay.integers(case["det_lo"], case["det_hi"] + 1))
            pitch = float(lay.uniform(0.5, 1.5)) if lay.random() < 0.5 else 0.0
            g = _scan(views, d, d, 1.5 * n * VOX / d, float(rng.uniform(0, 2 * np.pi)), helical=pitch, rng=rng)
            scans.append(dict(g=g, shape=(n, n, n), blobs=_blobs(rng, 8, VOX * np.array([n, n, n]) / 2)))
        return dict(scans=scans)
    if op == "fan_fbp":
        n = case["n"]
        pix = _pix(VOX * n * 0.9, case["nu"])
        g = _scan(case["views"], case["nu"], 1, pix, theta0)
        half = VOX * np.array([n, n, 1]) / 2 * np.array([0.7, 0.7, 0])
        return dict(g=g, n=n, blobs=[_blobs(rng, 6, half, flat=True) for _ in range(case["slices"])])
    if op in ("cone_fbp", "gbc"):
        shape = (case["n"], case["n"], case["nz"])
        vw = VOX if op == "cone_fbp" else 1.0
        pix = _pix(vw * case["n"] * (1.0 if op == "cone_fbp" else 0.65), case["nu"])
        height = case["turn"] * 2 * vw * case["nz"] if op == "cone_fbp" else 0.65 * vw * case["nz"]
        g = _cylinder(case["views"], case["nu"], case["nv"], pix, height, theta0)
        return dict(g=g, shape=shape, vw=vw, blobs=_blobs(rng, 12, 0.6 * vw * np.array(shape) / 2), rot=int(rng.integers(1 << 30)))
    if op == "gbc_weights":
        return dict(pitch=float(rng.uniform(0.9, 1.1)), off=float(rng.uniform(0, 0.5)), nu=int(rng.integers(180, 257)))
    L = 1200.0 / 1000.0  # noqa: N806  (a larger phantom: the scan scaled)
    g = _scan(case["views"], case["nu"], case["nv"], 0.175 * 1024 / max(case["nu"], case["nv"]) * 1.0123 * L, theta0)
    return dict(g=g, shapes=int(rng.integers(1 << 30)))


def _f32(x: float) -> float:
    return float(np.float32(x))


def _gbc_windows(g: dict) -> tuple[float, float]:
    pw, L = float(np.linalg.norm(g["u"][0])), R + LMR  # noqa: N806
    nu, nv = g["nu"], g["nv"]
    return (float(np.arctan2(nv * pw / 2 - pw / 2, np.sqrt(L**2 + (nu * pw / 2 - pw / 2) ** 2))),
            float(np.arctan2(nu * pw / 2 - pw / 2, L)))


# ------------------------------------------------------------------ the calls
def _geom(g: dict):
    from aprict_b200.cb import flatpanel as fp

    return fp.ProjGeom(source_pos=g["src"], det_pos=g["det"], det_uvec=g["u"], det_vvec=g["v"], nu=g["nu"], nv=g["nv"])


def _bp_config(case: dict, shape) -> dict:
    cfg = dict(cyl_mask_rad=min(shape[:2]) / 2 * VOX if case["mask"] else None, apply_summand_multiplier=case["mult"],
               soften_det_edges_proportion=case["taper"])
    if case["mode"] != "exact":
        cfg["fast_approx"] = True
    if case["mode"] == "bilinear":
        cfg["approx_mode_bilinear_interpolate"] = True
    if case["mode"] == "raycast":
        cfg.update(approx_mode_direct_raycast=True, Z_on_val_factor_power=-2, Z_on_val_factor_val=R)
    return cfg


def _multiplier(shape, seed: int) -> torch.Tensor:
    return 0.5 + torch.rand(shape, device="cuda", generator=_gen(seed + 3))


def prepare(case: dict, seed: int) -> dict:
    """What a program holds before the call: device inputs, geometry and the iterator or config it keeps."""
    from aprict_b200 import FBVolume, Volume, autograd, iterators, phantoms
    from aprict_b200.cb import flatpanel as fp

    op, i = case["op"], _inputs(case, seed)
    if op == "project":
        x = _phantom(i["blobs"], i["shape"], VOX, seed)
        ps = fp.ProjectionSet(_geom(i["g"]), data=None)
        ps.create_buffer()
        return dict(op=op, cfg=fp.ConfigProject(ssu=case["ss"], ssv=case["ss"]), ps=ps,
                    vol=Volume(x.half() if case["half"] else x, voxwid=VOX, order=case["order"]))
    if op == "gradient":
        pr = autograd.SiddonProjector(_geom(i["g"]), i["shape"], voxwid=VOX)
        return dict(op=op, pr=pr, x=_phantom(i["blobs"], i["shape"], VOX, seed).requires_grad_(True),
                    b=_measured(i["blobs"], i["g"], seed))
    if op == "backproject":
        ps = fp.ProjectionSet(_geom(i["g"]), data=_measured(i["blobs"], i["g"], seed))
        m = Volume(_multiplier(i["shape"], seed), voxwid=VOX, order=case["order"]) if case["mult"] else None
        return dict(op=op, cfg=fp.ConfigBackproject(**_bp_config(case, i["shape"])), ps=ps, mult=m,
                    vol=Volume.zeros(i["shape"], voxwid=VOX, order=case["order"]))
    if op in ("sirt", "sirt_batch"):
        its = []
        for k, s in enumerate([i] if op == "sirt" else i["scans"]):
            x = _phantom(s["blobs"], s["shape"], VOX, seed + k)
            ps = fp.ProjectionSet(_geom(s["g"]), data=_measured(s["blobs"], s["g"], seed + k))
            its.append(iterators.SIRT_flatpanel(iterators.SIRT_flatpanel.Config(), Volume(x * 0.9, voxwid=VOX), ps))
        return dict(op=op, it=its[0] if op == "sirt" else iterators.SIRTBatch(its))
    if op == "fan_fbp":
        pg, n = _geom(i["g"]), i["n"]
        projs = [fp.ProjectionSet(pg, data=_measured(b, i["g"], seed + 31 * k)) for k, b in enumerate(i["blobs"])]
        return dict(op=op, projs=projs, vols=[Volume.zeros((n, n, 1), voxwid=VOX) for _ in projs],
                    stacked=torch.cat([p.data for p in projs]), hann=case["hann"])
    if op == "cone_fbp":
        ps = fp.ProjectionSet(_geom(i["g"]), data=_measured(i["blobs"], i["g"], seed))
        return dict(op=op, ps=ps, vol=Volume.zeros(i["shape"], voxwid=VOX), rot=i["rot"], interpolate=case["interpolate"],
                    views=case["views"])
    if op == "gbc":
        ps = fp.ProjectionSet(_geom(i["g"]), data=_measured(i["blobs"], i["g"], seed))
        tv, th = _gbc_windows(i["g"])
        cfg = fp.ConfigBackproject(fast_approx=True, Z_on_val_factor_val=R, backproj_weighting_preset=7,
                                   approx_mode_direct_raycast=True, approx_mode_bilinear_interpolate=case["interpolate"],
                                   soft_vartheta_v=tv, soft_vartheta_v_softspan=0.05, soft_vartheta_h=th, soft_vartheta_h_softspan=0.05)
        return dict(op=op, cfg=cfg, ps=ps, vol=Volume.zeros(i["shape"], voxwid=1.0), ws=Volume.zeros(i["shape"], voxwid=1.0))
    if op == "gbc_weights":
        tv, th = _weights_windows(i)
        cfg = fp.ConfigBackproject(fast_approx=True, Z_on_val_factor_val=R, backproj_weighting_preset=7,
                                   approx_mode_direct_raycast=True, soft_vartheta_v=tv, soft_vartheta_v_softspan=0.05,
                                   soft_vartheta_h=th, soft_vartheta_h_softspan=0.05)
        return dict(op=op, cfg=cfg, xs=_weights_axis(case, i), z=case["z_samps"], ang=case["ang_samps"])
    shapes = phantoms.random_quadric_phantom(i["shapes"], n_ellipsoids=case["ellipsoids"], n_cylinders=case["cylinders"])
    ps = fp.ProjectionSet(_geom(i["g"]), data=None)
    ps.create_buffer()
    return dict(op=op, vol=FBVolume(shapes), ps=ps, cfg=fp.ConfigProject(overlap_addition=case["additive"]))


def run(s: dict):
    """One pass."""
    from aprict_b200 import recon
    from aprict_b200.cb import flatpanel as fp
    from aprict_b200.gbc import weightinteg

    op = s["op"]
    if op in ("project", "quadric"):
        s["ps"].data.zero_()
        fp.project(s["cfg"], s["vol"], s["ps"])
        return s["ps"].data
    if op == "gradient":
        y = s["pr"](s["x"])
        loss = 0.5 * (y - s["b"]).square().sum()
        (grad,) = torch.autograd.grad(loss, s["x"])
        return y.detach(), grad
    if op == "backproject":
        s["vol"].fill(0)
        fp.backproject(s["cfg"], s["vol"], s["ps"], summand_multiplier=s["mult"])
        return s["vol"].data
    if op == "sirt":
        s["it"].iterate()
        return s["it"].volume.data
    if op == "sirt_batch":
        s["it"].iterate()
        return [x.volume.data for x in s["it"].sirts]
    if op == "fan_fbp":
        for v in s["vols"]:
            v.fill(0)
        recon.fbp_fan_circ_batch(s["projs"], s["vols"], apodization="hann" if s["hann"] else None, stacked=s["stacked"])
        return [v.data for v in s["vols"]]
    if op == "cone_fbp":
        s["vol"].fill(0)
        recon.fbp_cone_cyl(s["ps"], s["vol"], seed_proj_rots=s["rot"], interpolate=s["interpolate"], num_projs_per_chunk=s["views"])
        return s["vol"].data
    if op == "gbc":
        s["vol"].fill(0)
        s["ws"].fill(0)
        fp.backproject(s["cfg"], s["vol"], s["ps"], secondary_volume=s["ws"])
        return s["vol"].data, s["ws"].data
    return weightinteg.backproj_gbc_weight_integ_xygrid_GPU(s["xs"], s["xs"], R, s["cfg"], s["z"], s["ang"])


def _weights_windows(i: dict) -> tuple[float, float]:
    pw = 1.5 * i["pitch"]
    return _gbc_windows(dict(u=np.array([[pw, 0, 0]]), nu=i["nu"], nv=i["nu"]))


def _weights_axis(case: dict, i: dict) -> np.ndarray:
    return (np.arange(case["n"], dtype=np.float32) - (case["n"] - 1) / 2 + np.float32(i["off"])).astype(np.float32)


# ------------------------------------------------- what a pass cannot do without
def work(case: dict) -> dict:
    """Bytes in and out once, and the arithmetic of one multiply-add per ray segment, voxel-view or ray-shape pair (plus
    the coordinate it is taken at)."""
    op = case["op"]
    if op in ("project", "gradient"):
        vox, rays = case["nx"] * case["ny"] * case["nz"], case["views"] * case["nu"] * case["nv"]
        segs = rays * case.get("ss", 1) ** 2 * 0.6 * (case["nx"] + case["ny"] + 0.2 * case["nz"]) / 2
        both = 2 if op == "gradient" else 1
        return dict(bytes=both * 4 * (vox * (0.5 if case.get("half") else 1) + rays), flops=both * 6 * segs)
    if op == "backproject":
        vox, rays = case["nx"] * case["ny"] * case["nz"], case["views"] * case["nu"] * case["nv"]
        return dict(bytes=4 * (vox * (2 if case["mult"] else 1) + rays),
                    flops=vox * case["views"] * dict(exact=60, nearest=10, bilinear=16, raycast=12)[case["mode"]])
    if op == "sirt":
        vox, rays = case["n"] ** 2 * case["nz"], case["views"] * case["nu"] * case["nv"]
        return dict(bytes=4 * (3 * vox + rays), flops=vox * case["views"] * 10 + rays * 0.7 * case["n"] * 6)
    if op == "sirt_batch":
        b = f = 0
        lay = np.random.default_rng(case["layout"])
        for _ in range(case["scans"]):
            n = int(round(math.exp(lay.uniform(math.log(case["edge_lo"]), math.log(case["edge_hi"])))))
            views, d = int(lay.integers(case["views_lo"], case["views_hi"] + 1)), int(lay.integers(case["det_lo"], case["det_hi"] + 1))
            if lay.random() < 0.5:
                lay.uniform(0.5, 1.5)
            b += 4 * (3 * n**3 + views * d * d)
            f += n**3 * views * 10 + views * d * d * 0.5 * n * 6
        return dict(bytes=b, flops=f)
    if op == "fan_fbp":
        s, n, m, nu = case["slices"], case["n"], case["views"], case["nu"]
        return dict(bytes=4 * s * (n * n + m * nu), flops=n * n * m * (10 + 2 * s) + s * m * nu * 40)
    if op == "cone_fbp":
        vox, rays = case["n"] ** 2 * case["nz"], case["views"] * case["nu"] * case["nv"]
        return dict(bytes=4 * (vox + rays), flops=vox * case["views"] * 12 + rays * 60)
    if op == "gbc":
        vox, rays = case["n"] ** 2 * case["nz"], case["views"] * case["nu"] * case["nv"]
        return dict(bytes=4 * (2 * vox + rays), flops=vox * case["views"] * (30 if case["interpolate"] else 24))
    if op == "gbc_weights":
        return dict(bytes=4 * (case["n"] ** 2), flops=2 * case["n"] * case["z_samps"] * case["ang_samps"] * 8)
    rays = case["views"] * case["nu"] * case["nv"]
    return dict(bytes=4 * rays, flops=rays * 0.15 * (case["ellipsoids"] + case["cylinders"]) * 40)


def tolerance(case: dict) -> dict:
    """32-bit sums of some hundred terms, about four times the distance seen from ``exact``. The exact mode takes its chords
    from 32-bit slab crossings: few rays through each voxel (pixels coarser than voxels, few views) leave their errors unaveraged."""
    op = case["op"]
    nearest = op in ("sirt", "fan_fbp") or case.get("mode") in ("nearest", "raycast") or case.get("interpolate") is False
    if nearest and case.get("nx", case.get("n", 0)) % 2 and case.get("ny", case.get("n", 0)) % 2 and case["nu"] % 2 == 0:
        # the axis of an odd grid lies on the edge between two detector columns in every view: either is its nearest one
        return dict(rel=6e-4, max=0.5)
    if op == "project":
        return dict(rel=2e-6, max=4e-3)
    if op == "quadric":
        return dict(rel=1e-6, max=2e-2)
    if op == "gradient":
        return dict(rel=1.2e-5, max=4e-3)
    if op == "backproject" and case["mode"] == "exact":
        coarse = max(1.0, _pix(VOX * max(case["nx"], case["ny"]), case["nu"], case["nv"], VOX * case["nz"]) / VOX)
        rel = min(3e-3, 4e-5 * coarse**2 * max(1.0, math.sqrt(180 / case["views"])))
        return dict(rel=rel, max=min(0.9, 250 * rel))
    if op in ("backproject", "sirt", "sirt_batch"):
        return dict(rel=4e-6, max=1e-2)
    if op in ("fan_fbp", "cone_fbp"):
        return dict(rel=2e-5, max=2e-2)
    if op == "gbc":
        return dict(rel=1.2e-5, max=1e-2)
    return dict(rel=4e-6, max=1e-3)


# ------------------------------------------------------ the same in 64 bits
def _march(o, d, shape, visit) -> None:
    """Calls visit(rays, flat voxel index, parameter length) along the segments o + t d, t in [0, 1], of the unit grid ``shape``."""
    inf = float("inf")
    n = [float(k) for k in shape]
    a_in, a_out = torch.zeros_like(o[:, 0]), torch.ones_like(o[:, 0])
    for a in range(3):
        inside = (o[:, a] > 0) & (o[:, a] <= n[a])
        par = d[:, a] == 0
        t0, t1 = -o[:, a] / d[:, a], (n[a] - o[:, a]) / d[:, a]
        lo = torch.where(par, torch.where(inside, -inf, inf), torch.minimum(t0, t1))
        hi = torch.where(par, torch.where(inside, inf, -inf), torch.maximum(t0, t1))
        a_in, a_out = torch.maximum(a_in, lo), torch.minimum(a_out, hi)
    ids = torch.nonzero(a_in < a_out)[:, 0]
    o, d, a_in, a_out = o[ids], d[ids], a_in[ids], a_out[ids]
    if not len(ids):
        return
    st = [shape[1] * shape[2], shape[2], 1]
    flat = torch.zeros(len(ids), dtype=torch.int64, device=o.device)
    nxt, inc, move = [], [], []
    for a in range(3):
        p = o[:, a] + a_in * d[:, a]
        fwd = d[:, a] > 0
        k = torch.where(fwd, p.floor(), p.ceil() - 1).clamp_(0, n[a] - 1)
        par = d[:, a] == 0
        flat += k.long() * st[a]
        nxt.append(torch.where(par, inf, (k + fwd.double() - o[:, a]) / d[:, a]))
        inc.append(torch.where(par, inf, 1 / d[:, a].abs()))
        move.append(torch.where(fwd, st[a], -st[a]))
    first = [x.clone() for x in nxt]
    cnt = [torch.zeros_like(a_in) for _ in range(3)]
    t, last = a_in, shape[0] * shape[1] * shape[2] - 1
    for step in range(sum(shape) + 3):
        cut = torch.minimum(torch.minimum(nxt[0], nxt[1]), torch.minimum(nxt[2], a_out))
        visit(ids, flat.clamp(0, last), cut - t)
        if step % 32 == 31 and not bool((cut < a_out).any()):
            break
        for a in range(3):
            hit = nxt[a] <= cut
            cnt[a] += hit
            flat += move[a] * hit
            nxt[a] = torch.where(hit, first[a] + cnt[a] * inc[a], nxt[a])
        t = cut


def _rays(g: dict, shape, vw: float, ss: int, per: int = 6_000_000):
    """(first view, past the last, sub-ray weight, o, d, world lengths) of chunks of views in voxel units."""
    corner = np.float64(-np.float32(vw) * np.array(shape, np.float32) / 2)
    c = torch.tensor(corner, device="cuda")
    m = len(g["src"])
    k = max(1, per // (g["nu"] * g["nv"]))
    for a in range(0, m, k):
        b = min(m, a + k)
        s, p = _directions(g, a, b, torch.float64)
        u, v = (torch.tensor(g[w][a:b], device="cuda", dtype=torch.float64)[:, None, None, :] for w in "uv")
        for i in range(ss):
            for j in range(ss):
                q = p + u * ((i + 0.5) / ss - 0.5) + v * ((j + 0.5) / ss - 0.5)
                o = ((s - c) / _f32(vw)).expand(q.shape).reshape(-1, 3)
                d = ((q - s) / _f32(vw)).reshape(-1, 3)
                yield a, b, 1.0 / ss**2, o, d, (q - s).norm(dim=-1).reshape(-1)


def _project64(x, g: dict, vw: float, ss: int = 1):
    out = torch.zeros((len(g["src"]), g["nu"], g["nv"]), dtype=torch.float64, device="cuda")
    flatx = x.double().contiguous().reshape(-1)
    for a, b, w, o, d, length in _rays(g, x.shape, vw, ss):
        acc = torch.zeros(len(o), dtype=torch.float64, device="cuda")
        part = {}

        def visit(ids, flat, seg):
            if "s" not in part:
                part["ids"], part["s"] = ids, torch.zeros_like(seg)
            part["s"].addcmul_(seg, flatx[flat])

        _march(o, d, x.shape, visit)
        if part:
            acc[part["ids"]] = part["s"]
        out[a:b] += (acc * length * w).reshape(out[a:b].shape)
    return out


def _adjoint64(y, g: dict, shape, vw: float):
    out = torch.zeros(shape[0] * shape[1] * shape[2], dtype=torch.float64, device="cuda")
    for a, b, w, o, d, length in _rays(g, shape, vw, 1):
        val = y[a:b].double().reshape(-1) * length * w
        _march(o, d, shape, lambda ids, flat, seg: out.index_add_(0, flat, seg * val[ids]))  # noqa: B023
    return out.reshape(shape)


def _taper64(c, n: int, sep: float):
    r = (1 - c.abs() * 2 / n) / sep
    return ((1 + torch.cos(np.pi * (1 - r.clamp(0, 1)))) / 2).clamp(0, 1)


def _backproject64(y, g: dict, shape, vw: float, *, bilinear=False, raycast=False, power=0, mask=None, sep=0.0):
    """Fast backprojection: nearest or bilinear samples times voxwid^3 Dn^2 / (|u||v| D^2), or (Z/R)^power in raycast mode."""
    vw = _f32(vw)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) * vw for n in shape]
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    nu, nv = g["nu"], g["nv"]

    def form(c, k):
        return (c[0] * ax[0])[:, None, None] + (c[1] * ax[1])[None, :, None] + (c[2] * ax[2] + k)[None, None, :]

    for m in range(len(g["src"])):
        s, p, u, v = (g[k][m].astype(np.float64) for k in ("src", "det", "u", "v"))
        nrm = np.cross(u, v)
        dn = (p - s) @ nrm
        den = form(nrm, -(s @ nrm))
        co = []
        for w, n in ((u, nu), (v, nv)):
            cw = (dn * w - (w @ (p - s)) * nrm) / (w @ w) + nrm * (n - 1) / 2
            co.append(form(cw, -(s @ cw)) / den)
        fu, fv = co
        data = y[m].double()

        def at(i, j):
            ok = (i >= 0) & (i < nu) & (j >= 0) & (j < nv)  # noqa: B023
            return torch.where(ok, data.reshape(-1)[(i.clamp(0, nu - 1) * nv + j.clamp(0, nv - 1))], 0.0)  # noqa: B023

        if bilinear:
            i, j = fu.floor().clamp(-2, nu + 1), fv.floor().clamp(-2, nv + 1)
            fx, fy = fu - i, fv - j
            i, j = i.long(), j.long()
            val = (at(i, j) * (1 - fx) + at(i + 1, j) * fx) * (1 - fy) + (at(i, j + 1) * (1 - fx) + at(i + 1, j + 1) * fx) * fy
        else:
            val = at((fu + 0.5).floor().clamp(-2, nu + 1).long(), (fv + 0.5).floor().clamp(-2, nv + 1).long())
        if sep > 0:
            val = val * _taper64(fu - (nu - 1) / 2, nu, sep) * _taper64(fv - (nv - 1) / 2, nv, sep)
        if raycast:
            lh = (p - s) / np.linalg.norm(p - s)
            val = val * (form(lh, -(s @ lh)) / R) ** power if power else val
        else:
            val = val * (vw**3 * dn * dn / (np.linalg.norm(u) * np.linalg.norm(v))) / den**2
        out += val
    if mask:
        out *= ((ax[0][:, None] ** 2 + ax[1][None, :] ** 2) <= _f32(mask) ** 2)[:, :, None]
    return out


def _adjoint_tapered64(y, g, shape, vw, sep, mask):
    """The exact mode: A^T with the taper taken at the voxel centre's coordinate."""
    if sep == 0:
        out = _adjoint64(y, g, shape, vw)
    else:
        one = dict(g)
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for m in range(len(g["src"])):
            for k in ("src", "det", "u", "v"):
                one[k] = g[k][m : m + 1]
            ones = torch.ones((1, g["nu"], g["nv"]), device="cuda")
            out += _adjoint64(y[m : m + 1], one, shape, vw) * _taper_at_centres(ones, one, shape, vw, sep)
    if mask:
        ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) * _f32(vw) for n in shape[:2]]
        out *= ((ax[0][:, None] ** 2 + ax[1][None, :] ** 2) <= _f32(mask) ** 2)[:, :, None]
    return out


def _taper_at_centres(ones, g, shape, vw, sep):
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) * _f32(vw) for n in shape]
    s, p, u, v = (g[k][0].astype(np.float64) for k in ("src", "det", "u", "v"))
    nrm = np.cross(u, v)
    dn = (p - s) @ nrm
    form = lambda c: (c[0] * ax[0])[:, None, None] + (c[1] * ax[1])[None, :, None] + (c[2] * ax[2] - s @ c)[None, None, :]  # noqa: E731
    den = form(nrm)
    t = 1.0
    for w, n in ((u, g["nu"]), (v, g["nv"])):
        t = t * _taper64(form((dn * w - (w @ (p - s)) * nrm) / (w @ w)) / den, n, sep)
    return t


def _softmask64(shape, r0: float):
    i, j = (torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2 for n in shape[:2])
    r = (i[:, None] ** 2 + j[None, :] ** 2).sqrt() * 2 / min(shape[:2])
    m = torch.zeros_like(r) if r0 >= 1 else (1 + torch.cos(np.pi * ((r - r0) / (1 - r0)).clamp(max=1))) / 2
    return torch.where(r < r0, 1.0, m.clamp(0, 1))[:, :, None]


def _sirt64(s: dict, seed: int):
    g, shape = s["g"], s["shape"]
    x = (_phantom(s["blobs"], shape, VOX, seed) * 0.9).double()
    b = _measured(s["blobs"], g, seed).double()
    rad, sep = min(shape[:2]) / 2 * VOX, _f32(1 - 0.95)
    scale = 1 / float(np.mean(shape))
    p = _project64(torch.full(shape, _f32(scale), dtype=torch.float64, device="cuda") * _softmask64(shape, 1.0), g, VOX)
    mean = float(p.mean())
    p /= mean / scale
    scale /= mean / scale
    m = _backproject64(p, g, shape, VOX, mask=rad, sep=sep)
    m = torch.where(m == 0, 0.0, 1 / (m + 0.1 * torch.exp(-m / 0.1))) * scale * _softmask64(shape, _f32(0.95))
    return x + m * _backproject64(b - _project64(x, g, VOX), g, shape, VOX, mask=rad, sep=sep)


def _ramlak64(n: int, pitch: float, hann: bool) -> np.ndarray:
    k = np.arange(-(n - 1), n, dtype=np.float64)
    odd = np.abs(k) % 2 == 1
    h = np.where(odd, -4 / np.where(odd, k, 1) ** 2, 0.0)
    h[n - 1] = np.pi**2
    h /= pitch
    return np.convolve(h, [0.25, 0.5, 0.25], mode="same") if hann else h


def _convolve64(rows: torch.Tensor, taps: np.ndarray) -> torch.Tensor:
    """Linear convolution along axis 1 of (m, nu, k) with 2 nu - 1 taps."""
    nu = rows.shape[1]
    size = 1 << (3 * nu).bit_length()
    h = torch.fft.rfft(torch.tensor(taps, device="cuda"), n=size)
    return torch.fft.irfft(torch.fft.rfft(rows.double(), n=size, dim=1) * h[None, :, None], n=size, dim=1)[:, nu - 1 : 2 * nu - 1]


def _fan64(case: dict, i: dict, seed: int):
    g, n, m, nu = i["g"], i["n"], case["views"], case["nu"]
    pw = float(np.linalg.norm(g["u"][0].astype(np.float64)))
    Ld = R + LMR  # noqa: N806
    taps = _ramlak64(nu, pw / Ld, case["hann"])
    uu = torch.tensor(pw / Ld * (np.arange(nu) - (nu - 1) / 2), device="cuda")
    wts = (1 / (1 + uu**2).sqrt())[None, :, None]
    y = torch.cat([_measured(b, g, seed + 31 * k) for k, b in enumerate(i["blobs"])], dim=2)  # (m, nu, slices)
    f = torch.cat([_convolve64(y[a : a + 60].double() * wts, taps) for a in range(0, m, 60)]) / (4 * np.pi * R * m)
    support = R * np.sin(np.arctan(pw * nu / 2 / Ld))
    ax = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) * VOX
    out = torch.zeros((n * n, y.shape[2]), dtype=torch.float64, device="cuda")
    for k in range(m):
        s, p, u = (g[w][k].astype(np.float64) for w in ("src", "det", "u"))
        nrm = np.cross(u, g["v"][k].astype(np.float64))
        dn = (p - s) @ nrm
        form = lambda c: (c[0] * (ax[:, None] - s[0]) + c[1] * (ax[None, :] - s[1])).reshape(-1)  # noqa: B023, E731
        den = form(nrm)
        j = (form((dn * u - (u @ (p - s)) * nrm) / (u @ u)) / den + (nu - 1) / 2 + 0.5).floor().clamp(-1, nu).long()
        lh = (p - s) / np.linalg.norm(p - s)
        w = torch.where((j >= 0) & (j < nu), (form(lh) / R) ** -2, 0.0)
        out += f[k][j.clamp(0, nu - 1)] * w[:, None]
    out *= ((ax[:, None] ** 2 + ax[None, :] ** 2) <= _f32(support) ** 2).reshape(-1, 1)
    return [out[:, k].reshape(n, n, 1) for k in range(y.shape[2])]


def _rotate64(img, c, s, out_shape, centre, in_off=(0, 0), out_off=(0, 0)):
    """Order-1 resampling of (m, nu, nv) images rotated about ``centre`` (zero outside); c, s per image."""
    nu, nv = img.shape[1:]
    i = (torch.arange(out_shape[0], device="cuda", dtype=torch.float64) + out_off[0] - centre[0])[None, :, None]
    j = (torch.arange(out_shape[1], device="cuda", dtype=torch.float64) + out_off[1] - centre[1])[None, None, :]
    qu = c * i + s * j + centre[0] - in_off[0]
    qv = -s * i + c * j + centre[1] - in_off[1]
    iu, iv = qu.floor(), qv.floor()
    tu, tv = qu - iu, qv - iv
    iu, iv = iu.long(), iv.long()
    flat = img.double().reshape(img.shape[0], -1)

    def at(a, b):
        ok = (a >= 0) & (a < nu) & (b >= 0) & (b < nv)
        idx = (a.clamp(0, nu - 1) * nv + b.clamp(0, nv - 1)).reshape(img.shape[0], -1)
        return torch.where(ok, flat.gather(1, idx).reshape(ok.shape), 0.0)

    return (1 - tu) * ((1 - tv) * at(iu, iv) + tv * at(iu, iv + 1)) + tu * ((1 - tv) * at(iu + 1, iv) + tv * at(iu + 1, iv + 1))


def _cone64(case: dict, i: dict, seed: int):
    g, shape, m = i["g"], i["shape"], case["views"]
    nu, nv, Ld = g["nu"], g["nv"], R + LMR  # noqa: N806
    pw = float(np.linalg.norm(g["u"][0]))
    zeta = float(np.arctan2(nv * pw / 2, np.sqrt(Ld**2 + (nu * pw / 2) ** 2)))
    we, he = int(np.ceil(nv * np.sin(zeta) + nu * np.cos(zeta))), nv
    we += (we - nu) % 2
    rng = np.random.default_rng(seed=i["rot"])
    ang = np.array([-zeta + 2 * zeta * rng.random() for _ in range(m)], dtype=np.float32)
    u = pw / Ld * (np.arange(we, dtype=np.float32) - (we - 1) / 2)
    v = pw / Ld * (np.arange(he, dtype=np.float32) - (he - 1) / 2)
    mask = 1 / (np.sqrt(1 + v[None, :] ** 2) ** 3 * np.sqrt(1 + v[None, :] ** 2 + u[:, None] ** 2))
    mask = torch.tensor(np.asarray(mask, np.float64), device="cuda")
    mid, col = (he - 1) / 2, np.ones((m, he))
    disc = Ld / pw * np.sqrt(np.maximum((np.cos(ang) / np.cos(zeta)) ** 2 - 1, 0))
    for k in range(m):
        lo, hi = mid - disc[k], mid + disc[k]
        a, b = round(lo), round(hi)
        col[k, :a], col[k, b + 1 :] = 0, 0
        if a == b:
            col[k, a] = hi - lo
        else:
            col[k, a], col[k, b] = a + 0.5 - lo, hi - (b - 0.5)
    col = torch.tensor(col, device="cuda")
    y = _measured(i["blobs"], g, seed)
    taps, pad, centre = _ramlak64(we, pw / Ld, False), ((we - nu) // 2, (he - nv) // 2), ((we - 1) / 2, (he - 1) / 2)
    out = torch.empty((m, nu, nv), dtype=torch.float64, device="cuda")
    for a in range(0, m, 16):
        sl = slice(a, min(m, a + 16))
        c, s = (torch.tensor(f(np.deg2rad(180 / np.pi * ang[sl]).astype(np.float64)), device="cuda")[:, None, None] for f in (np.cos, np.sin))
        e = _rotate64(y[sl], c, -s, (we, he), centre, in_off=pad) * mask * col[sl, None, :]
        out[sl] = _rotate64(_convolve64(e, taps), c, s, (nu, nv), centre, out_off=pad)
    z = g["src"][:, 2].astype(np.float64)
    out *= 2 * zeta / np.sin(zeta / 2) ** 2 * (z.max() - z.min()) / (16 * np.pi**2 * R**2 * m)
    rad = R * np.sin(np.arctan(pw * nu / 2 / Ld))
    return _backproject64(out, g, shape, VOX, bilinear=case["interpolate"], raycast=True, power=-3, mask=rad)


def _window64(s, a: float, b: float):
    """The GBC soft window of an angle given by its sine."""
    gamma = 1 / (np.sin(a - b) - np.sin(a))
    x = gamma * s - gamma * np.sin(a)
    w = (3 * x * x - 2 * x**3).clamp(0, 1)
    return torch.where(s > np.sin(a), 0.0, torch.where(s < np.sin(a - b), 1.0, w))


def _gbc64(case: dict, i: dict, seed: int):
    g, shape, vw = i["g"], i["shape"], i["vw"]
    y = _measured(i["blobs"], g, seed)
    tv, th = (_f32(t) for t in _gbc_windows(g))
    span = _f32(0.05)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - 0.5 * n) * vw for n in shape]
    vol, ws = (torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(2))
    one = dict(g)
    for m in range(case["views"]):
        s = g["src"][m].astype(np.float64)
        rx, ry, rz = (ax[0] - s[0])[:, None], (ax[1] - s[1])[None, :], (ax[2] - s[2])[None, None, :]
        q = (rx**2 + ry**2).sqrt()
        ell = q / R
        c = ((rx * s[0] + ry * s[1]).abs() / np.hypot(s[0], s[1]) / q).clamp(0, 1)
        hor = c / (c**2 + (c - ell) ** 2).clamp(min=1e-9) * _window64((1 - c**2).clamp(min=0).sqrt(), th, span)
        h = (ell[:, :, None] ** 2 + (rz / R) ** 2).sqrt()
        w = hor[:, :, None] * (ell[:, :, None] / h) ** 3 * _window64((rz / R).abs() / h, tv, span)
        ws += w
        for k in ("src", "det", "u", "v"):
            one[k] = g[k][m : m + 1]
        vol += w * _backproject64(y[m : m + 1], one, shape, vw, bilinear=case["interpolate"], raycast=True)
    return vol, ws


def _weights64(case: dict, i: dict):
    tv, th = (_f32(t) for t in _weights_windows(i))
    span = _f32(0.05)
    xs = _weights_axis(case, i)
    rel = np.sqrt(np.square(xs[:, None]) + np.square(xs[None, :])) / R
    grid = np.linspace(rel.min(), rel.max(), num=2 * case["n"])
    r32 = grid.astype(np.float32).astype(np.float64)
    nz, na = case["z_samps"], case["ang_samps"]
    zmax = np.tan(tv) * (1 + r32[-1])
    z = (torch.arange(nz, device="cuda", dtype=torch.float64) * (zmax / (nz - 1)))[None, :]
    half = torch.ones_like(z)
    half[0, 0] = 0.5
    t = torch.arange(na, device="cuda", dtype=torch.float64) / na * np.pi
    out = np.empty(len(r32))
    for k, r in enumerate(r32):
        rx, ry = r - torch.cos(t), -torch.sin(t)
        ell = (rx**2 + ry**2).sqrt()
        c = ((rx * torch.cos(t) + ry * torch.sin(t)).abs() / ell).nan_to_num(1.0).clamp(0, 1)
        a = c / (c**2 + (c - ell) ** 2).clamp(min=1e-9) * _window64((1 - c**2).clamp(min=0).sqrt(), th, span)
        tot = 0.0
        for b in range(0, na, 1500):
            e = ell[b : b + 1500, None]
            h = (e**2 + z**2).sqrt()
            tot += float((a[b : b + 1500, None] * (e / h) ** 3 * _window64(z / h, tv, span) * half).sum())
        out[k] = tot * 4 * zmax * np.pi / (nz * na)
    return np.interp(rel, grid, out)


def _quadric64(case: dict, i: dict):
    from aprict_b200 import phantoms  # the phantom's records: inputs, as in prepare

    g = i["g"]
    recs = phantoms.random_quadric_phantom(i["shapes"], n_ellipsoids=case["ellipsoids"], n_cylinders=case["cylinders"])
    out = torch.zeros((case["views"], g["nu"], g["nv"]), dtype=torch.float64, device="cuda")
    vec = lambda v: np.array([v["x"], v["y"], v["z"]], np.float64)  # noqa: E731
    unit = lambda v: v / np.linalg.norm(v)  # noqa: E731
    per = max(1, 4_000_000 // (g["nu"] * g["nv"]))
    for a in range(0, case["views"], per):
        b = min(case["views"], a + per)
        s, p = _directions(g, a, b, torch.float64)
        d = p - s
        acc = torch.zeros(d.shape[:-1], dtype=torch.float64, device="cuda")
        left = []  # intervals of the later shapes
        for rec in recs[::-1]:
            cyl = int(rec["type"]) == 12
            rows = [unit(vec(rec["a_x"])) / float(rec["dx"]), unit(vec(rec["a_y"])) / float(rec["dy"]),
                    unit(vec(rec["axis"])) if cyl else unit(vec(rec["a_z"])) / float(rec["dz"])]
            c = np.array([rec["x"], rec["y"], rec["z"]], np.float64)
            dot = lambda w, v: sum(float(v[k]) * w[..., k] for k in range(3))  # noqa: E731
            o = s - torch.tensor(c, device="cuda")
            oo, dd = [dot(o, r) for r in rows], [dot(d, r) for r in rows]
            k = 2 if cyl else 3
            qa, qb = sum(w * w for w in dd[:k]), sum(x * w for x, w in zip(oo[:k], dd[:k]))
            disc = qb * qb - qa * (sum(x * x for x in oo[:k]) - 1)
            root = disc.clamp(min=0).sqrt()
            lo, hi = ((-qb - root) / qa).clamp(min=0), ((-qb + root) / qa).clamp(max=1)
            hi = torch.where(disc > 0, hi, -1.0)
            if cyl:
                h = float(rec["l"]) / 2
                t0, t1 = (-h - oo[2]) / dd[2], (h - oo[2]) / dd[2]
                lo, hi = torch.maximum(lo, torch.minimum(t0, t1)), torch.minimum(hi, torch.maximum(t0, t1))
            for cas in ("cas1", "cas2", "cas3"):
                mode = int(rec[cas]["mode"])
                if mode:
                    sg = 1.0 if mode == 1 else -1.0
                    n = vec(rec[cas]["axis"]) * sg
                    f0, f1 = dot(s, n) - sg * float(rec[cas]["dotprod"]), dot(d, n)
                    t = -f0 / f1
                    hi = torch.where(f1 > 0, torch.minimum(hi, t), hi)
                    lo = torch.where(f1 < 0, torch.maximum(lo, t), lo)
            length = (hi - lo).clamp(min=0)
            if case["additive"]:
                acc += float(rec["rho"]) * length
            else:
                left.append((float(rec["rho"]), lo, torch.where(length > 0, hi, lo)))
        if not case["additive"]:
            # sweep the sorted interval ends; each piece belongs to the first interval of `left` that holds it
            ends = torch.stack([e for _, lo, hi in left for e in (lo, hi)]).sort(dim=0).values
            for k in range(len(ends) - 1):
                mid, piece = (ends[k] + ends[k + 1]) / 2, ends[k + 1] - ends[k]
                rho, free = torch.zeros_like(mid), torch.ones_like(mid, dtype=torch.bool)
                for value, lo, hi in left:
                    inside = free & (mid > lo) & (mid < hi)
                    rho = torch.where(inside, value, rho)
                    free &= ~inside
                acc += rho * piece
            acc *= d.norm(dim=-1)
        out[a:b] = acc
    return out


def exact(case: dict, seed: int):
    """``run``'s outputs in 64 bits; None where that would take too long."""
    i, op = _inputs(case, seed), case["op"]
    if op == "project":
        x = _phantom(i["blobs"], i["shape"], VOX, seed)
        return _project64(x.half() if case["half"] else x, i["g"], VOX, case["ss"])
    if op == "gradient":
        y = _project64(_phantom(i["blobs"], i["shape"], VOX, seed), i["g"], VOX)
        return y, _adjoint64(y - _measured(i["blobs"], i["g"], seed).double(), i["g"], i["shape"], VOX)
    if op == "backproject":
        y = _measured(i["blobs"], i["g"], seed)
        cfg = _bp_config(case, i["shape"])
        if case["mode"] == "exact":
            if case["taper"] and case["views"] * sum(i["shape"]) > 150_000:
                return None  # one march per view: too many launches
            out = _adjoint_tapered64(y, i["g"], i["shape"], VOX, _f32(case["taper"]), cfg["cyl_mask_rad"])
        else:
            out = _backproject64(y, i["g"], i["shape"], VOX, bilinear=case["mode"] == "bilinear", raycast=case["mode"] == "raycast",
                                 power=-2, mask=cfg["cyl_mask_rad"], sep=_f32(case["taper"]))
        return out * _multiplier(i["shape"], seed).double() if case["mult"] else out
    if op == "sirt":
        return _sirt64(i, seed)
    if op == "sirt_batch":
        return [_sirt64(s, seed + k) for k, s in enumerate(i["scans"])]
    if op == "fan_fbp":
        return _fan64(case, i, seed)
    if op == "cone_fbp":
        return _cone64(case, i, seed)
    if op == "gbc":
        return _gbc64(case, i, seed)
    if op == "gbc_weights":
        return _weights64(case, i)
    if not case["additive"] and case["views"] * case["nu"] * case["nv"] * (case["ellipsoids"] + case["cylinders"]) ** 2 > 3e10:
        return None  # the sweep over all interval ends
    return _quadric64(case, i)
