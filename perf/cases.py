"""The work that programs on this package have it do, as measurable cases.

Every case images, or prepares for imaging, a side-looking stripmap scene of the package's own scene
definitions (``bp_project_gb300.scenes.CONFIGS``): the near geometry of c0 / c1 / c3 (9.6 GHz, 180 MHz
sampling, 4 km slant range from 3 km altitude) or the far one of c2 (10 GHz, 360 MHz, 30 km).  The pulses
hold seeded point targets over Gaussian clutter and noise, the track has centimetre motion errors, the
pulse weights are an aperture taper and the pulse phases small corrections, as after motion
compensation.

Kinds and what they stand for:

* ``lattice``  direct BP onto a ground lattice (``core.backproject_lattice``), the package's main call:
  a quick-look chip where latency counts, the 4096-pulse / 2048^2 scene, ragged far-range sizes;
* ``polar``    direct BP onto a polar grid, the ``run_direct`` surface (split and the reference's mixed policy);
* ``points``   direct BP at the points of a terrain model in raster order (``core.backproject_points``);
* ``grad``     differentiable BP, forward and backward, as in one step of gradient autofocus;
* ``ffbp``     a kept FFBP program, then its polar image onto the ground lattice (a processing chain);
* ``form``     the whole ``ffbp.form_ffbp`` call, planning included (the reference's image-formation call);
* ``ground``   a polar image at terrain points (``core.evaluate_image``);
* ``compress`` range compression of raw echoes, without and with oversampling;
* ``pga``      one phase-gradient trajectory update of the reference's autofocus loop;
* ``batch``    many uneven scenes formed by one schedule (``batch.SceneBatch``).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bp_project_gb300 import autofocus, autograd, batch, core, ffbp, gpu_backend, sar_io
from bp_project_gb300.scenes import CONFIGS

DEV = "cuda"


def listed():
    return [
        # A quick-look chip around a detection: a call of tens of microseconds.
        dict(name="lattice_chip", kind="lattice", geometry="c0", pulses=192, samples=1536, rows=96, cols=128,
             spacing=0.5),
        # The benchmark scene: 4096 pulses onto 2048 x 2048.
        dict(name="lattice_c1", kind="lattice", geometry="c1", pulses=4096, samples=8192, rows=2048, cols=2048,
             spacing=0.5),
        # Far-range stripmap of odd sizes at the fine pixel spacing.
        dict(name="lattice_far_ragged", kind="lattice", geometry="c2", pulses=1777, samples=4999, rows=901, cols=1213,
             spacing=0.25),
        # run_direct: the 1024-pulse scene's polar sector, default precision, and the reference's mixed policy.
        dict(name="polar_c0", kind="polar", geometry="c0", pulses=1024, samples=2048, rows=512, cols=512, spacing=0.5,
             leaf=64, mode="split"),
        dict(name="polar_mixed", kind="polar", geometry="c0", pulses=256, samples=2048, rows=257, cols=257,
             spacing=0.5, leaf=64, mode="mixed"),
        # Orthorectified imaging: a terrain model's points in raster order.
        dict(name="points_terrain", kind="points", geometry="c3", pulses=1024, samples=4096, rows=384, cols=501,
             spacing=0.5),
        # One evaluation of gradient autofocus on the autofocus scene (image, then gradients).
        dict(name="grad_c3", kind="grad", geometry="c3", pulses=2048, samples=4096, rows=1024, cols=1024, spacing=0.5),
        # The 4096-pulse FFBP chain with its plan kept, onto the ground lattice.
        dict(name="ffbp_c1", kind="ffbp", geometry="c1", pulses=4096, samples=8192, rows=2048, cols=2048, spacing=0.5,
             leaf=16),
        # The whole image-formation call on the small scene.
        dict(name="form_c0", kind="form", geometry="c0", pulses=1024, samples=2048, rows=512, cols=512, spacing=0.5,
             leaf=64),
        # Raw echoes of the 4096-pulse scene to BP input.
        dict(name="compress_c1", kind="compress", pulses=4096, samples=8192, oversample=1),
        # One update of the reference's trajectory autofocus: 144 targets.
        dict(name="pga_c3", kind="pga", geometry="c3", pulses=2048, samples=4096, rows=1024, cols=1024, spacing=0.5,
             targets=144, cutoff=8.0),
        # A queue of small uneven scenes, half direct BP and half FFBP.
        dict(name="batch_small", kind="batch", geometry="c0", scenes=24, pulses=512, side=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice", "lattice", "lattice", "polar", "points", "grad", "ffbp", "ffbp", "form", "ground",
                       "compress", "pga", "batch"])
    if kind == "compress":
        return dict(kind=kind, pulses=_log_int(rng, 64, 4096), samples=_log_int(rng, 1000, 8192),
                    oversample=rng.choice([1, 1, 1, 2]))
    if kind == "batch":
        return dict(kind=kind, geometry="c0", scenes=rng.randint(8, 32), pulses=rng.choice([256, 512, 1024]),
                    side=rng.choice([128, 256, 512]))
    geometry = rng.choice(["c0", "c1", "c2", "c3"]) if kind in ("lattice", "points", "ground") else rng.choice(
        ["c0", "c1", "c3"])
    top_side = {"lattice": 2048, "polar": 700, "points": 600, "grad": 1200, "ffbp": 2048, "form": 700, "ground": 2048,
                "pga": 1024}[kind]
    top_pulses = {"lattice": 4096, "polar": 2048, "points": 2048, "grad": 2048, "ffbp": 4096, "form": 2048,
                  "ground": 1024, "pga": 2048}[kind]
    rows, cols = _log_int(rng, 64, top_side), _log_int(rng, 64, top_side)
    spacing = CONFIGS[geometry].pixel_spacing * rng.choice([0.5, 1.0, 1.0, 1.0, 1.25])
    case = dict(kind=kind, geometry=geometry, pulses=_log_int(rng, 128, top_pulses), samples=0, rows=rows, cols=cols,
                spacing=spacing)
    case["samples"] = _samples_for(case) + rng.randint(0, 511)
    if kind in ("ffbp", "form", "polar", "ground"):
        case["leaf"] = rng.choice([16, 16, 32, 64])
    if kind == "polar":
        case["mode"] = "split" if rng.random() < 0.8 else "mixed"
        if case["mode"] == "mixed":  # the FP64 policies are used on small sectors, to check against
            case.update(pulses=min(case["pulses"], 256), rows=min(rows, 257), cols=min(cols, 257))
    if kind == "pga":
        case.update(targets=rng.randint(16, 144), cutoff=rng.choice([12.0, 8.0, 5.0, 3.0]),
                    pulses=max(case["pulses"], 600))
    return case


# ---- geometry and inputs -----------------------------------------------------------------


def _samples_for(case):
    """Range bins that cover the scene from every pulse."""
    cfg = CONFIGS[case["geometry"]]
    far_x = cfg.near_ground + (case["rows"] + 2) * case["spacing"]
    y = 0.5 * case["cols"] * case["spacing"] + 0.5 * case["pulses"] * cfg.pulse_spacing
    far = math.sqrt(far_x**2 + y**2 + cfg.altitude**2)
    return int((far - cfg.range_start) / cfg.data_dr) + 160


def _track(cfg, pulses):
    """Antenna positions; the flown track is part of the case, so that plans keep their sizes."""
    rng = np.random.default_rng(pulses)
    t = (np.arange(pulses) - 0.5 * (pulses - 1)) / max(pulses, 2)
    pos = np.zeros((pulses, 3))
    pos[:, 1] = (np.arange(pulses) - 0.5 * (pulses - 1)) * cfg.pulse_spacing
    pos[:, 2] = cfg.altitude
    for c in range(3):  # smooth motion errors of a few centimetres
        pos[:, c] += rng.uniform(0.01, 0.04) * np.sin(2 * np.pi * rng.uniform(1.0, 4.0) * t + rng.uniform(0, 6.28))
    return pos


def _lattice(cfg, case):
    s = case["spacing"]
    origin = (cfg.near_ground + s, -0.5 * (case["cols"] - 1) * s, 0.0)
    return origin, (s, 0.0, 0.0), (0.0, s, 0.0)


def _extent(case, pos):
    """Polar sector about the mean track point that covers the ground lattice."""
    cfg = CONFIGS[case["geometry"]]
    origin, sr, sc = _lattice(cfg, case)
    o = pos.mean(axis=0)
    x = np.array([origin[0], origin[0] + (case["rows"] - 1) * sr[0]]) - o[0]
    y = np.array([origin[1], origin[1] + (case["cols"] - 1) * sc[1]]) - o[1]
    xx, yy = np.meshgrid(x, y)
    g = np.sqrt(xx**2 + yy**2)
    r = np.sqrt(g**2 + o[2] ** 2)
    rmin = math.sqrt(x.min() ** 2 + o[2] ** 2)
    u = yy / g
    return rmin - 2.0, float(r.max()) + 2.0, float(u.min()) - 1e-3, float(u.max()) + 1e-3


def _echoes(cfg, case, pos, rng, gen):
    """Range-compressed pulses: point targets with the exact two-way phase over clutter and noise."""
    p, s = case["pulses"], case["samples"]
    data = torch.complex(torch.randn(p, s, device=DEV, generator=gen), torch.randn(p, s, device=DEV, generator=gen))
    data *= 0.2
    origin, sr, sc = _lattice(cfg, case)
    n = 16
    tx = origin[0] + rng.uniform(0.05, 0.95, n) * case["rows"] * sr[0]
    ty = origin[1] + rng.uniform(0.05, 0.95, n) * case["cols"] * sc[1]
    amp = rng.uniform(1.0, 10.0, n) * np.exp(2j * np.pi * rng.uniform(size=n))
    pt = torch.from_numpy(pos).to(DEV)
    offs = torch.arange(-16, 17, device=DEV)
    row = torch.arange(p, device=DEV)[:, None].expand(p, offs.numel())
    for i in range(n):
        d = torch.sqrt((pt[:, 0] - tx[i]) ** 2 + (pt[:, 1] - ty[i]) ** 2 + pt[:, 2] ** 2)
        b = torch.floor((d - cfg.range_start) / cfg.data_dr).long()[:, None] + offs
        env = torch.sinc((cfg.range_start + b * cfg.data_dr - d[:, None]) / cfg.resolution)
        v = complex(amp[i]) * torch.polar(torch.ones_like(d), -cfg.k * d)[:, None] * env
        ok = (b >= 0) & (b < s)
        b = b.clamp(0, s - 1)
        # one target touches each (pulse, bin) once, so this read-add-write is exact and repeatable
        add = torch.where(ok, v, torch.zeros_like(v)).to(torch.complex64)
        old = data[row, b]
        keep = ok.reshape(-1)
        data[row.reshape(-1)[keep], b.reshape(-1)[keep]] = (old + add).reshape(-1)[keep]
    return data


def _scene(case, seed):
    cfg = CONFIGS[case["geometry"]]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    pos = _track(cfg, case["pulses"])
    p = case["pulses"]
    weight = 0.54 - 0.46 * np.cos(2 * np.pi * (np.arange(p) + 0.5) / p)
    phase = rng.normal(0.0, 0.2, p)
    st = dict(kind=case["kind"], cfg=cfg, host_pos=pos, data=_echoes(cfg, case, pos, rng, gen))
    for name, v in (("pos", pos), ("weight", weight), ("phase", phase)):
        st[name] = torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
    st["lattice"] = (*_lattice(cfg, case), case["rows"], case["cols"])
    st["radar"] = (cfg.range_start, cfg.data_dr, cfg.k)
    return st, rng, gen


def _terrain(case, st, rng):
    """The lattice's points on gentle hills, row by row."""
    origin, sr, sc, rows, cols = st["lattice"]
    x = origin[0] + sr[0] * torch.arange(rows, dtype=torch.float64, device=DEV)[:, None].expand(rows, cols)
    y = origin[1] + sc[1] * torch.arange(cols, dtype=torch.float64, device=DEV)[None, :].expand(rows, cols)
    a = rng.uniform(0, 6.28, 2)
    z = 6.0 * torch.sin(x / 90.0 + a[0]) + 4.0 * torch.cos(y / 70.0 + a[1])
    return torch.stack([x, y, z], dim=2).reshape(-1, 3).contiguous()


def _plan(case, st):
    cfg = CONFIGS[case["geometry"]]
    return gpu_backend.build_ffbp_plan(st["host_pos"], cfg.fc, _extent(case, st["host_pos"]), leaf_size=case["leaf"],
                                       range_spacing=cfg.range_spacing, angular_oversample=cfg.angular_oversample)


def _batch_cases(case):
    """The scenes of a batch: pulses and sides around the nominal ones, kinds in turn."""
    out = []
    for i in range(case["scenes"]):
        side = case["side"] * (1 + i % 3) // 2
        sub = dict(kind="lattice" if i % 2 == 0 else "ffbp", geometry=case["geometry"],
                   pulses=case["pulses"] * (2 + i % 4) // 4, rows=side, cols=side, spacing=0.5, leaf=16)
        sub["samples"] = _samples_for(sub)
        out.append(sub)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "compress":
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        shape = (case["pulses"], case["samples"])
        raw = torch.complex(torch.randn(shape, device=DEV, generator=gen), torch.randn(shape, device=DEV, generator=gen))
        raw = raw * 60.0 + (1.5 - 0.75j)  # the receiver's DC offset; converter counts are whole numbers
        return dict(kind=kind, raw=torch.complex(raw.real.round(), raw.imag.round()), oversample=case["oversample"])
    if kind == "batch":
        scenes = []
        for i, sub in enumerate(_batch_cases(case)):
            st, _, _ = _scene(sub, seed * 1000 + i)
            args = (st["data"], st["pos"], st["weight"], st["phase"], *st["radar"])
            if sub["kind"] == "lattice":
                scenes.append(batch.DirectScene(*args, *st["lattice"]))
            else:
                scenes.append(batch.FFBPScene(*args, plan=_plan(sub, st)))
        return dict(kind=kind, batch=batch.SceneBatch(scenes))
    st, rng, gen = _scene(case, seed)
    if kind == "polar":
        st["grid"], st["mode"] = _plan(case, st).grid(), case["mode"]
    elif kind == "points":
        st["xyz"] = _terrain(case, st, rng)
    elif kind == "grad":
        shape = st["lattice"][3:]
        st["upstream"] = torch.complex(torch.randn(shape, device=DEV, generator=gen),
                                       torch.randn(shape, device=DEV, generator=gen))
        for name in ("pos", "weight", "phase"):
            st[name].requires_grad_(True)
    elif kind == "ffbp":
        plan = _plan(case, st)
        st["plan"], st["grid"] = plan, plan.grid()
        st["program"] = core.FFBPProgram(plan.nodes(), plan.crop_r, plan.crop_u)
    elif kind == "form":
        st["extent"], st["leaf"] = _extent(case, st["host_pos"]), case["leaf"]
    elif kind == "ground":
        st["grid"] = _plan(case, st).grid()
        shape = (st["grid"].nr, st["grid"].nu)
        st["image"] = torch.complex(torch.randn(shape, device=DEV, generator=gen),
                                    torch.randn(shape, device=DEV, generator=gen))
        st["xyz"] = _terrain(case, st, rng)
        st["xyz"][:, 2] = 0.0
    elif kind == "pga":
        origin, sr, sc, rows, cols = st["lattice"]
        n = case["targets"]
        pts = np.zeros((n, 3))
        pts[:, 0] = origin[0] + rng.uniform(0, rows, n) * sr[0]
        pts[:, 1] = origin[1] + rng.uniform(0, cols, n) * sc[1]
        st["points"], st["cutoff"] = torch.from_numpy(pts).to(DEV), case["cutoff"]
    return st


# ---- one pass ------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "compress":
        return sar_io.range_compress(state["raw"], oversample=state["oversample"])
    if kind == "batch":
        state["batch"].execute()
        return state["batch"].outputs
    inputs = (state["data"], state["pos"], state["weight"], state["phase"])
    if kind == "lattice":
        return core.backproject_lattice(*inputs, *state["lattice"], *state["radar"])
    if kind == "polar":
        return core.direct_polar(*inputs, state["grid"], *state["radar"], mode=state["mode"])
    if kind == "points":
        return core.backproject_points(*inputs, state["xyz"], *state["radar"])
    if kind == "grad":
        image = autograd.backproject_lattice(*inputs, *state["lattice"], *state["radar"])
        grads = torch.autograd.grad(image, [state["pos"], state["weight"], state["phase"]], state["upstream"])
        return [image.detach(), *grads]
    if kind == "ffbp":
        polar = state["program"].execute(*inputs, *state["radar"])
        return [polar, core.evaluate_lattice(polar, state["grid"], *state["lattice"], state["cfg"].k)]
    if kind == "form":
        cfg = state["cfg"]
        result, _ = ffbp.form_ffbp(state["data"], state["pos"], cfg.range_start, cfg.data_dr, cfg.fc, state["extent"],
                                   leaf_size=state["leaf"], range_spacing=cfg.range_spacing,
                                   angular_oversample=cfg.angular_oversample, weight=state["weight"],
                                   phase=state["phase"], verbose=False)
        return result.image
    if kind == "ground":
        return core.evaluate_image(state["image"], state["grid"], state["xyz"], state["cfg"].k)
    if kind == "pga":
        delta, stats = autofocus.estimate_update(state["data"], state["pos"], state["points"], *state["radar"],
                                                 state["cfg"].prf, state["cutoff"])
        return [delta, stats["median_gradient_coherence"]]
    raise ValueError(kind)


# ---- what a pass cannot do without -----------------------------------------------------------

# Floating-point operations (FMA = 2): per pixel and pulse, range, interpolation, rotation and sum; per
# parent pixel of an FFBP merge, both children's 4 x 4 stencils, coordinates and rotations.
BP_FLOPS, MERGE_FLOPS, POINT_FLOPS = 54.0, 300.0, 120.0


def _node_sizes(case):
    cfg = CONFIGS[case["geometry"]]
    pos = _track(cfg, case["pulses"])
    plan = gpu_backend.build_ffbp_plan(pos, cfg.fc, _extent(case, pos), leaf_size=case["leaf"],
                                       range_spacing=cfg.range_spacing, angular_oversample=cfg.angular_oversample)
    leaf = sum(n.nr * n.nu * (n.b - n.a) for n in plan.nodes() if n.is_leaf)
    merged = sum(n.nr * n.nu for n in plan.nodes() if not n.is_leaf)
    every = sum(n.nr * n.nu for n in plan.nodes())
    return plan, leaf, merged, every


def work(case):
    kind = case["kind"]
    if kind == "compress":
        p, s, o = case["pulses"], case["samples"], case["oversample"]
        n = s + 399
        return dict(bytes=8.0 * p * s * (1 + o), flops=p * (5.0 * n * math.log2(n) * (1 + o) + 6.0 * n))
    if kind == "batch":
        parts = [work(sub) for sub in _batch_cases(case)]
        return dict(bytes=sum(w["bytes"] for w in parts), flops=sum(w["flops"] for w in parts))
    p, pixels = case["pulses"], case["rows"] * case["cols"]
    bins = min(case["samples"], _samples_for(case))  # the part of each pulse that the scene lies in
    base = 8.0 * p * bins + 40.0 * p
    if kind == "lattice":
        return dict(bytes=base + 8.0 * pixels, flops=BP_FLOPS * p * pixels)
    if kind == "points":
        return dict(bytes=base + 32.0 * pixels, flops=BP_FLOPS * p * pixels)
    if kind == "grad":
        return dict(bytes=2 * base + 16.0 * pixels + 40.0 * p, flops=3 * BP_FLOPS * p * pixels)
    if kind == "pga":
        n = case["targets"] * p
        return dict(bytes=(32.0 + 24.0) * n, flops=(POINT_FLOPS + 2 * 4 * 2 * 9.0) * n)
    plan, leaf, merged, every = _node_sizes(case)
    if kind == "polar":
        return dict(bytes=base + 8.0 * plan.nr * plan.nu, flops=BP_FLOPS * p * plan.nr * plan.nu)
    if kind == "ground":
        return dict(bytes=8.0 * plan.nr * plan.nu + 32.0 * pixels, flops=POINT_FLOPS * pixels)
    # FFBP: each node's image written once and read once by its parent.
    flops = BP_FLOPS * leaf + MERGE_FLOPS * merged
    if kind == "ffbp":
        return dict(bytes=base + 16.0 * every + 8.0 * pixels, flops=flops + POINT_FLOPS * pixels)
    return dict(bytes=base + 16.0 * every, flops=flops)


# ---- the same in 64 bits -----------------------------------------------------------------------

EXACT_PAIRS = 2.0e10  # pixel-pulse pairs that plain torch forms in 64 bits within the time there is


def _weights(t):
    return (-t * (t - 1) * (t - 2) / 6, (t + 1) * (t - 1) * (t - 2) / 2, -(t + 1) * t * (t - 2) / 2,
            (t + 1) * t * (t - 1) / 6)


def _unit(turns):
    a = (turns - torch.round(turns)) * (2 * math.pi)
    return torch.complex(torch.cos(a), torch.sin(a))


def _sample(rows, q):
    """The four-point Lagrange sample of each row (dim 0) at fractional bins q, zero off the row."""
    i = torch.floor(q)
    t = q - i
    ok = (i >= 1) & (i + 2 < rows.shape[1])
    i = torch.where(ok, i, torch.ones_like(i)).long()
    v = torch.zeros_like(q, dtype=torch.complex128)
    for a, w in enumerate(_weights(t)):
        v += w * torch.gather(rows, 1, i + (a - 1))
    return torch.where(ok, v, torch.zeros_like(v))


def _bp64(st, xyz, demod=None, pulses=None, adjoint=None):
    """Direct BP at xyz [M, 3]; with `adjoint` (the upstream gradient [M]) the per-pulse gradients instead."""
    rs, dr, k = st["radar"]
    a, b = pulses or (0, st["pos"].shape[0])
    pos, w, ph = st["pos"].detach()[a:b], st["weight"].detach()[a:b], st["phase"].detach()[a:b]
    m = xyz.shape[0]
    out = torch.zeros(m, dtype=torch.complex128, device=DEV)
    g = [torch.zeros(b - a, 3, dtype=torch.float64, device=DEV), torch.zeros(b - a, dtype=torch.float64, device=DEV),
         torch.zeros(b - a, dtype=torch.float64, device=DEV)]
    step = min(b - a, 64)
    block = max(1, 2**23 // step)
    for c in range(0, b - a, step):
        e = min(b - a, c + step)
        rows = st["data"][a + c:a + e].to(torch.complex128)
        for s in range(0, m, block):
            x = xyz[s:s + block]
            v = [x[None, :, i] - pos[c:e, i, None] for i in range(3)]
            d = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            q = (d - rs) / dr
            turns = d if demod is None else d - demod[None, s:s + block]
            z = _unit(k / (2 * math.pi) * turns + ph[c:e, None] / (2 * math.pi))
            f = _sample(rows, q)
            if adjoint is None:
                out[s:s + block] += (w[c:e, None] * f * z).sum(0)
                continue
            gz = adjoint[None, s:s + block].conj() * z
            i = torch.floor(q)
            t = q - i
            ok = (i >= 1) & (i + 2 < rows.shape[1])
            i = torch.where(ok, i, torch.ones_like(i)).long()
            slope = (-(3 * t * t - 6 * t + 2) / 6, (3 * t * t - 4 * t - 1) / 2, -(3 * t * t - 2 * t - 2) / 2,
                     (3 * t * t - 1) / 6)
            df = torch.zeros_like(f)
            for n, y in enumerate(slope):
                df += y * torch.gather(rows, 1, i + (n - 1))
            df = torch.where(ok, df, torch.zeros_like(df))
            along = w[c:e, None] * (gz * (df / dr + 1j * k * f)).real / d
            for n in range(3):
                g[0][c:e, n] -= (along * v[n]).sum(1)
            g[1][c:e] += (gz * f).real.sum(1)
            g[2][c:e] -= w[c:e] * (gz * f).imag.sum(1)
    return out if adjoint is None else g


def _lattice_points(lat):
    origin, sr, sc, rows, cols = lat
    i = torch.arange(rows, dtype=torch.float64, device=DEV)[:, None, None]
    j = torch.arange(cols, dtype=torch.float64, device=DEV)[None, :, None]
    o, r, c = (torch.tensor(v, dtype=torch.float64, device=DEV) for v in (origin, sr, sc))
    return (o + i * r + j * c).reshape(-1, 3)


def _polar_points(g, r0, u0, nr, nu):
    """(xyz [nr nu, 3], r [nr nu]) of a polar grid's pixels; g has origin, dr, du, side."""
    o = [float(v) for v in g.origin]
    r = (r0 + g.dr * torch.arange(nr, dtype=torch.float64, device=DEV))[:, None].expand(nr, nu)
    u = (u0 + g.du * torch.arange(nu, dtype=torch.float64, device=DEV))[None, :].expand(nr, nu)
    ground = torch.sqrt(torch.clamp(r * r - o[2] ** 2, min=0.0))
    x = o[0] + g.side * ground * torch.sqrt(torch.clamp(1 - u * u, min=0.0))
    return torch.stack([x, o[1] + ground * u, torch.zeros_like(x)], 2).reshape(-1, 3), r.reshape(-1)


def _image_at(img, g, r0, u0, xyz):
    """The 4 x 4 Lagrange sample of a polar image (first pixel at r0, u0) at ground points, and their ranges."""
    vx, vy = xyz[:, 0] - float(g.origin[0]), xyz[:, 1] - float(g.origin[1])
    ground = torch.sqrt(vx * vx + vy * vy)
    r = torch.sqrt(ground * ground + float(g.origin[2]) ** 2)
    qr, qu = (r - r0) / g.dr, (vy / ground - u0) / g.du
    ir, iu = torch.floor(qr), torch.floor(qu)
    wr, wu = _weights(qr - ir), _weights(qu - iu)
    ok = (ir >= 1) & (iu >= 1) & (ir + 2 < img.shape[0]) & (iu + 2 < img.shape[1])
    at = torch.where(ok, (ir - 1) * img.shape[1] + iu - 1, torch.zeros_like(ir)).long()
    flat, v = img.reshape(-1), torch.zeros_like(r, dtype=torch.complex128)
    for a in range(4):
        row = torch.zeros_like(v)
        for b in range(4):
            row += wu[b] * flat[torch.where(ok, at + a * img.shape[1] + b, at)]
        v += wr[a] * row
    return torch.where(ok, v, torch.zeros_like(v)), r


def _ffbp64(st, plan):
    """The plan's FFBP image (cropped) in 64 bits."""
    k = st["radar"][2] / (2 * math.pi)

    def form(n, r_off, u_off, nr, nu):
        r0, u0 = n.r0 + n.dr * r_off, n.u0 + n.du * u_off
        if n.is_leaf:
            xyz, r = _polar_points(n, r0, u0, nr, nu)
            return _bp64(st, xyz, demod=r, pulses=(n.a, n.b)).reshape(nr, nu)
        kids = [(c, form(c, 0, 0, c.nr, c.nu)) for c in (n.left, n.right)]
        out = torch.zeros(nr, nu, dtype=torch.complex128, device=DEV)
        block = max(1, 2**22 // nu)
        for s in range(0, nr, block):
            e = min(nr, s + block)
            xyz, r = _polar_points(n, r0 + n.dr * s, u0, e - s, nu)
            for c, img in kids:
                v, rr = _image_at(img, c, c.r0, c.u0, xyz)
                out[s:e] += (v * _unit(k * (rr - r))).reshape(e - s, nu)
        return out

    return form(plan.root, plan.crop_r[0], plan.crop_u[0], plan.nr, plan.nu)


def _compress64(raw, oversample):
    """Correlation with the centred, Hamming-weighted chirp of range_compress's default radar."""
    fs, tp, bandwidth, sign = 400e6, 1e-6, 200e6, -1
    n = round(tp * fs)
    t = (np.arange(n) - n // 2) / fs
    ref = np.exp(1j * np.pi * sign * bandwidth / tp * t**2).astype(np.complex64)
    ref *= np.hamming(n + 1)[:-1].astype(np.float32)  # periodic window; the reference chirp is a complex64 table
    h = torch.from_numpy(np.conj(ref[::-1]).astype(np.complex128)).to(DEV)
    samples = raw.shape[1]
    nfft = samples + n - 1
    while not _smooth(nfft):
        nfft += 1
    filt = torch.fft.fft(h, n=nfft)
    out = torch.empty(raw.shape[0], samples * oversample, dtype=torch.complex128, device=DEV)
    first = (n - 1 - n // 2) * oversample
    for s in range(0, raw.shape[0], 512):
        x = raw[s:s + 512].to(torch.complex128)
        spec = torch.fft.fft(x - x.mean(dim=1, keepdim=True), n=nfft, dim=1) * filt
        if oversample > 1:  # Fourier interpolation, the even length's middle bin in two halves
            long = torch.zeros(x.shape[0], nfft * oversample, dtype=torch.complex128, device=DEV)
            half = (nfft + 1) // 2
            long[:, :half] = spec[:, :half]
            long[:, nfft * oversample - nfft // 2:] = spec[:, nfft - nfft // 2:]
            if nfft % 2 == 0:
                mid = 0.5 * spec[:, nfft // 2]
                long[:, nfft // 2] = mid
                long[:, nfft * oversample - nfft // 2] = mid
            spec = long * oversample
        out[s:s + 512] = torch.fft.ifft(spec, dim=1)[:, first:first + samples * oversample]
    return out


def _smooth(n):
    """Whether n has no prime factor over 11: the lengths that scipy's complex next_fast_len picks from."""
    for f in (2, 3, 5, 7, 11):
        while n % f == 0:
            n //= f
    return n == 1


def _smooth_histories(x, cutoff, prf):
    """Zero-phase fourth-order Butterworth smoothing of each row: odd extension by 15 samples, forward and
    backward, each from the steady state of the first sample."""
    pad, warped = 15, 4.0 * math.tan(math.pi * cutoff / prf)
    poles = warped * np.exp(1j * np.pi * (2 * np.arange(2) + 5) / 8)
    z = (4 + poles) / (4 - poles)
    sections = [((1 - 2 * p.real + abs(p) ** 2) / 4, -2 * p.real, abs(p) ** 2) for p in z]
    x = np.concatenate([2 * x[:, :1] - x[:, pad:0:-1], x, 2 * x[:, -1:] - x[:, -2:-pad - 2:-1]], axis=1)
    for _ in range(2):
        x = np.ascontiguousarray(x.T)
        for g, a1, a2 in sections:
            s0, s1 = (1 - g) * x[0], (g - a2) * x[0]
            for i in range(len(x)):
                y = g * x[i] + s0
                s0 = 2 * g * x[i] - a1 * y + s1
                s1 = g * x[i] - a2 * y
                x[i] = y
        x = x.T[:, ::-1]
    return x[:, pad:-pad]


def _update64(st):
    """[trajectory update, median coherence] of one phase-gradient autofocus pass."""
    rs, dr, k = st["radar"]
    n, xyz = st["pos"].shape[0], st["points"]
    xi = torch.empty(xyz.shape[0], n, dtype=torch.complex128, device=DEV)
    for c in range(0, n, 256):
        d = torch.linalg.norm(xyz[None] - st["pos"][c:c + 256, None], dim=2)
        xi[:, c:c + 256] = (_sample(st["data"][c:c + 256].to(torch.complex128), (d - rs) / dr)
                            * _unit(k / (2 * math.pi) * d)).T
    y = _smooth_histories(xi.cpu().numpy(), st["cutoff"], st["cfg"].prf)
    pos, xyz = st["host_pos"], xyz.cpu().numpy()
    cross = y[:, 1:] * y[:, :-1].conj()
    amp = np.abs(cross)
    power = amp.mean(axis=1)
    coherence = np.abs(cross.sum(axis=1)) / amp.sum(axis=1)
    w = amp / (power[:, None] + 1e-12) * np.minimum(np.sqrt(power / np.median(power)), 3.0)[:, None]
    w = np.minimum(w * np.clip(coherence, 0, 1)[:, None] ** 2, 4.0)
    vec = xyz[:, None] - pos[None, 1:]
    dist = np.linalg.norm(vec, axis=2)
    ux, uy, rhs = vec[..., 0] / dist, vec[..., 1] / dist, np.angle(cross) / k
    for _ in range(3):
        a, b, c = (w * ux * ux).sum(0), (w * ux * uy).sum(0), (w * uy * uy).sum(0)
        ex, ey = (w * ux * rhs).sum(0), (w * uy * rhs).sum(0)
        reg = 0.002 * (a + c)
        det = np.maximum((a + reg) * (c + reg) - b * b, 1e-12)
        dx, dy = (ex * (c + reg) - ey * b) / det, (ey * (a + reg) - ex * b) / det
        left = np.abs(rhs - ux * dx - uy * dy)
        w = w * np.minimum(2.5 * (1.4826 * np.median(left, axis=0) + 1e-6) / (left + 1e-12), 1.0)
    xy = np.zeros((n, 2))
    xy[1:, 0], xy[1:, 1] = np.cumsum(dx), np.cumsum(dy)
    line = np.vander(np.arange(n) - 0.5 * (n - 1), 2)
    xy = xy - line @ np.linalg.lstsq(line, xy, rcond=None)[0]
    window = min(501, n // 2 * 2 - 1)
    half, basis = window // 2, np.linalg.qr(np.vander(np.linspace(-1, 1, window), 4))[0]
    hat, out = basis @ basis.T, np.empty_like(xy)
    for i in range(half, n - half):
        out[i] = hat[half] @ xy[i - half:i + half + 1]
    out[:half], out[n - half:] = hat[:half] @ xy[:window], hat[window - half:] @ xy[n - window:]
    delta = np.zeros((n, 3))
    delta[:, :2] = out / max(1.0, np.linalg.norm(out, axis=1).max())
    return [torch.from_numpy(delta), float(np.median(coherence))]


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("compress", "batch", "ground", "pga"):
        pairs = case["pulses"] * case["rows"] * case["cols"]
        if kind == "polar":
            plan = _node_sizes(case)[0]
            pairs = plan.nr * plan.nu * case["pulses"]
        if kind in ("ffbp", "form"):
            pairs = 0.02 * pairs * (2 if case["leaf"] > 16 else 1)
        if pairs * (2 if kind == "grad" else 1) > EXACT_PAIRS:
            return None
    st = prepare(case, seed)
    if kind == "compress":
        return _compress64(st["raw"], st["oversample"])
    if kind == "batch":
        out = []
        for i, sub in enumerate(_batch_cases(case)):
            one, _, _ = _scene(sub, seed * 1000 + i)
            if sub["kind"] == "lattice":
                out.append(_bp64(one, _lattice_points(one["lattice"])).reshape(one["lattice"][3:]))
            else:
                out.append(_ffbp64(one, _plan(sub, one)))
        return out
    if kind == "lattice":
        return _bp64(st, _lattice_points(st["lattice"])).reshape(st["lattice"][3:])
    if kind == "polar":
        g = st["grid"]
        xyz, r = _polar_points(g, g.r0, g.u0, g.nr, g.nu)
        return _bp64(st, xyz, demod=r).reshape(g.nr, g.nu)
    if kind == "points":
        return _bp64(st, st["xyz"])
    if kind == "grad":
        pts = _lattice_points(st["lattice"])
        up = st["upstream"].to(torch.complex128).reshape(-1)
        image = _bp64(st, pts).reshape(st["lattice"][3:])
        return [image, *_bp64(st, pts, adjoint=up)]
    if kind == "pga":
        return _update64(st)
    k = st["radar"][2] / (2 * math.pi)
    if kind == "ground":
        v, r = _image_at(st["image"].to(torch.complex128), st["grid"], st["grid"].r0, st["grid"].u0, st["xyz"])
        return v * _unit(k * r)
    polar = _ffbp64(st, _plan(case, st))
    if kind == "form":
        return polar
    g = st["grid"]
    pts = _lattice_points(st["lattice"])
    v, r = torch.zeros(0), None
    ground = torch.zeros(pts.shape[0], dtype=torch.complex128, device=DEV)
    for s in range(0, pts.shape[0], 2**22):
        v, r = _image_at(polar, g, g.r0, g.u0, pts[s:s + 2**22])
        ground[s:s + 2**22] = v * _unit(k * r)
    return [polar, ground.reshape(st["lattice"][3:])]
