"""The work that users of the cone-beam operators have them do, as timed cases.

Each case is one pass through the public entry points: projecting a volume,
differentiating a projection (for the volume, for the scan geometry, for
both), a calibration, FDK reconstructions, a differentiable FDK layer, a
self-calibration step, a batch of uneven problems and a training step of the
warm-start network.  ``exact`` restates the operators in plain float64 torch
where that is quick enough.
"""

import math
import sys
from pathlib import Path

import torch

_PACKAGE = str(Path.cwd() / "diff-geocali_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import cbct_backprojector as cb  # noqa: E402
from dgc_b200 import batch, calibration, phantoms, warmstart  # noqa: E402

DEVICE = "cuda"
GEOMETRY = 8  # angles, sid, sod, det_u0, det_v0, src_x, src_y, src_z


# ------------------------------------------------------------------- the cases


def _scan(kind, shape, views, detector, pixel=1.0, voxel=1.0, step=0.5, sid=1000.0, sod=600.0,
          offset=(0.0, 0.0, 0.0), **more):
    D, H, W = shape
    return dict(kind=kind, D=D, H=H, W=W, A=views, U=detector[0], V=detector[1], pixel=pixel,
                voxel=voxel, step=step, sid=sid, sod=sod, off_x=offset[0], off_y=offset[1],
                off_z=offset[2], **more)


def listed():
    return [
        # The README's example size, forward and all nine gradients: what a
        # first program, a unit test or a toy optimisation calls in a loop.
        dict(_scan("project_grad", (16, 20, 24), 24, (48, 40), sid=180.0, sod=120.0, want="all"),
             name="example-step"),
        # An odd-sized region of interest off the axis, with a voxel size that
        # divides and the projector's default step.
        dict(_scan("project", (101, 150, 133), 77, (333, 257), pixel=0.9, voxel=0.7, step=0.2,
                   offset=(5.0, -3.0, 2.5)), name="project-roi"),
        # Simulating a full-size scan.
        dict(_scan("project", (512, 512, 512), 720, (768, 768)), name="project-512"),
        # One iteration of an iterative reconstruction: project the current
        # volume and differentiate the projection for the volume alone.
        dict(_scan("project_grad", (256, 256, 256), 360, (384, 384), want="volume"),
             name="iterate-256"),
        # Joint reconstruction and geometry refinement: all nine gradients.
        dict(_scan("project_grad", (128, 192, 192), 180, (256, 384), want="all"),
             name="joint-192"),
        # Geometry calibration against a known object, two Adam iterations on
        # noisy, partly starved measurements (the acquisition that the
        # warm-start network is trained on).
        dict(_scan("calibrate", (128, 128, 128), 180, (256, 256), pixel=3.0, voxel=4.0, step=2.0,
                   iterations=2), name="calibrate-128"),
        # Reconstructing a full-size scan.
        dict(_scan("fdk", (512, 512, 512), 720, (768, 768), short=False, offset_weight=False),
             name="fdk-512"),
        # A small odd-sized short scan with the offset-aware preweight.
        dict(_scan("fdk", (90, 133, 121), 200, (187, 161), sid=900.0, sod=500.0, short=True,
                   offset_weight=True), name="fdk-short"),
        # A differentiable FDK layer inside a learned reconstruction: filter
        # and backproject, then the gradient for the projections alone.
        dict(_scan("fdk_layer", (256, 256, 256), 360, (384, 384)), name="fdk-layer-256"),
        # A step of self-calibration: filter and backproject under the current
        # geometry and differentiate for the geometry alone.
        dict(_scan("selfcal", (64, 64, 64), 90, (128, 128)), name="selfcal-64"),
        # Sixteen small uneven problems, forward and backward, as one batch.
        dict(kind="batch", n=16, low=48, high=96, views_low=30, views_high=90, det_low=96,
             det_high=160, step=0.5, name="batch-16"),
        # Training the warm-start network: forward and backward over a stack.
        dict(kind="net", A=180, name="net-step"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["project", "project", "project_grad", "project_grad", "project_grad",
                       "calibrate", "fdk", "fdk", "fdk_layer", "selfcal", "batch", "net"])
    if kind == "net":
        return dict(kind="net", A=_log_int(rng, 45, 360))
    if kind == "batch":
        low = _log_int(rng, 24, 64)
        views = _log_int(rng, 16, 60)
        det = _log_int(rng, 48, 128)
        return dict(kind="batch", n=rng.randint(4, 20), low=low, high=int(low * rng.uniform(1.2, 2)),
                    views_low=views, views_high=int(views * rng.uniform(1.2, 3)), det_low=det,
                    det_high=int(det * rng.uniform(1.1, 1.7)), step=rng.choice([0.2, 0.5, 1.0]))
    top = dict(project=448, fdk=448, project_grad=224, fdk_layer=224, calibrate=160, selfcal=128)
    n = _log_int(rng, 16, top[kind])
    shape = [max(8, int(n * rng.uniform(0.5, 1.0))) for _ in range(3)]
    shape[rng.randrange(3)] = n
    voxel = rng.choice([1.0, 1.0, 0.5, 2.0, 0.7])
    pixel = round(voxel * rng.choice([1.0, 1.0, 1.3]), 3)
    step = round(voxel * rng.choice([0.5, 0.5, 0.2, 1.0]), 3)
    wide = 1.6 * n * voxel / pixel
    detector = [max(8, int(wide * rng.uniform(0.7, 1.1))) for _ in range(2)]
    extent = n * voxel
    sod = 600.0 if 150.0 < extent <= 512.0 else 3.0 * extent + 40.0
    more = {}
    if kind == "project_grad":
        more["want"] = rng.choice(["volume", "geometry", "all"])
    if kind == "calibrate":
        more["iterations"] = rng.randint(1, 3)
    if kind == "fdk":
        more["short"] = rng.random() < 0.3
        more["offset_weight"] = rng.random() < 0.3
    views = _log_int(rng, 60 if more.get("short") else 12, 720)
    # keep a drawn case well below the largest listed ones
    rays = views * detector[0] * detector[1]
    if kind in ("project", "project_grad", "calibrate"):
        cost = rays * n * voxel / step * (1 if kind == "project" else 3 * more.get("iterations", 1))
        views = max(8, min(views, int(views * 1.2e11 / cost)))
    else:
        cost = views * shape[0] * shape[1] * shape[2] * (4 if kind != "fdk" else 1)
        views = max(60, min(views, int(views * 4e10 / cost)))
    offset = [0.0, 0.0, 0.0]
    if rng.random() < 0.3:
        offset = [round(rng.uniform(-0.05, 0.05) * extent, 2) for _ in range(3)]
    return _scan(kind, shape, views, detector, pixel=pixel, voxel=voxel, step=step,
                 sid=sod * 5.0 / 3.0, sod=sod, offset=offset, **more)


# ------------------------------------------------------------------ their inputs


def _geometry(case, seed):
    """A nominal circular scan and the perturbed per-view geometry of a real one."""
    nominal = phantoms.circular_geometry(case["A"], case["U"], case["V"], case["sid"], case["sod"],
                                         case["pixel"], device=DEVICE)
    if case.get("short"):
        fan = math.atan((case["U"] - 1) / 2 * case["pixel"] / case["sid"])
        span = math.pi + 2 * fan + 0.15
        nominal[0] = torch.linspace(0.0, span, case["A"], dtype=torch.float64).to(
            DEVICE, torch.float32)
    true = calibration.perturb_geometry(nominal, seed, src_mm=case["pixel"], det_px=2.0)
    if case["kind"] == "fdk":
        true[0] = nominal[0]  # a reconstruction's views are uniformly spaced
    return nominal, true


def _axis_range(case):
    n = max(case["D"], case["H"], case["W"])
    return (n * 10.0 / 256.0, n * 80.0 / 256.0)


def _volume(case, seed):
    """A phantom of twelve ellipsoids, or noise for the smallest volumes."""
    shape = (case["D"], case["H"], case["W"])
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    if max(shape) <= 32:
        return torch.rand(shape, generator=gen, device=DEVICE)
    vol = phantoms.ellipsoid_phantom(
        shape, seed=seed, voxel_size=case["voxel"], axis_range=_axis_range(case),
        offset=(case["off_x"], case["off_y"], case["off_z"]), device=DEVICE)
    if case["kind"] == "project_grad":  # an iterate: no region of it is exactly empty
        vol += 0.01 * torch.randn(shape, generator=gen, device=DEVICE)
    return vol


def _line_integrals(case, geometry, seed):
    """Noisy line integrals of the phantom's ellipsoids, in closed form: what a detector gives."""
    params = phantoms.ellipsoid_parameters((case["D"], case["H"], case["W"]), seed=seed,
                                           voxel_size=case["voxel"], axis_range=_axis_range(case))
    A, U, V = case["A"], case["U"], case["V"]
    out = torch.empty((A, U, V), device=DEVICE)
    per = max(1, (1 << 24) // (U * V))
    for a in range(0, A, per):
        part = [g[a:a + per] for g in geometry]
        origin, target = _rays(part, case["pixel"], U, V)
        d = (target - origin[:, None, None, :]).float()
        d = d / d.norm(dim=-1, keepdim=True)
        acc = torch.zeros(d.shape[:3], device=DEVICE)
        for centre, axes, rot, mu in params:
            to_body = (rot / axes).to(DEVICE, torch.float32)  # columns scaled: (R^T p) / axes
            o = (origin.float() - centre.to(DEVICE, torch.float32)) @ to_body
            e = d @ to_body
            aa = e.square().sum(-1)
            bb = (e * o[:, None, None, :]).sum(-1)
            cc = o.square().sum(-1)[:, None, None] - 1.0
            acc += mu * 2.0 * (bb * bb - aa * cc).clamp_min(0.0).sqrt() / aa
        out[a:a + per] = acc
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 1)
    scale = min(1.0, 8.0 / float(out.max().clamp_min(1e-6)))
    counts = torch.poisson(1e5 * torch.exp(-out * scale), generator=gen).clamp_min(1.0)
    return -torch.log(counts / 1e5) / scale, (counts >= 50).float()


def _randn(shape, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    return torch.randn(shape, generator=gen, device=DEVICE)


def _batch_cases(case, seed):
    rng = torch.Generator().manual_seed(seed)

    def pick(low, high):
        return int(torch.randint(low, high + 1, (1,), generator=rng))

    # the shapes belong to the case, the data to the seed
    rng.manual_seed(case["low"] * 1000 + case["n"])
    out = []
    for _ in range(case["n"]):
        shape = [pick(case["low"], case["high"]) for _ in range(3)]
        views = pick(case["views_low"], case["views_high"])
        detector = [pick(case["det_low"], case["det_high"]) for _ in range(2)]
        out.append(_scan("project_grad", shape, views, detector, step=case["step"], want="all"))
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case, kind=kind)
    if kind == "net":
        state["net"] = warmstart.WarmStartNet(seed=seed).to(DEVICE)
        # a smooth reprojection and a noisy residual, as network_input makes them
        x = torch.nn.functional.interpolate(_randn((case["A"], 2, 12, 12), seed), size=(96, 96),
                                            mode="bilinear")
        x[:, 0] = x[:, 0].abs()
        x[:, 1] += 0.1 * _randn((case["A"], 96, 96), seed + 1)
        state["x"] = x.permute(0, 2, 3, 1).contiguous().to(torch.bfloat16)
        state["up"] = _randn((case["A"], GEOMETRY), seed + 2) / case["A"]
        return state
    if kind == "batch":
        problems = []
        for i, c in enumerate(_batch_cases(case, seed)):
            problems.append(batch.Problem(
                _volume(c, seed + i), _geometry(c, seed + i)[1], c["pixel"], c["U"], c["V"],
                step_size=c["step"], voxel_size=c["voxel"],
                grad_projections=_randn((c["A"], c["U"], c["V"]), seed + 100 + i)))
        state["problems"] = problems
        state["batch"] = batch.ProjectionBatch(problems)
        return state
    nominal, true = _geometry(case, seed)
    state["geometry"] = true
    if kind in ("project", "project_grad"):
        state["volume"] = _volume(case, seed)
        if kind == "project_grad":
            state["up"] = _randn((case["A"], case["U"], case["V"]), seed + 2)
            if case["want"] != "geometry":
                state["volume"].requires_grad_(True)
            if case["want"] != "volume":
                for g in true:
                    g.requires_grad_(True)
        return state
    state["measured"], mask = _line_integrals(case, true, seed)
    if kind == "calibrate":
        state["volume"] = _volume(case, seed)
        state["mask"] = mask
        state["nominal"] = nominal
    elif kind == "fdk_layer":
        state["measured"].requires_grad_(True)
        state["up"] = _randn((case["D"], case["H"], case["W"]), seed + 2)
    elif kind == "selfcal":
        for g in true:
            g.requires_grad_(True)
        state["up"] = _randn((case["D"], case["H"], case["W"]), seed + 2)
    return state


# -------------------------------------------------------------------- one pass


def _offset(c):
    return (c["off_x"], c["off_y"], c["off_z"])


def _project(state):
    c = state["case"]
    return cb.project(state["volume"], *state["geometry"], c["pixel"], c["U"], c["V"],
                      step_size=c["step"], voxel_size=c["voxel"], off_x=c["off_x"],
                      off_y=c["off_y"], off_z=c["off_z"])


def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "project":
        return _project(state)
    if kind == "project_grad":
        p = _project(state)
        wrt = [t for t in (state["volume"], *state["geometry"]) if t.requires_grad]
        return [p.detach(), *torch.autograd.grad(p, wrt, grad_outputs=state["up"])]
    if kind == "calibrate":
        scan = calibration.ScanSetup(U=c["U"], V=c["V"], pixel_size=c["pixel"],
                                     step_size=c["step"], voxel_size=c["voxel"],
                                     volume_offset=_offset(c))
        r = calibration.calibrate(state["volume"], state["measured"], state["nominal"], scan,
                                  iterations=c["iterations"], mask=state["mask"])
        return [*r.geometry, r.final_loss]
    shape = (c.get("D"), c.get("H"), c.get("W"))
    if kind == "fdk":
        return cb.reconstruct_fdk(state["measured"], *state["geometry"], c["pixel"], shape,
                                  c["voxel"], _offset(c), short_scan=c["short"],
                                  offset_preweight=c["offset_weight"])
    if kind in ("fdk_layer", "selfcal"):
        g = state["geometry"]
        filtered = cb.fdk_filter(state["measured"], c["pixel"], g[2], g[1])
        vol = cb.backproject(filtered, *g, c["pixel"], shape, c["voxel"], _offset(c)) * (
            math.pi / c["A"])
        wrt = [state["measured"]] if kind == "fdk_layer" else g
        return [vol.detach(), *torch.autograd.grad(vol, wrt, grad_outputs=state["up"])]
    if kind == "batch":
        b = state["batch"]
        b.step()
        return [b.projections, b.grad_volumes, b.grad_geometry]
    net = state["net"]
    out = net(state["x"])
    return [out.detach(), *torch.autograd.grad(out, list(net.parameters()),
                                               grad_outputs=state["up"])]


# ------------------------------------------------- what a pass cannot do without


def _samples(c):
    """Samples of a projection: the rays' chords through the box over the step."""
    extent = [c[k] * c["voxel"] for k in "DHW"]
    mag = c["sid"] / c["sod"]
    rays = c["U"] * c["V"]
    inside = min(rays, mag * mag * extent[0] * math.hypot(extent[1], extent[2]) / c["pixel"] ** 2)
    chord = min(math.prod(extent) * mag * mag / c["pixel"] ** 2 / max(inside, 1.0),
                math.hypot(extent[1], extent[2]))
    return c["A"] * inside * chord / c["step"]


_SAMPLE = 21.0     # position, seven lerps and the sum
_GRADIENT = 24.0   # three derivatives and six running sums
_ADJOINT = 24.0    # eight weights and their sums
_TAP = 16.0        # detector position, three lerps and the sum


def work(case):
    c, kind = case, case["kind"]
    if kind == "net":
        macs, size, cin = 0.0, 96, 2
        for cout in (32, 64, 128, 256):
            size //= 2
            macs += size * size * 9 * (cin * cout + cout * cout)
            cin = cout
        return {"bytes": c["A"] * 96 * 96 * 2 * 2.0, "flops": 2.0 * 3.0 * macs * c["A"]}
    if kind == "batch":
        parts = [work(p) for p in _batch_cases(c, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    voxels, rays = c["D"] * c["H"] * c["W"], c["A"] * c["U"] * c["V"]
    geometry = 4.0 * GEOMETRY * c["A"]
    if kind == "project":
        return {"bytes": 4.0 * (voxels + rays) + geometry, "flops": _SAMPLE * _samples(c)}
    if kind == "project_grad":
        vol, geo = c["want"] != "geometry", c["want"] != "volume"
        return {"bytes": 4.0 * (voxels * (2 if vol else 1) + 2 * rays) + geometry * (2 if geo else 1),
                "flops": _samples(c) * (_SAMPLE + _ADJOINT * vol + (_GRADIENT + 7.0) * geo)}
    if kind == "calibrate":
        passes = c["iterations"] + 1
        return {"bytes": 4.0 * (voxels + 2 * rays) + geometry,
                "flops": _samples(c) * (_SAMPLE * passes + _GRADIENT * c["iterations"])}
    # the ramp filter as a padded real FFT there and back per detector column
    points = 1 << (2 * c["U"] - 1).bit_length()
    ramp = c["A"] * c["V"] * (5.0 * points * math.log2(points) + 6.0 * points)
    taps = float(voxels) * c["A"]
    scale = {"fdk": 1, "fdk_layer": 2, "selfcal": 2}[kind]
    more = {"fdk": 0.0, "fdk_layer": 4.0 * rays, "selfcal": geometry}[kind]
    return {"bytes": 4.0 * (voxels * scale + rays) + geometry + more,
            "flops": scale * (ramp + _TAP * taps)}


# ------------------------------------------------------ the same in 64 bits


def _rays(geometry, pixel, U, V):
    """Source [a, 3] and detector points [a, U, V, 3] of the views, in float64."""
    angles, sid, sod, u0, v0, sx, sy, sz = (g.double() for g in geometry)
    c, s = torch.cos(angles), torch.sin(angles)
    origin = torch.stack([sx - sod * s, sy + sod * c, sz], -1)
    up = (torch.arange(U, device=DEVICE, dtype=torch.float64)[None] - u0[:, None]) * pixel
    vp = (torch.arange(V, device=DEVICE, dtype=torch.float64)[None] - v0[:, None]) * pixel
    dn = (sod - sid)[:, None]
    tx = up * c[:, None] - dn * s[:, None]
    ty = up * s[:, None] + dn * c[:, None]
    shape = (angles.numel(), U, V)
    target = torch.stack([tx[:, :, None].expand(shape), ty[:, :, None].expand(shape),
                          vp[:, None, :].expand(shape)], -1)
    return origin, target


def _exact_projection(c, vol, geometry):
    """Line integrals of some views, differentiable in the volume and the geometry."""
    origin, target = _rays(geometry, c["pixel"], c["U"], c["V"])
    ray = (target - origin[:, None, None, :]).reshape(-1, 3)
    origin = origin[:, None, None, :].expand(target.shape).reshape(-1, 3)
    d = ray / ray.norm(dim=-1, keepdim=True)
    size = torch.tensor([c["W"], c["H"], c["D"]], device=DEVICE, dtype=torch.float64)
    off = torch.tensor(_offset(c), device=DEVICE, dtype=torch.float64)
    lo = (-size / 2 - 0.5) * c["voxel"] + off
    hi = (size / 2 - 0.5) * c["voxel"] + off
    t0, t1 = (lo - origin) / d, (hi - origin) / d
    tmin = torch.minimum(t0, t1).amax(-1).clamp_min(0.0)
    tmax = torch.maximum(t0, t1).amin(-1)
    hit = torch.nonzero(tmax.detach() >= tmin.detach()).flatten()
    out = torch.zeros(d.shape[0], device=DEVICE, dtype=torch.float64)
    if hit.numel():
        o, e, tmin, tmax = origin[hit], d[hit], tmin[hit], tmax[hit]
        count = int(((tmax - tmin).detach().max() / c["step"]).floor()) + 1
        t = tmin[:, None] + c["step"] * torch.arange(count, device=DEVICE, dtype=torch.float64)
        on = t.detach() <= tmax.detach()[:, None]
        value = on.double()
        # trilinear interpolation with neighbours clamped to the volume
        cells, parts = [], []
        for k, n in enumerate((c["W"], c["H"], c["D"])):
            x = (o[:, k, None] + t * e[:, k, None] - off[k]) / c["voxel"] + n / 2
            f = x.detach().floor()
            cells.append((f.long().clamp(0, n - 1), (f.long() + 1).clamp(0, n - 1)))
            parts.append(x - f)
        flat = vol.reshape(-1)

        def at(iz, iy, ix):
            index = (cells[2][iz] * c["H"] + cells[1][iy]) * c["W"] + cells[0][ix]
            return flat[index]

        def along_x(iz, iy):
            a, b = at(iz, iy, 0), at(iz, iy, 1)
            return a + parts[0] * (b - a)

        def along_y(iz):
            a, b = along_x(iz, 0), along_x(iz, 1)
            return a + parts[1] * (b - a)

        a, b = along_y(0), along_y(1)
        value = value * (a + parts[2] * (b - a))
        out = out.index_put((hit,), value.sum(-1) * c["step"])
    return out.reshape(-1, c["U"], c["V"])


def _exact_project_grad(c, vol, geometry, up, want):
    """[projection, gradients asked for] view by view."""
    vol = vol.detach().double()
    geometry = [g.detach().double() for g in geometry]
    per = max(1, int(1.2e7 * c["step"] / (c["U"] * c["V"] * c["voxel"] *
                                          math.hypot(c["D"], c["H"], c["W"]))))
    p = torch.empty((c["A"], c["U"], c["V"]), device=DEVICE, dtype=torch.float64)
    gv = torch.zeros_like(vol)
    gg = [torch.zeros_like(g) for g in geometry]
    for a in range(0, c["A"], per):
        part = [g[a:a + per].requires_grad_(want in ("geometry", "all")) for g in geometry]
        v = vol.detach().requires_grad_(want in ("volume", "all"))
        with torch.set_grad_enabled(want != ""):
            q = _exact_projection(c, v, part)
        p[a:a + per] = q.detach()
        wrt = [t for t in (v, *part) if t.requires_grad]
        if wrt:
            got = list(torch.autograd.grad(q, wrt, grad_outputs=up[a:a + per].double()))
            if v.requires_grad:
                gv += got.pop(0)
            for k, g in enumerate(got):
                gg[k][a:a + per] = g
        del q
    out = [p]
    if want in ("volume", "all"):
        out.append(gv)
    if want in ("geometry", "all"):
        out += gg
    return out


def _exact_filter(c, p, sid, sod, frame=None, weights=None, alpha=0.8):
    """The cosine-weighted, Hann-windowed ramp filter of some views by a padded FFT."""
    U, V, px = c["U"], c["V"], c["pixel"]
    points = 1 << (2 * U - 1).bit_length()
    dist, cu, cv = frame if frame is not None else (
        sid, torch.full_like(sid, (U - 1) / 2), torch.full_like(sid, (V - 1) / 2))
    u = (torch.arange(U, device=DEVICE, dtype=torch.float64)[None] - cu[:, None]) * px
    v = (torch.arange(V, device=DEVICE, dtype=torch.float64)[None] - cv[:, None]) * px
    w = dist[:, None, None] / (dist[:, None, None] ** 2 + u[:, :, None] ** 2 +
                               v[:, None, :] ** 2).sqrt()
    if weights is not None:
        w = w * weights[:, :, None]
    n = torch.arange(points, device=DEVICE, dtype=torch.float64)
    n = torch.where(n > points // 2, n - points, n)
    r = torch.where(n.long() % 2 != 0, -1.0 / (math.pi * n * px) ** 2, torch.zeros_like(n))
    r[0] = 1.0 / (4.0 * px * px)
    f = torch.fft.rfftfreq(points, device=DEVICE, dtype=torch.float64)
    hann = torch.where(f <= alpha / 2, 0.5 + 0.5 * torch.cos(2 * math.pi * f / alpha),
                       torch.zeros_like(f))
    response = torch.fft.rfft(r).real * hann
    y = torch.fft.irfft(torch.fft.rfft(p * w, n=points, dim=1) * response[None, :, None],
                        n=points, dim=1)[:, :U]
    return y * (px * sid / sod)[:, None, None]


def _exact_backprojection(c, p, geometry):
    """Sum over some views of the FDK-weighted bilinear detector samples."""
    axes = [(torch.arange(n, device=DEVICE, dtype=torch.float64) - n / 2) * c["voxel"] + o
            for n, o in ((c["D"], c["off_z"]), (c["H"], c["off_y"]), (c["W"], c["off_x"]))]
    z, y, x = axes[0][:, None, None], axes[1][:, None], axes[2][None]
    U, V = c["U"], c["V"]
    out = torch.zeros((c["D"], c["H"], c["W"]), device=DEVICE, dtype=torch.float64)
    for a in range(p.shape[0]):
        beta, sid, sod, u0, v0, sx, sy, sz = (g[a] for g in geometry)
        co, si = torch.cos(beta), torch.sin(beta)
        px, py = x * co + y * si, -x * si + y * co
        du, dn = sx * co + sy * si, -sx * si + sy * co
        q = sod + dn - py
        t = (sid + dn) / q
        ui = (du + t * (px - du)) / c["pixel"] + u0
        vi = (sz + t * (z - sz)) / c["pixel"] + v0
        fu, fv = ui.detach().floor(), vi.detach().floor()
        on = (q > 1e-6) & (ui >= 0) & (ui < U - 1) & (vi >= 0) & (vi < V - 1)
        iu, iv = fu.long().clamp(0, U - 2), fv.long().clamp(0, V - 2)
        flat = p[a].reshape(-1)
        base = iu * V + iv
        wu, wv = ui - fu, vi - fv
        a0 = flat[base] + wu * (flat[base + V] - flat[base])
        a1 = flat[base + 1] + wu * (flat[base + V + 1] - flat[base + 1])
        out = out + on * ((sod + dn) / q) ** 2 * (a0 + wv * (a1 - a0))
    return out


def _exact_parker(c, angles, dist, cu):
    beta = angles - angles[0]
    gamma_max = 0.5 * (float(beta[-1]) - math.pi)
    u = (torch.arange(c["U"], device=DEVICE, dtype=torch.float64)[None] - cu[:, None]) * c["pixel"]
    g, b = torch.atan(u / dist[:, None]), beta[:, None]
    first = torch.sin(math.pi / 4 * b / (gamma_max - g)) ** 2
    last = torch.sin(math.pi / 4 * (math.pi + 2 * gamma_max - b) / (gamma_max + g)) ** 2
    w = torch.where(b <= math.pi - 2 * g, torch.ones_like(first), last)
    w = torch.where(b < 2 * (gamma_max - g), first, w)
    return torch.where(b <= math.pi + 2 * gamma_max, w, torch.zeros_like(w))


def _exact_fdk(c, p, geometry):
    geometry = [g.double() for g in geometry]
    angles, sid, sod, u0, v0, sx, sy, sz = geometry
    co, si = torch.cos(angles), torch.sin(angles)
    frame = None
    if c["offset_weight"]:
        frame = (sid - sx * si + sy * co, u0 + (sx * co + sy * si) / c["pixel"],
                 v0 + sz / c["pixel"])
    weights, scale = None, math.pi / c["A"]
    if c["short"]:
        dist, cu = frame[:2] if frame else (sid, torch.full_like(sid, (c["U"] - 1) / 2))
        weights = _exact_parker(c, angles, dist, cu)
        scale = float(angles[-1] - angles[0]) / (c["A"] - 1)
    out = torch.zeros((c["D"], c["H"], c["W"]), device=DEVICE, dtype=torch.float64)
    for a in range(0, c["A"], 16):
        s = slice(a, a + 16)
        y = _exact_filter(c, p[s].double(), sid[s], sod[s],
                          None if frame is None else [f[s] for f in frame],
                          None if weights is None else weights[s])
        out += _exact_backprojection(c, y, [g[s] for g in geometry])
    return (out * scale).clamp_min(0.0)


def _exact_layer(c, p, geometry, up, wrt_projections):
    out = torch.zeros((c["D"], c["H"], c["W"]), device=DEVICE, dtype=torch.float64)
    scale = math.pi / c["A"]
    per = max(1, int(1.2e7 / out.numel()))
    gp = torch.zeros_like(p, dtype=torch.float64)
    gg = [torch.zeros_like(g, dtype=torch.float64) for g in geometry]
    for a in range(0, c["A"], per):
        s = slice(a, a + per)
        q = p[s].detach().double().requires_grad_(wrt_projections)
        g = [t[s].detach().double().requires_grad_(not wrt_projections) for t in geometry]
        vol = _exact_backprojection(c, _exact_filter(c, q, g[1], g[2]), g) * scale
        got = torch.autograd.grad(vol, [q] if wrt_projections else g, grad_outputs=up.double())
        out += vol.detach()
        if wrt_projections:
            gp[s] = got[0]
        else:
            for t, r in zip(gg, got):
                t[s] = r
        del vol
    return [out, gp] if wrt_projections else [out, *gg]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("net", "calibrate"):
        return None  # 16-bit products; optimiser steps of a gradient's sign
    if kind == "batch":
        parts = _batch_cases(case, seed)
        if sum(_samples(p) for p in parts) > 1.5e9:
            return None
        state = prepare(case, seed)
        got = [_exact_project_grad(c, pr.volume, pr.geometry, pr.grad_projections, "volume")
               for c, pr in zip(parts, state["problems"])]
        return [[g[0] for g in got], [g[1] for g in got], [None for _ in got]]
    voxel_views = case["D"] * case["H"] * case["W"] * case["A"]
    if kind in ("project", "project_grad"):
        if _samples(case) > (3e9 if kind == "project" else 1.5e9):
            return None
        s = prepare(case, seed)
        if kind == "project":
            with torch.no_grad():
                return _exact_project_grad(case, s["volume"], s["geometry"], None, "")[0]
        return _exact_project_grad(case, s["volume"], s["geometry"], s["up"], case["want"])
    if voxel_views > (1.2e10 if kind == "fdk" else 1.5e9):
        return None
    s = prepare(case, seed)
    if kind == "fdk":
        with torch.no_grad():
            return _exact_fdk(case, s["measured"], s["geometry"])
    return _exact_layer(case, s["measured"], s["geometry"], s["up"], kind == "fdk_layer")
