"""Timing cases of the projector framework, through its public calls.

Each case is one call, or the few calls that a program makes together, on the
geometries of the configurations, tests and benchmark of this repository or on
odd sizes of the same kinds:

``pair``       fan beam DD forward projection, then the normalised back projection
``fp``         DD forward projection of a stack
``fbp``        filtered back projection: FP64 ramp filter, FBP-weighted DD back projection
``fbp_stock``  the fan beam's default calls: default ramp filter, pixel-driven back projection
``sqs``        one SQS-TV iteration: forward projection of the stored iterate, residual,
               back projection, fused TV update
``grad``       least-squares training step through the differentiable DD projectors
``cone_fp``, ``cone_bp``, ``cone_grad``   the Siddon cone pair, and its training step
``tomo``       the tomosynthesis pair
``host``       the host-array calls: forward projection, filter, back projection

Phantoms are sums of ellipses (ellipsoids); measured projections are their
analytic line integrals with Poisson noise, so inputs do not depend on the
code that is timed.  ``exact`` evaluates the same operators in 64 bits with
plain torch.
"""
import math

import numpy as np
import torch

from ctprojector_b200 import autograd as AG
from ctprojector_b200 import recon
from ctprojector_b200 import synthetic as S
from ctprojector_b200.projector.cupy import cone, fan_equiangular, parallel, tomo
from ctprojector_b200.projector.cupy.ct_projector import ct_projector
from ctprojector_b200.projector.numpy import parallel as host_parallel

DSD, DSO = 1085.6, 595.0
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}


# --------------------------------------------------------------------------- the cases
def listed():
    fan512 = dict(geom="fan", ny=512, nx=512, pixel=0.8, nview=984, nu=888, cell=1.2858)
    par512 = dict(geom="parallel", ny=512, nx=512, pixel=0.8, nview=720, nu=768, cell=0.8)
    cone64 = dict(nz=64, ny=512, nx=512, pixel=0.7, dz=1.0, nview=360, turns=1.0, nu=736, nv=64, cell=1.2858, row=1.0)
    return [
        # the smallest scan in use, one fan slice: launches and latency count
        dict(name="fan256_pair", op="pair", geom="fan", batch=1, ny=256, nx=256, pixel=1.0, nview=360, nu=736,
             cell=1.2858),
        # fan reconstruction with the default calls of the module
        dict(name="fan512x4_fbp_stock", op="fbp_stock", batch=4, **fan512),
        # the benchmark batch: forward projection, and filtered back projection
        dict(name="par512x16_fp", op="fp", batch=16, **par512),
        dict(name="par512x16_fbp", op="fbp", batch=16, **par512),
        # iterative reconstruction, image and sinogram stored in 16 bits
        dict(name="fan512x4_sqs_bf16", op="sqs", batch=4, storage="bfloat16", **fan512),
        # training steps through the differentiable projectors
        dict(name="fan512x2_grad", op="grad", batch=2, **fan512),
        dict(name="par_ragged_grad", op="grad", geom="parallel", batch=3, ny=317, nx=413, pixel=0.93, nview=501,
             nu=601, cell=0.87),
        # helical cone beam: one volume of the served protocol in each direction, and a small odd training step
        dict(name="cone64_fp", op="cone_fp", **cone64),
        dict(name="cone64_bp", op="cone_bp", **cone64),
        dict(name="cone_ragged_grad", op="cone_grad", nz=33, ny=187, nx=201, pixel=1.3, dz=1.1, nview=97, turns=1.0,
             nu=251, nv=37, cell=2.1, row=1.9),
        # tomosynthesis, forward and back
        dict(name="tomo64_pair", op="tomo", nz=64, ny=256, nx=512, pixel=0.4, dz=1.0, nview=25, arc=30.0, nu=1024,
             nv=512, cell=0.25),
        # the same reconstruction from and to host arrays
        dict(name="host_par512x4", op="host", batch=4, **par512),
    ]


def draw(rng):
    """One more case: an operation, then sizes over the range of its listed cases."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["pair", "fp", "fbp", "fbp_stock", "sqs", "grad", "cone_fp", "cone_bp", "cone_grad", "tomo", "host"])
    if op.startswith("cone"):
        nx, nz = log(96, 448), log(8, 64)
        ny = max(64, int(nx * rng.uniform(0.8, 1.2)))
        pixel = round(358.0 / max(nx, ny), 3)
        nu = int(nx * rng.uniform(1.0, 1.6))
        nv = max(4, int(nz * rng.uniform(0.7, 1.2)))
        nview = log(60, 360) if op != "cone_grad" else log(48, 160)
        return dict(op=op, nz=nz, ny=ny, nx=nx, pixel=pixel, dz=round(rng.uniform(0.8, 1.5), 2), nview=nview,
                    turns=rng.choice([1.0, 2.0]), nu=nu, nv=nv, cell=round(946.0 / nu, 3),
                    row=round(rng.uniform(1.0, 2.0), 2))
    if op == "tomo":
        nx, ny, nz = log(128, 512), log(96, 256), log(16, 64)
        cell = round(rng.uniform(0.2, 0.6), 3)
        return dict(op=op, nz=nz, ny=ny, nx=nx, pixel=0.4, dz=1.0, nview=rng.randint(9, 25),
                    arc=round(rng.uniform(20, 50), 1), nu=min(1024, int(nx * 0.5 / cell)),
                    nv=min(512, int(ny * 0.5 / cell)), cell=cell)
    geom = "fan" if op in ("pair", "fbp_stock") else "parallel" if op == "host" else rng.choice(["fan", "parallel"])
    nx = log(128, 512)
    ny = max(96, min(512, int(nx * rng.uniform(0.75, 1.25))))
    pixel = round(410.0 / max(nx, ny) * rng.uniform(0.6, 1.0), 3)
    nu = int(nx * rng.uniform(1.2, 1.75))
    cell = round((1.35 if geom == "parallel" else 2.6) * math.hypot(nx, ny) * pixel / 1.3 / nu, 4)
    case = dict(op=op, geom=geom, batch=log(1, 16) if op != "host" else log(1, 4), ny=ny, nx=nx, pixel=pixel,
                nview=log(90, 984 if geom == "fan" else 720), nu=nu, cell=cell)
    if op in ("grad", "sqs", "pair"):
        case["batch"] = min(case["batch"], 6)
    if op == "sqs":
        case["storage"] = rng.choice(sorted(DTYPES))
    return case


# --------------------------------------------------------------------------- geometry
def _scan(c):
    op = c["op"]
    if op.startswith("cone"):
        return S.Scan(c["nx"], c["ny"], c["nz"], c["pixel"], c["pixel"], c["dz"], c["nu"], c["nv"], c["cell"],
                      c["row"], c["nview"], dsd=DSD, dso=DSO)
    if op == "tomo":
        return S.Scan(c["nx"], c["ny"], c["nz"], c["pixel"], c["pixel"], c["dz"], c["nu"], c["nv"], c["cell"],
                      c["cell"], c["nview"])
    return S.Scan(c["nx"], c["ny"], 1, c["pixel"], c["pixel"], 1.0, c["nu"], 1, c["cell"], 1.0, c["nview"], dsd=DSD,
                  dso=DSO)


def _angles(c):
    """Views from half a step past 0, over the full circle (fan) or half (parallel)."""
    span = 2 * math.pi if c["geom"] == "fan" else math.pi
    return (S.angles(c["nview"], span) + np.float32(span / c["nview"] / 2)).astype(np.float32)


def _trajectory(c):
    """Rows (det_center, det_u, det_v, src) of the cone scan, or (det_center, src) of the tomosynthesis arc."""
    if c["op"] == "tomo":
        return S.tomo_geometry(c["nview"], c["arc"], 650.0, -(c["nz"] * c["dz"] / 2 + 20.0))
    return S.helical(c["nview"], c["turns"], DSO, DSD, c["nz"] * c["dz"] / c["turns"])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dev(a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device(), dtype=dtype)


def _f(x):
    return float(np.float32(x))


# --------------------------------------------------------------------------- inputs
N_SHAPES = 10


def _shapes(gen, n, size, height=1.0):
    """[n, N_SHAPES, 8] ellipsoids (x, y, z, a, b, c, phi, mu): a body of
    0.019 /mm and inserts of up to 0.011 /mm around it."""
    u = torch.rand((n, N_SHAPES, 8), generator=gen, device=gen.device, dtype=torch.float64)
    R = 0.45 * size
    r, t = 0.6 * R * torch.sqrt(u[..., 0]), 2 * math.pi * u[..., 1]
    s = torch.stack([r * torch.cos(t), r * torch.sin(t), (u[..., 2] - 0.5) * height, R * (0.04 + 0.21 * u[..., 3]),
                     R * (0.04 + 0.21 * u[..., 4]), height * (0.1 + 0.3 * u[..., 5]), math.pi * u[..., 6],
                     0.022 * (u[..., 7] - 0.5)], -1)
    s[:, 0, :3] = 0
    s[:, 0, 3:5] = R
    s[:, 0, 5] = 0.8 * height
    s[:, 0, 7] = 0.019
    return s


def _axis(n, d, dev):
    return (torch.arange(n, device=dev, dtype=torch.float64) + 0.5 - n / 2) * d


def _image(shapes, ny, nx, d, nz=None, dz=1.0):
    """Phantom sampled at the pixel centres: [n, 1, ny, nx], or [n, nz, ny, nx] for a volume."""
    dev = shapes.device
    y, x = _axis(ny, d, dev)[:, None], _axis(nx, d, dev)[None, :]
    z = torch.zeros(1, device=dev, dtype=torch.float64) if nz is None else _axis(nz, dz, dev)
    out = torch.zeros((shapes.shape[0], z.numel(), ny, nx), device=dev)
    for b in range(shapes.shape[0]):
        for x0, y0, z0, a, bb, cc, phi, mu in shapes[b].tolist():
            c, s = math.cos(phi), math.sin(phi)
            q = (((x - x0) * c + (y - y0) * s) / a) ** 2 + (((y - y0) * c - (x - x0) * s) / bb) ** 2
            h = ((z - z0) / cc) ** 2 if nz is not None else z
            out[b] += mu * (q[None] + h[:, None, None] <= 1)
    return out


def _integrals(shapes, src, end):
    """Line integrals of one phantom [N_SHAPES, 8] from src to the points of end ([..., 3], mm)."""
    d = end - src
    length = d.norm(dim=-1)
    out = torch.zeros_like(length)
    for x0, y0, z0, a, b, cc, phi, mu in shapes.tolist():
        c, s = math.cos(phi), math.sin(phi)
        o = src - torch.tensor([x0, y0, z0], device=d.device, dtype=d.dtype)

        def unit(v):
            return torch.stack([(v[..., 0] * c + v[..., 1] * s) / a, (v[..., 1] * c - v[..., 0] * s) / b,
                                v[..., 2] / cc], -1)

        p, q = unit(o), unit(d)
        qq, pq = (q * q).sum(-1), (p * q).sum(-1)
        disc = pq * pq - qq * ((p * p).sum(-1) - 1)
        out += mu * length * 2 * torch.sqrt(disc.clamp_min(0)) / qq
    return out


def _noisy(p, gen, photons=1e5):
    counts = torch.poisson((photons * torch.exp(-p.clamp_min(0))).float(), generator=gen)
    return -torch.log(counts.clamp_min(1) / photons)


def _sinogram(c, shapes, gen):
    """Measured fan or parallel projections of a stack of phantoms, [batch, nview, 1, nu]."""
    dev = shapes.device
    th = _dev(_angles(c)).double()[:, None]
    k = torch.arange(c["nu"], device=dev, dtype=torch.float64)[None, :]
    out = torch.empty((c["batch"], c["nview"], 1, c["nu"]), device=dev)
    for b in range(c["batch"]):
        if c["geom"] == "fan":
            a = -(k + 0.5 - c["nu"] / 2) * c["cell"] / DSD
            src = torch.stack([DSO * torch.sin(th), -DSO * torch.cos(th), 0 * th], -1)
            lx, ly = DSD * torch.sin(a), DSD * torch.cos(a) - DSO
        else:
            lx = -(k + 0.5 - c["nu"] / 2) * c["cell"] + 0 * th
            src = torch.stack([lx * torch.cos(th) + 1e3 * torch.sin(th), lx * torch.sin(th) - 1e3 * torch.cos(th),
                               0 * lx], -1)
            ly = 0 * lx + 1e3
        end = torch.stack([lx * torch.cos(th) - ly * torch.sin(th), lx * torch.sin(th) + ly * torch.cos(th),
                           0 * lx + 0 * th], -1)
        out[b, :, 0] = _noisy(_integrals(shapes[b], src, end), gen)
    return out


def _cell_points(c, geo, view):
    """Cell centres [nv, nu, 3] of one view of a cone or tomosynthesis scan."""
    dc = geo[0][view].double()
    eu = geo[1][view].double() if len(geo) == 4 else dc.new_tensor([1.0, 0, 0])
    ev = geo[2][view].double() if len(geo) == 4 else dc.new_tensor([0, 1.0, 0])
    row = c.get("row", c["cell"])
    u = (torch.arange(c["nu"], device=dc.device) - (c["nu"] - 1) / 2) * _f(c["cell"])
    v = (torch.arange(c["nv"], device=dc.device) - (c["nv"] - 1) / 2) * _f(row)
    return dc + u[None, :, None].double() * eu + v[:, None, None].double() * ev


def _projections(c, shapes, geo, gen):
    """Measured cone or tomosynthesis projections, [1, nview, nv, nu]."""
    out = torch.empty((1, c["nview"], c["nv"], c["nu"]), device=shapes.device)
    for view in range(c["nview"]):
        p = _integrals(shapes[0], geo[-1][view].double(), _cell_points(c, geo, view))
        out[0, view] = _noisy(p, gen)
    return out


def prepare(case, seed):
    c = case
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    p = _scan(c).projector(ct_projector)
    st = {"case": c, "p": p}
    if c["op"].startswith("cone") or c["op"] == "tomo":
        geo = [_dev(a) for a in _trajectory(c)]
        shapes = _shapes(gen, 1, min(c["nx"], c["ny"]) * c["pixel"], c["nz"] * c["dz"])
        st["geo"] = geo
        if c["op"] != "cone_bp":
            st["img"] = _image(shapes, c["ny"], c["nx"], c["pixel"], c["nz"], c["dz"])
        if c["op"] == "cone_grad":  # an early iterate against the measured projections
            st["img"] = 0.7 * st["img"] + 0.002 * torch.rand(st["img"].shape, generator=gen, device=dev)
        if c["op"] != "cone_fp":
            st["prj"] = _projections(c, shapes, geo, gen)
        return st
    shapes = _shapes(gen, c["batch"], min(c["nx"], c["ny"]) * c["pixel"])
    st["ang"] = _dev(_angles(c))
    if c["op"] in ("pair", "fp", "sqs", "grad", "host"):
        st["img"] = _image(shapes, c["ny"], c["nx"], c["pixel"])
    if c["op"] in ("fbp", "fbp_stock", "sqs", "grad"):
        st["prj"] = _sinogram(c, shapes, gen)
    if c["op"] in ("sqs", "grad"):
        st["img"] = 0.7 * st["img"] + 0.002 * torch.rand(st["img"].shape, generator=gen, device=dev)
    if c["op"] == "sqs":
        lp = DTYPES[c["storage"]]
        st["x_lp"] = st["img"].to(lp)
        st["prj"] = st["prj"].to(lp)
        st["norm"] = torch.full((1, c["ny"], c["nx"]), 0.8 * c["nview"] * c["nx"] * c["pixel"], device=dev)
        st["zlink"] = torch.zeros(c["batch"], dtype=torch.uint8, device=dev)
    if c["op"] == "host":
        st["img"] = st["img"].cpu().numpy()
        st["ang"] = _angles(c)
    return st


# --------------------------------------------------------------------------- one pass
def run(state):
    st, c, p = state, state["case"], state["p"]
    op = c["op"]
    if op == "cone_fp":
        return cone.siddon_fp_arbitrary(p, st["img"], *st["geo"])
    if op == "cone_bp":
        return cone.siddon_bp_arbitrary(p, st["prj"], *st["geo"])
    if op == "tomo":
        return (tomo.distance_driven_fp(p, st["img"], *st["geo"]), tomo.distance_driven_bp(p, st["prj"], *st["geo"]))
    if op in ("grad", "cone_grad"):
        x = st["img"].detach().requires_grad_(True)
        y = AG.siddon_fp(p, x, *st["geo"]) if op == "cone_grad" else AG.dd_fp(p, x, st["ang"], c["geom"])
        loss = 0.5 * ((y - st["prj"]) ** 2).sum()
        loss.backward()
        return {"loss": loss.detach(), "grad": x.grad}
    if op == "host":
        y = host_parallel.distance_driven_fp(p, st["img"], st["ang"])
        f = host_parallel.ramp_filter(p, y, "hann", exact=True)
        return y, f, host_parallel.distance_driven_bp(p, f, st["ang"], True)
    M = fan_equiangular if c["geom"] == "fan" else parallel
    if op == "fp":
        return M.distance_driven_fp(p, st["img"], st["ang"])
    if op == "pair":
        y = M.distance_driven_fp(p, st["img"], st["ang"])
        return y, M.distance_driven_bp(p, y, st["ang"])
    if op == "fbp":
        f = M.ramp_filter(p, st["prj"], "hann", exact=True)
        return f, M.distance_driven_bp(p, f, st["ang"], True)
    if op == "fbp_stock":
        f = M.ramp_filter(p, st["prj"], "hann")
        return f, M.fbp_bp(p, f, st["ang"])
    if op == "sqs":
        r = M.distance_driven_fp(p, st["x_lp"], st["ang"])
        r.sub_(st["prj"])
        bp = M.distance_driven_bp(p, r, st["ang"])
        x_lp = torch.empty_like(st["x_lp"]) if c["storage"] != "float32" else None
        x = recon.sqs_tv_update(st["img"], bp, st["norm"], 2e-4, (0.0, 1.0, 1.0), 1e-6, zlink=st["zlink"], x_lp=x_lp)
        return (x, bp) if x_lp is None else (x, bp, x_lp)
    raise ValueError(op)


# --------------------------------------------------------------------------- work and tolerance
def work(case):
    """Each input read once and each output written once; one multiply-add per
    ray and image line (DD), per pixel and view (back projections), or per
    voxel that a ray crosses (Siddon)."""
    c, op = case, case["op"]
    if op.startswith("cone"):
        vol, prj = c["nz"] * c["ny"] * c["nx"], c["nview"] * c["nv"] * c["nu"]
        crossed = 2.0 * prj * 0.8 * (c["nx"] + c["ny"]) / 2
        both = 2 if op == "cone_grad" else 1
        return {"bytes": 4 * both * (vol + prj), "flops": both * crossed}
    if op == "tomo":
        vol, prj = c["nz"] * c["ny"] * c["nx"], c["nview"] * c["nv"] * c["nu"]
        return {"bytes": 8 * (vol + prj), "flops": 2.0 * (prj * c["nz"] + vol * c["nview"])}
    img, prj = c["batch"] * c["ny"] * c["nx"], c["batch"] * c["nview"] * c["nu"]
    fp, bp = 2.0 * prj * (c["nx"] + c["ny"]) / 2, 2.0 * img * c["nview"]
    filt = 2.0 * prj * 2.5 * 2 * math.log2(2 * c["nu"])
    e = 2 if c.get("storage", "float32") != "float32" else 4
    return {"fp": {"bytes": 4 * (img + prj), "flops": fp},
            "pair": {"bytes": 8 * img + 4 * prj, "flops": fp + bp},
            "fbp": {"bytes": 4 * (img + 2 * prj), "flops": bp + filt},
            "fbp_stock": {"bytes": 4 * (img + 2 * prj), "flops": bp + filt},
            "sqs": {"bytes": 2 * e * img + 12 * img + e * prj, "flops": fp + bp},
            "grad": {"bytes": 8 * img + 8 * prj, "flops": fp + bp},
            "host": {"bytes": 8 * img + 8 * prj, "flops": fp + bp + filt}}[op]


def tolerance(case):
    """32-bit sums.  The pixel-driven and filtered reconstructions add filtered
    views that largely cancel, and the default filter is built in 32 bits."""
    if case["op"] == "fbp_stock":
        return {"rel": 2e-4, "max": 8e-3}
    if case["op"] in ("fbp", "host"):
        return {"rel": 3e-5, "max": 2e-3}
    if case["op"] == "sqs" and case["storage"] != "float32":  # a 16-bit copy of the iterate rounds on
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 1e-5, "max": 1e-3}


# --------------------------------------------------------------------------- 64-bit evaluation
def _interp(C, x):
    """C: running sums [..., n+1] of cells; the integral up to the positions x ([m], clamped to [0, n])."""
    n = C.shape[-1] - 1
    x = x.clamp(0, n)
    i = x.floor().clamp(max=n - 1).long()
    f = x - i
    return C[..., i] * (1 - f) + C[..., i + 1] * f


def _running(a):
    return torch.nn.functional.pad(a.cumsum(-1), (1, 0))


def _params(c):
    """(pixel, cell, dso) as the 32-bit values the calls pass on."""
    cell = _f(np.float32(c["cell"] / DSD)) if c["geom"] == "fan" else _f(c["cell"])
    return _f(c["pixel"]), cell, _f(DSO)


def _blend(th):
    return min(1.0, max(0.0, (abs(math.cos(th)) - abs(math.sin(th)) + 0.12) / 0.24))


def _dd_fp_view(c, rows, cols, th):
    """Forward projection [batch, nu] of one view from the running sums of the image's rows and columns."""
    d, cell, dso = _params(c)
    nx, ny, nu = c["nx"], c["ny"], c["nu"]
    dev = rows.device
    j = torch.arange(nu + 1, device=dev, dtype=torch.float64)
    e = -(j - nu / 2) * cell
    s, co = math.sin(th), math.cos(th)
    if c["geom"] == "fan":
        sx, sy = dso * s + 0 * e, -dso * co + 0 * e
        lx, ly = _f(DSD) * torch.sin(e), _f(DSD) * torch.cos(e) - dso
        ex, ey = lx * co - ly * s, lx * s + ly * co
        a = -(j[:-1] - (nu - 1) / 2) * cell
    else:
        r = (nx + ny) * d
        sx, sy, ex, ey = e * co + r * s, e * s - r * co, e * co - r * s, e * s + r * co
        a = 0 * j[:-1]
    sx, ex, sy, ey = sx / d + nx / 2, ex / d + nx / 2, sy / d + ny / 2, ey / d + ny / 2
    out = 0.0
    for w, C, (p0, q0, p1, q1), length in ((_blend(th), rows, (sx, sy, ex, ey), d / torch.cos(th - a).abs()),
                                          (1 - _blend(th), cols, (sy, sx, ey, ex), d / torch.sin(th - a).abs())):
        if w == 0:
            continue
        nl, n = C.shape[1], C.shape[2] - 1
        t = torch.arange(nl, device=dev, dtype=torch.float64)[:, None] + 0.5
        x = p0 + (p1 - p0) / (q1 - q0) * (t - q0)  # [nl, nu+1]
        xc = x.clamp(0, n)
        i = xc.floor().clamp(max=n - 1).long()
        f = xc - i
        at = (torch.arange(nl, device=dev)[:, None] * (n + 1) + i).reshape(-1)
        flat = C.reshape(C.shape[0], -1)
        F = (flat[:, at] * (1 - f.reshape(-1)) + flat[:, at + 1] * f.reshape(-1)).reshape(C.shape[0], nl, nu + 1)
        out = out + w * length * ((F[..., 1:] - F[..., :-1]) / (x[:, 1:] - x[:, :-1])).sum(1)
    return out


def _dd_fp(c, img):
    """[batch, nview, 1, nu] in 64 bits; img [batch, 1, ny, nx]."""
    x = img.double()[:, 0]
    rows, cols = _running(x), _running(x.transpose(1, 2))
    return torch.stack([_dd_fp_view(c, rows, cols, float(th)) for th in _angles(c)], 1)[:, :, None]


def _dd_adjoint(c, prj):
    """Transpose of _dd_fp: [batch, 1, ny, nx]."""
    out = 0.0
    for v, th in enumerate(_angles(c)):
        x = torch.zeros((prj.shape[0], c["ny"], c["nx"]), device=prj.device, dtype=torch.float64, requires_grad=True)
        y = _dd_fp_view(c, _running(x), _running(x.transpose(1, 2)), float(th))
        out = out + torch.autograd.grad(y, x, prj[:, v, 0].double())[0]
    return out[:, None]


def _dd_bp(c, prj, is_fbp):
    """Normalised back projection: mean of the detector row over the pixel's footprint, per view."""
    d, cell, dso = _params(c)
    nx, ny, nu = c["nx"], c["ny"], c["nu"]
    dev = prj.device
    y = prj[:, :, 0].double()
    xc, yc = _axis(nx, d, dev), _axis(ny, d, dev)
    xe = torch.cat([xc - d / 2, xc[-1:] + d / 2])
    ye = torch.cat([yc - d / 2, yc[-1:] + d / 2])
    k = torch.arange(nu, device=dev, dtype=torch.float64)
    out = torch.zeros((prj.shape[0], ny, nx), device=dev, dtype=torch.float64)
    for v, th in enumerate(_angles(c)):
        th = float(th)
        s, co = math.sin(th), math.cos(th)
        y_main = abs(co) > abs(s)
        fan = c["geom"] == "fan"

        def at(x, yy):
            a = torch.atan((x * co + yy * s) / (yy * co - x * s + dso)) if fan else x * co + yy * s
            return -a / cell + nu / 2

        row = y[:, v]
        if fan and not is_fbp:
            a = -(k - (nu - 1) / 2) * cell
            row = row * (d / (torch.cos(th - a) if y_main else torch.sin(th - a)).abs())
        C = _running(row)
        wx = (1.0 if y_main else 0.0) if fan else _blend(th)
        val = 0.0
        if wx > 0:
            j = at(xe[None, :], yc[:, None])
            F = _interp(C, j.reshape(-1)).reshape(-1, ny, nx + 1)
            val = val + wx * (F[..., 1:] - F[..., :-1]) / (j[:, 1:] - j[:, :-1])
        if wx < 1:
            j = at(xc[None, :], ye[:, None])
            F = _interp(C, j.reshape(-1)).reshape(-1, ny + 1, nx)
            val = val + (1 - wx) * (F[:, 1:] - F[:, :-1]) / (j[1:] - j[:-1])
        if fan and is_fbp:
            rx, ry = xc[None, :] * co + yc[:, None] * s, yc[:, None] * co - xc[None, :] * s
            val = val * (dso * dso / (rx * rx + (dso + ry) ** 2))
        if not fan and not is_fbp:
            val = val * (d / abs(co) if y_main else d / abs(s))
        out += val
    return out[:, None]


def _ramp(c, prj):
    """Hann-windowed ramp filter: convolution with the windowed kernel of length 2 nu - 1."""
    _, cell, dso = _params(c)
    fan, nu = c["geom"] == "fan", c["nu"]
    L = 2 * nu - 1
    k = torch.arange(L, dtype=torch.float64, device=prj.device) - (nu - 1)
    odd = (k.abs() % 2) == 1
    den = torch.where(odd, torch.sin(k * cell) if fan else k * cell, torch.ones_like(k))
    h = torch.where(odd, -1 / (math.pi * den) ** 2, torch.zeros_like(k))
    h[nu - 1] = 1 / (4 * cell * cell)
    w = 0.5 + 0.5 * torch.cos(2 * math.pi * torch.arange(L, device=prj.device, dtype=torch.float64) / L)
    g = torch.fft.ifft(torch.fft.fft(h) * w).real
    x = prj.double()
    if fan:
        x = x * torch.cos((torch.arange(nu, device=prj.device) - (nu - 1) / 2) * cell)
    n = 2 * L
    y = torch.fft.irfft(torch.fft.rfft(x, n) * torch.fft.rfft(g, n), n)[..., nu - 1:2 * nu - 1]
    return y * (math.pi / c["nview"] * cell / (dso if fan else 1.0))


def _pixel_bp(c, prj):
    """Pixel-driven fan back projection with the FBP distance weight."""
    d, cell, dso = _params(c)
    nx, ny, nu = c["nx"], c["ny"], c["nu"]
    x, y = _axis(nx, d, prj.device)[None, :], _axis(ny, d, prj.device)[:, None]
    out = torch.zeros((prj.shape[0], ny, nx), device=prj.device, dtype=torch.float64)
    for v, th in enumerate(_angles(c)):
        s, co = math.sin(float(th)), math.cos(float(th))
        rx, ry = x * co + y * s, y * co - x * s
        pu = -torch.atan(rx / (ry + dso)) / cell + (nu - 1) / 2
        i = pu.floor().clamp(0, nu - 1).long()
        f = pu - i
        row = prj[:, v, 0].double()
        val = row[:, i.reshape(-1)] * (1 - f).reshape(-1) + row[:, (i + 1).clamp(max=nu - 1).reshape(-1)] * f.reshape(-1)
        wgt = ((pu >= 0) & (pu < nu)) * dso * dso / (rx * rx + (dso + ry) ** 2)
        out += val.reshape(-1, ny, nx) * wgt
    return out[:, None]


def _tv_update(c, x, bp, norm, beta, eps):
    """x - (bp + beta s1) / (norm + beta s2), the TV terms of the x and y differences."""
    x = x.double()
    dx, dy = torch.zeros_like(x), torch.zeros_like(x)
    dx[..., 1:] = x[..., 1:] - x[..., :-1]
    dy[..., 1:, :] = x[..., 1:, :] - x[..., :-1, :]
    var = torch.sqrt(dx * dx + dy * dy + eps)
    vx, vy = var.clone(), var.clone()
    vx[..., :-1] = var[..., 1:]
    vy[..., :-1, :] = var[..., 1:, :]
    fx, fy = torch.zeros_like(x), torch.zeros_like(x)
    fx[..., :-1] = -dx[..., 1:]
    fy[..., :-1, :] = -dy[..., 1:, :]
    s1 = (dx + dy) / var + fx / vx + fy / vy
    s2 = 2 / var + 1 / vx + 1 / vy
    return x - (bp + beta * s1) / (norm.double() + beta * s2)


def _cone_segments(c, geo, view):
    """Voxel indices and lengths of the rays of one view, slab by slab of each
    ray's main axis (x or y): per slab a ray meets at most one plane of each
    other axis, so it crosses up to three voxels.  Yields (rays, index, length)
    with rays the flat detector cells."""
    n = (c["nx"], c["ny"], c["nz"])
    sp = torch.tensor([_f(c["pixel"]), _f(c["pixel"]), _f(c["dz"])], device=geo[0].device, dtype=torch.float64)
    half = torch.tensor(n, device=sp.device, dtype=torch.float64) / 2
    end = _cell_points(c, geo, view).reshape(-1, 3)
    src = geo[3][view].double()
    length = (end - src).norm(dim=-1)
    a, b = src / sp + half, end / sp + half
    dirs = b - a
    main_x = dirs[:, 0].abs() >= dirs[:, 1].abs()
    stride = (1, n[0], n[0] * n[1])
    for m, o in ((0, 1), (1, 0)):
        rays = torch.nonzero(main_x if m == 0 else ~main_x)[:, 0]
        if rays.numel() == 0:
            continue
        dr = dirs[rays]
        i = torch.arange(n[m], device=sp.device, dtype=torch.float64)[None, :]
        t0, t1 = (i - a[m]) / dr[:, m:m + 1], (i + 1 - a[m]) / dr[:, m:m + 1]
        cuts = [t0]
        for k in (o, 2):
            p0, p1 = a[k] + t0 * dr[:, k:k + 1], a[k] + t1 * dr[:, k:k + 1]
            lo, hi = torch.minimum(p0, p1), torch.maximum(p0, p1)
            plane = lo.floor() + 1
            crosses = (plane < hi) & (dr[:, k:k + 1] != 0)
            cuts.append(torch.where(crosses, (plane - a[k]) / dr[:, k:k + 1], t1))
        same = torch.sign(dr[:, m:m + 1])
        lo2, hi2 = torch.minimum(cuts[1] * same, cuts[2] * same) * same, torch.maximum(cuts[1] * same, cuts[2] * same) * same
        cuts = [t0, lo2, hi2, t1]
        for s0, s1 in zip(cuts[:-1], cuts[1:]):
            mid = 0.5 * (s0 + s1)
            jo = (a[o] + mid * dr[:, o:o + 1]).floor()
            jz = (a[2] + mid * dr[:, 2:3]).floor()
            inside = (jo >= 0) & (jo < n[o]) & (jz >= 0) & (jz < n[2])
            idx = (i * stride[m] + jo.clamp(0, n[o] - 1) * stride[o] + jz.clamp(0, n[2] - 1) * stride[2]).long()
            yield rays, idx, (s1 - s0).abs() * length[rays][:, None] * inside


def _cone_fp(c, img, geo):
    vol = img.double().reshape(-1)
    out = torch.zeros((c["nview"], c["nv"] * c["nu"]), device=img.device, dtype=torch.float64)
    for v in range(c["nview"]):
        for rays, idx, length in _cone_segments(c, geo, v):
            out[v, rays] += (vol[idx] * length).sum(1)
    return out.reshape(1, c["nview"], c["nv"], c["nu"])


def _cone_bp(c, prj, geo):
    out = torch.zeros(c["nz"] * c["ny"] * c["nx"], device=prj.device, dtype=torch.float64)
    for v in range(c["nview"]):
        y = prj[0, v].double().reshape(-1)
        for rays, idx, length in _cone_segments(c, geo, v):
            out.index_add_(0, idx.reshape(-1), (y[rays][:, None] * length).reshape(-1))
    return out.reshape(1, c["nz"], c["ny"], c["nx"])


def _box2d(plane, x, y):
    """Mean of plane [ny, nx] over the rectangles between the edges y and x (both monotonic)."""
    C = _running(_running(plane).transpose(0, 1)).transpose(0, 1)
    B = _interp(_interp(C, x).transpose(0, 1), y).transpose(0, 1)
    box = B[1:, 1:] - B[:-1, 1:] - B[1:, :-1] + B[:-1, :-1]
    return box / ((x[1:] - x[:-1]) * (y[1:] - y[:-1])[:, None])


def _tomo(c, img, prj, geo):
    """(forward projection of img, back projection of prj)."""
    dev = img.device
    d, dz, cell = _f(c["pixel"]), _f(c["dz"]), _f(c["cell"])
    nu, nv, nx, ny, nz = c["nu"], c["nv"], c["nx"], c["ny"], c["nz"]
    ue = (torch.arange(nu + 1, device=dev, dtype=torch.float64) - nu / 2) * cell
    ve = (torch.arange(nv + 1, device=dev, dtype=torch.float64) - nv / 2) * cell
    xe = (torch.arange(nx + 1, device=dev, dtype=torch.float64) - nx / 2) * d
    ye = (torch.arange(ny + 1, device=dev, dtype=torch.float64) - ny / 2) * d
    z = _axis(nz, dz, dev).tolist()
    fp = torch.zeros((1, c["nview"], nv, nu), device=dev, dtype=torch.float64)
    bp = torch.zeros((1, nz, ny, nx), device=dev, dtype=torch.float64)
    vol = img.double()[0]
    for v in range(c["nview"]):
        (cx, cy, cz), (sx, sy, sz) = geo[0][v].double().tolist(), geo[1][v].double().tolist()
        pts = _cell_points(c, geo, v)
        w = dz / abs(sz - cz) * (pts - geo[1][v].double()).norm(dim=-1)
        y = prj[0, v].double() * w
        for k in range(nz):
            # the cell edges in plane z[k], then the pixel edges on the detector
            r = (z[k] - sz) / (cz - sz)
            # the forward footprints lie where the image's centre planes do
            x_at = (sx + (cx + ue - sx) * ((k - (sz / dz + 0.5 * nz)) / (cz / dz - sz / dz))) / d + nx / 2
            y_at = (sy + (cy + ve - sy) * ((k - (sz / dz + 0.5 * nz)) / (cz / dz - sz / dz))) / d + ny / 2
            fp[0, v] += _box2d(vol[k], x_at, y_at)
            u_at = (sx - cx + (xe - sx) / r) / cell + (nu - 1) / 2
            v_at = (sy - cy + (ye - sy) / r) / cell + (nv - 1) / 2
            bp[0, k] += _box2d(y, u_at, v_at)
        fp[0, v] *= w
    return fp, bp


def exact(case, seed):
    c, st = case, prepare(case, seed)
    op = c["op"]
    if op == "cone_fp":
        return _cone_fp(c, st["img"], st["geo"])
    if op == "cone_bp":
        return _cone_bp(c, st["prj"], st["geo"])
    if op == "tomo":
        return _tomo(c, st["img"], st["prj"], st["geo"])
    if op in ("grad", "cone_grad"):
        y = _cone_fp(c, st["img"], st["geo"]) if op == "cone_grad" else _dd_fp(c, st["img"])
        r = y - st["prj"].double()
        g = _cone_bp(c, r, st["geo"]) if op == "cone_grad" else _dd_adjoint(c, r)
        return {"loss": 0.5 * (r ** 2).sum(), "grad": g}
    if op == "host":
        y = _dd_fp(c, _dev(st["img"]))
        f = _ramp(c, y)
        return tuple(t.cpu().numpy() for t in (y, f, _dd_bp(c, f, True)))
    if op == "fp":
        return _dd_fp(c, st["img"])
    if op == "pair":
        y = _dd_fp(c, st["img"])
        return y, _dd_bp(c, y, False)
    if op == "fbp":
        f = _ramp(c, st["prj"])
        return f, _dd_bp(c, f, True)
    if op == "fbp_stock":
        f = _ramp(c, st["prj"])
        return f, _pixel_bp(c, f)
    bp = _dd_bp(c, _dd_fp(c, st["x_lp"]) - st["prj"].double(), False)
    x = _tv_update(c, st["img"], bp, st["norm"], 2e-4, 1e-6)
    return (x, bp) if c["storage"] == "float32" else (x, bp, None)
