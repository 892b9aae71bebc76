"""Performance cases: the work a user has the cone-beam package do.

Every case is a dict of plain values with a ``kind``:

* ``operator``  - one forward projection, one backprojection, or both,
  through ``XrayTransform`` (frames in one array) or
  ``ForwardProjector``/``BackProjector`` (one array per frame);
* ``fdk``       - a whole ``kk.fdk`` call, from host or device projections
  to a host volume;
* ``sirt``      - a whole SIRT solve, ``kk.sirt`` (float32, host to host) or
  ``kk.SIRT`` with 16-bit storage;
* ``batch``     - a whole ``BatchedSIRT`` solve of several uneven problems;
* ``gradient``  - one step of a differentiable reconstruction: projection,
  squared-error loss and its backward pass through the exact adjoint.

Scans are circular with a flat detector at twice the source-object
distance, volumes hold random ellipsoids with a little noise, and measured
projections are the ellipsoids' line integrals with Poisson noise.
``exact`` evaluates the same operations in float64 with plain torch: Joseph
rays (one bilinear sample per slice of the dominant axis), voxel-driven
backprojection and the float64 row filter.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(
    os.path.abspath(__file__))), "astra-kernelkit_b200"))

import kernelkit as kk  # noqa: E402
from kernelkit.batch import BatchedSIRT  # noqa: E402
from kernelkit.projector import BackProjector, ForwardProjector  # noqa: E402
from kernelkit.torch_support import ExactXrayForwardProjection  # noqa: E402

#: float64 samples that ``exact`` evaluates at most (about ten seconds)
EXACT_SAMPLES = 4e10
PITCH = 1.3


def _scan(nx, ny, nz, angles, rows, cols, sod, pitch=PITCH, tilt=0.0):
    return dict(nx=nx, ny=ny, nz=nz, angles=angles, rows=rows, cols=cols,
                sod=float(sod), pitch=float(pitch), tilt=float(tilt))


def listed():
    return [
        # the smallest call: a 64^3 volume, where launches and host work
        # count (interactive previews, unit-sized problems)
        dict(name="small_pair", kind="operator", direction="both",
             interpolation="texture", frames="array",
             **_scan(64, 64, 64, 96, 96, 96, 200, 1.5)),
        # an ordinary scan with odd, uneven extents
        dict(name="ragged_pair", kind="operator", direction="both",
             interpolation="texture", frames="array",
             **_scan(251, 233, 190, 333, 289, 367, 790)),
        # the largest scan, each direction by itself: 512^3 voxels, 720
        # angles, 768^2 detector
        dict(name="large_forward", kind="operator", direction="forward",
             interpolation="texture", frames="array",
             **_scan(512, 512, 512, 720, 768, 768, 1600)),
        dict(name="large_back", kind="operator", direction="back",
             interpolation="texture", frames="array",
             **_scan(512, 512, 512, 720, 768, 768, 1600)),
        # exact interpolation weights instead of the texture unit's
        dict(name="exact_weights", kind="operator", direction="both",
             interpolation="exact", frames="array",
             **_scan(160, 160, 160, 240, 240, 240, 500)),
        # a scan with a calibrated (slightly rotated) detector whose frames
        # arrive one array each
        dict(name="tilted_frames", kind="operator", direction="both",
             interpolation="texture", frames="list",
             **_scan(192, 192, 160, 300, 250, 288, 600, tilt=0.6)),
        # filtered backprojection from host memory, the usual first look at
        # a scan, and from projections that are on the device already
        dict(name="fdk_host", kind="fdk", source="host",
             **_scan(256, 256, 256, 360, 384, 384, 800)),
        dict(name="fdk_device", kind="fdk", source="device",
             **_scan(405, 405, 330, 501, 512, 620, 1200)),
        # iterative reconstruction: float32 from host memory with a lower
        # bound, and 16-bit storage of the same kind of scan at 256^3
        dict(name="sirt_host", kind="sirt", storage="float32", iters=20,
             **_scan(128, 128, 100, 180, 150, 192, 400)),
        dict(name="sirt_16bit", kind="sirt", storage="16bit", iters=10,
             **_scan(256, 256, 256, 360, 384, 384, 800)),
        # many small uneven problems solved together
        dict(name="batch_uneven", kind="batch", problems=8, iters=10,
             smallest=64, largest=192),
        # one step of a differentiable reconstruction at 256^3
        dict(name="gradient_step", kind="gradient",
             **_scan(256, 256, 256, 360, 384, 384, 800)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scan(rng, lo, hi, tilt=0.0):
    n = _log(rng, lo, hi)
    nx = max(16, int(n * rng.uniform(0.9, 1.1)))
    nz = max(16, int(n * rng.uniform(0.7, 1.1)))
    nx, ny, nz = min(nx, hi), min(n, hi), min(nz, hi)
    m = max(nx, ny)
    return _scan(nx, ny, nz, max(24, int(1.4 * m * rng.uniform(0.7, 1.0))),
                 int(1.5 * nz * rng.uniform(0.9, 1.0)),
                 int(1.5 * m * rng.uniform(0.9, 1.0)),
                 m * rng.uniform(2.5, 4.0), tilt=tilt)


def draw(rng: random.Random):
    kind = rng.choice(["operator", "operator", "operator", "fdk", "sirt",
                       "batch", "gradient"])
    if kind == "operator":
        form = rng.choice(["plain", "plain", "plain", "exact", "tilted"])
        if form == "exact":
            return dict(kind=kind, direction="both", interpolation="exact",
                        frames="array", **_draw_scan(rng, 48, 200))
        if form == "tilted":
            return dict(kind=kind, direction="both", interpolation="texture",
                        frames="list", **_draw_scan(
                            rng, 48, 224, tilt=rng.uniform(0.2, 1.0)))
        return dict(kind=kind, interpolation="texture", frames="array",
                    direction=rng.choice(["both", "forward", "back"]),
                    **_draw_scan(rng, 48, 400))
    if kind == "fdk":
        return dict(kind=kind, source=rng.choice(["host", "device"]),
                    **_draw_scan(rng, 96, 400))
    if kind == "sirt":
        return dict(kind=kind, storage=rng.choice(["float32", "16bit"]),
                    iters=rng.randint(8, 20), **_draw_scan(rng, 64, 224))
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 10),
                    iters=rng.randint(5, 10), smallest=48 + rng.randint(0, 24),
                    largest=160 + rng.randint(0, 32))
    return dict(kind=kind, **_draw_scan(rng, 48, 224))


# ---------------------------------------------------------------------------
# geometry, objects and measurements
# ---------------------------------------------------------------------------
def _vectors(c):
    """float64 source, detector centre, u and v (unit vectors) per angle."""
    n = c["angles"]
    th = 2.0 * np.pi * np.arange(n) / n
    cs, sn, z = np.cos(th), np.sin(th), np.zeros(n)
    src = c["sod"] * np.stack([-cs, -sn, z], 1)
    det = -src
    u, v = np.array([0.0, 1.0, 0.0]), np.array([0.0, 0.0, 1.0])
    if c["tilt"]:
        # in-plane rotation of the panel, half of it out of plane, and an
        # off-centre position: what a geometric calibration finds
        a, b = math.radians(c["tilt"]), math.radians(0.5 * c["tilt"])
        roll = np.array([[1, 0, 0], [0, math.cos(a), -math.sin(a)],
                         [0, math.sin(a), math.cos(a)]])
        pitch = np.array([[math.cos(b), 0, math.sin(b)], [0, 1, 0],
                          [-math.sin(b), 0, math.cos(b)]])
        u, v = pitch @ roll @ u, pitch @ roll @ v
        det = det + np.stack([-sn, cs, z], 1) * 1.7 + np.array([0, 0, -0.9])
    rot = np.stack([np.stack([cs, -sn, z], 1), np.stack([sn, cs, z], 1),
                    np.stack([z, z, z + 1.0], 1)], 1)
    return src, det, rot @ u, rot @ v


def _geometry(c):
    d = kk.Detector(rows=c["rows"], cols=c["cols"], pixel_height=c["pitch"],
                    pixel_width=c["pitch"])
    pgs = [kk.ProjectionGeometry(s, p, d, u=u, v=v)
           for s, p, u, v in zip(*_vectors(c))]
    return pgs, kk.resolve_volume_geometry(
        shape=(c["nx"], c["ny"], c["nz"]), voxel_size=1.0)


def _ellipsoids(c, seed, k=12):
    rng = np.random.default_rng(seed)
    n = np.array([c["nx"], c["ny"], c["nz"]], np.float64)
    q, _ = np.linalg.qr(rng.normal(size=(k, 3, 3)))
    return (rng.uniform(-0.25, 0.25, (k, 3)) * n,
            rng.uniform(0.05, 0.22, (k, 3)) * n.min(), q,
            rng.uniform(0.1, 1.0, k))


def _volume(c, seed):
    """Voxelised ellipsoids with a little noise, on the GPU."""
    centres, semi, rot, dens = _ellipsoids(c, seed)
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) - n / 2 + 0.5
          for n in (c["nx"], c["ny"], c["nz"])]
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    vol = 0.01 * torch.randn((c["nx"], c["ny"], c["nz"]), generator=gen,
                             device="cuda")
    for e in range(len(dens)):
        m = (rot[e] / semi[e][:, None]).astype(np.float32)
        r2 = 0.0
        for j in range(3):
            p = [float(m[j, i]) * (ax[i] - float(centres[e][i]))
                 for i in range(3)]
            r2 = r2 + (p[0][:, None, None] + p[1][None, :, None]
                       + p[2][None, None, :]).square_()
        vol.add_((r2 <= 1.0).float(), alpha=float(dens[e]))
    return vol


def _pixels(c, k):
    """float64 source and pixel centres (rows, cols, 3) of angle ``k``."""
    src, det, u, v = (torch.as_tensor(x[k], device="cuda")
                      for x in _vectors(c))
    r = (torch.arange(c["rows"], device="cuda", dtype=torch.float64) + 0.5
         - c["rows"] / 2) * c["pitch"]
    q = (torch.arange(c["cols"], device="cuda", dtype=torch.float64) + 0.5
         - c["cols"] / 2) * c["pitch"]
    return src, (det + r[:, None, None] * v + q[None, :, None] * u)


def _measured(c, seed):
    """Line integrals with Poisson noise at 1e5 photons, float32, GPU."""
    centres, semi, rot, dens = _ellipsoids(c, seed)
    dev = dict(device="cuda", dtype=torch.float32)
    out = torch.zeros((c["angles"], c["rows"], c["cols"]), **dev)
    vec = [torch.as_tensor(x, **dev) for x in _vectors(c)]
    r = (torch.arange(c["rows"], **dev) + 0.5 - c["rows"] / 2) * c["pitch"]
    q = (torch.arange(c["cols"], **dev) + 0.5 - c["cols"] / 2) * c["pitch"]
    step = max(1, (1 << 23) // (c["rows"] * c["cols"]))
    for a in range(0, c["angles"], step):
        src, det, u, v = (x[a:a + step] for x in vec)
        d = (det - src)[:, None, None, :] + r[:, None, None] * v[
            :, None, None, :] + q[:, None] * u[:, None, None, :]
        d /= d.norm(dim=-1, keepdim=True)
        for e in range(len(dens)):
            m = torch.as_tensor(rot[e] / semi[e][:, None], **dev)
            w = d @ m.T
            q0 = (src - torch.as_tensor(centres[e], **dev)) @ m.T
            ww = w.square().sum(-1)
            qw = (w @ q0[:, None, :, None])[..., 0]
            qq = q0.square().sum(-1)[:, None, None] - 1.0
            disc = (qw.square() - ww * qq).clamp_(min=0.0)
            out[a:a + step] += float(dens[e]) * 2.0 * disc.sqrt_() / ww
    k = 3.0 / out.max().clamp(min=1e-6)
    gen = torch.Generator(device="cuda").manual_seed(seed + 2)
    for a in range(0, c["angles"], step):
        counts = torch.poisson(1e5 * torch.exp(-k * out[a:a + step]),
                               generator=gen).clamp_(min=1.0)
        out[a:a + step] = -torch.log(counts / 1e5) / k
    return out


def _problems(c, seed):
    """Scans of a batch: edges, angles and distances as drawn per problem
    (the same for every seed, so that seeds change the data alone)."""
    rng = np.random.default_rng(1000 * c["problems"] + c["smallest"]
                                + c["largest"])
    edges = np.linspace(c["smallest"], c["largest"], 5).astype(int)
    out = []
    for _ in range(c["problems"]):
        n = int(rng.choice(edges))
        out.append(_scan(n, n, n, int(rng.integers(60, 361)), 3 * n // 2,
                         3 * n // 2, max(2.0 * n, rng.uniform(150, 1000))))
    return out


# ---------------------------------------------------------------------------
# states and passes
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return dict(kind=kind, case=case, problems=[
            (_measured(p, seed + 17 * i), *_geometry(p))
            for i, p in enumerate(_problems(case, seed))])
    pgs, vg = _geometry(case)
    s = dict(kind=kind, case=case, pgs=pgs, vg=vg)
    if kind == "operator":
        forward = case["direction"] in ("forward", "both")
        back = case["direction"] in ("back", "both")
        kw = dict(interpolation=case["interpolation"])
        if forward:
            s["x"] = _volume(case, seed)
        if back:
            s["y"] = _measured(case, seed)
        if case["frames"] == "list":
            s["fp"], s["bp"] = ForwardProjector(**kw), BackProjector(**kw)
            for p in (s["fp"], s["bp"]):
                p.volume_geometry, p.projection_geometry = vg, pgs
            s["y"] = [f.clone() for f in s["y"]]
            s["out"] = [torch.empty_like(f) for f in s["y"]]
            s["out_x"] = torch.empty_like(s["x"])
        else:
            s["op"] = kk.XrayTransform(pgs, vg, fp_kwargs=kw, bp_kwargs=kw)
    elif kind == "fdk":
        y = _measured(case, seed)
        s["y"] = y.cpu().numpy() if case["source"] == "host" else y
    elif kind == "sirt":
        y = _measured(case, seed)
        s["y"] = y.cpu().numpy() if case["storage"] == "float32" else y
    else:
        s["x"] = 0.5 * _volume(case, seed)[None, None]
        s["y"] = _measured(case, seed)[None, None]
        s["module"] = ExactXrayForwardProjection(pgs, vg)
    return s


def run(s):
    c = s["case"]
    if s["kind"] == "operator":
        if c["frames"] == "list":
            s["fp"].volume, s["fp"].projections = s["x"], s["out"]
            s["fp"]()
            s["bp"].projections, s["bp"].volume = s["y"], s["out_x"]
            s["bp"]()
            return {"projections": torch.stack(s["out"]),
                    "volume": s["out_x"]}
        out = {}
        if "x" in s:
            out["projections"] = s["op"](s["x"])
        if "y" in s:
            out["volume"] = s["op"].T(s["y"])
        return out
    if s["kind"] == "fdk":
        # device projections are filtered in place, so the program that
        # keeps its measurement passes a copy
        y = s["y"] if c["source"] == "host" else s["y"].clone()
        return {"volume": kk.fdk(y, s["pgs"], s["vg"])}
    if s["kind"] == "sirt":
        if c["storage"] == "float32":
            return {"volume": kk.sirt(s["y"], s["pgs"], s["vg"],
                                      iters=c["iters"], verbose=False,
                                      min_constraint=0.0)}
        solver = kk.SIRT(s["y"], s["pgs"], s["vg"],
                         volume_dtype=torch.bfloat16,
                         projection_dtype=torch.float16)
        return {"volume": solver.run(c["iters"])}
    if s["kind"] == "batch":
        solver = BatchedSIRT(s["problems"], min_constraint=0.0)
        return {"volumes": list(solver.run(c["iters"]))}
    x = s["x"].detach().requires_grad_()
    y = s["module"](x)
    loss = (y - s["y"]).square().sum()
    loss.backward()
    return {"projections": y.detach(), "loss": loss.detach(),
            "gradient": x.grad}


def work(case):
    """Compulsory bytes (inputs read once, outputs written once) and
    operations: eight per voxel and angle for each projection or
    backprojection, and the row transforms of the filter."""
    if case["kind"] == "batch":
        w = [work(dict(p, kind="sirt", storage="float32",
                       iters=case["iters"]))
             for p in _problems(case, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    v = case["nx"] * case["ny"] * case["nz"]
    p = case["angles"] * case["rows"] * case["cols"]
    once, one_way = 4.0 * (v + p), 8.0 * v * case["angles"]
    if case["kind"] == "operator":
        n = 2 if case["direction"] == "both" else 1
        return {"bytes": n * once, "flops": n * one_way}
    if case["kind"] == "fdk":
        m = 2.0 ** math.ceil(math.log2(2 * case["cols"]))
        return {"bytes": once, "flops": one_way + 5.0 * m * math.log2(m)
                * case["angles"] * case["rows"]}
    if case["kind"] == "sirt":
        # set-up projects twice; the iterate and the data move once each
        return {"bytes": once, "flops": 2 * (case["iters"] + 1) * one_way}
    return {"bytes": 2 * once, "flops": 2 * one_way}


# ---------------------------------------------------------------------------
# float64 evaluation
# ---------------------------------------------------------------------------
def _rays(c, k):
    """Joseph rays of angle ``k`` in the voxel frame (volume centre at the
    origin): dominant axis, in-slice axes, slice positions, slopes and
    offsets (rows * cols) and the path-length factor."""
    src, pix = _pixels(c, k)
    centre = torch.as_tensor(_vectors(c)[1][k], device="cuda")
    A = int((src - centre).abs().argmax())
    D1, D2 = [i for i in range(3) if i != A]
    d = (pix - src).reshape(-1, 3)
    a1, a2 = d[:, D1] / d[:, A], d[:, D2] / d[:, A]
    b1, b2 = src[D1] - a1 * src[A], src[D2] - a2 * src[A]
    return A, D1, D2, a1, a2, b1, b2, torch.sqrt(1 + a1 ** 2 + a2 ** 2)


def _footprints(c, k, rays_per_step=1 << 17):
    """For batches of rays of angle ``k``: (first ray, flat voxel indices,
    weights) of the four texels of every sample, zero outside."""
    A, D1, D2, a1, a2, b1, b2, corr = _rays(c, k)
    n = (c["nx"], c["ny"], c["nz"])
    stride = (n[1] * n[2], n[2], 1)
    s = torch.arange(n[A], device="cuda")
    t = s.double() - n[A] / 2 + 0.5
    step = max(1, rays_per_step * 64 // n[A])
    for r in range(0, a1.numel(), step):
        e = slice(r, r + step)
        y = a1[e, None] * t + b1[e, None] + (n[D1] / 2 - 0.5)
        z = a2[e, None] * t + b2[e, None] + (n[D2] / 2 - 0.5)
        j, i = torch.floor(y), torch.floor(z)
        fy, fz = y - j, z - i
        j, i = j.long(), i.long()
        terms = []
        for dj in (0, 1):
            for di in (0, 1):
                jj, ii = j + dj, i + di
                w = (fy if dj else 1 - fy) * (fz if di else 1 - fz)
                ok = (jj >= 0) & (jj < n[D1]) & (ii >= 0) & (ii < n[D2])
                terms.append((
                    s * stride[A] + jj.clamp_(0, n[D1] - 1) * stride[D1]
                    + ii.clamp_(0, n[D2] - 1) * stride[D2],
                    torch.where(ok, w, 0.0) * corr[e, None]))
        yield r, terms


def _project(c, vol):
    x = vol.double().reshape(-1)
    out = torch.zeros((c["angles"], c["rows"] * c["cols"]),
                      dtype=torch.float64, device="cuda")
    for k in range(c["angles"]):
        for r, terms in _footprints(c, k):
            out[k, r:r + terms[0][0].shape[0]] = sum(
                (x[i] * w).sum(1) for i, w in terms)
    return out.reshape(c["angles"], c["rows"], c["cols"])


def _transpose(c, proj):
    p = proj.double().reshape(c["angles"], -1)
    out = torch.zeros(c["nx"] * c["ny"] * c["nz"], dtype=torch.float64,
                      device="cuda")
    for k in range(c["angles"]):
        for r, terms in _footprints(c, k):
            v = p[k, r:r + terms[0][0].shape[0], None]
            for i, w in terms:
                out.index_add_(0, i.reshape(-1), (w * v).reshape(-1))
    return out.reshape(c["nx"], c["ny"], c["nz"])


def _backproject(c, proj):
    p = proj.double()
    rows, cols = c["rows"], c["cols"]
    n = (c["nx"], c["ny"], c["nz"])
    ax = [torch.arange(m, device="cuda", dtype=torch.float64) - m / 2 + 0.5
          for m in n]
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    src, det, uu, vv = _vectors(c)
    for k in range(c["angles"]):
        u, v, s = uu[k] * c["pitch"], vv[k] * c["pitch"], src[k]
        d = det[k] - u * cols / 2 - v * rows / 2
        flat = p[k].reshape(-1)
        nrm = np.cross(u, v)
        near = float(nrm @ (d - s))

        def affine(q, w, near=near):
            # q . (x - s) for all voxels, over w . (x - s), times near
            return [q[0] * (ax[0] - s[0])[:, None, None],
                    q[1] * (ax[1] - s[1])[None, :, None],
                    q[2] * (ax[2] - s[2])[None, None, :]]

        lam = near / sum(affine(nrm, None))  # s + lam (x - s) on the panel
        e1, e2 = np.cross(v, nrm), np.cross(nrm, u)
        e1, e2 = e1 / (e1 @ u), e2 / (e2 @ v)
        U = lam * sum(affine(e1, None)) + float(e1 @ (s - d)) - 0.5
        V = lam * sum(affine(e2, None)) + float(e2 @ (s - d)) - 0.5
        iu, iv = torch.floor(U), torch.floor(V)
        fu, fv = U - iu, V - iv
        iu, iv = iu.long(), iv.long()
        val = torch.zeros_like(out)
        for dv in (0, 1):
            for du in (0, 1):
                a, b = iv + dv, iu + du
                w = (fv if dv else 1 - fv) * (fu if du else 1 - fu)
                ok = (a >= 0) & (a < rows) & (b >= 0) & (b < cols)
                val += torch.where(ok, w, 0.0) * flat[
                    a.clamp_(0, rows - 1) * cols + b.clamp_(0, cols - 1)]
        out += val * lam ** 2 / float(np.linalg.norm(nrm))
    return out


def _filtered(c, proj):
    """Cosine weights (at the pixels' corners) and Ram-Lak row filter."""
    p = proj.double().clone()
    src, det, uu, vv = _vectors(c)
    rows, cols = c["rows"], c["cols"]
    r = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None, None]
    q = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :, None]
    for k in range(c["angles"]):
        u, v = uu[k] * c["pitch"], vv[k] * c["pitch"]
        d = det[k] - u * cols / 2 - v * rows / 2 - src[k]
        pix = (torch.as_tensor(d, device="cuda")
               + q * torch.as_tensor(u, device="cuda")
               + r * torch.as_tensor(v, device="cuda"))
        p[k] *= float(np.linalg.norm(det[k] - src[k])) / pix.norm(dim=-1)
    m = max(64, 2 ** math.ceil(math.log2(2 * cols)))
    h = np.zeros(m)
    h[0] = 0.25
    odd = np.arange(1, m // 2, 2)
    h[odd] = h[m - odd] = -1.0 / (np.pi * odd) ** 2
    H = torch.as_tensor(4 * np.real(np.fft.rfft(h)), device="cuda")
    for k in range(c["angles"]):
        p[k] = torch.fft.irfft(torch.fft.rfft(p[k], n=m) * H, n=m)[:, :cols]
    return p


def _solve(c, y, iters, low):
    """SIRT in float64 with the projector pair above."""
    v = (c["nx"], c["ny"], c["nz"])
    one = dict(dtype=torch.float64, device="cuda")
    C = 1.0 / _backproject(c, torch.ones(y.shape, **one))
    R = 1.0 / _project(c, torch.ones(v, **one))
    C[torch.isinf(C)] = 0.0
    R[torch.isinf(R)] = 0.0
    x = torch.zeros(v, **one)
    for _ in range(iters):
        x = x - C * _backproject(c, R * (_project(c, x) - y.double()))
        if low is not None:
            x = x.clamp(min=low)
    return x


def _samples(c):
    """float64 samples of one projection and one backprojection."""
    back = c["nx"] * c["ny"] * c["nz"]
    rays = c["rows"] * c["cols"] * max(c["nx"], c["ny"])
    return float(c["angles"]) * (back if c.get("kind") == "fdk"
                                 else rays + back)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        probs = _problems(case, seed)
        if sum(_samples(p) for p in probs) * case["iters"] > EXACT_SAMPLES:
            return None
        return {"volumes": [_solve(p, _measured(p, seed + 17 * i),
                                   case["iters"], 0.0)
                            for i, p in enumerate(probs)]}
    cost = _samples(case) * (case["iters"] + 1 if kind == "sirt" else 1)
    if cost > EXACT_SAMPLES:
        return None
    if kind == "operator":
        out = {}
        if case["direction"] in ("forward", "both"):
            out["projections"] = _project(case, _volume(case, seed))
        if case["direction"] in ("back", "both"):
            out["volume"] = _backproject(case, _measured(case, seed))
        return out
    y = _measured(case, seed)
    if kind == "fdk":
        return {"volume": _backproject(case, _filtered(case, y))}
    if kind == "sirt":
        low = 0.0 if case["storage"] == "float32" else None
        return {"volume": _solve(case, y, case["iters"], low)}
    p = _project(case, 0.5 * _volume(case, seed))
    res = p - y.double()
    return {"projections": p[None, None], "loss": res.square().sum(),
            "gradient": 2.0 * _transpose(case, res)[None, None]}
