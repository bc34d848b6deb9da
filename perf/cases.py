"""Workloads of the forward projector for timing it: single poses, scans, batches,
the sampling options, the one-shot host call and the post-projection steps, each
through the calls a program makes.

Every case is a dict of plain values.  ``kind`` says which calls it makes:

  scan      Context.project of a resident volume, matrices and result on the device
  batch     Context.project_batch over several volumes and detectors
  plan      Plan.launch of requests on resident volumes (a DRR service's replay)
  oneshot   Context.project_volume with host volume, matrices and result
  poisson   Context.poisson_noise on a copy of given extinctions
  spectral  SpectralEffectsExtension.project of resident material volumes

Volumes are seeded water cylinders with random ellipsoids and a fine texture,
generated on the device; geometries are circular or helical cone beams.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import ctl_b200
from ctl_b200.extensions import SpectralEffectsExtension
from ctl_b200.projector import Settings, VoxelVolume, torch_stream_handle

_STORAGE = {"f32": ctl_b200.F32, "bf16": ctl_b200.BF16, "f16": ctl_b200.F16}
_ACCUM = {"kahan": ctl_b200.ACCUM_KAHAN, "fp64": ctl_b200.ACCUM_FP64}
_TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_MOST_EXACT = 3.0e10  # samples; the 64-bit evaluation of more takes too long
_BINS = 30

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = ctl_b200.Context(0)
    return _context


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------

def _case(name, kind, **kw):
    c = {"kind": kind, "nx": 256, "ny": 256, "nz": 256, "voxel_mm": 1.0, "views": 1, "channels": 512, "rows": 512,
         "pixel_mm": 0.6, "modules": 1, "helical": False, "sid_mm": 750.0, "sdd_mm": 1200.0, "storage": "f32",
         "accum": "kahan", "sampling": 0.3, "upsampling": 1, "interpolate": True, "rays_x": 1, "rays_y": 1,
         "requests": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one pose of a 2D/3D registration loop on a small volume: latency and launches
        _case("pose_64", "scan", nx=64, ny=64, nz=64, voxel_mm=2.0, channels=128, rows=128, pixel_mm=1.0,
              sdd_mm=1000.0),
        # an ordered subset of a C-arm scan, odd volume and detector sizes, double accumulator
        _case("subset_odd", "scan", nx=201, ny=173, nz=155, views=23, channels=479, rows=361, accum="fp64"),
        # the flagship: a whole short scan of a 256^3 volume
        _case("scan_256", "scan", views=360),
        # half a turn of a clinical helical scan: 512^3, curved detector of 64 modules of 16 x 16
        _case("helical_512", "scan", nx=512, ny=512, nz=512, voxel_mm=0.5, views=180, channels=16, rows=16,
              pixel_mm=1.0, modules=64, helical=True, sid_mm=570.0, sdd_mm=1040.0),
        # coarse voxels seen by fine pixels: the settings' optimizedFor() gives volume up-sampling 3
        _case("upsampled", "scan", nx=101, ny=97, nz=89, voxel_mm=2.0, views=60, channels=512, rows=384,
              upsampling=3),
        # nearest-voxel sampling (interpolation off)
        _case("nearest", "scan", views=45, interpolate=False),
        # fine voxels seen by large pixels: optimizedFor() gives 2 x 2 rays per pixel; half-precision storage
        _case("subrays_f16", "scan", nx=320, ny=320, nz=256, voxel_mm=0.5, views=60, channels=160, rows=120,
              pixel_mm=1.2, storage="f16", rays_x=2, rays_y=2),
        # a simulation run over uneven volumes and detectors in one call
        _case("batch_uneven", "batch", nx=192, ny=160, nz=128, views=48, channels=384, rows=256, pixel_mm=0.75,
              sdd_mm=1000.0, requests=6),
        # DRR serving: a replayed plan of eight short requests on resident 16-bit volumes
        _case("drr_plan", "plan", views=6, channels=256, rows=256, pixel_mm=1.2, storage="bf16", requests=8),
        # the drop-in call as CTL makes it: host volume in, host projections out
        _case("oneshot_host", "oneshot", views=30),
        # quantum noise on a scan's extinctions
        _case("poisson", "poisson", views=60),
        # polychromatic scan: two density projections, 30 energy bins per pixel
        _case("spectral", "spectral", nx=128, ny=128, nz=128, voxel_mm=2.0, views=90),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """A case of the same kinds: mostly scans, sizes over the whole range, odd ones among them."""
    kind = rng.choice(["scan"] * 7 + ["batch", "plan", "oneshot", "poisson", "spectral"])
    edge = _log(rng, 48, 384)
    n = [max(24, int(edge * rng.uniform(0.6, 1.0))) for _ in range(3)]
    voxel = round(256.0 / max(n) * rng.uniform(0.7, 1.3), 3)
    ch, rows = _log(rng, 64, 640), _log(rng, 64, 512)
    kw = dict(nx=n[0], ny=n[1], nz=n[2], voxel_mm=voxel, channels=ch, rows=rows, views=_log(rng, 1, 180),
              pixel_mm=round(330.0 / max(ch, rows) * rng.uniform(0.8, 1.2), 3),
              storage=rng.choice(["f32", "f32", "f32", "bf16", "f16"]),
              accum=rng.choice(["kahan", "kahan", "fp64"]),
              sampling=rng.choice([0.2, 0.3, 0.3, 0.3, 0.3, 0.5, 0.75, 1.0]))
    if kind == "scan":
        what = rng.choice(["plain", "plain", "plain", "helical", "upsampled", "nearest", "rays"])
        if what == "helical":
            m = rng.choice([16, 20, 40, 64])
            kw.update(helical=True, modules=m, channels=rng.choice([12, 16, 24]), rows=rng.choice([16, 24, 32]),
                      pixel_mm=1.0, sid_mm=570.0, sdd_mm=1040.0, views=_log(rng, 30, 360))
        elif what == "upsampled":
            f = rng.choice([2, 2, 3, 4])
            kw.update(upsampling=f, nx=max(24, n[0] // f), ny=max(24, n[1] // f), nz=max(24, n[2] // f),
                      voxel_mm=round(voxel * f, 3))
        elif what == "nearest":
            kw.update(interpolate=False)
        elif what == "rays":
            kw.update(rays_x=rng.choice([1, 2, 3]), rays_y=rng.choice([2, 3]), channels=max(32, ch // 2),
                      rows=max(32, rows // 2), pixel_mm=round(2 * kw["pixel_mm"], 3))
    elif kind == "batch":
        kw.update(requests=rng.randint(2, 8), views=min(kw["views"], 60))
    elif kind == "plan":
        kw.update(requests=rng.randint(1, 8), views=rng.randint(1, 16), channels=min(ch, 384), rows=min(rows, 384))
    elif kind == "spectral":
        kw.update(sampling=0.3)
    c = _case(None, kind, **kw)
    for _ in range(64):  # no costlier than a whole short scan
        if _samples(c) <= 6.0e10:
            break
        c["views"] = max(1, c["views"] // 2)
    return c


# ---------------------------------------------------------------------------------------------
# volumes and geometries
# ---------------------------------------------------------------------------------------------

def _phantom(nx, ny, nz, voxel, seed):
    """(Z, Y, X) float32 on the GPU: water cylinder, 24 ellipsoids, 1% texture; 1/mm."""
    rng = np.random.default_rng(seed)
    dev = "cuda"
    x = ((torch.arange(nx, device=dev, dtype=torch.float32) - (nx - 1) / 2) * voxel).view(1, 1, nx)
    y = ((torch.arange(ny, device=dev, dtype=torch.float32) - (ny - 1) / 2) * voxel).view(1, ny, 1)
    z = ((torch.arange(nz, device=dev, dtype=torch.float32) - (nz - 1) / 2) * voxel).view(nz, 1, 1)
    radius = 0.45 * min(nx, ny) * voxel
    inside = ((x * x + y * y) <= radius * radius).expand(nz, ny, nx)
    vol = inside.to(torch.float32) * 0.02
    for _ in range(24):
        semi = rng.uniform(0.03, 0.18, 3) * radius * 2
        r, phi = rng.uniform(0.0, 0.6) * radius, rng.uniform(0, 2 * math.pi)
        c = (r * math.cos(phi), r * math.sin(phi), rng.uniform(-0.4, 0.4) * nz * voxel)
        mu = float(rng.uniform(0.002, 0.02))
        lo = [max(0, int((c[k] - semi[k]) / voxel + (n - 1) / 2)) for k, n in enumerate((nx, ny, nz))]
        hi = [min(n, int((c[k] + semi[k]) / voxel + (n - 1) / 2) + 2) for k, n in enumerate((nx, ny, nz))]
        if any(h <= l for l, h in zip(lo, hi)):
            continue
        e = (((x[..., lo[0]:hi[0]] - c[0]) / semi[0]) ** 2 + ((y[:, lo[1]:hi[1]] - c[1]) / semi[1]) ** 2
             + ((z[lo[2]:hi[2]] - c[2]) / semi[2]) ** 2) <= 1.0
        vol[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += mu * e
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    vol *= 1.0 + 0.01 * torch.randn(vol.shape, generator=g, device=dev)
    return vol.contiguous()


def _matrices(c, seed, views=None, channels=None, rows=None):
    """(views, modules, 3, 4) float64 projection matrices of a case."""
    rng = np.random.default_rng(seed + 77)
    V = c["views"] if views is None else views
    C = c["channels"] if channels is None else channels
    R = c["rows"] if rows is None else rows
    pitch, sid, sdd, M = c["pixel_mm"], c["sid_mm"], c["sdd_mm"], c["modules"]
    start = rng.uniform(0, 2 * math.pi)
    if c["helical"]:
        th = start + 2 * math.pi * np.arange(V) / 360.0
        feed = 0.25 * c["nz"] * c["voxel_mm"]
        z = feed * (np.arange(V) / 360.0 - 0.5 * V / 360.0)
        dphi = C * pitch / sdd
    else:
        span = math.radians(200.0) + 2 * math.atan(0.5 * C * pitch / sdd)
        th = start + span * np.arange(V) / max(V, 1)
        z = np.zeros(V)
        dphi = 0.0
    cos, sin, nul, one = np.cos(th), np.sin(th), np.zeros(V), np.ones(V)
    src = np.stack([sid * cos, sid * sin, z], -1) + rng.uniform(-0.5, 0.5, (V, 3))
    R0 = np.stack([np.stack([-sin, cos, nul], -1), np.stack([nul, nul, -one], -1), np.stack([-cos, -sin, nul], -1)], 1)
    if not c["helical"]:  # small detector tilts, as a C-arm has
        t = np.deg2rad(rng.uniform(-0.2, 0.2, (V, 2)))
        rx, ry = np.tile(np.eye(3), (V, 1, 1)), np.tile(np.eye(3), (V, 1, 1))
        rx[:, 1, 1] = rx[:, 2, 2] = np.cos(t[:, 0])
        rx[:, 2, 1] = np.sin(t[:, 0])
        rx[:, 1, 2] = -rx[:, 2, 1]
        ry[:, 0, 0] = ry[:, 2, 2] = np.cos(t[:, 1])
        ry[:, 0, 2] = np.sin(t[:, 1])
        ry[:, 2, 0] = -ry[:, 0, 2]
        R0 = rx @ ry @ R0
    K = np.array([[sdd / pitch, 0, (C - 1) / 2], [0, sdd / pitch, (R - 1) / 2], [0, 0, 1.0]])
    P = np.empty((V, M, 3, 4))
    for m in range(M):
        phi = (m - (M - 1) / 2) * dphi
        Rm = np.array([[math.cos(phi), 0, math.sin(phi)], [0, 1, 0], [-math.sin(phi), 0, math.cos(phi)]])
        KR = K @ (Rm @ R0)
        P[:, m, :, :3] = KR
        P[:, m, :, 3] = -np.einsum("vij,vj->vi", KR, src)
    return P


def _shape(c, k):
    """Volume, views and detector of request k of a batch or plan: uneven around the case's."""
    r = random.Random(1000 * k + 7)
    s = dict(c)
    if c["kind"] == "batch":
        for a in ("nx", "ny", "nz"):
            s[a] = max(24, int(c[a] * r.uniform(0.6, 1.2)))
        s["views"] = max(1, int(c["views"] * r.uniform(0.4, 1.2)))
        s["channels"], s["rows"] = max(32, int(c["channels"] * r.uniform(0.7, 1.2))), max(32, int(c["rows"] * r.uniform(0.7, 1.2)))
    elif c["kind"] == "plan":
        s["views"] = max(1, int(c["views"] * r.uniform(0.3, 1.7)))
    return s


# ---------------------------------------------------------------------------------------------
# preparing and running
# ---------------------------------------------------------------------------------------------

class _State(dict):
    """What a program holds; gives its resident volumes and plan back when it goes."""

    def __del__(self):
        try:
            if "plan" in self:
                self["plan"].close()
            for v in self.get("volumes", ()):
                v.release()
        except Exception:
            pass


def _resident(c, seed):
    """A volume in the projector's memory.  The projector reads it on its own stream, so it has to be complete."""
    v = _phantom(c["nx"], c["ny"], c["nz"], c["voxel_mm"], seed)
    torch.cuda.synchronize()
    return _ctx().volume(VoxelVolume(v, (c["voxel_mm"],) * 3), _STORAGE[c["storage"]])


def _settings(c):
    return Settings(rays_per_pixel=[c["rays_x"], c["rays_y"]], ray_sampling=c["sampling"],
                    volume_upsampling=c["upsampling"], interpolate=c["interpolate"], accum=_ACCUM[c["accum"]],
                    storage=_STORAGE[c["storage"]])


def _spectrum(c, seed):
    """Bin intensities per view, attenuation of two materials and a response per bin."""
    rng = np.random.default_rng(seed + 5)
    E = np.linspace(25.0, 120.0, _BINS)
    mu = np.stack([0.02 * (0.6 + (45.0 / E) ** 3), 0.03 * (0.5 + (60.0 / E) ** 3)], 1) / 0.02
    flux = 1e5 * np.exp(-0.5 * ((E - 60.0) / 22.0) ** 2)[:, None] * (1 + 0.05 * rng.uniform(-1, 1, (1, c["views"])))
    flux = np.ascontiguousarray(flux)
    resp = (E / 60.0).astype(np.float32)
    return mu.astype(np.float32), flux, (flux * resp[:, None].astype(np.float64)).sum(0), resp


def _extinctions(c, seed):
    """Smooth extinctions 0..6 of a scan, (views, 1, rows, channels) on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    V, R, C = c["views"], c["rows"], c["channels"]
    y = torch.linspace(-1, 1, R, device="cuda").view(1, 1, R, 1)
    x = torch.linspace(-1, 1, C, device="cuda").view(1, 1, 1, C)
    t = torch.rand((V, 1, 1, 1), generator=g, device="cuda") * 6.28
    p = 5.5 * torch.sqrt(torch.clamp(1.0 - (1.1 * x) ** 2, min=0.0)) * (1.0 + 0.1 * torch.cos(3 * y + t))
    return (p * (1.0 + 0.02 * torch.randn(p.shape, generator=g, device="cuda"))).clamp_(min=0.0).contiguous()


def prepare(case, seed):
    ctx = _ctx()
    c = case
    s = _State(kind=c["kind"], settings=_settings(c))
    if c["kind"] == "poisson":
        s.update(data=_extinctions(c, seed), seed=int(seed))
        return s
    if c["kind"] == "oneshot":
        v = _phantom(c["nx"], c["ny"], c["nz"], c["voxel_mm"], seed).cpu().numpy()
        s.update(volume=VoxelVolume(v, (c["voxel_mm"],) * 3), P=_matrices(c, seed), C=c["channels"], R=c["rows"])
        return s
    if c["kind"] in ("batch", "plan"):
        vols, reqs = [], []
        for k in range(c["requests"]):
            q = _shape(c, k)
            if c["kind"] == "batch" or k < 2:  # a service keeps a few volumes; each batch job has its own
                vols.append(_resident(q, seed + k))
            P = torch.from_numpy(_matrices(q, seed + k)).cuda()
            out = torch.empty((q["views"], q["modules"], q["rows"], q["channels"]), device="cuda")
            reqs.append((vols[k % len(vols)], P, out))
        s.update(volumes=vols, requests=reqs)
        torch.cuda.synchronize()
        if c["kind"] == "plan":
            s["plan"] = ctx.plan(reqs, s["settings"])
        return s
    P = torch.from_numpy(_matrices(c, seed)).cuda()
    if c["kind"] == "spectral":
        vols = [_resident(c, seed + k) for k in range(2)]
        mu, flux, total, resp = _spectrum(c, seed)
        ext = SpectralEffectsExtension(ctx, s["settings"])
        ext.configure(P, c["channels"], c["rows"], mu, flux, total, resp)
        s.update(volumes=vols, ext=ext)
        return s
    s.update(volumes=[_resident(c, seed)], P=P, C=c["channels"], R=c["rows"])
    return s


def run(state):
    ctx, s = _ctx(), state
    kind = s["kind"]
    if kind == "scan":
        return ctx.project(s["volumes"][0], s["P"], s["C"], s["R"], s["settings"])
    if kind == "batch":
        ctx.project_batch(s["requests"], s["settings"])
        return [r[2] for r in s["requests"]]
    if kind == "plan":
        s["plan"].launch(torch_stream_handle(torch.cuda.current_stream()))
        return [r[2] for r in s["requests"]]
    if kind == "oneshot":
        return ctx.project_volume(s["volume"], s["P"], s["C"], s["R"], s["settings"])
    if kind == "poisson":
        return ctx.poisson_noise(s["data"].clone(), 1.0e5, s["seed"])
    return s["ext"].project(s["volumes"])


# ---------------------------------------------------------------------------------------------
# work and 64-bit values
# ---------------------------------------------------------------------------------------------

def _grid(c):
    """Virtual voxel grid the rays see: counts, voxel size, step length (mm)."""
    f = c["upsampling"] if c["interpolate"] else 1
    vox = float(np.float32(c["voxel_mm"]))
    if f > 1:
        vox = float(np.float32(c["voxel_mm"]) / np.float32(f))
    return np.array([c["nx"] * f, c["ny"] * f, c["nz"] * f], np.float64), vox, vox * float(np.float32(c["sampling"])), f


def _samples(c):
    """About how many samples a pass takes, from every 16th pixel of a few views."""
    if c["kind"] == "poisson":
        return 0.0
    total = 0.0
    for k in range(c["requests"]):
        q = _shape(c, k)
        n, vox, inc, _ = _grid(q)
        few = dict(q, views=min(q["views"], 4))
        P = _matrices(few, 1).reshape(-1, 3, 4)
        P = P[:: max(1, len(P) // 16)]
        x, y = np.meshgrid(np.arange(0, q["channels"], 16.0), np.arange(0, q["rows"], 16.0))
        d = np.einsum("pij,jn->pni", np.linalg.inv(P[:, :, :3]), np.stack([x.ravel(), y.ravel(), np.ones(x.size)]))
        d /= np.linalg.norm(d, axis=-1, keepdims=True)
        src = -np.einsum("pij,pj->pi", np.linalg.inv(P[:, :, :3]), P[:, :, 3])[:, None]
        with np.errstate(divide="ignore"):
            a, b = (-0.5 * n * vox - src) / d, (0.5 * n * vox - src) / d
        chord = np.maximum(np.maximum(a, b).min(-1) - np.minimum(a, b).max(-1), 0.0)
        total += chord.mean() / inc * q["views"] * q["modules"] * q["channels"] * q["rows"] * q["rays_x"] * q["rays_y"]
    return total * (2 if c["kind"] == "spectral" else 1)


def work(case):
    """bytes: volumes, matrices and results once; flops: 7 interpolations (14) and an addition per sample."""
    c = case
    if c["kind"] == "poisson":
        px = c["views"] * c["channels"] * c["rows"]
        return {"bytes": 8.0 * px, "flops": 60.0 * px}
    n_bytes, flops = 0.0, 15.0 * _samples(c)
    size = 4.0 if c["storage"] == "f32" else 2.0
    for k in range(c["requests"]):
        q = _shape(c, k)
        px = float(q["views"] * q["modules"] * q["channels"] * q["rows"])
        vol = float(q["nx"] * q["ny"] * q["nz"]) * (4.0 if c["kind"] == "oneshot" else size)
        if c["kind"] == "plan" and k >= 2:
            vol = 0.0
        n_bytes += vol * (2 if c["kind"] == "spectral" else 1) + 4.0 * px + 96.0 * q["views"] * q["modules"]
        if c["kind"] == "spectral":
            flops += 8.0 * _BINS * px
    return {"bytes": n_bytes, "flops": flops}


def _exact_projections(c, vol, P):
    """increment * sum of the samples source + i * step, i >= 0, in 64 bits; zero outside the grid."""
    n, vox, inc, f = _grid(c)
    dev = vol.device
    v64 = vol.to(torch.float64)[None, None]
    P = torch.from_numpy(P).to(dev)
    V, M, R, C = P.shape[0], P.shape[1], c["rows"], c["channels"]
    N = torch.tensor(n, device=dev)
    inv = torch.linalg.inv(P[..., :3])
    src = -(inv[:, 0] @ P[:, 0, :, 3:])[..., 0]
    rx, ry = c["rays_x"], c["rays_y"]
    out = torch.zeros((V, M, R, C), dtype=torch.float64, device=dev)
    steps = int(math.ceil(float((N + 2).norm()) * vox / inc)) + 3
    rows_at_once = max(1, int(2.4e7 / (steps * C)))
    xs, ys = torch.arange(C, device=dev, dtype=torch.float64), torch.arange(R, device=dev, dtype=torch.float64)
    k = torch.arange(steps, device=dev, dtype=torch.float64).view(-1, 1, 1, 1)
    for vi in range(V):
        s = src[vi] / vox + N / 2  # source in grid units from the grid's low corner
        for m in range(M):
            for r0 in range(0, R, rows_at_once):
                yy = ys[r0: r0 + rows_at_once]
                for i in range(rx):
                    for j in range(ry):
                        px = (xs - 0.5 + (i + 0.5) / rx).view(1, C).expand(len(yy), C)
                        py = (yy - 0.5 + (j + 0.5) / ry).view(-1, 1).expand(len(yy), C)
                        d = torch.stack([px, py, torch.ones_like(px)], -1) @ inv[vi, m].T
                        d = d / d.norm(dim=-1, keepdim=True) * (inc / vox)
                        a, b = (-1.0 - s) / d, (N + 1.0 - s) / d
                        first = torch.minimum(a, b).nan_to_num(-1e30).amax(-1).clamp(min=0.0)
                        first = torch.ceil(first.clamp(max=1e9))
                        last = torch.maximum(a, b).nan_to_num(1e30).amin(-1)
                        at = first[None, ..., None] + k
                        p = s + at * d  # position in grid units from the low corner
                        if not c["interpolate"]:
                            q = torch.floor(p)
                            ok = ((q >= 0) & (q < N)).all(-1) & (at[..., 0] <= last)
                            q = torch.where(ok[..., None], q, torch.zeros_like(q)).long()
                            val = v64[0, 0][q[..., 2], q[..., 1], q[..., 0]] * ok
                            got = val.sum(0)
                        else:
                            if f > 1:  # replicated grid: a ramp of one fine voxel about each coarse face
                                face = torch.round(p / f)
                                u = face - 0.5 + (p - f * face).clamp(-0.5, 0.5)
                            else:
                                u = p - 0.5
                            size = torch.tensor([c["nx"], c["ny"], c["nz"]], device=dev, dtype=torch.float64)
                            g = (2.0 * u + 1.0) / size - 1.0
                            g = torch.where((at <= last[None, ..., None]), g, torch.full_like(g, 9.0))
                            got = torch.nn.functional.grid_sample(v64, g.reshape(1, steps, len(yy), C, 3), mode="bilinear",
                                                                  padding_mode="zeros", align_corners=False)[0, 0].sum(0)
                        out[vi, m, r0: r0 + len(yy)] += got
    return out * (inc / (rx * ry))


def exact(case, seed):
    c = case
    if c["kind"] == "poisson" or _samples(c) > _MOST_EXACT or c["modules"] * c["views"] * c["rays_x"] * c["rays_y"] > 12000:
        return None
    stored = lambda v: v.to(_TORCH[c["storage"]]).to(torch.float32)  # noqa: E731
    if c["kind"] in ("batch", "plan"):
        outs = []
        for k in range(c["requests"]):
            q = _shape(c, k)
            at = k if c["kind"] == "batch" else k % min(2, c["requests"])
            v = _shape(c, at)
            vol = stored(_phantom(v["nx"], v["ny"], v["nz"], v["voxel_mm"], seed + at))
            outs.append(_exact_projections(dict(q, nx=v["nx"], ny=v["ny"], nz=v["nz"]), vol, _matrices(q, seed + k)))
        return outs
    P = _matrices(c, seed)
    if c["kind"] == "spectral":
        proj = [_exact_projections(c, stored(_phantom(c["nx"], c["ny"], c["nz"], c["voxel_mm"], seed + k)), P)
                for k in range(2)]
        mu, flux, total, resp = (torch.from_numpy(np.asarray(a, np.float64)).cuda() for a in _spectrum(c, seed))
        acc = torch.zeros_like(proj[0])
        for b in range(_BINS):
            acc += flux[b].view(-1, 1, 1, 1) * torch.exp(-(proj[0] * mu[b, 0] + proj[1] * mu[b, 1])) * resp[b]
        return torch.log(total.view(-1, 1, 1, 1) / acc)
    got = _exact_projections(c, stored(_phantom(c["nx"], c["ny"], c["nz"], c["voxel_mm"], seed)), P)
    return got.cpu().numpy() if c["kind"] == "oneshot" else got
