"""The work that users have the engine do, as cases that can be timed and checked.

Every case is one call sequence through the public Python API on a synthetic
scan: a circular cone-beam orbit (ideal, with per-view detector shifts and
tilts, or tilted out of plane), an ellipsoid phantom, Poisson noise, per-pixel
gain and offset.  Scans and frames are made here from the seed alone.

  reconstruct  raw frames on the GPU -> HU volume (FDKEngine.reconstruct)
  host         the same from and to host buffers (FDKEngine.reconstruct_host)
  batch        several scans of uneven size at once (FDKBatch.run)
  stages       the agents' chain, one chunk of views after another
               (preprocess, filter, bp_accumulate, finalize)
  filter       the ramp filter of one chunk of preprocessed views (filter)
  gradient     forward and backward through FDKFunction under per-view motion

A case holds the form ("fp32" or "mixed"), the views, the detector (u x v
pixels of `pix` mm), the volume (x, y, z voxels of `vox` mm) and what the scan
is like: `flex` (per-view detector shift up to 0.5 px and in-plane tilt up to
0.2 deg), `tilt` (deg, the orbit plane about x), `offset` (a detector whose
principal point lies `offset` columns from its left edge, read with
conjugate-view compositing and the z-filter; 0: centred), `metal` inserts.

exact() restates the whole method in FP64 with plain torch.
"""
import math
import random

import numpy as np
import torch

from jenhine_b200.autograd import FDKFunction
from jenhine_b200.fdk import FDKBatch, FDKEngine, ReconConfig, ScanConfig

SID, SDD = 500.0, 800.0      # source to isocentre, source to detector, mm
BRIGHT = 50000.0             # ADU of an unattenuated pixel
MU_WATER = 0.02
BHC = (1.0, 0.05, 0.01)      # beam-hardening polynomial of the scans with metal


def _case(name, do, form, views, u, v, pix, x, y, z, vox, flex=False, tilt=0.0, offset=0, metal=False, chunk=32,
          scans=1):
    c = dict(do=do, form=form, views=views, u=u, v=v, pix=pix, x=x, y=y, z=z, vox=vox, flex=flex, tilt=tilt,
             offset=offset, metal=metal, chunk=chunk, scans=scans)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest call: a quick look at a cropped scan, ragged in every size
        _case("quick_look_fp32", "reconstruct", "fp32", 11, 33, 17, 4.0, 13, 37, 5, 2.0),
        # an everyday small volume from an ideal orbit, in both forms
        _case("small_fp32", "reconstruct", "fp32", 360, 256, 256, 0.5, 128, 128, 128, 0.5),
        _case("small_mixed", "reconstruct", "mixed", 360, 256, 256, 0.5, 128, 128, 128, 0.5),
        # the full dental-size scan with a calibrated-like flexing gantry and metal, in both forms
        _case("dental_fp32", "reconstruct", "fp32", 600, 768, 768, 0.2, 640, 640, 480, 0.125, flex=True, metal=True),
        _case("dental_mixed", "reconstruct", "mixed", 600, 768, 768, 0.2, 640, 640, 480, 0.125, flex=True, metal=True),
        # projection matrices with P[10] != 0, as calibrations give, at a ragged size
        _case("tilted_fp32", "reconstruct", "fp32", 301, 510, 411, 0.3, 300, 253, 207, 0.3, flex=True, tilt=1.0),
        # an offset detector: compositing and z-filter
        _case("offset_mixed", "reconstruct", "mixed", 360, 512, 384, 0.3, 360, 360, 200, 0.25, flex=True, offset=70),
        # a program that keeps its scans in host memory
        _case("host_fp32", "host", "fp32", 360, 512, 512, 0.3, 256, 256, 200, 0.35, flex=True),
        # a queue of scans of uneven size
        _case("queue_fp32", "batch", "fp32", 360, 512, 512, 0.4, 256, 256, 256, 0.4, scans=5),
        # the agents' chain: frames arrive in chunks of views
        _case("stages_fp32", "stages", "fp32", 180, 512, 400, 0.3, 256, 256, 160, 0.35, flex=True),
        # the filter agent's work on one chunk of full-size frames
        _case("filter_fp32", "filter", "fp32", 600, 768, 768, 0.2, 64, 64, 64, 1.0, flex=True),
        # motion estimation: value and gradient with respect to the projections and six motions per view
        _case("motion_gradient", "gradient", "fp32", 360, 512, 512, 0.5, 256, 256, 256, 0.4, chunk=64),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    do = rng.choice(["reconstruct"] * 5 + ["host", "batch", "stages", "filter", "gradient"])
    form = rng.choice(["fp32", "fp32", "mixed"])
    chunk, scans, offset, tilt, metal = 32, 1, 0, 0.0, False
    flex = rng.random() < 0.6
    if do in ("reconstruct", "host"):
        views, u, v = _log(rng, 12, 600), _log(rng, 32, 768), _log(rng, 24, 768)
        x, y, z = _log(rng, 16, 512), _log(rng, 16, 512), _log(rng, 5, 400)
        kind = rng.random() if do == "reconstruct" else 1.0
        tilt = round(rng.uniform(0.2, 2.0), 2) if kind < 0.25 else 0.0
        if 0.25 <= kind < 0.4:
            u, views, offset = max(u, 200), 2 * _log(rng, 30, 240), rng.randint(50, 90)
        metal = rng.random() < 0.3
        tilt *= form == "fp32" or rng.random() < 0.5
    elif do == "batch":
        views, u, v, scans = _log(rng, 90, 360), _log(rng, 128, 512), _log(rng, 128, 512), rng.randint(2, 6)
        x = y = _log(rng, 64, 256)
        z = _log(rng, 32, 256)
        form, flex = "fp32", False
    elif do == "stages":
        views, u, v, x, y, z = _log(rng, 30, 300), _log(rng, 64, 600), _log(rng, 48, 500), _log(rng, 32, 300), \
            _log(rng, 32, 300), _log(rng, 16, 200)
        chunk = rng.choice([8, 16, 32])
    elif do == "filter":
        views, u, v, x, y, z = 360, _log(rng, 96, 1024), _log(rng, 64, 1024), 32, 32, 32
        chunk = rng.choice([1, 4, 16, 32])
    else:
        views, u, v = _log(rng, 30, 200), _log(rng, 64, 400), _log(rng, 64, 400)
        x = y = _log(rng, 32, 180)
        z = _log(rng, 16, 180)
        form, flex, chunk = "fp32", False, rng.choice([16, 64])
    # detector about 150 mm wide (a little more for the tall ones), volume inside its view in z
    pix = round(154.0 / u, 4)
    vox = round(min(75.0 / max(x, y), 0.42 * v * pix / z), 4)
    return _case(None, do, form, views, u, v, pix, x, y, z, vox, flex, tilt, offset, metal, chunk, scans)


# ---- scans --------------------------------------------------------------------

def _matrices(c, seed):
    """(views, 3, 4) FP64 matrices scaled to P[2][3] = 1 and the frames (source, normal, u and v axes, centre)."""
    n, rng = c["views"], np.random.default_rng(seed + 7919)
    shift = rng.uniform(-1.0, 1.0, (n, 2)) * (0.5 if c["flex"] else 0.0)
    spin = np.deg2rad(rng.uniform(-1.0, 1.0, n) * (0.2 if c["flex"] else 0.0))
    b = 2.0 * math.pi * np.arange(n) / n
    zero, one = np.zeros(n), np.ones(n)
    src = SID * np.stack([np.cos(b), np.sin(b), zero], 1)
    nrm = np.stack([-np.cos(b), -np.sin(b), zero], 1)
    eu0, ev0 = np.stack([-np.sin(b), np.cos(b), zero], 1), np.stack([zero, zero, one], 1)
    ct, st = np.cos(spin)[:, None], np.sin(spin)[:, None]
    eu, ev = ct * eu0 + st * ev0, -st * eu0 + ct * ev0
    g = math.radians(c["tilt"])
    if g:
        rx = np.array([[1.0, 0.0, 0.0], [0.0, math.cos(g), -math.sin(g)], [0.0, math.sin(g), math.cos(g)]])
        src, nrm, eu, ev = (m @ rx.T for m in (src, nrm, eu, ev))
    cu = (c["offset"] if c["offset"] else c["u"] / 2.0 - 1.0) + shift[:, 0]
    cv = c["v"] / 2.0 - 1.0 + shift[:, 1]

    def row(e):
        return np.concatenate([e, -(src * e).sum(1, keepdims=True)], 1)

    r2 = row(nrm)
    P = np.stack([SDD / c["pix"] * row(eu) + cu[:, None] * r2, SDD / c["pix"] * row(ev) + cv[:, None] * r2, r2], 1)
    return P / P[:, 2:, 3:], (src, nrm, eu, ev, cu, cv)


def _raw(c, seed, frames):
    """(views, v, u) uint16 frames on the GPU: line integrals of an ellipsoid phantom, Poisson noise, gain, offset."""
    dev = "cuda"
    rng = np.random.default_rng(seed + 1)
    half = 0.5 * c["vox"] * np.array([c["x"], c["y"], c["z"]])
    parts = [(np.zeros(3), half * [0.8, 0.7, 0.85], np.eye(3), 0.02)]
    for k in range(12 + 3 * c["metal"]):
        rot = np.linalg.qr(rng.standard_normal((3, 3)))[0]
        metal = k >= 12
        parts.append((rng.uniform(-0.4, 0.4, 3) * half, rng.uniform(*((0.01, 0.03) if metal else (0.05, 0.3)), 3) * half.max(),
                      rot, 0.5 if metal else float(rng.uniform(0.0, 0.05))))
    src, nrm, eu, ev, cu, cv = frames
    g = torch.Generator(device=dev)
    g.manual_seed(seed + 104729)
    shape = (c["v"], c["u"])
    gain = 1.0 + (torch.rand(shape, generator=g, device=dev) * 2 - 1) * 0.05
    dark = torch.rand(shape, generator=g, device=dev) * 50.0
    raw = torch.empty((c["views"],) + shape, dtype=torch.uint16, device=dev)
    step = max(1, 2 ** 25 // (shape[0] * shape[1]))
    i0 = 5e4 if c["metal"] else 1e5

    def t(v):
        return torch.as_tensor(v, dtype=torch.float32, device=dev)

    for k in range(0, c["views"], step):
        s = slice(k, k + step)
        a = ((torch.arange(c["u"], device=dev) - 0.5)[None] - t(cu[s])[:, None])[:, None, :] * c["pix"]
        b = ((torch.arange(c["v"], device=dev) - 0.5)[None] - t(cv[s])[:, None])[:, :, None] * c["pix"]
        total = torch.zeros((len(src[s]),) + shape, device=dev)
        for centre, axes, rot, mu in parts:   # ray SDD n + a eu + b ev, in the ellipsoid's unit-sphere frame
            m = rot.T / axes[:, None]
            q, d0, d1, d2 = (w @ m.T for w in (src[s] - centre, SDD * nrm[s], eu[s], ev[s]))
            dot = [[t((p * r).sum(1))[:, None, None] for r in (d0, d1, d2)] for p in (d0, d1, d2, q)]
            qq = t((q * q).sum(1) - 1.0)[:, None, None]
            A = dot[0][0] + a * (2 * dot[0][1] + a * dot[1][1]) + b * (2 * dot[0][2] + 2 * a * dot[1][2] + b * dot[2][2])
            B = dot[3][0] + a * dot[3][1] + b * dot[3][2]
            total += (B * B - A * qq).clamp_min_(0).sqrt_().mul_(2 * mu).div_(A)
        total *= (SDD * SDD + a * a + b * b).sqrt_()
        adu = torch.poisson(total.neg_().exp_().mul_(i0), generator=g) * (BRIGHT / i0)
        raw[s] = adu.mul_(gain).add_(dark).round_().clamp_(0, 65535).to(torch.int32).to(torch.uint16)
    return raw


def _engine(c, P):
    scan = ScanConfig(num_views=c["views"], dso=SID, dsd=SDD, num_dets_u=c["u"], num_dets_v=c["v"],
                      detector_pixel_size=c["pix"], bright_field=BRIGHT,
                      beam_hardening=BHC if c["metal"] else (1.0, 0.0, 0.0))
    recon = ReconConfig(c["x"], c["y"], c["z"], c["vox"], c["vox"], mu_water=MU_WATER, z_filter=bool(c["offset"]))
    if c["offset"]:
        scan.filter_input_width, scan.detector_on_right = 2 * c["u"], True
    return FDKEngine(scan, recon, P, precision=c["form"])


def _scans(c):
    """The scans of a batch: the case's own, then smaller and larger ones down to a quarter of its sizes."""
    rng = random.Random(c["views"] * 1000003 + c["x"])
    out = [dict(c)]
    for _ in range(c["scans"] - 1):
        f, g, h = (rng.choice([0.25, 0.5, 0.75, 1.0]) for _ in range(3))
        s = dict(c, views=max(9, int(c["views"] * f)), u=int(c["u"] * g), v=int(c["v"] * g), pix=c["pix"] / g,
                 x=int(c["x"] * h), y=int(c["y"] * h), z=max(4, int(c["z"] * h)), vox=c["vox"] / h)
        out.append(s)
    return out


def _rigid(theta):
    """(n, 4, 4) motions of theta (n, 6: mm and degrees about x, y, z; R = Rz Ry Rx), FP64 torch."""
    n, r = theta.shape[0], theta[:, 3:] * (math.pi / 180.0)
    c, s = torch.cos(r), torch.sin(r)
    o, i = torch.zeros_like(c[:, 0]), torch.ones_like(c[:, 0])

    def m(*rows):
        return torch.stack(rows, 1).reshape(n, 3, 3)

    rx = m(i, o, o, o, c[:, 0], -s[:, 0], o, s[:, 0], c[:, 0])
    ry = m(c[:, 1], o, s[:, 1], o, i, o, -s[:, 1], o, c[:, 1])
    rz = m(c[:, 2], -s[:, 2], o, s[:, 2], c[:, 2], o, o, o, i)
    top = torch.cat([rz @ ry @ rx, theta[:, :3, None]], 2)
    return torch.cat([top, torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=theta.dtype, device=theta.device).expand(n, 1, 4)], 1)


def _motion(c, seed):
    rng = np.random.default_rng(seed + 31)
    th = np.concatenate([rng.uniform(-0.5, 0.5, (c["views"], 3)), rng.uniform(-0.3, 0.3, (c["views"], 3))], 1)
    return th.astype(np.float32)   # an optimiser's parameters


def _target(c, seed):
    """A volume to fit, water in a noisy ellipse, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 17)
    z, y, x = (torch.linspace(-1, 1, c[k], device="cuda") for k in "zyx")
    r2 = z[:, None, None] ** 2 + y[:, None] ** 2 + x ** 2
    noise = torch.rand((c["z"], c["y"], c["x"]), generator=g, device="cuda")
    return MU_WATER * (r2 < 0.6) * (0.8 + 0.4 * noise)


def prepare(case, seed):
    s = {"case": case, "do": case["do"]}
    if case["do"] == "batch":
        s["raw"], engines = [], []
        for k, c in enumerate(_scans(case)):
            P, frames = _matrices(c, seed + k)
            s["raw"].append(_raw(c, seed + k, frames))
            engines.append(_engine(c, P.astype(np.float32)))
        s["out"] = [torch.empty((c["z"], c["y"], c["x"]), device="cuda") for c in _scans(case)]
        s["batch"] = FDKBatch(engines, autotune=False, schedule="pipelined")
        return s
    P, frames = _matrices(case, seed)
    P = P.astype(np.float32)
    s["engine"] = e = _engine(case, P)
    if case["do"] == "filter":
        sub = dict(case, views=case["chunk"])
        raw = _raw(sub, seed, tuple(f[:case["chunk"]] for f in frames))
        s["frames"] = -(raw.float().clamp_min(1.0) / BRIGHT).log()
        s["out"] = torch.empty_like(s["frames"])
        return s
    raw = _raw(case, seed, frames)
    if case["do"] == "gradient":
        s["P"] = P
        s["p"] = e.preprocess(raw).requires_grad_()
        s["theta"] = torch.from_numpy(_motion(case, seed)).cuda().requires_grad_()
        s["target"] = _target(case, seed)
        return s
    shape = (case["z"], case["y"], case["x"])
    if case["do"] == "host":
        s["pinned"] = raw.cpu().pin_memory(), torch.empty(shape, pin_memory=True)
        s["raw"], s["out"] = (t.numpy() for t in s["pinned"])
    else:
        s["raw"], s["out"] = raw, torch.empty(shape, device="cuda")
    return s


def run(s):
    if s["do"] == "reconstruct":
        return s["engine"].reconstruct(s["raw"], s["out"])
    if s["do"] == "host":
        return s["engine"].reconstruct_host(s["raw"], s["out"])
    if s["do"] == "batch":
        return s["batch"].run(s["raw"], s["out"])
    if s["do"] == "filter":
        return s["engine"].filter(s["frames"], 0, out=s["out"])
    if s["do"] == "stages":
        e, n = s["engine"], s["case"]["chunk"]
        e.bp_reset()
        for v0 in range(0, s["case"]["views"], n):
            e.bp_accumulate(e.filter(e.preprocess(s["raw"][v0:v0 + n]), v0), v0)
        return e.finalize(out=s["out"])
    p, theta = s["p"], s["theta"]
    p.grad = theta.grad = None
    vol = FDKFunction.apply(p, theta, s["engine"], s["P"], s["case"]["chunk"])
    loss = torch.nan_to_num(vol - s["target"]).square().sum()
    loss.backward()
    return {"vol": vol.detach(), "p": p.grad, "theta": theta.grad}


def work(case):
    """Frames read and volumes written once; per voxel and view 15 operations (2 products and 2 sums for the sample's
    place, 2 products with 1/W, 2 fractions, 6 for the bilinear form, 1 to sum up); the filter of a row as two FFTs
    of its padded length."""
    if case["do"] == "batch":
        parts = [work(dict(c, do="reconstruct")) for c in _scans(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px, vox = case["u"] * case["v"], case["x"] * case["y"] * case["z"]
    wide = 2 * case["u"] if case["offset"] else case["u"]
    L = 1 << max(1, (2 * wide - 2).bit_length())
    row = 2 * 2.5 * L * math.log2(L) + 3 * L
    if case["do"] == "filter":
        return {"bytes": 8.0 * px * case["chunk"], "flops": row * case["v"] * case["chunk"]}
    flops = case["views"] * (15.0 * vox + row * case["v"])
    if case["do"] == "gradient":   # p, target in; vol, two gradients out; the adjoint and the six derivatives besides
        return {"bytes": 8.0 * px * case["views"] + 8.0 * vox, "flops": flops * 2 + 25.0 * vox * case["views"]}
    return {"bytes": 2.0 * px * case["views"] + 4.0 * vox, "flops": flops}


# ---- the method in FP64 -----------------------------------------------------------

class _Exact:
    """FDK with the engine's geometry conventions: pixel (i, j) of a frame at matrix coordinates (i - 0.5, j - 0.5)."""

    def __init__(self, c, P, dev="cuda"):
        self.c, self.dev, self.N = c, dev, c["views"]
        self.P = torch.as_tensor(P.astype(np.float64), device=dev).reshape(-1, 3, 4)   # the FP32 matrices' values
        self.mirror = bool(c["offset"])
        self.W, self.H = c["u"], c["v"]
        self.in_w = 2 * self.W if c["offset"] else self.W
        self.L = 1
        while self.L < 2 * self.in_w - 1:
            self.L *= 2
        self._operators()

    def _operators(self):
        L, dev = self.L, self.dev
        i = torch.arange(L, device=dev, dtype=torch.float64)
        d = torch.minimum(i, L - i)
        lak = torch.where(d % 2 == 1, -1.0 / (math.pi * d.clamp_min(1)) ** 2, 0.0)
        lak[0] = 0.25
        if L // 2 % 2 == 1:
            lak[L // 2] = -1.0 / (math.pi * (L // 2)) ** 2
        hsr = 0.5 / (np.float32(self.c["pix"]).item() / SDD * SID)
        f = torch.arange(L // 2 + 1, device=dev, dtype=torch.float64) * hsr * 2 / L
        self.spectrum = torch.fft.rfft(lak).real * torch.where(f < hsr, torch.cos(f / hsr * math.pi / 2), 0.0) * math.pi * hsr * 2
        far, near = (1 + 1 / SID) * SID, (1 - 1 / SID) * SID
        s20, s23 = (far + near) / (far - near), ((far + near) - 2 * far * near / SID) / (far - near) / SID
        P = self.P
        last = torch.stack([s20 * P[:, 2, 0], s20 * P[:, 2, 1], torch.zeros_like(P[:, 2, 0]), s23 * P[:, 2, 3]], 1)
        self.inv = torch.linalg.inv(torch.stack([P[:, 0], P[:, 1], last, P[:, 2]], 1))
        taper = torch.ones((self.N, self.W), dtype=torch.float64)
        for v, uf in enumerate((P[:, 0, 3] / P[:, 2, 3]).tolist()):
            u = int(uf)
            n = 2 * ((self.W - u) if u > self.W // 2 else u)
            ramp = torch.cos(torch.arange(n, dtype=torch.float64) * math.pi / max(n, 1)) * 0.5
            if u > self.W // 2:
                taper[v, self.W - n:] = ramp + 0.5
            else:
                taper[v, :n] = 0.5 - ramp
        self.taper = taper.to(dev)

    def preprocess(self, raw):
        p = -(raw.to(torch.int32).double().clamp_min(1.0) / BRIGHT).log()
        if self.c["metal"]:
            b = [np.float32(x).item() for x in BHC]
            p = p * (b[0] + p * (b[1] + b[2] * p))
        return p

    def composite(self, pre, k):
        """The (v, 2u) row of view k: its conjugate resampled to the left of it."""
        W, H, tw = self.W, self.H, 40
        q = self.P[(k + self.N // 2) % self.N] @ self.inv[k]
        i = torch.arange(W, device=self.dev, dtype=torch.float64) - W
        j = torch.arange(H, device=self.dev, dtype=torch.float64)[:, None]
        w = q[2, 0] * i + q[2, 1] * j + q[2, 3]
        u = (q[0, 0] * i + q[0, 1] * j + q[0, 3]) / w
        v = ((q[1, 0] * i + q[1, 1] * j + q[1, 3]) / w).clamp(0.0, H - 1.0)
        other = self._sample(pre[(k + self.N // 2) % self.N], u, v)[0]
        edge = pre[k][:, :5].mean(1, keepdim=True)
        m = 0.5 - 0.5 * torch.cos(torch.arange(tw, device=self.dev, dtype=torch.float64) / tw * math.pi)
        other[:, W - tw:] = other[:, W - tw:] * (1 - m) + edge * m
        return torch.cat([other, pre[k]], 1)

    def _sample(self, img, u, v):
        """Bilinear samples of img inside [0, W-1] x [0, H-1] (0 elsewhere), the mask, columns, rows and fractions."""
        inside = (u >= 0) & (u <= self.W - 1) & (v >= 0) & (v <= self.H - 1)
        u, v = torch.where(inside, u, 0.0), torch.where(inside, v, 0.0)
        i, j = u.floor().clamp_max_(max(self.W - 2, 0)), v.floor().clamp_max_(max(self.H - 2, 0))
        fu, fv = u - i, v - j
        at = (j * self.W + i).long()
        flat = img.reshape(-1)
        right, down = (1 if self.W > 1 else 0), (self.W if self.H > 1 else 0)
        top = torch.lerp(flat[at], flat[at + right], fu)
        val = torch.lerp(top, torch.lerp(flat[at + down], flat[at + down + right], fu), fv)
        return torch.where(inside, val, 0.0), inside, i, at, fu, fv, right, down

    def weights(self, k):
        """The cosine pre-weight (v, in_w) of view k: of the middle view of its group of nine."""
        T = self.inv[min(9 * (k // 9) + 4, self.N - 1)]
        j = torch.arange(self.H, device=self.dev, dtype=torch.float64)[:, None]
        i = torch.arange(self.L, device=self.dev, dtype=torch.float64) - (self.in_w / 2 if self.mirror else 0)
        at = [[T[r, 0] * i + T[r, 1] * j + w * T[r, 2] + T[r, 3] for r in range(4)] for w in (0.0, 1.0)]
        d2 = sum((at[0][r] / at[0][3] - at[1][r] / at[1][3]) ** 2 for r in range(3))
        return d2.min().sqrt() / d2[:, :self.in_w].sqrt()

    def filter(self, pre, k):
        """Ramp-filtered rows of (preprocessed, composited) frame k."""
        x, n, L = pre, self.in_w, self.L
        R = (L - n) // 2
        buf = torch.zeros((self.H, L), dtype=torch.float64, device=self.dev)
        buf[:, :n] = x * self.weights(k)
        ramp = torch.arange(R, device=self.dev, dtype=torch.float64) / max(R, 1)
        if self.mirror:
            buf[:, n:n + R] = x[:, n - 3:].mean(1, keepdim=True) * ((R - 1) / max(R, 1) - ramp)
        else:
            buf[:, L - R:] = x[:, :3].mean(1, keepdim=True) * ramp
        y = torch.fft.irfft(torch.fft.rfft(buf) * self.spectrum, n=L)
        y = y[:, self.W:2 * self.W] if self.mirror else y[:, :self.W]
        if self.c["offset"]:   # the z-filter
            y = 0.5 * y + 0.25 * torch.cat([y[:1], y[:-1]]) + 0.25 * torch.cat([y[1:], y[-1:]])
        return y

    def filter_transposed(self, ybar, k):
        """The transpose of filter() (no compositing, not mirrored) applied to ybar."""
        L, n = self.L, self.in_w
        R = (L - n) // 2
        g = torch.fft.irfft(torch.fft.rfft(torch.nn.functional.pad(ybar, (0, L - n))) * self.spectrum, n=L)
        ramp = torch.arange(R, device=self.dev, dtype=torch.float64) / max(R, 1)
        x = g[:, :n] * self.weights(k)
        x[:, :3] += (g[:, L - R:] * ramp).sum(1, keepdim=True) / 3
        return x

    def places(self, P, z0, z1):
        """u, v, W of the voxels of slices [z0, z1), and their coordinates."""
        c, t = self.c, dict(device=self.dev, dtype=torch.float64)
        vox = np.float32(c["vox"]).item()
        x, y, z = ((torch.arange(c[k], **t) - (c[k] - 1) / 2) * vox for k in "xyz")
        y, z = y[:, None], z[z0:z1, None, None]
        U, V, W = (P[r, 2] * z + (P[r, 0] * x + (P[r, 1] * y + P[r, 3])) for r in range(3))
        return U / W + 0.5, V / W + 0.5, W, (x, y, z)

    def frames(self, raw):
        pre = None
        if self.c["offset"]:
            pre = self.preprocess(raw)
        out = torch.empty((self.N, self.H, self.W), dtype=torch.float64, device=self.dev)
        for k in range(self.N):
            out[k] = self.filter(self.composite(pre, k) if pre is not None else self.preprocess(raw[k]), k)
        return out

    def backproject(self, q, P=None):
        """(sum of tapered samples, sum of tapers) of every voxel."""
        c, P = self.c, self.P if P is None else P
        q = q * self.taper[:, None, :]
        shape = (c["z"], c["y"], c["x"])
        S, C = (torch.zeros(shape, dtype=torch.float64, device=self.dev) for _ in range(2))
        slab = max(1, 2 ** 23 // (c["x"] * c["y"]))
        for z0 in range(0, c["z"], slab):
            z1 = min(c["z"], z0 + slab)
            for k in range(self.N):
                u, v, _, _ = self.places(P[k], z0, z1)
                val, inside, i, _, fu, _, right, _ = self._sample(q[k], u, v)
                S[z0:z1] += val
                i = i.long()
                C[z0:z1] += torch.where(inside, torch.lerp(self.taper[k][i], self.taper[k][i + right], fu), 0.0)
        return S, C

    def volume(self, raw):
        S, C = self.backproject(self.frames(raw))
        h = S / C * (1000.0 / np.float32(MU_WATER).item()) - 1000.0
        return torch.where(h > 300.0, h.clamp_max(8191.0), h)

    def gradient(self, p, theta, target):
        """vol, dL/dp and dL/dtheta of L = sum (vol - target)^2 over the voxels that some view sees."""
        th = torch.as_tensor(theta, device=self.dev, dtype=torch.float64).requires_grad_()
        moved = self.P @ _rigid(th)
        # the backprojector takes FP32 matrices
        P = moved.detach().float().double()
        q = torch.stack([self.filter(p[k].double(), k) for k in range(self.N)])
        S, C = self.backproject(q, P)
        vol = S / C
        bar = torch.nan_to_num(2 * (vol - target.double()))
        r = torch.where(C != 0, bar / C, 0.0)
        vol0 = torch.nan_to_num(vol)
        pbar = torch.empty((self.N, self.H, self.W), dtype=torch.float64, device=self.dev)
        Pbar = torch.zeros_like(P)
        for k in range(self.N):
            img = torch.zeros(self.H * self.W, dtype=torch.float64, device=self.dev)
            t = q[k] * self.taper[k]
            u, v, W, xyz = self.places(P[k], 0, self.c["z"])
            _, inside, i, at, fu, fv, right, down = self._sample(t, u, v)
            g = torch.where(inside, r, 0.0)
            for dx, dy, w in ((0, 0, (1 - fu) * (1 - fv)), (right, 0, fu * (1 - fv)), (0, down, (1 - fu) * fv),
                              (right, down, fu * fv)):
                img.index_add_(0, (at + dx + dy).reshape(-1), (g * w).reshape(-1))
            pbar[k] = self.filter_transposed(img.reshape(self.H, self.W) * self.taper[k], k)
            f = t.reshape(-1)
            a, b, d, e = f[at], f[at + right], f[at + down], f[at + down + right]
            tap = self.taper[k]
            i = i.long()
            gu = g / W * ((1 - fv) * (b - a) + fv * (e - d) - vol0 * (tap[i + right] - tap[i]))
            gv = g / W * ((1 - fu) * (d - a) + fu * (e - b))
            gw = -(gu * (u - 0.5) + gv * (v - 0.5))
            for row, m in enumerate((gu, gv, gw)):
                for col, s in enumerate((*xyz, 1.0)):
                    Pbar[k, row, col] = (m * s).sum()
        (moved * Pbar).sum().backward()
        return {"vol": vol, "p": pbar, "theta": th.grad}


def exact(case, seed):
    if case["do"] == "batch":
        out = []
        for k, c in enumerate(_scans(case)):
            P, frames = _matrices(c, seed + k)
            out.append(_Exact(c, P.astype(np.float32)).volume(_raw(c, seed + k, frames)))
        return out
    P, frames = _matrices(case, seed)
    P = P.astype(np.float32)
    x = _Exact(case, P)
    if case["do"] == "filter":
        n = case["chunk"]
        raw = _raw(dict(case, views=n), seed, tuple(f[:n] for f in frames))
        pre = -(raw.float().clamp_min(1.0) / BRIGHT).log()   # the call's own FP32 input
        return torch.stack([x.filter(pre[k].double(), k) for k in range(n)])
    raw = _raw(case, seed, frames)
    if case["do"] == "gradient":
        return x.gradient(x.preprocess(raw).float(), _motion(case, seed), _target(case, seed))
    vol = x.volume(raw)
    return vol.cpu().numpy() if case["do"] == "host" else vol
