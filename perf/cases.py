"""The work that a program has this engine do, as cases to be timed and checked.

A case is a dict of plain values; ``prepare`` makes what the program has in
hand (the tilt series, the geometry, buffers) and ``run`` is one pass through
``autom2_b200.tiltrec``.  As a program that reconstructs series after series
does, one Engine (and one Scheduler) is kept per process: a pass sets the
series' problem on it and then calls the method, so that geometry-dependent
weights belong to the pass.

Kinds:

* ``wbp``, ``fbp``: row filter and back-projection from zeros (the stack is
  filtered in place, so a pass works on a copy of it);
* ``sirt``, ``sart``, ``admm``: iterations from a zero volume;
* ``sirt16``: the stack quantised to FP16, SIRT with FP16 residuals;
* ``project``: forward projection of a volume with its weights;
* ``batch``: uneven series through the scheduler, WBP then SIRT each;
* ``resample``: area binning of a stack;
* ``bytes``: the byte output of a volume.

Geometries: ``ideal`` (single axis), ``shift`` (per-tilt shifts N(0, 1 px)),
``rot`` (XTILT 0.3 degrees and per-tilt in-plane rotations N(0, 0.5 degrees)).
"""
import math

import numpy as np
import torch

from autom2_b200 import tiltrec as T

MU, SOFT = 0.5, 0.02  # ADMM penalty and threshold


def listed():
    return [
        # A binned overview series: WBP of 41 tilts of 256 x 256, where launches count.
        dict(name="wbp_256", kind="wbp", geo="shift", layout=0, nx=256, ny=256, nt=41, th=64),
        # The ordinary WBP of a full series at half the camera's resolution.
        dict(name="wbp_1024", kind="wbp", geo="shift", layout=0, nx=1024, ny=1024, nt=81, th=256),
        # Iterative reconstruction of a binned series, thickness as it comes.
        dict(name="sirt_512", kind="sirt", geo="shift", layout=0, nx=512, ny=512, nt=41, th=97, iters=10),
        # The headline geometry: XTILT and in-plane rotations, 61 tilts of 1024 x 1024.
        dict(name="sirt_1024_rot", kind="sirt", geo="rot", layout=0, nx=1024, ny=1024, nt=61, th=256, iters=3),
        # Large images in the Z layout with 16-bit storage.
        dict(name="sirt16_2048_z", kind="sirt16", geo="ideal", layout=1, nx=2048, ny=2048, nt=61, th=128, iters=2),
        # A cropped field of view (odd sizes) re-projected, as in a residual check.
        dict(name="project_725_rot", kind="project", geo="rot", layout=0, nx=725, ny=517, nt=45, th=131),
        # FBP of an odd-sized field of view.
        dict(name="fbp_717", kind="fbp", geo="shift", layout=0, nx=717, ny=523, nt=61, th=150),
        # SART, whose updates go tilt by tilt.
        dict(name="sart_512", kind="sart", geo="shift", layout=0, nx=512, ny=512, nt=61, th=128, iters=1),
        # ADMM in the Z layout.
        dict(name="admm_256_z", kind="admm", geo="shift", layout=1, nx=256, ny=256, nt=61, th=64, iters=2),
        # Uneven series through the scheduler with 16-bit storage.
        dict(name="batch_4", kind="batch", geo="shift", layout=0, nx=512, ny=512, nt=41, th=90, jobs=4, iters=2),
        # Binning of full camera frames before the reconstruction.
        dict(name="resample_4096", kind="resample", nx=4096, ny=4096, nt=10, bin=4),
        # Byte output of the reconstruction, slabs of 64 rows.
        dict(name="bytes_1024", kind="bytes", nx=1024, ny=1024, th=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wbp", "wbp", "fbp", "sirt", "sirt", "sirt16", "project", "sart", "admm",
                       "batch", "resample", "bytes"])
    if kind == "resample":
        return dict(kind=kind, nx=_log_int(rng, 512, 4096), ny=_log_int(rng, 512, 4096),
                    nt=rng.randint(2, 10), bin=rng.choice([2, 3, 4, 4, 6, 8]))
    if kind == "bytes":
        return dict(kind=kind, nx=_log_int(rng, 256, 1024), ny=_log_int(rng, 256, 1024),
                    th=_log_int(rng, 48, 256))
    c = dict(kind=kind, geo=rng.choice(["ideal", "shift", "shift", "rot"]),
             layout=rng.choice([0, 0, 1]), nx=_log_int(rng, 192, 1024), ny=_log_int(rng, 192, 1024),
             nt=rng.choice([41, 45, 61, 81]), th=_log_int(rng, 48, 256))
    if rng.random() < 0.6:  # most cameras' and crops' rows are whole groups of 8 pixels
        c["nx"] -= c["nx"] % 8
    if kind in ("sirt", "sirt16"):
        c["iters"] = rng.choice([2, 3, 5])
    elif kind == "sart":
        c["iters"], c["th"] = 1, min(c["th"], 128)
    elif kind == "admm":
        c.update(iters=1, th=min(c["th"], 96), nx=min(c["nx"], 512), ny=min(c["ny"], 512))
    elif kind == "batch":  # the scheduler takes rows of whole 16-byte groups
        c.update(geo=rng.choice(["ideal", "shift", "rot"]), jobs=rng.randint(2, 4), iters=2,
                 nx=min(c["nx"], 512) // 8 * 8, ny=min(c["ny"], 512), th=min(c["th"], 90))
    while c["nx"] * c["ny"] * c["th"] * c["nt"] * (c.get("iters", 1) + 1) > 6e10:
        c["th"] = max(32, c["th"] // 2)
        c["ny"] = max(64, c["ny"] * 3 // 4)
    return c


# --------------------------------------------------------------- inputs


def _coeffs(case, rng):
    """[nt][8] coefficients of tilts over +-60..70 degrees."""
    nt = case["nt"]
    amax = 60.0 if case["geo"] != "shift" else rng.uniform(60.0, 70.0)
    th = np.deg2rad(np.linspace(-amax, amax, nt))
    al = np.deg2rad(-0.3) if case["geo"] == "rot" else 0.0
    a1, a3 = np.cos(th), -np.sin(th)
    z = np.zeros(nt)
    a = np.stack([z, a1, -a3 * np.sin(al), a3 * np.cos(al)], 1)
    b = np.stack([z, z, z + np.cos(al), z + np.sin(al)], 1)
    if case["geo"] == "rot":
        psi = np.deg2rad(rng.normal(0.0, 0.5, nt))[:, None]
        a, b = np.cos(psi) * a - np.sin(psi) * b, np.sin(psi) * a + np.cos(psi) * b
    if case["geo"] == "shift":
        a[:, 0] += rng.normal(0.0, 1.0, nt)
        b[:, 0] += rng.normal(0.0, 1.0, nt)
    return np.ascontiguousarray(np.concatenate([a, b], 1))


def _texture(shape, gen):
    """Smooth features over the last two axes plus noise, float32 on the GPU."""
    n, h, w = shape
    low = torch.randn((n, 1, max(2, h // 16), max(2, w // 16)), generator=gen, device="cuda")
    x = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=False)[:, 0]
    return x + 0.3 * torch.randn(shape, generator=gen, device="cuda")


def _stack(case, gen):
    return (_texture((case["nt"], case["ny"], case["nx"]), gen) * 2.0 + 8.0).contiguous()


def _vol_shape(case):
    nx, ny, th = case["nx"], case["ny"], case["th"]
    return (ny, th, nx) if case["layout"] == 0 else (th, ny, nx)


def _jobs(case):
    """The series of a batch: the case's own and uneven others."""
    sizes = [(1.0, 1.0, 0), (0.75, 0.7, 0), (1.0, 0.5, 20), (0.5, 1.0, 0)]
    out = []
    for k in range(case["jobs"]):
        s, d, more = sizes[k]
        out.append(dict(case, nx=max(64, int(case["nx"] * s) // 8 * 8), ny=max(64, int(case["ny"] * s)),
                        th=max(24, int(case["th"] * d)), nt=case["nt"] + more))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "resample":
        s["stack"] = _stack(case, gen)
        return s
    if kind == "bytes":
        s["vol"] = _texture((case["ny"], case["th"], case["nx"]), gen).contiguous()
        _engine()
        return s
    if kind == "batch":
        s["series"] = []
        for j in _jobs(case):
            s["series"].append(dict(coeff=_coeffs(j, rng), proj=_stack(j, gen), layout=j["layout"],
                                    vol=torch.zeros(_vol_shape(j), device="cuda")))
        _scheduler()
        torch.cuda.synchronize()  # the scheduler's streams are its own
        return s
    s["coeff"] = _coeffs(case, rng)
    if kind == "project":
        s["vol"] = (_texture(_vol_shape(case), gen).clamp(min=0) * 0.5).contiguous()
        s["val"] = torch.zeros((case["nt"], case["ny"], case["nx"]), device="cuda")
        s["wt"] = torch.zeros_like(s["val"])
    else:
        s["proj"] = _stack(case, gen)
        s["vol"] = torch.zeros(_vol_shape(case), device="cuda")
        if kind in ("wbp", "fbp"):
            s["rows"] = torch.empty_like(s["proj"])
    _engine()
    return s


_kept = {}


def _engine():
    if "engine" not in _kept:
        _kept["engine"] = T.Engine(torch.cuda.current_device())
    return _kept["engine"]


def _scheduler():
    if "sched" not in _kept:
        _kept["sched"] = T.Scheduler(torch.cuda.current_device(), 0, "f16", "f16")
    return _kept["sched"]


def _problem(case, coeff):
    """The process's Engine, set to the series."""
    e = _engine()
    e.set_problem(case["nx"], case["ny"], case["nt"], case["th"], coeff, case["layout"])
    return e


# ----------------------------------------------------------------- a pass


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "resample":
        return T.resample_bin(s["stack"], case["bin"])
    if kind == "bytes":
        return _engine().volume_to_bytes(s["vol"], 64 * case["th"] * case["nx"])
    if kind == "batch":
        d = _scheduler()
        for j in s["series"]:
            d.submit(d.job(j["proj"], j["vol"], j["coeff"], j["layout"], wbp=True,
                           sirt_iters=case["iters"], gamma=0.5))
        d.drain()
        return [j["vol"] for j in s["series"]]
    e = _problem(case, s["coeff"])
    if kind == "project":
        s["val"].zero_()
        s["wt"].zero_()
        e.forward_project(s["vol"], s["val"], s["wt"])
        return s["val"], s["wt"]
    vol = s["vol"].zero_()
    if kind == "wbp":
        e.wbp(s["rows"].copy_(s["proj"]), vol)
    elif kind == "fbp":
        e.filter_fbp(s["rows"].copy_(s["proj"]), 0)
        e.backproject(s["rows"], vol)
    elif kind == "sirt":
        e.sirt(s["proj"], vol, case["iters"], 0.5)
    elif kind == "sirt16":
        p16, scale = e.quantize(s["proj"], torch.float16)
        e.sirt_lp(p16, scale, vol, case["iters"], 0.5, "f16")
    elif kind == "sart":
        e.sart(s["proj"], vol, case["iters"], 0.2)
    elif kind == "admm":
        e.admm(s["proj"], vol, case["iters"], 1, MU, SOFT)
    return vol


def work(case):
    """Bytes: inputs read once, results written once.  Flops: 14 for each
    voxel and tilt of a projection (two weights, four taps, the sum), and a
    filter's as its FFTs or taps take."""
    kind = case["kind"]
    if kind == "resample":
        n = case["nx"] * case["ny"] * case["nt"]
        return dict(bytes=4.0 * n * (1 + 1 / case["bin"] ** 2), flops=2.0 * n)
    if kind == "bytes":
        n = case["nx"] * case["ny"] * case["th"]
        return dict(bytes=5.0 * n, flops=8.0 * n)
    total = dict(bytes=0.0, flops=0.0)
    for c in _jobs(case) if kind == "batch" else [case]:
        p, v = c["nx"] * c["ny"] * c["nt"], c["nx"] * c["ny"] * c["th"]
        upd = 14.0 * v * c["nt"]
        total["bytes"] += 4.0 * (p + v)
        if kind == "project":
            total["bytes"] += 4.0 * p
            total["flops"] += 2 * upd
        if kind in ("wbp", "batch"):
            total["flops"] += upd + 10.0 * p * math.log2(4 * c["nx"])
        elif kind == "fbp":
            total["flops"] += upd + 2.0 * 251 * p
        if kind in ("sirt", "sirt16", "sart", "batch"):
            total["flops"] += 2 * upd * c["iters"]
        elif kind == "admm":
            total["flops"] += upd * (1 + 6 * c["iters"])
    return total


# ------------------------------------------------- the same in 64 bits


class _Exact:
    """The operators of one series in float64 with plain torch, rows of the
    volume in pieces of bounded size.  Volumes are [ny][th][nx]."""

    def __init__(self, case, coeff):
        self.nx, self.ny, self.nt, self.th = (case[k] for k in ("nx", "ny", "nt", "th"))
        self.c = coeff
        self.o = T.default_origin(case["layout"], self.nx, self.ny, self.th)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.step = max(1, int(2.4e7 // (self.nx * self.th)))

    def zeros(self):
        return torch.zeros((self.ny, self.th, self.nx), dtype=torch.float64, device=self.dev)

    def pieces(self):
        for y0 in range(0, self.ny, self.step):
            yield slice(y0, min(self.ny, y0 + self.step))

    def taps(self, t, rows):
        """(pixel index, weight) of the four in-image taps of each voxel."""
        ox, oy, oz = self.o
        f = dict(dtype=torch.float64, device=self.dev)
        x = torch.arange(self.nx, **f) - ox
        y = (torch.arange(rows.start, rows.stop, **f) - oy)[:, None, None]
        z = (torch.arange(self.th, **f) - oz)[:, None]
        k = [float(v) for v in self.c[t]]
        u = k[0] + k[1] * x + k[2] * y + k[3] * z + ox
        v = k[4] + k[5] * x + k[6] * y + k[7] * z + oy
        u0, v0 = u.floor(), v.floor()
        dx, dy = u - u0, v - v0
        u0, v0 = u0.to(torch.int32), v0.to(torch.int32)
        for j, wy in ((v0, 1 - dy), (v0 + 1, dy)):
            inj = (j >= 0) & (j < self.ny)
            for i, wx in ((u0, 1 - dx), (u0 + 1, dx)):
                ok = inj & (i >= 0) & (i < self.nx)
                w = torch.where(ok, wx * wy, 0.0)
                yield (j.clamp(0, self.ny - 1) * self.nx + i.clamp(0, self.nx - 1)).long(), w

    def gather(self, img, t, rows):
        s = c = 0.0
        img = img.reshape(-1)
        for n, w in self.taps(t, rows):
            s = s + w * img[n]
            c = c + w
        return s, c

    def project(self, vol, t):
        val = torch.zeros(self.ny * self.nx, dtype=torch.float64, device=self.dev)
        wt = torch.zeros_like(val)
        for rows in self.pieces():
            for n, w in self.taps(t, rows):
                w = w.expand(n.shape).reshape(-1)
                val.index_add_(0, n.reshape(-1), w * vol[rows].reshape(-1))
                wt.index_add_(0, n.reshape(-1), w)
        return val.reshape(self.ny, self.nx), wt.reshape(self.ny, self.nx)

    def normalised(self, img, t, vol, gamma):
        for rows in self.pieces():
            s, c = self.gather(img, t, rows)
            vol[rows] += torch.where(c != 0, s / torch.where(c != 0, c, 1.0), 0.0) * gamma

    def residual(self, p, vol, t):
        val, wt = self.project(vol, t)
        return p.double() - torch.where(wt != 0, val / torch.where(wt != 0, wt, 1.0), val)

    def backproject(self, proj, vol):
        for t in range(self.nt):
            self.normalised(proj[t].double(), t, vol, 1.0)
        return vol

    def sirt(self, proj, vol, iters, gamma):
        for _ in range(iters):
            s, c = self.zeros(), self.zeros()
            for t in range(self.nt):
                r = self.residual(proj[t], vol, t)
                for rows in self.pieces():
                    a, b = self.gather(r, t, rows)
                    s[rows] += a
                    c[rows] += b
            vol += torch.where(c != 0, s / torch.where(c != 0, c, 1.0), 0.0) * gamma
        return vol

    def sart(self, proj, vol, iters, gamma):
        for _ in range(iters):
            for t in range(self.nt):
                self.normalised(self.residual(proj[t], vol, t), t, vol, gamma)
        return vol

    def admm(self, proj, vol, outer):
        def adjoint(imgs):
            out = self.zeros()
            for t in range(self.nt):
                for rows in self.pieces():
                    out[rows] += self.gather(imgs[t].double(), t, rows)[0]
            return out

        def apply(x):
            def normal(t):
                val, wt = self.project(x, t)
                return torch.where(wt > 1e-5, val / torch.where(wt > 1e-5, wt, 1.0), 0.0)
            return adjoint([normal(t) for t in range(self.nt)]) + MU * x

        atb, u, d = adjoint(proj), self.zeros(), self.zeros()
        for _ in range(outer):
            atb += (u - d) * MU
            r = atb - apply(vol)
            h = apply(r)
            vol += ((r * r).sum() / (h * r).sum()) * r
            v = vol + d
            u = torch.where(v < -SOFT, v + SOFT, torch.where(v > SOFT, v - SOFT, 0.0))
            d += vol - u
        return vol


def _weighted(proj):
    """The R-weighting row filter in float64: the row padded by a ramp back to
    its first sample, its spectrum weighted, cropped, divided by the length."""
    nx = proj.shape[-1]
    n = nx + nx // 10
    r, sg = int(math.floor(np.float32(n) * np.float32(0.05))), 0.5 * n
    w = np.array([0.2 if k == 0 else k if k <= r else r * math.exp(-((k - r) / sg) ** 2)
                  for k in range(n // 2 + 1)])
    w = torch.from_numpy(w).to(proj.device)
    j = torch.arange(nx, n, device=proj.device, dtype=torch.float64)
    out = torch.empty(proj.shape, dtype=torch.float64, device=proj.device)
    for t in range(proj.shape[0]):
        x = proj[t].double()
        pad = ((j - nx + 1) * x[:, :1] + (n - j) * x[:, -1:]) / (n - nx + 1)
        f = torch.fft.rfft(torch.cat([x, pad], 1), dim=1) * w
        out[t] = torch.fft.irfft(f, n=n, dim=1)[:, :nx] * (n / nx)
    return out


def _shepp_logan(proj):
    """The FBP row filter in float64: 251 taps over the row padded by an edge
    sample and mirrored about its right end."""
    nx, taps = proj.shape[-1], 251
    length = nx + 252
    while True:
        m = length
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            break
        length += 1
    n = np.arange(taps) - taps // 2
    f = torch.from_numpy((-2.0 / (np.pi * (4.0 * n * n - 1.0))).astype(np.float32).astype(np.float64))
    f = f.to(proj.device)
    out = torch.empty(proj.shape, dtype=torch.float64, device=proj.device)
    for t in range(proj.shape[0]):
        x = proj[t].double()
        x = torch.cat([x[:, :1], x, x[:, -1:]], 1)
        x = torch.cat([x, x.flip(1)], 1)[:, :length]
        x = torch.nn.functional.pad(x, (0, length - x.shape[1]))
        spec = torch.fft.rfft(x, dim=1) * torch.fft.rfft(torch.nn.functional.pad(f, (0, length - taps)))
        out[t] = torch.fft.irfft(spec, n=length, dim=1)[:, 126:126 + nx]
    return out


def _binned(stack, b):
    def axis(n):
        d = n // b
        edge = torch.arange(d + 1, dtype=torch.float64, device=stack.device) * (n / d)
        i = torch.arange(n, dtype=torch.float64, device=stack.device)
        lo = torch.maximum(edge[:-1, None], i)
        hi = torch.minimum(edge[1:, None].clamp(max=n), i + 1)
        return (hi - lo).clamp(min=0) / (n / d)

    wy, wx = axis(stack.shape[1]), axis(stack.shape[2])
    return torch.stack([wy @ s.double() @ wx.T for s in stack])


def exact(case, seed):
    kind = case["kind"]
    if kind == "bytes":
        return None
    parts = _jobs(case) if kind == "batch" else [case]
    if kind != "resample":
        passes = {"wbp": 0.3, "fbp": 0.3, "project": 2.0, "sart": 2.5, "admm": 13.0,
                  "sirt": 2.5, "sirt16": 2.5, "batch": 2.8}[kind]
        cost = sum(c["nx"] * c["ny"] * c["th"] * c["nt"] for c in parts) * passes
        if cost * (case.get("iters", 1) if kind != "admm" else 1) > 3.5e10:
            return None
    s = prepare(case, seed)
    if kind == "resample":
        return _binned(s["stack"], case["bin"])

    def placed(vol, layout):
        return vol if layout == 0 else vol.permute(1, 0, 2).contiguous()

    if kind == "batch":
        out = []
        for c, j in zip(parts, s["series"]):
            e = _Exact(c, j["coeff"])
            vol = e.backproject(_weighted(j["proj"]), e.zeros())
            out.append(placed(e.sirt(j["proj"], vol, case["iters"], 0.5), j["layout"]))
        return out
    e = _Exact(case, s["coeff"])
    if kind == "project":
        vol = s["vol"] if case["layout"] == 0 else s["vol"].permute(1, 0, 2)
        both = [e.project(vol.double(), t) for t in range(e.nt)]
        return torch.stack([v for v, _ in both]), torch.stack([w for _, w in both])
    if kind == "wbp":
        vol = e.backproject(_weighted(s["proj"]), e.zeros())
    elif kind == "fbp":
        vol = e.backproject(_shepp_logan(s["proj"]), e.zeros())
    elif kind in ("sirt", "sirt16"):
        vol = e.sirt(s["proj"], e.zeros(), case["iters"], 0.5)
    elif kind == "sart":
        vol = e.sart(s["proj"], e.zeros(), case["iters"], 0.2)
    else:
        vol = e.admm(s["proj"], e.zeros(), case["iters"])
    return placed(vol, case["layout"])
