"""The calls that a user of the library has it do, at the sizes they come in, as timed cases.

Each case names one call through the Python binding (fa_b200.py) and its sizes; `prepare` makes the
inputs and the handles that a program keeps between calls, `run` makes the call once and returns
what it returned, and `exact` computes the same outputs in FP64 with torch alone. Kinds of call:

  evaluate   Frame.get_error + get_jacobian at one displacement set (the warper's two calls per
             optimiser step when the caller drives the solve)
  warp       Frame.warp: the realigned image of one registered frame
  reference  Reference + hessian: a new reference volume (gradient, Hessian, its factor)
  shift      Correlator.compute_shift_device: one volume's rigid shift
  solve      Frame.align: one registered frame's non-rigid solve
  align      Aligner.add_frames(_device): raw frames in, displacements out, a batch at a time
  results    Aligner.results: correlations and coverage of aligned frames
  serve      Server.submit_ptr / wait: frames of several acquisitions in flight at once

Contexts use the default configuration (no timing-based tile choice: with it the order of summation,
and so the last bits, would depend on what the timing of that process found).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "frame-aligner_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import fa_b200 as fa  # noqa: E402

DEV = "cuda"
TYPES = {"f32": torch.float32, "u16": torch.uint16}


def listed():
    return [
        # The smallest call: one evaluation of a 256 x 256 plane (a caller's own optimiser makes one
        # per step). Launches and round trips.
        dict(name="evaluate_plane", kind="evaluate", nz=1, ny=256, nx=256, nD=10, mixed=False),
        # The same for a volume stored in mixed precision, the headline volume size.
        dict(name="evaluate_volume", kind="evaluate", nz=16, ny=512, nx=512, nD=32, mixed=True),
        # A camera region of odd size: rows that are no multiple of four voxels.
        dict(name="evaluate_odd", kind="evaluate", nz=5, ny=301, nx=423, nD=20, mixed=False),
        # The realigned image of one plane, read back to the host.
        dict(name="warp_plane", kind="warp", nz=1, ny=512, nx=512, nD=32, mixed=False),
        # A new acquisition: gradient and Hessian of its reference volume.
        dict(name="reference_volume", kind="reference", nz=16, ny=512, nx=512, nD=32, mixed=True),
        # One volume's rigid shift (FP64 phase correlation).
        dict(name="shift_volume", kind="shift", nz=16, ny=512, nx=512),
        # One plane's solve, frame by frame, FP32: an interactive single-frame call.
        dict(name="solve_plane", kind="solve", nz=1, ny=512, nx=512, nD=32, mixed=False),
        # A short time series of small planes: 20 raw uint16 frames.
        dict(name="align_planes", kind="align", nz=1, ny=256, nx=256, nD=10, mixed=True, frames=20, dtype="u16",
             host=False, binning=1),
        # The headline workload: 50 raw volumes in device memory.
        dict(name="align_volumes", kind="align", nz=16, ny=512, nx=512, nD=32, mixed=True, frames=50, dtype="u16",
             host=False, binning=1),
        # The same call fed from page-locked host memory, as an acquisition computer feeds it.
        dict(name="align_host", kind="align", nz=16, ny=512, nx=512, nD=32, mixed=True, frames=16, dtype="u16",
             host=True, binning=1),
        # The largest volumes.
        dict(name="align_large", kind="align", nz=64, ny=1024, nx=1024, nD=64, mixed=True, frames=3, dtype="u16",
             host=False, binning=1),
        # Three acquisitions of different sizes served at once, eight frames of each in flight.
        dict(name="serve_mix", kind="serve", sizes="1x256x256 1x512x512 8x512x512", frames=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _control_points(nz, ny):
    """16 per 256 lines of a plane, at least two per plane of a stack, at most 64."""
    return int(min(64, max(4, 16 * ny // 256, 2 * nz if nz > 1 else 0)))


def _size(rng, most, least=64):
    """A volume of at most `most` voxels: a plane or a stack, of even, odd or power-of-two sides."""
    while True:
        nz = 1 if rng.random() < 0.4 else rng.choice([2, 3, 4, 5, 8, 11, 16, 20, 32])
        form = rng.random()
        if form < 0.4:
            ny, nx = 2 ** rng.randint(6, 10), 2 ** rng.randint(6, 10)
        elif form < 0.7:
            ny, nx = _log(rng, 64, 1024), 4 * _log(rng, 16, 256)
        else:
            ny, nx = _log(rng, 64, 1024), _log(rng, 64, 1024)
        if nz * ny * nx <= most and nz < ny and min(ny, nx) >= least:
            return dict(nz=nz, ny=ny, nx=nx)


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "warp", "reference", "shift", "solve", "align", "align", "align", "serve"])
    if kind == "serve":
        a = [_size(rng, 1 << 21, 128) for _ in range(rng.randint(1, 3))]
        return dict(kind=kind, sizes=" ".join("%dx%dx%d" % (s["nz"], s["ny"], s["nx"]) for s in a),
                    frames=rng.randint(2, 12))
    s = _size(rng, 1 << 23)
    c = dict(kind=kind, **s)
    if kind == "shift":
        return c
    c["nD"] = _control_points(s["nz"], s["ny"])
    c["mixed"] = rng.random() < 0.6
    if kind == "align":
        voxels = s["nz"] * s["ny"] * s["nx"]
        c["frames"] = _log(rng, 1, max(1, min(64, (1 << 26) // voxels)))
        c["dtype"] = rng.choice(["u16", "u16", "f32"])
        c["host"] = rng.random() < 0.3
        c["binning"] = 2 if rng.random() < 0.15 else 1
    return c


# ---------------------------------------------------------------- inputs --------------------------


def _sizes(case):
    if case["kind"] == "serve":
        out = []
        for s in case["sizes"].split():
            nz, ny, nx = (int(v) for v in s.split("x"))
            out.append(dict(kind="serve", nz=nz, ny=ny, nx=nx, nD=_control_points(nz, ny)))
        return out
    return [case]


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rate(shape, g):
    """A photon rate of mean 20: Gaussian blobs of three widths on a background."""
    nz, ny, nx = shape
    n = max(30, int(200 * ny * nx / 65536) * (1 if nz == 1 else max(1, nz // 4)))
    freq = [torch.fft.fftfreq(s, device=DEV) for s in (nz, ny)] + [torch.fft.rfftfreq(nx, device=DEV)]
    r2 = freq[1][:, None] ** 2 + freq[2][None, :] ** 2
    spec = 0
    for sigma in (1.5, 3.0, 6.0):
        seeds = torch.zeros(nz * ny * nx, device=DEV)
        at = torch.randint(0, nz * ny * nx, (n // 3 + 1,), generator=g, device=DEV)
        seeds.scatter_add_(0, at, (5 + 45 * torch.rand(at.shape, generator=g, device=DEV)) * sigma ** 2)
        gauss = torch.exp(-2 * math.pi ** 2 * sigma ** 2 * r2)
        if nz > 1:
            gauss = gauss * torch.exp(-2 * math.pi ** 2 * 1.5 ** 2 * freq[0] ** 2)[:, None, None]
        spec = spec + torch.fft.rfftn(seeds.view(nz, ny, nx)) * gauss
    blobs = torch.fft.irfftn(spec, s=(nz, ny, nx)).clamp_(min=0)
    return 2.0 + blobs * (18.0 / blobs.mean())


def _walk(c, g):
    """A clipped random walk of the displacement over the control points, pixels (x, y, z), about a
    drift of the whole frame (a served stream's frames follow one another and stay near)."""
    n = c["nD"]
    r = torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float64).cpu().numpy()
    drift = torch.rand(3, generator=g, device=DEV, dtype=torch.float64).cpu().numpy() * 2 - 1
    deep = min(1.0, c["nz"] / 16) if c["nz"] > 1 else 0.0
    step, bound = np.array([0.8, 0.8, 0.3 * deep]), np.array([3.0, 3.0, deep])
    far = 0.0 if c["kind"] == "serve" else min(6.0, 0.03 * min(c["ny"], c["nx"]))
    return np.round(drift * np.array([far, far, 0.0])) + _clipped(r * step, bound)


def _clipped(steps, bound):
    out, cur = np.empty_like(steps), np.zeros(steps.shape[1])
    for k, s in enumerate(steps):
        cur = np.clip(cur + s, -bound, bound)
        out[k] = cur
    return out


def _scan(c):
    return fa.scan_params(1.0, 1.01, c["ny"] * 1.01, c["nx"], c["ny"], c["nz"])


def _times(c, dtype):
    """The control-point coordinate of every voxel: q = t / stack * (nD - 1), the scan's own timing."""
    nz, ny, nx, nD = c["nz"], c["ny"], c["nx"], c["nD"]
    frame = ny * 1.01
    between = frame  # from the start of one plane to the start of the next
    stack = (nz - 1) * between + frame
    z, y, x = (torch.arange(s, device=DEV, dtype=dtype) for s in (nz, ny, nx))
    t = (z * between)[:, None, None] + (y * 1.01)[None, :, None] + (x * (1.0 / nx))[None, None, :]
    return t / stack * (nD - 1)


def _displacement(c, D, dtype):
    """Interval, fraction within it and displacement (x, y, z) of every voxel."""
    q = _times(c, dtype)
    i = q.floor().long().clamp_(max=c["nD"] - 2)
    f = q - i
    Dt = torch.as_tensor(D, device=DEV, dtype=dtype)
    d = [Dt[i, k] + f * (Dt[i + 1, k] - Dt[i, k]) for k in range(3 if c["nz"] > 1 else 2)]
    return i, f, d


def _frame(c, rate, D, g):
    """Poisson photon counts of the scene displaced along the scan: frame(x) = rate(x - d(t(x)))."""
    nz, ny, nx = rate.shape
    _, _, d = _displacement(c, D, torch.float32)
    gx = (torch.arange(nx, device=DEV)[None, None, :] - d[0]) * (2 / (nx - 1)) - 1
    gy = (torch.arange(ny, device=DEV)[None, :, None] - d[1]) * (2 / (ny - 1)) - 1
    if nz > 1:
        gz = (torch.arange(nz, device=DEV)[:, None, None] - d[2]) * (2 / (nz - 1)) - 1
        grid = torch.stack([gx, gy, gz], -1)[None]
        lam = torch.nn.functional.grid_sample(rate[None, None], grid, padding_mode="border", align_corners=True)
    else:
        grid = torch.stack([gx, gy], -1)
        lam = torch.nn.functional.grid_sample(rate[None], grid, mode="bicubic", padding_mode="border",
                                              align_corners=True)
    return torch.poisson(lam.reshape(nz, ny, nx).clamp_(min=0), generator=g)


def _inputs(c, seed, frames):
    """Reference counts (FP32), raw frames (FP32) and their true displacements, on the GPU."""
    g = _generator(seed)
    rate = _rate((c["nz"], c["ny"], c["nx"]), g)
    reference = torch.poisson(rate * 16, generator=g) / 16  # the mean of 16 frames
    raw, D = [], []
    for _ in range(frames):
        D.append(_walk(c, g))
        raw.append(_frame(c, rate, D[-1], g))
    return reference, raw, D


def _stored(frame, dtype):
    """A raw frame as the acquisition delivers it."""
    return frame if dtype == "f32" else frame.to(torch.int32).to(torch.uint16)


def _rigid(D):
    """The rigid start that a correlation would give: the mean displacement in whole pixels."""
    return np.round(D.mean(axis=0)) + 0.0


def _precision(c):
    return fa.PREC_MIXED if c["mixed"] else fa.PREC_F32


def prepare(case, seed):
    kind = case["kind"]
    ctx = fa.Context(0)
    st = dict(case, ctx=ctx)
    if kind == "serve":
        server = fa.Server(ctx)
        st.update(server=server, order=[], keep=[])
        per = []
        for j, c in enumerate(_sizes(case)):
            reference, raw, _ = _inputs(c, seed * 16 + j, case["frames"])
            a = server.add_acquisition(reference.cpu().numpy(), _scan(c), nD=c["nD"])
            server.reserve(a, case["frames"])
            frames = [_stored(r, "u16") for r in raw]
            st["keep"] += frames
            per.append([(a, f.data_ptr()) for f in frames])
        st["order"] = [f for turn in zip(*per) for f in turn]
        torch.cuda.synchronize()
        return st
    c = dict(case)
    if kind == "shift":
        c["nD"] = _control_points(c["nz"], c["ny"])
        reference, raw, _ = _inputs(c, seed, 1)
        st.update(correlator=fa.Correlator(ctx, reference.cpu().numpy()), volume=raw[0])
        torch.cuda.synchronize()
        return st
    if kind == "reference":
        reference, _, _ = _inputs(c, seed, 0)
        st.update(reference=reference + 1, scan=_scan(c))
        torch.cuda.synchronize()
        return st
    n = case.get("frames", 1)
    reference, raw, D = _inputs(c, seed, n)
    if kind == "align":
        aligner = fa.Aligner(ctx, spatial_binning=case["binning"], nD=c["nD"], precision=_precision(c))
        aligner.set_reference(reference.cpu().numpy(), _scan(c))
        frames = [_stored(r, case["dtype"]) for r in raw]
        if case["host"]:
            pinned = [torch.empty(f.shape, dtype=f.dtype, pin_memory=True) for f in frames]
            for p, f in zip(pinned, frames):
                p.copy_(f)
            frames = pinned
            st["host_frames"] = [p.numpy() for p in pinned]
        torch.cuda.synchronize()
        st.update(aligner=aligner, frames_data=frames, ptrs=[f.data_ptr() for f in frames],
                  code=fa.U16 if case["dtype"] == "u16" else fa.F32)
        return st
    ref = fa.Reference(ctx, (reference + 1).cpu().numpy(), c["nD"], _scan(c), _precision(c))
    frame = (raw[0] + 1).contiguous()
    torch.cuda.synchronize()
    st.update(ref=ref, frame=fa.Frame(ref, device_ptr=frame.data_ptr(), dtype=fa.F32), rigid=_rigid(D[0]),
              D=0.9 * D[0] + 0.05)
    if c["nz"] == 1:
        st["D"][:, 2] = 0.0
    return st


# ---------------------------------------------------------------- the calls -----------------------


def run(s):
    kind = s["kind"]
    if kind == "evaluate":
        f = s["frame"].get_error(s["D"])
        return {"f": np.array([f]), "jacobian": s["frame"].get_jacobian(s["D"])}
    if kind == "warp":
        return s["frame"].warp(s["D"])
    if kind == "reference":
        ref = fa.Reference(s["ctx"], None, s["nD"], s["scan"], _precision(s), device_ptr=s["reference"].data_ptr(),
                           shape=(s["nz"], s["ny"], s["nx"]))
        H = ref.hessian()
        ref.close()
        return H
    if kind == "shift":
        return s["correlator"].compute_shift_device(s["volume"].data_ptr())
    if kind == "solve":
        D, stats = s["frame"].align(s["rigid"])
        return {"D": D, "f": np.array([stats["f_final"]])}
    if kind == "align":
        if s["host"]:
            D, stats = s["aligner"].add_frames(s["host_frames"])
        else:
            D, stats = s["aligner"].add_frames_device(s["ptrs"], s["code"], len(s["ptrs"]))
        return {"D": D, "f": np.array([t["f_final"] for t in stats])}
    if kind == "serve":
        tickets = [s["server"].submit_ptr(a, p, True) for a, p in s["order"]]
        got = [s["server"].wait(t) for t in tickets]
        return {"D": np.concatenate([g[0] for g in got]), "f": np.array([g[1]["f_final"] for g in got])}
    raise ValueError(kind)


# ---------------------------------------------------------------- what cannot be done without -----


def work(case):
    """Each input read once and each output written once. Operations: a correlation is a real 3-D
    DFT and its inverse; an evaluation's trilinear sample, error and two control points' gradient
    terms are about 45 a voxel; a solve needs at least three (two starting points, one step)."""
    kind = case["kind"]
    nbytes, flops = 0.0, 0.0
    for c in _sizes(case):
        n = c["nz"] * c["ny"] * c["nx"]
        P = c.get("nD", 0) * (3 if c["nz"] > 1 else 2)
        ev, fft = 45.0 * n, 5.0 * n * math.log2(n)
        frames = case.get("frames", 1)
        elem = 2 if kind == "serve" or case.get("dtype") == "u16" else 4
        if kind == "evaluate":
            nbytes += n * ((2 + 8) if case["mixed"] else (4 + 16)) + 8 * P
            flops += ev
        elif kind == "warp":
            nbytes += n * ((2 + 4) if case["mixed"] else (4 + 4))
            flops += 20.0 * n
        elif kind == "reference":
            nbytes += n * (4 + 4 + 12 + (8 if case["mixed"] else 0)) + 8 * P * P
            flops += 70.0 * n
        elif kind == "shift":
            nbytes += n * 4 + 8 * n
            flops += fft
        elif kind == "solve":
            nbytes += n * ((2 + 8) if case["mixed"] else (4 + 16)) + 8 * P
            flops += 3 * ev
        else:
            nbytes += n * (elem * frames + 8 + 8) + 8 * P * frames
            flops += frames * (3 * ev + fft)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the same in FP64 ----------------

MOST_EXACT = 4.5e9  # voxel evaluations of one case's FP64 solves (about 15 s); more: no value


def _smooth(m, dim, n, single):
    """One 3-tap pass of the Sobel gradient's smoothing: [1/4, 1/2, 1/4], 2/3 of each of two at the ends."""
    if n == 1 and single:
        return m
    a = lambda i, k: m.narrow(dim, i, k)  # noqa: E731
    first = (a(0, 1) + a(1, 1)) * (2.0 / 3.0)
    last = (a(n - 1, 1) + a(n - 2, 1)) * (2.0 / 3.0)
    mid = 0.25 * a(0, n - 2) + 0.5 * a(1, n - 2) + 0.25 * a(2, n - 2)
    return torch.cat([first, mid, last], dim)


def _difference(m, dim, n):
    a = lambda i, k: m.narrow(dim, i, k)  # noqa: E731
    first = 0.5 * (a(1, 1) - a(0, 1))
    last = 0.5 * (a(n - 1, 1) - a(n - 2, 1))
    return torch.cat([first, 0.5 * (a(2, n - 2) - a(0, n - 2)), last], dim)


class _Model:
    """The warper's model in FP64: error, gradient and Hessian of one reference."""

    def __init__(self, c, reference):
        self.c = c
        nz, ny, nx = self.shape = (c["nz"], c["ny"], c["nx"])
        self.nd = 3 if nz > 1 else 2
        self.t = t = reference.double()
        sx = lambda m: _smooth(m, 2, nx, False)  # noqa: E731
        sy = lambda m: _smooth(m, 1, ny, False)  # noqa: E731
        sz = lambda m: _smooth(m, 0, nz, True)  # noqa: E731
        self.g = [_difference(sz(sy(t)), 2, nx), _difference(sz(sx(t)), 1, ny)]
        if nz > 1:
            self.g.append(_difference(sy(sx(t)), 0, nz))
        q = _times(c, torch.float64)
        self.i = q.floor().long().clamp_(max=c["nD"] - 2)
        self.fr = q - self.i
        flat = self.i.reshape(-1)
        self.ends = torch.searchsorted(flat, torch.arange(c["nD"] - 1, device=DEV), right=True)
        # the last voxel of every interval has no weight
        self.w1 = self.fr.clone().reshape(-1)
        self.w0 = 1.0 - self.w1
        self.w1[self.ends - 1] = 0.0
        self.w0[self.ends - 1] = 0.0

    def intervals(self, v):
        """Sums over each interval's voxels."""
        s = torch.cumsum(v.reshape(-1), 0)[self.ends - 1]
        return torch.diff(s, prepend=s.new_zeros(1))

    def hessian(self):
        nD, nd = self.c["nD"], self.nd
        H = torch.zeros((nD, nd, nD, nd), dtype=torch.float64, device=DEV)
        k = torch.arange(nD - 1, device=DEV)
        for a in range(nd):
            for b in range(nd):
                gg = (self.g[a] * self.g[b]).reshape(-1)
                H[k, a, k, b] += self.intervals(gg * self.w0 * self.w0)
                H[k + 1, a, k + 1, b] += self.intervals(gg * self.w1 * self.w1)
                both = self.intervals(gg * self.w0 * self.w1)
                H[k + 1, a, k, b] += both
                H[k, a, k + 1, b] += both
        return H.reshape(nD * nd, nD * nd)

    def warp(self, frame, D):
        """The zero-padded linear sample of the frame at x + d(x)."""
        nz, ny, nx = self.shape
        Dt = torch.as_tensor(D, device=DEV, dtype=torch.float64)
        base = [torch.arange(nx, device=DEV)[None, None, :], torch.arange(ny, device=DEV)[None, :, None],
                torch.arange(nz, device=DEV)[:, None, None]]
        low, w = [], []
        for k in range(self.nd):
            p = Dt[self.i, k] + self.fr * (Dt[self.i + 1, k] - Dt[self.i, k])
            n = p.floor()
            w.append(p - n)
            low.append(base[k] + n.long())
        if self.nd == 2:
            low.append(base[2].expand(self.shape))
        flat = frame.reshape(-1)
        val = torch.zeros(self.shape, dtype=torch.float64, device=DEV)
        for corner in range(1 << self.nd):
            weight, idx, ok = 1.0, 0, True
            for k, n in reversed(list(enumerate((nx, ny, nz)))):
                up = (corner >> k) & 1 if k < self.nd else 0
                at = low[k] + up
                ok = ok & (at >= 0) & (at < n)
                idx = idx * n + at.clamp(0, n - 1)
                if k < self.nd:
                    weight = weight * (w[k] if up else 1.0 - w[k])
            val += torch.where(ok, flat[idx], 0.0) * weight
        return val

    def evaluate(self, frame, D):
        """The error sum and its gradient, in the parameter order D0.x, D0.y, (D0.z), D1.x, ..."""
        v = self.warp(frame, D)
        e = torch.where(v > 0, v - self.t, 0.0)
        f = float((e * e).sum())
        g = torch.zeros((self.c["nD"], self.nd), dtype=torch.float64, device=DEV)
        for k in range(self.nd):
            ge = (e * self.g[k]).reshape(-1)
            g[:-1, k] += self.intervals(ge * self.w0)
            g[1:, k] += self.intervals(ge * self.w1)
        return f, g.reshape(-1)

    def solve(self, frame, rigid, earlier=None):
        """The trust-region solve from the best of zero, the rigid shift and an earlier solution, to
        where FP64 no longer lowers the error: (D, f)."""
        nD, nd = self.c["nD"], self.nd
        if not hasattr(self, "eig"):
            self.H = self.hessian()
            self.eig = torch.linalg.eigh(self.H)
        vals, vecs = self.eig

        def point(x):
            D = np.zeros((nD, 3))
            D[:, :nd] = x.reshape(nD, nd).cpu().numpy()
            return D

        x = torch.zeros(nD * nd, dtype=torch.float64, device=DEV)
        f, g = self.evaluate(frame, point(x))
        starts = [np.tile(rigid, (nD, 1))] if np.any(rigid[:nd] != 0) else []
        for s in starts + ([] if earlier is None else [earlier]):
            fs, gs = self.evaluate(frame, s)
            if fs < f:
                x, f, g = torch.as_tensor(s[:, :nd], device=DEV, dtype=torch.float64).reshape(-1), fs, gs
        radius = 40.0
        for _ in range(100):
            c = vecs.T @ g
            step = lambda lam: -c / (vals + lam)  # noqa: E731
            lam, inside = 0.0, vals[0] > 0 and float(step(0.0).norm()) <= radius
            if not inside:
                lo, hi = max(0.0, -float(vals[0])), float(g.norm()) / radius + float(vals[-1])
                for _ in range(60):
                    lam = 0.5 * (lo + hi)
                    lo, hi = (lam, hi) if float(step(lam).norm()) > radius else (lo, lam)
            p = vecs @ step(lam)
            predicted = -float(g @ p + 0.5 * p @ (self.H @ p))
            ft, gt = self.evaluate(frame, point(x + p))
            rho = (f - ft) / predicted if predicted > 0 else -1.0
            if rho < 0.25:
                radius *= 0.25
            elif rho > 0.75 and not inside:
                radius = min(1000.0, 2 * radius)
            if not rho > 0:
                break
            small = float(p.abs().max()) < 1e-9
            x, f, g = x + p, ft, gt
            if small:
                break
        return point(x), f


def _correlate(reference, volume):
    """The whole-pixel shift (x, y, z) at the first maximum of the normalised phase correlation."""
    nz, ny, nx = reference.shape

    def window(n):
        i = torch.arange(n, device=DEV, dtype=torch.float64)
        return torch.sqrt(0.5 * (1 - torch.cos(2 * math.pi / (n - 1) * i))) if n > 1 else torch.ones_like(i)

    w = window(ny)[None, :, None] * window(nx)[None, None, :]
    c = torch.fft.rfftn(volume.double() * w) * torch.fft.rfftn(reference.double() * w).conj()
    c = c / (c.abs() + 2.2250738585072014e-308)
    at = int(torch.argmax(torch.fft.irfftn(c, s=(nz, ny, nx))))
    s = [at % nx, at // nx % ny, at // (nx * ny)]
    return np.array([v - n if v > n // 2 else v for v, n in zip(s, (nx, ny, nz))], dtype=np.float64)


def _binned(v, b):
    if b == 1:
        return v
    nz, ny, nx = v.shape
    v = torch.nn.functional.pad(v, (0, -nx % b, 0, -ny % b))
    return v.reshape(nz, v.shape[1] // b, b, v.shape[2] // b, b).sum((2, 4))


def _exact_solves(c, reference, raw, binning=1, chained=False):
    model = _Model(c, reference + 1)
    D, f = [], []
    for r in raw:
        shift = _correlate(_binned(reference, binning), _binned(r, binning))
        shift[:2] *= binning
        d, v = model.solve(r.double() + 1, shift, D[-1] if chained and D else None)
        D.append(d)
        f.append(v)
    return np.stack(D), np.array(f)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("align", "serve"):
        voxels = sum(c["nz"] * c["ny"] * c["nx"] for c in _sizes(case)) * case["frames"]
        if 20.0 * voxels > MOST_EXACT:  # about 20 evaluations a solve
            return None
    if kind == "serve":
        per = []
        for j, c in enumerate(_sizes(case)):
            reference, raw, _ = _inputs(c, seed * 16 + j, case["frames"])
            per.append(list(zip(*_exact_solves(c, reference, raw, chained=True))))
        got = [f for turn in zip(*per) for f in turn]
        return {"D": np.concatenate([g[0] for g in got]), "f": np.array([g[1] for g in got])}
    c = dict(case)
    if kind == "shift":
        c["nD"] = _control_points(c["nz"], c["ny"])
        reference, raw, _ = _inputs(c, seed, 1)
        return _correlate(reference, raw[0])
    if kind == "reference":
        reference, _, _ = _inputs(c, seed, 0)
        return _Model(c, reference + 1).hessian()
    reference, raw, D = _inputs(c, seed, case.get("frames", 1))
    if kind == "align":
        d, f = _exact_solves(c, reference, raw, case["binning"])
        return {"D": d, "f": f}
    model, frame = _Model(c, reference + 1), raw[0].double() + 1
    at = 0.9 * D[0] + 0.05
    if c["nz"] == 1:
        at[:, 2] = 0.0
    if kind == "evaluate":
        f, g = model.evaluate(frame, at)
        return {"f": np.array([f]), "jacobian": g}
    if kind == "warp":
        return model.warp(frame, at)
    d, f = model.solve(frame, _rigid(D[0]))
    return {"D": d, "f": np.array([f])}
