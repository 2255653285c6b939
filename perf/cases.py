"""Performance cases of the framework: the work its users have it do, through
the public entry points, over the range of sizes and options in real use.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` makes what a program has in hand before the call (inputs
and the long-lived handle), ``run`` is one pass, ``work`` the bytes and
operations a pass cannot do without, and ``exact`` the result in 64 bits by
plain torch.

Kinds of case (``kind``):

- ``frame``     one frame of a DPRA handle (least squares, WFF2, phase update)
- ``sequence``  a block of host frames through the sequence call
- ``batch``     one step of several sequences of uneven sizes
- ``surrogate`` one frame with the learned network in WFF2's place
- ``train``     one training pass of that network, with the optimizer's step
- ``wff``       the windowed Fourier filter alone
- ``wfr``       windowed Fourier ridges
- ``aia``       initial phase from frames with unknown shifts
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "g-ls3u_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import glsu  # noqa: E402
from glsu import train_surrogate  # noqa: E402

_IMG = {"u8": glsu.U8, "f32": glsu.F32, "f64": glsu.F64}
_REAL = {"f32": torch.float32, "f64": torch.float64}
_CPLX = {"f32": torch.complex64, "f64": torch.complex128}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _grid(sigma, half_range, step, thr):
    return {"sigma": sigma, "wl": -half_range, "wh": half_range, "step": step, "thr": thr}


def listed():
    return [
        # a small camera's frame with the parameters that DPRA hard-wires (3 x 3
        # window, sigma 20, 7 x 7 frequencies): the shortest call
        {"name": "frame_256_defaults_u8", "kind": "frame", "h": 256, "w": 256, "r": 1, "img": "u8", "prec": "f32",
         "graph": False, **_grid(20.0, 0.15, 0.05, 15.0)},
        # the benchmark's frame: 7 x 7 window, sigma 10, 21 x 21 frequencies, replayed from a CUDA graph
        {"name": "frame_1024_sigma10", "kind": "frame", "h": 1024, "w": 1024, "r": 3, "img": "f32", "prec": "f32",
         "graph": True, **_grid(10.0, 1.0, 0.1, 0.2)},
        # a sensor's odd size, 8-bit, a narrower window and fewer frequencies
        {"name": "frame_733x1021_sigma7_u8", "kind": "frame", "h": 733, "w": 1021, "r": 2, "img": "u8", "prec": "f32",
         "graph": False, **_grid(7.0, 0.75, 0.125, 0.3)},
        # the FP64 form on the 256 x 256 workload
        {"name": "frame_256_f64", "kind": "frame", "h": 256, "w": 256, "r": 3, "img": "f64", "prec": "f64",
         "graph": False, **_grid(10.0, 1.0, 0.1, 0.2)},
        # a recorded 8-bit clip from pinned host memory, copies overlapped, results on the host
        {"name": "sequence_480x640_u8", "kind": "sequence", "h": 480, "w": 640, "r": 2, "img": "u8", "prec": "f32",
         "frames": 8, **_grid(10.0, 1.0, 0.1, 0.2)},
        # one step of a batch of uneven sequences, windows of radius 2 to 4
        {"name": "batch_uneven_6", "kind": "batch", "sizes": "256x256,256x256,384x512,384x512,1024x1024,480x640",
         "img": "f32", "prec": "f32", **_grid(10.0, 1.0, 0.1, 0.2)},
        # the learned form at the benchmark's size with the shipped network
        {"name": "surrogate_1024", "kind": "surrogate", "h": 1024, "w": 1024, "r": 3, "img": "f32", "prec": "f32",
         "tile": 256, **_grid(10.0, 1.0, 0.1, 0.2)},
        # one training pass at the trainer's batch and crop, gradients read back
        {"name": "train_16x256", "kind": "train", "batch": 16, "h": 256, "w": 256},
        # the filter alone with its class defaults (47 x 47 frequencies, automatic threshold)
        {"name": "wff_384x512_defaults", "kind": "wff", "h": 384, "w": 512, "prec": "f32", **_grid(10.0, 2.3, 0.1, -1.0)},
        # the large workload's window and grid (sigma 15, 31 x 31) on a large field: the longest call
        {"name": "wff_1536x2048_sigma15", "kind": "wff", "h": 1536, "w": 2048, "prec": "f32",
         **_grid(15.0, 1.5, 0.1, 0.2)},
        # ridges of a field over a moderate frequency grid
        {"name": "wfr_256x320", "kind": "wfr", "h": 256, "w": 320, "prec": "f32", **_grid(10.0, 1.0, 0.05, 0.0)},
        # initial phase of five full frames with unknown shifts, at most 30 iterations
        {"name": "aia_5x1024", "kind": "aia", "m": 5, "h": 1024, "w": 1024, "img": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "sequence", "batch", "surrogate", "train", "wff", "wff", "wfr", "aia"])
    sigma = round(rng.uniform(5.0, 15.0), 1)
    n = rng.randint(7, 21)
    half = round(rng.uniform(0.3, 1.2), 2)
    grid = _grid(sigma, half, round(2 * half / (n - 0.5), 4), round(rng.uniform(0.1, 0.5), 2))
    if kind == "frame":
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        big = 1400 if prec == "f32" else 240
        return {"kind": kind, "h": _log_int(rng, 64, big), "w": _log_int(rng, 64, big), "r": rng.randint(1, 5),
                "img": rng.choice(["u8", prec]), "prec": prec, "graph": rng.random() < 0.5, **grid}
    if kind == "sequence":
        return {"kind": kind, "h": _log_int(rng, 96, 700), "w": _log_int(rng, 96, 700), "r": rng.randint(1, 4),
                "img": rng.choice(["u8", "f32"]), "prec": "f32", "frames": rng.randint(3, 8), **grid}
    if kind == "batch":
        sizes = ",".join("%dx%d" % (_log_int(rng, 64, 800), _log_int(rng, 64, 800)) for _ in range(rng.randint(2, 6)))
        return {"kind": kind, "sizes": sizes, "img": rng.choice(["u8", "f32"]), "prec": "f32", **grid}
    if kind == "surrogate":
        return {"kind": kind, "h": _log_int(rng, 256, 1400), "w": _log_int(rng, 256, 1400), "r": 3, "img": "f32",
                "prec": "f32", "tile": rng.choice([128, 256, 512]), **_grid(10.0, 1.0, 0.1, 0.2)}
    if kind == "train":
        return {"kind": kind, "batch": rng.randint(1, 16), "h": _log_int(rng, 96, 256), "w": _log_int(rng, 96, 256)}
    if kind == "wff":
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        big = 1400 if prec == "f32" else 240
        if rng.random() < 0.3:
            grid["thr"] = -1.0
        return {"kind": kind, "h": _log_int(rng, 64, big), "w": _log_int(rng, 64, big), "prec": prec, **grid}
    if kind == "wfr":
        return {"kind": kind, "h": _log_int(rng, 64, 320), "w": _log_int(rng, 64, 320), "prec": "f32",
                **_grid(round(rng.uniform(5.0, 12.0), 1), 1.0, rng.choice([0.05, 0.1]), 0.0)}
    return {"kind": kind, "m": rng.randint(3, 8), "h": _log_int(rng, 128, 1024), "w": _log_int(rng, 128, 1024),
            "img": rng.choice(["u8", "f32"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _bumps(rng, h, w, n, amp, width):
    """Sum of n Gaussians with random centres, amplitudes and widths (pixels at 256, scaled with the image)."""
    y = torch.arange(h, device="cuda", dtype=torch.float64)[:, None]
    x = torch.arange(w, device="cuda", dtype=torch.float64)[None, :]
    scale = max(h, w) / 256.0
    out = torch.zeros((h, w), device="cuda", dtype=torch.float64)
    for _ in range(n):
        cy, cx = rng.uniform(0, h), rng.uniform(0, w)
        a, s = rng.uniform(*amp), rng.uniform(*width) * scale
        out += a * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * s * s))
    return out


def _scene(h, w, seed, carrier):
    """Background, reference phase and per-frame phase change.  With a carrier
    the phase is tilt fringes of 8 to 16 pixels plus an object of a few
    radians, as an interferometer gives them; without, the generator that the
    network is trained on."""
    rng = np.random.default_rng(seed)
    a = 0.5 + _bumps(rng, h, w, 1, (0.1, 0.1), (80, 80))
    if carrier:
        phi0 = _bumps(rng, h, w, 3, (1.0, 3.0), (40, 80))
        k = 2 * math.pi / rng.uniform(8.0, 16.0)
        t = rng.uniform(0.4, 1.1)
        y = torch.arange(h, device="cuda", dtype=torch.float64)[:, None]
        x = torch.arange(w, device="cuda", dtype=torch.float64)[None, :]
        phi0 = phi0 + k * (math.cos(t) * x + math.sin(t) * y)
        delta = _bumps(rng, h, w, 2, (0.3, 0.5), (40, 80)) + 0.2
    else:
        phi0 = _bumps(rng, h, w, 4, (5.0, 15.0), (20, 60))
        delta = _bumps(rng, h, w, 2, (0.5, 1.0), (20, 60))
        delta = delta * (0.3 / delta.abs().max())
    return a, phi0, delta


def _frames(h, w, seed, n, img, carrier=True, noise=0.02):
    """(frames 1..n as device tensors, phi0 on the host in FP64).  Over a
    block the phase moves by less than half a turn, as the recursion asks."""
    a, phi0, delta = _scene(h, w, seed, carrier)
    delta = delta * min(1.0, 2.0 / n)
    g = _gen(seed)
    out = []
    for k in range(1, n + 1):
        f = a + 0.4 * torch.cos(phi0 + k * delta) + noise * torch.randn((h, w), generator=g, device="cuda",
                                                                        dtype=torch.float64)
        if img == "u8":
            f = torch.clamp(torch.round(f * 255), 0, 255).to(torch.uint8)
        else:
            f = f.to(_REAL[img])
        out.append(f.contiguous())
    return out, phi0.cpu().numpy()


def _field(h, w, seed, prec):
    """exp(j phi) of a smooth phase with complex noise, amplitude varying by 2x."""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    y = torch.arange(h, device="cuda", dtype=torch.float64)[:, None]
    x = torch.arange(w, device="cuda", dtype=torch.float64)[None, :]
    phi = _bumps(rng, h, w, 3, (3.0, 8.0), (30, 80)) + rng.uniform(-0.2, 0.2) * x + rng.uniform(-0.2, 0.2) * y
    amp = 1.0 + _bumps(rng, h, w, 1, (1.0, 1.0), (60, 100))
    f = amp * torch.exp(1j * phi)
    noise = torch.randn((h, w, 2), generator=g, device="cuda", dtype=torch.float64)
    return (f + 0.1 * torch.view_as_complex(noise)).to(_CPLX[prec]).contiguous()


def _params(c):
    return glsu.WffParams(c["sigma"], c["wl"], c["wh"], c["step"], c["sigma"], c["wl"], c["wh"], c["step"], c["thr"])


def _sizes(c):
    return [tuple(int(v) for v in s.split("x")) for s in c["sizes"].split(",")]


class _Batch(glsu.DpraBatch):
    """A batch that gives its streams and graphs back with its last reference."""

    def __del__(self):
        self.close()


class _Plane:
    """A device plane of a handle as an array that torch can take without a
    copy; the tensor made from it keeps the handle, and so the plane, alive."""

    def __init__(self, owner, ptr, shape):
        self._owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 2}


def _aia_frames(c, seed):
    a, phi0, _ = _scene(c["h"], c["w"], seed, False)
    rng = np.random.default_rng(seed + 1)
    # shifts spread over the circle, each off its place by up to a quarter step
    shifts = 2 * np.pi * (np.arange(c["m"]) + rng.uniform(-0.25, 0.25, c["m"])) / c["m"]
    g = _gen(seed)
    frames = []
    for s in shifts:
        f = a + 0.4 * torch.cos(phi0 + float(s)) + 0.02 * torch.randn(phi0.shape, generator=g, device="cuda",
                                                                      dtype=torch.float64)
        f = torch.clamp(torch.round(f * 255), 0, 255).to(torch.uint8) if c["img"] == "u8" else f.to(torch.float32)
        frames.append(f.cpu().numpy())
    start = (shifts - shifts[0] + rng.uniform(-0.3, 0.3, c["m"])).astype(np.float32)
    return frames, start


def _train_pair(c, seed):
    """(network input, target): a noisy unit-modulus field and the same field without noise, magnitude below one."""
    z, t = [], []
    g = _gen(seed)
    for b in range(c["batch"]):
        rng = np.random.default_rng((seed, b))
        d = _bumps(rng, c["h"], c["w"], 2, (0.1, 0.5), (20, 60))
        noise = rng.uniform(0.05, 0.6) * torch.randn(d.shape, generator=g, device="cuda", dtype=torch.float64)
        z.append(torch.exp(1j * (d + noise)))
        t.append(rng.uniform(0.6, 0.95) * torch.exp(1j * d))
    return torch.stack(z).to(torch.complex64).contiguous(), torch.stack(t).to(torch.complex64).contiguous()


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": dict(c), "kind": kind}
    if kind == "frame" or kind == "surrogate":
        fr, phi0 = _frames(c["h"], c["w"], seed, 1, c["img"], carrier=kind == "frame")
        s["frame"] = fr[0]
        s["out"] = torch.empty((c["h"], c["w"]), device="cuda", dtype=_REAL[c["prec"]])
        s["dpra"] = glsu.DPRA(phi0, 1, c["r"], c["prec"], _params(c))
        if kind == "surrogate":
            d = np.load(train_surrogate.DEFAULT_WEIGHTS)
            s["dpra"].set_surrogate(d["params"], d["dilations"], c["tile"], 0, 0.05)
        if c.get("graph", True):
            s["dpra"].set_graph(True)
    elif kind == "sequence":
        fr, phi0 = _frames(c["h"], c["w"], seed, c["frames"], c["img"])
        s["frames"] = torch.stack(fr).cpu().pin_memory()
        s["out"] = torch.empty((c["frames"], c["h"], c["w"]), dtype=torch.float32).pin_memory()
        s["dpra"] = glsu.DPRA(phi0, c["frames"], c["r"], c["prec"], _params(c))
        s["dpra"].set_graph(True)
    elif kind == "batch":
        s["frames"], s["handles"] = [], []
        for k, (h, w) in enumerate(_sizes(c)):
            fr, phi0 = _frames(h, w, seed * 64 + k, 1, c["img"])
            s["frames"].append(fr[0])
            s["handles"].append(glsu.DPRA(phi0, 1 << 20, 2 + k % 3, "f32", _params(c)))
        s["batch"] = _Batch(s["handles"], graph=True)
    elif kind == "train":
        s["z"], s["t"] = _train_pair(c, seed)
        s["net"] = glsu.Surrogate(c["batch"], c["w"], c["h"], train_surrogate.DILATIONS, training=True)
        s["net"].params = train_surrogate.init_params(seed)
    elif kind == "wff":
        s["f"] = _field(c["h"], c["w"], seed, c["prec"])
        s["out"] = torch.empty_like(s["f"])
        s["wff"] = glsu.WFF2(c["w"], c["h"], c["prec"], _params(c))
    elif kind == "wfr":
        s["f"] = _field(c["h"], c["w"], seed, c["prec"])
        s["maps"] = {k: torch.empty((c["h"], c["w"]), device="cuda", dtype=_REAL[c["prec"]]) for k in glsu.WFR_FIELDS}
        s["wfr"] = glsu.WFR2(c["w"], c["h"], c["prec"], _params(c))
        s["ptrs"] = {k: v.data_ptr() for k, v in s["maps"].items()}
    else:
        s["frames"], s["start"] = _aia_frames(c, seed)
        s["aia"] = glsu.AIA(c["m"], c["w"], c["h"])
        s["aia"].set_convergence(True)
    torch.cuda.synchronize()
    return s


def run(state):
    s, c, kind = state, state["case"], state["kind"]
    if kind == "frame" or kind == "surrogate":
        s["dpra"].per_frame_device(s["frame"].data_ptr(), _IMG[c["img"]], s["out"].data_ptr())
        return s["out"]
    if kind == "sequence":
        s["dpra"].sequence_ptr(c["frames"], s["frames"].data_ptr(), _IMG[c["img"]], s["out"].data_ptr())
        return s["out"]
    if kind == "batch":
        s["batch"].run([f.data_ptr() for f in s["frames"]], _IMG[c["img"]])
        return [torch.as_tensor(_Plane(d, d.device_ptr(glsu.DPHI), (d.height, d.width)), device="cuda")
                for d in s["handles"]]
    if kind == "train":
        loss, grad = s["net"].backward(s["z"].data_ptr(), s["t"].data_ptr(), want_grad=True)
        s["net"].adam(1e-4)
        return {"loss": loss, "grad": grad}
    if kind == "wff":
        s["wff"].run_async(s["f"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if kind == "wfr":
        s["wfr"].run_async(s["f"].data_ptr(), s["ptrs"])
        return s["maps"]
    phi, deltas, _, iters, _ = s["aia"].run(s["frames"], s["start"], max_iter=30, max_err=1e-4)
    return {"phi": phi, "deltas": deltas, "iters": iters}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _count(c):
    if c.get("prec", "f32") == "f64":
        return int((c["wh"] - c["wl"]) * (1.0 / c["step"])) + 1
    f = np.float32
    return int((f(c["wh"]) - f(c["wl"])) * (f(1) / f(c["step"]))) + 1


def _wff_flops(h, w, c, filters=2):
    """Row filters per x-frequency, and per (x, y) frequency pair `filters`
    column transforms with one product each: 5 L log2 L per transform."""
    n, s = _count(c), int(math.floor(3 * c["sigma"] + 0.5))
    length = h + 2 * s
    rows = filters * n * h * w * (4.0 * (2 * s + 1) + 8)
    cols = float(n) * n * w * filters * (5.0 * length * math.log2(length) + 8.0 * length)
    return rows + cols


def _frame_work(h, w, c, r):
    es = 4 if c["prec"] == "f32" else 8
    im = {"u8": 1, "f32": 4, "f64": 8}[c["img"]]
    # frame, phi_ref and dphi_ref in; phi_curr and dphi out; running sums of the 8 window moments and the solve
    return h * w * (im + 4 * es), h * w * (8 * 8 + 60.0)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("frame", "sequence"):
        b, f = _frame_work(c["h"], c["w"], c, c["r"])
        k = c.get("frames", 1)
        return {"bytes": k * b, "flops": k * (f + _wff_flops(c["h"], c["w"], c))}
    if kind == "batch":
        b = f = 0
        for h, w in _sizes(c):
            x, y = _frame_work(h, w, c, 3)
            b, f = b + x, f + y + _wff_flops(h, w, c)
        return {"bytes": b, "flops": f}
    if kind == "surrogate":
        b, f = _frame_work(c["h"], c["w"], c, c["r"])
        return {"bytes": b, "flops": f + 2.0 * c["h"] * c["w"] * 9 * (2 * 32 + 6 * 32 * 32 + 32 * 2)}
    if kind == "train":
        n = c["batch"] * c["h"] * c["w"]
        return {"bytes": 16.0 * n, "flops": 3 * 2.0 * n * 9 * (2 * 32 + 6 * 32 * 32 + 32 * 2)}
    if kind == "wff":
        es = 8 if c["prec"] == "f32" else 16
        return {"bytes": 2.0 * es * c["h"] * c["w"], "flops": _wff_flops(c["h"], c["w"], c)}
    if kind == "wfr":
        return {"bytes": (8 + 8 * 4.0) * c["h"] * c["w"], "flops": _wff_flops(c["h"], c["w"], c, filters=1)}
    n = c["h"] * c["w"]
    return {"bytes": n * (c["m"] * (1 if c["img"] == "u8" else 4) + 4.0), "flops": 10 * n * (12.0 * c["m"] + 30)}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
def _box(a, r):
    """Sums over the (2r+1)^2 window clipped to the image, for each shift."""
    return torch.nn.functional.pad(a, (r, r, r, r))


def _ls(img, phi, r):
    """exp(j dphi) of the windowed 3 x 3 least squares; sums shifted by the centre pixel's own values."""
    h, w = img.shape
    mc, ms, mi = torch.cos(phi), torch.sin(phi), img
    pad = [_box(a, r) for a in (mc, ms, mi, torch.ones_like(img))]
    t = {k: torch.zeros_like(img) for k in ("c", "s", "i", "cc", "ss", "cs", "ic", "is", "n")}
    for dy in range(2 * r + 1):
        for dx in range(2 * r + 1):
            c, s, i, one = (a[dy:dy + h, dx:dx + w] for a in pad)
            c, s, i = (c - mc) * one, (s - ms) * one, (i - mi) * one
            for k, v in (("c", c), ("s", s), ("i", i), ("cc", c * c), ("ss", s * s), ("cs", c * s), ("ic", i * c),
                         ("is", i * s), ("n", one)):
                t[k] += v
    n0 = float((2 * r + 1) ** 2)
    rho = 1 - t["n"] / n0

    def moment(p, u, v, mu, mv):
        return p - u * v / n0 + rho * (mu * v + mv * u + t["n"] * mu * mv)

    a, d = moment(t["cc"], t["c"], t["c"], mc, mc), moment(t["ss"], t["s"], t["s"], ms, ms)
    b = moment(t["cs"], t["c"], t["s"], mc, ms)
    p, q = moment(t["ic"], t["i"], t["c"], mi, mc), moment(t["is"], t["i"], t["s"], mi, ms)
    x, y = d * p - b * q, a * q - b * p
    sg = torch.where(a * d - b * b < 0, -1.0, 1.0).to(x)
    z = torch.complex(sg * x, -sg * y)
    m = z.abs()
    return torch.where(m > 0, z / torch.where(m > 0, m, torch.ones_like(m)), torch.ones_like(z))


def _fft_size(n):
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _window_spectra(c, length, s, g):
    m = torch.arange(-s, s + 1, device="cuda", dtype=torch.float64)
    out = []
    for k in range(_count(c)):
        v = torch.zeros(length, device="cuda", dtype=torch.complex128)
        v[(torch.arange(-s, s + 1, device="cuda")) % length] = g * torch.exp(1j * (c["wl"] + k * c["step"]) * m)
        out.append(torch.fft.fft(v))
    return out


def _windows(c, h, w):
    s = int(math.floor(3 * c["sigma"] + 0.5))
    m = torch.arange(-s, s + 1, device="cuda", dtype=torch.float64)
    g = torch.exp(-m * m / (2 * c["sigma"] ** 2))
    g = g / torch.sqrt((g * g).sum())
    lh, lw = _fft_size(h + 2 * s), _fft_size(w + 2 * s)
    return s, m, g, lh, lw, _window_spectra(c, lh, s, g), _window_spectra(c, lw, s, g)


def _wff(f, c):
    h, w = f.shape
    thr = c["thr"] if c["thr"] >= 0 else 6 * math.sqrt(float((f.abs() ** 2).mean()) / 3)
    _, _, _, lh, lw, ys, xs = _windows(c, h, w)
    spec = torch.fft.fft2(f, s=(lh, lw))
    acc = torch.zeros_like(spec)
    for kx in xs:
        row = spec * kx[None, :]
        for ky in ys:
            sf = torch.fft.ifft2(row * ky[:, None])[:h, :w]
            sf = torch.where(sf.abs() >= thr, sf, torch.zeros_like(sf))
            acc += torch.fft.fft2(sf, s=(lh, lw)) * kx[None, :] * ky[:, None]
    return torch.fft.ifft2(acc)[:h, :w] * (c["step"] ** 2 / (4 * math.pi ** 2))


def _wfr(f, c):
    h, w = f.shape
    s, m, g, lh, lw, ys, xs = _windows(c, h, w)
    spec = torch.fft.fft2(f, s=(lh, lw))
    r = torch.zeros((h, w), device="cuda", dtype=torch.float64)
    wx, wy, ph = torch.zeros_like(r), torch.zeros_like(r), torch.zeros_like(r)
    for k, ky in enumerate(ys):
        col = spec * ky[:, None]
        for i, kx in enumerate(xs):
            sf = torch.fft.ifft2(col * kx[None, :])[:h, :w]
            mag = sf.abs()
            t = mag >= r
            r, ph = torch.where(t, mag, r), torch.where(t, sf.angle(), ph)
            wx = torch.where(t, torch.full_like(wx, c["wl"] + i * c["step"]), wx)
            wy = torch.where(t, torch.full_like(wy, c["wl"] + k * c["step"]), wy)

    def conv(a, ky, kx):
        # separable, border replicated; out(y, x) = sum k(n) a(y, x - n)
        a = torch.nn.functional.pad(a[None, None], (s, s, s, s), mode="replicate")
        a = sum(float(kx[s + n]) * a[..., s - n:s - n + w] for n in range(-s, s + 1))
        return sum(float(ky[s + n]) * a[..., s - n:s - n + h, :] for n in range(-s, s + 1))[0, 0]

    cxx = -conv(wx, g, g * m) / float((g * m * m).sum() * g.sum())
    cyy = -conv(wy, g * m, g) / float((g * m * m).sum() * g.sum())
    s2 = c["sigma"] ** 2
    pc = ph - 0.5 * torch.atan(s2 * cxx) - 0.5 * torch.atan(s2 * cyy)
    q = 0.25 / math.pi / s2
    b = r * ((1 + (s2 * cxx) ** 2) * q) ** 0.25 * ((1 + (s2 * cyy) ** 2) * q) ** 0.25
    return {"wx": wx, "wy": wy, "phase": ph, "phase_comp": torch.atan2(torch.sin(pc), torch.cos(pc)), "b": b, "r": r,
            "cxx": cxx, "cyy": cyy}


def _net(params, z, dil):
    """The residual network in 64 bits: eight dilated 3 x 3 layers, output renormalised."""
    x = torch.stack([z.real, z.imag], 1)
    a, off = x, 0
    sizes = [(32, 2)] + [(32, 32)] * 6 + [(2, 32)]
    for k, (co, ci) in enumerate(sizes):
        wt = params[off:off + co * ci * 9].reshape(co, ci, 3, 3)
        b = params[off + co * ci * 9:off + co * ci * 9 + co]
        off += co * ci * 9 + co
        d = int(dil[k])
        p = torch.nn.functional.pad(a, (d, d, d, d))
        h, w = a.shape[2:]
        o = b[None, :, None, None].expand(a.shape[0], co, h, w)
        for dy in range(3):
            for dx in range(3):
                o = o + torch.einsum("oc,bchw->bohw", wt[:, :, dy, dx], p[:, :, dy * d:dy * d + h, dx * d:dx * d + w])
        a = x + o if k == 7 else torch.relu(o)
    return a / torch.sqrt((a * a).sum(1, keepdim=True))


def _exact_frame(frame, phi, c, r):
    return _wff(_ls(frame.double(), phi, r), c).angle()


def _ref(phi0, prec):
    return torch.from_numpy(phi0).cuda().to(_REAL[prec]).double()


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("frame", "surrogate"):
        fr, phi0 = _frames(c["h"], c["w"], seed, 1, c["img"], carrier=kind == "frame")
        phi = _ref(phi0, c["prec"])
        if kind == "frame":
            return _exact_frame(fr[0], phi, c, c["r"])
        d = np.load(train_surrogate.DEFAULT_WEIGHTS)
        y = _net(torch.from_numpy(d["params"]).cuda().double(), _ls(fr[0].double(), phi, c["r"])[None], d["dilations"])
        return torch.atan2(y[0, 1], y[0, 0])
    if kind == "sequence":
        fr, phi0 = _frames(c["h"], c["w"], seed, c["frames"], c["img"])
        phi, dref, out = _ref(phi0, "f32"), 0.0, []
        for k, f in enumerate(fr):
            t = _exact_frame(f, phi, c, c["r"])
            out.append(dref + t)
            if k == 0:  # the reference moves after the first frame of the block only
                phi, dref = phi + t, dref + t
        return torch.stack(out).cpu()
    if kind == "batch":
        out = []
        for k, (h, w) in enumerate(_sizes(c)):
            fr, phi0 = _frames(h, w, seed * 64 + k, 1, c["img"])
            out.append(_exact_frame(fr[0], _ref(phi0, "f32"), c, 2 + k % 3))
        return out
    if kind == "train":
        z, t = _train_pair(c, seed)
        p = torch.from_numpy(train_surrogate.init_params(seed)).cuda().double().requires_grad_()
        loss = 0.0
        for b in range(c["batch"]):
            y = _net(p, z[b:b + 1].to(torch.complex128), train_surrogate.DILATIONS)[0]
            tb = t[b].to(torch.complex128)
            u = tb / tb.abs()
            e = (tb.abs().clamp(max=1) * ((y[0] - u.real) ** 2 + (y[1] - u.imag) ** 2)).sum()
            e = e / (c["batch"] * c["h"] * c["w"])
            e.backward()
            loss += float(e.detach())
        return {"loss": loss, "grad": p.grad.cpu().numpy()}
    if kind == "wff":
        return _wff(_field(c["h"], c["w"], seed, c["prec"]).to(torch.complex128), c)
    if kind == "wfr":
        return _wfr(_field(c["h"], c["w"], seed, c["prec"]).to(torch.complex128), c)
    frames, start = _aia_frames(c, seed)
    f = torch.stack([torch.from_numpy(v) for v in frames]).cuda().double().reshape(c["m"], -1)
    d = torch.from_numpy(start).cuda().double()

    def phase(d):
        a = torch.stack([torch.ones_like(d), torch.cos(d), torch.sin(d)])
        x = torch.linalg.solve(a @ a.T, a @ f)
        return torch.atan2(-x[2], x[1])

    iters = 0
    for iters in range(1, 31):
        phi = phase(d)
        b = torch.stack([torch.ones_like(phi), torch.cos(phi), torch.sin(phi)])
        y = torch.linalg.solve(b @ b.T, b @ f.T)
        new = torch.atan2(-y[2], y[1])
        err = float(((new - new[0]) - (d - d[0])).abs().max())
        d = new
        if not err > 1e-4:
            break
    phi = phase(d) + d[0]
    d = d - d[0]
    return {"phi": torch.atan2(torch.sin(phi), torch.cos(phi)).reshape(c["h"], c["w"]).cpu().numpy(),
            "deltas": torch.atan2(torch.sin(d), torch.cos(d)).cpu().numpy(), "iters": iters}
