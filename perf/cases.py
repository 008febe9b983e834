"""Performance cases: what a user of this framework has it compute, through its public entry points.

Three kinds of work:

* projections (``lfdeconv.ForwardProjectACC`` / ``BackwardProjectACC``) of camera frames and volumes that
  stay on the device, as a program that goes on working with them there calls them;
* Richardson-Lucy deconvolution: ``lfdeconv.DeconvRL`` on host images (the reference's whole call), and a
  batch of a time series on the device (back projection, then ``Projector_gb300.RichardsonLucy``), as
  ``deconvolve_time_series`` does it;
* the warm-start network: single layers (``_flf.conv3d``, its data gradient with the ReLU mask,
  ``conv3d_wgrad`` / ``bias_grad``) and the whole forward pass of ``warmstart.UNet3D``.

``listed`` gives the fixed cases, ``draw`` more of the same ranges, ``prepare`` the inputs and what a
program keeps, ``run`` one pass, ``work`` the bytes and operations a pass cannot do without, ``exact`` the
result in 64 bits in plain torch.
"""

import collections
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "fast-light-field_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import _flf  # noqa: E402
import lfdeconv  # noqa: E402
import projector as proj  # noqa: E402
import psfmatrix  # noqa: E402
import warmstart  # noqa: E402


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one frame of a few lenslets, as in an interactive check or a test
        {"name": "bp_smallest", "kind": "backward", "nnum": 5, "y": 30, "x": 35, "planes": 3, "reach": 3, "frames": 1},
        # one frame of the small field of view, 30 x 30 lenslets of 15 px, planes -25..25 um
        {"name": "fp_frame", "kind": "forward", "nnum": 15, "y": 450, "x": 450, "planes": 11, "reach": 7, "frames": 1},
        # three frames of a cropped camera image, no side a multiple of the lenslet
        {"name": "bp_ragged", "kind": "backward", "nnum": 15, "y": 437, "x": 608, "planes": 31, "reach": 14, "frames": 3},
        # the full field of view, 67 x 67 lenslets, planes -100..100 um: forward model of a volume
        {"name": "fp_fullfield", "kind": "forward", "nnum": 15, "y": 1005, "x": 1005, "planes": 41, "reach": 28, "frames": 1},
        # the same field of view: first estimate Htf of a frame
        {"name": "bp_fullfield", "kind": "backward", "nnum": 15, "y": 1005, "x": 1005, "planes": 41, "reach": 28, "frames": 1},
        # a user's whole deconvolution of one camera frame: host image in, host volume out, 8 iterations
        {"name": "rl_frame", "kind": "rl", "nnum": 15, "y": 450, "x": 450, "planes": 21, "reach": 14, "frames": 1,
         "iters": 8, "trust": False},
        # a batch of a time series on the device: Htf as start, 8 iterations, 8 frames at once
        {"name": "rl_series", "kind": "series", "nnum": 15, "y": 450, "x": 450, "planes": 31, "reach": 14, "frames": 8,
         "iters": 8},
        # the standard update with a trust mask (dead lenslets), coarser lenslets of 19 px, two frames
        {"name": "rl_trust", "kind": "rl", "nnum": 19, "y": 380, "x": 437, "planes": 7, "reach": 5, "frames": 2,
         "iters": 4, "trust": True},
        # a full-resolution layer of the warm-start network at the 450 x 450 px, 21-plane volume's padded size
        {"name": "conv_level0", "kind": "conv", "ci": 16, "co": 16, "b": 1, "z": 24, "y": 456, "x": 456, "grad": False},
        # a deep layer's data gradient (ReLU mask) on a training batch of 4 crops
        {"name": "conv_wide_grad", "kind": "conv", "ci": 64, "co": 64, "b": 4, "z": 6, "y": 32, "x": 32, "grad": True},
        # weight and bias gradients of a full-resolution layer on a training batch of 4 crops
        {"name": "wgrad_level0", "kind": "wgrad", "ci": 16, "co": 16, "b": 4, "z": 24, "y": 128, "x": 128},
        # the network's whole forward pass on one volume
        {"name": "unet_forward", "kind": "unet", "b": 1, "z": 24, "y": 456, "x": 456},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# input and output channels of the network's layers
_PAIRS = [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 64), (64, 32), (32, 16)]


def draw(rng):
    kind = rng.choice(["forward", "backward", "backward", "forward", "rl", "series", "conv", "conv", "wgrad", "unet"])
    if kind == "unet":
        z, y, x = 8 * rng.randint(1, 3), 8 * _log_int(rng, 3, 57), 8 * _log_int(rng, 3, 57)
        return {"kind": kind, "b": 1, "z": z, "y": y, "x": x}
    if kind in ("conv", "wgrad"):
        ci, co = rng.choice(_PAIRS)
        level = int(math.log2(max(ci, co) / 16))
        hi = (456 if kind == "conv" else 128) >> level
        case = {"kind": kind, "ci": ci, "co": co, "b": rng.choice([1, 1, 2, 4]), "z": rng.randint(3, max(3, 24 >> level)),
                "y": _log_int(rng, 6, hi), "x": _log_int(rng, 6, hi)}
        if kind == "conv":
            if case["y"] * case["x"] > (228 >> level) ** 2:
                case["b"] = 1
            case["grad"] = rng.random() < 0.4
        return case
    while True:
        nnum = rng.choice([5, 7, 15, 15, 15, 19])
        ly, lx = _log_int(rng, 5, 67), _log_int(rng, 5, 67)
        case = {"kind": kind, "nnum": nnum, "y": ly * nnum - rng.choice([0, 0, rng.randrange(nnum)]),
                "x": lx * nnum - rng.choice([0, 0, rng.randrange(nnum)]), "planes": _log_int(rng, 3, 41),
                "reach": _log_int(rng, 2, 28), "frames": rng.choice([1, 1, 1, 2, 3, 4, 5, 8])}
        if kind in ("rl", "series"):
            case["iters"] = rng.randint(1, 8)
        if kind == "rl":
            case["trust"] = rng.random() < 0.4
        most = listed()[6 if kind in ("rl", "series") else 4]
        w, m = work(case), work(most)
        if max(ly, lx) + case["reach"] <= 96 and w["bytes"] <= m["bytes"] and w["flops"] <= m["flops"]:
            return case


# ---------------------------------------------------------------------------
# The microscope: a PSF set with the shapes and symmetries of a light-field PSF
# ---------------------------------------------------------------------------
def _plane_sizes(case):
    """PSF side of each plane: 2 * Nnum * max(2, lenslets reached at that depth) + 1."""
    n = case["planes"]
    zs = [abs(2.0 * k / (n - 1) - 1.0) if n > 1 else 1.0 for k in range(n)]
    return [2 * case["nnum"] * max(2, math.ceil(case["reach"] * z - 1e-9)) + 1 for z in zs]


def _profiles(N, h, spread, sigma, gamma, alpha):
    """Spots under successive lenslets along one axis, for each of the N offsets; each sums to 1."""
    c, ch, K = N // 2, (h - 1) // 2, max(1, (h // 2) // N - 1)
    d = np.arange(-ch, ch + 1, dtype=np.float64)
    ks = np.arange(-K, K + 1, dtype=np.float64)
    weight = np.exp(-ks ** 2 / (2.0 * (0.5 + 0.6 * spread) ** 2))
    u = np.zeros((N, h))
    for b in range(N):
        centre = ks * N + gamma * (b - c) + alpha * ks
        u[b] = (weight[:, None] * np.exp(-(d[None, :] - centre[:, None]) ** 2 / (2.0 * sigma ** 2))).sum(0)
        u[b] /= u[b].sum()
    return u


@functools.lru_cache(maxsize=1)
def _psf_set(nnum, planes, reach):
    """(H, Ht): per plane the float32 quadrant [n_h, n_h, h, h] of the offsets' PSFs on the host.  Ht is the
    adjoint of H: Ht_ba(y, x) = H_{(b+y-ch) % N, (a+x-ch) % N}(2ch - y, 2ch - x)."""
    N, nh = nnum, (nnum + 1) // 2
    case = {"nnum": nnum, "planes": planes, "reach": reach}
    H, Ht = [], []
    for k, h in enumerate(_plane_sizes(case)):
        z = 2.0 * k / (planes - 1) - 1.0 if planes > 1 else 1.0
        rel, sgn, ch = abs(z), (1.0 if z >= 0 else -1.0), (h - 1) // 2
        yy = np.arange(h)
        h2 = torch.zeros((nh, nh, h, h), dtype=torch.float64, device="cuda")
        t2 = torch.zeros_like(h2)
        for weight, u in ((0.75, _profiles(N, h, reach * rel, 0.9 + 0.8 * rel, 0.55, 0.35 * sgn * rel)),
                          (0.25, _profiles(N, h, 0.5 * reach * rel + 0.5, 1.6 + 1.2 * rel, -0.3, 0.15 * sgn * rel))):
            ut = np.stack([u[(b + yy - ch) % N, 2 * ch - yy] for b in range(nh)])
            a, b = (torch.as_tensor(v, device="cuda") for v in (np.ascontiguousarray(u[:nh]), ut))
            h2 += weight * a[:, None, :, None] * a[None, :, None, :]
            t2 += weight * b[:, None, :, None] * b[None, :, None, :]
        H.append(h2.float().cpu().numpy())
        Ht.append(t2.float().cpu().numpy())
    return H, Ht


Microscope = collections.namedtuple("Microscope", "matrix projector")


@functools.lru_cache(maxsize=1)
def _microscope(nnum, planes, reach):
    """What a program keeps for its microscope: the PSF matrix and a projector for it."""
    H, Ht = _psf_set(nnum, planes, reach)
    return Microscope(psfmatrix.HMatrixArrays(H, Ht), proj.Projector_gb300(device=0))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _beads(shape, per_pixel, rng):
    """[..., Y, X] float64 on the device: Gaussian beads (sigma 1 pixel, amplitude 500..1000) at random places."""
    v = np.zeros(shape)
    n = max(3, int(v.size * per_pixel))
    np.put(v, rng.integers(0, v.size, n), rng.uniform(500.0, 1000.0, n))
    t = torch.as_tensor(v, device="cuda")
    for axis in (-1, -2):
        t = sum(math.exp(-s * s / 2.0) * torch.roll(t, s, axis) for s in range(-3, 4))
    return t


def _image(case, seed):
    """Camera frames [T, Y, X] float32 on the host: spots of unequal brightness on a background of 100, Poisson noise."""
    rng = np.random.default_rng([seed, 1])
    clean = _beads((case["frames"], case["y"], case["x"]), 2e-2, rng).cpu().numpy()
    return rng.poisson(0.3 * clean + 100.0).astype(np.float32)


def _volume(case, seed):
    """Volume [Z, T, Y, X] float32 on the device: beads over a faint background."""
    rng = np.random.default_rng([seed, 2])
    return (_beads((case["planes"], case["frames"], case["y"], case["x"]), 1e-4, rng) + 1.0).float()


def _trust(case):
    """Trust mask [Y, X]: one lenslet in the middle of the image is dead."""
    m, n = np.ones((case["y"], case["x"]), np.float32), case["nnum"]
    y, x = (case["y"] // n // 2) * n, (case["x"] // n // 2) * n
    m[y:y + n, x:x + n] = 0
    return m


def _randn(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda")


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _layer(case, seed):
    """Tensors of one layer: activations after a ReLU, He-scaled weights, bias, gradients, mask."""
    g, (B, Z, Y, X, ci, co) = _gen(seed), (case[k] for k in ("b", "z", "y", "x", "ci", "co"))
    bf = torch.bfloat16
    if case["kind"] == "wgrad":
        return {"x": _randn((B, Z, Y, X, ci), g).clamp_min(0).to(bf), "dy": (1e-2 * _randn((B, Z, Y, X, co), g)).to(bf)}
    t = {"w": (_randn((27, ci, co), g) * math.sqrt(2.0 / (27 * ci))).to(bf)}
    if case["grad"]:
        t["x"] = (1e-2 * _randn((B, Z, Y, X, ci), g)).to(bf)
        t["mask"] = _randn((B, Z, Y, X, co), g).clamp_min(0).to(bf)
    else:
        t["x"] = _randn((B, Z, Y, X, ci), g).clamp_min(0).to(bf)
        t["bias"] = 0.1 * _randn((co,), g)
    return t


def _net_weights(seed):
    """The network's state dict: He-scaled weights, small biases; the head predicts channel 0, the first layer is 3x3x1."""
    rng, d = np.random.default_rng([seed, 3]), {}
    for name, ci, co, relu in warmstart.LAYERS:
        w = rng.standard_normal((27, ci, co)).astype(np.float32) * math.sqrt((2.0 if relu else 1.0) / (27 * ci))
        if name == "head":
            w[:, :, 1:] = 0
        if name == "e0a":
            w[[t for t in range(27) if t % 3 != 1]] = 0
        d[name + ".w"] = w
        d[name + ".b"] = (0.05 * rng.standard_normal(co)).astype(np.float32)
    return d


def _net_input(case, seed):
    """[B, Z, Y, X, 16] bf16: four features of x - 1, x and x + 1 (the first RL iterate, a smoother one, two sensitivity maps)."""
    g = _gen(seed)
    shape = tuple(case[k] for k in ("b", "z", "y", "x"))
    f = torch.stack([_randn(shape, g).abs(), 1 + 0.3 * _randn(shape, g), 1 + 0.1 * _randn(shape, g),
                     1 + 0.1 * _randn(shape, g)], -1)
    x = torch.zeros(shape + (16,), device="cuda")
    for k in range(3):
        s = torch.roll(f, 1 - k, 3)
        if k != 1:
            s[:, :, :, 0 if k == 0 else -1] = 0
        x[..., 4 * k:4 * k + 4] = s
    return x.to(torch.bfloat16)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "backward", "rl", "series"):
        m = _microscope(case["nnum"], case["planes"], case["reach"])
        m.projector.storeVolumesOnGPU = True
        s = {"kind": kind, "m": m, "case": case}
        if kind == "forward":
            s["volume"] = _volume(case, seed)
        elif kind == "backward" or kind == "series":
            s["image"] = torch.as_tensor(_image(case, seed), device="cuda")
        else:
            s["image"] = _image(case, seed)
            s["mask"] = _trust(case) if case["trust"] else None
            if case["trust"]:
                s["image"] *= s["mask"]
            # the program's own host buffer for the result
            s["out"] = torch.empty((case["planes"], case["frames"], case["y"], case["x"]), pin_memory=True).numpy()
        return s
    if kind == "unet":
        net = warmstart.UNet3D(device=0, seed=0)
        net.load_state_dict(_net_weights(seed))
        return {"kind": kind, "net": net, "x": _net_input(case, seed)}
    s = _layer(case, seed)
    s["kind"], s["case"] = kind, case
    n = s["x"][..., 0].numel()
    if kind == "conv":
        if max(case["ci"], case["co"]) >= 64:      # the deep layers' weights are laid out once
            s["wp"] = torch.empty_like(s["w"])
            _flf.conv3d_pack(s["w"], s["wp"], torch.cuda.current_stream().cuda_stream)
        out = n * case["co"]
        s["ws"] = torch.empty(out * (4 if out < (1 << 23) else 1), dtype=torch.float32, device="cuda")
    else:
        s["ws"] = torch.empty(max(64 * 27 * case["ci"] * case["co"], n * case["co"] // 2048 + case["co"]),
                              dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "forward":
        return lfdeconv.ForwardProjectACC(s["m"].matrix, s["volume"], projector=s["m"].projector, logPrint=False)
    if kind == "backward":
        return lfdeconv.BackwardProjectACC(s["m"].matrix, s["image"], projector=s["m"].projector, logPrint=False)
    if kind == "rl":
        trust = s["mask"] is not None
        return lfdeconv.DeconvRL(s["m"].matrix, None, s["case"]["iters"], None, logPrint=False,
                                 projector=s["m"].projector, im=s["image"], prevedel=not trust, trustMask=s["mask"],
                                 out=s["out"])
    if kind == "series":
        m = s["m"]
        htf = lfdeconv.BackwardProjectACC(m.matrix, s["image"], projector=m.projector, logPrint=False)
        return m.projector.RichardsonLucy(m.matrix, htf.clone(), htf, s["case"]["iters"])
    if kind == "unet":
        return s["net"].forward(s["x"])[0]
    x, case, stream = s["x"], s["case"], torch.cuda.current_stream().cuda_stream
    if kind == "conv":
        y = torch.empty(tuple(x.shape[:4]) + (case["co"],), dtype=torch.bfloat16, device="cuda")
        _flf.conv3d(x, s["w"], s.get("bias"), y, relu=not case["grad"], mask=s.get("mask"), stream=stream, ws=s["ws"],
                    wp=s.get("wp"))
        return y
    dw = torch.zeros((27, case["ci"], case["co"]), dtype=torch.float32, device="cuda")
    db = torch.zeros(case["co"], dtype=torch.float32, device="cuda")
    _flf.conv3d_wgrad(x, s["dy"], dw, stream, ws=s["ws"])
    _flf.bias_grad(s["dy"], db, stream, ws=s["ws"])
    return dw, db


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
_UNET = [("e0a", 0, 16, 16, 9), ("e0b", 0, 16, 16, 27), ("e1a", 1, 16, 32, 27), ("e1b", 1, 32, 32, 27), ("e2a", 2, 32, 64, 27),
         ("e2b", 2, 64, 64, 27), ("e3a", 3, 64, 128, 27), ("e3b", 3, 128, 128, 27), ("u2", 3, 128, 64, 27),
         ("d2", 2, 64, 64, 27), ("u1", 2, 64, 32, 27), ("d1", 1, 32, 32, 27), ("u0", 1, 32, 16, 27), ("d0", 0, 16, 16, 27),
         ("head", 0, 16, 1, 27)]


def work(case):
    """Bytes: the inputs and outputs once, weights once, and for projections the stored PSF quadrants once per
    projection (they exceed the caches, so each projection streams them).  Operations: per plane, frame and
    projection one complex multiply-add per lenslet offset and frequency of an F x F real transform that holds
    image and PSF, 8 N^2 F (F/2 + 1); for layers 2 per multiply-add."""
    kind = case["kind"]
    if kind in ("conv", "wgrad", "unet"):
        m = case["b"] * case["z"] * case["y"] * case["x"]
        if kind == "unet":
            flops = sum(2.0 * taps * (m >> (3 * lv)) * ci * co for _, lv, ci, co, taps in _UNET)
            return {"bytes": m * 2 * 16 * 2, "flops": flops}
        ci, co = case["ci"], case["co"]
        flops = 2.0 * 27 * m * ci * co
        if kind == "wgrad":
            return {"bytes": m * 2 * (ci + co) + 4 * (27 * ci * co + co), "flops": flops + m * co}
        return {"bytes": m * 2 * (ci + co * (2 if case["grad"] else 1)) + 2 * 27 * ci * co, "flops": flops}
    N, Y, X, T = (case[k] for k in ("nnum", "y", "x", "frames"))
    psf, flops = 0.0, 0.0
    for h in _plane_sizes(case):
        psf += 4.0 * ((N + 1) // 2) ** 2 * h * h
        F = N * -(-(max(Y, X) + h - 1) // N)
        flops += 8.0 * N * N * F * (F / 2 + 1) * T
    projections = 1                             # RL: Htf, two projections an iteration, the trust mask's back projection
    if kind in ("rl", "series"):
        projections += 2 * case["iters"] + (1 if case.get("trust") else 0)
    return {"bytes": projections * psf + 4.0 * T * Y * X * (1 + case["planes"]), "flops": projections * flops}


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """Projections in 64 bits: per plane, the sum over lenslet offsets (b, a) of the image masked to that
    offset and convolved ('same') with the offset's PSF, taken apart into the N x N pixel positions under a
    lenslet, so that every convolution is one over lenslets, done by an FFT that holds it without wrapping."""

    def __init__(self, case, directions):
        self.N, self.Y, self.X = case["nnum"], case["y"], case["x"]
        N = self.N
        self.Ly, self.Lx = -(-self.Y // N), -(-self.X // N)
        H, Ht = _psf_set(case["nnum"], case["planes"], case["reach"])
        self.sets = {"H": H, "Ht": Ht}
        self.kept = {}
        size = sum((16.0 * N ** 4 * self._f(q.shape[-1])[0] * (self._f(q.shape[-1])[1] // 2 + 1)) for q in H)
        self.keep = size * len(directions) < 60e9

    def _f(self, h):
        r = ((h - 1) // 2 + self.N - 1) // self.N
        return self.Ly + r, self.Lx + r, r

    def transfer(self, name, z):
        """T[i, j, u]: from pixel position i to j under a lenslet, complex128."""
        if (name, z) in self.kept:
            return self.kept[name, z]
        N, c, q = self.N, self.N // 2, torch.as_tensor(self.sets[name][z], device="cuda").double()
        h = q.shape[-1]
        fy, fx, r = self._f(h)
        fy, fx = max(fy, 2 * r + 1), max(fx, 2 * r + 1)
        ch, side = (h - 1) // 2, (2 * r + 1) * N
        T = torch.empty((N * N, N * N, fy, fx // 2 + 1), dtype=torch.complex128, device="cuda")
        for b in range(N):
            for a in range(N):
                bb, aa = min(b, N - 1 - b), min(a, N - 1 - a)
                p = q[bb, aa] if aa >= bb else q[aa, bb].T      # the stored quadrant's symmetry map
                if b > c:
                    p = p.flip(0)
                if a > c:
                    p = p.flip(1)
                # entry (m, beta), (n, alpha) of the padded PSF is its value at pixel (mN + beta - b, nN + alpha - a)
                k = torch.zeros((side + 2 * N, side + 2 * N), dtype=torch.float64, device="cuda")
                oy, ox = r * N + b - ch, r * N + a - ch
                k[N + oy:N + oy + h, N + ox:N + ox + h] = p
                k = k[N:N + side, N:N + side].reshape(2 * r + 1, N, 2 * r + 1, N).permute(1, 3, 0, 2)
                full = torch.zeros((N, N, fy, fx), dtype=torch.float64, device="cuda")
                full[:, :, :2 * r + 1, :2 * r + 1] = k
                full = torch.roll(full, (-r, -r), (2, 3))
                T[b * N + a] = torch.fft.rfft2(full).reshape(N * N, fy, fx // 2 + 1)
        if self.keep:
            self.kept[name, z] = T
        return T

    def _project(self, name, z, image):
        """One plane: [T, Y, X] -> [T, Y, X]."""
        N, t = self.N, image.shape[0]
        T = self.transfer(name, z)
        _, _, r = self._f(self.sets[name][z].shape[-1])
        fy, fx = max(self.Ly + r, 2 * r + 1), max(self.Lx + r, 2 * r + 1)
        pad = torch.zeros((t, self.Ly * N, self.Lx * N), dtype=torch.float64, device="cuda")
        pad[:, :self.Y, :self.X] = image
        s = pad.reshape(t, self.Ly, N, self.Lx, N).permute(2, 4, 0, 1, 3).reshape(N * N, t, self.Ly, self.Lx)
        S = torch.fft.rfft2(s, s=(fy, fx))
        O = torch.stack([(T * S[:, None, k]).sum(0) for k in range(t)], 1)
        o = torch.fft.irfft2(O, s=(fy, fx))[:, :, :self.Ly, :self.Lx]
        o = o.reshape(N, N, t, self.Ly, self.Lx).permute(2, 3, 0, 4, 1).reshape(t, self.Ly * N, self.Lx * N)
        return o[:, :self.Y, :self.X].contiguous()

    def forward(self, vol):
        return sum(self._project("H", z, vol[z]) for z in range(vol.shape[0]))

    def backward(self, img):
        return torch.stack([self._project("Ht", z, img) for z in range(len(self.sets["Ht"]))])


def _exact_conv(x, w, bias=None):
    """3x3x3 convolution of channels-last x in 64 bits, zeros outside; w [27, ci, co]."""
    B, Z, Y, X, ci = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = torch.zeros((B, Z, Y, X, w.shape[2]), dtype=torch.float64, device="cuda")
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        y += p[:, dz:dz + Z, dy:dy + Y, dx:dx + X] @ w[t]
    return y if bias is None else y + bias


def _exact_unet(case, seed):
    d, x = _net_weights(seed), _net_input(case, seed).double()

    def conv(name, v):
        w = torch.as_tensor(d[name + ".w"], device="cuda").to(torch.bfloat16).double()
        y = _exact_conv(v, w, torch.as_tensor(d[name + ".b"], device="cuda").double())
        return y if name == "head" else y.clamp_min(0)

    def pool(v):
        B, Z, Y, X, C = v.shape
        return v.reshape(B, Z // 2, 2, Y // 2, 2, X // 2, 2, C).mean((2, 4, 6))

    def up(v, skip):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3) + skip

    e0 = conv("e0b", conv("e0a", x))
    e1 = conv("e1b", conv("e1a", pool(e0)))
    e2 = conv("e2b", conv("e2a", pool(e1)))
    e3 = conv("e3b", conv("e3a", pool(e2)))
    d2 = conv("d2", up(conv("u2", e3), e2))
    d1 = conv("d1", up(conv("u1", d2), e1))
    return conv("head", conv("d0", up(conv("u0", d1), e0)))


def _update(x, num, den):
    r = x * (num / den)
    return torch.where(torch.isnan(r), torch.zeros_like(r), r)


def exact(case, seed):
    kind = case["kind"]
    if kind == "unet":
        return _exact_unet(case, seed)
    if kind == "conv":
        t = _layer(case, seed)
        y = _exact_conv(t["x"].double(), t["w"].double(), t["bias"].double() if "bias" in t else None)
        return y * (t["mask"] > 0) if case["grad"] else y.clamp_min(0)
    if kind == "wgrad":
        t = _layer(case, seed)
        x, dy = torch.nn.functional.pad(t["x"].double(), (0, 0, 1, 1, 1, 1, 1, 1)), t["dy"].double()
        B, Z, Y, X, co = dy.shape
        g = dy.reshape(-1, co)
        dw = torch.stack([x[:, k // 9:k // 9 + Z, k // 3 % 3:k // 3 % 3 + Y, k % 3:k % 3 + X].reshape(-1, x.shape[-1]).T @ g
                          for k in range(27)])
        return dw, g.sum(0)
    e = _Exact(case, ("H",) if kind == "forward" else ("Ht",) if kind == "backward" else ("H", "Ht"))
    if kind == "forward":
        return e.forward(_volume(case, seed).double())
    if kind != "backward" and not e.keep:
        return None                             # the transfer matrices of both directions, again in each iteration: minutes
    img = torch.as_tensor(_image(case, seed), device="cuda").double()
    if kind == "rl" and case["trust"]:
        mask = torch.as_tensor(_trust(case), device="cuda").double()
        img = img * mask
        norm = e.backward(mask[None])
        x = e.backward(img)
        for _ in range(case["iters"]):
            x = _update(x, e.backward(img / e.forward(x)), norm)
        return x.cpu().numpy()
    htf = e.backward(img)
    if kind == "backward":
        return htf
    x = htf.clone()
    for _ in range(case["iters"]):
        x = _update(x, htf, e.backward(e.forward(x)))
    return x.cpu().numpy() if kind == "rl" else x
