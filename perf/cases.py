"""Performance cases: the calls that a reconstruction makes, over the sizes it makes them at.

Five families, each through the entry points a program calls:

* ``single``  -- the drop-in NUFFT of one image or one coil's k-space
  (``NufftBackend.forward`` / ``.adjoint``), what a host program that keeps its
  own coil loop calls per (bin, echo, coil);
* ``bin``     -- the batched NUFFT of every (echo, coil) column of a motion bin
  (``forward_bin`` with the samples brought back to acquisition order, as k-space is
  simulated; ``adjoint_bin`` with density weights, as gradients and adjoint
  images are made);
* ``pdhg``    -- ``PdhgSolver.run`` of TVM, TVME and TVMW for a few iterations;
* ``wavelet`` -- the db6 analysis and synthesis of TVMW on every image;
* ``conv``    -- one 3x3x3 convolution layer of the learned warm start:
  inference, and a training step's forward and backward.

Sizes: the workloads of ``synthetic.CONFIGS``, the drop-in calls of a small
scan, and odd sizes as field-of-view scaling makes them.  ``draw`` spreads
further cases over the same ranges.  ``exact`` restates every operation in 64
bits with plain torch: Kaiser-Bessel NUFFT (width 4, oversampling 1.25, the
window by the Abramowitz & Stegun Bessel formulas, coordinates scaled in 32
bits: these are the operation's definition), the PDHG iterations, db6, and the
convolution of operands rounded to bf16.
"""

import importlib
import itertools
import math

import numpy as np
import torch

PKG = "multinodemri-miccai26_b200"


def _mod(name):
    return importlib.import_module(PKG + "." + name)


# ---------------------------------------------------------------------- the cases
def listed():
    return [
        # one image of a small scan at odd sizes: a call whose latency and launches count
        {"name": "single-forward-small", "kind": "single", "adjoint": False, "z": 36, "y": 51, "x": 57,
         "cones": 48, "readout": 120},
        # one coil's k-space of a field-of-view scaled (odd) geometry, in a host program's coil loop
        {"name": "single-adjoint-odd", "kind": "single", "adjoint": True, "z": 84, "y": 117, "x": 100,
         "cones": 170, "readout": 600},
        # a motion bin of the 128 x 128 x 96 four-echo workload: k-space simulation and data duals
        {"name": "bin-forward-128", "kind": "bin", "adjoint": False, "z": 96, "y": 128, "x": 128, "coils": 8,
         "echoes": 4, "cones": 170, "readout": 600},
        # a motion bin of the 160 x 160 x 112 wavelet workload (12 coils): data gradient
        {"name": "bin-adjoint-160", "kind": "bin", "adjoint": True, "z": 112, "y": 160, "x": 160, "coils": 12,
         "echoes": 6, "cones": 266, "readout": 700},
        # a motion bin of the 256 x 256 x 128 workload, the largest: both directions
        {"name": "bin-forward-256", "kind": "bin", "adjoint": False, "z": 128, "y": 256, "x": 256, "coils": 16,
         "echoes": 6, "cones": 683, "readout": 800},
        {"name": "bin-adjoint-256", "kind": "bin", "adjoint": True, "z": 128, "y": 256, "x": 256, "coils": 16,
         "echoes": 6, "cones": 683, "readout": 800},
        # whole reconstructions, a few iterations each: the small single-echo one ...
        {"name": "pdhg-tvm-64", "kind": "pdhg", "algorithm": "tvm", "l2": False, "z": 48, "y": 64, "x": 64,
         "coils": 4, "echoes": 1, "bins": 6, "cones": 85, "readout": 400, "iters": 20},
        # ... the four-echo one with the motion dual coupled over echoes ...
        {"name": "pdhg-tvme-128", "kind": "pdhg", "algorithm": "tvme", "l2": True, "z": 96, "y": 128, "x": 128,
         "coils": 8, "echoes": 4, "bins": 6, "cones": 170, "readout": 600, "iters": 4},
        # ... and the six-echo wavelet one
        {"name": "pdhg-tvmw-160", "kind": "pdhg", "algorithm": "tvmw", "l2": False, "z": 112, "y": 160, "x": 160,
         "coils": 12, "echoes": 6, "bins": 6, "cones": 266, "readout": 700, "iters": 2},
        # the spatial wavelet pair on every image of that workload
        {"name": "wavelet-160", "kind": "wavelet", "z": 112, "y": 160, "x": 160, "echoes": 6, "bins": 6},
        # warm-start inference at full resolution: the decoder's widest layer on one 256 x 256 x 128 volume
        {"name": "conv-inference-256", "kind": "conv", "train": False, "n": 1, "z": 128, "y": 256, "x": 256,
         "cin": 64, "cout": 32},
        # warm-start training on four 32^3 crops: a middle layer's forward and backward
        {"name": "conv-train-32", "kind": "conv", "train": True, "n": 4, "z": 32, "y": 32, "x": 32, "cin": 64,
         "cout": 32},
    ]


def _smooth(n):
    """Whether the oversampled length of n image points factors into 2, 3, 5, 7 (what a plan accepts)."""
    m = math.ceil(1.25 * n)
    for r in (2, 3, 5, 7):
        while m % r == 0:
            m //= r
    return m == 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axis(rng, lo, hi):
    while True:
        n = _log_int(rng, lo, hi)
        if _smooth(n):
            return n


def draw(rng):
    kind = rng.choice(("single", "bin", "bin", "pdhg", "wavelet", "conv"))
    if kind == "single":
        return {"kind": kind, "adjoint": rng.random() < 0.5, "z": _axis(rng, 24, 128), "y": _axis(rng, 32, 256),
                "x": _axis(rng, 32, 256), "cones": _log_int(rng, 40, 700), "readout": _log_int(rng, 100, 800)}
    if kind == "bin":
        while True:
            c = {"kind": kind, "adjoint": rng.random() < 0.5, "z": _axis(rng, 32, 128), "y": _axis(rng, 48, 256),
                 "x": _axis(rng, 48, 256), "coils": rng.choice((1, 3, 4, 5, 6, 8, 8, 10, 12, 16, 16)),
                 "echoes": rng.randint(1, 6), "cones": _log_int(rng, 80, 680), "readout": _log_int(rng, 300, 800)}
            if c["z"] * c["y"] * c["x"] * c["coils"] * c["echoes"] <= 2 ** 23 * 96:
                return c
    if kind == "pdhg":
        while True:
            alg = rng.choice(("tvm", "tvme", "tvmw"))
            c = {"kind": kind, "algorithm": alg, "l2": rng.random() < 0.5, "z": _axis(rng, 32, 112),
                 "y": _axis(rng, 48, 160), "x": _axis(rng, 48, 160), "coils": rng.choice((1, 4, 5, 8, 12)),
                 "echoes": 1 if alg == "tvm" else rng.randint(2, 6), "bins": rng.randint(2, 8),
                 "cones": _log_int(rng, 60, 270), "readout": _log_int(rng, 200, 700), "iters": rng.randint(2, 6)}
            cols = c["coils"] * c["echoes"] * c["bins"] * c["iters"]
            if c["z"] * c["y"] * c["x"] * cols <= 112 * 160 * 160 * 12 * 6 * 6 * 2:
                return c
    if kind == "wavelet":
        return {"kind": kind, "z": _axis(rng, 24, 112), "y": _axis(rng, 40, 160), "x": _axis(rng, 40, 160),
                "echoes": rng.randint(1, 6), "bins": rng.randint(1, 6)}
    cin, cout = rng.choice(((2, 32), (32, 32), (64, 32), (32, 64), (64, 64), (128, 64), (64, 128), (128, 128),
                            (32, 8), (16, 16), (48, 24)))
    if rng.random() < 0.5:                       # training crops at one of the three levels
        s = rng.choice((8, 12, 16, 24, 32))
        return {"kind": "conv", "train": True, "n": rng.randint(1, 8), "z": s, "y": s, "x": s, "cin": cin,
                "cout": cout}
    while True:
        c = {"kind": "conv", "train": False, "n": 1, "z": _log_int(rng, 12, 128), "y": _log_int(rng, 16, 256),
             "x": _log_int(rng, 16, 256), "cin": cin, "cout": cout}
        if c["z"] * c["y"] * c["x"] * cin * cout <= 2 ** 23 * 64 * 32:
            return c


# ---------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _shape(c):
    return (c["z"], c["y"], c["x"])


def _cones(c, bins, seed):
    """Per bin (cones, readout, 3) float32 zyx grid units on the GPU: each bin's share of one set of
    interleaved 3-D cones in shuffled acquisition order, |k| < n / 2 per axis."""
    Z, Y, X = _shape(c)
    tr, ro = c["cones"], c["readout"]
    total = tr * max(bins, 6)
    rng = np.random.default_rng(seed)
    out = []
    order = rng.permutation(total)
    for b in range(bins):
        i = torch.from_numpy(order[b * tr:(b + 1) * tr]).cuda().double()[:, None]
        cos_t = 1.0 - 2.0 * (i + 0.5) / total
        theta = torch.arccos(cos_t)
        r = torch.linspace(0.0, 1.0, ro, dtype=torch.float64, device="cuda")[None, :]
        phi = i * (math.pi * (3.0 - math.sqrt(5.0))) + 2.0 * math.pi * (2.0 + 6.0 * torch.sin(theta)) * r
        st = torch.sin(theta)
        k = torch.stack([cos_t * r * Z, st * torch.sin(phi) * r * Y, st * torch.cos(phi) * r * X], dim=-1)
        out.append((k * (0.5 - 1e-4)).float())
    return out


def _density(c, coords):
    half = torch.tensor(_shape(c), device="cuda", dtype=torch.float32) / 2.0
    return [((k / half) ** 2).sum(-1).clamp(1e-4, 1.0) for k in coords]


def _axes(c):
    return [((torch.arange(n, device="cuda") - n // 2).float() / (n / 2.0)).view(
        [-1 if j == i else 1 for j in range(3)]) for i, n in enumerate(_shape(c))]


def _maps(c, g):
    """(C, Z, Y, X) complex64: Gaussian coils on a cylinder with random linear phase, unit root sum of squares."""
    zz, yy, xx = _axes(c)
    C = c["coils"]
    maps = []
    par = torch.rand((C, 4), generator=g, device="cuda").cpu().tolist()
    for i in range(C):
        ang = 2.0 * math.pi * i / C
        mag = torch.exp(-((zz - 0.5 * math.cos(7.0 * ang)) ** 2 + (yy - 1.1 * math.sin(ang)) ** 2
                          + (xx - 1.1 * math.cos(ang)) ** 2) / 1.28)
        p = par[i]
        phase = 3.0 * ((p[0] - 0.5) * zz + (p[1] - 0.5) * yy + (p[2] - 0.5) * xx) + 6.283 * p[3]
        maps.append(torch.polar(mag, phase.expand_as(mag).contiguous()))
    m = torch.stack(maps)
    return m / m.abs().square().sum(0).sqrt().clamp_min(1e-12)


def _ellipsoids(g, count=6):
    """Rows (centre zyx, semi-axes zyx, amplitude, phase): centres and axes as fractions of half the volume."""
    r = torch.rand((count, 8), generator=g, device="cuda").cpu()
    r[:, 0:3] = (r[:, 0:3] - 0.5) * 0.9
    r[:, 3:6] = 0.16 + 0.34 * r[:, 3:6]
    r[:, 6] = 0.4 + 0.6 * r[:, 6]
    r[:, 7] = 6.283 * r[:, 7]
    return r.tolist()


def _images(c, g, lead):
    """Ellipsoid phantoms with 1 % complex noise, lead + (Z, Y, X) complex64."""
    zz, yy, xx = _axes(c)
    n = int(np.prod(lead))
    out = torch.empty((n,) + _shape(c), dtype=torch.complex64, device="cuda")
    ells = _ellipsoids(g)
    masks = [(((zz - e[0]) / e[3]) ** 2 + ((yy - e[1]) / e[4]) ** 2 + ((xx - e[2]) / e[5]) ** 2 <= 1.0) for e in ells]
    for i in range(n):
        im = 0.01 * torch.randn(_shape(c), generator=g, dtype=torch.complex64, device="cuda")
        for j, (e, m) in enumerate(zip(ells, masks)):
            decay = e[6] * math.exp(-0.15 * (j + 1) * (i % 6))
            im += m * complex(decay * math.cos(e[7] + 0.4 * i), decay * math.sin(e[7] + 0.4 * i))
        out[i] = im
    return out.reshape(tuple(lead) + _shape(c))


def _kspace(c, g, k, ncol):
    """(ncol, M) complex64 ellipsoid k-space at the samples k (per-column gains), with 1 % noise and
    largest magnitude near one: the closed-form transform 3 (sin q - q cos q) / q^3 of each ellipsoid."""
    kk = k.reshape(-1, 3)
    half = torch.tensor(_shape(c), device="cuda", dtype=torch.float32) / 2.0
    f = kk / half                                # cycles over half the volume are pi f
    basis, gains = [], []
    for e in _ellipsoids(g):
        q = math.pi * (f * torch.tensor(e[3:6], device="cuda")).norm(dim=1) * half.min()
        q = q.clamp_min(1e-2)
        mag = 3.0 * (torch.sin(q) - q * torch.cos(q)) / q ** 3
        ph = -math.pi * (f * torch.tensor(e[0:3], device="cuda") * half).sum(1) + e[7]
        basis.append(torch.polar(mag.abs(), ph + math.pi * (mag < 0)))
        gains.append(e[6] * e[3] * e[4] * e[5])
    mix = torch.randn((ncol, len(basis)), generator=g, dtype=torch.complex64, device="cuda")
    mix = mix * torch.tensor(gains, device="cuda") / sum(gains)
    out = torch.empty((ncol, kk.shape[0]), dtype=torch.complex64, device="cuda")
    basis = torch.stack(basis)
    for i in range(ncol):
        col = (mix[i][:, None] * basis).sum(0)
        out[i] = col + 0.01 * torch.randn(col.shape, generator=g, dtype=torch.complex64, device="cuda")
    return out


def _inputs(case, seed):
    """Everything a case's plan, run and 64-bit restatement are made from."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "conv":
        shp = (case["n"], case["z"], case["y"], case["x"])
        x = torch.randn(shp + (case["cin"],), generator=g, device="cuda").relu_()     # activations after a CReLU
        w = torch.randn((case["cout"], 27, case["cin"]), generator=g, device="cuda") / math.sqrt(27 * case["cin"])
        b = 0.1 * torch.randn(case["cout"], generator=g, device="cuda")
        gy = 1e-3 * torch.randn(shp + (case["cout"],), generator=g, device="cuda") if case["train"] else None
        return {"x": x, "w": w, "b": b, "gy": gy}
    if kind == "wavelet":
        return {"images": _images(case, g, (case["bins"], case["echoes"])), "gen": g}
    bins = case.get("bins", 1)
    d = {"coords": _cones(case, bins, seed)}
    if kind == "single":
        d["in"] = _kspace(case, g, d["coords"][0], 1)[0] if case["adjoint"] else _images(case, g, (1,))[0]
        return d
    d["dcf"] = _density(case, d["coords"])
    d["maps"] = _maps(case, g)
    ncol = case["coils"] * case["echoes"]
    if kind == "pdhg":
        d["ksp"] = [_kspace(case, g, k, ncol).reshape((case["echoes"], case["coils"]) + tuple(k.shape[:2]))
                    for k in d["coords"]]
    elif case["adjoint"]:
        d["in"] = _kspace(case, g, d["coords"][0], ncol)
    else:
        d["in"] = _images(case, g, (case["echoes"],))
    return d


def _tree(case, width, g):
    """Random (bins * echoes, width) dual coefficients within the projection radius."""
    return 1e-2 * torch.randn((case["bins"] * case["echoes"], width), generator=g, dtype=torch.complex64,
                              device="cuda")


# ---------------------------------------------------------------------- the calls
def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "conv":
        st = {"kind": kind, "train": case["train"], "b": d["b"], "w": d["w"], "x": d["x"], "gy": d["gy"]}
        if case["train"]:
            for name in ("x", "w", "b"):
                st[name].requires_grad_(True)
        return st
    nb = _mod("nufft_backend")
    if kind == "wavelet":
        be = nb.B200NufftBackend(_shape(case), [np.zeros((1, 3), np.float32)] * case["bins"], 0, n_coils=1,
                                 n_echoes=case["echoes"])
        return {"kind": kind, "be": be, "images": d["images"], "tree": _tree(case, be.wavelet_coeffs, d["gen"])}
    if kind == "single":
        be = nb.create_nufft_backend("b200", img_shape=_shape(case), coordinates=d["coords"], device=0)
        return {"kind": kind, "adjoint": case["adjoint"], "be": be, "in": d["in"].reshape(
            d["coords"][0].shape[:2] if case["adjoint"] else _shape(case))}
    if kind == "bin":
        be = nb.B200NufftBackend(_shape(case), d["coords"], 0, dcf=d["dcf"], n_coils=case["coils"],
                                 n_echoes=case["echoes"])
        be.set_maps(d["maps"])
        x = be.sort_kspace(d["in"], 0) if case["adjoint"] else d["in"]
        return {"kind": kind, "adjoint": case["adjoint"], "be": be, "in": x}
    solver = _mod("solver").PdhgSolver(case["algorithm"], _shape(case), d["coords"], d["dcf"], d["maps"], d["ksp"],
                                       l2_coupling=case["l2"])
    return {"kind": kind, "solver": solver, "iters": case["iters"]}


def run(state):
    kind = state["kind"]
    if kind == "single":
        return (state["be"].adjoint if state["adjoint"] else state["be"].forward)(state["in"], 0)
    if kind == "bin":
        if state["adjoint"]:
            return state["be"].adjoint_bin(state["in"], 0)
        return state["be"].unsort_kspace(state["be"].forward_bin(state["in"], 0), 0)
    if kind == "pdhg":
        res = state["solver"].run(max_iter=state["iters"], tol=0.0)
        return {"image": res.image, "u": state["solver"].u, "tols": res.tols}
    if kind == "wavelet":
        return state["be"].wavelet_forward(state["images"]), state["be"].wavelet_adjoint(state["tree"])
    conv3d = _mod("warmstart").conv3d
    if not state["train"]:
        with torch.no_grad():
            return conv3d(state["x"], state["w"], state["b"])
    y = conv3d(state["x"], state["w"], state["b"])
    gx, gw, gb = torch.autograd.grad(y, (state["x"], state["w"], state["b"]), state["gy"])
    return {"y": y.detach(), "gx": gx, "gw": gw, "gb": gb}


# ---------------------------------------------------------------------- unavoidable work
def _tree_sizes(shape):
    """(coefficients per image, [(input shape, output shape) per level, finest first])."""
    levels = min(max(0, int(math.floor(math.log2(n / 11)))) if n >= 11 else 0 for n in shape)
    cur, sizes, total = tuple(shape), [], 0
    for _ in range(levels):
        out = tuple((n + 11) // 2 for n in cur)
        sizes.append((cur, out))
        total += 7 * out[0] * out[1] * out[2]
        cur = out
    return total + cur[0] * cur[1] * cur[2], sizes


def _nufft_flops(case, ncol, samples):
    os_ = [math.ceil(1.25 * n) for n in _shape(case)]
    Z, Y, X = _shape(case)
    fft = (Z * Y * os_[2] * 5 * math.log2(os_[2]) + Z * os_[1] * os_[2] * 5 * math.log2(os_[1])
           + os_[0] * os_[1] * os_[2] * 5 * math.log2(os_[0]))
    return ncol * (fft + samples * 64 * 4)


def work(case):
    kind = case["kind"]
    if kind == "conv":
        v = case["n"] * case["z"] * case["y"] * case["x"]
        ci, co = case["cin"], case["cout"]
        wb = 27 * ci * co * 4
        if case["train"]:    # x, gy, w in; y, gx, gw, gb out
            return {"bytes": 4.0 * v * (2 * ci + 2 * co) + 2 * wb, "flops": 3 * 2.0 * v * 27 * ci * co}
        return {"bytes": 4.0 * v * (ci + co) + wb, "flops": 2.0 * v * 27 * ci * co}
    n = case["z"] * case["y"] * case["x"]
    if kind == "wavelet":
        ncoef, sizes = _tree_sizes(_shape(case))
        images = case["bins"] * case["echoes"]
        points = sum(2 * o[0] * i[1] * i[2] + 4 * o[0] * o[1] * i[2] + 8 * o[0] * o[1] * o[2] for i, o in sizes)
        return {"bytes": 16.0 * images * (n + ncoef), "flops": 2 * images * points * 12 * 4.0}
    m = case["cones"] * case["readout"]
    if kind == "single":
        return {"bytes": 8.0 * (n + m) + 12.0 * m, "flops": _nufft_flops(case, 1, m)}
    ncol = case["coils"] * case["echoes"]
    if kind == "bin":
        return {"bytes": 8.0 * (case["echoes"] * n + case["coils"] * n + m * ncol) + 16.0 * m,
                "flops": _nufft_flops(case, ncol, m)}
    # an iteration reads and writes the primal and dual state once and reads the k-space, maps and samples
    be = case["bins"] * case["echoes"]
    arrays = {"tvm": 3, "tvme": 6, "tvmw": 4}[case["algorithm"]]
    state = 16.0 * be * n * arrays + 24.0 * case["bins"] * m * ncol + 8.0 * case["coils"] * n
    flops = 2 * case["bins"] * _nufft_flops(case, ncol, m) + 60.0 * be * n
    if case["algorithm"] == "tvmw":
        state += 16.0 * be * _tree_sizes(_shape(case))[0]
        flops += 2 * be * 12 * 4.0 * 10 * n
    return {"bytes": case["iters"] * state, "flops": case["iters"] * flops}


# ---------------------------------------------------------------------- 64-bit restatements
def _bessel_i0(x):
    t = (x / 3.75) ** 2
    small = 1.0 + t * (3.5156229 + t * (3.0899424 + t * (1.2067492 + t * (0.2659732 + t * (0.0360768
                       + t * 0.0045813)))))
    u = 3.75 / x.clamp_min(3.75)
    poly = 0.39894228 + u * (0.01328592 + u * (0.00225319 + u * (-0.00157565 + u * (0.00916281 + u * (
        -0.02057706 + u * (0.02635537 + u * (-0.01647633 + u * 0.00392377)))))))
    big = torch.exp(x) / torch.sqrt(x.clamp_min(1.0)) * poly
    return torch.where(x < 3.75, small, big)


class _Nufft:
    """Width-4, 1.25x Kaiser-Bessel NUFFT of (ncol, Z, Y, X) complex128 images at one bin's samples."""

    def __init__(self, shape, coords):
        self.n = tuple(shape)
        self.os = tuple(math.ceil(1.25 * n) for n in shape)
        beta = math.pi * math.sqrt((4 / 1.25 * (1.25 - 0.5)) ** 2 - 0.8)
        k = coords.reshape(-1, 3).float()
        self.taps, self.apod = [], []
        for i, (n, o) in enumerate(zip(self.n, self.os)):
            ks = (k[:, i] * float(np.float32(o / n)) + float(o // 2)).double()        # scaled in 32 bits
            first = torch.ceil(ks - 2.0)
            at = first[:, None] + torch.arange(5, device="cuda")
            d = (at - ks[:, None]) / 2.0
            w = torch.where(d.abs() <= 1.0, _bessel_i0(beta * torch.sqrt((1.0 - d * d).clamp_min(0.0))), 0.0)
            self.taps.append((torch.remainder(at, o).long(), w))
            r = torch.sqrt(beta ** 2 - (math.pi * 4 * (torch.arange(n, device="cuda").double() - n // 2) / o) ** 2)
            self.apod.append((r / torch.sinh(r)).view([-1 if j == i else 1 for j in range(3)]))
        self.scale = 1.0 / (math.sqrt(float(np.prod(self.n))) * 64.0)
        self.box = tuple(slice(o // 2 - n // 2, o // 2 - n // 2 + n) for n, o in zip(self.n, self.os))

    def _pairs(self):
        """(grid index, weight, sample index or None for all) of every tap that some sample has."""
        (tz, wz), (ty, wy), (tx, wx) = self.taps
        for a, b, c in itertools.product(range(5), repeat=3):
            w = wz[:, a] * wy[:, b] * wx[:, c]
            idx = (tz[:, a] * self.os[1] + ty[:, b]) * self.os[2] + tx[:, c]
            if 4 in (a, b, c):                       # the fifth tap: integer coordinates only
                s = torch.nonzero(w)[:, 0]
                if s.numel():
                    yield idx[s], w[s], s
            else:
                yield idx, w, None

    def forward(self, x):
        grid = torch.zeros((x.shape[0],) + self.os, dtype=torch.complex128, device="cuda")
        grid[(slice(None),) + self.box] = x * (self.apod[0] * self.apod[1] * self.apod[2]) * self.scale
        dims = (1, 2, 3)
        grid = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(grid, dim=dims), dim=dims), dim=dims)
        grid = grid.reshape(x.shape[0], -1).T.contiguous()
        out = torch.zeros((self.taps[0][0].shape[0], x.shape[0]), dtype=torch.complex128, device="cuda")
        for idx, w, s in self._pairs():
            if s is None:
                out += w[:, None] * grid[idx]
            else:
                out[s] += w[:, None] * grid[idx]
        return out.T

    def adjoint(self, y):
        ncol = y.shape[0]
        grid = torch.zeros((int(np.prod(self.os)), 2 * ncol), dtype=torch.float64, device="cuda")
        v = y.T.contiguous()
        for idx, w, s in self._pairs():
            t = w[:, None] * (v if s is None else v[s])
            grid.index_add_(0, idx, torch.view_as_real(t).reshape(-1, 2 * ncol))
        grid = torch.view_as_complex(grid.view(-1, ncol, 2)).T.reshape((ncol,) + self.os)
        dims = (1, 2, 3)
        im = torch.fft.ifftn(torch.fft.ifftshift(grid, dim=dims), dim=dims, norm="forward")
        im = torch.fft.fftshift(im, dim=dims)[(slice(None),) + self.box]
        return im * (self.apod[0] * self.apod[1] * self.apod[2]) * self.scale


def _chunk(shape):
    """Columns that one step of the restatement holds at a time (about 4 GB of grids)."""
    return max(1, int(2e8 / np.prod([1.25 * n for n in shape])) // 2)


def _bin_forward(nf, images, maps, echoes, coils):
    """images (E, Z, Y, X), maps (C, Z, Y, X) -> (E * C, M) complex128."""
    out, step = [], _chunk(nf.n)
    for e in range(echoes):
        for c in range(0, coils, step):
            out.append(nf.forward(images[e].to(torch.complex128) * maps[c:c + step]))
    return torch.cat(out)


def _bin_adjoint(nf, ksp, maps, echoes, coils, dcf):
    out, step = [], _chunk(nf.n)
    for e in range(echoes):
        im = 0
        for c in range(0, coils, step):
            m = maps[c:c + step].to(torch.complex128)
            im = im + (m.conj() * nf.adjoint(ksp[e * coils + c:e * coils + c + len(m)].to(torch.complex128)
                                             * dcf)).sum(0)
        out.append(im)
    return torch.stack(out)


_DB6 = (0.11154074335010940, 0.49462389039845290, 0.75113390802109490, 0.31525035170919800, -0.22626469396543930,
        -0.12976686756726188, 0.09750160558732306, 0.02752286553030561, -0.03158203931748598, 0.00055384220116150,
        0.00477725751094551, -0.00107730108530848)
_REC_HI = tuple((-1.0 if j % 2 else 1.0) * h for j, h in enumerate(reversed(_DB6)))


def _analyse(x, dim):
    """(low, high) halves along one axis: c[o] = sum_j f[j] x[2 o + 1 - j], zeros outside."""
    n = x.shape[dim]
    no = (n + 11) // 2
    x = x.movedim(dim, -1)
    x = torch.nn.functional.pad(torch.view_as_real(x.contiguous()), (0, 0, 10, 2 * no - n + 1))
    lo = hi = 0
    for j in range(12):
        v = x[..., 11 - j:11 - j + 2 * no - 1:2, :]
        lo = lo + _DB6[11 - j] * v
        hi = hi + _REC_HI[11 - j] * v
    return tuple(torch.view_as_complex(v.contiguous()).movedim(-1, dim) for v in (lo, hi))


def _synthesise(lo, hi, dim, n):
    """y[o] = sum_j rec_lo[2 j + o % 2] lo[i - j] + rec_hi[...] hi[i - j], i = o // 2 + 5, for o < n."""
    lo, hi = (torch.nn.functional.pad(torch.view_as_real(v.movedim(dim, -1).contiguous()), (0, 0, 0, 6))
              for v in (lo, hi))
    half = (n + 1) // 2
    out = []
    for par in (0, 1):
        s = 0
        for j in range(6):
            s = s + _DB6[2 * j + par] * lo[..., 5 - j:5 - j + half, :] + _REC_HI[2 * j + par] * hi[
                ..., 5 - j:5 - j + half, :]
        out.append(s)
    y = torch.stack(out, dim=-2).flatten(-3, -2)[..., :n, :]
    return torch.view_as_complex(y.contiguous()).movedim(-1, dim)


def _wavedec(x):
    """(coefficients,) tree of one (Z, Y, X) complex128 image: coarsest first."""
    _, sizes = _tree_sizes(x.shape)
    parts = []
    for _ in sizes:
        bands = []
        for a in _analyse(x, 0):
            for b in _analyse(a, 1):
                bands += list(_analyse(b, 2))
        parts.append(torch.stack(bands[1:]).reshape(-1))
        x = bands[0]
    return torch.cat([x.reshape(-1)] + parts[::-1])


def _waverec(tree, shape):
    _, sizes = _tree_sizes(shape)
    top = sizes[-1][1]
    at = top[0] * top[1] * top[2]
    x = tree[:at].reshape(top)
    for inp, out in reversed(sizes):
        sub = out[0] * out[1] * out[2]
        d = tree[at:at + 7 * sub].reshape((7,) + out)
        at += 7 * sub
        x = x[:out[0], :out[1], :out[2]]
        bands = [x] + list(d)
        bands = [_synthesise(bands[2 * i], bands[2 * i + 1], 2, inp[2]) for i in range(4)]
        bands = [_synthesise(bands[2 * i], bands[2 * i + 1], 1, inp[1]) for i in range(2)]
        x = _synthesise(bands[0], bands[1], 0, inp[0])
    return x


def _forward_diff(u, dim):
    d = torch.zeros_like(u)
    n = u.shape[dim]
    d.narrow(dim, 0, n - 1).copy_(u.narrow(dim, 1, n - 1) - u.narrow(dim, 0, n - 1))
    return d


def _forward_diff_adjoint(p, dim):
    d = torch.zeros_like(p)
    n = p.shape[dim]
    d.narrow(dim, 0, n - 1).sub_(p.narrow(dim, 0, n - 1))
    d.narrow(dim, 1, n - 1).add_(p.narrow(dim, 0, n - 1))
    return d


def _echo_pair(u, adjoint):
    """db1 pair along the echo axis (dim 1); an odd last echo meets a zero."""
    E = u.shape[1]
    out = torch.empty_like(u)
    s = math.sqrt(0.5)
    for e in range(E):
        other = e + 1 if e % 2 == 0 else e - 1
        v = u[:, other] if other < E else torch.zeros_like(u[:, e])
        if e % 2 == 0:
            out[:, e] = s * (u[:, e] - v if adjoint else u[:, e] + v)
        else:
            out[:, e] = s * (u[:, e] + v if adjoint else u[:, e] - v)
    return out


def _pdhg(case, d):
    alg, B, E, C = case["algorithm"], case["bins"], case["echoes"], case["coils"]
    sigma = tau = 1.0 / 6.0
    lam = 1e-5
    shape = _shape(case)
    nf = [_Nufft(shape, k) for k in d["coords"]]
    maps = d["maps"].to(torch.complex128)
    z = lambda: torch.zeros((B, E) + shape, dtype=torch.complex128, device="cuda")  # noqa: E731
    u, ub, pm = z(), z(), z()
    pe = [z(), z(), z()] if alg == "tvme" else None
    pw1 = z() if alg == "tvmw" else None
    pw2 = (torch.zeros((B * E, _tree_sizes(shape)[0]), dtype=torch.complex128, device="cuda")
           if alg == "tvmw" else None)
    y = [k.reshape(E * C, -1).to(torch.complex128) for k in d["ksp"]]
    q = [torch.zeros_like(v) for v in y]
    tols = []
    clip = lambda p, r: p / torch.clamp(r / lam, min=1.0)  # noqa: E731
    for _ in range(case["iters"]):
        for b in range(B):
            q[b] = (q[b] + sigma * (_bin_forward(nf[b], ub[b], maps, E, C) - y[b])) / (1.0 + sigma)
        pm = pm + sigma * _forward_diff(ub, 0)
        pm = clip(pm, pm.abs().square().sum(1, keepdim=True).sqrt() if case["l2"] else pm.abs())
        if alg == "tvme":
            de = _forward_diff(ub, 1)
            pe = [p + sigma * _forward_diff(de, k) for p, k in zip(pe, (4, 3, 2))]
            r = sum(p.abs().square() for p in pe).sqrt()
            pe = [clip(p, r) for p in pe]
        if alg == "tvmw":
            pw1 = pw1 + sigma * _echo_pair(ub, False)
            pw1 = clip(pw1, pw1.abs())
            w2 = z()
            for i in range(B * E):
                t = pw2[i] + sigma * _wavedec(ub[i // E, i % E])
                t = t * torch.clamp(lam / torch.sqrt(t.abs().square() + 1e-12), max=1.0)
                pw2[i] = t
                w2[i // E, i % E] = _waverec(t, shape)
        g = torch.stack([_bin_adjoint(nf[b], q[b], maps, E, C, d["dcf"][b].reshape(1, -1).double())
                         for b in range(B)])
        if alg == "tvmw":    # the motion divergence without the last bin's edge row
            dm = pm.clone()
            dm[1:] -= pm[:-1]
            r = g - dm + _echo_pair(pw1, True) + w2
        else:
            r = g + _forward_diff_adjoint(pm, 0)
            if alg == "tvme":
                r = r + _forward_diff_adjoint(sum(_forward_diff_adjoint(p, k) for p, k in zip(pe, (4, 3, 2))), 1)
        un = u - tau * r
        new = 2.0 * un - u
        if alg == "tvmw":
            tols.append(float((ub - new).norm()) / max(float(ub.norm()), 1e-12))
        else:
            tols.append(float((un - u).norm()) / float(un.norm()))
        u, ub = un, new
    # the first iteration's TVMW tolerance divides by the clamped zero image: no number to compare
    return {"image": ub, "u": u, "tols": [t if t < 1e6 else None for t in tols]}


def _conv(x, w):
    """(N, D, H, W, Cin) x (Cout, 27, Cin) in 64 bits, zero padding one."""
    N, D, H, W, ci = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = torch.empty((N, D, H, W, w.shape[0]), dtype=torch.float64, device="cuda")
    for n in range(N):
        for d0 in range(0, D, 16):
            d1 = min(D, d0 + 16)
            acc = 0
            for t in range(27):
                a, b, c = t // 9, (t // 3) % 3, t % 3
                acc = acc + p[n, d0 + a:d1 + a, b:b + H, c:c + W].double() @ w[:, t].double().T
            out[n, d0:d1] = acc
    return out


def _conv_wgrad(x, gy):
    N, D, H, W, ci = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    g = gy.double().reshape(-1, gy.shape[-1])
    rows = []
    for t in range(27):
        a, b, c = t // 9, (t // 3) % 3, t % 3
        v = p[:, a:a + D, b:b + H, c:c + W].double().reshape(-1, ci)
        rows.append(g.T @ v)
    return torch.stack(rows, dim=1)


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "conv":
        x, w = d["x"].bfloat16(), d["w"].bfloat16()
        y = _conv(x, w) + d["b"].double()
        if not case["train"]:
            return y
        gy = d["gy"].bfloat16()
        return {"y": y, "gx": _conv(gy, w.flip(1).permute(2, 1, 0)), "gw": _conv_wgrad(x, gy),
                "gb": d["gy"].double().sum(dim=(0, 1, 2, 3))}
    if kind == "wavelet":
        images = d["images"].to(torch.complex128)
        ncoef, sizes = _tree_sizes(_shape(case))
        tree = _tree(case, ncoef, d["gen"])
        fwd = torch.stack([_wavedec(im) for im in images.reshape((-1,) + _shape(case))])
        adj = torch.stack([_waverec(t.to(torch.complex128), _shape(case)) for t in tree])
        return fwd, adj.reshape(images.shape)
    if kind == "single":
        nf = _Nufft(_shape(case), d["coords"][0])
        x = d["in"].to(torch.complex128)[None]
        return nf.adjoint(x)[0] if case["adjoint"] else nf.forward(x)[0].reshape(d["coords"][0].shape[:2])
    if kind == "bin":
        nf = _Nufft(_shape(case), d["coords"][0])
        if case["adjoint"]:
            return _bin_adjoint(nf, d["in"], d["maps"], case["echoes"], case["coils"],
                                d["dcf"][0].reshape(1, -1).double())
        return _bin_forward(nf, d["in"], d["maps"].to(torch.complex128), case["echoes"], case["coils"])
    # two NUFFTs per column, bin and iteration: about 20 s of 64-bit work at this bound
    if np.prod(_shape(case)) * case["coils"] * case["echoes"] * case["bins"] * case["iters"] > 2.6e9:
        return None
    return _pdhg(case, d)
