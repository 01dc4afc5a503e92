"""Performance cases: the work that programs on this package give it, with inputs made on the GPU from a seed.

Every case goes through the package's public entry points: the functional interpolation, gridding, NUFFT, block
and sampling calls, the SENSE normal operator of the CG reconstruction, and the convolution layer of the learned
preconditioner. ``exact`` restates each one in float64 with plain torch."""

import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "torch-named-linops_gb300"))

import torchlinops_gb300 as T  # noqa: E402
from torchlinops_gb300 import linops, mri, precond  # noqa: E402

DEV = "cuda"
OVERSAMP = 1.25


def kb_beta(width):
    """The NUFFT's Kaiser-Bessel shape parameter at an oversampling of 1.25."""
    return math.pi * (((width / OVERSAMP) * (OVERSAMP - 0.5)) ** 2 - 0.8) ** 0.5


def _interp(name, op, size, entries, npts, density, **kw):
    """An interpolation case: ``size`` is the (oversampled) grid as "X" joined text, e.g. "64x64"."""
    c = dict(name=name, op=op, size=size, entries=entries, npts=npts, density=density, width=4.0, kernel="kaiser_bessel",
             pad="circular", beta=kb_beta(4.0), dtype="complex64")
    c.update(kw)
    return c


def listed():
    return [
        # The smallest calls of a 2D program: one image, one slice (64^2, 4096 points), forward and adjoint.
        # Launches and the host path count here.
        _interp("interp2d_small", "both", "64x64", 1, 4096, "uniform"),
        # One coil or one combined image in 3D (a single-coil scan, one basis image of a subspace fit), forward
        # and adjoint, points spread evenly, with the functional default beta = 1.
        _interp("interp3d_one_entry", "both", "128x128x128", 1, 262144, "uniform", beta=1.0),
        # The large multicoil 3D workload: 256^3 oversampled grid, 8 coils, 2^21 points with a dense centre.
        # Its forward and its adjoint are what a CG iteration spends its time in.
        _interp("ungrid3d_multicoil", "ungrid", "256x256x256", 8, 1 << 21, "ball"),
        _interp("grid3d_multicoil", "grid", "256x256x256", 8, 1 << 21, "ball"),
        # A clinical matrix that is no power of two (100 x 120 x 108, oversampled by 1.25) and a coil count that
        # is no multiple of 8: 3D radial spokes, forward and adjoint.
        _interp("interp3d_ragged", "both", "125x150x135", 12, 400000, "radial"),
        # A wider kernel chosen for accuracy (width 6), zero padding, a 2D multislice batch, forward and adjoint.
        _interp("interp2d_wide", "both", "320x320", 20, 131072, "radial", width=6.0, pad="zero", beta=kb_beta(6.0)),
        # One application of the 3D SENSE normal operator: what every CG iteration of a reconstruction does
        # (128^3 image, 8 coils, 2^20 radial points, regularised).
        dict(name="sense3d_normal", op="sense", n=128, coils=8, spokes=2048, readout=512),
        # One step of trajectory optimisation: the differentiable 2D NUFFT of 32 slices x 8 coils, forward,
        # gradients of the images and of the trajectory, which is another one at every step.
        dict(name="nufft2d_train", op="train2d", n=256, slices=32, coils=8, spokes=402, readout=512),
        # Dynamic imaging: each frame comes with its own trajectory, in physical units, and is gridded once.
        dict(name="grid3d_new_trajectory", op="frame", size="160x160x160", entries=8, npts=1 << 18),
        # Overlapping blocks of a 3D series (locally low-rank regularisation): all blocks out, and summed back.
        dict(name="blocks3d", op="blocks", size="160x160x160", entries=16, block="8x8x8", stride="4x4x4",
             dtype="complex64"),
        # Cartesian-like sampling at integer locations: gather and the accumulating adjoint, 8 coils.
        dict(name="sampling3d", op="sampling", size="160x160x160", entries=8, npts=1 << 20),
        # One hidden layer of the preconditioner network in training: forward, data gradient, weight gradient.
        dict(name="conv_layer_train", op="conv", size="128x128x128"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _x(dims):
    return "x".join(str(int(d)) for d in dims)


def draw(rng):
    op = rng.choice(["interp3d", "interp3d", "interp3d", "interp2d", "interp2d", "sense", "train2d", "frame", "blocks",
                     "sampling", "conv"])
    if op == "interp3d":
        n = _log(rng, 32, 224)
        size = [max(24, n + rng.randint(-n // 4, n // 8)) for _ in range(3)]
        return _draw_interp(rng, size, _log(rng, 1, 16), _log(rng, 2000, 1 << 20))
    if op == "interp2d":
        n = _log(rng, 48, 512)
        size = [max(32, n + rng.randint(-n // 4, n // 8)) for _ in range(2)]
        wide = rng.random() < 0.25
        kw = dict(width=6.0, beta=kb_beta(6.0)) if wide else {}
        return _draw_interp(rng, size, _log(rng, 1, 64), _log(rng, 1000, 200000), **kw)
    if op == "sense":
        n = rng.randint(32, 128)
        return dict(op="sense", n=n, coils=rng.randint(1, 12), spokes=_log(rng, 64, 2048), readout=2 * n)
    if op == "train2d":
        n = rng.randint(48, 256)
        return dict(op="train2d", n=n, slices=_log(rng, 1, 24), coils=rng.randint(1, 8), spokes=_log(rng, 32, 400),
                    readout=2 * n)
    if op == "frame":
        n = _log(rng, 32, 176)
        size = [max(24, n + rng.randint(-n // 4, n // 8)) for _ in range(3)]
        entries = max(1, min(_log(rng, 1, 12), (1 << 25) // math.prod(size)))
        return dict(op="frame", size=_x(size), entries=entries, npts=_log(rng, 2000, 1 << 19))
    if op == "blocks":
        nd = rng.choice([2, 3])
        block = [rng.randint(4, 9) for _ in range(nd)]
        stride = [rng.randint((b + 1) // 2, b) for b in block]
        size = [rng.randint(64, 320) if nd == 2 else rng.randint(32, 128) for _ in range(nd)]
        return dict(op="blocks", size=_x(size), entries=_log(rng, 1, 16), block=_x(block), stride=_x(stride),
                    dtype=rng.choice(["complex64", "complex64", "float32"]))
    if op == "sampling":
        nd = rng.choice([2, 3])
        size = [rng.randint(64, 320) if nd == 2 else rng.randint(32, 160) for _ in range(nd)]
        return dict(op="sampling", size=_x(size), entries=_log(rng, 1, 12), npts=_log(rng, 2000, 1 << 20))
    return dict(op="conv", size=_x([rng.randint(24, 128) for _ in range(3)]))


def _draw_interp(rng, size, entries, npts, **kw):
    entries = max(1, min(entries, (1 << 25) // math.prod(size)))  # at most 2^25 grid values
    c = _interp("", rng.choice(["both", "ungrid", "grid"]), _x(size), entries, npts,
                rng.choice(["uniform", "ball", "radial"]), pad=rng.choice(["circular", "circular", "zero"]), **kw)
    del c["name"]
    if rng.random() < 0.15:
        c["dtype"] = "float32"
    if rng.random() < 0.15:
        c["kernel"], c["beta"] = "spline", 1.0
    return c


# ------------------------------------------------------------------- inputs


def _dims(text):
    return tuple(int(v) for v in text.split("x"))


def _gen(seed, stream=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + stream)


def _randn(shape, gen, dtype=torch.complex64):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=dtype)


def _directions(n, nd, gen):
    u = torch.randn(n, nd, generator=gen, device=DEV)
    return u / u.norm(dim=-1, keepdim=True)


def _locs(size, npts, density, width, gen):
    """[npts, D] float32 points in grid units."""
    s = torch.tensor(size, device=DEV, dtype=torch.float32)
    nd = len(size)
    if density == "uniform":  # half a kernel width away from the edges
        return torch.rand(npts, nd, generator=gen, device=DEV) * (s - width) + width / 2
    if density == "ball":  # r ~ U(0, 1): density ~ 1/r^2 in 3D, 1/r in 2D
        r = torch.rand(npts, 1, generator=gen, device=DEV)
        return s / 2 + r * (s / 2) * _directions(npts, nd, gen)
    # radial spokes through the centre, rotated and slightly jittered per seed
    read = max(16, min(512, 2 * max(size)))
    spokes = -(-npts // read)
    d = _directions(spokes, nd, gen)
    r = (torch.arange(read, device=DEV, dtype=torch.float32) - read // 2) / read
    l = (d[:, None, :] * r[None, :, None]).reshape(-1, nd)[:npts] * s
    return l + s / 2 + 0.05 * torch.randn(npts, nd, generator=gen, device=DEV)


def _spokes(case, nd, gen):
    """Centred radial trajectory in [-n/2, n/2): [spokes, readout, nd] float32, with the jitter of a real scan."""
    n, read = case["n"], case["readout"]
    d = _directions(case["spokes"], nd, gen)
    r = (torch.arange(read, device=DEV, dtype=torch.float32) - read // 2) * (n / read)
    l = d[:, None, :] * r[None, :, None]
    return (l + 0.1 * torch.randn(l.shape, generator=gen, device=DEV)).clamp_(-n / 2, n / 2 - 1e-3).contiguous()


def _coil_maps(n, coils, gen):
    """[coils, n, n, n] complex64 smooth sensitivities, normalised."""
    ax = torch.linspace(-0.5, 0.5, n, device=DEV)
    c = _directions(coils, 3, gen) * 0.3
    g = [torch.exp(-((ax[None, :] - c[:, e:e + 1]) ** 2) / (2 * 0.4**2)) for e in range(3)]
    ph = torch.rand(coils, 3, generator=gen, device=DEV)
    p = [torch.exp(2j * math.pi * ph[:, e:e + 1] * ax[None, :]) for e in range(3)]
    m = [a * b for a, b in zip(g, p)]
    S = m[0][:, :, None, None] * m[1][:, None, :, None] * m[2][:, None, None, :]
    return (S / (S.abs() ** 2).sum(0, keepdim=True).sqrt()).to(torch.complex64).contiguous()


def _inputs(case, seed):
    op, g = case["op"], _gen(seed)
    if op in ("both", "ungrid", "grid"):
        size, dt = _dims(case["size"]), getattr(torch, case["dtype"])
        s = {"locs": _locs(size, case["npts"], case["density"], case["width"], g)}
        if op != "grid":
            s["img"] = _randn((case["entries"], *size), g, dt)
        if op != "ungrid":
            s["vals"] = _randn((case["entries"], case["npts"]), g, dt)
        return s
    if op == "sense":
        n = case["n"]
        return {"locs": _spokes(case, 3, g).reshape(-1, 3), "maps": _coil_maps(n, case["coils"], g),
                "x": _randn((n, n, n), g)}
    if op == "train2d":
        n = case["n"]
        l = _spokes(case, 2, g)
        b = (case["slices"], case["coils"])
        return {"locs": l, "x": _randn((*b, n, n), g), "w": _randn((*b, *l.shape[:-1]), g)}
    if op == "frame":
        size = _dims(case["size"])
        # k-space positions in cycles per metre over a field of view of 0.24 m
        k = (_locs(size, case["npts"], "ball", 4.0, g) - torch.tensor(size, device=DEV) / 2) / 0.24
        return {"k": k, "vals": _randn((case["entries"], case["npts"]), g)}
    if op == "blocks":
        return {"x": _randn((case["entries"], *_dims(case["size"])), g, getattr(torch, case["dtype"]))}
    if op == "sampling":
        size = _dims(case["size"])
        # variable density: Gaussian around the centre, clipped to the grid
        idx = tuple((s / 2 + torch.randn(case["npts"], generator=g, device=DEV) * (s / 5)).long().clamp_(0, s - 1)
                    for s in size)
        return {"idx": idx, "img": _randn((case["entries"], *size), g), "vals": _randn((case["entries"], case["npts"]), g)}
    if op == "conv":
        size = _dims(case["size"])
        b16 = torch.bfloat16
        return {"x": torch.randn(*size, 16, generator=g, device=DEV).to(b16),
                "w": (torch.randn(27, 16, 16, generator=g, device=DEV) / math.sqrt(27 * 16)).to(b16),
                "gy": torch.randn(*size, 16, generator=g, device=DEV).to(b16)}
    raise ValueError(op)


def prepare(case, seed):
    s = _inputs(case, seed)
    op = s["op"] = case["op"]
    if op in ("both", "ungrid", "grid"):
        kp = dict(beta=case["beta"]) if case["kernel"] == "kaiser_bessel" else {}
        s["size"] = _dims(case["size"])
        s["opts"] = dict(width=case["width"], kernel=case["kernel"], pad_mode=case["pad"], kernel_params=kp)
    elif op == "sense":
        s["A"] = mri.SenseNormal(s.pop("locs"), s.pop("maps"), lam=1e-3, normalise=False)
    elif op == "train2d":
        s["x"].requires_grad_(True)
        s["locs"].requires_grad_(True)
    elif op == "frame":
        s["size"] = _dims(case["size"])
        s["centre"] = torch.tensor(s["size"], device=DEV) / 2
        s["kp"] = dict(beta=kb_beta(4.0))
    elif op == "blocks":
        s["size"], s["block"], s["stride"] = (_dims(case[k]) for k in ("size", "block", "stride"))
    elif op == "sampling":
        s["size"] = _dims(case["size"])
    return s


def run(s):
    op = s["op"]
    if op == "both":
        return (T.interpolate(s["img"], s["locs"], **s["opts"]),
                T.interpolate_adjoint(s["vals"], s["locs"], s["size"], **s["opts"]))
    if op == "ungrid":
        return T.interpolate(s["img"], s["locs"], **s["opts"])
    if op == "grid":
        return T.interpolate_adjoint(s["vals"], s["locs"], s["size"], **s["opts"])
    if op == "sense":
        return s["A"](s["x"])
    if op == "train2d":
        y = linops.nufft(s["x"], s["locs"])
        gx, gl = torch.autograd.grad(y, (s["x"], s["locs"]), s["w"])
        return y.detach(), gx, gl
    if op == "frame":
        locs = s["k"] * 0.24 + s["centre"]
        return T.interpolate_adjoint(s["vals"], locs, s["size"], 4.0, kernel_params=s["kp"])
    if op == "blocks":
        y = T.array_to_blocks(s["x"], s["block"], s["stride"])
        return y, T.blocks_to_array(y, s["size"], s["block"], s["stride"])
    if op == "sampling":
        return T.index(s["img"], s["idx"]), T.index_adjoint(s["vals"], s["idx"], s["size"])
    if op == "conv":
        return (precond.conv3d(s["x"], s["w"]), precond.conv3d(s["gy"], precond.flip_weights(s["w"])),
                precond.conv3d_wgrad(s["x"], s["gy"]))
    raise ValueError(op)


def work(case):
    """Bytes: each input read once and each output written once. Flops: the taps' multiply-adds, the FFTs at
    5 n log2 n, the convolutions' products."""
    op = case["op"]
    if op in ("both", "ungrid", "grid", "frame"):
        size = _dims(case["size"])
        vol, nd = math.prod(size), len(size)
        es = 4 if case.get("dtype") == "float32" else 8
        e, p = case["entries"], case["npts"]
        taps = int(case.get("width", 4.0)) ** nd
        k = 2 if op == "both" else 1
        return {"bytes": e * es * (vol + p) * k + 4 * nd * p, "flops": k * p * e * taps * es / 2}
    if op == "sense":
        n, c, p = case["n"], case["coils"], case["spokes"] * case["readout"]
        m = int(n * OVERSAMP) ** 3
        return {"bytes": 8 * (2 + c) * n**3 + 12 * p, "flops": c * (10 * m * math.log2(m) + 2 * p * 64 * 4)}
    if op == "train2d":
        n, e, p = case["n"], case["slices"] * case["coils"], case["spokes"] * case["readout"]
        m = int(n * OVERSAMP) ** 2
        return {"bytes": e * 8 * (2 * n * n + 2 * p) + 16 * p, "flops": e * (10 * m * math.log2(m) + 4 * p * 16 * 4)}
    if op == "blocks":
        size, block, stride = (_dims(case[k]) for k in ("size", "block", "stride"))
        nb = math.prod((a - b) // s + 1 for a, b, s in zip(size, block, stride))
        es = 4 if case["dtype"] == "float32" else 8
        blocks, arr = nb * math.prod(block), math.prod(size)
        return {"bytes": es * case["entries"] * 2 * (blocks + arr), "flops": case["entries"] * blocks * es / 4}
    if op == "sampling":
        size = _dims(case["size"])
        vol, e, p = math.prod(size), case["entries"], case["npts"]
        return {"bytes": 8 * (e * 3 * p + e * vol + min(vol, p) * e) + 8 * len(size) * p, "flops": 2 * p * e}
    vox = math.prod(_dims(case["size"]))
    return {"bytes": vox * 16 * 2 * 4, "flops": 3 * vox * 2 * 27 * 256}


# ------------------------------------------------------- the same in 64 bits
#
# The kernel is the Kaiser-Bessel window by the Abramowitz & Stegun expansions 9.8.1 and 9.8.2 of I0, as the
# reference defines it; which taps a window has is decided by the float32 coordinates, as there.

_AS1 = (1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813)
_AS2 = (0.39894228, 0.01328592, 0.00225319, -0.00157565, 0.00916281, -0.02057706, 0.02635537, -0.01647633, 0.00392377)


def _horner(c, t):
    y = torch.full_like(t, c[-1])
    for a in reversed(c[:-1]):
        y = y * t + a
    return y


def _kb(d, beta):
    z = beta * (1 - d * d).clamp_min(0).sqrt()
    zb = z.clamp_min(3.75)
    return torch.where(z < 3.75, _horner(_AS1, (z / 3.75) ** 2), zb.exp() / zb.sqrt() * _horner(_AS2, 3.75 / zb))


def _kb_slope(d, beta):
    """d KB / d d."""
    z = beta * (1 - d * d).clamp_min(0).sqrt()
    u = (z / 3.75) ** 2
    small = -2 * beta**2 * d / 3.75**2 * _horner([k * a for k, a in enumerate(_AS1)][1:], u)
    zb = z.clamp_min(3.75)
    v = 3.75 / zb
    q, dq = _horner(_AS2, v), _horner([k * a for k, a in enumerate(_AS2)][1:], v)
    big = zb.exp() / zb.sqrt() * (q * (1 - 0.5 / zb) - dq * 3.75 / zb**2) * (-(beta**2) * d / zb)
    return torch.where(z < 3.75, small, big)


def _axis(x, n, width, kernel, beta, pad, slope=False):
    """(cells [P, K] in [0, n), weights [P, K], slopes or None) of one coordinate (float32 [P])."""
    r = torch.tensor(width, dtype=torch.float32, device=x.device) / 2
    cell = torch.ceil(x - r)[:, None] + torch.arange(math.ceil(width + 1), device=x.device)
    d32 = (x[:, None] - cell) / r
    ok = (d32.abs() <= r) & (d32.abs() <= 1 if kernel == "kaiser_bessel" else True)
    if pad == "zero":
        ok = ok & (cell >= 0) & (cell < n)
    d = (x[:, None].double() - cell.double()) / r.double()
    w = _kb(d, beta) if kernel == "kaiser_bessel" else (1 - d.abs()).clamp_min(0)
    zero = torch.zeros_like(w)
    cell = torch.remainder(cell.long(), n)
    return cell, torch.where(ok, w, zero), torch.where(ok, _kb_slope(d, beta) / r.double(), zero) if slope else None


def _taps(locs, size, width, kernel, beta, pad, slope=False):
    """Yields (cells [P], weights [P], slopes [D, P] or None) for each tap of the windows."""
    ax = [_axis(locs[:, e], n, width, kernel, beta, pad, slope) for e, n in enumerate(size)]
    used = [[k for k in range(a[0].shape[1]) if bool((a[1][:, k] != 0).any())] for a in ax]

    def visit(e, picked):
        if e == len(size):
            cell, w = 0, 1.0
            for a, n, k in zip(ax, size, picked):
                cell, w = cell * n + a[0][:, k], w * a[1][:, k]
            s = None
            if slope:
                s = [math.prod([ax[f][2 if f == g else 1][:, picked[f]] for f in range(len(size))]) for g in range(len(size))]
            yield cell, w, s
            return
        for k in used[e]:
            yield from visit(e + 1, picked + [k])

    yield from visit(0, [])


def _ungrid64(img, locs, size, **o):
    flat = img.reshape(-1, math.prod(size))
    out = torch.zeros(flat.shape[0], locs.shape[0], dtype=flat.dtype, device=flat.device)
    for cell, w, _ in _taps(locs, size, **o):
        out += flat[:, cell] * w
    return out


def _grid64(vals, locs, size, **o):
    v = vals.reshape(-1, locs.shape[0]).T.contiguous()
    cplx = v.is_complex()
    v = torch.view_as_real(v).reshape(v.shape[0], -1) if cplx else v
    out = torch.zeros(math.prod(size), v.shape[1], dtype=v.dtype, device=v.device)
    for cell, w, _ in _taps(locs, size, **o):
        out.index_add_(0, cell, v * w[:, None])
    out = torch.view_as_complex(out.reshape(out.shape[0], -1, 2)) if cplx else out
    return out.T.contiguous().reshape(-1, *size)


def _prepared(locs, n, p):
    return torch.remainder(locs * (p / n) + p // 2, p)


class _Nufft64:
    """Apodisation, centred padded FFT and interpolation (width 4) of an n^nd image, and its adjoint."""

    def __init__(self, n, nd, locs):
        self.n, self.nd, self.p = n, nd, int(n * OVERSAMP)
        self.locs = _prepared(locs.reshape(-1, nd), n, self.p)
        self.size = (self.p,) * nd
        beta = kb_beta(4.0)
        self.opts = dict(width=4.0, kernel="kaiser_bessel", beta=beta, pad="circular")
        g = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
        a = (beta**2 - (math.pi * 4.0 * g / self.p) ** 2).sqrt()
        self.apod = 1.0
        for e in range(nd):
            self.apod = self.apod * (a / torch.sinh(a)).reshape([-1 if f == e else 1 for f in range(nd)])
        t = self.p - n
        left = t // 2 + (1 if t % 2 and n % 2 else 0)
        self.crop = (..., *[slice(left, left + n)] * nd)
        self.dim = tuple(range(-nd, 0))
        self.scale = 1.0 / (4.0**nd * (n / self.p) ** (nd / 2))

    def kspace(self, x):
        z = torch.zeros(*x.shape[: x.ndim - self.nd], *self.size, dtype=torch.complex128, device=x.device)
        z[self.crop] = x.to(torch.complex128) * self.apod
        z = torch.fft.fftn(torch.fft.ifftshift(z, dim=self.dim), dim=self.dim, norm="ortho")
        return torch.fft.fftshift(z, dim=self.dim)

    def image(self, z):
        z = torch.fft.ifftn(torch.fft.ifftshift(z, dim=self.dim), dim=self.dim, norm="ortho")
        return torch.fft.fftshift(z, dim=self.dim)[self.crop] * self.apod

    def points(self, k):
        return _ungrid64(k, self.locs, self.size, **self.opts) * self.scale

    def adjoint(self, y):
        return self.image(_grid64(y * self.scale, self.locs, self.size, **self.opts))


def exact(case, seed):
    op = case["op"]
    s = _inputs(case, seed)
    if op in ("both", "ungrid", "grid"):
        size = _dims(case["size"])
        o = dict(width=case["width"], kernel=case["kernel"], beta=case["beta"], pad=case["pad"])
        up = torch.complex128 if case["dtype"] == "complex64" else torch.float64
        a = _ungrid64(s["img"].to(up), s["locs"], size, **o) if op != "grid" else None
        b = _grid64(s["vals"].to(up), s["locs"], size, **o) if op != "ungrid" else None
        return (a, b) if op == "both" else (a if op == "ungrid" else b)
    if op == "sense":
        F = _Nufft64(case["n"], 3, s["locs"])
        maps = s["maps"].to(torch.complex128)
        out = 1e-3 * s["x"].to(torch.complex128)
        for c in range(maps.shape[0]):
            y = F.points(F.kspace(maps[c] * s["x"])[None])
            out = out + maps[c].conj() * F.adjoint(y)[0]
        return out
    if op == "train2d":
        n, l = case["n"], s["locs"]
        F = _Nufft64(n, 2, l)
        x, w = s["x"].reshape(-1, n, n), s["w"].reshape(s["x"].shape[0] * s["x"].shape[1], -1)
        ys, gx, gl = [], [], torch.zeros(F.locs.shape[0], 2, dtype=torch.float64, device=DEV)
        for b in range(0, x.shape[0], 16):
            k, wb = F.kspace(x[b:b + 16]), w[b:b + 16].to(torch.complex128)
            ys.append(F.points(k))
            gx.append(F.adjoint(wb))
            flat = k.reshape(k.shape[0], -1)
            for cell, _, slope in _taps(F.locs, F.size, slope=True, **F.opts):
                dot = (wb.conj() * flat[:, cell]).real.sum(0)
                for e in range(2):
                    gl[:, e] += dot * slope[e]
        return (torch.cat(ys).reshape(s["w"].shape), torch.cat(gx).reshape(s["x"].shape),
                (gl * (F.scale * F.p / n)).reshape(l.shape))
    if op == "frame":
        size = _dims(case["size"])
        locs = s["k"] * 0.24 + torch.tensor(size, device=DEV) / 2
        return _grid64(s["vals"].to(torch.complex128), locs, size, width=4.0, kernel="kaiser_bessel", beta=kb_beta(4.0),
                       pad="circular")
    if op == "blocks":
        size, block, stride = (_dims(case[k]) for k in ("size", "block", "stride"))
        y, nd = s["x"].to(torch.complex128 if case["dtype"] == "complex64" else torch.float64), len(size)
        out = torch.zeros_like(y)
        for e in range(nd):
            y = y.unfold(1 + e, block[e], stride[e])
        count = [torch.zeros(n, dtype=torch.float64, device=DEV) for n in size]
        for c, n, b, st in zip(count, size, block, stride):
            for i in range((n - b) // st + 1):
                c[i * st:i * st + b] += 1
        out = s["x"].to(out.dtype)
        for e, c in enumerate(count):  # each element comes back once per block that covers it
            out = out * c.reshape([1] + [-1 if f == e else 1 for f in range(nd)])
        return y.contiguous(), out
    if op == "sampling":
        size = _dims(case["size"])
        cell = 0
        for i, n in zip(s["idx"], size):
            cell = cell * n + i
        e = case["entries"]
        out = torch.zeros(math.prod(size), 2 * e, dtype=torch.float64, device=DEV)
        v = torch.view_as_real(s["vals"].to(torch.complex128).T.contiguous()).reshape(-1, 2 * e)
        out.index_add_(0, cell, v)
        adj = torch.view_as_complex(out.reshape(-1, e, 2)).T.contiguous().reshape(e, *size)
        return s["img"].reshape(e, -1)[:, cell].to(torch.complex128), adj
    x, w, gy = (s[k].double() for k in ("x", "w", "gy"))
    D, H, W, _ = x.shape
    pad = torch.nn.functional.pad
    xp, gp = (pad(t, (0, 0, 1, 1, 1, 1, 1, 1)) for t in (x, gy))
    y, gx, dw = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(w)
    for t in range(27):
        a, b, c = t // 9, t // 3 % 3, t % 3
        v = xp[a:a + D, b:b + H, c:c + W]
        y += v @ w[t].T
        gx += gp[2 - a:2 - a + D, 2 - b:2 - b + H, 2 - c:2 - c + W] @ w[t]
        dw[t] = gy.reshape(-1, 16).T @ v.reshape(-1, 16)
    return y, gx, dw
