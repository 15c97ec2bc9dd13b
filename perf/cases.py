"""What a user of this framework has it do, as a list of timed cases.

A case is a dict of plain values. ``kind`` says which public entry point runs:

  nufft      b200_nufft forward and adjoint of a multi-coil image batch
  forward    the forward alone, ``adjoint`` the adjoint alone
  grad       loss ||A(k) x - y||^2 with gradients for image and trajectory
  sense      one normal operator A^H D A of a density-weighted sense_linop
             (what every CG / FISTA iteration applies)
  toeplitz   the same normal with use_toeplitz (FFT-only)
  segments   the normal of a time-segmented off-resonance sense_linop
  batch      CG-SENSE of uneven slices in one plan, replayed from its graph
  dcf        Pipe-Menon density compensation of a trajectory, the whole call

Inputs follow the repository's own workloads: golden-angle radial and
variable-density spiral trajectories in 2D, kooshballs in 3D, Gaussian coil
maps of unit root-sum-of-squares, random images and samples.

``exact`` computes what ``run`` returns in 64 bits with plain torch. The grid
coordinate of a sample and the set of its kernel taps are float32 by the
operator's definition (|j - u| <= W/2 in float32 selects a tap), so those two
are formed in float32 there as well; weights, sums and transforms are 64-bit.
"""

import math

import numpy as np
import torch

from mr_recon_b200.algs import SenseCG, density_compensation
from mr_recon_b200.fourier import b200_nufft
from mr_recon_b200.linops import sense_linop
from mr_recon_b200.plan import Plan

DEV = "cuda"
C64, C128, F64 = torch.complex64, torch.complex128, torch.float64


def listed():
    return [
        # the smallest call: one coil, 128^2, 64 golden-angle spokes x 256, oversampling 2
        # (launch and call latency; a quick look at one channel, a unit of a learned model)
        dict(name="radial128_c1", kind="nufft", n0=128, n1=128, n2=0, coils=1, shots=64, readout=256, os=2.0, width=6.0),
        # the benchmark's headline: 256^2, 32 coils, 48 x 2048 spiral
        dict(name="spiral256_c32", kind="nufft", n0=256, n1=256, n2=0, coils=32, shots=48, readout=2048, os=1.25,
             width=6.0),
        # ragged 2D: odd rectangular matrix whose grid (272 x 326) has large prime factors, 7 coils,
        # an odd width (a protocol's own field of view, coil compression)
        dict(name="odd181x217_c7", kind="nufft", n0=181, n1=217, n2=0, coils=7, shots=37, readout=509, os=1.5, width=5.0),
        # the CG-SENSE iteration at the headline size: density-weighted normal operator
        dict(name="sense256_c32", kind="sense", n0=256, n1=256, n2=0, coils=32, shots=48, readout=2048, os=1.25,
             width=6.0),
        # the same iteration through the Toeplitz embedding
        dict(name="toep256_c32", kind="toeplitz", n0=256, n1=256, n2=0, coils=32, shots=48, readout=2048, os=1.25,
             width=6.0),
        # time-segmented off-resonance: 4 long interleaves, 16 coils, 20 zero-order segments
        dict(name="segments256_c16", kind="segments", n0=256, n1=256, n2=0, coils=16, shots=4, readout=16384, os=1.25,
             width=6.0, nseg=20),
        # a whole solve: uneven slices (160..256 matrix, 8-32 coils, 10k-100k samples) in one graph
        dict(name="batch16_cg", kind="batch", slices=16, mix=4, nmin=160, nmax=256, cmin=8, cmax=32, mmin=10000,
             mmax=100000, os=1.25, width=6.0, iters=8),
        # 3D, 16 coils, 7.68 M kooshball samples: the largest, each direction
        dict(name="koosh192_c16_fwd", kind="forward", n0=192, n1=192, n2=192, coils=16, shots=20000, readout=384, os=1.25,
             width=4.0),
        dict(name="koosh192_c16_adj", kind="adjoint", n0=192, n1=192, n2=192, coils=16, shots=20000, readout=384, os=1.25,
             width=4.0),
        # trajectory optimisation in 3D: image and trajectory gradients of the data loss
        dict(name="koosh128_c8_grad", kind="grad", n0=128, n1=128, n2=128, coils=8, shots=8000, readout=256, os=1.25,
             width=4.0),
        # 3D CG-SENSE iteration at the operator's default kernel (oversampling 1.25, width 6), 12 coils
        dict(name="sense120_c12_w6", kind="sense", n0=120, n1=120, n2=120, coils=12, shots=8000, readout=240, os=1.25,
             width=6.0),
        # density compensation of a 3D trajectory, 30 iterations on one channel
        dict(name="dcf128", kind="dcf", n0=128, n1=128, n2=128, shots=8000, readout=256, iters=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nufft", "nufft", "sense", "toeplitz", "segments", "batch", "forward3", "adjoint3", "grad3", "sense3",
                       "dcf"])
    os = rng.choice([1.25, 1.25, 1.5, 2.0])
    width = rng.choice([4.0, 5.0, 6.0, 6.0, 7.0])
    if kind == "batch":
        nmin = _log(rng, 96, 200)
        mmin = _log(rng, 5000, 40000)
        cmin = _log(rng, 2, 12)
        return dict(kind="batch", slices=_log(rng, 2, 24), mix=rng.randrange(1000), nmin=nmin, nmax=nmin + rng.randrange(8, 64),
                    cmin=cmin, cmax=cmin + rng.randrange(1, 20), mmin=mmin, mmax=mmin * rng.randrange(2, 4), os=1.25,
                    width=rng.choice([4.0, 6.0]), iters=8)
    if kind == "dcf":
        d3 = rng.random() < 0.6
        n = [_log(rng, 40, 144) if d3 else _log(rng, 64, 320) for _ in range(3 if d3 else 2)] + ([] if d3 else [0])
        return dict(kind="dcf", n0=n[0], n1=n[1], n2=n[2], shots=_log(rng, 500, 8000) if d3 else _log(rng, 16, 256),
                    readout=_log(rng, 100, 300), iters=rng.choice([10, 20, 30]))
    if kind in ("forward3", "adjoint3", "grad3", "sense3"):
        top = 176 if kind in ("forward3", "adjoint3") else 128
        n0 = _log(rng, 40, top)
        n1, n2 = (max(24, min(top, int(n0 * rng.uniform(0.6, 1.4)))) for _ in range(2))
        w = rng.choice([4.0, 4.0, 5.0, 6.0])
        return dict(kind=kind[:-1], n0=n0, n1=n1, n2=n2, coils=_log(rng, 1, 16), shots=_log(rng, 500, 8000),
                    readout=_log(rng, 80, 300), os=1.25 if n0 > 100 else rng.choice([1.25, 1.5]), width=w)
    n0 = _log(rng, 64, 384)
    n1 = n0 if rng.random() < 0.4 else max(48, min(384, int(n0 * rng.uniform(0.6, 1.4))))
    case = dict(kind=kind, n0=n0, n1=n1, n2=0, coils=_log(rng, 1, 40), shots=_log(rng, 4, 96), readout=_log(rng, 200, 4000),
                os=os, width=width)
    if kind == "toeplitz":
        # the padded (doubled) grid has to exceed the image by an even number of cells
        case.update(n0=n0 + n0 % 2, n1=n1 + n1 % 2)
    if kind == "segments":
        case.update(os=1.25, nseg=rng.randrange(4, 24), coils=_log(rng, 2, 24))
    return case


# ------------------------------------------------------------------ inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(shape, g):
    return torch.randn(shape, dtype=C64, device=DEV, generator=g)


def _im(case):
    return (case["n0"], case["n1"]) + ((case["n2"],) if case["n2"] else ())


def _clip(unit, im):
    """Trajectory in grid units [-N/2, N/2) from coordinates in [-1, 1]."""
    half = torch.tensor([n / 2.0 for n in im], dtype=F64, device=DEV)
    top = torch.nextafter(half.float(), torch.zeros_like(half.float()))
    return torch.minimum(torch.maximum((unit * half).float(), -half.float()), top).contiguous()


def _spiral(shots, readout, im, g, alpha=1.5):
    """(shots, readout, 2) variable-density spiral and its density weights
    (r dr/dt), rotated by a random angle."""
    turn = torch.rand((), dtype=F64, device=DEV, generator=g) * 2 * math.pi
    t = torch.arange(readout, dtype=F64, device=DEV) / readout
    turns = max(1.0, float(max(im)) / shots)
    th = 2 * math.pi * turns * t + 2 * math.pi * torch.arange(shots, dtype=F64, device=DEV)[:, None] / shots + turn
    r = t ** alpha
    w = (t + 0.5 / readout) ** (2 * alpha - 1)
    return _clip(torch.stack([r * torch.cos(th), r * torch.sin(th)], -1), im), w.expand(shots, readout)


def _radial(shots, readout, im, g):
    """(shots, readout, 2) golden-angle radial spokes from a random first angle."""
    turn = torch.rand((), dtype=F64, device=DEV, generator=g) * 2 * math.pi
    r = torch.arange(readout, dtype=F64, device=DEV) * (2.0 / readout) - 1.0
    a = torch.arange(shots, dtype=F64, device=DEV)[:, None] * math.pi * (3 - math.sqrt(5)) + turn
    return _clip(torch.stack([r * torch.cos(a), r * torch.sin(a)], -1), im), (r.abs() + 0.5 / readout).expand(shots, readout)


def _kooshball(shots, readout, im, g):
    """(shots, readout, 3) spokes through the centre along a phyllotaxis
    half-sphere, turned about the last axis by a random angle."""
    turn = torch.rand((), dtype=F64, device=DEV, generator=g) * 2 * math.pi
    i = torch.arange(shots, dtype=F64, device=DEV) + 0.5
    phi = torch.acos(1 - i / shots)
    th = math.pi * (1 + 5 ** 0.5) * i + turn
    d = torch.stack([torch.sin(phi) * torch.cos(th), torch.sin(phi) * torch.sin(th), torch.cos(phi)], -1)
    r = torch.arange(readout, dtype=F64, device=DEV) * (2.0 / readout) - 1.0
    return _clip(r[None, :, None] * d[:, None, :], im), (r.abs() + 0.5 / readout).square().expand(shots, readout)


def _traj(case, im, g):
    """Trajectory (shots, readout, d) and density weights (shots, readout) that
    sum to the k-space area, so that A^H D A is near the identity."""
    make = _kooshball if len(im) == 3 else _radial if case.get("readout", 0) <= 512 and case["shots"] > 8 else _spiral
    trj, w = make(case["shots"], case["readout"], im, g)
    return trj, (w * (0.7 * math.prod(im) / w.sum())).float().contiguous()


def _maps(coils, im, g):
    """(C, *im) complex Gaussian bumps on a circle, unit root-sum-of-squares."""
    axes = [(torch.arange(n, device=DEV, dtype=torch.float32) - n // 2) / (n / 2) for n in im]
    grids = torch.meshgrid(*axes, indexing="ij")
    a0 = float(torch.rand((), device=DEV, generator=g)) * 2 * math.pi
    m = torch.empty((coils, *im), dtype=C64, device=DEV)
    for c in range(coils):
        a = a0 + 2 * math.pi * c / coils
        cen = [0.8 * math.cos(a), 0.8 * math.sin(a), 0.8 * math.cos(2.4 * a)]
        d2 = sum((x - ci) ** 2 for x, ci in zip(grids, cen))
        m[c] = torch.polar(torch.exp(-d2 / 0.72), a + 0.5 * grids[0] * math.cos(a) + 0.5 * grids[1] * math.sin(a))
    return m / m.abs().square().sum(0).sqrt()


def _segment_functions(case, im, g):
    """Zero-order time segments of a smooth off-resonance map within +-200 Hz
    over a 25 ms readout: b_l(r) = exp(-2 pi i f(r) t_l), one-hot h_l(t)."""
    L, ro = case["nseg"], case["readout"]
    axes = [torch.linspace(-1, 1, n, device=DEV, dtype=F64) for n in im]
    yy, xx = torch.meshgrid(*axes, indexing="ij")
    s = float(torch.rand((), device=DEV, generator=g)) * 0.2
    f = (0.6 - s) * xx + (0.4 + s) * yy - 0.5 * xx * yy + 0.3 * yy ** 2 + torch.exp(-((xx - 0.25) ** 2 + (yy + 0.1) ** 2) / 0.08)
    f = 200.0 * f / f.abs().max()
    tl = (torch.arange(L, device=DEV, dtype=F64) + 0.5) / L * 25e-3
    spatial = torch.polar(torch.ones_like(f), -2 * math.pi * f * tl[:, None, None]).to(C64)
    seg = (torch.arange(ro, device=DEV) * L) // ro
    temporal = (seg[None, None, :] == torch.arange(L, device=DEV)[:, None, None]).to(C64)
    return spatial, temporal.expand(L, case["shots"], ro).contiguous()


def _batch_shapes(case):
    """Matrix, coils and samples of each slice: a property of the case."""
    r = np.random.RandomState(case["mix"])
    S = case["slices"]
    n = r.randint(case["nmin"] // 2, case["nmax"] // 2 + 1, S) * 2
    return ([(int(v), int(v)) for v in n], [int(v) for v in r.randint(case["cmin"], case["cmax"] + 1, S)],
            [int(v) for v in r.randint(case["mmin"], case["mmax"] + 1, S)])


def _inputs(case, seed):
    """The plain tensors of a case."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        out = []
        for im, c, m in zip(*_batch_shapes(case)):
            shots = 16
            trj, w = _spiral(shots, -(-m // shots), im, g)
            trj = trj.reshape(-1, 2)[:m].contiguous()
            w = w.reshape(-1)[:m]
            dcf = (w * (0.7 * math.prod(im) / w.sum())).float()
            out.append(dict(im=im, trj=trj, dcf=dcf, mps=_maps(c, im, g), ksp=_randn((c, m), g)))
        return out
    im = _im(case)
    trj, dcf = _traj(case, im, g)
    s = dict(im=im, trj=trj, dcf=dcf)
    if kind in ("nufft", "forward", "grad"):
        s["img"] = _randn((1, case["coils"], *im), g)
    if kind in ("nufft", "adjoint", "grad"):
        s["ksp"] = _randn((1, case["coils"], *trj.shape[:-1]), g)
    if kind in ("sense", "toeplitz", "segments"):
        s["img"] = _randn(im, g)
        s["mps"] = _maps(case["coils"], im, g)
    if kind == "segments":
        s["spatial"], s["temporal"] = _segment_functions(case, im, g)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        plan = Plan([x["im"] for x in s], [x["trj"].shape[0] for x in s], [x["mps"].shape[0] for x in s], case["os"],
                    (case["width"],) * 2)
        plan.set_traj(torch.cat([x["trj"].reshape(-1) for x in s]))
        cg = SenseCG(plan, torch.cat([x["mps"].reshape(-1) for x in s]), torch.cat([x["dcf"] for x in s]), case["iters"], 1e-2,
                     1.0)
        ksp = torch.cat([x["ksp"].reshape(-1) for x in s])
        return dict(kind=kind, cg=cg.capture(), ksp=ksp)
    s["kind"] = kind
    if kind == "dcf":
        s["iters"] = case["iters"]
        return s
    s["op"] = b200_nufft(s["im"], oversamp=case["os"], width=case["width"])
    if kind in ("sense", "toeplitz"):
        s["A"] = sense_linop(s["trj"], s["mps"], dcf=s["dcf"], nufft=s["op"], use_toeplitz=kind == "toeplitz")
    elif kind == "segments":
        s["A"] = sense_linop(s["trj"], s["mps"], dcf=s["dcf"], nufft=s["op"], spatial_funcs=s["spatial"],
                             temporal_funcs=s["temporal"])
    else:
        s["trj"] = s["trj"][None]
        if kind == "grad":
            s["trj"].requires_grad_(True)
            s["img"].requires_grad_(True)
    return s


def run(state):
    kind = state["kind"]
    if kind == "nufft":
        return state["op"].forward(state["img"], state["trj"]), state["op"].adjoint(state["ksp"], state["trj"])
    if kind == "forward":
        return state["op"].forward(state["img"], state["trj"])
    if kind == "adjoint":
        return state["op"].adjoint(state["ksp"], state["trj"])
    if kind in ("sense", "toeplitz", "segments"):
        return state["A"].normal(state["img"])
    if kind == "batch":
        return state["cg"].solve(state["ksp"])
    if kind == "dcf":
        return density_compensation(state["trj"], state["im"], num_iters=state["iters"])
    loss = (state["op"].forward(state["img"], state["trj"]) - state["ksp"]).abs().square().sum()
    gi, gt = torch.autograd.grad(loss, (state["img"], state["trj"]))
    return loss.detach(), gi, gt


# ------------------------------------------------------------------ work


def _nufft_work(im, os, width, coils, m, fft=1):
    """Bytes and operations of one interpolation or gridding with its FFT."""
    gos = math.prod(math.ceil(os * n) for n in im)
    return 4.0 * coils * m * width ** len(im) + fft * 5.0 * coils * gos * math.log2(max(2, gos))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for im, c, m in zip(*_batch_shapes(case)):
            n = math.prod(im)
            b += 8.0 * c * m + 8.0 * c * n + 8.0 * n + 12.0 * m
            f += (2 * case["iters"] + 3) * _nufft_work(im, case["os"], case["width"], c, m)
        return dict(bytes=b, flops=f)
    im = _im(case)
    n, d, m = math.prod(im), len(im), case["shots"] * case["readout"]
    if kind == "dcf":
        return dict(bytes=4.0 * m * (d + 1), flops=2.0 * case["iters"] * _nufft_work(im, 1.0, 4.0, 1, m, 0))
    c = case["coils"]
    one = _nufft_work(im, case["os"], case["width"], c, m)
    image, samples, coords = 8.0 * c * n, 8.0 * c * m, 4.0 * d * m
    if kind == "nufft":
        return dict(bytes=2 * (image + samples) + coords, flops=2 * one)
    if kind in ("forward", "adjoint"):
        return dict(bytes=image + samples + coords, flops=one)
    if kind == "grad":
        return dict(bytes=2 * image + samples + 2 * coords, flops=2 * one + _nufft_work(im, case["os"], case["width"], c * d, m, 0))
    if kind == "toeplitz":
        gp = math.prod(2 * v for v in im)
        return dict(bytes=image + 16.0 * n + 8.0 * gp, flops=10.0 * c * gp * math.log2(gp) + 6.0 * c * gp)
    if kind == "segments":
        L = case["nseg"]
        return dict(bytes=image + 16.0 * n + 4.0 * m + coords + 8.0 * L * n,
                    flops=2 * (L * (one - _nufft_work(im, case["os"], case["width"], c, m, 0)) +
                               _nufft_work(im, case["os"], case["width"], c, m, 0)))
    return dict(bytes=image + 16.0 * n + 4.0 * m + coords, flops=2 * one)


# ------------------------------------------------------------------ 64-bit values


def _beta(os, width):
    return math.pi * math.sqrt((width / os * (os - 0.5)) ** 2 - 0.8)


class _Exact:
    """Kaiser-Bessel gridding NUFFT in 64 bits on grids [cells, C]."""

    def __init__(self, im, trj, os, width, beta=None, raw=False):
        self.im, self.d, self.width, self.raw = im, len(im), float(width), raw
        self.nos = tuple(im) if raw else tuple(math.ceil(os * n) for n in im)
        self.beta = _beta(os, width) if beta is None else beta
        t = trj.reshape(-1, self.d).float()
        u = []
        for i, (n, k) in enumerate(zip(im, self.nos)):
            scale = np.float32(1.0 if raw else k / n)
            shift = np.float32(n // 2 if raw else k // 2)
            u.append(torch.remainder(t[:, i] * float(scale) + float(shift), float(k)))
        self.u = torch.stack(u, 1)
        self.m = t.shape[0]
        self.taps = int(width) + 1

    def _axis(self, u, i, deriv=False):
        """(m, K) cells and weights (or their derivatives) along axis i."""
        r = torch.tensor(self.width / 2, dtype=torch.float32, device=u.device)
        j = torch.ceil(u - r)[:, None] + torch.arange(self.taps, device=u.device, dtype=torch.float32)
        dx = j - u[:, None]
        ok = dx.abs() <= r
        x = dx.double() / (self.width / 2)
        z = self.beta * (1 - x * x).clamp(min=0).sqrt()
        if deriv:
            # d/du I0(z): dz/du = beta^2 x / (z r), and I1(z)/z -> 1/2 at z = 0
            ratio = torch.where(z > 1e-8, torch.special.i1(z) / z.clamp(min=1e-8), torch.full_like(z, 0.5))
            w = ratio * self.beta ** 2 * x / (self.width / 2)
        else:
            w = torch.special.i0(z)
        return j.long() % self.nos[i], torch.where(ok, w, torch.zeros_like(w))

    def _chunks(self, coils):
        step = max(1, int(6e7 // (self.taps ** self.d * max(coils, 2))))
        for a in range(0, self.m, step):
            yield a, min(self.m, a + step)

    def _taps(self, a, b, deriv=-1):
        """(m, K^d) linear cells and weights of samples a..b; along axis
        ``deriv`` the derivative of the weight."""
        cell, w = None, None
        for i in range(self.d):
            c, v = self._axis(self.u[a:b, i], i, deriv == i)
            cell = c if cell is None else (cell[:, :, None] * self.nos[i] + c[:, None, :]).flatten(1)
            w = v if w is None else (w[:, :, None] * v[:, None, :]).flatten(1)
        return cell, w

    def interp(self, grid, deriv=-1):
        """grid (cells, C) -> samples (m, C), without the 1 / W^d."""
        out = torch.empty((self.m, grid.shape[1]), dtype=C128, device=grid.device)
        for a, b in self._chunks(grid.shape[1]):
            cell, w = self._taps(a, b, deriv)
            out[a:b] = (grid[cell] * w[..., None]).sum(1)
        return out

    def grid(self, y):
        """samples (m, C) -> grid (cells, C), without the 1 / W^d."""
        C = y.shape[1]
        out = torch.zeros((math.prod(self.nos), 2 * C), dtype=F64, device=y.device)
        yr = torch.view_as_real(y.contiguous()).reshape(self.m, 2 * C)
        for a, b in self._chunks(C):
            cell, w = self._taps(a, b)
            out.index_add_(0, cell.reshape(-1), (w[..., None] * yr[a:b, None, :]).reshape(-1, 2 * C))
        return torch.view_as_complex(out.reshape(-1, C, 2))

    def _apod(self, dev):
        a = torch.ones((), dtype=F64, device=dev)
        for n, k in zip(self.im, self.nos):
            x = (torch.arange(n, dtype=F64, device=dev) - n // 2) / k
            s = (self.beta ** 2 - (math.pi * self.width * x) ** 2).sqrt()
            a = a[..., None] * (s / torch.sinh(s))
        return a / math.sqrt(math.prod(self.im))

    def _place(self):
        return tuple(slice(k // 2 - n // 2, k // 2 - n // 2 + n) for n, k in zip(self.im, self.nos))

    def to_grid(self, img):
        """img (C, *im) -> centred spectrum (cells, C)."""
        C, dims = img.shape[0], tuple(range(1, self.d + 1))
        p = torch.zeros((C, *self.nos), dtype=C128, device=img.device)
        p[(slice(None), *self._place())] = img.to(C128) * self._apod(img.device)
        f = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(p, dim=dims), dim=dims), dim=dims)
        return f.reshape(C, -1).T.contiguous()

    def from_grid(self, grid):
        C, dims = grid.shape[1], tuple(range(1, self.d + 1))
        p = grid.T.reshape(C, *self.nos)
        f = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(p, dim=dims), dim=dims, norm="forward"), dim=dims)
        return f[(slice(None), *self._place())] * self._apod(grid.device)

    def forward(self, img):
        """(C, *im) -> (C, m)."""
        return (self.interp(self.to_grid(img)) / self.width ** self.d).T

    def adjoint(self, ksp):
        """(C, m) -> (C, *im)."""
        return self.from_grid(self.grid(ksp.to(C128).T) / self.width ** self.d)

    def normal(self, x, mps, dcf):
        m = mps.to(C128)
        y = self.forward(m * x.to(C128)) * dcf.reshape(-1).double()
        return (m.conj() * self.adjoint(y)).sum(0)


def _exact_batch(case, seed):
    xs = []
    for s in _inputs(case, seed):
        op = _Exact(s["im"], s["trj"], case["os"], case["width"])
        m = s["mps"].to(C128)
        b = (m.conj() * op.adjoint(s["ksp"].to(C128) * s["dcf"].double())).sum(0)
        x = b.clone()
        r = b - op.normal(x, m, s["dcf"]) - 1e-2 * x
        p = r.clone()
        rz = r.abs().square().sum()
        for _ in range(case["iters"]):
            ap = op.normal(p, m, s["dcf"]) + 1e-2 * p
            a = rz / (p.conj() * ap).real.sum()
            x, r = x + a * p, r - a * ap
            rr = r.abs().square().sum()
            p, rz = r + rr / rz * p, rr
        xs.append(x.reshape(-1))
    return torch.cat(xs)


def _exact_toeplitz(case, s):
    """crop IFFT K FFT pad with K the centred FFT of the doubled-size adjoint
    of the weights, all transforms orthonormal."""
    im, d = s["im"], len(s["im"])
    im2 = tuple(2 * n for n in im)
    dims = tuple(range(-d, 0))

    def cfft(x, f):
        return torch.fft.fftshift(f(torch.fft.ifftshift(x, dim=dims), dim=dims, norm="ortho"), dim=dims)

    big = _Exact(im2, (s["trj"] * 2.0), case["os"], case["width"])
    kern = cfft(big.adjoint(s["dcf"].reshape(1, -1))[0], torch.fft.fftn) * 2.0 ** d
    m = s["mps"].to(C128)
    place = (slice(None),) + tuple(slice((k - n) // 2, (k - n) // 2 + n) for n, k in zip(im, im2))
    p = torch.zeros((m.shape[0], *im2), dtype=C128, device=m.device)
    p[place] = m * s["img"].to(C128)
    y = cfft(cfft(p, torch.fft.fftn) * kern, torch.fft.ifftn)[place]
    return (m.conj() * y).sum(0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    s = _inputs(case, seed)
    im, trj = s["im"], s["trj"]
    if kind == "dcf":
        op = _Exact(im, trj, 1.0, 4.0, beta=8.0, raw=True)
        w = torch.ones((op.m, 1), dtype=C128, device=DEV)
        for _ in range(case["iters"]):
            w = w / op.interp(op.grid(w)).abs()
        w = w.real.reshape(trj.shape[:-1])
        return w / w.max()
    if kind == "toeplitz":
        return _exact_toeplitz(case, s)
    op = _Exact(im, trj, case["os"], case["width"])
    if kind == "sense":
        return op.normal(s["img"], s["mps"], s["dcf"])
    if kind == "segments":
        x = s["img"].to(C128)
        out = torch.zeros_like(x)
        hot = s["temporal"].reshape(case["nseg"], -1).real > 0
        flat, dcf = trj.reshape(-1, 2), s["dcf"].reshape(-1)
        for b, h in zip(s["spatial"].to(C128), hot):
            part = _Exact(im, flat[h], case["os"], case["width"])
            out += b.conj() * part.normal(b * x, s["mps"], dcf[h])
        return out
    shape = trj.shape[:-1]
    fwd = (lambda: op.forward(s["img"][0]).reshape(1, -1, *shape))
    adj = (lambda: op.adjoint(s["ksp"].reshape(case["coils"], -1))[None])
    if kind == "nufft":
        return fwd(), adj()
    if kind == "forward":
        return fwd()
    if kind == "adjoint":
        return adj()
    # grad: L = sum |A x - y|^2, dL/dx = 2 A^H r, dL/dk = 2 Re <r, (dA/dk) x>
    grid = op.to_grid(s["img"][0])
    wd = op.width ** op.d
    r = op.interp(grid) / wd - s["ksp"].reshape(case["coils"], -1).to(C128).T
    gt = torch.stack([2 * (r.conj() * op.interp(grid, i)).real.sum(1) / wd * (op.nos[i] / im[i]) for i in range(op.d)], 1)
    return r.abs().square().sum(), 2 * op.adjoint(r.T)[None], gt.reshape(1, *trj.shape)
