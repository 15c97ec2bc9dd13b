"""The grid in coil blocks: the native FFT passes over every kind of length
(two, three and four stages, all radices, odd image sizes) and coil counts
around the block widths, and the interpolation kernels that read it, against
64-bit transforms and the oracle."""
import math

import numpy as np
import pytest
import torch

from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _image_of(n):
    """An image length whose 1.25-oversampled grid has n points, or n itself (no oversampling)."""
    k = int(n / 1.25)
    return (k, 1.25) if math.ceil(1.25 * k) == n else (n, 1.0)


LENGTHS = [98, 112, 121, 143, 169, 187, 209, 247, 289, 304, 361, 374, 539, 616, 1001,  # 7, 11, 13, 17, 19
           97, 111, 163, 206, 254, 326, 401, 466, 509,  # chirp convolutions
           5, 6, 15, 16, 20, 27, 36, 50, 64, 81, 96, 100, 125, 144, 162, 200, 225, 240, 243, 250, 256, 288, 320, 375,
           400, 432, 500, 512, 600, 625, 640, 729, 768, 810, 960, 1000, 1024]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("last", [False, True])
def test_native_fft_lengths(n, last):
    from mr_recon_b200.plan import Plan
    k, os_ = _image_of(n)
    other = 8 if os_ > 1 else 10  # 10 grid points
    im = (other, k) if last else (k, other)
    C = 3
    rng = np.random.RandomState(n + last)
    # a second slice of another grid size: lengths without direct radices then run as chirp convolutions
    p = Plan([im, (20, 16)], [0, 0], [C, 1], os_, (4.0, 4.0), beta=9.0, device=DEV)
    assert p.fft_kind == 1
    nos = p.os_sizes[0]
    img = (rng.randn(C, *im) + 1j * rng.randn(C, *im)).astype(np.complex64)
    both = torch.zeros(p.n_img, dtype=torch.complex64, device=DEV)
    both[:img.size] = torch.from_numpy(img).reshape(-1).to(DEV)
    grid = torch.empty(p.n_grid, dtype=torch.complex64, device=DEV)
    back = torch.empty(p.n_img, dtype=torch.complex64, device=DEV)
    p.forward_ft(both, grid)
    src = (rng.randn(C, *nos) + 1j * rng.randn(C, *nos)).astype(np.complex64)
    gsrc = torch.zeros_like(grid)
    gsrc[:src.size] = torch.from_numpy(src).reshape(-1).to(DEV)
    p.adjoint_ift(gsrc, back)
    grid, back = grid[:src.size].reshape(src.shape), back[:img.size].reshape(img.shape)
    a = np.ones(())
    for m, o in zip(im, nos):
        t = np.sqrt(9.0 ** 2 - (np.pi * 4.0 * (np.arange(m) - m // 2) / o) ** 2 + 0j)
        a = a[..., None] * (t / np.sinh(t)).real
    a = a / math.sqrt(np.prod(im))
    at = tuple(slice(o // 2 - m // 2, o // 2 - m // 2 + m) for m, o in zip(im, nos))
    pad = np.zeros((C, *nos), np.complex128)
    pad[(slice(None), *at)] = img * a
    ax = (1, 2)
    want = np.fft.fftshift(np.fft.fftn(np.fft.ifftshift(pad, axes=ax), axes=ax), axes=ax)
    wback = np.fft.fftshift(np.fft.ifftn(np.fft.ifftshift(src.astype(np.complex128), axes=ax), axes=ax, norm="forward"),
                            axes=ax)[(slice(None), *at)] * a
    # float32 butterflies: a few ulp (6e-8) per stage, at most five stages an axis
    assert _rel(grid.cpu().numpy(), want) < 1e-6
    assert _rel(back.cpu().numpy(), wback) < 1e-6


CASES = [((40, 32), 1.25, 4, 1), ((40, 32), 1.25, 6, 2), ((48, 40), 1.25, 6, 3), ((40, 32), 2.0, 5, 7), ((40, 32), 1.25, 7, 8),
         ((48, 40), 1.25, 6, 9), ((40, 32), 1.25, 6, 17), ((40, 32), 1.5, 4, 33),
         ((16, 12, 20), 1.25, 4, 1), ((16, 12, 20), 1.25, 6, 2), ((12, 16, 8), 2.0, 5, 4), ((16, 12, 20), 1.25, 4, 8),
         ((12, 16, 20), 1.25, 6, 9), ((12, 8, 16), 1.25, 7, 19)]


@pytest.mark.parametrize("im,os_,W,C", CASES)
@pytest.mark.parametrize("M", [1, 33, 700])
def test_interpolation_from_coil_blocks(im, os_, W, C, M):
    """Forward over coil counts on both sides of a block, with samples on grid points, at exact kernel edges, at
    the grid's seam and outside it."""
    from mr_recon_b200.fourier import b200_nufft
    d = len(im)
    rng = np.random.RandomState(C * 1000 + M)
    trj = ((rng.rand(1, M, d) - 0.5) * np.array(im) * 1.2).astype(np.float32)
    trj[:, ::7] = np.round(trj[:, ::7])
    trj[:, 1::11] = -np.array(im) / 2.0
    img = (rng.randn(1, C, *im) + 1j * rng.randn(1, C, *im)).astype(np.complex64)
    nf = b200_nufft(im, oversamp=os_, width=W)
    on = O.KBNufftOracle(im, os_, W)
    t = torch.from_numpy(trj).to(DEV)
    # the tolerance of the repository's parity tests (float32 weights and sums)
    assert _rel(nf.forward(torch.from_numpy(img).to(DEV), t).cpu().numpy(), on.forward(img, trj)) < 1e-5


GRID_CASES = [((40, 32), 1.25, 4, 1), ((40, 32), 1.25, 6, 3), ((40, 32), 2.0, 5, 6), ((40, 32), 1.25, 7, 8),
              ((48, 40), 1.25, 6, 11), ((40, 32), 1.25, 6, 17), ((40, 32), 1.5, 4, 35),
              ((16, 12, 20), 1.25, 4, 1), ((16, 20, 12), 1.5, 6, 3), ((12, 16, 16), 2.0, 5, 7), ((16, 16, 16), 1.5, 7, 12),
              ((16, 12, 20), 1.25, 4, 19)]


@pytest.mark.parametrize("im,os_,W,C", GRID_CASES)
@pytest.mark.parametrize("chunk", [1, 40, 100000])
def test_register_tile_gridding(im, os_, W, C, chunk):
    """Gridding over coil counts on both sides of its lane groups, with a dense centre (split tiles, several
    trajectory parts and windows per batch of entries), grid points and exact kernel edges, and the seam; and the
    density-weighted normal operator, which passes rows, against the adjoint of the forward."""
    from mr_recon_b200 import _lib
    from mr_recon_b200.linops import sense_linop
    from mr_recon_b200.fourier import b200_nufft
    d, M = len(im), 500
    rng = np.random.RandomState(C * 100 + W)
    trj = ((rng.rand(M, d) - 0.5) * np.array(im) * 1.1).astype(np.float32)
    trj[::2] *= 0.15
    trj[::9] = np.round(trj[::9])
    ksp = (rng.randn(C, M) + 1j * rng.randn(C, M)).astype(np.complex64)
    nf = b200_nufft(im, oversamp=os_, width=W)
    on = O.KBNufftOracle(im, os_, W)
    t = torch.from_numpy(trj).to(DEV)
    mps = torch.from_numpy((rng.randn(C, *im) + 1j * rng.randn(C, *im)).astype(np.complex64)).to(DEV)
    dcf = torch.from_numpy((0.5 + rng.rand(M)).astype(np.float32)).to(DEV)
    A = sense_linop(t, mps, dcf=dcf, nufft=nf)
    A.plan.set_option(_lib.MRN_OPT_GRID_CHUNK, chunk)
    A.plan.set_traj(t.reshape(-1))
    assert (A.plan.stats()["split_tiles"] > 0) == (chunk < 500)
    g = torch.empty((C, *A.plan.os_sizes[0]), dtype=torch.complex64, device=DEV)
    A.plan.grid(torch.from_numpy(ksp).to(DEV), g, 1.0 / W ** d)
    # the tolerance of the repository's parity tests (float32 weights and sums)
    assert _rel(g.cpu().numpy(), on.adjoint_grid_only(ksp[None], trj[None])[0]) < 1e-5
    x = torch.from_numpy((rng.randn(*im) + 1j * rng.randn(*im)).astype(np.complex64)).to(DEV)
    assert torch.equal(A.normal(x), A.adjoint(A.forward(x)))


# (lengths of the grid, coils): lengths with factors 11 to 19, or a large prime, with columns enough for the widest CTAs (16
# direct, 8 as a chirp convolution), on each axis, in whole and ragged blocks of 8 coils
WIDE = [((209, 323), 9), ((323, 209), 32), ((539, 40), 9), ((40, 616), 8), ((361, 96), 32), ((96, 361), 9),
        ((206, 400), 9), ((100, 254), 32), ((254, 96), 33), ((401, 200), 9), ((180, 509), 17), ((509, 320), 32),
        ((206, 50, 40), 9), ((50, 206, 40), 9), ((40, 50, 206), 11), ((254, 254, 30), 8), ((121, 48, 60), 17),
        ((48, 121, 60), 9), ((48, 60, 121), 12)]


@pytest.mark.parametrize("nos,C", WIDE)
def test_wide_transforms(nos, C):
    """Transforms of many columns against 64 bits, and the coil-map source and sum against the plain ones."""
    from mr_recon_b200.plan import Plan
    d = len(nos)
    os_ = next(o for o in (1.25, 1.5, 1.375, 1.125, 1.0) if all(math.ceil(o * int(n / o)) == n for n in nos))
    im = tuple(int(n / os_) for n in nos)
    rng = np.random.RandomState(sum(nos) + C)
    M = 300
    p = Plan([im], [M], [C], os_, (4.0,) * d, beta=9.0, device=DEV)
    assert tuple(p.os_sizes[0]) == nos and p.fft_kind == 1
    cplx = lambda *s: (rng.randn(*s) + 1j * rng.randn(*s)).astype(np.complex64)  # noqa: E731
    dev = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    img, src = cplx(C, *im), cplx(C, *nos)
    grid = torch.empty(src.shape, dtype=torch.complex64, device=DEV)
    back = torch.empty(img.shape, dtype=torch.complex64, device=DEV)
    p.forward_ft(dev(img), grid)
    p.adjoint_ift(dev(src), back)
    a = np.ones(())
    for m, o in zip(im, nos):
        t = np.sqrt(9.0 ** 2 - (np.pi * 4.0 * (np.arange(m) - m // 2) / o) ** 2 + 0j)
        a = a[..., None] * (t / np.sinh(t)).real
    a = a / math.sqrt(np.prod(im))
    at = (slice(None),) + tuple(slice(o // 2 - m // 2, o // 2 - m // 2 + m) for m, o in zip(im, nos))
    pad = np.zeros(src.shape, np.complex128)
    pad[at] = img * a
    ax = tuple(range(1, d + 1))
    want = np.fft.fftshift(np.fft.fftn(np.fft.ifftshift(pad, axes=ax), axes=ax), axes=ax)
    wback = np.fft.fftshift(np.fft.ifftn(np.fft.ifftshift(src.astype(np.complex128), axes=ax), axes=ax, norm="forward"),
                            axes=ax)[at] * a
    # float32 butterflies: a few ulp (6e-8) per stage, at most five stages an axis
    assert _rel(grid.cpu().numpy(), want) < 1e-6
    assert _rel(back.cpu().numpy(), wback) < 1e-6
    p.set_traj(dev(((rng.rand(M, d) - 0.5) * np.array(im)).astype(np.float32).reshape(-1)))
    x, mps = dev(cplx(*im)), dev(cplx(C, *im))
    ks, kp = (torch.empty(C * M, dtype=torch.complex64, device=DEV) for _ in range(2))
    p.sense_forward(x, mps, ks)
    p.forward(mps * x, kp)
    xs = torch.empty_like(x)
    p.sense_adjoint(kp, None, mps, xs)
    p.adjoint(kp, back)
    # one rounding of the coil product (and of the sum of up to 33 coils) apart
    assert _rel(ks.cpu().numpy(), kp.cpu().numpy()) < 1e-6
    assert _rel(xs.cpu().numpy(), (mps.conj() * back).sum(0).cpu().numpy()) < 1e-6


@pytest.mark.parametrize("W", [4.5, 5.25, 6.5])
@pytest.mark.parametrize("im,C", [((48, 40), 1), ((48, 40), 4), ((64, 45), 9), ((12, 10), 3), ((24, 20, 28), 2), ((24, 20, 28), 9),
                                  ((13, 24, 24), 5)])
def test_widths_that_are_not_whole(im, C, W):
    """Half of the footprints of an axis have floor(W) taps there and half one more: forward, and adjoint with split
    tiles, with samples on grid points and at the seam, on grids with room for one more tap and without."""
    from mr_recon_b200.fourier import b200_nufft
    from mr_recon_b200 import _lib
    d, M = len(im), 900
    rng = np.random.RandomState(C + int(8 * W))
    trj = ((rng.rand(1, M, d) - 0.5) * np.array(im) * 1.2).astype(np.float32)
    trj[:, ::7] = np.round(trj[:, ::7])
    trj[:, 1::3] *= 0.2
    trj[:, 2::11] = -np.array(im) / 2.0
    img = (rng.randn(1, C, *im) + 1j * rng.randn(1, C, *im)).astype(np.complex64)
    ksp = (rng.randn(1, C, M) + 1j * rng.randn(1, C, M)).astype(np.complex64)
    nf = b200_nufft(im, oversamp=1.25, width=W)
    on = O.KBNufftOracle(im, 1.25, W)
    t = torch.from_numpy(trj).to(DEV)
    # the tolerance of the repository's parity tests (float32 weights and sums)
    assert _rel(nf.forward(torch.from_numpy(img).to(DEV), t).cpu().numpy(), on.forward(img, trj)) < 1e-5
    assert _rel(nf.adjoint(torch.from_numpy(ksp).to(DEV), t).cpu().numpy(), on.adjoint(ksp, trj)) < 1e-5
    from mr_recon_b200.plan import Plan
    p = Plan([im], [M], [C], 1.25, (W,) * d, device=DEV)
    p.set_option(_lib.MRN_OPT_GRID_CHUNK, 40)
    p.set_traj(t.reshape(-1))
    back = torch.empty(p.n_img, dtype=torch.complex64, device=DEV)
    p.adjoint(torch.from_numpy(ksp).to(DEV), back)
    assert _rel(back.cpu().numpy().reshape(img.shape), on.adjoint(ksp, trj)) < 1e-5


@pytest.mark.parametrize("im,os_,W,C", [((40, 32), 1.25, 6, 1), ((40, 32), 1.25, 4, 3), ((48, 40), 1.25, 4.5, 12), ((40, 32), 2.0, 7, 35),
                                        ((16, 12, 20), 1.25, 4, 1), ((16, 20, 12), 1.5, 6, 3), ((12, 16, 16), 2.0, 5, 12),
                                        ((16, 12, 20), 1.25, 4, 19)])
@pytest.mark.parametrize("chunk", [40, 100000])
def test_samples_that_are_not_finite_stay_in_their_footprints(im, os_, W, C, chunk):
    """Gridding with infinite and NaN samples of some coils: exactly the cells with weight of theirs are not finite,
    and the others are what they are with those samples zero."""
    from mr_recon_b200 import _lib
    from mr_recon_b200.plan import Plan
    d, M = len(im), 500
    rng = np.random.RandomState(C + int(W))
    trj = ((rng.rand(M, d) - 0.5) * np.array(im) * 1.1).astype(np.float32)
    trj[::2] *= 0.3
    trj[::9] = np.round(trj[::9])
    p = Plan([im], [M], [C], os_, (W,) * d, device=DEV)
    p.set_option(_lib.MRN_OPT_GRID_CHUNK, chunk)
    p.set_traj(torch.from_numpy(trj).to(DEV).reshape(-1))
    shape = (C, *p.os_sizes[0])

    def grid(k):
        g = torch.empty(shape, dtype=torch.complex64, device=DEV)
        p.grid(k, g, 0.5)
        return g

    ksp = torch.from_numpy((rng.randn(C, M) + 1j * rng.randn(C, M)).astype(np.complex64)).to(DEV)
    where = torch.zeros((C, M), dtype=torch.bool, device=DEV)
    for c, m, v in [(0, 3, complex("inf")), (C - 1, 9, complex("nan")), (C // 2, 18, complex(0, float("-inf")))]:
        ksp[c, m] = v
        where[c, m] = True
    got = grid(ksp)
    bad = ~(torch.isfinite(got.real) & torch.isfinite(got.imag))
    assert torch.equal(bad, grid(where.to(torch.complex64)) != 0)
    want = grid(torch.where(where, torch.zeros_like(ksp), ksp))
    got, want = got[~bad].cpu().numpy(), want[~bad].cpu().numpy()
    # the same terms in another order: a few ulp of float32 sums of up to a few hundred
    assert _rel(got, want) < 1e-6
