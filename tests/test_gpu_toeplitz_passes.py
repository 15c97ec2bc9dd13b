"""The Toeplitz normal operator on the native FFT passes (2D and 3D padded
sizes with direct radices) against numpy's float64 FFTs: one to four stages in
the turning pass, radices with primes, odd sizes, partial coil blocks, several
padded sizes in one plan, and a size without direct radices (cuFFT).

Tolerance: two transforms of at most 2.8e-7 relative L2 each (the passes'
largest error against float64), the product and the coil sum: 1e-6."""

import numpy as np
import pytest
import torch

from mr_recon_b200.plan import Plan

pytestmark = pytest.mark.gpu
DEV = "cuda"


def cplx(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def exact(x, kern):
    d = kern.ndim
    ax = tuple(range(x.ndim - d, x.ndim))
    off = [(p - n) // 2 for p, n in zip(kern.shape, x.shape[-d:])]
    box = (Ellipsis,) + tuple(slice(o, o + n) for o, n in zip(off, x.shape[-d:]))
    y = np.zeros(x.shape[:x.ndim - d] + kern.shape, np.complex128)
    y[box] = x
    y = np.fft.fftshift(np.fft.fftn(np.fft.ifftshift(y, ax), axes=ax), ax) * kern
    return np.fft.fftshift(np.fft.ifftn(np.fft.ifftshift(y, ax), axes=ax), ax)[box]


CASES = [
    ([((2, 3), (4, 5))], [1]),
    ([((8, 30), (16, 60))], [3]),
    ([((15, 9), (25, 45))], [9]),
    ([((64, 50), (128, 100))], [8]),
    ([((256, 40), (512, 80))], [12]),
    ([((33, 200), (99, 400))], [5]),
    ([((66, 98), (132, 196))], [2]),
    ([((24, 24), (48, 48)), ((30, 20), (60, 40)), ((24, 24), (48, 48))], [4, 11, 1]),
    ([((48, 24), (98, 48)), ((16, 20), (32, 40))], [3, 6]),
    ([((46, 20), (92, 40))], [3]),
    ([((12, 10, 9), (24, 20, 27))], [5]),
    ([((50, 6, 8), (100, 12, 16))], [8]),
    ([((20, 18, 16), (20, 18, 16))], [2]),
]


@pytest.mark.parametrize("slices,coils", CASES)
def test_toeplitz_passes(slices, coils):
    rng = np.random.default_rng(len(slices) * 100 + coils[0])
    ims, pads = [s[0] for s in slices], [s[1] for s in slices]
    d = len(ims[0])
    plan = Plan(ims, [0] * len(ims), coils, 1.25, (4.0,) * d, device=DEV)
    kerns = [cplx(rng, p) for p in pads]
    imgs = [cplx(rng, (c, *im)) for c, im in zip(coils, ims)]
    x = [cplx(rng, im) for im in ims]
    flat = lambda a: torch.from_numpy(np.concatenate([v.reshape(-1) for v in a])).to(DEV)  # noqa: E731
    plan.set_toeplitz(flat(kerns), pads)
    out = torch.empty(plan.n_img, dtype=torch.complex64, device=DEV)
    plan.toeplitz_normal(flat(imgs), out)
    sense = torch.empty(sum(v.size for v in x), dtype=torch.complex64, device=DEV)
    plan.sense_normal_toeplitz(flat(x), flat(imgs), sense)
    out, sense = out.cpu().numpy(), sense.cpu().numpy()
    a = b = 0
    for k, i, v in zip(kerns, imgs, x):
        k64, i64 = k.astype(np.complex128), i.astype(np.complex128)
        ref = exact(i64, k64)
        sref = (np.conj(i64) * exact(i64 * v, k64)).sum(0)
        got, sgot = out[a:a + i.size].reshape(i.shape), sense[b:b + v.size].reshape(v.shape)
        a, b = a + i.size, b + v.size
        assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
        assert np.linalg.norm(sgot - sref) <= 1e-6 * np.linalg.norm(sref)


def test_kernels_set_again_follow_the_fft_option():
    """The same padded sizes after MRN_OPT_NATIVE_FFT changed: the bits of a plan that had the value from the start."""
    from mr_recon_b200 import _lib
    rng = np.random.default_rng(5)
    kern = torch.from_numpy(cplx(rng, (96, 80))).to(DEV)
    img = torch.from_numpy(cplx(rng, (3, 48, 40))).to(DEV)

    def normal(plan, native):
        plan.set_option(_lib.MRN_OPT_NATIVE_FFT, native)
        plan.set_toeplitz(kern, [(96, 80)])
        out = torch.empty_like(img)
        plan.toeplitz_normal(img, out)
        return out

    make = lambda: Plan([(48, 40)], [0], [3], 1.25, (4.0, 4.0), device=DEV)  # noqa: E731
    plan, fresh = make(), {n: normal(make(), n) for n in (0, 1)}
    assert not torch.equal(fresh[0], fresh[1])
    for native in (1, 0, 1):
        assert torch.equal(normal(plan, native), fresh[native])


@pytest.mark.parametrize("slices,coils", [
    ([((24, 24), (48, 48)), ((46, 20), (92, 40)), ((30, 20), (60, 40)), ((46, 20), (92, 40))], [4, 3, 11, 9]),
    ([((10, 12, 9), (20, 24, 23)), ((12, 10, 9), (24, 20, 27))], [5, 2]),
])
def test_normal_does_not_depend_on_the_other_slices(slices, coils):
    """Padded sizes without direct radices (92, 23) beside others: each slice's normal, and its CG sum, has the bits
    that it has in a plan of its own."""
    rng = np.random.default_rng(len(slices))
    ims, pads = [s[0] for s in slices], [s[1] for s in slices]
    d = len(ims[0])
    kerns = [cplx(rng, p) for p in pads]
    imgs = [cplx(rng, (c, *im)) for c, im in zip(coils, ims)]
    xs = [cplx(rng, im) for im in ims]
    flat = lambda a: torch.from_numpy(np.concatenate([v.reshape(-1) for v in a])).to(DEV)  # noqa: E731

    def run(sel):
        pick = lambda a: [a[s] for s in sel]  # noqa: E731
        plan = Plan(pick(ims), [0] * len(sel), pick(coils), 1.25, (4.0,) * d, device=DEV)
        plan.set_toeplitz(flat(pick(kerns)), pick(pads))
        img, x = flat(pick(imgs)), flat(pick(xs))
        out, sense = torch.empty_like(img), torch.empty_like(x)
        pap = torch.zeros(len(sel), dtype=torch.float64, device=DEV)
        plan.toeplitz_normal(img, out)
        plan.sense_normal_toeplitz(x, img, sense, 1.0, 0.5, pap)
        return out, sense, pap

    out, sense, pap = run(range(len(slices)))
    a = b = 0
    for s in range(len(slices)):
        o1, s1, p1 = run([s])
        assert torch.equal(out[a:a + o1.numel()], o1) and torch.equal(sense[b:b + s1.numel()], s1)
        assert pap[s] == p1[0]
        a, b = a + o1.numel(), b + s1.numel()
