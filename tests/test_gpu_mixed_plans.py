"""Plans whose slices differ in ways that the kernels' choices depend on: grids
of any number of points before one that is read 16 bytes at a time, slices
without samples, and slices that take different kernels from their neighbours."""
import numpy as np
import pytest
import torch

from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-5  # the repository's parity tests (float32 weights and sums)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _cplx(rng, shape):
    return (rng.randn(*shape) + 1j * rng.randn(*shape)).astype(np.complex64)


def _check(plan, ims, ms, coils, os_, W, rng):
    """Forward and adjoint of every slice against the oracle."""
    d = len(ims[0])
    trjs = [((rng.rand(m, d) - 0.5) * np.array(im)).astype(np.float32) for im, m in zip(ims, ms)]
    imgs = [_cplx(rng, (c, *im)) for im, c in zip(ims, coils)]
    flat = lambda a: torch.from_numpy(np.concatenate([v.reshape(-1) for v in a])).to(DEV)  # noqa: E731
    plan.set_traj(flat(trjs))
    ksp = torch.empty(plan.n_ksp, dtype=torch.complex64, device=DEV)
    back = torch.empty(plan.n_img, dtype=torch.complex64, device=DEV)
    plan.forward(flat(imgs), ksp)
    plan.adjoint(ksp, back)
    ksp, back = ksp.cpu().numpy(), back.cpu().numpy()
    for s, (im, m, c) in enumerate(zip(ims, ms, coils)):
        bo = back[plan.img_off[s]:][:c * int(np.prod(im))].reshape(c, *im)
        if m == 0:
            assert not bo.any()
            continue
        on = O.KBNufftOracle(im, os_, W)
        ko = ksp[plan.ksp_off[s]:][:c * m].reshape(c, m)
        assert _rel(ko, on.forward(imgs[s][None], trjs[s][None])[0]) < TOL, f"forward, slice {s}"
        assert _rel(bo, on.adjoint(ko[None], trjs[s][None])[0]) < TOL, f"adjoint, slice {s}"


@pytest.mark.parametrize("ims,ms,coils", [
    ([(36, 36), (64, 64)], [0, 500], [1, 8]),              # 45 x 45 points before the grid of 8 coils
    ([(36, 36), (36, 36), (20, 20)], [0, 300, 200], [1, 16, 9]),  # the same grid size
    ([(36, 36), (12, 12), (64, 60)], [0, 0, 400], [1, 2, 11]),
])
def test_grids_start_on_whole_sectors(ims, ms, coils):
    """A slice without samples whose grid has an odd number of points, before slices whose coil blocks are copied
    16 bytes at a time."""
    from mr_recon_b200 import _lib
    from mr_recon_b200.plan import Plan
    for native in (1, 0):
        plan = Plan(ims, ms, coils, 1.25, (6.0, 6.0), device=DEV)
        plan.set_option(_lib.MRN_OPT_NATIVE_FFT, native)
        _check(plan, ims, ms, coils, 1.25, 6.0, np.random.RandomState(len(ims) + ms[0]))
