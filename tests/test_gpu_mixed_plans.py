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


@pytest.mark.parametrize("ims,coils", [
    ([(203, 203), (163, 150), (64, 64), (181, 217), (331, 150), (203, 203)], [4, 8, 1, 7, 3, 32]),
    ([(82, 20, 24), (48, 48, 48), (82, 96, 80)], [3, 5, 8]),
])
def test_transforms_do_not_depend_on_the_other_slices(ims, coils):
    """Grids with large prime factors (254 = 2 x 127, 326 = 2 x 163, 103) beside others, the same size with few and
    with many coils: each slice's transforms have the bits that they have in a plan of their own."""
    from mr_recon_b200.plan import Plan
    rng = np.random.RandomState(len(ims))
    d = len(ims[0])

    def transforms(ims, coils, img, src):
        p = Plan(ims, [0] * len(ims), coils, 1.25, (4.0,) * d, device=DEV)
        grid, back = torch.empty_like(src), torch.empty_like(img)
        p.forward_ft(img, grid)
        p.adjoint_ift(src, back)
        return p, grid, back

    n_img = [c * int(np.prod(im)) for im, c in zip(ims, coils)]
    n_grid = [c * int(np.prod([-(-5 * n // 4) for n in im])) for im, c in zip(ims, coils)]
    img = torch.from_numpy(_cplx(rng, (sum(n_img),))).to(DEV)
    src = torch.from_numpy(_cplx(rng, (sum(n_grid),))).to(DEV)
    both, grid, back = transforms(ims, coils, img, src)
    for s in range(len(ims)):
        i = slice(int(both.img_off[s]), int(both.img_off[s]) + n_img[s])
        g = slice(int(both.grid_off[s]), int(both.grid_off[s]) + n_grid[s])
        _, one_grid, one_back = transforms([ims[s]], [coils[s]], img[i].contiguous(), src[g].contiguous())
        assert torch.equal(grid[g], one_grid), f"forward, slice {s}"
        assert torch.equal(back[i], one_back), f"inverse, slice {s}"


@pytest.mark.parametrize("ims,ms,coils,W", [
    ([(48, 48), (203, 203), (64, 64), (160, 150), (56, 56)], [1600, 9000, 4800, 100000, 2000], [3, 4, 12, 20, 1], 6.0),
    ([(48, 48), (64, 60), (90, 80)], [1600, 4800, 60000], [8, 8, 8], 4.5),
    ([(24, 24, 24), (32, 28, 30), (24, 20, 16)], [6000, 500000, 3000], [2, 8, 5], 4.0),
])
def test_samples_and_grids_do_not_depend_on_the_other_slices(ims, ms, coils, W):
    """Forward and adjoint of slices of very different sample counts, with a dense centre (split gridding tiles): the
    bits of each slice in a plan of its own, at the default work-item sizes."""
    from mr_recon_b200 import _lib
    from mr_recon_b200.plan import Plan
    rng = np.random.RandomState(len(ims) + coils[0])
    d = len(ims[0])
    trjs = []
    for im, m in zip(ims, ms):
        t = (rng.rand(m, d) - 0.5) * np.array(im)
        t[::2] *= 0.3
        trjs.append(t.astype(np.float32))
    flat = lambda a: torch.from_numpy(np.concatenate([v.reshape(-1) for v in a])).to(DEV)  # noqa: E731

    def run(ims, ms, coils, trj, img, ksp):
        p = Plan(ims, ms, coils, 1.25, (W,) * d, device=DEV)
        if d == 2:
            p.set_option(_lib.MRN_OPT_GRID_LANES, 32)
        p.set_traj(trj)
        k, b = torch.empty_like(ksp), torch.empty_like(img)
        p.forward(img, k)
        p.adjoint(ksp, b)
        return p, k, b

    img = flat([_cplx(rng, (c, *im)) for im, c in zip(ims, coils)])
    ksp = flat([_cplx(rng, (c, m)) for m, c in zip(ms, coils)])
    both, k, b = run(ims, ms, coils, flat(trjs), img, ksp)
    assert both.stats()["split_tiles"] > 0
    for s in range(len(ims)):
        i = slice(int(both.img_off[s]), int(both.img_off[s]) + coils[s] * int(np.prod(ims[s])))
        q = slice(int(both.ksp_off[s]), int(both.ksp_off[s]) + coils[s] * ms[s])
        _, k1, b1 = run([ims[s]], [ms[s]], [coils[s]], flat([trjs[s]]), img[i].contiguous(), ksp[q].contiguous())
        assert torch.equal(k[q], k1), f"forward, slice {s}"
        assert torch.equal(b[i], b1), f"adjoint, slice {s}"


def test_cg_sums_do_not_depend_on_the_other_slices():
    """Re<x, A x> of rows of 40, 100 and 200 pixels in one plan and alone: the same float64 bits."""
    from mr_recon_b200 import _lib
    from mr_recon_b200.plan import Plan
    rng = np.random.RandomState(3)
    ims, coils, m = [(30, 40), (20, 100), (24, 200)], [2, 3, 8], 400
    xs = [(_cplx(rng, im) * np.exp(rng.uniform(-9, 9, im))).astype(np.complex64) for im in ims]  # sums that round
    mps = [_cplx(rng, (c, *im)) for c, im in zip(coils, ims)]
    trjs = [((rng.rand(m, 2) - 0.5) * np.array(im)).astype(np.float32) for im in ims]
    flat = lambda a: torch.from_numpy(np.concatenate([v.reshape(-1) for v in a])).to(DEV)  # noqa: E731

    def sums(sel):
        pick = lambda a: [a[s] for s in sel]  # noqa: E731
        p = Plan(pick(ims), [m] * len(sel), pick(coils), 1.25, (6.0, 6.0), device=DEV)
        p.set_option(_lib.MRN_OPT_GRID_LANES, 8)
        p.set_traj(flat(pick(trjs)))
        x = flat(pick(xs))
        out, pap = torch.empty_like(x), torch.zeros(len(sel), dtype=torch.float64, device=DEV)
        p.sense_normal(x, flat(pick(mps)), None, out, 1.0, 0.1, pap)
        return out, pap

    out, pap = sums([0, 1, 2])
    at = 0
    for s in range(3):
        o1, p1 = sums([s])
        assert torch.equal(out[at:at + o1.numel()], o1) and pap[s] == p1[0]
        at += o1.numel()
