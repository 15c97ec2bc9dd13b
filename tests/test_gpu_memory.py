"""Plans with little device memory left: partly filled coil blocks and sample-major
rows are for speed, so a plan that fits without them is made without them."""
import numpy as np
import pytest
import torch

from mr_recon_b200.plan import Plan

pytestmark = pytest.mark.gpu
DEV = "cuda"
MB = 1 << 20


@pytest.fixture(autouse=True)
def _give_back():
    yield
    torch.cuda.empty_cache()


def _leave(nbytes):
    """A tensor that leaves about nbytes of the device free."""
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - nbytes, 1), dtype=torch.uint8, device=DEV)


def _inputs(im, C, M, seed):
    rng = np.random.RandomState(seed)
    trj = torch.from_numpy(((rng.rand(M, 3) - 0.5) * np.array(im)).astype(np.float32).reshape(-1)).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda n: torch.randn(n, dtype=torch.complex64, device=DEV, generator=g)  # noqa: E731
    return trj, rand(C * im[0] * im[1] * im[2]), rand(C * M)


def _both(plan, trj, img, ksp, k, b):
    plan.set_traj(trj)
    plan.forward(img, k)
    plan.adjoint(ksp, b)
    torch.cuda.synchronize()


def test_grid_without_partly_filled_blocks():
    """9 coils of a 120^3 grid take 124 MB, in whole blocks of 8 they take 221 MB: the same bits in less room."""
    im, C, M = (96, 96, 96), 9, 2000
    trj, img, ksp = _inputs(im, C, M, 0)
    out = [(torch.empty_like(ksp), torch.empty_like(img)) for _ in range(2)]
    plan = Plan([im], [M], [C], 1.25, (4.0,) * 3, device=DEV)
    _both(plan, trj, img, ksp, *out[0])
    del plan
    filler = _leave(190 * MB)
    plan = Plan([im], [M], [C], 1.25, (4.0,) * 3, device=DEV)
    assert plan.fft_kind == 1
    _both(plan, trj, img, ksp, *out[1])
    del filler
    torch.cuda.empty_cache()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_trajectory_takes_the_room_of_the_rows():
    """Rows of 2 M samples of 9 coils (256 MB) give way to the gridding entries (about 200 MB)."""
    im, C, M = (64, 64, 64), 9, 2000000
    trj, img, ksp = _inputs(im, C, M, 1)
    out = [(torch.empty_like(ksp), torch.empty_like(img)) for _ in range(2)]
    plan = Plan([im], [M], [C], 1.25, (4.0,) * 3, device=DEV)
    _both(plan, trj, img, ksp, *out[0])
    del plan
    plan = Plan([im], [M], [C], 1.25, (4.0,) * 3, device=DEV)
    filler = _leave(90 * MB)
    _both(plan, trj, img, ksp, *out[1])
    del filler
    torch.cuda.empty_cache()
    rel = lambda a, b: float(torch.linalg.norm(a - b) / torch.linalg.norm(b))  # noqa: E731
    assert torch.equal(out[0][0], out[1][0])
    assert rel(out[1][1], out[0][1]) < 1e-5  # other kernels: the tolerance of the repository's parity tests
