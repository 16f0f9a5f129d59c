"""The oversampling-2 grid kernel at its edges: the smallest and largest L0, grids whose columns
straddle warps (n = 12, 20, 44, 60), beta values that do not fill a pass, batches around the
cluster sizes' changes, 1 to 32 kept points, ties and values that are not numbers.

The grid is compared with the oracle's (FP32 sums of at most a few thousand terms: 2e-5 of the
maximum, the tolerance of the other grid tests); the kept points, exactly, with a sort of the
kernel's own grid by (value, then smaller index)."""
import numpy as np
import pytest
import torch

from oracle import matcha as OM
from oracle import wigner as OW

pytestmark = pytest.mark.gpu


def _run(dev, sig, L0, C):
    from matcha_b200.core.SOFFT import SOFFT

    a, g = SOFFT(L=L0, device=dev, batchsize=sig.shape[0], oversampling_factor=2)._run(
        torch.from_numpy(sig).to(dev), C, True)
    return a.cpu().numpy(), g.cpu().numpy()


def _kept(grid, C):
    n = grid.shape[1]
    out = np.empty((3, grid.shape[0], C), dtype=np.float32)
    for b in range(grid.shape[0]):
        flat = grid[b].ravel()
        idx = np.lexsort((np.arange(flat.size), -flat))[:C]
        out[1, b] = (idx // (n * n)).astype(np.float32) * np.float32(np.pi / (n - 1))
        out[0, b] = ((idx // n) % n).astype(np.float32) * np.float32(2 * np.pi / n)
        out[2, b] = (idx % n).astype(np.float32) * np.float32(2 * np.pi / n)
    return out


@pytest.mark.parametrize("L0,B,C", [(3, 1, 1), (3, 200, 32), (4, 5, 10), (5, 149, 7), (7, 3, 10), (8, 16, 10),
                                    (8, 700, 10), (11, 2, 17), (12, 75, 10), (13, 1, 32), (15, 2, 10), (16, 3, 10)])
def test_grid_and_kept_points(cuda_device, L0, B, C):
    rng = np.random.default_rng(L0 * 1000 + B)
    n = OW.dsize(L0 - 1)
    sig = (rng.standard_normal((B, n)) + 1j * rng.standard_normal((B, n))).astype(np.complex64)
    a, g = _run(cuda_device, np.concatenate([sig, np.full((B, 5), np.nan, np.complex64)], 1), L0, C)
    for b in {0, B - 1}:
        ref = OM.sofft_eval(sig[b:b + 1].astype(np.complex128), L0, 2)[0]
        np.testing.assert_allclose(g[b], ref, rtol=0, atol=2e-5 * np.abs(ref).max())
    np.testing.assert_array_equal(a, _kept(g, C))


def test_ties_and_not_a_number(cuda_device):
    n = OW.dsize(7)
    sig = np.zeros((4, n), dtype=np.complex64)
    sig[1, 0] = 1.0       # one constant grid
    sig[2, 0] = -1.0
    sig[3] = np.nan
    a, g = _run(cuda_device, sig, 8, 10)
    assert np.isnan(g[3]).all()
    np.testing.assert_array_equal(a[:, :3], _kept(g[:3], 10))
    # no comparable value: still angles of the grid
    assert np.isfinite(a[:, 3]).all() and a[1, 3].max() <= np.float32(np.pi)
