"""The FP32 product of the shift match outside its Fourier ball: zero, whatever the shared memory of
columns that are not transformed holds."""
import numpy as np
import pytest
import torch

from tests.test_shift_gpu import _matcher

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 16, 32, 48, 64, 80, 96, 128])
def test_results_survive_other_data_on_the_chip(cuda_device, N):
    """The continuous score reads every point of the product, so a not-a-number outside the ball
    would show.  Between two calls a search of volumes that hold infinities leaves such values in
    every SM's shared memory; the second call repeats the first (the norms' atomic sums differ by
    FP32 rounding, 1e-6 of a score of order one)."""
    rng = np.random.default_rng(N)
    B = 3
    vols = torch.from_numpy(rng.standard_normal((B, N, N, N)).astype(np.float32)).to(cuda_device)
    sm = _matcher(N, max(B, 148 * 8 // N + 1), 2, 1, cuda_device, precision="fp32")
    sm.set_reference(rng.standard_normal((N, N, N)).astype(np.float32))
    z = torch.from_numpy(rng.uniform(-0.5, 0.5, (B, 3)).astype(np.float32)).to(cuda_device)
    rot = torch.eye(3, device=cuda_device).reshape(1, 9).repeat(B, 1)
    first = [t.clone() for t in sm.score_and_gradient(vols, z, rot, z)]
    bad = torch.full((148 * 8 // N + 1, N, N, N), float("inf"), device=cuda_device)
    sm.score_and_gradient(bad, bad.new_zeros((bad.shape[0], 3)), rot[:1].repeat(bad.shape[0], 1),
                          bad.new_zeros((bad.shape[0], 3)))
    again = sm.score_and_gradient(vols, z, rot, z)
    for a, b in zip(again, first):
        assert torch.isfinite(b).all()
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)
