"""The shift search's Fourier ball: content up to the ball's edge, in every box and operand layout."""
import numpy as np
import pytest
import torch

from oracle import shift as OS
from tests.test_shift_gpu import _matcher

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,precision", [(8, "fp32"), (16, "fp32"), (16, "bf16x3"), (32, "fp32"), (32, "bf16x3"),
                                         (48, "fp32"), (48, "bf16x3"), (64, "fp32"), (64, "bf16x3"), (80, "fp32"),
                                         (96, "bf16x3"), (128, "bf16x3")])
def test_white_content_matches_oracle(cuda_device, N, precision):
    """White volumes, so that the points at the ball's edge weigh as much as those inside.  The score
    is at most one and its error that of the operands: 3e-5 in FP32 and 1e-4 with bf16 pairs, as in
    the other comparisons with the oracle, here absolute since white volumes score below one."""
    rng = np.random.default_rng(N)
    B, uf, r = 2, 4, 1
    tmpl = rng.standard_normal((N, N, N)).astype(np.float32)
    vols = (np.repeat(tmpl[None], B, 0) + 0.3 * rng.standard_normal((B, N, N, N))).astype(np.float32)
    half = np.array([0.5, 2.0]) * 2.0 / N  # turns that move the ball's edge by about 0.5 and 2 points
    axis = np.array([[0.6, 0.0, 0.8], [0.0, -0.8, 0.6]])
    q = np.concatenate([np.cos(half)[:, None], np.sin(half)[:, None] * axis], 1)
    prior = rng.uniform(-0.4, 0.4, (B, 3)).astype(np.float32)
    sm = _matcher(N, B, uf, r, cuda_device, precision=precision)
    sm.set_reference(tmpl)
    _, score = sm.search_shifts(subtomos=torch.from_numpy(vols).to(cuda_device), ctfs=None,
                                shift_zyx=torch.from_numpy(prior).to(cuda_device), rotation_tracker=q)
    sm.status()
    assert sm.effective_precision == precision
    ref = OS.load_reference_full(tmpl, N, 1.0)
    ang = OS.euler_zyz_deg_from_quat_conj(q)
    want = [OS.estimate_shift_like_relion(ref, vols[b], prior[b], ang[b], uf, r)[1] for b in range(B)]
    np.testing.assert_allclose(score.cpu().numpy(), want, rtol=0, atol=3e-5 if precision == "fp32" else 1e-4)
