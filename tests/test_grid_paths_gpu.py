"""The two SO(3) grid kernels round alike.  Oversampling 2 runs the column kernel and 4 the general
one; at beta = 0 both sample the same function, the finer grid at every second alpha and gamma, and
with a power of two of points per axis the scale of the values is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L0,B", [(4, 3), (8, 40), (16, 2)])
def test_common_points_agree_bit_by_bit(cuda_device, L0, B):
    from matcha_b200.core.SOFFT import SOFFT
    from matcha_b200.core.wigner_index import dsize

    rng = np.random.default_rng(L0)
    n = dsize(L0 - 1)
    sig = torch.from_numpy((rng.standard_normal((B, n)) + 1j * rng.standard_normal((B, n))).astype(np.complex64))
    g2, g4 = (SOFFT(L=L0, device=cuda_device, batchsize=B, oversampling_factor=K)._run(
        sig.to(cuda_device), 1, True)[1][:, 0] for K in (2, 4))
    assert g2.abs().max() > 0
    assert torch.equal(g2, 4.0 * g4[:, ::2, ::2])
