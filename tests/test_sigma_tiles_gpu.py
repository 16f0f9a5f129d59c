"""The sigma contraction's tiles of rows and columns, at every remainder of a degree's width."""
import numpy as np
import pytest
import torch

from oracle import fle as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L", [(12, 4), (16, 8), (32, 16)])
def test_every_degree_matches_oracle(cuda_device, N, L):
    """Widths 1, 3, 5, .. of the degrees against tiles of 4 x 3, one subtomogram and several.  FP32 sums
    of at most K = 32 products of the oracle's own coefficients rounded to FP32: 34 roundings of 6e-8
    each, relative to the sum of the products' magnitudes, itself at most the norms' product."""
    from matcha_b200 import _native as nat
    from matcha_b200.core.FLEBasis3D import FLEBasis3D

    fle = FLEBasis3D(N=N, bandlimit=L, eps=1e-4, batchsize=4, radius=int(N // 2 * 0.95), device=cuda_device,
                     dtype=torch.complex64)
    t = fle.tables
    rng = np.random.default_rng(N)
    ne = fle.ne
    c = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    av, at = c(4, ne), c(ne)
    ref = F.compute_sigma(t, at.astype(np.complex128), av.astype(np.complex128))
    for B in (1, 4):
        sig = torch.zeros((B, ref.shape[1]), dtype=torch.complex64, device=cuda_device)
        dv, dt = torch.from_numpy(av[:B]).to(cuda_device), torch.from_numpy(at).to(cuda_device)
        with torch.cuda.device(cuda_device):
            nat.check(fle._lib.mtb_sigma(fle._h, nat.ptr(dv), dv.stride(0), nat.ptr(dt), B, nat.ptr(sig),
                                         sig.stride(0), nat.stream_ptr(cuda_device)), "mtb_sigma")
        bound = 34 * 6e-8 * np.linalg.norm(at) * np.linalg.norm(av[:B], axis=1)[:, None]
        assert np.all(np.abs(sig.cpu().numpy() - ref[:B]) <= bound)
