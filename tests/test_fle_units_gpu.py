"""The work units of the tensor-core ball expansion: tiles cut along K into parts (a batch of one,
a batch block and one row, two batch blocks), both orders of the hi/lo products (a basis of
less than 1 GB and one of more), and the coefficients' independence of the batch where the
parts' sums are added chunk by chunk.

Tolerance 1e-4 of the result's norm, as for the hi+lo split elsewhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fle(dev, N, L, cap, precision):
    from matcha_b200.core.FLEBasis3D import FLEBasis3D

    return FLEBasis3D(N=N, bandlimit=L, eps=1e-4, batchsize=cap, radius=int(N // 2 * 0.95), device=dev,
                      dtype=torch.complex64, precision=precision)


@pytest.mark.parametrize("N,L,batches", [(16, 8, (1, 40)), (32, 16, (1, 127, 128, 129, 300)), (47, 20, (3, 130)),
                                         (48, 24, (1, 129)), (64, 32, (1, 128, 129, 257, 520)), (80, 40, (1, 128, 150))])
def test_units_match_fp32(cuda_device, N, L, batches):
    cap = max(batches)
    tc, fp = _fle(cuda_device, N, L, cap, "bf16x3"), _fle(cuda_device, N, L, cap, "fp32")
    g = torch.Generator(device=cuda_device).manual_seed(N)
    v = torch.randn((cap, N, N, N), generator=g, device=cuda_device) + 0.5
    ref, nref = fp._forward(v, True)
    whole, _ = tc._forward(v, True)
    for B in batches:
        a, n = tc._forward(v[:B], True)
        tc.status()
        for b in {0, B // 2, B - 1}:
            assert torch.linalg.norm(a[b] - ref[b]) < 1e-4 * torch.linalg.norm(ref[b]), (B, b)
        torch.testing.assert_close(n, nref[:B], rtol=1e-4, atol=0)
        if N <= 64:
            assert torch.equal(a, whole[:B])
