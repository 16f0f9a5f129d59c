"""A subtomogram's results do not depend on the batch that it is sent in: every sum whose split over
CTAs follows the batch adds the same groups in the same order.  Compared bit by bit, but for the
preparation, whose statistics meet by FP64 atomics in no order."""
import numpy as np
import pytest
import torch

from tests.helpers import haar_quaternions, synthetic_sigma
from tests.test_prepare import _prepare_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,batches", [(16, 8, (1, 75, 149)), (48, 24, (1, 130, 300)), (64, 32, (1, 129, 300)),
                                         (80, 40, (1, 128, 150, 300))])
def test_coefficients(cuda_device, N, L, batches):
    """80^3 lies past the size from which hi and lo tiles share a stage; batches of one, two and three
    blocks of 128, whose tiles are cut differently."""
    from matcha_b200.core.FLEBasis3D import FLEBasis3D

    cap = max(batches) + 300
    fle = FLEBasis3D(N=N, bandlimit=L, eps=1e-4, batchsize=cap, radius=N // 2 - 1, device=cuda_device,
                     dtype=torch.complex64, precision="bf16x3")
    g = torch.Generator(device=cuda_device).manual_seed(N)
    v = torch.randn((cap, N, N, N), generator=g, device=cuda_device) + 0.5
    whole = fle._forward(v, False)[0].clone()
    for B in batches:
        assert torch.equal(fle._forward(v[:B], False)[0], whole[:B]), B
    fle.status()


@pytest.mark.parametrize("N,L", [(16, 8), (48, 24), (64, 32)])
def test_norms(cuda_device, N, L):
    """Batches of every cluster size of the coefficients' sums of squares, eight CTAs to one."""
    from matcha_b200.core.FLEBasis3D import FLEBasis3D

    fle = FLEBasis3D(N=N, bandlimit=L, eps=1e-4, batchsize=1200, radius=N // 2 - 1, device=cuda_device,
                     dtype=torch.complex64, precision="bf16x3")
    g = torch.Generator(device=cuda_device).manual_seed(N)
    v = (torch.randn((100, N, N, N), generator=g, device=cuda_device) + 0.5).repeat(12, 1, 1, 1)
    whole = fle._forward(v, True)[1].clone()
    for B in (1, 149, 297, 593):
        assert torch.equal(fle._forward(v[:B], True)[1], whole[:B]), B
    fle.status()


@pytest.mark.parametrize("L,Li,C,steps", [(32, [8, 16, 24], 10, 1), (64, [16, 32, 48], 4, 1), (24, [8, 16], 2, 3)])
def test_marches_of_several_stages(cuda_device, L, Li, C, steps):
    """One and two candidates of a subtomogram per CTA, by the number of CTAs."""
    from matcha_b200.core.Matcha import Matcha

    big = 2 * 148 // C + 2
    sig, _ = synthetic_sigma(np.random.default_rng(L), 4, L)
    sig = torch.from_numpy(sig).to(cuda_device)[torch.arange(big) % 4]
    sig = sig * (1 + torch.arange(big, device=cuda_device)[:, None] / big)
    m = Matcha(batchsize=big, device=cuda_device, L_max=L, matcha_config=dict(Li=Li, candidates=C, num_steps=steps))
    g = torch.Generator(device=cuda_device).manual_seed(L)
    start = torch.rand((3, big, C), generator=g, device=cuda_device) * 3
    whole = m.march(*start, sig)
    for B in (1, 5, big - 3):
        for x, y in zip(m.march(*start[:, :B], sig[:B]), whole):
            assert torch.equal(x, y[:B]), B


@pytest.mark.parametrize("N,radius", [(16, 7.0), (64, 30.0), (90, 40.0)])
def test_preparation(cuda_device, N, radius):
    """Batches of CTAs of one plane and of two: the statistics are FP64 sums of the same FP32 sums (in
    any order), so mean and deviation agree but for a rounding to FP32, and the values to 3e-7 of
    the largest.  The mean far above the deviation makes any other change of the sums show."""
    B = -(-1184 // ((N + 3) // 4))
    rng = np.random.default_rng(N)
    base = (rng.standard_normal((3, N, N, N)) + 200.0).astype(np.float32)
    vols = base[np.arange(B) % 3]
    shifts = rng.uniform(-2, 2, (3, 3)).astype(np.float32)[np.arange(B) % 3]
    q = haar_quaternions(rng, 3)[np.arange(B) % 3]
    got = _prepare_gpu(vols, shifts, q, radius, cuda_device)
    for b in range(3):
        one = _prepare_gpu(vols[b:b + 1], shifts[b:b + 1], q[b:b + 1], radius, cuda_device)
        np.testing.assert_allclose(got[b:b + 1], one, rtol=0, atol=3e-7 * np.abs(one).max())
