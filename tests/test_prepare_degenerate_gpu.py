"""Preparation of a subtomogram without deviation in its mask: not a number up to two voxels past the
mask, as 0 / 0, and zero beyond, beside ordinary subtomograms of the same batch."""
import numpy as np
import pytest

from tests.helpers import haar_quaternions
from tests.test_prepare import _prepare_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,radius,B", [(16, 5.0, 2), (33, 10.5, 2), (64, 20.0, 2), (64, 20.0, 80), (240, 30.0, 2)])
def test_constant_volume(cuda_device, N, radius, B):
    rng = np.random.default_rng(N)
    vols = rng.standard_normal((2, N, N, N)).astype(np.float32)
    vols[1] = 0.0
    got = _prepare_gpu(vols[np.arange(B) % 2], np.zeros((B, 3), np.float32), haar_quaternions(rng, B), radius,
                       cuda_device)
    g = np.arange(N) - N // 2
    near = (g[:, None, None] ** 2 + g[:, None] ** 2 + g ** 2) < (radius + 2.0) ** 2
    assert np.isfinite(got[0]).all()
    for b in {1, B - 1}:
        np.testing.assert_array_equal(np.isnan(got[b]), near)
        assert not got[b][~near].any()
