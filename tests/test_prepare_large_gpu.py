"""Preparation of boxes whose planes are not staged: 31 columns of a warp at a time, odd boxes, masks up
to and past the faces."""
import numpy as np
import pytest

from oracle import prepare as OP
from tests.helpers import haar_quaternions
from tests.test_prepare import _prepare_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,radius", [(236, 118.0), (237, 118.5), (249, 140.0)])
def test_large_boxes_match_oracle(cuda_device, N, radius):
    """236: the last step holds 19 columns; 237: the mask reaches the first voxel of a row; 249 = 8 x 31 + 1,
    its mask past the faces.  Tolerance: 2e-4 for coordinates of a box of 64, which lose two bits here."""
    rng = np.random.default_rng(N)
    vols = (rng.standard_normal((1, N, N, N)) + 1.0).astype(np.float32)
    shifts = np.array([[-0.4, 1.6, 0.25]], dtype=np.float32)
    q = haar_quaternions(rng, 1)
    got = _prepare_gpu(vols, shifts, q, radius, cuda_device)
    np.testing.assert_allclose(got, OP.prepare(vols, shifts, q, radius), atol=8e-4)
