"""Preparation of large batches: planes and bricks shared differently than in small ones."""
import numpy as np
import pytest

from oracle import prepare as OP
from tests.helpers import haar_quaternions
from tests.test_prepare import _prepare_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,radius", [(9, 5.0), (15, 7.9), (16, 8.0), (30, 17.0), (63, 32.0), (66, 31.0), (130, 60.0)])
def test_large_batches_match_small_ones_and_the_oracle(cuda_device, N, radius):
    """Boxes around the 63-column steps and odd ones whose mask reaches the first voxel of a row.  The
    same volume and shift under many rotations, axis-aligned ones among them, in a batch that is
    large enough for CTAs of several planes, against batches of one: the two differ by the order of
    the statistics' FP32 partial sums of at most 2 N terms, 6e-8 each of an O(1) value."""
    B = -(-1184 // ((N + 3) // 4))
    rng = np.random.default_rng(N)
    base = (rng.standard_normal((4, N, N, N)) + 1.0).astype(np.float32)
    vols = base[np.arange(B) % 4]
    shifts = np.array([[0.3, -1.7, 2.2], [0, 0, 0], [-0.5, 0.25, 0.75], [1, -1, 0]], dtype=np.float32)[np.arange(B) % 4]
    q = haar_quaternions(rng, B)
    h = np.sqrt(0.5)
    q[:4] = [[h, h, 0, 0], [h, 0, h, 0], [h, 0, 0, h], [1, 0, 0, 0]]
    got = _prepare_gpu(vols, shifts, q, radius, cuda_device)
    for b in (0, 1, 2, 3, 5, B - 1):
        one = _prepare_gpu(vols[b:b + 1], shifts[b:b + 1], q[b:b + 1], radius, cuda_device)
        np.testing.assert_allclose(got[b:b + 1], one, rtol=0, atol=2 * N * 6e-8 * max(1.0, np.abs(one).max()))
    if N <= 66:
        picks = [0, 3, 5, B - 1]
        ref = OP.prepare(vols[picks], shifts[picks], q[picks], radius)
        np.testing.assert_allclose(got[picks], ref, atol=2e-4)  # as in the comparison of small batches


def test_box_past_the_staged_planes_matches_oracle(cuda_device):
    """A plane of 236^2 and up does not fit in shared memory: voxel by voxel from global memory."""
    N = 238
    rng = np.random.default_rng(N)
    vols = (rng.standard_normal((1, N, N, N)) + 1.0).astype(np.float32)
    shifts = np.array([[0.4, -1.6, 2.3]], dtype=np.float32)
    q = haar_quaternions(rng, 1)
    got = _prepare_gpu(vols, shifts, q, 40.0, cuda_device)
    # coordinates of up to 238 carry four times the rounding of those in the comparisons above
    np.testing.assert_allclose(got, OP.prepare(vols, shifts, q, 40.0), atol=8e-4)
