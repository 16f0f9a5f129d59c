"""The Newton march's two launch shapes (one or two candidates of a subtomogram per CTA, by the
number of CTAs): a subtomogram's result does not depend on the batch it is in, for degrees at the
edges of the 128-thread deal of the chains ((L + 1)^2 around 128 and 256) and the largest."""
import numpy as np
import pytest
import torch

from tests.helpers import synthetic_sigma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Li", [(5, [3]), (10, [4]), (11, [5]), (15, [7]), (16, [8])])
@pytest.mark.parametrize("C,steps", [(10, 1), (4, 3), (2, 0)])
def test_result_does_not_depend_on_the_batch(cuda_device, L, Li, C, steps):
    from matcha_b200.core.Matcha import Matcha

    big = 2 * 148 // C + 2
    sig, _ = synthetic_sigma(np.random.default_rng(L), big, L)
    sig = torch.from_numpy(sig).to(cuda_device)
    m = Matcha(batchsize=big, device=cuda_device, L_max=L,
               matcha_config=dict(Li=Li, candidates=C, num_steps=steps))
    whole = m.search_orientations(sig)
    for B in (1, 3, big - 3, big - 2):
        part = m.search_orientations(sig[:B])
        for x, y in zip(part, whole):
            assert torch.equal(x, y[:B]), B
