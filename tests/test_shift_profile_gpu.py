"""The stages of the shift search's profile hold the launches that they are named after."""
import numpy as np
import pytest
import torch

from tests.test_shift_gpu import _matcher

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,uf,r", [(64, 8, 5), (48, 8, 3)])
def test_stages_hold_their_launches(cuda_device, N, uf, r):
    """Each kernel's own events lie between its stage's, so a stage lasts as long as its kernels at
    least (less 2 us a call for the events' resolution).  64: fused passes, the Nyquist plane's second
    pass a launch of its own; 48: unfused, all of it in the planes' launches."""
    from matcha_b200 import _native as nat

    B, calls = 64, 5
    rng = np.random.default_rng(N)
    sm = _matcher(N, B, uf, r, cuda_device, precision="bf16x3")
    sm.set_reference(rng.standard_normal((N, N, N)).astype(np.float32))
    args = dict(subtomos=torch.from_numpy(rng.standard_normal((B, N, N, N)).astype(np.float32)).to(cuda_device),
                ctfs=None, shift_zyx=torch.zeros((B, 3), device=cuda_device),
                rotation_tracker=np.tile([1.0, 0, 0, 0], (B, 1)))
    sm.search_shifts(**args)
    sm.profile(calls)
    nat.profile_start(calls * 16)
    for _ in range(calls):
        sm.search_shifts(**args)
    nat.profile_stop()
    kernels = {k: v["ms"] for k, v in nat.profile_read()[0].items()}
    ms, n = sm.profile_read()
    sm.profile(0)
    assert n == calls
    slack = 0.002 * calls
    nyquist = kernels.pop("updft1_tc_kernel (Nyquist plane, pass 2)", None)
    assert (nyquist is None) == (N == 48)
    if nyquist is not None:
        assert ms["nyquist"] >= nyquist - slack > 0
    assert ms["updft_pass1"] >= kernels["updft1_tc_kernel"] - slack
    assert ms["updft_pass23"] >= sum(v for k, v in kernels.items() if k.startswith("updft")
                                     and k != "updft1_tc_kernel") - slack
