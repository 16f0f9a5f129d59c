"""Handles of different sizes used by two threads at once, each on its own stream: the kernels they
share are launched with different amounts of shared memory, and no launch may be refused because
the other thread asked for less just before it.  The threads call the library itself, thousands of
times, since the window between a call's setting and its launch is about a microsecond."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expansion(N, dev):
    from matcha_b200 import _native as nat
    from matcha_b200.core.CrossCorrelationMatcher import CrossCorrelationMatcher
    from matcha_b200.core.wigner_index import dsize

    cc = CrossCorrelationMatcher(N=N, device=dev, batchsize=1, bandlimit=N // 2, radius=N // 2 - 1,
                                 precision="bf16x3")
    L = cc.lmax
    v = torch.ones((1, N, N, N), device=dev)
    t = torch.ones((cc.fle.ne + 1,), device=dev, dtype=torch.complex64)
    sig = torch.zeros((1, dsize(L)), device=dev, dtype=torch.complex64)
    grad = torch.zeros_like(t)
    lib, h, c, p = nat.load(), cc.fle._h, cc._coeffs, nat.ptr

    def go(stream, keep=(cc, v, t, sig)):
        return (lib.mtb_fle_forward(h, p(v), 1, p(c), c.stride(0), None, stream)
                or lib.mtb_sigma_upto(h, p(c), c.stride(0), p(t), 1, L, p(sig), sig.stride(0), stream)
                or lib.mtb_sigma_backward_template(h, p(c), c.stride(0), p(sig), sig.stride(0), 1, L, p(grad),
                                                   stream))

    return go, grad


def _shift(N, precision, dev):
    from matcha_b200 import _native as nat
    from tests.test_shift_gpu import _matcher

    sm = _matcher(N, 1, 4, N // 16, dev, precision=precision)
    rng = np.random.default_rng(N)
    sm.set_reference(rng.standard_normal((N, N, N)).astype(np.float32))
    v = torch.from_numpy(rng.standard_normal((1, N, N, N)).astype(np.float32)).to(dev)
    z, rot = torch.zeros((1, 3), device=dev), torch.eye(3, device=dev).reshape(1, 9).contiguous()
    out, score = torch.empty((1, 3), device=dev), torch.empty((1,), device=dev)
    sm.search_shifts(subtomos=v, ctfs=None, shift_zyx=z, rotation_tracker=np.array([[1.0, 0, 0, 0]]))
    lib, p = nat.load(), nat.ptr

    def go(stream, keep=(sm, v, z, rot, score)):
        return lib.mtb_shift_search(sm._h, p(v), p(z), p(rot), None, 1, p(out), p(score), stream)

    return go, out


def _grid(L0, dev):
    from matcha_b200 import _native as nat
    from matcha_b200.core.SOFFT import SOFFT
    from matcha_b200.core.wigner_index import dsize

    s = SOFFT(L=L0, device=dev, batchsize=1, oversampling_factor=1)
    sig = torch.ones((1, dsize(L0 - 1)), dtype=torch.complex64, device=dev)
    out = torch.empty((3, 1, 4), device=dev)
    h, lib, p = s._handle(4), nat.load(), nat.ptr

    def go(stream, keep=(s, sig)):
        return lib.mtb_so3_grid_topk(h, p(sig), sig.stride(0), 1, p(out[0]), p(out[1]), p(out[2]), None, stream)

    return go, out


CASES = {"expansion": (lambda dev: _expansion(64, dev), lambda dev: _expansion(16, dev)),
         "shift-bf16x3": (lambda dev: _shift(64, "bf16x3", dev), lambda dev: _shift(16, "bf16x3", dev)),
         "shift-fp32": (lambda dev: _shift(64, "fp32", dev), lambda dev: _shift(16, "fp32", dev)),
         "grid": (lambda dev: _grid(12, dev), lambda dev: _grid(4, dev))}


@pytest.mark.parametrize("case", CASES)
def test_two_sizes_in_two_threads(cuda_device, case):
    calls = [make(cuda_device) for make in CASES[case]]
    want = []
    for go, out in calls:
        assert go(torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        want.append(out.clone())
    refused = [0, 0]

    def work(i):
        stream = torch.cuda.Stream()
        for k in range(6000):
            refused[i] += calls[i][0](stream.cuda_stream) != 0
            if k % 20 == 19:
                stream.synchronize()
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert refused == [0, 0]
    for (_, out), w in zip(calls, want):
        assert torch.equal(out, w)
