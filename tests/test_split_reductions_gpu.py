"""The reductions that a cluster of CTAs shares: template gradient, score backward and the
continuous shift score, at batches around the cluster sizes' changes and at ragged sizes,
against plain FP64 numpy and the oracle.

Tolerances: inputs and outputs are FP32 and sums run over at most a few thousand terms of mixed
sign, so an FP32 sum is within 2e-6 of the largest output and an FP64 one within FP32 rounding
(6e-8 of each value); the factors below leave ten times that."""
import numpy as np
import pytest
import torch

from oracle import shift as OS
from oracle import wigner as OW

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 7, 9, 33, 70])
@pytest.mark.parametrize("L", [0, 3, 16])
def test_template_gradient(cuda_device, B, L):
    from matcha_b200.autograd import template_sigma
    from matcha_b200.core.CrossCorrelationMatcher import CrossCorrelationMatcher
    from matcha_b200.core.fle_tables import sht_index
    from matcha_b200.core.wigner_index import dsize

    rng = np.random.default_rng(10 * B + L)
    cc = CrossCorrelationMatcher(N=32, device=cuda_device, batchsize=B, bandlimit=16, radius=15, precision="fp32")
    cc.expand(torch.from_numpy(rng.standard_normal((B, 32, 32, 32)).astype(np.float32)).to(cuda_device))
    aV = cc._coeffs[:B].cpu().numpy().astype(np.complex128)
    t = torch.from_numpy((rng.standard_normal(cc.fle.ne + 1) + 1j * rng.standard_normal(cc.fle.ne + 1))
                         .astype(np.complex64)).to(cuda_device).requires_grad_(True)
    G = (rng.standard_normal((B, dsize(L))) + 1j * rng.standard_normal((B, dsize(L)))).astype(np.complex64)
    template_sigma(t, cc, L).backward(torch.from_numpy(G).to(cuda_device))
    ref = np.zeros(cc.fle.ne + 1, dtype=np.complex128)
    for l in range(L + 1):
        g = G[:, dsize(l - 1):dsize(l)].reshape(B, 2 * l + 1, 2 * l + 1).astype(np.complex128)
        for mu in range(-l, l + 1):  # sigma[m, m'] = (-1)^(m+m') sum_k T[-m', k] conj(V[-m, k])
            for k, i in enumerate(cc.fle.idlm_list[l][sht_index(mu)]):
                for m in range(-l, l + 1):
                    row = cc.fle.idlm_list[l][sht_index(-m)]
                    if k < len(row):
                        ref[i] += (-1) ** (m + mu) * np.sum(aV[:, row[k]] * g[:, m + l, l - mu])
    np.testing.assert_allclose(t.grad.cpu().numpy(), ref, rtol=0, atol=2e-5 * np.abs(ref).max())


@pytest.mark.parametrize("B,L", [(1, 0), (1, 1), (3, 6), (74, 5), (75, 2), (149, 3), (300, 2), (600, 1), (2, 17)])
def test_score_backward(cuda_device, B, L):
    from matcha_b200 import _native as nat

    rng = np.random.default_rng(B + L)
    n = OW.dsize(L)
    ang = np.stack([rng.uniform(-3, 3, B), rng.uniform(0, np.pi, B), rng.uniform(-3, 3, B)]).astype(np.float32)
    ang[1, 0] = 0.0
    sig = ((rng.standard_normal((B, n)) + 1j * rng.standard_normal((B, n))) / np.sqrt(n)).astype(np.complex64)
    w = rng.standard_normal(B).astype(np.float32)
    dev = [torch.from_numpy(x).to(cuda_device) for x in (sig, ang, w)]
    gs = torch.zeros((B, n), dtype=torch.complex64, device=cuda_device)
    gb = torch.zeros((B, 3), dtype=torch.float64, device=cuda_device)
    nat.check(nat.load().mtb_score_backward(nat.ptr(dev[0]), n, B, L, nat.ptr(dev[1][0]), nat.ptr(dev[1][1]),
                                            nat.ptr(dev[1][2]), nat.ptr(dev[2]), nat.ptr(gs), n, nat.ptr(gb),
                                            nat.stream_ptr(cuda_device)), "mtb_score_backward")
    D = OW.wigner_D(*ang.astype(np.float64), L)
    np.testing.assert_allclose(gs.cpu().numpy(), w[:, None] * np.conj(D), rtol=0, atol=1e-6 * np.abs(w).max())
    ref = np.zeros((B, 3))
    for l in range(L + 1):
        m = np.arange(-l, l + 1)
        up = np.sqrt((l - m[:-1]) * (l + m[:-1] + 1)) / 2
        gen = [1j * (np.diag(up, 1) + np.diag(up, -1)), np.diag(up, 1) - np.diag(up, -1), np.diag(1j * m)]
        sl = slice(OW.dsize(l - 1), OW.dsize(l))
        Dl, s = D[:, sl].reshape(B, 2 * l + 1, -1), sig[:, sl].reshape(B, 2 * l + 1, -1).astype(np.complex128)
        for k in range(3):
            ref[:, k] += w * np.sum((Dl @ gen[k]) * s, (1, 2)).real
    np.testing.assert_allclose(gb.cpu().numpy(), ref, rtol=0, atol=1e-6 * max(np.abs(ref).max(), 1e-3))


@pytest.mark.parametrize("N,B", [(4, 2), (8, 1), (8, 149), (8, 300), (8, 600), (16, 5), (48, 2), (80, 1)])
def test_shift_score_gradient(cuda_device, N, B):
    from matcha_b200.core.ShiftMatcher import ShiftMatcher

    rng = np.random.default_rng(N + B)
    sm = ShiftMatcher(dict(N=N, num_subtomograms_per_batch=B, shift_upsample_factor=4, shift_search_radius=1,
                           do_ctf_correction=False), cuda_device, torch.complex64)
    template = rng.standard_normal((N, N, N))
    sm.set_reference(template)
    vols = rng.standard_normal((B, N, N, N)).astype(np.float32)
    prior = rng.uniform(-1, 1, (B, 3)).astype(np.float32)
    ang = rng.uniform(10, 170, (B, 3))
    from scipy.spatial.transform import Rotation as R

    rot = R.from_euler("ZYZ", ang, degrees=True).as_matrix().reshape(B, 9).astype(np.float32)
    q = rng.uniform(-1.5, 1.5, (B, 3)).astype(np.float32)
    c, g = sm.score_and_gradient(torch.from_numpy(vols).to(cuda_device), torch.from_numpy(prior),
                                 torch.from_numpy(rot), torch.from_numpy(q))
    ref = sm.reference_data_fourier[0].cpu().numpy()
    for b in {0, B // 2, B - 1}:
        c_ref, g_ref = OS.shift_score_and_grad(ref, vols[b], prior[b], ang[b], q[b])
        # the FP32 transforms in front of the sum: 2e-5 of the score's scale (unit-norm products)
        assert abs(c[b].item() - c_ref) < 2e-5
        np.testing.assert_allclose(g[b].cpu().numpy(), g_ref, rtol=0, atol=2e-5 * np.pi)


@pytest.mark.parametrize("B", [1, 63, 64, 65, 200])
def test_rotation_angles_and_gradient(cuda_device, B):
    """The one-launch rotations against the module's own torch functions in FP64: the rotation of
    the angles within FP32 rounding of angles up to pi (2e-7 each), the gradient in FP64."""
    from matcha_b200 import _native as nat
    from matcha_b200.autograd import right_jacobian, so3_exp, zyz_matrix

    rng = np.random.default_rng(B)
    omega, base = torch.tensor(rng.standard_normal((B, 3))), torch.tensor(rng.uniform(-3, 3, (B, 3)))
    omega[0] = 0
    base[0, 1] = 0.0
    if B > 2:
        omega[1], base[1, 1] = 0, np.pi
        omega[2] = torch.tensor([1e-9, -2e-9, 1e-7], dtype=torch.float64)
    body = torch.tensor(rng.standard_normal((B, 3)))
    w, e, g = (t.to(cuda_device) for t in (omega, base, body))
    ang, out = torch.empty((3, B), device=cuda_device), torch.empty_like(w)
    lib = nat.load()
    nat.check(lib.mtb_rotation_angles(nat.ptr(w), nat.ptr(e), B, nat.ptr(ang[0]), nat.ptr(ang[1]), nat.ptr(ang[2]),
                                      nat.stream_ptr(cuda_device)), "mtb_rotation_angles")
    nat.check(lib.mtb_rotation_gradient(nat.ptr(w), nat.ptr(g), B, nat.ptr(out), nat.stream_ptr(cuda_device)),
              "mtb_rotation_gradient")
    R = zyz_matrix(base[:, 0], base[:, 1], base[:, 2]) @ so3_exp(omega)
    torch.testing.assert_close(zyz_matrix(*ang.cpu().double()), R, atol=1e-6, rtol=0)
    assert bool((ang[1] >= 0).all())
    ref = (right_jacobian(omega).transpose(-1, -2) @ body[..., None])[..., 0]
    torch.testing.assert_close(out.cpu(), ref, atol=1e-9, rtol=0)


@pytest.mark.parametrize("B", [2, 4, 5, 8])
def test_template_gradient_of_few(cuda_device, B):
    """A batch that one CTA gathers whole, and the smallest ones that a cluster shares, against the sum
    of the subtomograms' gradients one by one (FP32 sums of a few hundred terms: 2e-6 of the largest)."""
    from matcha_b200.autograd import template_sigma
    from matcha_b200.core.CrossCorrelationMatcher import CrossCorrelationMatcher

    g = torch.Generator(device=cuda_device).manual_seed(B)
    cc = CrossCorrelationMatcher(N=32, device=cuda_device, batchsize=B, bandlimit=16, radius=15, precision="fp32")
    v = torch.randn((B, 32, 32, 32), generator=g, device=cuda_device)
    w = torch.randn((B, cc.sigma.shape[1]), generator=g, device=cuda_device, dtype=torch.complex64)

    def grad(sl):
        cc.expand(v[sl])
        t = torch.ones((cc.fle.ne + 1,), device=cuda_device, dtype=torch.complex64, requires_grad=True)
        template_sigma(t, cc, cc.lmax).backward(w[sl])
        return t.grad.to(torch.complex128)

    want = sum(grad(slice(b, b + 1)) for b in range(B))
    assert (grad(slice(0, B)) - want).abs().max() < 2e-6 * want.abs().max()


@pytest.mark.parametrize("B", [1, 9])
def test_template_gradient_of_an_infinite_coefficient(cuda_device, B):
    """An infinite coefficient makes its own entries infinite, not all that rows past the end touch."""
    from matcha_b200.autograd import template_sigma
    from matcha_b200.core.CrossCorrelationMatcher import CrossCorrelationMatcher
    from matcha_b200.core.fle_tables import sht_index

    cc = CrossCorrelationMatcher(N=16, device=cuda_device, batchsize=B, bandlimit=8, radius=7, precision="fp32")
    cc.expand(torch.ones((B, 16, 16, 16), device=cuda_device))
    cc._coeffs.fill_(1.0 + 1.0j)
    at = int(cc.fle.idlm_list[0][sht_index(0)][0])
    cc._coeffs[0, at] = complex(float("inf"), 1.0)
    t = torch.ones((cc.fle.ne + 1,), device=cuda_device, dtype=torch.complex64, requires_grad=True)
    template_sigma(t, cc, 1).backward(torch.full((B, 1 + 9), 1.0 + 1.0j, device=cuda_device, dtype=torch.complex64))
    grad = torch.view_as_real(t.grad)
    assert torch.isinf(grad[at]).all()
    others = torch.ones(cc.fle.ne + 1, dtype=torch.bool, device=cuda_device)
    others[at] = False
    assert torch.isfinite(grad[others]).all()
