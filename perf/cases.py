"""The measured workload: what a subtomogram alignment run has this framework do, stage by
stage through the classes a program calls, and two whole calls.

expand    CrossCorrelationMatcher.get_sigma: ball expansion of a batch, correlation with the template
search    Matcha.search_orientations: SO(3) grid, frequency-marched Newton refinement
shift     ShiftMatcher.search_shifts: the sub-voxel shift match
prepare   AlignmentStep.prepare: patch at the current shift, normalised, masked and rotated
align     AlignmentStep(...): one whole alternation
gradient  autograd.summed_aligned_correlation and its backward (template refinement)

A run keeps one plan per configuration (its tables, template and workspaces) and sends batch
after batch through it, and so does this file: plans are made once per configuration, the
inputs of every state from its seed alone.  Boxes 32-128, bandlimits N/2, batches from one
particle (a template, the rest of a run) to the benchmark's 1000 come from bench.py, its
mixed-box and high-bandlimit shapes, and the tests.

Particles are rotated, shifted copies of a template of Gaussian blobs of both signs (the
contrast that a microscope's transfer function leaves: little power at the lowest
frequencies) in white noise, at 0 dB, and 5 dB (the top of the mixed workload) where a shift
is searched.  There the offsets lie on the searched 1/upsample_factor grid (the last axis of
the match is sampled by fftfreq(N/2+1), so its step is N/(N/2+1) times larger): half-way
offsets would make the returned peak a toss between two equal grid values.
"""
import math

import numpy as np
import torch

from matcha_b200.autograd import summed_aligned_correlation
from matcha_b200.core.CrossCorrelationMatcher import CrossCorrelationMatcher
from matcha_b200.core.Matcha import Matcha
from matcha_b200.core.ShiftMatcher import ShiftMatcher
from matcha_b200.pipeline import AlignmentStep, StepConfig

DEV = "cuda"
# frequency march below the final degree: the configurations' L/4 steps (8, 16, 24 at L = 32)
MARCH = {8: (4,), 16: (8,), 20: (7, 13), 24: (8, 16), 32: (8, 16, 24), 40: (10, 20, 30), 48: (12, 24, 36),
         64: (16, 32, 48)}
# largest batch of each box in a drawn case: no dearer than the listed large cases
MOST = {"expand": {32: 1000, 48: 1000, 64: 1000, 80: 240, 96: 100},
        "search": {8: 1000, 16: 1000, 20: 1000, 24: 1000, 32: 1000, 40: 400, 48: 200, 64: 64},
        "shift": {32: 1000, 48: 1000, 64: 900, 80: 60, 96: 200, 128: 48},
        "prepare": {32: 1000, 48: 1000, 64: 1000, 80: 500, 96: 250},
        "align": {32: 1000, 48: 400, 64: 256}, "gradient": {32: 256, 48: 256, 64: 200}}


def listed():
    return [
        # the smallest call of a run: one volume (the template, a run's last particle)
        {"name": "expand-48-b1", "kind": "expand", "N": 48, "L": 24, "B": 1, "cap": 1},
        # the benchmark batch
        {"name": "expand-64-b1000", "kind": "expand", "N": 64, "L": 32, "B": 1000, "cap": 1000},
        # the large box of the mixed workload, a batch short of the plan's capacity
        {"name": "expand-96-b100", "kind": "expand", "N": 96, "L": 48, "B": 100, "cap": 128},
        # the reference's default search settings (10 candidates, 5 Newton steps) on a small set
        {"name": "search-L16-b16", "kind": "search", "L": 16, "B": 16, "C": 10, "steps": 5},
        # the benchmark batch: one Newton step per stage of the march 8, 16, 24, 32
        {"name": "search-L32-b1000", "kind": "search", "L": 32, "B": 1000, "C": 10, "steps": 1},
        # the high-bandlimit march 16, 32, 48, 64
        {"name": "search-L64-b64", "kind": "search", "L": 64, "B": 64, "C": 10, "steps": 1},
        # the reference's default shift settings (1/16 voxel, radius 2) with CTF weights, odd batch
        {"name": "shift-48-b37-ctf", "kind": "shift", "N": 48, "B": 37, "uf": 16, "r": 2, "ctf": True},
        # the benchmark batch: 1/8 voxel, radius 5
        {"name": "shift-64-b1000", "kind": "shift", "N": 64, "B": 1000, "uf": 8, "r": 5, "ctf": False},
        # the high-bandlimit box: 1/8 voxel, radius 8
        {"name": "shift-128-b48", "kind": "shift", "N": 128, "B": 48, "uf": 8, "r": 8, "ctf": False},
        # the benchmark batch, before every alternation
        {"name": "prepare-64-b1000", "kind": "prepare", "N": 64, "L": 32, "B": 1000},
        # a whole alternation of the smallest configuration
        {"name": "align-32-b16", "kind": "align", "N": 32, "L": 16, "B": 16, "uf": 8, "r": 3},
        # the differentiation workload: score of a batch, backward to rotations, shifts, template
        {"name": "gradient-64-b256", "kind": "gradient", "N": 64, "L": 32, "B": 256},
    ]


def draw(rng):
    kind = rng.choice(["expand", "expand", "search", "search", "shift", "shift", "prepare", "align", "gradient"])
    key = rng.choice(sorted(MOST[kind]))
    B = int(round(math.exp(rng.uniform(0.0, math.log(MOST[kind][key])))))
    if kind == "search":
        return {"kind": kind, "L": key, "B": B, "C": rng.choice([4, 7, 10, 16]), "steps": rng.choice([1, 1, 2, 5])}
    case = {"kind": kind, "N": key, "B": B}
    if kind != "shift":
        case["L"] = key // 2
    if kind == "expand":
        case["cap"] = B + rng.choice([0, 0, rng.randint(1, 40)])
    if kind in ("shift", "align"):
        case["uf"], case["r"] = rng.choice([(8, 5), (8, 3), (16, 2), (4, 6), (10, 4)])
    if kind == "shift":
        case["ctf"] = rng.random() < 0.3
    return case


# ---------------------------------------------------------------- synthetic data
def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _radius(N):
    return min(N // 2, int(N // 2 * 0.95))


def _matrix(q):
    w, x, y, z = q.unbind(-1)
    rows = [1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
            2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
            2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]
    return torch.stack(rows, -1).reshape(q.shape[:-1] + (3, 3))


def _haar(g, B):
    q = torch.randn((B, 4), generator=g, device=DEV, dtype=torch.float64)
    return q / q.norm(dim=1, keepdim=True)


def _blobs(N):
    """The box's template as Gaussian blobs: centres (x, y, z) about N/2 in two lobes, widths, amplitudes."""
    g = _rng(N)
    n = min(1500, max(60, round(400 * (N / 64) ** 2)))
    d = torch.randn((n, 3), generator=g, device=DEV)
    d = d / d.norm(dim=1, keepdim=True) * torch.rand((n, 1), generator=g, device=DEV) ** (1 / 3)
    off = torch.tensor([[-0.05, 0.02, 0.0], [0.1, -0.07, 0.05]], device=DEV)
    which = torch.arange(n, device=DEV) % 2
    c = N * (off[which] + d * torch.where(which == 0, 0.32, 0.2)[:, None])
    u = torch.rand((2, n), generator=g, device=DEV)
    return c, 1.5 + u[0], (0.5 + 0.5 * u[1]) * (1 - 2 * (torch.arange(n, device=DEV) // 2 % 2))


def _render(c, s, a, N):
    """Volumes [b, z, y, x] of blobs at c (B, J, 3) (x, y, z offsets from N/2); separable per blob."""
    g = torch.arange(N, device=DEV) - N // 2
    out = torch.empty((c.shape[0], N, N, N), device=DEV)
    step = max(1, (1 << 28) // (c.shape[1] * N * N))
    for i in range(0, c.shape[0], step):
        e = torch.exp(-(g - c[i:i + step, :, :, None]) ** 2 / (2 * s[:, None, None] ** 2))
        yx = (e[:, :, 1, :, None] * e[:, :, 0, None, :]).flatten(2)
        out[i:i + step] = torch.bmm((a[:, None] * e[:, :, 2]).transpose(1, 2), yx).view(-1, N, N, N)
    return out


def _template(N):
    c, s, a = _blobs(N)
    return _render(c[None], s, a, N)[0]


def _particles(g, q, move, N, snr_db=0.0):
    """Copies of the template turned by q (v(p) = template(M p)), moved by `move` (x, y, z), in white noise."""
    c, s, a = _blobs(N)
    v = _render((c.double() @ _matrix(q)).float() + move[:, None], s, a, N)
    p = torch.arange(N, device=DEV) - N // 2
    ball = (p[:, None, None] ** 2 + p[:, None] ** 2 + p ** 2) < (0.45 * N) ** 2
    for b in range(v.shape[0]):
        power = (v[b][ball] ** 2).mean()
        v[b] += torch.randn(v[b].shape, generator=g, device=DEV) * (power * 10 ** (-snr_db / 10)).sqrt()
    return v


def _offsets(g, case):
    """(prior shift (x, y, z), true offset): the residual lies on the searched grid."""
    B, N, uf = case["B"], case["N"], case["uf"]
    reach = max(1, int(uf * min(case["r"], 3) * 0.5))
    prior = torch.randint(-16, 17, (B, 3), generator=g, device=DEV) / 8.0
    rest = torch.randint(-reach, reach + 1, (B, 3), generator=g, device=DEV) / uf
    rest[:, 0] *= N / (N // 2 + 1)
    return prior, prior + rest


def _zyz(R):
    return torch.stack([torch.atan2(R[:, 1, 2], R[:, 0, 2]), torch.acos(R[:, 2, 2].clamp(-1, 1)),
                        torch.atan2(R[:, 2, 1], -R[:, 2, 0])], -1)


def _generators(l):
    """Generators A_x, A_y, A_z of the degree-l rotation matrices D(R exp(t e_k)) = D(R) exp(t A_k)."""
    m = torch.arange(-l, l + 1, device=DEV, dtype=torch.float64)
    up = torch.sqrt((l - m[:-1]) * (l + m[:-1] + 1)) / 2
    Ay = torch.diag(up, 1) - torch.diag(up, -1)
    Ax = 1j * (torch.diag(up, 1) + torch.diag(up, -1))
    return Ax.to(torch.complex128), Ay.to(torch.complex128), torch.diag(1j * m)


def _wigner(l, angles):
    """D^l(a, b, g) = e^{i m' a} d^l(b) e^{i m g}, (B, 2l+1, 2l+1) complex128."""
    m = torch.arange(-l, l + 1, device=DEV, dtype=torch.float64)
    lam, U = torch.linalg.eigh(1j * _generators(l)[1])
    a, b, g = angles.double().unbind(-1)
    d = (U * torch.exp(-1j * b[:, None, None] * lam)) @ U.mH
    return torch.exp(1j * a[:, None] * m)[:, :, None] * d * torch.exp(1j * g[:, None] * m)[:, None, :]


def _dsize(L):
    return (L + 1) * (2 * L + 1) * (2 * L + 3) // 3


def _sigma(seed, L, B):
    """Correlation coefficients of B noisy, turned copies of a band-limited template."""
    g = _rng(seed)
    q = _haar(g, B)
    ang = _zyz(_matrix(q))
    out = torch.empty((B, _dsize(L)), device=DEV, dtype=torch.complex64)
    for l in range(L + 1):
        K = max(1, int((L * math.pi / 2 - l - 1.86 * l ** (1 / 3)) / math.pi))
        t = torch.randn((2 * l + 1, K), generator=_rng(1000 + l), device=DEV, dtype=torch.complex128)
        sign = (-1.0) ** torch.arange(-l, l + 1, device=DEV, dtype=torch.float64)[:, None]
        t = (t + sign * t.flip(0).conj()) * math.exp(-l / (0.35 * L))  # of a real volume
        v = _wigner(l, ang).transpose(1, 2) @ t
        v = v + 0.1 * torch.randn(v.shape, generator=g, device=DEV, dtype=torch.complex128)
        out[:, _dsize(l - 1):_dsize(l)] = (t @ v.mH).flatten(1)
    return out


# ---------------------------------------------------------------- plans and inputs
_plans = {}


def _plan(key, make):
    if key not in _plans:
        _plans[key] = make()
    return _plans[key]


def _march(L):
    return list(MARCH[L])


def _step(case):
    N, L, B, uf, r = case["N"], case["L"], case["B"], case.get("uf", 8), case.get("r", 5)

    def make():
        step = AlignmentStep(StepConfig(N=N, L=L, Li=_march(L), batch=B, shift_upsample_factor=uf,
                                        shift_search_radius=r), DEV)
        step.set_template(_template(N).cpu().numpy())
        return step

    return _plan(("step", N, L, B, uf, r), make)


def _correlator(case):
    def make():
        c = CrossCorrelationMatcher(N=case["N"], device=DEV, batchsize=case["cap"], bandlimit=case["L"],
                                    radius=_radius(case["N"]), precision_mode="fast")
        c.set_template(_template(case["N"]).cpu().numpy())
        return c

    return _plan(("expand", case["N"], case["L"], case["cap"]), make)


def _shifter(case):
    def make():
        s = ShiftMatcher(dict(N=case["N"], num_subtomograms_per_batch=case["B"], shift_upsample_factor=case["uf"],
                              shift_search_radius=case["r"], do_ctf_correction=case["ctf"], precision_mode="fast"),
                         DEV, torch.complex64)
        s.set_reference(_template(case["N"]).cpu().numpy())
        return s

    return _plan(("shift", case["N"], case["B"], case["uf"], case["r"], case["ctf"]), make)


def _matcher(case):
    return _plan(("search", case["L"], case["B"], case["C"], case["steps"]),
                 lambda: Matcha(case["B"], DEV, case["L"], dict(Li=_march(case["L"]), candidates=case["C"],
                                                                 num_steps=case["steps"])))


def _inputs(case, seed):
    g = _rng(seed)
    kind, B = case["kind"], case["B"]
    if kind == "search":
        return {"sigma": _sigma(seed, case["L"], B)}
    N, q = case["N"], _haar(g, B)
    conj = q * torch.tensor([1.0, -1, -1, -1], device=DEV, dtype=torch.float64)
    if kind == "expand":
        move = torch.rand((B, 3), generator=g, device=DEV) - 0.5
        return {"volumes": _particles(g, q, move, N)}
    if kind == "prepare":
        shift = 4 * torch.rand((B, 3), generator=g, device=DEV) - 2
        return {"volumes": _particles(g, q, shift, N), "shift": shift, "tracker": conj}
    if kind == "shift":
        prior, true = _offsets(g, case)
        d = {"volumes": _particles(g, q, true, N, 5.0), "shift": prior, "tracker": conj, "ctf": None}
        if case["ctf"]:
            k = torch.fft.fftfreq(N, device=DEV)
            r2 = k[:, None, None] ** 2 + k[:, None] ** 2 + torch.fft.rfftfreq(N, device=DEV) ** 2
            defocus = 20 + 20 * torch.rand((B, 1, 1, 1), generator=g, device=DEV)
            d["ctf"] = torch.sin(0.3 + defocus * r2).abs() * torch.exp(-2 * r2)
        return d
    if kind == "align":
        prior, true = _offsets(g, case)
        return {"volumes": _particles(g, q, torch.zeros((B, 3), device=DEV), N, 5.0),
                "subtomos": _particles(g, q, true, N, 5.0), "shift": prior}
    # gradient: near the optimum, as in the steps of a refinement
    swap = torch.eye(3, device=DEV, dtype=torch.float64).flip(0)
    R = _matrix(q)
    small = 0.02 * torch.randn((2, B, 3), generator=g, device=DEV, dtype=torch.float64)
    move = 2 * torch.rand((B, 3), generator=g, device=DEV) - 1
    return {"volumes": _particles(g, q, move, N), "base": _zyz(swap @ R.mT @ swap) + small[0], "omega": small[1],
            "rot": R.float().reshape(B, 9), "zero": torch.zeros((B, 3), device=DEV),
            "shift": move * torch.tensor([(N // 2 + 1) / N, 1.0, 1.0], device=DEV)
            + 0.1 * torch.randn((B, 3), generator=g, device=DEV)}


def prepare(case, seed):
    state = dict(_inputs(case, seed), kind=case["kind"])
    plan = {"expand": _correlator, "search": _matcher, "shift": _shifter}.get(case["kind"], _step)(case)
    state["plan"] = plan
    if case["kind"] == "align":
        # the trackers are updated in place: a pass starts from the identity, as a run's first one
        state["start"] = torch.tensor([[1.0, 0, 0, 0]], device=DEV, dtype=torch.float64).repeat(case["B"], 1)
    if case["kind"] == "gradient":
        state["template"] = plan.correlator.template_coefficients_alphas_torch.clone()
    return state


def run(s):
    plan, kind = s["plan"], s["kind"]
    if kind == "expand":
        return plan.get_sigma(s["volumes"])
    if kind == "search":
        return plan.search_orientations(s["sigma"])
    if kind == "shift":
        return plan.search_shifts(subtomos=s["volumes"], ctfs=s["ctf"], shift_zyx=s["shift"],
                                  rotation_tracker=s["tracker"])
    if kind == "prepare":
        return plan.prepare(s["volumes"], s["shift"], s["tracker"])
    if kind == "align":
        out = plan(s["volumes"], s["subtomos"], s["start"].clone(), s["shift"])
        return {k: v.float() for k, v in out.items()}  # the trackers: 32-bit angles in 64-bit quaternions
    leaves = [s[k].detach().requires_grad_(True) for k in ("omega", "template", "shift")]
    total = summed_aligned_correlation(plan, s["volumes"], leaves[0], s["base"], leaves[1], leaves[2], s["zero"],
                                       s["rot"])
    grads = torch.autograd.grad(total, leaves)
    # sums of 32-bit scores, widened by the entry point
    return {"total": total.detach().float(), "omega": grads[0].float(), "template": grads[1], "shift": grads[2]}


# ---------------------------------------------------------------- what a pass cannot do without
def _expansion_size(N, L):
    """(octant voxels, real coefficients, degrees) of the expansion, from the volumes they fill."""
    r = _radius(N)
    c = np.arange(r + 1)
    reps = int(((c[:, None, None] ** 2 + c[:, None] ** 2 + c ** 2) <= r * r).sum())
    table = _spectrum(L)
    return reps, len(table), 1 + max(t[1] for t in table)


def _march_flops(case):
    """Terms of the score over the folded chains: value, gradient and Hessian once per step, the value of each trial."""
    n = 0
    for l in _march(case["L"]) + [case["L"]]:
        n += (l + 1) * (l + 2) * (2 * l + 3) // 6 * (case["steps"] * 50 + 14)
    return n * case["C"]


def work(case):
    kind, B = case["kind"], case["B"]
    if kind == "search":
        L0 = min(_march(case["L"]))
        n, p = 4 * L0, 2 * L0 - 1
        grid = n * (2 * _dsize(L0 - 1) + 4 * p * p * n + 2 * p * n * n)
        return {"bytes": B * (8 * _dsize(case["L"]) + 16), "flops": B * (grid + _march_flops(case))}
    N = case["N"]
    vol = 4 * N ** 3
    if kind == "prepare":
        return {"bytes": B * 2 * vol, "flops": B * 60 * N ** 3}
    fft = 5 * N ** 3 * math.log2(N)
    if kind == "expand":
        reps, cols, deg = _expansion_size(N, case["L"])
        return {"bytes": 4 * reps * cols + B * vol + case["cap"] * 8 * _dsize(deg - 1),
                "flops": 2.0 * B * reps * cols + B * 8.0 * cols * deg}
    if kind == "gradient":
        reps, cols, deg = _expansion_size(N, case["L"])
        sig = _dsize(case["L"])
        return {"bytes": 4 * reps * cols + B * vol + 16 * cols + B * 100,
                "flops": B * (2.0 * reps * cols + fft + 200 * sig + 16.0 * cols * case["L"] + 30 * N ** 3)}
    U = case["uf"] * (2 * case["r"] + 1)
    H = N // 2 + 1
    dft = 8.0 * (U * N * N * H + U * U * N * H) + 4.0 * U ** 3 * H
    shift = {"bytes": B * (vol + (4 * N * N * H if case.get("ctf") else 0)) + 8 * N ** 3,
             "flops": B * (fft + dft + 60 * N * N * H)}
    if kind == "shift":
        return shift
    reps, cols, deg = _expansion_size(N, case["L"])
    march = _march_flops({"L": case["L"], "C": 10, "steps": 1})
    return {"bytes": shift["bytes"] + 4 * reps * cols + B * vol, "flops": shift["flops"] + B * (2.0 * reps * cols + march)}


# ---------------------------------------------------------------- 64-bit values, in plain torch and numpy
def _upward(l, x):
    """j_0 .. j_l at x >= l (the upward recurrence is stable there)."""
    j = [np.sin(x) / x, np.sin(x) / x ** 2 - np.cos(x) / x]
    for n in range(1, l):
        j.append((2 * n + 1) / x * j[n] - j[n - 1])
    return j[:l + 1]


_spectra = {}


def _spectrum(L):
    """The expansion's (lambda, l, k, m): zeros lambda_lk < L pi / 2 of j_l in ascending order, m = 0, -1, 1, ..;
    the last coefficient is dropped, and with it the partner it leaves without one."""
    if L in _spectra:
        return _spectra[L]
    top = L * math.pi / 2
    z = np.pi * np.arange(1, int(top) + 4, dtype=np.float64)
    rows, l = [], 0
    while z.size and z[0] < top:
        rows += [(v, l, k) for k, v in enumerate(z, 1) if v < top]
        l += 1
        lo, hi = z[:-1].copy(), z[1:].copy()  # the zeros of j_l lie between those of j_{l-1}
        s = np.sign(_upward(l, lo)[l])
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            left = np.sign(_upward(l, mid)[l]) == s
            lo, hi = np.where(left, mid, lo), np.where(left, hi, mid)
        z = 0.5 * (lo + hi)
    out = [(v, l, k, m) for v, l, k in sorted(rows) for m in sorted(range(-l, l + 1), key=lambda m: (abs(m), m))]
    out = out[:-1]
    if out[-1][3] < 0:
        out = out[:-1]
    _spectra[L] = out
    return out


def _jl(l, x):
    """j_l(x) by downward recurrence from far above, scaled on j_0 and j_1."""
    x = x.clamp_min(1e-14)
    hi, f, keep = torch.zeros_like(x), torch.ones_like(x), None
    for n in range(max(l, int(x.max())) + 40, 0, -1):
        if n == l:
            keep = f
        hi, f = f, (2 * n + 1) / x * f - hi
        s = 1 / torch.maximum(f.abs(), hi.abs()).clamp_min(1.0)
        hi, f = hi * s, f * s
        keep = None if keep is None else keep * s
    keep = f if l == 0 else keep
    j0 = torch.sin(x) / x
    j1 = torch.where(x < 1e-3, x / 3, j0 / x - torch.cos(x) / x)
    return keep * (f * j0 + hi * j1) / (f * f + hi * hi)


def _expansion(vols, L):
    """{(l, m >= 0): coefficients (B, K_l) complex128} of volumes [b, x, y, z]."""
    N = vols.shape[1]
    r = _radius(N)
    g = torch.arange(N, device=DEV, dtype=torch.float64) - N // 2
    x, y, z = torch.meshgrid(g, g, g, indexing="ij")
    r2 = x * x + y * y + z * z
    at = (r2 <= r * r).flatten().nonzero()[:, 0]
    x, y, z, r2 = (t.flatten()[at] for t in (x, y, z, r2))
    f = vols.flatten(1)[:, at].double()
    rad, inv = torch.unique(r2, return_inverse=True)
    ct = torch.where(r2 > 0, z / r2.sqrt().clamp_min(1e-9), 1.0)
    st, phi = (x * x + y * y).sqrt() / r2.sqrt().clamp_min(1e-9), torch.atan2(y, x)
    have = {}
    for v, l, k, m in _spectrum(L):
        have.setdefault(l, {}).setdefault(abs(m), []).append(v)
    radial = {}
    for l, by in have.items():
        lam = torch.tensor(by[0], device=DEV, dtype=torch.float64)
        c = torch.tensor([math.sqrt(2) / abs(_upward(l + 1, np.float64(v))[l + 1]) for v in lam.tolist()],
                         device=DEV, dtype=torch.float64)
        radial[l] = _jl(l, rad.sqrt()[:, None] / r * lam) * c * r ** -1.5
    out, pmm = {}, torch.full_like(ct, 0.5 / math.sqrt(math.pi))
    for m in range(max(have) + 1):
        if m:
            pmm = -math.sqrt((2 * m + 1) / (2 * m)) * st * pmm
        fc, fs = f * torch.cos(m * phi), f * torch.sin(m * phi)
        p0, p1 = torch.zeros_like(pmm), pmm
        for l in range(m, max(have) + 1):
            if l > m:
                a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
                b = math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1)) if l > m + 1 else 0.0
                p0, p1 = p1, a * (ct * p1 - b * p0)
            n = len(have.get(l, {}).get(m, [])) // (2 if m else 1)
            if n:
                B = p1[:, None] * radial[l][inv, :n]
                out[l, m] = torch.complex(fc @ B, -(fs @ B))
    return out


def _rows(coef, l):
    """(B, 2l+1, K) of one degree: a_{-m} = (-1)^m conj(a_m); a dropped zero's orders stay 0."""
    K = max(v.shape[1] for (d, _), v in coef.items() if d == l)
    B = next(iter(coef.values())).shape[0]
    a = torch.zeros((B, 2 * l + 1, K), device=DEV, dtype=torch.complex128)
    for m in range(l + 1):
        v = coef.get((l, m))
        if v is not None:
            a[:, l + m, :v.shape[1]] = v
            a[:, l - m, :v.shape[1]] = (-1) ** m * v.conj() if m else v
    return a


def _correlate(T, V, l):
    """sigma[l, m, m'] = (-1)^(m+m') sum_k T[-m', k] conj(V[-m, k])."""
    s = (-1.0) ** torch.arange(2 * l + 1, device=DEV, dtype=torch.float64)
    return s[:, None] * s * (V.flip(1).conj() @ T.flip(0).T)


def _exact_expand(case, seed):
    coef = _expansion(_inputs(case, seed)["volumes"], case["L"])
    tmpl = _expansion(_template(case["N"])[None], case["L"])
    deg = 1 + max(l for l, _ in coef)
    out = torch.zeros((case["cap"], _dsize(deg - 1)), device=DEV, dtype=torch.complex128)
    norms = torch.zeros(case["cap"], device=DEV, dtype=torch.float64)
    for l in range(deg):
        V = _rows(coef, l)
        out[:case["B"], _dsize(l - 1):_dsize(l)] = _correlate(_rows(tmpl, l)[0], V, l).flatten(1)
        norms[:case["B"]] += (V.abs() ** 2).sum((1, 2))
    return out, norms.sqrt()


def _sample(vol, z, y, x):
    """Trilinear values of vol (B, D, H, W) at points (B, ...), zero outside the box."""
    out = 0.0
    D, H, W = vol.shape[1:]
    b = torch.arange(vol.shape[0], device=DEV).view((-1,) + (1,) * (z.ndim - 1))
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                zi, yi, xi = z.floor() + dz, y.floor() + dy, x.floor() + dx
                w = (1 - (z - zi).abs()) * (1 - (y - yi).abs()) * (1 - (x - xi).abs())
                ok = (zi >= 0) & (zi < D) & (yi >= 0) & (yi < H) & (xi >= 0) & (xi < W)
                v = vol[b, zi.clamp(0, D - 1).long(), yi.clamp(0, H - 1).long(), xi.clamp(0, W - 1).long()]
                out = out + torch.where(ok, w, 0.0) * v
    return out


def _grid(N, c):
    g = torch.arange(N, device=DEV, dtype=torch.float64) - c
    return torch.meshgrid(g, g, g, indexing="ij")


def _exact_prepare(case, seed):
    s, N = _inputs(case, seed), case["N"]
    z, y, x = _grid(N, N // 2)
    mask = ((z * z + y * y + x * x).sqrt() < _radius(N)).double()
    out = []
    for b in range(case["B"]):
        v, sh = s["volumes"][b:b + 1].double(), s["shift"][b].double()
        c = N // 2
        p = _sample(v, (z + c + sh[2])[None], (y + c + sh[1])[None], (x + c + sh[0])[None])
        mean = (p * mask).sum() / mask.sum()
        p = (p - mean) / ((p * p * mask).sum() / mask.sum() - mean ** 2).sqrt() * mask
        M = _matrix(s["tracker"][b])
        t = torch.stack([x, y, z]).flatten(1)
        t = (M @ t).view(3, N, N, N) + c
        out.append(_sample(p, t[2][None], t[1][None], t[0][None])[0].float())
    # a sample is a sum of eight products: rounding it to 32 bits is far below what either side is off
    return torch.stack(out)


def _reference(N):
    """The template's Fourier reference: soft low-pass (resolution 4 voxels, edge 2), gridding correction, centred
    transform in the ball mask."""
    t = _template(N).double()
    z, y, x = _grid(N, N // 2)
    r = (z * z + y * y + x * x).sqrt()
    rad, edge = N / 4.0 - 1.0, 2.0
    band = 0.5 - 0.5 * torch.cos(math.pi * (rad + edge - r) / edge)
    soft = torch.where(r > rad + edge, 0.0, torch.where(r >= rad, band, 1.0))
    f = torch.fft.fftshift(torch.fft.fftn(t, norm="forward")) * soft
    t = torch.fft.ifftn(torch.fft.ifftshift(f), norm="forward").real / torch.sinc(r / N) ** 2
    f = torch.fft.fftshift(torch.fft.fftn(torch.roll(t, (-(N // 2),) * 3, (0, 1, 2)), norm="forward"))
    return torch.where(r * r <= N // 2 * N // 2, f, 0.0)


def _products(ref, vols, prior, M, ctf, N):
    """conj(reference) x transform of the patch, (B, N, N, N/2+1), and the product of their norms."""
    H, h = N // 2 + 1, N // 2
    z, y, x = _grid(N, 0)
    vols, p = vols.double(), prior.double().view(-1, 3, 1, 1, 1)
    patch = _sample(vols, z + p[:, 2], y + p[:, 1], x + p[:, 0])
    for b in range(vols.shape[0]):
        for d, s in enumerate((p[b, 2].item(), p[b, 1].item(), p[b, 0].item())):
            if abs(s) != math.floor(abs(s)):
                patch[b].select(d, math.floor(abs(s)) if s < 0 else N - math.ceil(abs(s))).zero_()
    cz, cy, cx = _grid(N, h)
    r = (cz * cz + cy * cy + cx * cx).sqrt()
    fill = torch.where(r > h + 5.0, 1.0, torch.where(r >= h, 0.5 + 0.5 * torch.cos(math.pi * (h + 5.0 - r) / 5.0), 0.0))
    avg = (patch * fill).sum((1, 2, 3), keepdim=True) / fill.sum()
    patch = torch.roll((1 - fill) * patch + fill * avg, (-h, -h, -h), (1, 2, 3))
    tgt = torch.fft.rfftn(patch, dim=(1, 2, 3), norm="forward")
    k = torch.arange(N, device=DEV, dtype=torch.float64)
    k = torch.where(k < h, k, k - N)
    kx = torch.arange(H, device=DEV, dtype=torch.float64)
    ball = k[:, None, None] ** 2 + k[:, None] ** 2 + torch.where(kx < h, kx, kx - H) ** 2 <= h * h
    pts = torch.stack(torch.meshgrid(k, k, kx, indexing="ij")[::-1])  # (x, y, z)
    # index N/2 stands for -N/2 in z and y
    w = (M.double() @ pts.flatten(1)).view(-1, 3, N, N, H) + h
    src = _sample(ref[None].expand(vols.shape[0], -1, -1, -1), w[:, 2], w[:, 1], w[:, 0]) * ball
    if ctf is not None:
        src = src * ctf.double()
    return src.conj() * tgt, src.flatten(1).norm(dim=1) * tgt.flatten(1).norm(dim=1)


def _exact_shift(case, seed):
    s, N, uf = _inputs(case, seed), case["N"], case["uf"]
    M = _matrix(s["tracker"]).mT
    ref = _reference(N)
    U = uf * (2 * case["r"] + 1)
    u = (torch.arange(U, device=DEV, dtype=torch.float64) - U // 2) / uf
    E = [torch.exp(2j * math.pi * u[:, None] * torch.fft.fftfreq(n, device=DEV, dtype=torch.float64))
         for n in (N, N // 2 + 1)]
    shifts, scores, step = [], [], max(1, (1 << 22) // N ** 3)
    for i in range(0, case["B"], step):
        j = slice(i, i + step)
        P, den = _products(ref, s["volumes"][j], s["shift"][j], M[j], None if s["ctf"] is None else s["ctf"][j], N)
        for b in range(P.shape[0]):
            q = torch.tensordot(E[0], P[b], 1)                       # u0, m1, m2
            q = torch.einsum("vm,umk->uvk", E[0], q)
            v = (q @ E[1].T).real
            at = int(v.argmax())
            scores.append(v.flatten()[at] / den[b])
            shifts.append([u[at % U], u[at // U % U], u[at // (U * U)]])
    return torch.tensor(shifts, device=DEV, dtype=torch.float64), torch.stack(scores)


def _exact_gradient(case, seed):
    s, N, L, B = _inputs(case, seed), case["N"], case["L"], case["B"]
    coef, tmpl = _expansion(s["volumes"], L), _expansion(_template(N)[None], L)
    omega = s["omega"].clone().requires_grad_(True)
    rows = {l: _rows(tmpl, l)[0].requires_grad_(True) for l in range(L + 1)}
    f = 0.0
    for l in range(L + 1):
        V = _rows(coef, l)
        turn = torch.linalg.matrix_exp(sum(omega[:, k, None, None] * A for k, A in enumerate(_generators(l))))
        f = f + ((_wigner(l, s["base"]) @ turn) * _correlate(rows[l], V, l)).real.sum()
    shift = s["shift"].double().requires_grad_(True)
    ref, step = _reference(N), max(1, (1 << 22) // N ** 3)
    kz, kx = (torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) for n in (N, N // 2 + 1))
    total, gshift = f.detach(), torch.zeros_like(s["shift"], dtype=torch.float64)
    for i in range(0, B, step):
        j = slice(i, i + step)
        P, den = _products(ref, s["volumes"][j], s["zero"][j], s["rot"][j].view(-1, 3, 3), None, N)
        e = [torch.exp(2j * math.pi * shift[j, d, None] * k) for d, k in ((0, kx), (1, kz), (2, kz))]
        c = (torch.einsum("bzyx,bx,by,bz->b", P, *e).real / den).sum()
        gshift += torch.autograd.grad(c, shift)[0]
        total = total + c.detach()
    grads = torch.autograd.grad(f, [omega] + list(rows.values()))
    table = _spectrum(L)
    gt = torch.zeros(len(table) + 1, device=DEV, dtype=torch.complex128)
    for l in range(L + 1):
        at = [(n, m + l, k - 1) for n, (_, d, k, m) in enumerate(table) if d == l]
        n, row, k = (torch.tensor(t, device=DEV) for t in zip(*at))
        gt[n] = grads[1 + l][row, k]
    return {"total": total, "omega": grads[0], "template": gt, "shift": gshift}


def exact(case, seed):
    """None for the search and the whole alternation: their accepted Newton steps are a chain of
    comparisons, which has no 64-bit value of its own."""
    make = {"expand": _exact_expand, "prepare": _exact_prepare, "shift": _exact_shift,
            "gradient": _exact_gradient}.get(case["kind"])
    return None if make is None else make(case, seed)
