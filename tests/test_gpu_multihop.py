"""The one-call evaluation over several metasurfaces against autograd in
complex128 and the path-by-path one, where its tiles (32 codes, 16 elements, 64
inner terms) end: one element, one past a tile, eight metasurfaces, one to four
hops."""
import math

import numpy as np
import pytest
import torch

import objective_oracle as OO

pytestmark = pytest.mark.gpu

CASES = [  # S, sizes, hops, C, R
    (1, (1, 1), 2, 1, 40), (36, (16, 17), 2, 30, 130), (65, (63, 65), 3, 33, 200),
    (8, (40, 24, 33), 4, 64, 90), (5, (129, 7, 1), 1, 5, 70), (9, (3,) * 8, 2, 12, 64),
    (16, (576, 256), 2, 32, 300),
]


def _loss64(ch, W, phi, sizes, hops, w, drop):
    n, off = len(sizes), np.concatenate([[0], np.cumsum(sizes)])
    e = [torch.exp(1j * torch.remainder(phi[off[i]:off[i + 1]], 2 * math.pi)) for i in range(n)]
    mm = lambda a, b: ch["ms{%d}_to_ms{%d}" % (a, b)] if a < b else (  # noqa: E731
        ch["ms{%d}_to_ms{%d}" % (b, a)].T)
    V = [(W @ ch["src_to_ms{%d}" % i]) * e[i] for i in range(n)]
    Y = W @ ch["src_to_dst"]
    for _ in range(hops):
        for i in range(n):
            Y = Y + V[i] @ ch["ms{%d}_to_dst" % i]
        V = [sum(V[j] @ mm(j, i) for j in range(n) if j != i) * e[i] for i in range(n)]
    cap = torch.log2(1.0 + (Y.abs() + OO.EPS32) ** 2 / OO.N0) * (~drop)[:, None]
    mx, _ = cap.max(0)
    return -w * mx.sum() + torch.linalg.norm(cap * (cap != mx[None, :])), Y.abs()


@pytest.mark.parametrize("S,sizes,hops,C,R", CASES)
def test_against_fp64(S, sizes, hops, C, R):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    n, M = len(sizes), sum(sizes)
    rng = np.random.default_rng(S + M + R)
    mk = lambda s, *d: torch.as_tensor(  # noqa: E731
        ((rng.normal(size=d) + 1j * rng.normal(size=d)) * s).astype(np.complex64))
    ch = {"src_to_dst": mk(1e-4, S, R)}
    for i in range(n):
        ch["src_to_ms{%d}" % i] = mk(1e-2, S, sizes[i])
        ch["ms{%d}_to_dst" % i] = mk(1e-3, sizes[i], R)
        for j in range(i + 1, n):
            ch["ms{%d}_to_ms{%d}" % (i, j)] = mk(0.5 / math.sqrt(sizes[i] * n), sizes[i], sizes[j])
    W, phi = mk(1.0, C, S), torch.as_tensor(rng.uniform(0, 9, M).astype(np.float32))
    drop = torch.zeros(C, dtype=torch.bool)
    drop[C // 2] = C > 1
    w64 = W.to(torch.complex128).requires_grad_()
    p64 = phi.double().requires_grad_()
    # the phases wrap at the float32 value of 2 pi on the device: 2e-7 away
    lo, amp64 = _loss64({k: v.to(torch.complex128) for k, v in ch.items()}, w64, p64, sizes, hops,
                        0.5, drop)
    g64 = torch.autograd.grad(lo, [w64, p64])
    dch = {k: v.cuda() for k, v in ch.items()}
    plan = objective.StackedPlan(dch["src_to_dst"],
                                 [dch["ms{%d}_to_dst" % i] for i in range(n)], C)
    for fn, last in ((objective.FusedMultiHop, hops),
                     (objective.MultiHopObjective, objective.ms_paths(n, hops))):
        w, p = W.cuda().requires_grad_(), phi.cuda().requires_grad_()
        loss, amp = fn.apply(w, p, plan, dch, [2 * math.pi] * n, last, 0.5, drop, True)
        g = torch.autograd.grad(loss, [w, p])
        objective.check_status(plan)
        # bounds of the stacked tensor-core evaluation (products about 1e-5)
        np.testing.assert_allclose(float(loss.detach()), float(lo.detach()), rtol=1e-4)
        a = amp64.detach().numpy()
        assert np.abs(amp.cpu().numpy() - a).max() <= 1e-4 * a.max()
        for got, ref in zip(g, g64):
            ref = ref.numpy()
            assert np.abs(got.cpu().numpy() - ref).max() <= 1e-3 * np.abs(ref).max()
    plan.close()


def test_refuses_what_does_not_fit():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    z = lambda *s: torch.zeros(*s, dtype=torch.complex64, device="cuda")  # noqa: E731
    ch = {"src_to_dst": z(2, 8), "src_to_ms{0}": z(2, 3), "src_to_ms{1}": z(2, 4),
          "ms{0}_to_dst": z(3, 8), "ms{1}_to_dst": z(4, 8), "ms{0}_to_ms{1}": z(4, 3)}
    plan = objective.StackedPlan(ch["src_to_dst"], [ch["ms{0}_to_dst"], ch["ms{1}_to_dst"]], 2)
    run = lambda c: objective.FusedMultiHop.apply(  # noqa: E731
        torch.ones(2, 2, dtype=torch.complex64, device="cuda"), torch.zeros(7, device="cuda"),
        plan, c, [1.0, 1.0], 2, 1.0, None, True)
    with pytest.raises(ValueError):
        run(ch)
    run(dict(ch, **{"ms{0}_to_ms{1}": z(3, 4)}))
    plan.close()
