"""The clustered streaming kernel against the FP64 oracle where its split
changes over (cluster of 1, 2, 4; tiles of 16 and 8 Rx; one and two rows a
thread; H_d rows that share a CTA with H_r rows or fill several; the first K
beyond it), at Rx counts that end inside a tile, direct and through a plan."""
import math

import numpy as np
import pytest
import torch

import objective_oracle as OO

pytestmark = pytest.mark.gpu

SHAPES = [  # S, M, R, C
    (1, 1, 2, 1), (1, 0, 16, 2), (16, 250, 18, 1), (16, 300, 14, 1), (16, 511, 4098, 2),
    (16, 600, 130, 1), (16, 1030, 64, 1), (16, 1130, 46, 1), (7, 1300, 1000, 2),
    (300, 40, 66, 1), (300, 700, 34, 2), (16, 2304, 98, 1), (16, 2400, 40, 2), (16, 2600, 40, 1),
    (36, 0, 5930, 1),
]


@pytest.mark.parametrize("S,M,R,C", SHAPES)
@pytest.mark.parametrize("plan", (False, True))
def test_against_fp64(S, M, R, C, plan):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if plan and M == 0:
        pytest.skip("a plan needs a metasurface")
    from automs_gb300 import objective
    rng = np.random.default_rng(S + M + R)
    mk = lambda *s: ((rng.normal(size=s) + 1j * rng.normal(size=s)) * 1e-4).astype(  # noqa: E731
        np.complex64)
    Hd, Ha, Hr = mk(S, R), (mk(S, M) if M else None), (mk(M, R) if M else None)
    phi = rng.uniform(0, 9.0, M).astype(np.float32) if M else None
    W = mk(C, S) * 1e4
    drop = np.zeros(C, bool)
    drop[C - 1] = C > 1
    dev = lambda x: None if x is None else torch.as_tensor(x, device="cuda")  # noqa: E731
    w = dev(W).requires_grad_()
    ph = dev(phi).requires_grad_() if M else None
    hd, ha, hr = dev(Hd), dev(Ha), dev(Hr)
    pl = objective.ObjectivePlan(hd, ha, hr, c_max=C) if plan else None
    for _ in range(2):  # the second call finds what the first one left
        loss, amp = objective.capacity_objective(w, hd, ha, hr, ph, 2 * math.pi, 0.5,
                                                 dev(drop) if C > 1 else None, return_recv=True,
                                                 plan=pl)
        g = torch.autograd.grad(loss, [w] + ([ph] if M else []))
    lo, gW, gp = OO.objective_from_weights(Hd, Ha, Hr, phi, W, 0.5, drop)
    Y = W.astype(np.complex128) @ Hd.astype(np.complex128)
    if M:
        U = (W.astype(np.complex128) @ Ha) * np.exp(1j * np.mod(phi.astype(np.float64),
                                                                np.float32(2 * math.pi)))
        Y = Y + U @ Hr.astype(np.complex128)
    # FP32 sums of up to n terms: n units in the last place of their scale
    ulp = 2.0 ** -23
    assert abs(float(loss.detach()) - lo) <= 64 * ulp * abs(lo)
    scale = np.abs(Y).max()
    assert np.abs(amp.cpu().numpy() - np.abs(Y)).max() <= (M + S) * ulp * scale
    tol = (M + S + R) * ulp
    assert np.abs(g[0].cpu().numpy() - gW).max() <= tol * np.abs(gW).max()
    if M:
        assert np.abs(g[1].cpu().numpy() - gp).max() <= tol * np.abs(gp).max()
