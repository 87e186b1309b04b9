"""Objective calls of one or two codes on CTAs that work alone (no cluster): one Rx
or an exact tile of them, fewer tiles than CTAs and several a CTA, with and without
a metasurface, against FP64; and a NaN among the channels shows in the loss."""
import math

import numpy as np
import pytest
import torch

import objective_oracle as OO

pytestmark = pytest.mark.gpu


def _run(S, M, R, C, plan, nan=False):
    from automs_gb300 import objective
    rng = np.random.default_rng(S + M + R)
    mk = lambda s, *d: ((rng.normal(size=d) + 1j * rng.normal(size=d)) * s).astype(  # noqa: E731
        np.complex64)
    Hd, Ha, Hr, W = mk(1e-4, S, R), mk(1e-2, S, M), mk(1e-3, M, R), mk(1.0, C, S)
    phi = rng.uniform(0, 6.0, M).astype(np.float32)
    if nan:
        Hd[0, R // 2] = np.nan
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    p = objective.ObjectivePlan(dev(Hd), dev(Ha), dev(Hr), c_max=C) if plan else None
    w, f = dev(W).requires_grad_(), dev(phi).requires_grad_()
    loss, amp = objective.capacity_objective(
        w, dev(Hd), dev(Ha) if M else None, dev(Hr) if M else None, f if M else None, 2 * math.pi,
        0.5, None, return_recv=True, plan=p)
    g = torch.autograd.grad(loss, [w] + ([f] if M else []))
    objective.check_status(p)
    return Hd, Ha, Hr, phi, W, float(loss.detach()), amp.cpu().numpy(), [x.cpu().numpy() for x in g]


@pytest.mark.parametrize("plan", (False, True))
@pytest.mark.parametrize("S,M,R,C", [
    (1, 1, 2, 1), (4, 16, 16, 1), (4, 16, 18, 2), (16, 64, 1024, 1), (36, 0, 1200, 2),
    (9, 100, 8000, 2), (16, 200, 20000, 1),
])
def test_against_fp64(S, M, R, C, plan):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if plan and M == 0:
        pytest.skip("a plan needs a metasurface")
    Hd, Ha, Hr, phi, W, loss, amp, g = _run(S, M, R, C, plan)
    lo, gW, gp = OO.objective_from_weights(Hd, Ha if M else None, Hr if M else None,
                                           phi if M else None, W, 0.5, None)
    U = (W.astype(np.complex128) @ Ha) * np.exp(1j * np.mod(phi.astype(np.float64),
                                                            np.float32(2 * math.pi)))
    Y = np.abs(W.astype(np.complex128) @ Hd + U @ Hr.astype(np.complex128))
    # FP32 sums of up to 216 terms
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    assert np.abs(amp - Y).max() <= 2e-5 * Y.max()
    for got, ref in zip(g, (gW, gp)):
        assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("C", (1, 2))
def test_nan_shows(C):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert math.isnan(_run(4, 16, 64, C, False, nan=True)[5])
