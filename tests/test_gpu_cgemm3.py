"""The tensor-core plan's products against FP64 where their split changes: fewer
Rx than a tile, an odd number of tiles (the second CTA of the last pair has
none), tiles that end inside a k-block plane, several items a CTA, one k-block."""
import math

import numpy as np
import pytest
import torch

import objective_oracle as OO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,M,R,C", [
    (1, 1, 1, 3), (3, 5, 33, 64), (7, 57, 64, 5), (16, 130, 70, 17), (16, 500, 1300, 33),
    (36, 1100, 2116, 30), (4, 28, 30000, 60), (5, 60, 26000, 8), (16, 2300, 130, 64),
])
def test_against_fp64(S, M, R, C):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    rng = np.random.default_rng(S + M + R)
    mk = lambda s, *d: ((rng.normal(size=d) + 1j * rng.normal(size=d)) * s).astype(  # noqa: E731
        np.complex64)
    Hd, Ha, Hr, W = mk(1e-4, S, R), mk(1e-2, S, M), mk(1e-3, M, R), mk(1.0, C, S)
    phi = rng.uniform(0, 6.0, M).astype(np.float32)
    drop = np.zeros(C, bool)
    drop[C // 2] = True
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    plan = objective.ObjectivePlan(dev(Hd), dev(Ha), dev(Hr), c_max=C)
    w, p = dev(W).requires_grad_(), dev(phi).requires_grad_()
    for _ in range(2):
        loss, amp = objective.capacity_objective(w, dev(Hd), dev(Ha), dev(Hr), p, 2 * math.pi, 0.5,
                                                 dev(drop), return_recv=True, plan=plan)
        g = torch.autograd.grad(loss, [w, p])
    objective.check_status(plan)
    lo, gW, gp = OO.objective_from_weights(Hd, Ha, Hr, phi, W, 0.5, drop)
    U = (W.astype(np.complex128) @ Ha) * np.exp(1j * np.mod(phi.astype(np.float64),
                                                            np.float32(2 * math.pi)))
    Y = np.abs(W.astype(np.complex128) @ Hd + U @ Hr.astype(np.complex128))
    # three BF16 products: about 1e-5 (bounds of the plan's other tests)
    assert abs(float(loss.detach()) - lo) <= 1e-4 * abs(lo)
    assert np.abs(amp.cpu().numpy() - Y).max() <= 1e-4 * Y.max()
    for got, ref in zip(g, (gW, gp)):
        assert np.abs(got.cpu().numpy() - ref).max() <= 1e-3 * np.abs(ref).max()
    plan.close()
