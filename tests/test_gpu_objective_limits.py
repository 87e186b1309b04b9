"""One and two codes where a call changes kernels: the last K = M + S that the
clustered streaming kernel takes and the first that it does not (3,200 and 3,201
for one code, 3,072 and 3,073 for two), the last that a plan streams at all (4,096
and 2,048 where the clustered kernel does not take it), and an odd number of Rx,
which a plan streams over its transposed copy at every height of its tiles."""
import math

import numpy as np
import pytest
import torch

import objective_oracle as OO

pytestmark = pytest.mark.gpu

SHAPES = [  # S, M, R, C
    (16, 3184, 40, 1), (16, 3185, 40, 1), (16, 3056, 40, 2), (16, 3057, 40, 2),
    (16, 4080, 36, 1), (16, 4081, 36, 1),
    (16, 500, 41, 1), (16, 1000, 41, 1), (16, 2000, 41, 1), (16, 3500, 41, 1), (16, 4081, 41, 1),
    (16, 400, 41, 2), (16, 900, 41, 2), (16, 1600, 41, 2), (16, 2032, 41, 2), (16, 2033, 41, 2),
]


@pytest.mark.parametrize("S,M,R,C", SHAPES)
@pytest.mark.parametrize("plan", (False, True))
def test_against_fp64(S, M, R, C, plan):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    rng = np.random.default_rng(S + M + R)
    mk = lambda *s: ((rng.normal(size=s) + 1j * rng.normal(size=s)) * 1e-4).astype(  # noqa: E731
        np.complex64)
    Hd, Ha, Hr, W = mk(S, R), mk(S, M), mk(M, R), mk(C, S) * 1e4
    phi = rng.uniform(0, 9.0, M).astype(np.float32)
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    w, ph = dev(W).requires_grad_(), dev(phi).requires_grad_()
    hd, ha, hr = dev(Hd), dev(Ha), dev(Hr)
    pl = objective.ObjectivePlan(hd, ha, hr, c_max=C) if plan else None
    loss, amp = objective.capacity_objective(w, hd, ha, hr, ph, 2 * math.pi, 0.5, None,
                                             return_recv=True, plan=pl)
    g = torch.autograd.grad(loss, [w, ph])
    objective.check_status(pl)
    lo, gW, gp = OO.objective_from_weights(Hd, Ha, Hr, phi, W, 0.5, None)
    U = (W.astype(np.complex128) @ Ha) * np.exp(1j * np.mod(phi.astype(np.float64),
                                                            np.float32(2 * math.pi)))
    Y = np.abs(W.astype(np.complex128) @ Hd.astype(np.complex128) + U @ Hr.astype(np.complex128))
    # FP32 sums of up to n terms, n units in the last place of their scale; beyond
    # its streaming kernels a plan takes three BF16 products (about 1e-5)
    ulp, tc = 2.0 ** -23, 2e-5 * plan
    assert abs(float(loss.detach()) - lo) <= (64 * ulp + tc) * abs(lo)
    assert np.abs(amp.cpu().numpy() - Y).max() <= ((M + S) * ulp + tc) * Y.max()
    for got, ref in zip(g, (gW, gp)):
        assert np.abs(got.cpu().numpy() - ref).max() <= ((M + S + R) * ulp + tc) * np.abs(ref).max()
