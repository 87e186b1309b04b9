"""Error of a codebook plan's gradients against 64 bits.  The split of the inner
dimension bounds the FP32 chains of the products, and with them the error that
comes on top of the three-product split's (about 1.5e-6 for dW)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = float(torch.finfo(torch.float32).eps)


def _exact(W, phi, Hd, Ha, Hr):
    W, phi = W.to(torch.complex128).requires_grad_(), phi.double().requires_grad_()
    Hd, Ha, Hr = (x.to(torch.complex128) for x in (Hd, Ha, Hr))
    e = torch.polar(torch.ones_like(phi), torch.remainder(phi, float(torch.tensor(2 * math.pi))))
    Y = W @ Hd + ((W @ Ha) * e) @ Hr
    cap = torch.log2(1 + (Y.abs() + EPS) ** 2 / 1e-9)
    top = cap.max(0).values
    loss = torch.linalg.vector_norm(cap * (cap != top).double()) - top.sum()
    return torch.autograd.grad(loss, [W, phi])


# chains of 8 k-blocks gave 1.9e-6, of 10 2.15e-6, of 13 2.3e-6
@pytest.mark.parametrize("C,S,M,R,most", [(60, 16, 1024, 4096, 2.0e-6)])
def test_gradient_error(C, S, M, R, most):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    off = []
    for seed in (1, 2, 3):
        g = torch.Generator(device="cuda").manual_seed(seed + R)
        mk = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda",  # noqa: E731
                                    generator=g) * 1e-3
        Hd, Ha, Hr, W = mk(S, R), mk(S, M), mk(M, R), mk(C, S) * 1e3
        phi = torch.rand(M, device="cuda", generator=g) * 9
        ref = _exact(W, phi, Hd, Ha, Hr)
        plan = objective.ObjectivePlan(Hd, Ha, Hr, c_max=C)
        W.requires_grad_()
        phi.requires_grad_()
        loss = objective.capacity_objective(W, Hd, Ha, Hr, phi, 2 * math.pi, 1.0, plan=plan)
        got = torch.autograd.grad(loss, [W, phi])
        plan.close()
        off.append([float((x.to(y.dtype) - y).norm() / y.norm()) for x, y in zip(got, ref)])
    assert sum(x[0] for x in off) / 3 <= most, off
    assert sum(x[1] for x in off) / 3 <= 4 * most, off
