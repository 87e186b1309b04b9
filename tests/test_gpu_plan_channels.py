"""A plan evaluates the H_d and H_r that it was made of: writing into the arrays
afterwards changes nothing, whichever form the plan took (one or two codes with an
even or an odd number of Rx, long columns, a codebook)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,M,R,C", [
    (4, 60, 512, 1), (4, 60, 511, 1), (5, 33, 96, 2), (5, 33, 97, 2), (16, 3300, 64, 1),
    (8, 2200, 64, 2), (4, 60, 512, 5),
])
def test_channels_written_after_the_plan(S, M, R, C):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    g = torch.Generator(device="cuda").manual_seed(S + M + R)
    mk = lambda s, *d: torch.randn(*d, generator=g, dtype=torch.complex64,  # noqa: E731
                                   device="cuda") * s
    Hd, Ha, Hr, W = mk(1e-4, S, R), mk(1e-2, S, M), mk(1e-3, M, R), mk(1.0, C, S)
    phi = (torch.rand(M, generator=g, device="cuda") * 6).requires_grad_()
    W.requires_grad_()
    plan = objective.ObjectivePlan(Hd, Ha, Hr, c_max=C)

    def step():
        loss, amp = objective.capacity_objective(W, Hd, Ha, Hr, phi, 2 * math.pi, 1.0,
                                                 return_recv=True, plan=plan)
        return [loss.detach(), amp] + list(torch.autograd.grad(loss, [W, phi]))

    before = step()
    assert float(before[1].abs().sum()) > 0
    Hd.zero_()
    Hr.mul_(-3.0)
    # the kernels add in a fixed order: the same bits
    for x, y in zip(before, step()):
        assert torch.equal(x, y)
    plan.close()
