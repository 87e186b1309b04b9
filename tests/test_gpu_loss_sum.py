"""The loss over many Rx: its sums lose nothing however long they get.  All Rx have
the same channel, so that every capacity is the same float and a plain FP32 chain
of n of them is off by up to n / 2 roundings, always to the same side (1e-6 at 54).
The mean over the Rx has to be that of 32 of them."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# R: 54 groups of 32 Rx a CTA with four CTAs on each of 152 SMs; one and two codes:
# tiles of 16 Rx in at most 152 chains of two
SHAPES = [(8, 32 * 608 * 54), (60, 32 * 608 * 27), (1, 16 * 304 * 54), (2, 16 * 304 * 54)]


@pytest.mark.parametrize("plan", [True, False])
@pytest.mark.parametrize("C,R", SHAPES)
def test_mean_over_equal_rx(C, R, plan):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    if C > 8 and not plan:
        pytest.skip("the evaluation without a plan sums groups of 32 Rx by themselves")
    S, M = 2, 12
    g = torch.Generator(device="cuda").manual_seed(C)
    mk = lambda *d: torch.randn(*d, generator=g, dtype=torch.complex64,  # noqa: E731
                                device="cuda")
    Ha, W, hd, hr = mk(S, M) * 0.1, mk(C, S), mk(S, 1), mk(M, 1)
    phi = torch.rand(M, generator=g, device="cuda") * 6

    def means(scale, n):
        Hd, Hr = (x.mul(scale).expand(-1, n).contiguous() for x in (hd, hr))
        p = objective.ObjectivePlan(Hd, Ha, Hr, c_max=C) if plan else None
        # w = 0: the norm of the masked capacities, sqrt(n) times one Rx's
        with torch.no_grad():
            full = objective.capacity_objective(W, Hd, Ha, Hr, phi, 2 * math.pi, 1.0, plan=p)
            norm = objective.capacity_objective(W, Hd, Ha, Hr, phi, 2 * math.pi, 0.0, plan=p)
        full, norm = float(full), float(norm)
        if p is not None:
            p.close()
        return (norm - full) / n, norm / math.sqrt(n)

    for scale in (1e-4, 2.3e-4, 4.1e-4, 1e-3, 3.3e-3):
        (a, b), (x, y) = means(scale, 32), means(scale, R)
        # two losses of either side rounded to FP32 (2^-24 each), the norm being
        # up to sqrt(C) / sqrt(R) of the sum: 4 x 2^-24 of the mean, and the
        # subtraction's cancellation at n = 32, where both terms are of a size
        assert abs(x - a) <= 4 * 2.0**-24 * (abs(a) + b / math.sqrt(32))
        assert abs(y - b) <= 2 * 2.0**-24 * b
