"""Rounding of the one-call evaluation over several metasurfaces: its sums over
all sources of a level are no further off than the path-by-path products, whose
FP32 chains end with every path.  Equal real channels between the metasurfaces
make a chain's errors add up to one side, the same for every element."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(4, 600), (8, 300), (2, 1000)])
def test_no_further_off_than_by_path(n, m):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import objective
    S, C, R = 4, 3, 64
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=g, dtype=torch.complex64,  # noqa: E731
                                 device="cuda")
    flat = lambda v, *s: torch.full(s, v, dtype=torch.complex64, device="cuda")  # noqa: E731
    off = {"one call": [], "by path": []}
    for scale in (0.61, 0.7, 0.83, 0.97, 1.13):
        ch = {"src_to_dst": rnd(S, R) * 1e-9}
        for i in range(n):
            ch["src_to_ms{%d}" % i] = flat(scale, S, m)
            ch["ms{%d}_to_dst" % i] = rnd(m, R) * 1e-3
            for j in range(i + 1, n):
                ch["ms{%d}_to_ms{%d}" % (i, j)] = flat(0.9 * scale, m, m)
        W = torch.rand(C, S, generator=g, device="cuda").to(torch.complex64)
        phi = torch.zeros(n * m, device="cuda")
        wide = {k: v.to(torch.complex128) for k, v in ch.items()}
        V = [W.to(torch.complex128) @ wide["src_to_ms{%d}" % i] for i in range(n)]
        V2 = [sum(V[j] @ (wide["ms{%d}_to_ms{%d}" % (j, i)] if j < i else
                          wide["ms{%d}_to_ms{%d}" % (i, j)].T) for j in range(n) if j != i)
              for i in range(n)]
        Y = W.to(torch.complex128) @ wide["src_to_dst"] + sum(
            (V[i] + V2[i]) @ wide["ms{%d}_to_dst" % i] for i in range(n))
        plan = objective.StackedPlan(ch["src_to_dst"],
                                     [ch["ms{%d}_to_dst" % i] for i in range(n)], C)
        for name, fn, last in (("one call", objective.FusedMultiHop, 2),
                               ("by path", objective.MultiHopObjective,
                                objective.ms_paths(n, 2))):
            with torch.no_grad():
                _, amp = fn.apply(W, phi, plan, ch, [2 * math.pi] * n, last, 1.0, None, True)
            off[name].append(float((amp.double() - Y.abs()).norm() / Y.abs().norm()))
        plan.close()
    assert max(off["by path"]) < 1e-4, off
    # (the products that follow are the same in both: 3e-6)
    assert max(off["one call"]) <= 1.05 * max(off["by path"]), off
