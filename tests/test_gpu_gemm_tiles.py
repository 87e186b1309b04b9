"""The tensor-core GEMM at each of its tile widths, and the network's passes at
batches that end inside a tile and into rows that are not 16-byte aligned."""
import ctypes as C

import numpy as np
import pytest
import torch

import mlp_oracle

pytestmark = pytest.mark.gpu


# half the SMs of a GB300 is 76 tiles: 128 x 128 from 76 of those on, then
# 128 x 64 from 76 of those on, else 128 x 32
@pytest.mark.parametrize("M,N,K", [(128, 64, 64), (128, 192, 576), (1280, 448, 64),
                                   (1280, 512, 128), (2048, 320, 192), (1280, 1024, 64)])
def test_tile_widths(M, N, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import surrogate
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    out = surrogate.gemm_bf16(A, B).double()
    a, b = A.double(), B.double()
    # products of bf16 are exact in FP32; K sums, each off by at most one unit
    # in the last place of the largest partial sum
    bound = K * 2.0 ** -23 * (a.abs() @ b.abs().T)
    assert bool(((out - a @ b.T).abs() <= bound).all())


@pytest.mark.parametrize("B", (1, 31, 128, 129, 700))
def test_batches_that_end_inside_a_tile(B):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import _lib, surrogate
    dims = [40, 256, 128, 384]
    net = surrogate.MLP(dims, max_batch=1024, seed=4)
    rng = np.random.default_rng(B)
    X = rng.normal(size=(B, dims[0])).astype(np.float32)
    T = rng.normal(size=(B, dims[-1])).astype(np.float32)
    p = net.get_params().cpu().numpy()
    # a larger batch before: what it left beyond row B must not count
    net.gradients(torch.ones(900, dims[0]), torch.ones(900, dims[-1]))
    loss, grad = net.gradients(torch.as_tensor(X), torch.as_tensor(T))
    lo, go = mlp_oracle.loss_and_grads(p, dims, X.astype(np.float64), T.astype(np.float64))
    # the oracle rounds where the network does; a value within FP32 rounding of
    # a bf16 midpoint may fall to the other side (2^-8 of it), seldom
    np.testing.assert_allclose(float(loss), lo, rtol=1e-4)
    assert np.linalg.norm(grad.cpu().numpy() - go) <= 2e-2 * np.linalg.norm(go)
    Y = net(torch.as_tensor(X))
    Xd = torch.as_tensor(X).cuda()
    off = torch.full((B * dims[-1] + 1,), -7.0, device="cuda")  # rows 4 bytes off
    _lib.call("ams_mlp_forward", net._h, C.c_void_p(Xd.data_ptr()), B,
              C.c_void_p(off.data_ptr() + 4), C.c_void_p(0))
    assert torch.equal(off[1:].view(B, -1), Y) and float(off[0]) == -7.0
    net.close()
