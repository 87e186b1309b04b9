"""Rx sets that form no grid, whose hierarchy is visited in one loop with the
scene's: against the oracle with one, two and more Rx beside none, one, two and
more triangles (a set or a scene of one primitive has no nodes), and where some
launches meet neither."""
import numpy as np
import pytest
import torch

import cases
import oracle

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9


def _scene(n):
    rng = np.random.default_rng(n)
    floor = np.array([[[-2, -2, 0], [9, -2, 0], [9, 8, 0]], [[-2, -2, 0], [9, 8, 0], [-2, 8, 0]]])
    c = rng.uniform([0.5, 0.5, 0.2], [5.5, 4.5, 2.6], (60, 1, 3))
    t = np.concatenate([floor, c + rng.uniform(-0.5, 0.5, (60, 3, 3))])[:n]
    return (t.astype(np.float32), np.zeros(n, np.int32),
            np.full((1, 19), 0.6, np.float32))


@pytest.mark.parametrize("n_tri", (1, 2, 3, 62))
@pytest.mark.parametrize("shape", ((1, 1), (1, 2), (2, 2), (3, 7), (40, 53)))
def test_against_oracle(n_tri, shape):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import scenes, tracer
    tris, mat, prop = _scene(n_tri)
    rng = np.random.default_rng(shape[0])
    n = shape[0] * shape[1]
    a = np.stack(np.meshgrid(np.arange(shape[0]), np.arange(shape[1]), indexing="ij"), -1)
    a = (a + 0.5) / shape * [3.0, 2.4]
    c, s = np.cos(0.6), np.sin(0.6)  # turned in its plane, and a little rough
    dst = np.stack([2.4 + c * a[..., 0] - s * a[..., 1], 1.0 + s * a[..., 0] + c * a[..., 1],
                    1.1 + rng.uniform(-0.2, 0.2, shape)], -1).astype(np.float32)
    src = scenes.ula((3.0, 1.0, 2.0), (1, 0, 0), 2, LAM / 2)
    p = dict(samples_per_launch=1, launch_x=150, launch_y=150, wave_len=LAM, max_reflection=2,
             reserve_size=100, src_bptype=0, dst_bptype=0, dst_gridsize=3, src_r=0.5e-5,
             dst_r=0.3 if n < 30 else 0.06, src_dir=[0., 1., 0.], dst_dir=[0., 0., 0.])
    sc = tracer.Scene(tris, mat, prop)
    res, st = sc.trace(src, dst, p)
    paths = sc.export_paths()
    sc.close()
    H = (res[..., 0] + 1j * res[..., 1]).cpu().numpy()
    Ho, so, po = oracle.trace_channel(tris, mat, prop, src, dst, p)
    for k in cases.STAT_KEYS + ("tasks", "overflow"):
        assert st[k] == so[k], (k, st[k], so[k])
    assert st["fwd_records"] > 0
    assert np.array_equal(paths, po)
    assert np.array_equal(H != 0, Ho != 0)
    # the same rays; sin and cos of the phase differ in their last bits
    assert np.linalg.norm(H - Ho) <= 1e-5 * np.linalg.norm(Ho)
