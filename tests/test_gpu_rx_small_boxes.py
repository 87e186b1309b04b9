"""Rx whose boxes do not hold all of their spheres: a hit then lies outside the box
that let the ray in, and which of two close Rx a ray meets is decided by the order of
the hierarchy.  A grid of such Rx goes by the hierarchy as well: the same Rx in a
mixed order, which are no grid, get the same rays (every Rx is a cell of its own)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9


# the sphere's distance of acceptance is 7.07 mm at least
@pytest.mark.parametrize("radius,half", [(0.1, 0.05), (0.1, 0.08), (0.02, 0.01), (0.003, None),
                                         (0.005, None)])
@pytest.mark.parametrize("step", [(0.011, 0.009), (0.0025, 0.0025)])
def test_grid_equals_mixed_order(radius, half, step):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import scenes, tracer
    tris, mat, prop = scenes.shoebox_scene(4, room=(6.0, 5.0, 3.0), box_tess=1, seed=3,
                                           keep_clear=[(3.0, 1.0, 2.0), (3.1, 1.6, 1.3)])
    n0, n1 = 23, 17
    dst = np.stack(np.meshgrid(3.0 + np.arange(n0) * step[0], 1.2 + np.arange(n1) * step[1],
                               indexing="ij"), -1)
    dst = np.stack([dst[..., 0], np.full((n0, n1), 1.4), dst[..., 1]], -1).astype(np.float32)
    mixed = np.random.default_rng(5).permutation(dst.reshape(-1, 3)).reshape(dst.shape)
    src = (np.array([3.0, 1.0, 2.0]) + np.random.default_rng(1).uniform(-0.3, 0.3, (1, 12, 3)))
    p = dict(samples_per_launch=2, launch_x=170, launch_y=170, wave_len=LAM, max_reflection=1,
             reserve_size=256, src_bptype=0, dst_bptype=0, dst_gridsize=1, src_r=0.5e-5,
             dst_r=radius, src_dir=[0., 1., 0.], dst_dir=[0., 0., 0.])
    got = []
    for d in (dst, np.ascontiguousarray(mixed)):
        box = None
        if half is not None:
            box = np.concatenate([d - np.float32(half), d + np.float32(half)], -1).reshape(-1, 6)
        sc = tracer.Scene(tris, mat, prop)
        _, st = sc.trace(src.astype(np.float32), d, p, dst_aabb=box)
        got.append(([st[k] for k in ("fwd_records", "unique_records", "unique_paths",
                                     "segments_fwd")], sc.export_paths()))
        sc.close()
    assert got[0][0][0] > 0
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
