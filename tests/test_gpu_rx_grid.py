"""Stage 1's Rx-grid rule against the oracle over the Rx sets that it takes and
those that it leaves to the hierarchy: every pair of axes, falling orders, one
row or column, jitter, rotation, boxes larger than the spheres, Tx in the plane
of the Rx."""
import numpy as np
import pytest
import torch

import cases
import oracle

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9
ROOM = (6.0, 5.0, 3.0)


def _grid(kind):
    """Rx positions [n0, n1, 3] and their half boxes."""
    rng = np.random.default_rng(11)
    half = 0.08
    lin = lambda a, b, n: np.linspace(a, b, n)  # noqa: E731
    u, v = np.meshgrid(lin(0.5, 5.5, 23), lin(0.5, 4.5, 17), indexing="ij")
    p = np.stack([u, v, np.full(u.shape, 1.2)], -1)
    if kind == "yx":
        p = np.stack([v, u * 0.8, np.full(u.shape, 1.2)], -1)
    elif kind == "xz":
        p = np.stack([u, np.full(u.shape, 3.0), v * 0.55], -1)
    elif kind == "zy":
        p = np.stack([np.full(u.shape, 4.0), v, u * 0.5], -1)
    elif kind == "falling":
        p = p[::-1, ::-1]
    elif kind == "row":
        p = p[:1]
    elif kind == "column":
        p = p[:, 4:5]
    elif kind == "same":      # a step of zero
        p = np.broadcast_to(p[3:4], (5,) + p.shape[1:])
    elif kind == "jitter":
        p = p + rng.uniform(-0.03, 0.03, p.shape)
    elif kind == "scatter":
        p = p + rng.uniform(-0.4, 0.4, p.shape)
    elif kind == "rotated":
        c, s = np.cos(0.5), np.sin(0.5)
        q = p - [3, 2.5, 0]
        p = np.stack([c * q[..., 0] - s * q[..., 1], s * q[..., 0] + c * q[..., 1], q[..., 2]],
                     -1) * [0.7, 0.7, 1] + [3, 2.5, 0]
    elif kind == "tilted":
        p = p + (u * 0.1)[..., None] * [0, 0, 1]
    elif kind == "boxes":
        half = 0.2
    elif kind == "dense":     # 32 x 32 elements, as a metasurface
        k = (np.arange(32) - 15.5) * LAM / 2
        p = np.stack(np.broadcast_arrays(3.0 + k[:, None], 4.99, 1.5 + k[None]), -1)
    return np.ascontiguousarray(p.astype(np.float32)), half


KINDS = ("xy", "yx", "xz", "zy", "falling", "row", "column", "same", "jitter", "scatter",
         "rotated", "tilted", "boxes", "dense", "in-plane")


@pytest.mark.parametrize("kind", KINDS)
def test_rx_sets(kind):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import scenes, tracer
    tris, mat, prop = scenes.shoebox_scene(5, room=ROOM, box_tess=1, seed=2,
                                           keep_clear=[(3.0, 1.0, 2.0), (3.0, 1.0, 1.2)])
    dst, half = _grid(kind)
    src = scenes.ula((3.0, 1.0, 1.2 if kind == "in-plane" else 2.0), (1, 0, 0), 3, LAM / 2)
    box = np.concatenate([dst - np.float32(half), dst + np.float32(half)], -1).reshape(-1, 6)
    p = dict(samples_per_launch=1, launch_x=120, launch_y=72, wave_len=LAM, max_reflection=2,
             reserve_size=100, src_bptype=0, dst_bptype=0, dst_gridsize=3, src_r=0.5e-5,
             dst_r=0.08, src_dir=[0., 1., 0.], dst_dir=[0., 0., 0.])
    sc = tracer.Scene(tris, mat, prop)
    res, st = sc.trace(src, dst, p, dst_aabb=box)
    paths = sc.export_paths()
    sc.close()
    H = (res[..., 0] + 1j * res[..., 1]).cpu().numpy()
    Ho, so, po = oracle.trace_channel(tris, mat, prop, src, dst, p, dst_box=box)
    for k in cases.STAT_KEYS + ("tasks", "overflow"):
        assert st[k] == so[k], (k, st[k], so[k])
    assert st["fwd_records"] > 0
    assert np.array_equal(paths, po)
    assert np.array_equal(H != 0, Ho != 0)
    # the same rays; sin and cos of the phase differ in their last bits
    assert np.linalg.norm(H - Ho) <= 1e-5 * np.linalg.norm(Ho)
