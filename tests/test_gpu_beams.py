"""Stage-2 beams against the oracle where their rules change over: the sizes
at which the 32-wide hierarchy gets its next node or level, and Tx arrays whose
rays pass through other Tx spheres (the rays go on behind them) or for which
the array has no thin direction."""
import numpy as np
import pytest
import torch

import cases
import oracle

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9


def _soup(n, seed):
    """n triangles in a 6 x 5 x 3 m room, the first two the floor; a fifth of
    the materials lets rays through."""
    rng = np.random.default_rng(seed)
    c = rng.uniform([0.3, 0.3, 0.2], [5.7, 4.7, 2.8], (n, 1, 3))
    t = c + rng.uniform(-0.4, 0.4, (n, 3, 3))
    # half of them axis-aligned, as walls and furniture are
    ax = rng.integers(0, 3, n)
    for i in range(0, n, 2):
        t[i, :, ax[i]] = t[i, 0, ax[i]]
    t[0] = [[-1, -1, 0], [7, -1, 0], [7, 6, 0]]
    if n > 1:
        t[1] = [[-1, -1, 0], [7, 6, 0], [-1, 6, 0]]
    prop = np.repeat(rng.uniform(0.3, 0.7, 5)[:, None], 19, 1)
    prop[4] *= -1.0
    return (t.astype(np.float32), rng.integers(0, 5, n).astype(np.int32),
            prop.astype(np.float32))


def _tx(kind):
    at = np.array([3.0, 1.0, 1.5])
    rng = np.random.default_rng(3)
    if kind == "one":
        p = at[None]
    elif kind == "line":        # towards the Rx row
        p = at + np.arange(40)[:, None] * np.array([LAM / 2, 0.0, 0.0])
    elif kind == "plane":       # the Rx row lies in its plane
        k = np.arange(35)
        p = at + np.stack([(k % 7) * LAM / 2, (k // 7) * LAM / 2, 0 * k], 1)
    elif kind == "cluster":
        p = at + rng.uniform(-0.02, 0.02, (33, 3))
    else:                       # two Tx in one place
        p = at + np.array([[0, 0, 0], [0, 0, 0], [LAM / 2, 0, 0]])
    return p.astype(np.float32)[None]


def _check(n_tri, kind, refl, seed):
    from automs_gb300 import tracer
    tris, mat, prop = _soup(n_tri, seed)
    src = _tx(kind)
    # 3 x 11 Rx, the middle row on the line through the Tx along x
    x = np.linspace(3.6, 5.4, 11)
    dst = np.stack(np.meshgrid(np.array([0.9, 1.0, 1.1]), x, indexing="ij"), -1)
    dst = np.stack([dst[..., 1], dst[..., 0], np.full(dst.shape[:2], 1.5)], -1)
    dst = dst.astype(np.float32)
    p = dict(samples_per_launch=1, launch_x=160, launch_y=160, wave_len=LAM, max_reflection=refl,
             reserve_size=100, src_bptype=0, dst_bptype=0, dst_gridsize=2, src_r=0.5e-5,
             dst_r=0.1, src_dir=[0., 1., 0.], dst_dir=[0., 0., 0.])
    sc = tracer.Scene(tris, mat, prop)
    res, st = sc.trace(src, dst, p)
    paths = sc.export_paths()
    sc.close()
    H = (res[..., 0] + 1j * res[..., 1]).cpu().numpy()
    Ho, so, po = oracle.trace_channel(tris, mat, prop, src, dst, p)
    for k in cases.STAT_KEYS + ("tasks", "overflow"):
        assert st[k] == so[k], (k, st[k], so[k])
    assert np.array_equal(paths, po)
    assert np.array_equal(H != 0, Ho != 0)
    # the same rays; sin and cos of the phase differ in their last bits
    assert np.linalg.norm(H - Ho) <= 1e-5 * np.linalg.norm(Ho)
    return st


@pytest.mark.parametrize("n_tri", (1, 2, 31, 32, 33, 34, 1025, 2000))
def test_wide_hierarchy_sizes(n_tri):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert _check(n_tri, "plane", 2, n_tri)["rx_paths"] > 0


@pytest.mark.parametrize("kind", ("one", "line", "plane", "cluster", "twice"))
@pytest.mark.parametrize("refl", (0, 3))
def test_tx_arrays(kind, refl):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert _check(60, kind, refl, 5)["rx_paths"] > 0
