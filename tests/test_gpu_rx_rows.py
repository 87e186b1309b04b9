"""Rx rows that lie on one another, with the ones between moved out of the common
plane by less than a box: a ray meets the moved ones first from one side, so the
set is no grid although its corners make one."""
import numpy as np
import pytest
import torch

import cases
import oracle

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9


@pytest.mark.parametrize("along", (0, 1))
@pytest.mark.parametrize("shift", (-0.05, 0.05))
def test_moved_rows_of_no_step(along, shift):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import scenes, tracer
    tris, mat, prop = scenes.shoebox_scene(5, room=(6.0, 5.0, 3.0), box_tess=1, seed=2,
                                           keep_clear=[(3.0, 1.0, 2.0), (3.0, 1.0, 1.2)])
    half = np.float32(0.08)
    row = np.stack([np.full(17, 2.0), np.linspace(0.5, 4.5, 17), np.full(17, 1.2)], -1)
    dst = np.repeat(row[None], 3, 0)
    dst[1, :, 2] += shift
    if along:
        dst = dst.transpose(1, 0, 2)
    dst = np.ascontiguousarray(dst.astype(np.float32))
    src = scenes.ula((3.0, 1.0, 2.0), (1, 0, 0), 3, LAM / 2)
    box = np.concatenate([dst - half, dst + half], -1).reshape(-1, 6)
    p = dict(samples_per_launch=1, launch_x=240, launch_y=144, wave_len=LAM, max_reflection=2,
             reserve_size=100, src_bptype=0, dst_bptype=0, dst_gridsize=1, src_r=0.5e-5,
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
