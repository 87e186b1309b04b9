"""Memory that a trace can do without is not a reason to refuse it: the call goes
on as it would for a larger scene and gives the same channel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LAM = 3e8 / 60e9
COUNTS = ("rx_paths", "rx_fail", "fwd_records", "unique_records", "unique_paths", "rounds",
          "tasks", "overflow")


def _room():
    from automs_gb300 import scenes
    return scenes.shoebox_scene(6, room=(6.0, 5.0, 3.0), box_tess=2, seed=4,
                                keep_clear=[(3.0, 1.0, 2.0)])


def _params(refl):
    return dict(samples_per_launch=1, launch_x=160, launch_y=160, wave_len=LAM,
                max_reflection=refl, reserve_size=100, src_bptype=0, dst_bptype=0,
                dst_gridsize=5, src_r=0.5e-5, dst_r=0.06, src_dir=[0., 1., 0.],
                dst_dir=[0., 0., 0.])


def _ends():
    from automs_gb300 import scenes
    return (scenes.ula((3.0, 1.0, 2.0), (1, 0, 0), 3, LAM / 2),
            scenes.rx_grid(0.25, 5.75, 100, 0.25, 4.75, 100, 1.2))


def _refuse(n):
    from automs_gb300._lib import lib
    lib().ams_debug_refuse_allocations(int(n))


def _same(a, b):
    assert all(a[1][k] == b[1][k] for k in COUNTS), (a[1], b[1])
    assert a[1]["rx_paths"] > 0
    assert torch.equal(a[0], b[0])  # sums of fixed-point numbers: the same bits


def test_task_list_of_every_path_in_every_cell():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import tracer
    src, dst = _ends()
    plain = tracer.Scene(*_room())
    want = plain.trace(src, dst, _params(3))
    plain.close()
    st = want[1]
    # a task takes 24 bytes; round by round no list is longer than twice all
    # tasks, and a list is 1 MB at least
    limit = max(1 << 20, 48 * st["tasks"]) + 1024
    assert 24 * 400 * st["unique_paths"] > limit  # 20 x 20 cells
    sc = tracer.Scene(*_room())
    sc.trace(src, dst, _params(0))  # the workspace, whose size is the same
    try:
        _refuse(limit)
        got = sc.trace(src, dst, _params(3))
    finally:
        _refuse(0)
    _same(got, want)
    _same(sc.trace(src, dst, _params(3)), want)
    sc.close()


def test_wide_nodes():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from automs_gb300 import tracer
    room = _room()
    src, dst = _ends()
    plain = tracer.Scene(*room)
    want = plain.trace(src, dst, _params(3))
    plain.close()
    n = len(room[0])
    try:
        _refuse(896 * (n // 3 + 64))  # nothing else of this scene is as large
        sc = tracer.Scene(*room)
    finally:
        _refuse(0)
    _same(sc.trace(src, dst, _params(3)), want)
    sc.close()
