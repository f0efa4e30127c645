"""The team step kernel's failures, injected on the host: a wait that gave up
and a launch that was refused repeat the level with launch-per-kernel steps,
and the call's results are bitwise those of PARRSB_GPU_PERSIST=0."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _call(vtx, xyz):
    part = P.part_mesh(vtx, xyz, 12, partitioner=0)
    s = P.last_stats()
    return part, s.lanczos_iters, s.lanczos_passes, s.spmv_launches, s.max_fiedler_resid


@pytest.mark.parametrize("mode", ["device_loop", "host_loop", "no_graphs"])
@pytest.mark.parametrize("start", ["0", "2"])
@pytest.mark.parametrize("fault", ["team_wait", "team_launch"])
def test_level_is_repeated(monkeypatch, capfd, fault, start, mode):
    monkeypatch.setenv("PARRSB_GPU_START", start)
    monkeypatch.setenv("PARRSB_GPU_FP32", "1")
    monkeypatch.setenv("PARRSB_GPU_RESID_STOP", "1")
    if mode == "host_loop":
        monkeypatch.setenv("PARRSB_GPU_DEVICE_LOOP", "0")
    if mode == "no_graphs":
        monkeypatch.setenv("PARRSB_GPU_GRAPHS", "0")
    vtx, xyz = meshgen.box_hex(30, 22, 16, jitter=0.1, seed=9)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "0")
    want = _call(vtx, xyz)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "1")
    monkeypatch.setenv("PARRSB_FAULT", fault)
    capfd.readouterr()
    got = _call(vtx, xyz)
    assert capfd.readouterr().err.count("team step kernel not available") == 1
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1:] == want[1:]
    monkeypatch.delenv("PARRSB_FAULT")  # and the next call takes the team kernel again
    np.testing.assert_array_equal(_call(vtx, xyz)[0], want[0])
    assert "not available" not in capfd.readouterr().err
