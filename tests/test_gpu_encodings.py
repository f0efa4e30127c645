"""The level encodings of the team step kernel and of the staged SpMV: which
of them a level makes, and what runs where one does not apply."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _launches(vtx, grp):
    P.fiedler_groups(vtx, grp, 1, rsb_max_passes=2)  # (decides the block size)
    f, it, _ = P.fiedler_groups(vtx, grp, 1, rsb_max_passes=2)
    return P.last_stats().kernel_launches, f, it


def test_one_encoding_per_level(monkeypatch):
    """A level of the team kernel is not encoded for the staged SpMV too."""
    monkeypatch.setenv("PARRSB_GPU_FP32", "1")
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "1")
    vtx, _ = meshgen.box_hex(24, 20, 16, jitter=0.1, seed=4)
    grp = np.zeros(len(vtx), np.int32)
    monkeypatch.setenv("PARRSB_GPU_SPMV", "0")
    plain, f0, i0 = _launches(vtx, grp)
    monkeypatch.setenv("PARRSB_GPU_SPMV", "2")
    staged, f2, i2 = _launches(vtx, grp)
    assert staged == plain
    np.testing.assert_array_equal(f0, f2)
    np.testing.assert_array_equal(i0, i2)


@pytest.mark.parametrize("persist,spmv", [("1", "0"), ("0", "2"), ("1", "2")])
def test_no_memory_for_an_encoding(monkeypatch, persist, spmv):
    """An encoding that does not fit the device's memory (injected on the
    host) leaves the level to the form that needs none."""
    monkeypatch.setenv("PARRSB_GPU_FP32", "1")
    vtx, _ = meshgen.box_hex(24, 20, 16, jitter=0.1, seed=4)
    grp = np.zeros(len(vtx), np.int32)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "0")
    monkeypatch.setenv("PARRSB_GPU_SPMV", "0")
    plain, f0, i0 = _launches(vtx, grp)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", persist)
    monkeypatch.setenv("PARRSB_GPU_SPMV", spmv)
    monkeypatch.setenv("PARRSB_FAULT", "encoding")
    got, f1, i1 = _launches(vtx, grp)
    assert got == plain
    np.testing.assert_array_equal(f0, f1)
    np.testing.assert_array_equal(i0, i1)


def test_staged_spmv_after_the_team_encoder_refuses(monkeypatch):
    """Planes of seven lines of 300 elements: the rows beside a block of 512 are
    more than the team kernel holds, those beside a staged run of 8192 are not.
    The team encoder has written its own buffers by then."""
    monkeypatch.setenv("PARRSB_GPU_FP32", "1")
    vtx, _ = meshgen.box_hex(300, 7, 14, jitter=0.1, seed=4)
    grp = np.zeros(len(vtx), np.int32)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "0")
    monkeypatch.setenv("PARRSB_GPU_SPMV", "0")
    plain, f0, i0 = _launches(vtx, grp)
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "1")
    monkeypatch.setenv("PARRSB_GPU_SPMV", "2")
    got, f1, i1 = _launches(vtx, grp)
    assert got == plain + 2  # both encoders, then a launch per kernel
    np.testing.assert_array_equal(f0, f1)
    np.testing.assert_array_equal(i0, i1)
