"""The early pass exit's stride and delay in the team step kernel: for every
pair that the settings allow, bitwise the launch-per-kernel steps.  A request
that applies one step after its check has no exchange to travel with, so a
delay of 1 keeps the launches."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _groups():
    vs, off = [], 0
    for g, d in enumerate([(9, 8, 7), (20, 16, 12), (24, 20, 18)]):
        v, _ = meshgen.box_hex(*d, jitter=0.1, seed=11 + g, id_offset=off)
        off += (d[0] + 1) * (d[1] + 1) * (d[2] + 1)
        vs.append(v)
    return np.concatenate(vs), np.repeat(np.arange(3, dtype=np.int32), [len(v) for v in vs])


@pytest.mark.parametrize("fp32", ["0", "1"])
@pytest.mark.parametrize("stride,delay", [(1, 1), (2, 1), (3, 1), (2, 2), (3, 2), (3, 3), (4, 2)])
def test_stride_and_delay(monkeypatch, fp32, stride, delay):
    monkeypatch.setenv("PARRSB_GPU_FP32", fp32)
    monkeypatch.setenv("PARRSB_GPU_RESID_STOP", "1")
    monkeypatch.setenv("PARRSB_GPU_EARLY_STRIDE", str(stride))
    monkeypatch.setenv("PARRSB_GPU_EARLY_DELAY", str(delay))
    vtx, grp = _groups()
    out, launches = [], []
    for ps in ("0", "1"):
        monkeypatch.setenv("PARRSB_GPU_PERSIST", ps)
        out.append(P.fiedler_groups(vtx, grp, 3, rsb_max_passes=4))
        launches.append(P.last_stats().kernel_launches)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    if delay == 1:
        assert launches[1] > launches[0] // 2
    else:
        assert launches[1] < launches[0] // 2
