"""The team step kernel (every Lanczos step of a pass in one launch) against
the launch-per-kernel steps: bitwise the same Fiedler vectors, step counts and
residuals at the sizes where its tiling can go wrong."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu

# groups by element count: one element short of, at and past a chunk (32), a
# vector chunk (64 / 128), a tile (512) and the largest single block; the
# starts that follow are unaligned
SIZES = {
    "edges": [2, 3, 31, 32, 33, 63, 65, 127, 129, 511, 512, 513, 1023, 1025, 2049],
    "teams": [20000, 513, 8193, 12289, 700],
    "one": [70001],
}


def _chain_boxes(sizes, seed):
    """Disjoint jittered boxes cut down to exactly sizes[g] elements."""
    vs, gs, off = [], [], 0
    for g, n in enumerate(sizes):
        side = max(1, int(round(n ** (1.0 / 3.0))))
        nx = -(-n // (side * side))
        v, _ = meshgen.box_hex(max(nx, 2), side, side, jitter=0.1, seed=seed + g, id_offset=off)
        off += (max(nx, 2) + 1) * (side + 1) ** 2
        vs.append(v[:n])
        gs.append(np.full(n, g, np.int32))
    return np.concatenate(vs), np.concatenate(gs)


def _both(monkeypatch, vtx, grp, ng, **kw):
    out = []
    for ps in ("0", "1"):
        monkeypatch.setenv("PARRSB_GPU_PERSIST", ps)
        out.append(P.fiedler_groups(vtx, grp, ng, **kw) + (P.last_stats().kernel_launches,))
    for a, b in zip(out[0][:3], out[1][:3]):
        np.testing.assert_array_equal(a, b)
    return out[0][3], out[1][3]


@pytest.mark.parametrize("stop", ["0", "1"])
@pytest.mark.parametrize("fp32", ["0", "1"])
@pytest.mark.parametrize("case", sorted(SIZES))
def test_team_steps_bitwise(monkeypatch, case, fp32, stop):
    monkeypatch.setenv("PARRSB_GPU_FP32", fp32)
    monkeypatch.setenv("PARRSB_GPU_RESID_STOP", stop)  # with it, the early pass exit
    sizes = SIZES[case]
    vtx, grp = _chain_boxes(sizes, 5)
    launches, team = _both(monkeypatch, vtx, grp, len(sizes), rsb_max_passes=3)
    assert team < launches // 2  # the steps ran in one launch per pass


@pytest.mark.parametrize("fp32", ["0", "1"])
def test_team_steps_other_weights(monkeypatch, fp32):
    """Two elements that share three vertices (weight 3) do not fit the
    16-bit entries: the level takes the launch-per-kernel steps."""
    monkeypatch.setenv("PARRSB_GPU_FP32", fp32)
    vtx, _ = meshgen.box_hex(12, 10, 8, jitter=0.1, seed=3)
    vtx[0, :] = vtx[200, :]
    vtx[0, 3:] = vtx.max() + 1 + np.arange(5)
    launches, team = _both(monkeypatch, vtx, np.zeros(len(vtx), np.int32), 1, rsb_max_passes=2)
    assert team > launches // 2
