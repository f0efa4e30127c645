"""Sorts of values that a linear map over their range does not separate (one far
point, clumps, geometric grading, last-bit forms of a value): RIB orders and RCB
parts against the oracle, gencon ids against those of the same mesh without its
far element."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _line(values):
    n = len(values)
    xyz = np.zeros((n, 4, 2))
    xyz[..., 0] = values[:, None]
    return np.arange(n * 4, dtype=np.int64).reshape(n, 4) + 1, xyz


def _values(kind, n):
    rng = np.random.Generator(np.random.PCG64(5))
    x = rng.random(n)
    if kind == "far":
        x[n // 3] = 1e9
    elif kind == "clumps":  # half of them within 1e-7, 1e-9, 1e-12 of the range
        x[: n // 2] *= 1e-7
    elif kind == "tight_clumps":
        x[: n // 2] *= 1e-9
    elif kind == "points":
        x[: n // 2] = 0.5 + x[: n // 2] * 1e-12
    elif kind == "fars":  # the refined values have a far one among them too
        x[: n // 2] *= 2.0 ** -40
        x[1] = 1e9
    elif kind == "deep":  # half of them closer than the fixed point tells apart
        x[: n // 2] *= 2.0 ** -70
    elif kind == "graded":
        x = np.expm1(np.log(1e12) * x)
    elif kind == "twins":  # many values, each in two forms
        x = (np.floor(n / 100.0 * x) + 1.0) * (1.0 + 2.0 ** -52 * rng.integers(0, 2, n))
    elif kind == "planes":  # 30 values, in their last bits apart
        x = np.floor(30.0 * x) / 30.0 * (1.0 + 2.0 ** -52 * rng.integers(-2, 3, n))
    return x


@pytest.mark.parametrize("n", [4097, 20000, 262144, 300001])
@pytest.mark.parametrize("kind", ["far", "clumps", "tight_clumps", "points", "fars", "deep",
                                  "graded", "twins", "planes"])
def test_ranges(oracle, kind, n):
    vtx, xyz = _line(_values(kind, n))
    for partitioner in (1, 2):
        part, seq = P.part_mesh_seq(vtx, xyz, 2, partitioner=partitioner)
        rc, ref, order, _, _ = oracle.part_mesh(vtx, xyz, 2, want_order=True,
                                                partitioner=partitioner)
        assert rc == 0
        np.testing.assert_array_equal(part, ref)
        np.testing.assert_array_equal(np.lexsort((seq, part)), order)


def test_segments_with_clumps(oracle):
    """Segments of more than 4096 elements, each with values that do not separate."""
    rng = np.random.Generator(np.random.PCG64(6))
    n = 40000
    for kind in range(3):
        x = rng.random((n, 2))
        if kind == 0:
            x[:, 0] = np.where(rng.random(n) < 0.7, x[:, 0] * 1e-11, x[:, 0])
        elif kind == 1:
            x[:, 0] = np.round(x[:, 0] * 4) / 4 * (1 + 2.0 ** -52 * rng.integers(0, 3, n))
        else:
            x[:, 0] *= np.where(rng.random(n) < 0.5, 2.0 ** -66, 1.0)
        xyz = np.ascontiguousarray(np.repeat(x[:, None, :], 4, axis=1))
        vtx = np.arange(n * 4, dtype=np.int64).reshape(n, 4) + 1
        part, seq = P.part_mesh_seq(vtx, xyz, 4, partitioner=2)
        rc, ref, order, _, _ = oracle.part_mesh(vtx, xyz, 4, want_order=True, partitioner=2)
        assert rc == 0
        np.testing.assert_array_equal(part, ref)
        np.testing.assert_array_equal(np.lexsort((seq, part)), order)


def test_gencon_far_element():
    _, xyz = meshgen.box_hex(40, 20, 20, jitter=0.1, seed=2)
    want = P.conn_mesh(xyz, 3)
    far = xyz[:1] + 1e9 * np.ones(3)
    got = P.conn_mesh(np.concatenate([xyz, far]), 3)
    np.testing.assert_array_equal(got[:-1], want)
    assert len(np.unique(got[-1])) == 8 and got[-1].min() > want.max()
