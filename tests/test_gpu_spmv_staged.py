"""FP32 SpMV on staged rows (k_spmv_loc) against k_spmv: the same Fiedler
vectors and iteration counts, bit for bit, at group sizes around the tile and
slice lengths, unaligned groups, wide rows and weights outside its range."""
import numpy as np
import pytest

import parrsb_gb300 as P

pytestmark = pytest.mark.gpu

OFF = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1],
                [0, 1, 1]])


def _box(nx, ny, nz):
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    i, j, k = i.ravel(), j.ravel(), k.ravel()
    v = (i[:, None] + OFF[:, 0]) + (nx + 1) * ((j[:, None] + OFF[:, 1]) +
                                               (ny + 1) * (k[:, None] + OFF[:, 2]))
    return v + 1, (nx + 1) * (ny + 1) * (nz + 1)


def _run(monkeypatch, vtx, grp, count, spmv):
    monkeypatch.setenv("PARRSB_GPU_FP32", "1")
    monkeypatch.setenv("PARRSB_GPU_PERSIST", "0")
    monkeypatch.setenv("PARRSB_GPU_SPMV", spmv)
    f, it, _ = P.fiedler_groups(vtx, grp, count, rsb_max_passes=2)
    return f, it


def _same(monkeypatch, vtx, grp, count):
    f0, i0 = _run(monkeypatch, vtx, grp, count, "0")
    f2, i2 = _run(monkeypatch, vtx, grp, count, "2")
    np.testing.assert_array_equal(i0, i2)
    np.testing.assert_array_equal(f0, f2)


@pytest.mark.parametrize("dims,count", [((5, 3, 2), 1), ((13, 9, 5), 7), ((31, 1, 1), 5),
                                        ((8, 8, 8), 9), ((33, 17, 9), 3), ((64, 32, 32), 2),
                                        ((63, 64, 65), 1)])
def test_same_bits_as_k_spmv(monkeypatch, dims, count):
    v, nv = _box(*dims)
    vtx = np.concatenate([v + g * nv for g in range(count)])
    grp = np.repeat(np.arange(count, dtype=np.int32), len(v))
    _same(monkeypatch, vtx, grp, count)


def test_rows_in_random_order_fall_back(monkeypatch):
    """Halos larger than the table: the other form takes over."""
    v, _ = _box(40, 40, 40)
    v = v[np.random.Generator(np.random.PCG64(1)).permutation(len(v))]
    _same(monkeypatch, v, np.zeros(len(v), dtype=np.int32), 1)


def test_wide_rows_and_other_weights(monkeypatch):
    """A fan of elements around one edge (rows wider than the registers hold)
    and elements that share three corners (a weight without a code)."""
    n = 90
    fan = np.stack([np.full(n, 1), np.full(n, 2)] +
                   [3 + 6 * np.arange(n) + c for c in range(6)], axis=1)
    _same(monkeypatch, fan.astype(np.int64), np.zeros(n, dtype=np.int32), 1)
    v, _ = _box(6, 5, 4)
    v = v.copy()
    v[::7, 6] = 10000 + np.arange(len(v[::7]))  # a corner of their own: three shared of a face
    _same(monkeypatch, v, np.zeros(len(v), dtype=np.int32), 1)
