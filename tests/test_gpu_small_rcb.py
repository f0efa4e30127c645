"""RCB of segments that one CTA finishes, against the oracle: sizes around the
rounds of 32 and 1024 positions, ranks that are unique (presorted lists and
sorts per level) and that tie (buckets, crowded buckets), recursion down to
single elements, and the same partition without allocation."""
import numpy as np
import pytest
import torch

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _points(kind, n, nv, seed=5):
    rng = np.random.Generator(np.random.PCG64(seed + n))
    d = 3 if nv == 8 else 2
    if kind == "unique":
        x = rng.uniform(-1.0, 1.0, (n, d))
    elif kind == "lattice":  # every axis ties
        x = rng.integers(0, 9, (n, d)).astype(np.float64)
    elif kind == "crowded":  # most in one bucket, a few far away
        x = 1.0 + rng.integers(0, 3000, (n, d)) * 2.0 ** -50
        x[rng.random(n) < 0.02] *= 1e6
    else:  # all the same point
        x = np.full((n, d), 0.3)
    return np.ascontiguousarray(np.repeat(x[:, None, :], nv, axis=1))


def _noalloc(xyz, nparts):
    """d_part of the entry point on torch buffers and the current stream."""
    lib = P.library()
    n, nv, _ = xyz.shape
    assert lib.parrsb_part_mesh_rcb_noalloc(None, None, 0, nv, 1, None) == 0
    x = torch.from_numpy(xyz).cuda()
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.parrsb_part_mesh_rcb_noalloc(out.data_ptr(), x.data_ptr(), n, nv, nparts, st) == 0
    return out.cpu().numpy()


def _check(oracle, xyz, nparts, noalloc):
    n, nv, _ = xyz.shape
    vtx = np.arange(n * nv, dtype=np.int64).reshape(n, nv) + 1
    part, seq = P.part_mesh_seq(vtx, xyz, nparts, partitioner=1)
    rc, ref, order, _, _ = oracle.part_mesh(vtx, xyz, nparts, want_order=True, partitioner=1)
    assert rc == 0
    np.testing.assert_array_equal(part, ref)
    np.testing.assert_array_equal(np.lexsort((seq, part)), order)
    if noalloc:
        np.testing.assert_array_equal(_noalloc(xyz, nparts), ref)


@pytest.mark.parametrize("presort", ["1", "0"])
@pytest.mark.parametrize("kind", ["unique", "lattice", "crowded", "same"])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 64, 1023, 1025, 4097, 8191, 8192])
def test_one_segment(oracle, monkeypatch, n, kind, presort):
    monkeypatch.setenv("PARRSB_GPU_RCB_PRESORT", presort)
    _check(oracle, _points(kind, n, 8), min(n, 7), presort == "1")


@pytest.mark.parametrize("kind", ["unique", "lattice", "crowded"])
@pytest.mark.parametrize("n,nparts", [(700, 700), (8192, 8192), (8190, 4097), (2050, 1000)])
def test_down_to_single_elements(oracle, n, nparts, kind):
    _check(oracle, _points(kind, n, 4), nparts, True)


@pytest.mark.parametrize("kind", ["unique", "lattice"])
def test_many_segments(oracle, kind):
    """Global levels above, then a CTA per segment."""
    _check(oracle, _points(kind, 40001, 8), 37, False)


def test_more_parts_than_elements():
    xyz = _points("lattice", 50, 8)
    vtx = np.arange(400, dtype=np.int64).reshape(50, 8) + 1
    a = P.part_mesh(vtx, xyz, 200, partitioner=1)
    np.testing.assert_array_equal(np.asarray(a), _noalloc(xyz, 200))
