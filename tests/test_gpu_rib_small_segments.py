"""RIB on many small segments against the oracle: the sums by a warp (up to 32
elements) and by a block (up to 1024) per segment, the axes by quads and, beyond
8192 segments, by single threads."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [63, 64, 65, 1023, 1025, 2047, 2049, 4100])
@pytest.mark.parametrize("per_part", [1, 2, 17, 33])
def test_around_the_forms(oracle, n, per_part):
    vtx, xyz = meshgen.box_hex(n, 1, 1, jitter=0.2, seed=3)
    o = np.random.Generator(np.random.PCG64(n)).permutation(n)
    vtx, xyz, nparts = vtx[o], np.ascontiguousarray(xyz[o]), max(2, n // per_part)
    part, seq = P.part_mesh_seq(vtx, xyz, nparts, partitioner=2)
    rc, ref, order, _, _ = oracle.part_mesh(vtx, xyz, nparts, want_order=True, partitioner=2)
    assert rc == 0
    np.testing.assert_array_equal(part, ref)
    np.testing.assert_array_equal(np.lexsort((seq, part)), order)


@pytest.mark.parametrize("ndim", [2, 3])
def test_many_segments(oracle, ndim):
    mesh = (meshgen.box_quad(250, 160, jitter=0.2, seed=5) if ndim == 2 else
            meshgen.box_hex(50, 40, 20, jitter=0.2, seed=5))
    vtx, xyz = mesh
    part = P.part_mesh(vtx, xyz, 20000, partitioner=2)
    rc, ref = oracle.part_mesh(vtx, xyz, 20000, partitioner=2)[:2]
    assert rc == 0
    np.testing.assert_array_equal(part, ref)
