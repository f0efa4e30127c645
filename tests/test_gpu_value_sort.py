"""Sorts of doubles inside segments through the entry points that use them:
RIB orders and gencon ids against the oracle at sizes around the limits of the
three forms (counting up to 32 items, one CTA up to 1024 and 8192, radix passes
beyond), with values that tie and values that differ in their last bits."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _rib(oracle, vtx, xyz, nparts):
    part, seq = P.part_mesh_seq(vtx, xyz, nparts, partitioner=2)
    rc, ref, order, _, _ = oracle.part_mesh(vtx, xyz, nparts, want_order=True, partitioner=2)
    assert rc == 0
    np.testing.assert_array_equal(part, ref)
    np.testing.assert_array_equal(np.lexsort((seq, part)), order)


@pytest.mark.parametrize("n", [2, 31, 33, 1023, 1025, 8191, 8193, 20011])
def test_rib_around_the_limits(oracle, n):
    vtx, xyz = meshgen.box_quad(n, 1, jitter=0.0, seed=1)
    rng = np.random.Generator(np.random.PCG64(n))
    o = rng.permutation(n)
    xyz = xyz[o] + rng.uniform(-1e-3, 1e-3, (n, 1, 2))
    _rib(oracle, vtx[o], np.ascontiguousarray(xyz), 2)


@pytest.mark.parametrize("values", ["equal", "last_bits", "few", "huge_range"])
def test_rib_ties_and_near_ties(oracle, values):
    """One coordinate that ties or nearly ties over thousands of elements: the
    32-bit keys of the radix form collide, in runs longer than a thread fixes."""
    n = 20000
    rng = np.random.Generator(np.random.PCG64(7))
    x = {"equal": np.full(n, 0.75),
         "last_bits": 0.75 + rng.integers(0, 64, n) * 2.0 ** -52,
         "few": rng.integers(0, 40, n) / 40.0,
         "huge_range": np.exp(rng.uniform(-300.0, 300.0, n)) * rng.choice([-1.0, 1.0], n)}[values]
    vtx = np.arange(n * 4, dtype=np.int64).reshape(n, 4) + 1
    xyz = np.zeros((n, 4, 2))
    xyz[..., 0] = x[:, None]
    _rib(oracle, vtx, xyz, 3)


@pytest.mark.parametrize("dims", [(2, 2, 2), (40, 3, 2), (7, 33, 9), (3, 2, 130)])
@pytest.mark.parametrize("noise", [0.0, 1e-12])
def test_gencon_settled_or_not(oracle, dims, noise):
    """Copies of a vertex with the same bits (the later rounds are skipped)
    and with noise in the last digits (they run on segments of a few points)."""
    _, xyz = meshgen.box_hex(*dims, jitter=0.1, seed=2)
    rng = np.random.Generator(np.random.PCG64(3))
    xyz = np.ascontiguousarray((xyz + noise * rng.uniform(-1, 1, xyz.shape))[rng.permutation(len(xyz))])
    rc, ref, _, _ = oracle.conn_mesh(xyz, 3, 0.2)
    if rc:  # flat elements: the jitter exceeds the tolerance, both refuse
        with pytest.raises(P.ParrsbError) as e:
            P.conn_mesh(xyz, 3, 0.2)
        assert e.value.code == rc
        return
    np.testing.assert_array_equal(P.conn_mesh(xyz, 3, 0.2), ref)
