"""Sorts of doubles inside segments through the entry points that use them:
RIB orders and gencon ids against the oracle at sizes around the limits of the
three forms (counting up to 32 items, one CTA up to 1024 and 4096, radix passes
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


@pytest.mark.parametrize("n", [2, 31, 33, 1023, 1025, 4096, 4097, 8191, 20011])
def test_rib_around_the_limits(oracle, n):
    vtx, xyz = meshgen.box_quad(n, 1, jitter=0.0, seed=1)
    rng = np.random.Generator(np.random.PCG64(n))
    o = rng.permutation(n)
    xyz = xyz[o] + rng.uniform(-1e-3, 1e-3, (n, 1, 2))
    _rib(oracle, vtx[o], np.ascontiguousarray(xyz), 2)


@pytest.mark.parametrize("values", ["equal", "last_bits", "few", "huge_range"])
@pytest.mark.parametrize("n", [900, 4001, 20000])
def test_rib_ties_and_near_ties(oracle, values, n):
    """One coordinate that ties or nearly ties over many elements: the 32-bit
    keys of the radix form collide, in runs longer than a thread fixes, and the
    buckets of the shared-memory form overflow."""
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


def _same_gencon(oracle, xyz, tol):
    rc, ref, _, _ = oracle.conn_mesh(xyz, 3, tol)
    if rc:
        with pytest.raises(P.ParrsbError) as e:
            P.conn_mesh(xyz, 3, tol)
        assert e.value.code == rc
    else:
        np.testing.assert_array_equal(P.conn_mesh(xyz, 3, tol), ref)
    return rc


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 70, 2.0 ** -70])
@pytest.mark.parametrize("ulps", [-(1 << 30), -1, 0, 1, 1 << 30])
def test_gencon_gap_at_the_tolerance(oracle, scale, ulps):
    """Two unit cubes whose touching faces are tol apart, to the last bit: the
    single-precision screen has to leave the decision to FP64, also where its
    range ends."""
    _, xyz = meshgen.box_hex(2, 1, 1, jitter=0.0, seed=1)
    xyz = np.ascontiguousarray(xyz * (1.0 / np.ptp(xyz.reshape(-1, 3), axis=0)) * [2.0, 1.0, 1.0])
    second = xyz[..., 0].mean(axis=1) > 1.0
    xyz[second, :, 0] += 0.25 + ulps * 2.0 ** -52
    _same_gencon(oracle, np.ascontiguousarray(xyz * scale), 0.25)


@pytest.mark.parametrize("copies", [2, 64, 65, 66, 150])
@pytest.mark.parametrize("split", [False, True])
def test_gencon_many_elements_around_a_face(oracle, copies, split):
    """As many elements on the same corners as the face check's table holds,
    and more; with one that has three corners of a face of the others."""
    _, one = meshgen.box_hex(1, 1, 1, jitter=0.0, seed=1)
    xyz = np.repeat(one, copies, axis=0)
    if split:
        xyz[copies // 2, 0] -= 0.4
    assert bool(_same_gencon(oracle, np.ascontiguousarray(xyz), 0.1)) == split
