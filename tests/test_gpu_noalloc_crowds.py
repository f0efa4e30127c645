"""Allocation-free RCB on values that crowd into few of its buckets, against
the oracle: a far element, clumps and a graded axis, at sizes around the 256
elements that a block ranks."""
import numpy as np
import pytest
import torch

import parrsb_gb300 as P

pytestmark = pytest.mark.gpu


def _points(kind, n):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.random((n, 3))
    if kind == "far":
        x[n // 2] = 1e9
    elif kind == "clumps":  # three quarters, a third of these in one place
        x[: 3 * n // 4] *= 1e-9
        x[: n // 4] = 0.5
    else:
        x = np.expm1(np.log(1e12) * x)
    return np.ascontiguousarray(np.repeat(x[:, None, :], 8, axis=1))


@pytest.mark.parametrize("n", [66, 255, 256, 257, 2049, 8192])
@pytest.mark.parametrize("kind", ["far", "clumps", "graded"])
def test_crowds(oracle, kind, n):
    xyz = _points(kind, n)
    vtx = np.arange(n * 8, dtype=np.int64).reshape(n, 8) + 1
    rc, ref = oracle.part_mesh(vtx, xyz, 5, partitioner=1)[:2]
    assert rc == 0
    lib = P.library()
    assert lib.parrsb_part_mesh_rcb_noalloc(None, None, 0, 8, 1, None) == 0
    x = torch.from_numpy(xyz).cuda()
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.parrsb_part_mesh_rcb_noalloc(out.data_ptr(), x.data_ptr(), n, 8, 5, st) == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
