"""Dual-graph rows around the sizes of the candidate list (32 a round, 256 in
the table, longer ones pairwise), for every number of corners per element: each
row in the order of first occurrence, the weights the numbers of occurrences."""
import numpy as np
import pytest

import parrsb_gb300 as P

pytestmark = pytest.mark.gpu


def _first_occurrence(vtx, a):
    """Elements that share a vertex with a: vertex by vertex, each vertex's
    corners in element order."""
    seen = {}
    for v in vtx[a]:
        for b in np.nonzero(vtx == v)[0]:
            if b != a:
                seen[int(b)] = seen.get(int(b), 0) + 1
    return seen


@pytest.mark.parametrize("nv", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("run", [1, 2, 8, 31, 33, 65, 300])
def test_rows_of_random_incidence(nv, run):
    """Every vertex id is shared by about `run` element corners; corners of an
    element may coincide."""
    rng = np.random.Generator(np.random.PCG64(100 * nv + run))
    n = 700
    vtx = rng.integers(1, max(2, n * nv // run) + 1, (n, nv)).astype(np.int64)
    rp, col, w = P.dual_graph(vtx)
    for a in range(0, n, 11):
        ref = _first_occurrence(vtx, a)
        assert list(ref) == list(col[rp[a]:rp[a + 1]])
        assert [min(c, 255) for c in ref.values()] == list(w[rp[a]:rp[a + 1]])
