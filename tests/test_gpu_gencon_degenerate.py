"""gencon on corners that run together: the element check fails, and the call
says so without the face check's walk over vertices that every element shares
(its work grows with the square of their number)."""
import numpy as np
import pytest

import parrsb_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.0, 1e-9])
def test_collapsed_elements(spread):
    n = 150000
    rng = np.random.Generator(np.random.PCG64(7))
    xyz = np.zeros((n, 8, 3))  # every corner of an element in one of two places
    xyz += spread * rng.integers(0, 2, size=(n, 1, 1))
    with pytest.raises(P.ParrsbError) as ei:
        P.conn_mesh(xyz, 3)
    assert ei.value.code == 1
    # 0.1 ms here; seconds where every corner is compared with every element
    assert P.last_stats().stage_ms[P.STAGES.index("check")] < 100.0
