"""Training step of the warm-start network at the edges of its tiles: rows
around 64 (layer kernels), around 2048 (loss tiles) and groups of one tile and
several, against the FP64 forward and backward on the GPU's own features."""
import numpy as np
import pytest

import parrsb_gb300 as P
from parrsb_gb300 import meshgen
from parrsb_gb300 import warm as Wm

pytestmark = pytest.mark.gpu


def _batch(shapes):
    vtx, xyz, grp, top = [], [], [], 0
    for g, s in enumerate(shapes):
        v, x = meshgen.box_hex(*s, jitter=0.1, seed=g)
        vtx.append(v + top)
        xyz.append(x)
        grp.append(np.full(len(v), g, dtype=np.int32))
        top += int(v.max())
    return np.concatenate(vtx), np.concatenate(xyz), np.concatenate(grp)


@pytest.mark.parametrize("shapes", [
    [(3, 1, 1)],
    [(7, 3, 3)],                       # 63 rows
    [(4, 4, 4)],                       # 64
    [(13, 5, 1)],                      # 65
    [(23, 89, 1), (2, 1, 1)],          # 2047 and a group of two
    [(16, 16, 8), (4, 4, 4)],          # 2048, whole tiles
    [(683, 3, 1), (31, 3, 1), (1, 1, 2)],  # 2049
    [(20, 19, 18), (5, 3, 1), (17, 16, 15)],
])
def test_step_at_the_edges(shapes):
    import torch
    from oracle import oracle as O
    from oracle import warm_oracle as W
    vtx, xyz, group = _batch(shapes)
    G = len(shapes)
    b = Wm.Batch(vtx, xyz, group, G)
    X = b.features().cpu().numpy().astype(np.float64)
    rows, col, w = W.restrict(*O.dual_graph(vtx), group)
    rng = np.random.default_rng(5)
    params = Wm.init_params(3).astype(np.float64)
    params[W.OFF["b1"][0]:W.OFF["b1"][1]] = rng.normal(0, 0.1, 64)
    params[W.OFF["wo"][0]:W.OFF["wo"][1]] = rng.normal(0, 0.1, 64)
    # (a label far from zero mean: the moments are those of the centred one)
    label = np.ascontiguousarray(50.0 + np.cos(np.pi * X[:, 0] * 0.5) + 0.1 * rng.normal(size=len(X)))
    p32 = params.astype(np.float32)
    d_g = torch.zeros(len(p32), dtype=torch.float32, device="cuda")
    loss, pred = b.step(torch.from_numpy(p32).cuda(), torch.from_numpy(label).cuda(), d_g,
                        want_pred=True)
    b.close()
    p64 = p32.astype(np.float64)
    y, _ = W.forward(X, rows, col, w, p64)
    Lo, go = W.gradient(X, rows, col, w, p64, label, group.astype(np.int64))
    # BF16 activations through three layers (8 significant bits each)
    pred = pred.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(pred - y) <= 3e-2 * np.linalg.norm(y)
    assert abs(loss - Lo) <= 2e-2 * max(Lo, 1e-3) + 1e-4
    grad = d_g.cpu().numpy().astype(np.float64)
    assert np.all(np.isfinite(grad))
    for name, (a, z) in W.OFF.items():
        nrm = np.linalg.norm(go[a:z])
        err = np.linalg.norm(grad[a:z] - go[a:z])
        assert err <= 6e-2 * nrm + 6e-2 * np.linalg.norm(go) + 1e-6, (name, err, nrm)
