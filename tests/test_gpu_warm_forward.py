"""A forward pass of the warm-start network alone, whose layers share buffers,
gives bitwise the prediction of the training step, which keeps them all."""
import numpy as np
import pytest

from parrsb_gb300 import meshgen
from parrsb_gb300 import warm as Wm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(3, 1, 1)], [(13, 5, 1), (4, 4, 4)],
                                    [(40, 40, 30), (64, 40, 31), (5, 3, 2)]])
def test_forward_alone(shapes):
    import torch
    vtx, xyz, grp, top = [], [], [], 0
    for g, s in enumerate(shapes):
        v, x = meshgen.box_hex(*s, jitter=0.1, seed=g, id_offset=top)
        top += (s[0] + 1) * (s[1] + 1) * (s[2] + 1)
        vtx.append(v)
        xyz.append(x)
        grp.append(np.full(len(v), g, dtype=np.int32))
    vtx, xyz, grp = np.concatenate(vtx), np.concatenate(xyz), np.concatenate(grp)
    params = torch.from_numpy(np.asarray(Wm.init_params(3), np.float32)).cuda()
    label = torch.from_numpy(np.random.default_rng(1).normal(size=len(vtx))).cuda()
    preds = []
    for train in (False, True, False):
        b = Wm.Batch(vtx, xyz, grp, len(shapes))
        if train:
            preds.append(b.step(params, label, torch.zeros_like(params), want_pred=True)[1])
        else:
            preds.append(b.step(params, want_pred=True)[1])
        b.close()
    assert torch.equal(preds[0], preds[1]) and torch.equal(preds[0], preds[2])
    assert float(preds[0].abs().max()) > 0.0
