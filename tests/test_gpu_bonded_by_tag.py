"""Bonded terms by tag (more than 128 particles per SM) against the same chains alone, taken by slot: a
channel's bonded forces do not depend on the other replicas of its batch, bit for bit."""
import numpy as np
import pytest

from mfa_brush_gb300 import configs, md

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_mon", [2, 9, 33])
def test_batch_equals_single(precision, n_mon):
    p = configs.wca_params()
    reps = [configs.brush_channel(6.0 + k % 3, 12.0, 0.06, n_mon, 0.7, seed=5 + k) for k in range(64)]
    systems, t, r, v = configs.concat(reps)
    assert len(t) > 128 * 152

    def bonded(*a):
        with md.MdSystem(p, *a, precision=precision, skin=0.4) as g:
            g.zero_force()
            return g.intra_molec(), g.state()[3]

    e, f = bonded(systems, t, r, v)
    at = 0
    for k, (s, a, x, u) in enumerate(reps):
        if k % 13 == 0:
            e1, f1 = bonded(s, a, x, u)
            assert np.array_equal(f[at:at + len(a)], f1)
            # a few thousand positive terms in another order: 1e-12 in FP64, 1e-5 summed in FP32 by warps
            assert np.allclose(np.asarray(e)[k], np.asarray(e1)[0], rtol=1e-12 if precision == "fp64" else 1e-5)
        at += len(a)
