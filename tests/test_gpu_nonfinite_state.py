"""An uploaded coordinate that is not finite, or beyond any channel, is reported in both precisions: by the
rebuild that the upload causes, or by the next step's integration."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _report(precision, axis, value):
    p, (s, t, r, v) = configs.wca_params(), configs.brush_channel(11.0, 13.0, 0.1, 11, seed=7)
    i = s.n_mon * s.n_chain + 5  # a solvent bead
    with md.MdSystem(p, s, t, r, v, precision=precision, skin=0.4) as g:
        g.step(2)
        r = g.state()[0]
        r[i, axis] = value
        with pytest.raises(abi.MfaError) as e:
            g.set_state(r)
            g.step(1)
            g.synchronize()
    return e.value.code


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_not_finite(precision, axis, value):
    assert _report(precision, axis, value) == -6


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("value", [1e3, -1e3, 2.0 ** 128, -(2.0 ** 129), 1e300])
def test_far_out_of_the_channel(precision, value):
    assert _report(precision, 2, value) == -5


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_z_is_seen_by_the_upload_itself(precision, value):
    p, (s, t, r, v) = configs.wca_params(), configs.brush_channel(11.0, 13.0, 0.1, 11, seed=7)
    with md.MdSystem(p, s, t, r, v, precision=precision, skin=0.4) as g:
        r[s.n_mon * s.n_chain + 5, 2] = value
        with pytest.raises(abi.MfaError) as e:
            g.set_state(r)
        assert e.value.code == -6
