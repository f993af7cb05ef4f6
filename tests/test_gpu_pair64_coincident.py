"""FP64 mode: pairs so close that r^2 is below the FP32 range, and coincident ones, as IEEE arithmetic gives them."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _dpd_only():
    """The thermostat's pair forces alone, with a range of their own."""
    p = configs.wca_params()
    p.r_cut_dpd_2 = 1.0
    for k in range(len(p.range_2)):
        p.range_2[k] = 0.0
    return p


def _pair(gap):
    s = abi.System()
    s.boundary[0] = s.boundary[1] = 9.0
    s.boundary[2] = 10.0
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, 2, 0, 0
    s.n_mon_tot = s.n_part = 2
    s.s_time, s.seed = 1, 11
    r = np.array([[0.0, 3.0, 4.0], [gap, 3.0, 4.0]])
    v = np.array([[0.3, -0.2, 0.1], [-0.4, 0.2, 0.5]])
    return s, np.full(2, 3, np.int32), r, v


@pytest.mark.parametrize("block", [0, 32])  # lanes per particle, and one
@pytest.mark.parametrize("gap", [1e-30, 1e-25, 1e-20, 1e-19, 1.2e-19, 1e-18, 1e-9, 0.1])
def test_close_pairs(oracle_mod, gap, block):
    p = _dpd_only()
    s, t, r, v = _pair(gap)
    o = oracle_mod.Oracle(p, s, t, r, v)
    o.zero_force()
    o.fluid_fluid()
    want = o.state()[3]
    assert np.abs(want[0, 0]) > 0.1  # finite, along x
    with md.MdSystem(p, s, t, r, v, precision="fp64", skin=0.4, block_size=block) as g:
        g.zero_force()
        g.fluid_fluid()
        f = g.state()[3]
    # a handful of 64-bit roundings
    assert np.allclose(f, want, rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("block", [0, 32])
@pytest.mark.parametrize("model", ["dpd", "wca"])
def test_coincident_pair_is_not_a_number(model, block):
    p = _dpd_only() if model == "dpd" else configs.wca_params()
    s, t, r, v = _pair(0.0)
    with md.MdSystem(p, s, t, r, v, precision="fp64", skin=0.4, block_size=block) as g:
        g.zero_force()
        g.fluid_fluid()
        assert np.isnan(g.state()[3]).any(axis=1).all()
