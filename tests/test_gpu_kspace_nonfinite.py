"""A charge at a position that is not finite makes the reciprocal-space energy and every charge's force
NaN, in every form of the k-space sum (the integer tables have no NaN of their own)."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axis", [0, 1])
# dense and one-k-at-a-time kernels; in FP64 the first is the limb form
@pytest.mark.parametrize("precision,n_kmax", [("mixed", 5), ("mixed", 40), ("fp64", 5), ("fp64", 40)])
def test_energy_and_forces_are_nan(precision, n_kmax, axis, value):
    inp = configs.wca_inputs(thermostat=1)
    inp.flags.system, inp.flags.particle_4 = 2, 1
    inp.inter4 = 1
    inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
    inp.charge[2], inp.charge[3] = 1.0, -1.0
    inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, n_kmax, 2.0
    p = md.derive(inp)[0]
    n = 90
    g3 = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 1.9 + 0.01
    g3[:, 2] += 1.0
    s = abi.System()
    s.boundary[0] = s.boundary[1] = 10.0
    s.boundary[2] = 12.0
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, 45, 1, 45
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, 3
    t = np.array([3] * 45 + [4] * 45, np.int32)
    with md.MdSystem(p, s, t, g3, precision=precision, skin=0.4) as g:
        assert np.isfinite(g.ewald_k()[0])
        r = g3.copy()
        r[0, axis] = value  # at 0.01: the fixed point takes 0 for it, no list is rebuilt
        g.set_state(r)
        g.zero_force()
        assert np.isnan(g.ewald_k()[0])
        assert np.isnan(g.state()[3]).all()
        # a finite state gives finite sums again
        g.set_state(g3)
        g.zero_force()
        assert np.isfinite(g.ewald_k()[0])
        assert np.isfinite(g.state()[3]).all()
