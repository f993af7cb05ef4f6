"""FP64 mode: a pair one ulp inside the real-space Coulomb cut-off, at cut-offs where its place in the
table rounds onto the table's end."""
import math
from fractions import Fraction

import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu

LO = 0.49  # r^2 at the table's start


def _cut_offs(alpha, count):
    """Distances d whose square, rounded, is the last double below a cut-off r^2 = hi, where (r^2 - lo) / h
    is not below the number of intervals although r^2 < hi."""
    out = []
    for d in np.random.default_rng(1).uniform(1.3, 5.0, 40000):
        z = 1.0 + d
        d = z - 1.0  # what the kernel subtracts
        r2 = d * d
        hi = math.nextafter(r2, 99.0)
        n = math.ceil((hi - LO) / min(LO / 30.0, 0.1 / alpha))
        inv_h = 1.0 / ((hi - LO) / n)
        if Fraction(r2 - LO) * Fraction(inv_h) >= n:
            out.append((d, hi))
            if len(out) == count:
                break
    return out


@pytest.mark.parametrize("alpha", [0.81, 4.0])
def test_last_double_below_the_cut_off(alpha):
    cases = _cut_offs(alpha, 8)
    assert len(cases) == 8
    for d, hi in cases:
        inp = configs.wca_inputs(thermostat=1)
        inp.flags.system, inp.flags.particle_4 = 2, 1
        inp.inter4 = 1
        inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
        inp.charge[2], inp.charge[3] = 1.0, -1.0
        inp.alpha_c, inp.n_kmax, inp.rc_coul = alpha, 2, d
        p = md.derive(inp)[0]
        p.rc_coul_2 = hi
        s = abi.System()
        s.boundary[0] = s.boundary[1] = 3.2 * (d + 0.5)
        s.boundary[2] = d + 4.0
        s.n_mon, s.n_chain = 1, 0
        s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, 1, 1, 1
        s.n_mon_tot = s.n_part = 2
        s.s_time, s.seed = 1, 3
        r = np.array([[2.0, 2.0, 1.0], [2.0, 2.0, 1.0 + d]])
        with md.MdSystem(p, s, np.array([3, 4], np.int32), r, precision="fp64", skin=0.4) as g:
            g.zero_force()
            e = g.fluid_fluid()[1][0]
            F = g.state()[3]
        sa, isp = p.sqrt_alpha, p.inv_sqrt_pi
        ec = math.erfc(sa * d)
        f = 2.0 * sa * isp * math.exp(-alpha * d * d) / d + ec / (d * d)
        # the table's own error is 1e-15 of the value; erfc and exp here enlarge a rounding of alpha d^2
        # (up to 100) by that much: 3e-14
        self_energy = -2.0 * sa / math.sqrt(float(np.float32(3.1415926536)))
        assert F[0, 2] == pytest.approx(f, rel=1e-12)
        assert F[1, 2] == pytest.approx(-f, rel=1e-12)
        # (the call's energy holds the self energy as well)
        assert e - self_energy == pytest.approx(-ec / d, rel=1e-12, abs=1e-15 * abs(self_energy))
