"""Mixed precision: the tables of the k-space sum keep the relative precision of small phases.  A pair of opposite
charges 1e-6 sigma apart near x = 0: every rho(k) is the sine of a phase of 1e-7 turns."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu

PI = float(np.float32(3.1415926536))


@pytest.mark.parametrize("n_kmax", [5, 34])  # the dense force kernels and the others
@pytest.mark.parametrize("gap", [1e-3, 1e-5, 1e-6])
def test_energy_of_a_tiny_dipole(n_kmax, gap):
    inp = configs.wca_inputs(thermostat=1)
    inp.flags.system, inp.flags.particle_4 = 2, 1
    inp.inter4 = 1
    inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
    inp.charge[2], inp.charge[3] = 1.0, -1.0
    inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, n_kmax, 2.0
    p = md.derive(inp)[0]
    box = np.array([9.0, 10.0, 12.0])
    s = abi.System()
    s.boundary[0], s.boundary[1], s.boundary[2] = box
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, 1, 1, 1
    s.n_mon_tot = s.n_part = 2
    s.s_time, s.seed = 1, 3
    r = np.array([[3.0, 3.0, 4.0]] * 2)
    r[:, 0] = 0.0, gap
    with md.MdSystem(p, s, np.array([3, 4], np.int32), r, precision="mixed", skin=0.4) as g:
        g.zero_force()
        u = g.ewald_k()[0]
    dk = np.array([2 * PI / box[0], 2 * PI / box[1], 2 * PI / (3 * box[2])])
    kc = (dk[0] + dk[1]) * n_kmax / 2
    nm = (kc / dk).astype(int)
    n = np.stack(np.meshgrid(*[np.arange(-m, m + 1) for m in nm], indexing="ij"), -1).reshape(-1, 3)
    k = n * dk
    k2 = (k * k).sum(1)
    keep = (k2 <= kc * kc) & (n[:, 2] >= 0) & (k2 > 0)
    keep &= (n[:, 2] > 0) | ((n[:, 0] + n[:, 1] >= 0) & ~((-n[:, 0] == n[:, 1]) & (n[:, 1] > 0)))
    k, k2 = k[keep], k2[keep]
    # |1 - exp(i k gap)|^2 = 4 sin^2(k gap / 2), without cancellation
    want = 4 * PI / (3 * box.prod()) * (np.exp(-k2 / (4 * p.alpha_c)) / k2 * 4 * np.sin(k[:, 0] * gap / 2) ** 2).sum()
    # the rows' factors q Y Z are equal and opposite, and rho their product with the difference of the X, whose real
    # parts cancel exactly: four FP32 roundings (along y or z the products with Z would round first; cos = 1 - phase^2 / 2 has an
    # error of 2^-25, beside a sine of 1e-3 at the largest gap 3e-5 of it; none of it at the others)
    assert u == pytest.approx(want, rel=2e-6 if gap < 1e-4 else 1e-4, abs=0.0)
