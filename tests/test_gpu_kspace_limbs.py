"""FP64 mode: the k-space sums in integer limbs (up to 15 waves per axis, the plain FP64 kernels above)
and the tabulated real-space Coulomb factors against the oracle, far below the 1e-9 gate."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _system(n, L, D, seed, spread=1.0):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    r = 1.0 + g * ((min(L, D) - 2.0) / m) * spread + rng.uniform(-0.05, 0.05, (n, 3))
    s = abi.System()
    s.boundary[0], s.boundary[1], s.boundary[2] = L, L * 1.1, D
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d = 1, n - n // 2
    s.n_mon_e, s.n_chain_e = 1, n // 2
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, 9 + seed
    return s, np.array([3] * (n - n // 2) + [4] * (n // 2), np.int32), r, np.zeros((n, 3))


def _params(n_kmax, q3, q4, rc=3.0):
    inp = configs.wca_inputs(thermostat=1)
    inp.flags.system, inp.flags.particle_4 = 2, 1
    inp.inter4 = 1
    inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
    inp.charge[2], inp.charge[3] = q3, q4
    inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, n_kmax, rc
    return md.derive(inp)[0]


@pytest.mark.parametrize("n_kmax", [2, 7, 14, 15, 17])
@pytest.mark.parametrize("n,q3,q4", [(2, 1.0, -1.0), (31, 0.3, -2.5), (130, 1.0, -1.0), (513, 1e-3, -7.0)])
def test_kspace_against_the_oracle(oracle_mod, n_kmax, n, q3, q4):
    p = _params(n_kmax, q3, q4)
    s, t, r, v = _system(n, 12.0, 13.0, n)
    o = oracle_mod.Oracle(p, s, t, r, v)
    o.ewald_init()
    o.zero_force()
    uo = o.ewald_k()
    Fo, Wo = o.state()[3], o.virial()["kspace"]
    with md.MdSystem(p, s, t, r, v, precision="fp64", skin=0.4) as g:
        g.zero_force()
        u = g.ewald_k()[0]
        F, W = g.state()[3], g.virial()[0]["kspace"]
    # both sum the same terms in 64 bits; the oracle's phases alone carry ~1e-14
    assert u == pytest.approx(uo, rel=1e-11)
    for q in (3, 4):  # each charge against its own kind: a small charge next to a large one
        assert np.abs(F - Fo)[t == q].max() <= 1e-11 * np.abs(Fo[t == q]).max()
    assert np.abs(W - Wo).max() <= 1e-11 * np.abs(Wo).max()


@pytest.mark.parametrize("alpha", [0.81, 4.0])
@pytest.mark.parametrize("rc", [0.8, 3.0, 5.0])
def test_real_space_factors(oracle_mod, rc, alpha):
    """Pairs from inside the table's start to the cut-off, one pair per distance."""
    p = _params(3, 1.0, -1.0, rc)
    p.alpha_c, p.sqrt_alpha = alpha, np.sqrt(alpha)
    dist = np.concatenate([np.linspace(0.55, min(rc, 1.2), 40), np.linspace(0.69, 0.71, 9),
                           np.linspace(0.8, rc * (1 - 1e-9), 60)])
    dist = dist[dist < rc]
    n = len(dist)
    L = 13.0 * np.ceil(np.sqrt(n))
    m = int(np.ceil(np.sqrt(n)))
    base = np.stack([(np.arange(n) % m) * 13.0 + 5.0, (np.arange(n) // m) * 13.0 + 5.0, np.full(n, 6.0)], 1)
    u = np.random.default_rng(2).standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    r = np.concatenate([base, base + dist[:, None] * u])
    s = abi.System()
    s.boundary[0] = s.boundary[1] = L
    s.boundary[2] = 14.0
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, n, 1, n
    s.n_mon_tot = s.n_part = 2 * n
    s.s_time, s.seed = 1, 3
    t = np.array([3] * n + [4] * n, np.int32)
    o = oracle_mod.Oracle(p, s, t, r, np.zeros_like(r))
    o.zero_force()
    o.fluid_fluid()
    Fo = o.state()[3]
    with md.MdSystem(p, s, t, r, precision="fp64", skin=0.4) as g:
        g.zero_force()
        g.fluid_fluid()
        F = g.state()[3]
    # WCA and Coulomb of one pair; the minimum image of the positions carries 1e-15 x 150 sigma
    assert np.all(np.linalg.norm(F - Fo, axis=1) <= 1e-11 * np.linalg.norm(Fo, axis=1) + 1e-13)
