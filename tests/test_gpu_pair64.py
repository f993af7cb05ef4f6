"""The FP64 pair kernel puts a warp's kept pairs together: particle counts around the warp and block
edges, warps that span replicas, kept counts below and above a round, explicit wall beads."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _cluster(n, L, D, spacing, seed, n_wall=0):
    """n free beads on a jittered cubic lattice around the middle of the box, n_wall fixed ones at z = 0."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    r = g * spacing + 1.0 + rng.uniform(-0.04, 0.04, (n, 3))
    if n_wall:
        w = np.stack([1.0 + spacing * (np.arange(n_wall) % 4), 1.0 + spacing * (np.arange(n_wall) // 4),
                      np.zeros(n_wall)], 1)
        r = np.concatenate([r, w])
    s = abi.System()
    s.boundary[0] = s.boundary[1] = L
    s.boundary[2] = D
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d = 1, n
    s.n_mon_e = s.n_chain_e = 0
    s.n_mon_tot, s.n_part = n, n + n_wall
    s.s_time, s.seed = 1, 1000 + seed
    a_type = np.array([3] * n + [4] * n_wall, np.int32)
    v = rng.standard_normal((n + n_wall, 3))
    v[n:] = 0
    return s, a_type, r, v


@pytest.mark.parametrize("model", ["wca", "long", "walls"])
@pytest.mark.parametrize("sizes", [(1,), (31,), (33,), (1, 2, 31, 33, 127, 129), (128, 128), (300,)])
def test_forces_and_energies(oracle_mod, model, sizes):
    n_wall = 0
    if model == "long":  # 2 * 2^(1/6) sigma: tens of kept pairs a particle
        inp = configs.two_liquid_inputs(f_x=0.0)
        inp.flags.poiseuille = inp.flags.profiles = 0
        p, _ = md.derive(inp)
        L, D, a = 12.0, 12.0, 0.95
    elif model == "walls":
        p = configs.wca_params(wall=1, dpd_cut_off=1.0)
        L, D, a, n_wall = 12.0, 12.0, 0.95, 7
    else:
        p = configs.wca_params()
        L, D, a = 12.0, 12.0, 0.95
    reps = [_cluster(n, L, D, a, 10 * k + n, n_wall) for k, n in enumerate(sizes)]
    systems, a_type, r0, v = configs.concat(reps)
    with md.MdSystem(p, systems, a_type, r0, v, precision="fp64", skin=0.4) as g:
        g.zero_force()
        e = g.fluid_fluid()[0]
        F = g.state()[3]
        W = g.virial()
    at = 0
    for k, (s, t, r, vv) in enumerate(reps):
        o = oracle_mod.Oracle(p, s, t, r, vv)
        o.zero_force()
        o.fluid_fluid()
        Fo, m = o.state()[3], s.n_mon_tot
        # 64-bit sums of at most ~60 terms: a few 1e-16 of the largest force each
        assert np.allclose(F[at:at + m], Fo[:m], rtol=0, atol=1e-12 * max(1.0, np.abs(Fo).max()))
        assert e[k] == pytest.approx(o.energies()["v_fluid_fluid"], rel=1e-12, abs=1e-12)
        # the pair virial's trace is sum F_i r_i over isolated (non-wrapping) clusters of free beads
        if not n_wall:
            assert np.trace(W[k]["pair"]) == pytest.approx((Fo * r).sum(), rel=1e-9, abs=1e-8)
        at += s.n_part
