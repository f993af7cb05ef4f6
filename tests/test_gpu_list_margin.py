"""The list builder decides in FP32 on truncated positions: no pair inside the list cut-off may be lost.  Pairs are
put just inside it when the list is built, then brought just inside the interaction cut-off by moves a little
short of half a skin each, which rebuild nothing."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu

SKIN, INSIDE, SHORT = 0.4, 4e-5, 5e-6


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("L,D,few", [(30.0, 20.0, True), (30.0, 20.0, False), (2500.0, 60.0, True),
                                       (30.0, 2500.0, True)])
def test_pairs_at_the_list_cut_off(precision, uniform, L, D, few):
    inp = configs.two_liquid_inputs(f_x=0.0)
    f = inp.flags
    f.poiseuille = f.profiles = 0
    f.thermostat = 1  # conservative forces only
    f.brush_in_good_sv = 0 if uniform else 1
    p, _ = md.derive(inp)
    rc = np.sqrt(p.table("range_2")[2, 2])
    rng = np.random.default_rng(17)
    n = 12 if L < 100 else 300
    centre = []
    while len(centre) < n:
        c = rng.uniform([0, 0, 7.0], [L, L, D - 7.0])
        d = np.array(centre) - c if centre else np.full((1, 3), 99.0)
        d[:, :2] -= L * np.round(d[:, :2] / L)
        if np.min(np.linalg.norm(d, axis=1)) > 2 * (rc + SKIN):
            centre.append(c)
    u = rng.standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]

    def at(dist):
        r = np.concatenate([np.array(centre) - 0.5 * dist * u, np.array(centre) + 0.5 * dist * u])
        r[:, :2] %= L
        return r

    def system(r):
        s = abi.System()
        s.boundary[0] = s.boundary[1] = L
        s.boundary[2] = D
        s.n_mon, s.n_chain = 1, 0
        s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, len(r), 0, 0
        s.n_mon_tot = s.n_part = len(r)
        s.s_time, s.seed = 1, 5
        return s, np.full(len(r), 3, np.int32), r, np.zeros_like(r)

    # both forms of the list builder: several lanes per particle, and a thread per particle when there are more of
    # them than 2048 lanes per SM (beside the pairs a replica of beads on a lattice)
    reps = [system(at(rc + SKIN - INSIDE))]
    if not few:
        g = np.stack(np.meshgrid(*[np.arange(36)] * 3, indexing="ij"), -1).reshape(-1, 3) * 1.2 + 1.0
        s, t, r, v = system(g)
        s.boundary[0] = s.boundary[1] = s.boundary[2] = 36 * 1.2 + 1.0
        reps.append((s, t, r, v))
    systems, t, r0, v = configs.concat(reps)
    dist = rc + SKIN - INSIDE - 2 * (SKIN / 2 - SHORT)  # 3e-5 inside the interaction cut-off
    with md.MdSystem(p, systems, t, r0, v, precision=precision, skin=SKIN) as g:
        built = g.rebuild_count()
        r = r0.copy()
        r[: 2 * n] = at(dist)
        g.set_state(r)
        assert g.rebuild_count() == built
        g.zero_force()
        g.fluid_fluid()
        F = g.state()[3]
    s6 = (p.table("sigma_2")[2, 2] / dist ** 2) ** 3
    want = p.table("epsil")[2, 2] * (12 * s6 * s6 - 6 * s6) / dist
    # a lost pair has no force at all; the distance carries the rounding of the positions and, in mixed precision, of
    # the fixed point (L / 2^32) and FP32
    tol = 1e-8 if precision == "fp64" else 1e-4
    assert np.allclose(F[:n], -want * u, rtol=0, atol=tol * abs(want))
    assert np.allclose(F[n:2 * n], want * u, rtol=0, atol=tol * abs(want))
