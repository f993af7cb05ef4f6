"""The list build and the screening decide in FP32 on truncated fixed-point positions in both
precisions.  In a box of thousands of sigma the truncation is no longer far below the margin of a
normal box, so the thresholds widen with the box: no pair inside its cut-off may be lost."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("L,D", [(30.0, 20.0), (2500.0, 60.0)])
def test_pairs_at_the_cut_off(precision, uniform, L, D):
    inp = configs.two_liquid_inputs(f_x=0.0)
    f = inp.flags
    f.poiseuille = f.profiles = 0
    f.thermostat = 1  # conservative forces only
    if not uniform:  # brush-brush pairs keep their own range
        f.brush_in_good_sv = 1
    else:
        f.brush_in_good_sv = 0
    p, _ = md.derive(inp)
    rc = np.sqrt(p.table("range_2")[2, 2])
    rng = np.random.default_rng(7)
    # isolated pairs just inside the cut-off, in random directions, at random places
    n = 300 if L > 100 else 12
    centre = []
    while len(centre) < n:
        c = rng.uniform([0, 0, 8.0], [L, L, D - 8.0])
        d = np.array(centre) - c if centre else np.full((1, 3), 99.0)
        d[:, :2] -= L * np.round(d[:, :2] / L)
        if np.min(np.linalg.norm(d, axis=1)) > 6.0:
            centre.append(c)
    u = rng.standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    # the fixed point resolves L / 2^32 (6e-7 sigma at 2500); the pairs sit 4e-5 inside
    half = 0.5 * (rc - 4e-5) * u
    r = np.concatenate([np.array(centre) - half, np.array(centre) + half])
    r[:, :2] %= L
    s = abi.System()
    s.boundary[0] = s.boundary[1] = L
    s.boundary[2] = D
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d = 1, 2 * n
    s.n_mon_e = s.n_chain_e = 0
    s.n_mon_tot = s.n_part = 2 * n
    s.s_time, s.seed = 1, 5
    with md.MdSystem(p, s, np.full(2 * n, 3, np.int32), r, precision=precision, skin=0.4) as g:
        g.zero_force()
        e = g.fluid_fluid()[0][0]
        F = g.state()[3]
        assert len(g.pair_list()) == n
    eps4, sig2 = p.table("epsil")[2, 2], p.table("sigma_2")[2, 2]
    s6 = (sig2 / (rc - 4e-5) ** 2) ** 3
    want = eps4 * (12 * s6 * s6 - 6 * s6) / (rc - 4e-5)  # along r_i - r_j
    # one lost pair would change a force by its whole size; the distance carries the rounding of
    # the positions (2 x 2^-52 x 2500) and, in mixed precision, of the fixed point (L / 2^32)
    tol = 1e-9 if precision == "fp64" else 1e-5
    assert np.allclose(F[:n], -want * u, atol=tol * abs(want) * 10)
    assert np.allclose(F[n:], want * u, atol=tol * abs(want) * 10)
    assert e == pytest.approx(n * eps4 * (s6 * s6 - s6 - p.table("e_shift")[2, 2]), abs=n * 1e-5)
