"""z-profiles by a counting sort of each tile: one and many replicas per tile, tiles of both sizes, fine
and coarse bins, against sums over the states; and the one-pass profile step against the split one."""
import numpy as np
import pytest

from mfa_brush_gb300 import configs, md

pytestmark = pytest.mark.gpu


def _params(hist):
    inp = configs.two_liquid_inputs(f_x=0.01)
    inp.hist_dim = hist
    return md.derive(inp)[0]


def _expect(s, t, r, v, H):
    n0, n1 = s.n_mon * s.n_chain, s.n_mon * s.n_chain + s.n_mon_d * s.n_chain_d
    sp = np.where(np.arange(s.n_mon_tot) < n0, 0, np.where(np.arange(s.n_mon_tot) < n1, 1, 2))
    inv = 1.0 / (s.boundary[2] / H)
    z = np.clip((r[: s.n_mon_tot, 2] * inv).astype(int), 0, H - 1)
    d, vs, v2 = np.zeros((H, 3)), np.zeros((H, 3, 3)), np.zeros((H, 3, 3))
    np.add.at(d, (z, sp), 1.0)
    np.add.at(vs, (z, sp), v[: s.n_mon_tot])
    np.add.at(v2, (z, sp), v[: s.n_mon_tot] ** 2)
    return d, vs, v2


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("hist", [1, 7, 200, 1024])
@pytest.mark.parametrize("sizes", [(13.0,), (13.0, 11.0, 12.0, 11.5, 13.5), (70.0, 12.0)])
def test_profile_of_a_state(precision, hist, sizes):
    p = _params(hist)
    reps = [configs.two_liquid_channel(L=L, D=30.0 if L > 60 else 12.0, sigma_g=0.05, n_mon=6, seed=3 + k)
            for k, L in enumerate(sizes)]
    systems, t, r, v = configs.concat(reps)
    with md.MdSystem(p, systems, t, r, v, precision=precision, skin=0.4) as g:
        g.profiles_accumulate()
        g.profiles_accumulate()
        for k, (s, tt, rr, vv) in enumerate(reps):
            got, want = g.profiles(k)[:3], _expect(s, tt, rr, vv, hist)
            assert np.array_equal(got[0], 2 * want[0])
            for a, b in zip(got[1:], want[1:]):  # 64-bit sums of up to ~1e5 terms in another order
                assert np.allclose(a, 2 * b, rtol=0, atol=1e-11 * max(1.0, np.abs(b).max()))


@pytest.mark.parametrize("L", [13.0, 75.0])
def test_one_pass_step_equals_the_split_one(L):
    p = _params(200)
    s, t, r, v = configs.two_liquid_channel(L=L, D=24.0 if L > 60 else 12.0, sigma_g=0.05, n_mon=6, seed=5)
    out = []
    for every in (1000, 1):  # energies on every step keep the profile between two integrator kernels
        with md.MdSystem(p, s, t, r, v, precision="mixed", skin=0.4, energy_every=every) as g:
            g.step(9)
            out.append((g.state(), g.profiles(0)))
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    assert out[0][1][3] == out[1][1][3] == 9
    assert np.array_equal(out[0][1][0], out[1][1][0])
    for a, b in zip(out[0][1][1:3], out[1][1][1:3]):
        assert np.allclose(a, b, rtol=0, atol=1e-10 * np.abs(b).max())
