"""The lanes-per-particle pair kernel of small systems gives the sums of the thread-per-particle one
(chosen by an explicit block size) to the bit: every model, energies on every step or not, the
separate integrator, drop-in calls, particle counts around its blocks of 32."""
import numpy as np
import pytest

from mfa_brush_gb300 import configs, md

pytestmark = pytest.mark.gpu


def _model(name):
    if name == "melt":
        p, rep = configs.melt_brush(14.0, 14.0, 0.1, 12, n_mon_d=6, rho=0.8, seed=3)
    elif name == "two_liquid":
        inp = configs.two_liquid_inputs(f_x=0.02)
        inp.flags.profiles = 0
        p, _ = md.derive(inp)
        rep = configs.two_liquid_channel(L=13.0, D=12.0, sigma_g=0.1, n_mon=9, seed=4)
    elif name == "walls":
        p = configs.wca_params(wall=1, dpd_cut_off=1.0)
        rep = configs.brush_channel(12.0, 12.0, 0.1, 9, seed=5, z_lo=1.0, wall_spacing=1.0)
    elif name == "charged":
        inp = configs.wca_inputs()
        inp.flags.system = 3
        inp.charge[1], inp.charge[2] = -1.0, 0.25
        inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, 4, 3.0
        p, _ = md.derive(inp)
        rep = configs.brush_channel(12.0, 12.0, 0.08, 8, rho=0.5, seed=6, max_fill=0.75)
    else:
        p, rep = configs.wca_params(), configs.brush_channel(11.0, 13.0, 0.1, 11, seed=7)
    return p, rep


def _run(p, rep, block, **opt):
    s, t, r, v = rep
    with md.MdSystem(p, s, t, r, v, precision="mixed", skin=0.4, block_size=block, **opt) as g:
        g.step(13)
        g.step(4)
        a = g.state()
        g.md_step()  # the drop-in calls
        return a, g.state(), g.energies()[0], g.virial()[0]


@pytest.mark.parametrize("opt", [{}, {"energy_every": 1}, {"separate_integrator": True}])
@pytest.mark.parametrize("name", ["wca", "melt", "two_liquid", "walls", "charged"])
def test_same_bits(name, opt):
    p, rep = _model(name)
    a, b = _run(p, rep, 0, **opt), _run(p, rep, 128, **opt)
    for x, y in zip(a[0] + a[1], b[0] + b[1]):
        assert np.array_equal(x, y)
    # (energies are FP32 partial sums grouped differently: 1e-6 of the largest term)
    for k in ("v_fluid_fluid", "v_fluid_wall", "v_intra_molec", "v_bend_melt", "t_fluid", "e_total"):
        assert a[2][k] == pytest.approx(b[2][k], rel=1e-6, abs=1e-5 * abs(b[2]["t_fluid"]))
    assert np.allclose(a[3]["total"], b[3]["total"], rtol=0, atol=1e-5 * np.abs(b[3]["total"]).max())


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 95])
def test_particle_counts(n):
    p, (s, t, r, v) = _model("two_liquid")
    s = type(s).from_buffer_copy(s)
    keep = np.sort(np.random.default_rng(n).permutation(np.arange(s.n_mon * s.n_chain, s.n_mon_tot))[:n])
    s.n_chain, s.n_mon = 0, 1
    s.n_chain_d, s.n_chain_e = int((t[keep] == 3).sum()), int((t[keep] == 4).sum())
    s.n_mon_tot = s.n_part = n
    rep = (s, t[keep], r[keep], v[keep])
    a, b = _run(p, rep, 0), _run(p, rep, 128)
    for x, y in zip(a[0] + a[1], b[0] + b[1]):
        assert np.array_equal(x, y)
