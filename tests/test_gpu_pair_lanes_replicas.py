"""The lanes-per-particle pair kernel with several replicas in one block of 32 particles: the bits of the
thread-per-particle kernel, energies and virial with their own replica."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _cluster(n, seed, L):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    s = abi.System()
    s.boundary[0], s.boundary[1], s.boundary[2] = L, L + 1.0, 11.0
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, n, 0, 0
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, 300 + seed
    return s, np.full(n, 3, np.int32), g * 0.97 + 1.5 + rng.uniform(-0.03, 0.03, (n, 3)), rng.standard_normal((n, 3))


@pytest.mark.parametrize("opt", [{}, {"energy_every": 1}, {"separate_integrator": True}])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 5, 7, 11), (31, 1, 33, 40, 2), (20, 20, 20, 20)])
def test_same_bits(sizes, opt):
    p = configs.wca_params()
    reps = [_cluster(n, 10 * k + n, 9.0 + k) for k, n in enumerate(sizes)]
    systems, t, r, v = configs.concat(reps)
    out = []
    for block in (0, 128):
        with md.MdSystem(p, systems, t, r, v, precision="mixed", skin=0.4, block_size=block, **opt) as g:
            g.step(11)
            a, e, w = g.state(), g.energies(), g.virial()
            g.md_step()  # the drop-in calls
            out.append((a + g.state(), e + g.energies(), w + g.virial()))
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x, y)
    # (FP32 partial sums of at most 40 particles grouped differently: 1e-6 of the largest term)
    for x, y in zip(out[0][1], out[1][1]):
        for k in ("v_fluid_fluid", "v_fluid_wall", "t_fluid", "e_total"):
            assert x[k] == pytest.approx(y[k], rel=2e-6, abs=1e-5)
    for x, y in zip(out[0][2], out[1][2]):
        assert np.allclose(x["total"], y["total"], rtol=0, atol=2e-6 * max(1.0, np.abs(y["pair"]).max()))
