"""The FP64 pair kernel with four or eight lanes per particle (chosen by the particle count and the list
capacity) against one lane per particle (an explicit block size): the same pairs in the same order, so the
forces are the same bits; energies and virial are the same terms in another order of the sums."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _lattice(n, spacing, seed):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    s = abi.System()
    s.boundary[0] = s.boundary[1] = s.boundary[2] = max(12.0, m * spacing + 2.0)
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d = 1, n
    s.n_mon_e = s.n_chain_e = 0
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, 70 + seed
    return s, np.full(n, 3, np.int32), g * spacing + 1.0 + rng.uniform(-0.04, 0.04, (n, 3)), rng.standard_normal((n, 3))


def _run(p, reps, block, cap):
    systems, t, r, v = configs.concat(reps)
    with md.MdSystem(p, systems, t, r, v, precision="fp64", skin=0.4, block_size=block, nbr_capacity=cap) as g:
        g.zero_force()
        e = g.fluid_fluid()
        w = np.array([x["pair"] for x in g.virial()])
        return np.array(e), w, g.state()[3]


# (sizes, spacing, capacity): eight lanes up to 60 particles per entry of capacity, four above; in the long model
# 55 pairs a particle at 0.95 (a round of four lanes keeps 32) and 95 at 0.8 (of eight: 64)
@pytest.mark.parametrize("model,sizes,spacing,cap", [
    ("wca", (1,), 0.95, 64), ("wca", (3, 4, 5, 31, 33, 129), 0.95, 64), ("wca", (4001,), 0.95, 40),
    ("wca", (5, 2003, 1998, 7), 0.95, 40), ("long", (300,), 0.8, 256), ("long", (3, 290, 61), 0.8, 256),
    ("long", (13007,), 0.95, 144)])
def test_lanes_give_the_same_forces(model, sizes, spacing, cap):
    if model == "long":  # 2 * 2^(1/6) sigma
        inp = configs.two_liquid_inputs(f_x=0.0)
        inp.flags.poiseuille = inp.flags.profiles = 0
        p, _ = md.derive(inp)
    else:
        p = configs.wca_params()
    reps = [_lattice(n, spacing, 10 * k + n) for k, n in enumerate(sizes)]
    e1, w1, f1 = _run(p, reps, 32, cap)
    e, w, f = _run(p, reps, 0, cap)
    assert np.array_equal(f, f1)
    # up to 10^6 terms of both signs: 1e-12 of the largest
    assert np.abs(e - e1).max() <= 1e-12 * max(1.0, np.abs(e1).max())
    assert np.abs(w - w1).max() <= 1e-12 * max(1.0, np.abs(w1).max())
