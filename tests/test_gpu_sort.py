"""The cell sort: cells denser than their tag buckets, more replicas than the shared work list holds,
replicas of one particle, lists equal to brute force."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _free(r, L, D, seed):
    n = len(r)
    s = abi.System()
    s.boundary[0] = s.boundary[1] = L
    s.boundary[2] = D
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d = 1, n
    s.n_mon_e = s.n_chain_e = 0
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, 77 + seed
    return s, np.full(n, 3, np.int32), r, np.zeros((n, 3))


def _brute(r, L, rc):
    d = r[:, None] - r[None]
    d[..., :2] -= L * np.round(d[..., :2] / L)
    i, j = np.nonzero((d * d).sum(-1) < rc * rc)
    return {(a, b) for a, b in zip(i.tolist(), j.tolist()) if a < b}


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("dense", [False, True])
def test_lists_equal_brute_force(precision, dense):
    rng = np.random.default_rng(3)
    p = configs.wca_params()
    rc = np.sqrt(max(p.range_2))
    reps = []
    for k, (n, L, D) in enumerate([(700, 14.0, 11.0), (1, 9.0, 9.0), (333, 9.0, 30.0), (64, 40.0, 10.0)]):
        r = rng.uniform([0, 0, 0.8], [L, L, D - 0.8], (n, 3))
        if dense:  # half of them within one cell's reach of each other: far more than a bucket holds
            r[: n // 2] = [L - 0.2, 0.1, D / 2] + rng.uniform(-0.5, 0.5, (n // 2, 3))
            r[:, :2] %= L
        reps.append(_free(r, L, D, k))
    systems, a_type, r0, v = configs.concat(reps)
    with md.MdSystem(p, systems, a_type, r0, v, precision=precision, skin=0.4, nbr_capacity=420) as g:
        for k, (s, _, r, _) in enumerate(reps):
            got = {tuple(sorted(x)) for x in g.pair_list(k).tolist()}
            want = _brute(r, s.boundary[0], rc)
            # a pair within 1e-9 of the cut-off may count either way
            edge = _brute(r, s.boundary[0], rc + 1e-9) - _brute(r, s.boundary[0], rc - 1e-9)
            assert got ^ want <= edge
        # the caller's order comes back whatever the slot order
        assert np.array_equal(g.state()[0], r0)


@pytest.mark.parametrize("n_rep", [1023, 1025, 1500])
def test_more_replicas_than_the_shared_work_list(n_rep):
    p = configs.wca_params()
    rng = np.random.default_rng(5)
    reps = []
    for k in range(n_rep):
        n = 1 + k % 3
        r = np.array([[1.0, 1.0, 3.0]]) + np.arange(n)[:, None] * [1.0, 0.1, 0.05] + rng.uniform(0, 0.02, (n, 3))
        reps.append(_free(r, 8.0, 8.0, k))
    systems, a_type, r0, v = configs.concat(reps)
    with md.MdSystem(p, systems, a_type, r0, v, precision="fp64", skin=0.4) as g:
        g.step(40)
        r = g.state()[0]
        counts = g.replica_rebuild_counts()
    at = np.concatenate([[0], np.cumsum([len(x[2]) for x in reps])])
    assert counts.max() > 0
    for k in (0, 1, 2, n_rep // 2, n_rep - 2, n_rep - 1):
        s, t, rr, vv = reps[k]
        with md.MdSystem(p, s, t, rr, vv, precision="fp64", skin=0.4) as one:
            one.step(40)
            assert np.array_equal(one.state()[0], r[at[k]:at[k + 1]])
            assert one.replica_rebuild_counts()[0] == counts[k]
