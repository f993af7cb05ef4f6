"""A cell sort whose grid barrier runs out of patience: the call that reads the status returns an error,
no later sort or list builder touches the half-way counts, the context refuses further steps, and the
device stays usable.  The wait is made to run out by its limit: with none, all blocks but the last to
arrive give up."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _system(replicas=1):
    if replicas > 1:  # more than the shared work list holds
        reps = []
        for k in range(replicas):
            s = abi.System()
            s.boundary[0] = s.boundary[1] = s.boundary[2] = 8.0
            s.n_mon, s.n_chain, s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, 0, 1, 2, 0, 0
            s.n_mon_tot = s.n_part = 2
            s.s_time, s.seed = 1, 9 + k
            reps.append((s, np.full(2, 3, np.int32), np.array([[1.0, 1.0, 3.0], [2.0, 1.1, 3.1]]), np.zeros((2, 3))))
        return (configs.wca_params(),) + tuple(configs.concat(reps))
    return (configs.wca_params(),) + tuple(configs.brush_channel(12.0, 14.0, 0.1, 11, seed=7))


def _gives_up(call):
    with pytest.raises(abi.MfaError) as e:
        call()
    assert e.value.code == -2 and "barrier" in str(e.value)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("use_graphs", [True, False])
@pytest.mark.parametrize("replicas", [1, 1100])
def test_context_refuses_further_steps(precision, use_graphs, replicas):
    p, s, t, r, v = _system(replicas)
    opt = dict(precision=precision, use_graphs=use_graphs, skin=0.4)
    with md.MdSystem(p, s, t, r, v, **opt) as g:
        assert g.n > 1024  # several blocks of the sort
        g.step(5)
        ok = g.state()
        n0 = g.rebuild_count()
        assert g.lib.mfa_set_barrier_limit(g.ctx, -1) == -1
        assert g.lib.mfa_set_barrier_limit(g.ctx, 0) == 0
        moved = ok[0] + [0.5, 0.0, 0.0]
        _gives_up(lambda: g.set_state(moved, ok[1]))
        for _ in range(3):
            _gives_up(lambda: g.step(7))
        _gives_up(g.verlet_positions)
        _gives_up(g.synchronize)
        _gives_up(g.energies)
        assert g.lib.mfa_set_barrier_limit(g.ctx, 1 << 21) == 0  # the state stays lost
        _gives_up(lambda: g.set_state(moved, ok[1]))
        _gives_up(lambda: g.step(1))
        assert g.rebuild_count() == n0
    with md.MdSystem(p, s, t, r, v, **opt) as g:
        g.step(5)
        for a, b in zip(g.state(), ok):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("use_graphs", [True, False])
def test_within_a_call(use_graphs):
    """Steps issued together: the rebuilds after the one that gave up leave at once."""
    p, s, t, r, v = _system()
    with md.MdSystem(p, s, t, r, v, precision="mixed", use_graphs=use_graphs, skin=0.2) as g:
        g.step(40)
        g.synchronize()
        n0 = g.rebuild_count()
        assert n0 > 1
        assert g.lib.mfa_set_barrier_limit(g.ctx, 0) == 0
        g.step(60)
        _gives_up(g.synchronize)
        _gives_up(lambda: g.step(60))
        assert g.rebuild_count() == n0
