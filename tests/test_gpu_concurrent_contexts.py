"""Contexts stepped by several host threads at once: each has its own streams, and the rebuild's cooperative kernels
of all of them share the GPU.  Every context gives the trajectory that it gives alone."""
import threading

import numpy as np
import pytest

from mfa_brush_gb300 import configs, md

pytestmark = pytest.mark.gpu


def _trajectory(p, rep, precision, use_graphs, calls, steps):
    s, t, r, v = rep
    with md.MdSystem(p, s, t, r, v, precision=precision, use_graphs=use_graphs, skin=0.15) as g:
        for _ in range(calls):
            g.step(steps)
        out = g.state()[:2]
        return out, g.rebuild_count()


@pytest.mark.parametrize("precision,use_graphs", [("mixed", True), ("mixed", False), ("fp64", True)])
def test_threads_do_not_disturb_each_other(precision, use_graphs):
    p = configs.wca_params()
    # sizes from one block of the sort to two per SM
    reps = [configs.brush_channel(L, 20.0, 0.1, 11, seed=k) for k, L in enumerate([10.0, 40.0, 100.0, 100.0])]
    calls, steps = (12, 25) if precision == "mixed" else (6, 15)
    alone = [_trajectory(p, rep, precision, use_graphs, calls, steps) for rep in reps]
    assert min(n for _, n in alone) > 10
    got, errors = [None] * len(reps), []

    def work(k):
        try:
            got[k] = _trajectory(p, reps[k], precision, use_graphs, calls, steps)
        except Exception as e:  # reported by the test's own thread
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(reps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (a, na), (b, nb) in zip(alone, got):
        assert na == nb
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
