"""An error that the caller's own CUDA calls left behind is not taken for one of the library's: set-up, steps,
uploads, skin checks and energy reads go on."""
import ctypes

import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu


def _runtimes():
    paths = {l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l}
    return [ctypes.CDLL(p) for p in paths]


def _leave_an_error():
    for rt in _runtimes():
        assert rt.cudaSetDevice(9999) != 0
        assert rt.cudaPeekAtLastError() != 0


@pytest.fixture(autouse=True)
def _no_error_for_the_next_test():
    yield
    for rt in _runtimes():
        rt.cudaGetLastError()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_calls_go_on(gpu, precision):
    p = configs.wca_params()
    s, t, r, v = configs.brush_channel(11.0, 13.0, 0.1, 11, seed=7)

    def run(leave):
        leave()
        with md.MdSystem(p, s, t, r, v, precision=precision, skin=0.4) as g:
            leave()
            g.step(12)  # captured
            leave()
            x = g.state()
            g.set_state(x[0], x[1])
            leave()
            rebuilt = abi.i32(0)
            assert g.lib.mfa_check_skin(g.ctx, ctypes.byref(rebuilt)) == 0
            leave()
            g.step(5)
            leave()
            return g.state()[0], g.energies()[0]["t_fluid"]

    a, b = run(_leave_an_error), run(lambda: None)
    assert np.array_equal(a[0], b[0]) and a[1] == pytest.approx(b[1], rel=1e-12)
