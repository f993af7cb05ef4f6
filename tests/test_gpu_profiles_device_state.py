"""The profile kernel's shared-memory opt-in belongs to a kernel on one device: every context makes its own, and
reports its failure, instead of relying on the first context of the process (which may be on another GPU).
The calls are counted, and made to fail, by a stand-in for cudaFuncSetAttribute in front of the runtime's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
int cudaFuncSetAttribute(const void* f, int attr, int value) {
  const char* refuse = getenv("FAKE_REFUSE");
  const char* lie = getenv("FAKE_LIE");
  fprintf(stderr, "opt-in %d\n", value);
  if (lie && atoi(lie) == value) return 0; /* and does nothing: the launches will fail */
  if (refuse && atoi(refuse) == value) return 1; /* cudaErrorInvalidValue */
  void* rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD); /* the one that the library brought in */
  return rt ? ((int (*)(const void*, int, int))dlsym(rt, "cudaFuncSetAttribute"))(f, attr, value) : 999;
}
"""

SCRIPT = r"""
import sys
import numpy as np
from mfa_brush_gb300 import configs, md

inp = configs.two_liquid_inputs(f_x=0.01)
inp.hist_dim = 1024
p = md.derive(inp)[0]
s, t, r, v = configs.two_liquid_channel(L=70.0, D=30.0, sigma_g=0.05, n_mon=6, seed=3)
out = []
for k in range(2):
    print("context", k, file=sys.stderr, flush=True)
    with md.MdSystem(p, s, t, r, v, precision="mixed", skin=0.4, energy_every=100) as g:
        assert g.n > 80000  # four particles a thread
        g.step(3)
        out.append(g.profiles()[0])
assert np.array_equal(*out) and out[0].sum() > 0
"""
BYTES = 1024 * 24 + 1024 * 36  # the velocities of a tile, three words a (bin, species)


def _run(tmp_path, **env):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, lib = str(tmp_path / "fake.c"), str(tmp_path / "libfake.so")
    with open(src, "w") as f:
        f.write(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, src, "-ldl"], check=True)
    return subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, LD_PRELOAD=lib, **env))


def test_every_context_opts_in(gpu, tmp_path):
    r = _run(tmp_path)
    assert r.returncode == 0, r.stderr
    first, second = r.stderr.split("context 1")
    line = "opt-in %d" % BYTES
    assert first.count(line) == second.count(line) > 0


def test_a_refused_opt_in_fails_the_context(gpu, tmp_path):
    r = _run(tmp_path, FAKE_REFUSE=str(BYTES))
    assert r.returncode != 0 and "MFA_ERR_CUDA" in r.stderr


def test_a_launch_that_fails_is_an_error_of_the_call(gpu, tmp_path):
    """The steps are captured as a graph: the failed launch must not be left out of it, nor end the process."""
    r = _run(tmp_path, FAKE_LIE=str(BYTES))
    assert r.returncode == 1 and "MFA_ERR_CUDA" in r.stderr, (r.returncode, r.stderr)
