"""Charged channels that are long in y: the k set then has hundreds of waves along y, and the rho kernels
must not need shared memory for all of them."""
import numpy as np
import pytest

from mfa_brush_gb300 import abi, configs, md

pytestmark = pytest.mark.gpu

PI = float(np.float32(3.1415926536))


def _channel(box, n, seed):
    rng = np.random.default_rng(seed)
    r = np.stack([rng.uniform(0, box[0], n), np.arange(n) * (box[1] / n) + rng.uniform(0, 0.2, n),
                  rng.uniform(1.0, box[2] - 1.0, n)], 1)
    s = abi.System()
    s.boundary[0], s.boundary[1], s.boundary[2] = box
    s.n_mon, s.n_chain = 1, 0
    s.n_mon_d, s.n_chain_d, s.n_mon_e, s.n_chain_e = 1, n - n // 2, 1, n // 2
    s.n_mon_tot = s.n_part = n
    s.s_time, s.seed = 1, seed
    return s, np.array([3] * (n - n // 2) + [4] * (n // 2), np.int32), r


def _params(n_kmax):
    inp = configs.wca_inputs(thermostat=1)
    inp.flags.system, inp.flags.particle_4 = 2, 1
    inp.inter4 = 1
    inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
    inp.charge[2], inp.charge[3] = 1.0, -1.0
    inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, n_kmax, 1.5
    return md.derive(inp)[0]


def _direct(p, box, q, r):
    """ewald_k.f90:37-202 in 64 bits: energy and forces over the half space of k."""
    dk = np.array([2 * PI / box[0], 2 * PI / box[1], 2 * PI / (3 * box[2])])
    kc = (dk[0] + dk[1]) * p.n_kmax / 2
    nm = (kc / dk).astype(int)
    x = [np.exp(1j * np.outer(np.arange(-nm[d], nm[d] + 1) * dk[d], r[:, d])) for d in range(3)]
    kx, ky = np.meshgrid(np.arange(-nm[0], nm[0] + 1), np.arange(-nm[1], nm[1] + 1), indexing="ij")
    V = 3 * box[0] * box[1] * box[2]
    U, F = 0.0, np.zeros_like(r)
    for kz in range(nm[2] + 1):
        k2 = (kx * dk[0]) ** 2 + (ky * dk[1]) ** 2 + (kz * dk[2]) ** 2
        take = k2 <= kc * kc
        if kz == 0:
            take &= (kx + ky >= 0) & ~((-kx == ky) & (ky > 0)) & ((kx != 0) | (ky != 0))
        a, b = np.nonzero(take)
        k = np.stack([kx[a, b] * dk[0], ky[a, b] * dk[1], np.full(len(a), kz * dk[2])], 1)
        G = np.exp(-k2[a, b] / (4 * p.alpha_c)) / k2[a, b]
        for c in range(0, len(a), 4096):  # (bounded memory)
            e = x[0][a[c:c + 4096]] * x[1][b[c:c + 4096]] * x[2][kz + nm[2]]
            rho = e @ q
            U += (G[c:c + 4096] * np.abs(rho) ** 2).sum()
            t = (np.conj(e) * rho[:, None]).imag * G[c:c + 4096, None]
            F += -8 * PI / V * q[:, None] * np.einsum("kp,kd->pd", t, k[c:c + 4096])
    return 4 * PI / V * U, F, nm


# the waves along y past which the columns of all of them are more than 227 KB of shared memory: about 170
# in FP64 (170 x 33 particles x two tiles x 16 bytes), 390 in mixed precision
@pytest.mark.parametrize("precision,box,n_kmax,more_than", [
    ("fp64", (10.0, 200.0, 20.0), 17, 170),   # the limb kernels (at most 15 waves along x)
    ("fp64", (20.0, 120.0, 8.0), 50, 150),    # the plain FP64 kernels
    ("mixed", (8.0, 400.0, 6.0), 17, 390),    # the dense kernels
    ("mixed", (9.0, 120.0, 6.0), 60, 390),    # the one-k-at-a-time force kernel
    ("fp64", (9.0, 90.0, 8.0), 9, 20),        # a few: blocks of rows over several planes of k
])
def test_many_waves_along_y(precision, box, n_kmax, more_than):
    p = _params(n_kmax)
    n = 48
    s, t, r = _channel(box, n, 3)
    q = np.where(t == 3, 1.0, -1.0)
    U, F, nm = _direct(p, box, q, r)
    assert nm[1] > more_than
    with md.MdSystem(p, s, t, r, precision=precision, skin=0.4) as g:
        g.zero_force()
        u = g.ewald_k()[0]
        f = g.state()[3]
    # 64 bits: the phases of the direct sum, of hundreds of turns, carry ~1e-13; FP32: the tile sums
    # (2^-24 of a sum of 32 terms) and the phases, times the cancellation in a force
    tol = 1e-10 if precision == "fp64" else 2e-6
    assert u == pytest.approx(U, rel=tol)
    assert np.abs(f - F).max() <= tol * 5 * np.abs(F).max()
