"""FP64 mode: pair forces against extended precision (numpy's long double: 64 or 113 bits), not only inside a gate but
as close as plain double arithmetic with the library's root, logarithm and cosine gives them."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from mfa_brush_gb300 import configs, md

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")
M32 = np.uint64(0xFFFFFFFF)


def _noise(seed, step, ta, tb):
    """Philox2x32-10 keyed on (seed, step), counter (min tag, max tag); Box-Muller on 23-bit uniforms."""
    h = seed & (2 ** 64 - 1)
    for mul in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
        h ^= h >> 33
        h = h * mul & (2 ** 64 - 1)
    h ^= h >> 33
    k = (h ^ step) & 0xFFFFFFFF
    c0, c1 = np.minimum(ta, tb).astype(np.uint64), np.maximum(ta, tb).astype(np.uint64)
    for r in range(10):
        if r:
            k = (k + 0x9E3779B9) & 0xFFFFFFFF
        p = c0 * np.uint64(0xD256D193)
        c0, c1 = (p >> np.uint64(32)) ^ np.uint64(k) ^ c1, p & M32
    u1 = ((c0 >> np.uint64(9)).astype(LD) + LD(0.5)) / LD(2 ** 23)
    u2 = (c1 >> np.uint64(9)).astype(LD) / LD(2 ** 23)
    return np.sqrt(LD(-2) * np.log(u1)) * np.cos(LD(2) * PI * u2)


def _forces(p, rep):
    s, t, r, v = rep
    L = np.array(s.boundary)
    rc = np.sqrt(max(p.range_2))
    box = np.array([L[0], L[1], 1e4])
    ij = cKDTree(np.mod(r, box), boxsize=box).query_pairs(rc * (1 + 1e-9), output_type="ndarray")
    i, j = ij[:, 0], ij[:, 1]
    d = r[i].astype(LD) - r[j].astype(LD)
    for c in range(2):
        d[:, c] -= L[c] * np.where(d[:, c] > L[c] / 2, 1, np.where(d[:, c] < -L[c] / 2, -1, 0))
    a, b = t[i] - 1, t[j] - 1
    tab = lambda name: p.table(name)[a, b].astype(LD)
    r2 = (d * d).sum(1)
    s2 = tab("sigma_2") / r2
    s6 = s2 ** 3
    fs = tab("epsil") * (12 * s6 * s6 - 6 * s6) / r2
    if p.flags.thermostat == 0:
        rr = np.sqrt(r2)
        wr = 1 - rr * np.sqrt(p.table("inv_range_2"))[a, b].astype(LD)
        rdot = ((v[i].astype(LD) - v[j].astype(LD)) * d).sum(1) / rr
        fs += (LD(p.sig) * wr * _noise(s.seed, s.s_time, i, j) - LD(p.friction1) * wr * wr * rdot) / rr
    fs[r2 >= tab("range_2")] = 0
    F = np.zeros(r.shape, LD)
    np.add.at(F, i, fs[:, None] * d)
    np.add.at(F, j, -fs[:, None] * d)
    return F


# Double arithmetic with the library's functions and multiply-add sums is 5.830e-16 and, with the thermostat (0),
# 5.364e-16 of the r.m.s. force off on these 24 channels (mean of their r.m.s. errors); sums of rounded products
# 5.857e-16, and with a noise of rounded tables as well 5.400e-16.  The bounds lie between.
@pytest.mark.parametrize("thermostat,bound", [(1, 5.843e-16), (0, 5.382e-16)])
def test_rms_error(thermostat, bound):
    assert np.finfo(LD).nmant >= 63
    p = md.derive(configs.wca_inputs(thermostat=1))[0] if thermostat else configs.wca_params()
    err = []
    for k in range(24):
        rep = configs.brush_channel(20.0, 20.0, 0.1, 11, seed=7 + k)
        want = _forces(p, rep)
        with md.MdSystem(p, *rep, precision="fp64", skin=0.4) as g:
            g.zero_force()
            g.fluid_fluid()
            f = g.state()[3]
        err.append(float(np.sqrt(((f - want) ** 2).mean() / (want ** 2).mean())))
    assert np.mean(err) <= bound
