"""The calls whose speed this framework is judged by: channels of polymer brushes advanced through
`MdSystem` and the C ABI under it, over the range that its users run.

A pass advances every replica by `steps` MD steps and reads a frame back: positions, velocities and
accelerations of every particle, and the energies of every replica.  (The two models with the long
LJ cut-off, whose force jumps there, give positions and velocities: whether one pair in 10^7 counts
in the last step's acceleration is decided below FP32's resolution.)  Successive passes continue the
trajectory, as a production run does (`how` "roundtrip" uploads the state first on every pass, as a
host program that owns the state does).  Frames of the mixed-precision mode, whose forces are FP32,
are kept in single precision, as trajectory files are; the FP64 mode's are kept in double.

    listed()            the fixed cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) the context a user's program holds, made from the seed
    run(state)          one pass
    work(case)          bytes and operations that a pass cannot do without
    exact(case, seed)   what the first pass returns, from plain torch in 64 bits
"""
import ctypes
import functools
import math

import numpy as np
import torch

from mfa_brush_gb300 import abi, configs, md

SKIN = 0.5  # the skin that the tuner picks for these densities


def listed():
    return [
        # the smallest call: one reference-scale channel advanced by the md_main subroutines one by
        # one, each returning its energy to the host, as the Fortran host program calls them
        dict(name="dropin_channel", model="wca", how="dropin", precision="mixed", replicas=1, L=20.0, D=20.0,
             sigma_g=0.1, n_mon=30, rho=0.8, steps=1),
        # the same channel through the fused step: a small system, bound by latency and launches
        dict(name="small_channel", model="wca", how="step", precision="mixed", replicas=1, L=20.0, D=20.0,
             sigma_g=0.1, n_mon=30, rho=0.8, steps=20),
        # the reference's own kind of run: 20^3, explicit wall beads, own DPD cut-off, plain FP64
        dict(name="walls_fp64", model="walls", how="step", precision="fp64", replicas=1, L=20.0, D=20.0,
             sigma_g=0.1, n_mon=30, rho=0.8, steps=10),
        # a small parameter study in the FP64 mode: 16 uneven channels in one batch
        dict(name="replicas16_fp64", model="replicas", how="step", precision="fp64", replicas=16, shapes=2024,
             steps=10),
        # an ordinary study: 32 uneven channels batched in mixed precision
        dict(name="replicas32", model="replicas", how="step", precision="mixed", replicas=32, shapes=2024, steps=20),
        # the headline workload: 256 uneven channels, 4.66 M particles
        dict(name="replicas256", model="replicas", how="step", precision="mixed", replicas=256, shapes=2024,
             steps=20),
        # a host program that owns the state: upload, ten steps, read back
        dict(name="roundtrip64", model="replicas", how="roundtrip", precision="mixed", replicas=64, shapes=2024,
             steps=10),
        # one large melt in brush: long cut-off, cosine bending, chains everywhere (340 k particles)
        dict(name="melt_brush", model="melt", how="step", precision="mixed", replicas=1, L=100.0, D=40.0,
             sigma_g=0.2, n_mon=50, rho=0.85, steps=20),
        # one large two-liquid Poiseuille channel with z-profiles on every step (1.6 M particles)
        dict(name="two_liquid", model="two_liquid", how="step", precision="mixed", replicas=1, L=200.0, D=50.0,
             sigma_g=0.15, n_mon=30, rho=0.8, steps=10),
        # the charged brush with the slab Ewald sum (33.6 k particles, 8070 k-vectors)
        dict(name="charged_brush", model="charged", how="step", precision="mixed", replicas=1, L=40.0, D=30.0,
             sigma_g=0.1, n_mon=40, rho=0.7, n_kmax=12, steps=10),
        # the same in the FP64 mode, the reference point of a charged run
        dict(name="charged_fp64", model="charged", how="step", precision="fp64", replicas=1, L=40.0, D=30.0,
             sigma_g=0.1, n_mon=40, rho=0.7, n_kmax=12, steps=4),
        # a batch of small charged channels (a salt or grafting study)
        dict(name="charged_batch", model="charged", how="step", precision="mixed", replicas=12, L=16.0, D=16.0,
             sigma_g=0.08, n_mon=20, rho=0.6, n_kmax=6, steps=10),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["channel", "channel", "walls", "replicas", "replicas", "replicas", "melt", "two_liquid",
                       "charged", "charged"])
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    big = precision == "mixed"
    if kind == "channel":
        return dict(model="wca", how=rng.choice(["step", "dropin"]), precision=precision, replicas=1,
                    L=round(_log(rng, 12.0, 60.0 if big else 40.0), 2), D=round(rng.uniform(10.0, 40.0), 2),
                    sigma_g=round(rng.uniform(0.05, 0.15), 3), n_mon=rng.randint(10, 30), rho=0.8,
                    steps=rng.randint(1, 20))
    if kind == "walls":
        return dict(model="walls", how="step", precision=precision, replicas=1, L=round(_log(rng, 12.0, 40.0), 2),
                    D=round(rng.uniform(12.0, 24.0), 2), sigma_g=0.1, n_mon=rng.randint(10, 25), rho=0.8,
                    steps=rng.randint(5, 20))
    if kind == "replicas":
        return dict(model="replicas", how=rng.choice(["step", "step", "roundtrip"]), precision=precision,
                    replicas=int(round(_log(rng, 2, 256 if big else 24))), shapes=rng.randint(1, 9999),
                    steps=rng.randint(8, 20) if big else 10)
    if kind == "melt":
        return dict(model="melt", how="step", precision=precision, replicas=1,
                    L=round(_log(rng, 16.0, 100.0 if big else 40.0), 2), D=round(rng.uniform(16.0, 40.0), 2),
                    sigma_g=round(rng.uniform(0.1, 0.2), 3), n_mon=rng.randint(15, 40), rho=0.85,
                    steps=rng.randint(5, 20) if big else 5)
    if kind == "two_liquid":
        return dict(model="two_liquid", how="step", precision=precision, replicas=1,
                    L=round(_log(rng, 20.0, 200.0 if big else 40.0), 2), D=round(rng.uniform(16.0, 50.0), 2),
                    sigma_g=round(rng.uniform(0.08, 0.15), 3), n_mon=rng.randint(10, 30), rho=0.8,
                    steps=rng.randint(5, 10))
    n = rng.choice([1, 1, rng.randint(2, 16)])
    return dict(model="charged", how="step", precision=precision, replicas=n,
                L=round(_log(rng, 12.0, 40.0 if n == 1 else 20.0), 2), D=round(rng.uniform(12.0, 30.0 if n == 1 else 20.0), 2),
                sigma_g=round(rng.uniform(0.05, 0.1), 3), n_mon=rng.randint(10, 40 if n == 1 else 20), rho=0.65,
                n_kmax=rng.randint(5, 12 if n == 1 else 7), steps=rng.randint(4, 10) if big else 3)


# ---- configurations ----------------------------------------------------------------------------
def _charge(rep, seed):
    """Turns a neutral channel into the charged brush of configs.charged_brush: four charges' worth
    on each chain's non-head beads, as many +1 counterions among the free beads (type 4, stored last)."""
    s, a_type, r0, v = rep
    n_brush = s.n_mon * s.n_chain
    free = np.arange(n_brush, s.n_mon_tot)
    n_ci = min(4 * s.n_chain, len(free) // 2)
    ci = np.sort(np.random.default_rng(seed + 1).choice(free, n_ci, replace=False))
    solv = np.setdiff1d(free, ci)
    order = np.concatenate([np.arange(n_brush), solv, ci])
    a_type, r0, v = a_type[order].copy(), r0[order].copy(), v[order].copy()
    a_type[n_brush + len(solv):] = 4
    s.n_mon_d, s.n_chain_d = 1, len(solv)
    s.n_mon_e, s.n_chain_e = 1, n_ci
    return (s, a_type, r0, v), -float(n_ci) / max(1, s.n_chain * (s.n_mon - 1))


@functools.lru_cache(maxsize=2)
def _base(key):
    """(mfa_params, [(System, a_type, r0, v)]) of a case's sizes: lattice starts of the generators."""
    c = dict(key)
    kind, n = c["model"], c["replicas"]
    if kind == "replicas":
        return configs.wca_params(), configs.replicas(n, c["shapes"])
    if kind == "walls":
        p = configs.wca_params(wall=1, dpd_cut_off=1.0)
        return p, [configs.brush_channel(c["L"], c["D"], c["sigma_g"], c["n_mon"], rho=c["rho"], seed=1, z_lo=1.0,
                                         wall_spacing=1.0)]
    if kind == "melt":
        p, rep = configs.melt_brush(c["L"], c["D"], c["sigma_g"], c["n_mon"], rho=c["rho"])
        return p, [rep]
    if kind == "two_liquid":
        p, _ = md.derive(configs.two_liquid_inputs(f_x=0.01))
        return p, [configs.two_liquid_channel(c["L"], c["D"], c["sigma_g"], c["n_mon"], rho=c["rho"], seed=3)]
    if kind == "charged":
        reps, q = [], 0.0
        for k in range(n):
            rep = configs.brush_channel(c["L"], c["D"], c["sigma_g"], c["n_mon"], rho=c["rho"], seed=41 + k,
                                        max_fill=0.75)
            rep, q = _charge(rep, 41 + k)
            reps.append(rep)
        inp = configs.wca_inputs()
        inp.flags.system, inp.flags.particle_4 = 3, 1
        inp.inter4 = 1
        inp.a_w4, inp.sigma_w4 = inp.a_w, inp.sigma_w
        inp.charge[1], inp.charge[3] = q, 1.0
        inp.alpha_c, inp.n_kmax, inp.rc_coul = 0.81, c["n_kmax"], 3.0
        p, _ = md.derive(inp)
        return p, reps
    return configs.wca_params(), [configs.brush_channel(c["L"], c["D"], c["sigma_g"], c["n_mon"], rho=c["rho"],
                                                        seed=1 + k) for k in range(n)]


def _inputs(case, seed):
    """(params, systems, a_type, r0, v): the lattice starts moved by a random x, y shift each, with
    Maxwell velocities (heads and wall beads at rest) and noise keys of the seed."""
    p, reps = _base(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "how", "precision", "steps"))))
    rng = np.random.default_rng([int(seed), 77])
    systems, types, pos, vel = [], [], [], []
    for s, a_type, r0, _ in reps:
        s = type(s).from_buffer_copy(s)
        s.seed = int(rng.integers(1, 2**63 - 1))
        L = np.array([s.boundary[0], s.boundary[1]])
        r = r0.copy()
        r[:, :2] += rng.uniform(0.0, 1.0, 2) * L
        r[:, :2] -= L * (r[:, :2] >= L)
        v = rng.standard_normal((s.n_part, 3))
        v[s.n_mon_tot:] = 0.0
        v[: s.n_mon * s.n_chain : max(1, s.n_mon)] = 0.0
        systems.append(s)
        types.append(a_type)
        pos.append(r)
        vel.append(v)
    return p, systems, np.concatenate(types).astype(np.int32), np.concatenate(pos), np.concatenate(vel)


# ---- the pass ----------------------------------------------------------------------------------
def _pointer(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), abi.dp)


def _parts(case):
    return "rv" if case["model"] in ("melt", "two_liquid") else "rva"


def prepare(case, seed):
    p, systems, a_type, r0, v = _inputs(case, seed)
    g = md.MdSystem(p, systems, a_type, r0, v, precision=case["precision"], skin=SKIN, energy_every=10)
    n = len(a_type)
    st = dict(g=g, how=case["how"], steps=case["steps"], mixed=case["precision"] == "mixed",
              profiles=bool(p.flags.profiles), energies=(abi.Energies * len(systems))())
    # the frame: page-locked buffers that the library copies into
    parts = _parts(case)
    st["frame"] = [torch.empty((n, 3), dtype=torch.float64, pin_memory=True) for _ in parts]
    st["kept"] = [torch.empty((n, 3), dtype=torch.float32) for _ in parts] if st["mixed"] else None
    if st["how"] == "roundtrip":
        st["mine"] = [torch.from_numpy(x).pin_memory() for x in (r0, v, np.zeros_like(v))]
    return st


def run(st):
    g, lib = st["g"], st["g"].lib
    if st["how"] == "roundtrip":
        abi.check(lib.mfa_set_state(g.ctx, *[_pointer(t) for t in st["mine"]]), g.ctx)
    if st["how"] == "dropin":
        for _ in range(st["steps"]):
            e = g.md_step()
        e = np.array([[r[k] for k, _ in abi.Energies._fields_[1:]] for r in e])
    else:
        g.step(st["steps"])
        abi.check(lib.mfa_get_energies(g.ctx, st["energies"]), g.ctx)
        e = np.frombuffer(st["energies"], np.float64).reshape(g.nrep, -1)[:, 1:].copy()
    frame = st["frame"]
    abi.check(lib.mfa_sync_to_host(g.ctx, *([_pointer(t) for t in frame] + [None] * (4 - len(frame)))), g.ctx)
    if st["mixed"]:
        for kept, t in zip(st["kept"], frame):
            kept.copy_(t)
        frame, e = st["kept"], e.astype(np.float32)
    out = dict(zip("rva", frame), energies=e)
    if st["profiles"]:
        h = g.profiles(0)[:3]
        for k, x in zip(("dens", "vsum", "v2sum"), h):
            out[k] = x.astype(np.float32) if st["mixed"] else x
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    p, reps = _base(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "how", "precision", "steps"))))
    n = sum(r[0].n_part for r in reps)
    steps = case["steps"]
    # the state in and the frame out, once; a state that no cache holds (129 MB) moves every step
    state = 48 * n
    nbytes = 24 * (3 + len(_parts(case))) * n + (2 * state * (steps - 1) if state > 129e6 else 0)
    rc = math.sqrt(max(p.range_2))
    flops = 0.0
    for s, _, _, _ in reps:
        pairs = 0.5 * s.n_mon_tot * s.n_part / (s.boundary[0] * s.boundary[1] * s.boundary[2]) * 4.19 * rc**3
        flops += steps * (60.0 * pairs + 60.0 * s.n_mon_tot)  # LJ + DPD of each pair once; bonds, walls, drift
        if case["model"] == "charged":
            nk = 0.5 * 4.19 * case["n_kmax"] ** 3 * 3.0 * s.boundary[2] / s.boundary[0]
            nq = s.n_chain * (s.n_mon - 1) + s.n_chain_e
            flops += steps * nk * nq * 12.0  # rho and the force with the +-kx symmetry
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits, plain torch ------------------------------------------------------------
PI_F = float(np.float32(3.1415926536))  # the reference's single-precision literal
M32 = 0xFFFFFFFF


def _key(seed, step):
    h = seed & (2**64 - 1)
    for mul in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
        h ^= h >> 33
        h = h * mul & (2**64 - 1)
    h ^= h >> 33
    return (h ^ step) & M32


def _gauss(key, ta, tb):
    """Philox2x32-10 on (min tag, max tag), Box-Muller on 23-bit uniforms."""
    c0, c1, k, m = torch.minimum(ta, tb), torch.maximum(ta, tb), key.clone(), 0xD256D193
    for r in range(10):
        if r:
            k = (k + 0x9E3779B9) & M32
        hi = (m * (c0 >> 16) + ((m * (c0 & 0xFFFF)) >> 16)) >> 16
        lo = (m * c0) & M32
        c0, c1 = hi ^ k ^ c1, lo
    u1 = ((c0 >> 9).double() + 0.5) / 2.0**23
    u2 = (c1 >> 9).double() / 2.0**23
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)


def _pairs(r, L, rc):
    """Index pairs i < j of one replica within rc: cells at least rc wide, x and y periodic."""
    dev = r.device
    nc = [max(1, int(L[d] / rc)) for d in range(3)]
    if min(nc[0], nc[1]) < 3:
        d = r[:, None] - r[None]
        d[..., :2] -= L[:2] * torch.round(d[..., :2] / L[:2])
        i, j = torch.nonzero((d * d).sum(-1) < rc * rc, as_tuple=True)
        return i[i < j], j[i < j]
    c = torch.stack([(r[:, d] / L[d] * nc[d]).long().clamp(0, nc[d] - 1) for d in range(3)], 1)
    cell = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=nc[0] * nc[1] * nc[2])
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    rank = torch.empty_like(cell)
    rank[order] = torch.arange(len(r), device=dev) - start[cell[order]]
    table = torch.full((len(count), most), -1, dtype=torch.long, device=dev)
    table[cell, rank] = torch.arange(len(r), device=dev)
    me, got_i, got_j = torch.arange(len(r), device=dev), [], []
    for dz in (-1, 0, 1):
        z = c[:, 2] + dz
        for dy in (-1, 0, 1):
            y = (c[:, 1] + dy) % nc[1]
            for dx in (-1, 0, 1):
                x = (c[:, 0] + dx) % nc[0]
                j = table[(z.clamp(0, nc[2] - 1) * nc[1] + y) * nc[0] + x]
                j = torch.where(((z >= 0) & (z < nc[2]))[:, None] & (j > me[:, None]), j, -1)
                i = me[:, None].expand_as(j)[j >= 0]
                j = j[j >= 0]
                d = r[i] - r[j]
                d[:, :2] -= L[:2] * torch.round(d[:, :2] / L[:2])
                keep = (d * d).sum(1) < rc * rc
                got_i.append(i[keep])
                got_j.append(j[keep])
    return torch.cat(got_i), torch.cat(got_j)


class _Exact:
    def __init__(self, case, seed):
        self.p, self.systems, a_type, r0, v = _inputs(case, seed)
        p, dev = self.p, "cuda" if torch.cuda.is_available() else "cpu"
        f64 = dict(dtype=torch.float64, device=dev)
        self.dev, self.case, self.f64 = dev, case, f64
        n = len(a_type)
        self.type = torch.from_numpy(a_type.astype(np.int64) - 1).to(dev)
        self.r, self.v = torch.tensor(r0, **f64), torch.tensor(v, **f64)
        self.a = torch.zeros_like(self.r)
        size = [s.n_part for s in self.systems]
        self.p0 = np.concatenate([[0], np.cumsum(size)[:-1]])
        self.rep = torch.repeat_interleave(torch.arange(len(size), device=dev), torch.tensor(size, device=dev))
        self.L = torch.tensor([list(s.boundary) for s in self.systems], **f64)
        self.Li = self.L[self.rep]
        mob, head = np.zeros(n, bool), np.zeros(n, bool)
        first, second, angle = [], [], []  # bonds; (a, b, c) angles with the owner kind
        kind = []
        species = np.full(n, 3)
        for q, s in zip(self.p0, self.systems):
            mob[q:q + s.n_mon_tot] = True
            b = q
            for sp, (m, c) in enumerate(((s.n_mon, s.n_chain), (s.n_mon_d, s.n_chain_d), (s.n_mon_e, s.n_chain_e))):
                t = b + np.arange(m * c).reshape(c, m)
                species[b:b + m * c] = sp
                if sp == 0 and c:
                    head[t[:, 0]] = True
                if m > 1 and c:
                    first.append(t[:, :-1].ravel())
                    second.append(t[:, 1:].ravel())
                if m > 2 and c:
                    angle.append(np.stack([t[:, :-2].ravel(), t[:, 1:-1].ravel(), t[:, 2:].ravel()]))
                    kind.append(np.full(angle[-1].shape[1], sp))
                b += m * c
        cat = lambda x: torch.from_numpy(np.concatenate(x) if x else np.zeros(0, np.int64)).to(dev)  # noqa: E731
        self.mob, self.head = torch.from_numpy(mob).to(dev), torch.from_numpy(head).to(dev)
        self.species = torch.from_numpy(species).to(dev)
        self.b0, self.b1 = cat(first), cat(second)
        self.ang = torch.from_numpy(np.concatenate(angle, 1)).to(dev) if angle else None
        self.akind = cat(kind)
        tab = lambda x: torch.tensor(list(x), **f64)  # noqa: E731
        self.range2, self.eps4 = tab(p.range_2), tab(p.epsil)
        self.sig2, self.shift = tab(p.sigma_2), tab(p.e_shift)
        self.mass, self.charge = tab(p.mass_type), tab(p.charge)
        self.charged = p.flags.system in (2, 3)
        self.q = self.charge[self.type]
        self.rc = math.sqrt(max(max(p.range_2), p.r_cut_dpd_2, p.rc_coul_2 if self.charged else 0.0))
        self.local = torch.arange(n, device=dev) - torch.from_numpy(self.p0).to(dev)[self.rep]
        self.list_at = None
        self.done = 0

    def lists(self):
        """Pairs within rc + 0.6, renewed when a particle has moved 0.3."""
        if self.list_at is not None:
            d = self.r - self.list_at
            d[:, :2] -= self.Li[:, :2] * torch.round(d[:, :2] / self.Li[:, :2])
            if float((d * d).sum(1).max()) < 0.09:
                return
        gi, gj = [], []
        for k, s in enumerate(self.systems):
            q = int(self.p0[k])
            i, j = _pairs(self.r[q:q + s.n_part], self.L[k], self.rc + 0.6)
            gi.append(i + q)
            gj.append(j + q)
        self.i, self.j = torch.cat(gi), torch.cat(gj)
        self.list_at = self.r.clone()

    def per_rep(self, x, who):
        return torch.zeros(len(self.systems), **self.f64).index_add_(0, self.rep[who], x)

    def bond(self, a, b):
        d = self.r[a] - self.r[b]
        d[:, :2] -= self.Li[a, :2] * torch.round(d[:, :2] / self.Li[a, :2])
        return d

    def forces(self, energies):
        p, fl, R = self.p, self.p.flags, len(self.systems)
        F, E = torch.zeros_like(self.r), {}
        self.lists()
        i, j = self.i, self.j
        d = self.bond(i, j)
        r2 = (d * d).sum(1)
        near = r2 < self.rc**2
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        k = self.type[i] * abi.MAXT + self.type[j]
        lj = r2 < self.range2[k]
        s2 = self.sig2[k] / r2
        s6 = s2**3
        zero = torch.zeros_like(r2)
        fs = torch.where(lj, self.eps4[k] * (12.0 * s6 * s6 - 6.0 * s6) / r2, zero)
        E["ff"] = self.per_rep(torch.where(lj, self.eps4[k] * (s6 * s6 - s6 - self.shift[k]), zero), i)
        wall = torch.zeros_like(lj)
        if fl.wall == 1:
            wall = (self.type[i] == p.n_type - 1) | (self.type[j] == p.n_type - 1)
        if fl.thermostat == 0:
            if p.r_cut_dpd_2 == 0.0:
                dpd, rc = lj & ~wall, torch.sqrt(self.range2[k])
            else:
                dpd = (r2 < p.r_cut_dpd_2) & (self.type[i] != 0) & (self.type[j] != 0) & ~wall
                rc = torch.full_like(r2, math.sqrt(p.r_cut_dpd_2))
            w = torch.nonzero(dpd)[:, 0]
            iw, jw, dw = i[w], j[w], d[w]
            rr = torch.sqrt(r2[w])
            wr = 1.0 - rr / rc[w]
            keys = torch.tensor([_key(s.seed, s.s_time + self.done) for s in self.systems], device=self.dev)
            g = _gauss(keys[self.rep[iw]], self.local[iw], self.local[jw])
            rdot = ((self.v[iw] - self.v[jw]) * dw).sum(1) / rr
            fs[w] += (p.sig * wr * g - p.friction1 * wr * wr * rdot) / rr
        E["coul"] = torch.zeros(R, **self.f64)
        if self.charged:
            qq = self.q[i] * self.q[j]
            c = torch.nonzero((qq != 0.0) & (r2 < p.rc_coul_2))[:, 0]
            rr, qq = torch.sqrt(r2[c]), qq[c]
            erfc = torch.erfc(p.sqrt_alpha * rr)
            E["coul"] += self.per_rep(qq * erfc / rr, i[c])
            fs[c] += (qq * p.sqrt_alpha * p.inv_sqrt_pi * 2.0 * torch.exp(-p.alpha_c * r2[c]) / rr
                      + qq * erfc / r2[c]) / rr
        f = fs[:, None] * d
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        # FENE
        d = self.bond(self.b0, self.b1)
        x = (d * d).sum(1) * p.inv_r_chain_2
        f = (-p.k_chain / (1.0 - x) * p.inv_r_chain_2)[:, None] * d
        F.index_add_(0, self.b0, f)
        F.index_add_(0, self.b1, -f)
        E["intra"] = self.per_rep(-0.5 * p.k_chain * torch.log(1.0 - x), self.b0)
        # cosine bending
        for name, on, sp in (("bend", fl.bending, 0), ("bendm", fl.bending_melt, 1)):
            E[name] = torch.zeros(R, **self.f64)
            if not on or self.ang is None:
                continue
            a, b, c = self.ang[:, self.akind == sp]
            u, w = self.bond(b, a), self.bond(c, b)
            nu, nw = u.norm(dim=1, keepdim=True), w.norm(dim=1, keepdim=True)
            u, w = u / nu, w / nw
            cos = (u * w).sum(1, keepdim=True)
            gu, gw = (w - cos * u) / nu, (u - cos * w) / nw  # gradients of the cosine
            F.index_add_(0, a, -p.k_bend * gu)
            F.index_add_(0, b, p.k_bend * (gu - gw))
            F.index_add_(0, c, p.k_bend * gw)
            E[name] = self.per_rep(p.k_bend * (1.0 - cos[:, 0]), a)
        # 9-3 walls and the body force
        E["fw"] = torch.zeros(R, **self.f64)
        if fl.wall == 2:
            m = torch.nonzero(self.mob)[:, 0]
            t = self.type[m]
            sw, aw = torch.tensor(list(p.sigma_wall), **self.f64)[t], torch.tensor(list(p.a_wall), **self.f64)[t]
            for z, sign in ((self.r[m, 2], 1.0), (self.Li[m, 2] - self.r[m, 2], -1.0)):
                x = (sw / z) ** 3
                E["fw"] += self.per_rep(aw.abs() * x**3 - p.a_w * x, m)
                F[m, 2] += sign * (9.0 * aw.abs() * x**3 - 3.0 * aw * x) / z
        if fl.poiseuille:
            g = self.mass[self.type] * (self.type != 0) * self.mob
            F += g[:, None] * torch.tensor(list(p.const_force), **self.f64)
        if self.charged:
            self.ewald(F, E)
        F[~self.mob] = 0.0
        return F, E

    def ewald(self, F, E):
        p = self.p
        for n, s in enumerate(self.systems):
            q0 = int(self.p0[n])
            who = torch.nonzero(self.q[q0:q0 + s.n_mon_tot])[:, 0] + q0
            q, r = self.q[who], self.r[who]
            L = list(s.boundary)
            dk = [2.0 * PI_F * (1.0 / L[0]), 2.0 * PI_F * (1.0 / L[1]), 2.0 * PI_F / (L[2] + 2.0 * L[2])]
            kc = (dk[0] + dk[1]) * p.n_kmax / 2.0
            m = [int(kc / x) for x in dk]
            nx, ny, nz = np.meshgrid(np.arange(-m[0], m[0] + 1), np.arange(-m[1], m[1] + 1), np.arange(m[2] + 1),
                                     indexing="ij")
            a, b, c = nx * dk[0], ny * dk[1], nz * dk[2]
            k2 = a * a + b * b + c * c
            keep = (k2 <= kc * kc) & (k2 > 0) & ~((nz == 0) & (nx + ny < 0)) & ~((nz == 0) & (-nx == ny) & (ny > 0))
            kv = torch.tensor(np.stack([a[keep], b[keep], c[keep]], 1), **self.f64)
            k2 = (kv * kv).sum(1)
            G = torch.exp(-k2 / (4.0 * p.alpha_c)) / k2
            inv_V = 1.0 / (L[0] * L[1] * 3.0 * L[2])
            fk = torch.zeros_like(r)
            for lo in range(0, len(kv), 1024):
                k, g = kv[lo:lo + 1024], G[lo:lo + 1024]
                # (the phase in turns, reduced before the sine: kv / (2 pi) is n / L up to the literal)
                ph = 2.0 * math.pi * torch.remainder(r @ (k / (2.0 * math.pi)).T, 1.0)
                co, si = torch.cos(ph), torch.sin(ph)
                re, im = q @ co, q @ si
                E["coul"][n] += 4.0 * PI_F * inv_V * (g * (re * re + im * im)).sum()
                fk += (co * (g * im) - si * (g * re)) @ k
            F[who] -= 8.0 * PI_F * inv_V * q[:, None] * fk
            mz = (q * (r[:, 2] - L[2] / 2.0)).sum()
            E["coul"][n] += 2.0 * PI_F * mz * mz * inv_V - (q * q).sum() * p.sqrt_alpha / math.sqrt(PI_F)
            F[who, 2] -= 4.0 * PI_F * inv_V * mz * q

    def step(self, last, profile):
        p = self.p
        m = self.mob[:, None]
        self.r = torch.where(m, self.r + p.dt * self.v + 0.5 * p.dt**2 * self.a, self.r)
        xy, L = self.r[:, :2], self.Li[:, :2]
        self.r[:, :2] = torch.where(xy > L, xy - L, torch.where(xy < 0.0, xy + L, xy))
        self.v = self.v + 0.5 * p.dt * self.a
        F, E = self.forces(last)
        self.a = F / self.mass[self.type][:, None]
        self.a[self.head] = 0.0
        self.v = self.v + 0.5 * p.dt * self.a
        self.v[self.head] = 0.0
        self.done += 1
        if profile is not None:
            H = len(profile)
            w = torch.nonzero(self.mob & (self.species < 3))[:, 0]
            z = ((self.r[w, 2] * (H / self.Li[w, 2])).long()).clamp(0, H - 1)
            v = self.v[w]
            profile.view(H * 3, 7).index_add_(0, z * 3 + self.species[w], torch.cat([torch.ones_like(v[:, :1]), v, v * v], 1))
        return E

    def energies(self, E):
        p, fl, S = self.p, self.p.flags, self.systems
        who = torch.arange(len(self.r), device=self.dev)
        kin = self.per_rep(0.5 * self.mass[self.type] * (self.v**2).sum(1) * self.mob, who)
        D = self.L[:, 2]
        ww = 2.0 * (abs(p.a_w) * (p.sigma_w / D) ** 9 - p.a_w * (p.sigma_w / D) ** 3) if fl.wall == 2 else 0.0 * D
        total = ww + E["fw"] + E["ff"] + E["intra"] + E["bend"] + E["bendm"] + E["coul"]
        inv_n = torch.tensor([1.0 / (s.n_mon_tot - (0 if fl.system == 2 else s.n_chain)) for s in S], **self.f64)
        cols = [E["ff"], E["fw"], ww, E["intra"], E["bend"], E["bendm"], 0.0 * D, E["coul"], kin, total, total + kin, inv_n]
        return torch.stack(cols, 1)


def exact(case, seed):
    x = _Exact(case, seed)
    prof = torch.zeros((x.p.hist_dim, 3, 7), **x.f64) if x.p.flags.profiles else None
    for k in range(case["steps"]):
        E = x.step(k == case["steps"] - 1, prof)
    out = {k: getattr(x, k).cpu() for k in _parts(case)}
    out["energies"] = x.energies(E).cpu()
    if prof is not None and case["how"] != "dropin":
        prof = prof.cpu()
        out.update(dens=prof[:, :, 0].contiguous(), vsum=prof[:, :, 1:4].contiguous(), v2sum=prof[:, :, 4:].contiguous())
    return out
