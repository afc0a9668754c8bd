"""The work a program has this library do, as cases that can be timed: steps
of molecular dynamics with each polarization model and precision, a
constant-pressure step, the reference's own non-Ewald mode, an energy analysis
and a training step through the adjoint.

A case names a box (waters, Na+/Cl- pairs, edge, PME grid), the settings of a
context and the call:

  step      new coordinates in, energies and gradients out (amg_set_coords,
            amg_forward on the program's own gradient arrays), the call of an
            MD program at every time step
  pressure  the same with the virial, then the same atoms in a slightly
            larger box: two consecutive steps under pressure coupling, which
            changes the box at every step
  analyze   one evaluation with everything a structure analysis prints:
            energies per atom, pair counts, gradients, dipoles, multipoles
  train     an evaluation with dipoles, then the adjoint with cotangents of the
            energy and of both dipole sets: gradients of the parameters

Coordinates, box and cotangents are host data (the C ABI takes and returns
host arrays); a program keeps them in pinned memory.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from polmdqc_b200 import abi, systems
from polmdqc_b200.engine import OPT_COEF, Engine, Settings
from polmdqc_b200.prm import COULOMB

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
VOLUME = 29.88        # A^3 per water in the 32,768-water box (99.3 A)
SPACING = 1.085       # PME grid points per A in the 4,096- and 32,768-water boxes
MODELS = {"mutual": abi.POL_MUTUAL, "direct": abi.POL_DIRECT, "opt4": abi.POL_OPT, "none": abi.POL_NONE}
GRAD = abi.DO_ENERGY | abi.DO_GRADIENT
JITTER = 0.3          # A, of the sites of the water lattice


def case(name, call, waters, box, grid, pairs=0, model="mutual", precision="mixed", ewald=True, cutoff=7.0):
    return {"name": name, "call": call, "waters": waters, "pairs": pairs, "box": box, "grid": grid, "model": model,
            "precision": precision, "ewald": ewald, "cutoff": cutoff}


def listed():
    return [
        # the smallest production box (a solvated ion or a test molecule): launch latency
        case("step_216", "step", 216, 18.643, 24),
        # a ragged box a few nanometres wide, as a solvated small molecule has
        case("step_1500", "step", 1500, 35.52, 40),
        # the common size of a solvated protein domain
        case("step_4096", "step", 4096, 49.7, 54),
        # the largest box: a solvated protein complex
        case("step_32768", "step", 32768, 99.3, 108),
        # the same step in FP64: reference trajectories, energy-conservation checks; ions among the waters
        case("step_ions_fp64", "step", 8000, 62.1, 72, pairs=22, precision="fp64"),
        # the cheap polarization models: screening and equilibration runs
        case("step_direct", "step", 19683, 83.8, 90, model="direct"),
        case("step_opt4", "step", 6859, 58.96, 64, model="opt4"),
        # constant pressure: the virial, and a box that changes at every step
        case("pressure_4096", "pressure", 4096, 49.7, 54),
        # the reference's own electrostatics mode (no Ewald, no polarization), FP64, cutoff 9 A
        case("multipoles_fp64", "step", 13824, 74.5, 0, model="none", precision="fp64", ewald=False, cutoff=9.0),
        # a structure analysis, as the reference's analyze program asks for it
        case("analyze_2744", "analyze", 2744, 43.5, 48, precision="fp64"),
        # fitting parameters to energies and induced dipoles of an ion solution
        case("train_ions", "train", 8000, 62.1, 72, pairs=22),
    ]


def smooth_even(x):
    """The smallest even grid size of factors 2, 3 and 5 that is at least x."""
    k = max(16, 2 * math.ceil(x / 2))
    while True:
        m = k
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return k
        k += 2


def draw(rng):
    call = rng.choice(["step"] * 6 + ["pressure", "analyze", "train", "train"])
    model = rng.choice(["mutual"] * 5 + ["direct", "opt4", "none"]) if call in ("step", "analyze") else "mutual"
    precision = rng.choice(["mixed", "mixed", "fp64"])
    ewald = model != "none" or rng.random() < 0.5
    cutoff = 7.0 if ewald else 9.0
    top = {"pressure": 6000, "analyze": 6000, "train": 9000}.get(call, 14000 if precision == "fp64" else 30000)
    low = 216 if cutoff < 8 else 300
    waters = int(round(math.exp(rng.uniform(math.log(low), math.log(top)))))
    pairs = rng.choice([0, 0, max(1, waters // 360)])
    box = round(((waters + 3 * pairs) * VOLUME * rng.uniform(1.0, 1.04)) ** (1 / 3), 3)
    grid = smooth_even(SPACING * box) if ewald else 0
    c = case("", call, waters, box, grid, pairs, model, precision, ewald, cutoff)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
@dataclasses.dataclass
class Tiled(systems.System):
    """A System of many copies of few molecules: its lists as CSR arrays."""
    tiled: dict = None

    def csr(self, name):
        return self.tiled[name]


def rows(s, first, count, copies, at):
    """`copies` of the atoms first..first+count of s, the first copy at atom `at`."""
    off = np.repeat(at + count * np.arange(copies), count)
    num = at + np.arange(count * copies)
    pick = first + np.tile(np.arange(count), copies)

    def axis(a):
        a = np.asarray(a)[pick]
        return np.where(a > 0, a - first + off, 0).astype(np.int32)

    d = {k: np.asarray(getattr(s, k))[pick] for k in ("types", "pole", "polaxe", "polarity", "thole", "pdamp")}
    d.update(zaxis=axis(s.zaxis), xaxis=axis(s.xaxis), yaxis=axis(s.yaxis), num=num)
    lists = {}
    for k, v in s.lists.items():
        own = [np.asarray(v[first + a], np.int64) - first for a in range(count)]
        n = np.tile([len(o) for o in own], copies)
        one = np.concatenate(own) if own else np.zeros(0, np.int64)
        base = np.repeat(at + count * np.arange(copies), len(one))
        lists[k] = (n, np.tile(one, copies) + base)
    return d, lists


@functools.lru_cache(maxsize=4)
def topology(waters, pairs):
    """The parameters of `waters` waters followed by `pairs` Na+/Cl- pairs
    (water03, or amoebabio18 with ions), without coordinates."""
    s = systems.ion_solution(n_waters=8, n_pairs=1, box_len=14.0) if pairs else systems.water_box(8, 9.3)
    parts = [rows(s, 0, 3, waters, 0)]
    if pairs:
        parts.append(rows(s, 24, 2, pairs, 3 * waters))
    join = lambda k: np.concatenate([p[0][k] for p in parts])  # noqa: E731
    n = 3 * waters + 2 * pairs
    tiled = {}
    for k in s.lists:
        off = np.zeros(n + 1, np.int32)
        off[1:] = np.cumsum(np.concatenate([p[1][k][0] for p in parts]))
        tiled[k] = (off, np.concatenate([p[1][k][1] for p in parts]).astype(np.int32))
    mol = np.concatenate([np.repeat(np.arange(waters), 3), waters + np.arange(2 * pairs)]).astype(np.int32)
    return Tiled(n=n, xyz=np.zeros((n, 3)), types=join("types"), names=[], bonds=[], pole=join("pole"),
                 zaxis=join("zaxis"), xaxis=join("xaxis"), yaxis=join("yaxis"), polaxe=join("polaxe"), molcule=mol,
                 polarity=join("polarity"), thole=join("thole"), pdamp=join("pdamp"), lists={},
                 m_scale=s.m_scale, p_scale=s.p_scale, p_iscale=s.p_iscale, d_scale=s.d_scale, u_scale=s.u_scale,
                 box=np.zeros(6), use_bounds=True, prm_name=s.prm_name, tiled=tiled)


def coordinates(waters, pairs, box, seed):
    """Liquid-like coordinates: O and ions on random sites of a jittered
    lattice, uniform random orientations, redrawn while an H comes within
    1.7 A of another molecule."""
    rng = np.random.default_rng(seed)
    side = math.ceil((waters + 2 * pairs) ** (1 / 3) - 1e-9)
    a = box / side
    sites = np.sort(rng.permutation(side ** 3)[:waters + 2 * pairs])
    take = rng.permutation(len(sites))
    sites = np.concatenate([np.sort(sites[take[:waters]]), sites[take[waters:]]])
    grid = np.stack(np.unravel_index(sites, (side,) * 3), -1)
    where = np.full(side ** 3, -1)
    where[sites] = np.arange(len(sites))
    center = (grid + 0.5) * a + rng.uniform(-JITTER, JITTER, (len(sites), 3)) * (np.arange(len(sites)) < waters)[:, None]
    step = np.array([(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) != (0, 0, 0)])
    near = where[np.ravel_multi_index(np.moveaxis((grid[:waters, None] + step) % side, -1, 0), (side,) * 3)]
    at = torch.from_numpy(np.repeat(center[:, None], 3, 1)).to(DEVICE)  # [molecule, atom, xyz]; ions three times
    near = torch.from_numpy(near).to(DEVICE)
    redo = np.arange(waters)
    for _ in range(60):
        new = systems.water_geometry(center[redo], systems.random_rotations(rng, len(redo)))
        at[torch.from_numpy(redo).to(DEVICE), 1:] = torch.from_numpy(new).to(DEVICE)
        other = at[near.clamp(min=0)]                                    # [water, neighbour, atom, xyz]
        d = at[:waters, None, 1:, None] - other[:, :, None]              # from this water's two H
        d = d - box * torch.round(d / box)
        close = (d.square().sum(-1).amin((-1, -2)) < 1.7 ** 2) & (near >= 0)
        # of two waters in contact the later one turns; one at an ion always does
        later = (near < torch.arange(waters, device=DEVICE)[:, None]) | (near >= waters)
        redo = torch.nonzero((close & later).any(1) | hit_by_later(close, later, near, waters)).flatten().cpu().numpy()
        if not len(redo):
            break
    at = at.cpu().numpy()
    return np.ascontiguousarray(np.concatenate([at[:waters].reshape(-1, 3), center[waters:]]))


def hit_by_later(close, later, near, waters):
    """Waters that an earlier water's H touches: the earlier one reports the contact, the later one turns."""
    hit = torch.zeros(waters, dtype=torch.bool, device=close.device)
    hit[near[close & ~later]] = True
    return hit


def system_of(c, seed):
    xyz = coordinates(c["waters"], c["pairs"], c["box"], seed)
    return dataclasses.replace(topology(c["waters"], c["pairs"]), xyz=xyz, box=np.array([c["box"]] * 3 + [90.0] * 3))


def grown(c, xyz):
    """The atoms and the box after a step of the barostat: every molecule moved with its centre, 0.1% per edge."""
    w, scale = 3 * c["waters"], 1.001
    out = xyz * scale
    mol = xyz[:w].reshape(-1, 3, 3)
    out[:w] = (mol + (scale - 1) * mol.mean(1, keepdims=True)).reshape(-1, 3)
    return out, np.array([c["box"] * scale] * 3 + [90.0] * 3)


def cotangents(n, seed):
    rng = np.random.default_rng(seed + 7)
    return 0.7, 0.1 * rng.standard_normal((n, 3)), 0.1 * rng.standard_normal((n, 3))


def pinned(a):
    """A host array in pinned memory."""
    t = torch.from_numpy(np.array(a, np.float64).reshape(-1))
    return t.pin_memory().numpy() if DEVICE == "cuda" else t.numpy()


def prepare(case, seed):
    c = case
    s = system_of(c, seed)
    st = Settings(use_ewald=c["ewald"], nfft=(c["grid"],) * 3, cutoff=c["cutoff"], poltyp=MODELS[c["model"]],
                  precision=abi.PREC_MIXED if c["precision"] == "mixed" else abi.PREC_FP64)
    state = {"call": c["call"], "engine": Engine(s, st), "xyz": pinned(s.xyz), "box": s.box,
             "dem": pinned(np.zeros(3 * s.n)), "dep": pinned(np.zeros(3 * s.n))}
    if c["call"] == "pressure":
        xyz, box = grown(c, s.xyz)
        state.update(xyz2=pinned(xyz), box2=box)
    if c["call"] == "train":
        state["cotangents"] = [x if isinstance(x, float) else pinned(x) for x in cotangents(s.n, seed)]
    return state


def run(state):
    e, dem, dep = state["engine"], state["dem"], state["dep"]
    if state["call"] == "step":
        dem.fill(0.0)
        dep.fill(0.0)
        e.set_coords(state["xyz"])
        em, ep, _, _ = e.forward_into(GRAD, dem, dep)
        return {"em": em, "ep": ep, "dem": dem, "dep": dep}
    if state["call"] == "pressure":
        out = []
        for xyz, box in ((state["xyz"], state["box"]), (state["xyz2"], state["box2"])):
            e.set_coords(xyz, box)
            out.append(plain(e.forward(GRAD | abi.DO_VIRIAL), "em", "ep", "dem", "dep", "vir"))
        return out
    e.set_coords(state["xyz"])
    if state["call"] == "analyze":
        r = e.forward(GRAD | abi.DO_ANALYSIS | abi.DO_DIPOLES)
        return plain(r, "em", "ep", "einter", "nem", "nep", "aem", "aep", "dem", "dep", "uind", "uinp", "rpole")
    r = e.forward(abi.DO_ENERGY | abi.DO_DIPOLES)
    return {**plain(r, "em", "ep", "uind", "uinp"), **e.backward(*state["cotangents"])}


def plain(r, *names):
    return {k: getattr(r, k) for k in names}


# ------------------------------------------------------------------- floor
def work(case):
    """Bytes and operations of one pass: host arrays in and out once, the
    site records once; one pair evaluation per pair within the cutoff and
    term (multipoles ~220 operations, permanent field ~120, polarization
    forces ~300, one dipole field ~30 per iteration and dipole set), spline
    stencils (125 points) and the transforms of the PME grids."""
    c = case
    n = 3 * c["waters"] + 2 * c["pairs"]
    pairs = 0.5 * n * (4 / 3 * math.pi * c["cutoff"] ** 3 * n / c["box"] ** 3)
    iters = {"mutual": 9, "opt4": 4, "direct": 0, "none": 0}[c["model"]]
    solves = 1
    flops = pairs * 220
    if c["model"] != "none":
        flops += pairs * (120 + 300 + 60 * iters)
    if c["ewald"]:
        g = c["grid"] ** 3
        fft = 5 * g * math.log2(g)
        flops += 2 * n * 125 * 40 + fft
        if c["model"] != "none":
            flops += (iters + 1) * (2 * n * 125 * 12 + 2 * fft)
    size = 8 * n * (3 + 10 + 3)
    if c["call"] in ("step", "pressure", "analyze"):
        size += 8 * n * 6
    if c["call"] == "analyze":
        size += 8 * n * (2 + 6 + 13)
    if c["call"] == "train":
        size += 8 * n * (12 + 18)
        solves = 2
    if c["call"] == "pressure":
        solves = 2
    return {"bytes": solves * size, "flops": solves * flops}


# ------------------------------------------------------- values in 64 bits
class Reference:
    """The energies of a case in 64 bits from their definitions: every pair
    within the cutoff, smooth PME as sums over the transformed grids; the
    gradients are torch's derivatives of the energies."""

    def __init__(self, c, s, xyz, box):
        t = lambda a: torch.as_tensor(np.asarray(a), device=DEVICE)  # noqa: E731
        self.c, self.n = c, len(xyz)
        self.f, self.alpha = COULOMB, 0.5446
        self.x, self.L = t(xyz), float(box[0])
        self.pole, self.pol, self.thole = t(s.pole), t(s.polarity), t(s.thole)
        self.mol, self.water = t(s.molcule).long(), 3 * c["waters"]
        self.polarizable = c["model"] != "none"
        self.eps = torch.zeros(3, 3, device=DEVICE, dtype=torch.float64)  # strain of the cell
        self.pairs()

    def leaves(self):
        for k in ("x", "pole", "pol", "thole", "eps"):
            setattr(self, k, getattr(self, k).detach().requires_grad_(True))

    def pairs(self):
        x, i0, k0 = self.x, [], []
        for a in range(0, self.n, 4096):
            d = x[None] - x[a:a + 4096, None]
            d -= self.L * torch.round(d / self.L)
            i, k = torch.nonzero(d.square().sum(-1) <= self.c["cutoff"] ** 2, as_tuple=True)
            keep = k > i + a
            i0.append(i[keep] + a)
            k0.append(k[keep])
        self.i, self.k = torch.cat(i0), torch.cat(k0)
        d = x[self.k] - x[self.i]
        self.image = -torch.round(d / self.L)
        self.inside = self.mol[self.i] == self.mol[self.k]

    def cell(self):
        return self.L * (torch.eye(3, device=DEVICE, dtype=torch.float64) + 0.5 * (self.eps + self.eps.T))

    def strained(self):
        return self.x @ (self.cell() / self.L)

    def frames(self):
        """Global multipoles: O of a water on the bisector of its H, an H with
        z along its O and x towards the other H; ions as they are."""
        x = self.strained()
        w = x[:self.water].reshape(-1, 3, 3)
        unit = lambda v: v / v.norm(dim=-1, keepdim=True)  # noqa: E731
        u1, u2 = unit(w[:, 1] - w[:, 0]), unit(w[:, 2] - w[:, 0])
        zs, ts = [unit(u1 + u2)], [u2]
        for h, o in ((1, 2), (2, 1)):
            zs.append(unit(w[:, 0] - w[:, h]))
            ts.append(w[:, o] - w[:, h])
        z, t = torch.stack(zs, 1), torch.stack(ts, 1)
        xx = unit(t - (t * z).sum(-1, keepdim=True) * z)
        rot = torch.stack([xx, torch.linalg.cross(z, xx), z], -2).reshape(-1, 3, 3)
        eye = torch.eye(3, device=DEVICE, dtype=torch.float64).expand(self.n - self.water, 3, 3)
        rot = torch.cat([rot, eye])
        q = self.pole[:, 0]
        d = (self.pole[:, 1:4, None] * rot).sum(1)
        Q = rot.transpose(1, 2) @ self.pole[:, 4:].reshape(-1, 3, 3) @ rot
        up = torch.triu(Q)
        return q, d, up + torch.triu(Q, 1).transpose(1, 2)

    def geometry(self):
        x = self.strained()
        r = x[self.k] - x[self.i] + self.image @ self.cell()
        r2 = r.square().sum(-1)
        rr = r2.sqrt()
        bare = [1 / rr]
        for m in range(1, 6):
            bare.append(bare[-1] * (2 * m - 1) / r2)
        long = bare
        if self.c["ewald"]:
            a = self.alpha
            e = torch.exp(-a * a * r2)
            long = [torch.erfc(a * rr) / rr]
            for m in range(1, 6):
                long.append(((2 * m - 1) * long[-1] + (2 * a * a) ** m / (a * math.sqrt(math.pi)) * e) / r2)
        self.r, self.rr, self.bare, self.long = r, rr, bare, long

    def radial(self, scale, damped):
        """B_0..B_4 of a channel: the scaled (1-2 and 1-3) pairs are those of a molecule."""
        lam = [1.0] * 5
        if damped:
            pd = self.pol ** (1 / 6)
            a = torch.minimum(self.thole[self.i], self.thole[self.k])
            v = a * (self.rr / (pd[self.i] * pd[self.k])) ** 3
            e = torch.exp(-v)
            lam = [1.0, 1 - e, 1 - (1 + v) * e, 1 - (1 + v + 0.6 * v ** 2) * e,
                   1 - (1 + v + 18 / 35 * v ** 2 + 9 / 35 * v ** 3) * e]
        s = torch.where(self.inside, scale, 1.0)
        return [self.long[m] - (1 - s * lam[m]) * self.bare[m] for m in range(5)]

    # -- pair energies
    def permanent_pairs(self, M, scale=0.0):
        q, d, Q = M
        r, B = self.r, self.radial(scale, False)
        qi, qk, di, dk = q[self.i], q[self.k], d[self.i], d[self.k]
        Qi, Qk = Q[self.i], Q[self.k]
        dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
        Ri, Rk = (Qi @ r[..., None])[..., 0], (Qk @ r[..., None])[..., 0]
        ai, ak, bi, bk = dot(di, r), dot(dk, r), dot(Ri, r), dot(Rk, r)
        e = qi * qk * B[0] + (qk * ai - qi * ak + dot(di, dk)) * B[1]
        e = e + (qi * bk + qk * bi - ai * ak + 2 * (dot(dk, Ri) - dot(di, Rk) + (Qi * Qk).sum((-1, -2)))) * B[2]
        return e + (ai * bk - ak * bi - 4 * dot(Ri, Rk)) * B[3] + bi * bk * B[4]

    def field_pairs(self, M, v, scale):
        """Energy of the dipoles v in the field of the multipoles."""
        q, d, Q = M
        r, B = self.r, self.radial(scale, True)
        dot = lambda a, b: (a * b).sum(-1)  # noqa: E731
        total = 0.0
        for s, t, sign in ((self.i, self.k, 1.0), (self.k, self.i, -1.0)):  # dipole at t, multipole at s
            w, rr = v[t], sign * r
            wr, R = dot(w, rr), (Q[s] @ rr[..., None])[..., 0]
            e = (dot(d[s], w) - q[s] * wr) * B[1] + (2 * dot(w, R) - dot(d[s], rr) * wr) * B[2] - wr * dot(R, rr) * B[3]
            total = total + e.sum()
        return total

    def mutual_pairs(self, a, b):
        r, B = self.r, self.radial(1.0, True)
        dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
        ai, ak, bi, bk = a[self.i], a[self.k], b[self.i], b[self.k]
        e = (dot(ai, bk) + dot(ak, bi)) * B[1] - (dot(ai, r) * dot(bk, r) + dot(ak, r) * dot(bi, r)) * B[2]
        return e.sum()

    # -- smooth PME: structure factors and energies as sums over the grid
    def stencils(self):
        K, P = self.c["grid"], 5
        inv = torch.linalg.inv(self.cell())
        self.m = inv * K                                   # d(grid units) / d(Cartesian)
        u = self.strained() @ self.m
        u = u - K * torch.floor(u.detach() / K)
        lo = torch.floor(u.detach())
        w = u - lo
        b = {1: [torch.ones_like(w)]}
        for n in range(2, P + 1):
            b[n] = []
            for s in range(n):
                left = b[n - 1][s - 1] * (w + n - 1 - s) if s else 0.0
                right = b[n - 1][s] * (s + 1 - w) if s < n - 1 else 0.0
                b[n].append((left + right) / (n - 1))
        zero = torch.zeros_like(w)
        at = lambda n, s: b[n][s] if 0 <= s < n else zero  # noqa: E731
        t0 = torch.stack([at(P, s) for s in range(P)], -1)
        t1 = torch.stack([at(P - 1, s - 1) - at(P - 1, s) for s in range(P)], -1)
        t2 = torch.stack([at(P - 2, s - 2) - 2 * at(P - 2, s - 1) + at(P - 2, s) for s in range(P)], -1)
        self.theta = t0, t1, t2                            # each [n, axis, P]
        g = (lo.long()[..., None] - P + 1 + torch.arange(P, device=DEVICE)) % K
        self.index = ((g[:, 0, :, None, None] * K + g[:, 1, None, :, None]) * K + g[:, 2, None, None, :]).reshape(-1)
        # influence function over the half-complex grid, each point's weight in the full sum included
        h1 = torch.arange(K, device=DEVICE, dtype=torch.float64)
        f = torch.where(h1 <= K // 2, h1, h1 - K)
        half = torch.arange(K // 2 + 1, device=DEVICE, dtype=torch.float64)
        h = torch.stack(torch.meshgrid(f, f, half, indexing="ij"), -1) @ inv.T
        h2 = h.square().sum(-1)
        h2 = torch.where(h2 == 0, torch.ones_like(h2), h2)
        mod = self.modulus(K)
        V = torch.linalg.det(self.cell())
        G = torch.exp(-math.pi ** 2 * h2 / self.alpha ** 2) / (math.pi * V * h2)
        G = G / (mod[:, None, None] * mod[None, :, None] * mod[None, None, :K // 2 + 1])
        wgt = torch.full((K // 2 + 1,), 2.0, device=DEVICE, dtype=torch.float64)
        wgt[0] = 1
        if K % 2 == 0:
            wgt[-1] = 1
        keep = torch.ones_like(G)
        keep[0, 0, 0] = 0
        self.G = G * wgt * keep

    @staticmethod
    def modulus(K):
        v = torch.tensor([1, 11, 11, 1], dtype=torch.float64) / 24  # the order-5 spline at its inner knots
        m = torch.arange(K, dtype=torch.float64)
        z = (v * torch.exp(2j * math.pi / K * m[:, None] * torch.arange(4))).sum(-1)
        out = z.abs() ** 2
        bad = out < 1e-7
        out[bad] = 0.5 * (out.roll(1) + out.roll(-1))[bad]
        return out.to(DEVICE)

    def spread(self, q=None, d=None, Q=None):
        K = self.c["grid"]
        t = self.theta
        total = 0.0
        prod = lambda o: (t[o[0]][:, 0, :, None, None] * t[o[1]][:, 1, None, :, None] * t[o[2]][:, 2, None, None, :])  # noqa: E731
        wide = lambda v: v[:, None, None, None]  # noqa: E731
        if q is not None:
            total = total + wide(q) * prod((0, 0, 0))
        if d is not None:
            df = d @ self.m
            for a in range(3):
                total = total + wide(df[:, a]) * prod(tuple(int(a == b) for b in range(3)))
        if Q is not None:
            Qf = self.m.T @ Q @ self.m
            for a in range(3):
                for b in range(a, 3):
                    o = tuple(int(a == x) + int(b == x) for x in range(3))
                    total = total + wide(Qf[:, a, b] * (1 if a == b else 2)) * prod(o)
        grid = torch.zeros(K ** 3, device=DEVICE, dtype=torch.float64)
        return torch.fft.rfftn(grid.index_add(0, self.index, total.reshape(-1)).reshape(K, K, K))

    def product(self, A, B):
        return (self.G * (A.real * B.real + A.imag * B.imag)).sum()

    # -- energies without the factor f
    def update(self):
        self.M = self.frames()
        self.geometry()
        if self.c["ewald"]:
            self.stencils()
            self.SM = self.spread(*self.M)
        self.self_field = 4 * self.alpha ** 3 / (3 * math.sqrt(math.pi)) if self.c["ewald"] else 0.0

    def permanent(self):
        pairs = self.permanent_pairs(self.M)
        e = pairs.sum()
        self.between = pairs[~self.inside].sum()
        self.per_atom = torch.zeros(self.n, device=DEVICE, dtype=torch.float64)
        half = 0.5 * pairs.detach()
        self.per_atom.index_add_(0, self.i, half).index_add_(0, self.k, half)
        self.nonzero = int((pairs.detach() != 0).sum())
        if self.c["ewald"]:
            a, (q, d, Q) = self.alpha, self.M
            own = -a / math.sqrt(math.pi) * (q ** 2 + 2 / 3 * a ** 2 * d.square().sum(-1) + 8 / 5 * a ** 4 * Q.square().sum((-1, -2)))
            V = torch.linalg.det(self.cell())
            e = e + 0.5 * self.product(self.SM, self.SM) + own.sum() - math.pi * q.sum() ** 2 / (2 * V * a * a)
            self.per_atom += own.detach() + self.reciprocal_per_atom()
        return e

    def reciprocal_per_atom(self):
        """Half of each site's multipoles in the reciprocal potential."""
        with torch.enable_grad():
            s = torch.ones(self.n, device=DEVICE, dtype=torch.float64, requires_grad=True)
            q, d, Q = (v.detach() for v in self.M)
            S = self.spread(s * q, s[:, None] * d, s[:, None, None] * Q)
            return 0.5 * torch.autograd.grad(self.product(S, self.SM.detach()), s)[0]

    def with_multipoles(self, v, scale):
        e = self.field_pairs(self.M, v, scale)
        if self.c["ewald"]:
            e = e + self.product(self.spread(d=v), self.SM) - self.self_field * (v * self.M[1]).sum()
        return e

    def with_dipoles(self, a, b):
        e = self.mutual_pairs(a, b)
        if self.c["ewald"]:
            e = e + self.product(self.spread(d=a), self.spread(d=b)) - self.self_field * (a * b).sum()
        return e

    def minus_gradient(self, energy, graph=False):
        v = torch.zeros(self.n, 3, device=DEVICE, dtype=torch.float64, requires_grad=True)
        return -torch.autograd.grad(energy(v), v, create_graph=graph)[0]

    def fields(self, graph=False):
        """The permanent field; within a molecule both its scales (d and p) are 0."""
        return self.minus_gradient(lambda v: self.with_multipoles(v, 0.0), graph)

    def solve(self, E):
        """A u = E with A = 1/alpha - T, conjugate gradients to 1e-13."""
        pol = self.pol.detach()[:, None]
        A = lambda v: v / pol - self.minus_gradient(lambda w: self.with_dipoles(w, v))  # noqa: E731
        u = pol * E
        r = E - A(u)
        z = pol * r
        p, rz = z, (r * z).sum()
        stop = 1e-13 * float(E.norm())
        for _ in range(60):
            if float(r.norm()) <= stop:
                break
            Ap = A(p)
            a = rz / (p * Ap).sum()
            u, r = u + a * p, r - a * Ap
            z = pol * r
            new = (r * z).sum()
            p, rz = z + new / rz * p, new
        return u

    def dipoles(self):
        """Induced dipoles of the case's model; the d and p sets coincide for rigid waters and ions."""
        with torch.enable_grad():
            E = self.fields().detach()
        if self.c["model"] == "direct":
            return E, self.pol.detach()[:, None] * E
        return E, self.solve(E)

    def detached(self):
        """A copy of the geometry without its graph, for the fields and the solve."""
        with torch.no_grad():
            self.update()

    def polarization(self, u, E, lam=None, lam_p=None, c=1.0):
        """A function with the gradient of c ep + <g_d, u_d> + <g_p, u_p> at fixed
        vectors: lam_d (E_d - A u) + lam_p (E_p - A u) - c f/2 u E_p."""
        f, mutual = self.f, self.c["model"] == "mutual"
        lam = -0.5 * c * f * u if lam is None else lam
        total = lam if lam_p is None else lam + lam_p
        g = -self.with_multipoles(total - 0.5 * c * f * u, 0.0) - ((total * u) / self.pol[:, None]).sum()
        return g - self.with_dipoles(total, u) if mutual else g


def evaluate(c, s, xyz, box):
    """(em, ep, dem, dep, virial, the Reference) of one geometry."""
    R = Reference(c, s, xyz, box)
    zero = torch.zeros_like(R.x)
    E = u = None
    if R.polarizable and c["model"] != "opt4":
        R.detached()
        E, u = R.dipoles()
    R.leaves()
    R.update()
    em = R.f * R.permanent()
    dem, vir = torch.autograd.grad(em, [R.x, R.eps], retain_graph=True, allow_unused=True)
    ep, dep, vir_p = torch.zeros(()), zero, torch.zeros_like(vir)
    if c["model"] == "opt4":
        E = R.fields(graph=True)
        a, copt = R.pol[:, None], OPT_COEF[4]
        v = a * E
        u = sum(copt) * v
        for k in range(1, 5):
            w = v
            v = a * R.minus_gradient(lambda t: R.with_dipoles(t, w), graph=True)
            u = u + sum(copt[k:]) * v
        ep = -0.5 * R.f * (u * E).sum()
        dep, = torch.autograd.grad(ep, [R.x])
    elif R.polarizable:
        ep = -0.5 * R.f * (u * E).sum()
        dep, vir_p = torch.autograd.grad(R.polarization(u, E), [R.x, R.eps])
    R.E, R.u = E, u
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    v = host(vir + vir_p)
    return float(em.detach()), float(ep.detach()), host(dem), host(dep), 0.5 * (v + v.T), R


def exact(case, seed):
    c = case
    s = system_of(c, seed)
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    if c["call"] == "step":
        em, ep, dem, dep, _, _ = evaluate(c, s, s.xyz, s.box)
        return {"em": em, "ep": ep, "dem": dem.reshape(-1), "dep": dep.reshape(-1)}
    if c["call"] == "pressure":
        out = []
        for xyz, box in ((s.xyz, s.box), grown(c, s.xyz)):
            em, ep, dem, dep, vir, _ = evaluate(c, s, xyz, box)
            out.append({"em": em, "ep": ep, "dem": dem, "dep": dep, "vir": vir})
        return out
    if c["call"] == "analyze":
        em, ep, dem, dep, _, R = evaluate(c, s, s.xyz, s.box)
        q, d, Q = (host(v) for v in R.M)
        pol = R.polarizable
        u = host(R.u) if pol else np.zeros((s.n, 3))
        return {"em": em, "ep": ep, "einter": float(R.f * R.between.detach()), "nem": None, "nep": None, "aem": R.f * host(R.per_atom),
                "aep": -0.5 * R.f * host((R.u * R.E).sum(-1)) if pol else np.zeros(s.n), "dem": dem, "dep": dep, "uind": u,
                "uinp": u, "rpole": np.concatenate([q[:, None], d, Q.reshape(-1, 9)], 1)}
    # train: L = c (em + ep) + <g_d, u_d> + <g_p, u_p>
    seedE, gd, gp = cotangents(s.n, seed)
    R = Reference(c, s, s.xyz, s.box)
    R.detached()
    E, u = R.dipoles()
    wd, wp = (R.solve(torch.as_tensor(g, device=DEVICE)) for g in (gd, gp))
    R.leaves()
    R.update()
    L = seedE * R.f * R.permanent() + R.polarization(u, E, lam=wd - 0.5 * seedE * R.f * u, lam_p=wp, c=seedE)
    dpole, dpol, dthole, dx = torch.autograd.grad(L, [R.pole, R.pol, R.thole, R.x])
    em = R.f * float(R.permanent().detach())
    d = host(dpole).copy()
    trace = d[:, [4, 8, 12]].mean(1, keepdims=True)
    d[:, [4, 8, 12]] -= trace  # quadrupoles are traceless
    return {"em": em, "ep": float(-0.5 * R.f * (u * E).sum()), "uind": host(u), "uinp": host(u),
            "d_pole": d, "d_polarity": host(dpol), "d_thole": host(dthole), "d_xyz": host(dx).reshape(-1, 3)}
