"""The work that programs have this framework do, as cases that can be timed and checked.

Every case goes through a public entry point: ``FockBuilder`` (restricted, unrestricted,
Fock-matrix and incremental/mixed builds, host and device arrays, geometry steps) and
``BatchFockBuilder``.  The systems are the ones of the benchmark and the
tests: seeded water clusters from two to 32 molecules and all-trans alkanes up to C40H82, in
STO-3G, 6-31G(d), cc-pVDZ, def2-SVP and cc-pVTZ (f shells), spherical and Cartesian.

Inputs come from the seed alone: the geometry (the seeded jitter and orientations of the cluster
builders) and the density, the occupied projector of a seeded tight-binding model of the same
molecule (idempotent, decaying with distance, core orbitals doubly occupied, as an SCF's density).
"""

from __future__ import annotations

import dataclasses
import math
from functools import lru_cache

import numpy as np
import torch

from tonto_b200.basis import Molecule
from tonto_b200.fock import (TF_JK_DELTA, TF_JK_FULL, TF_JK_MIXED, BatchFockBuilder, FockBuilder)
from tonto_b200.molecules import alkane, water_cluster

SCHWARZ = 1e-12          # the SCF drivers' and the benchmark's Schwarz x density cutoff
TONTO_SCHWARZ = 1e-9     # Tonto's default
PAIR_CUTOFF = 1e-6       # Tonto's default primitive-pair cutoff


def _case(name=None, **kw):
    c = {"kind": "jk", "system": "water", "n": 4, "basis": "cc-pVDZ", "spherical": True, "density": "full",
         "mixed": False, "deterministic": False}
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: host arrays through the C ABI, 14 functions; latency and launches
        _case("h2o2-sto3g-host", kind="jk_host", n=2, basis="STO-3G"),
        # one Fock matrix of a Cartesian basis from host arrays at Tonto's default cutoff (make_r_Fock_mx)
        _case("h2o3-631gd-cartesian-fock", kind="fock", n=3, basis="6-31G(d)", spherical=False),
        # f shells: Tonto's cc-pVTZ runs, on device arrays
        _case("h2o2-ccpvtz", n=2, basis="cc-pVTZ"),
        # the same basis at the size of a small cluster, an ordinary triple-zeta job
        _case("h2o5-ccpvtz", n=5, basis="cc-pVTZ"),
        # an ordinary SCF cycle's build, odd size
        _case("h2o7-ccpvdz", n=7),
        # an open shell: both spins' J and K (cation, doublet)
        _case("h2o6-631gd-uhf", kind="uhf", n=6, basis="6-31G(d)"),
        # a bitwise-reproducible build
        _case("h2o12-ccpvdz-deterministic", n=12, deterministic=True),
        # a geometry step, as refinement and optimisation take them: moved atoms, S, T, V, then J and K
        _case("h2o9-ccpvdz-move", kind="move", n=9),
        # a late SCF cycle of the fast schedule: mixed precision, from the density change
        _case("h2o19-ccpvdz-delta-mixed", n=19, density="delta", mixed=True),
        # many molecules in one launch sequence: one cycle of a batched SCF
        _case("batch24-ccpvdz", kind="batch", n=24),
        # the long-chain workload: C40H82 (970 functions) in mixed precision
        _case("c40h82-def2svp-mixed", system="alkane", n=40, basis="def2-SVP", mixed=True),
        # the benchmark: (H2O)32 cc-pVDZ, 768 functions, a full FP64 build
        _case("h2o32-ccpvdz", n=32),
    ]


def draw(rng):
    """One more case of the listed ranges: an entry point, a system, a size over the logarithm of its range."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))

    kind = rng.choice(["jk", "jk", "jk", "jk_host", "fock", "uhf", "move", "batch"])
    if kind == "batch":
        return _case(kind="batch", n=size(2, 24), mixed=rng.random() < 0.5,
                     density=rng.choice(["full", "delta"]))
    system = rng.choice(["water", "water", "alkane"])
    basis = rng.choice(["STO-3G", "6-31G(d)", "cc-pVDZ", "cc-pVDZ", "def2-SVP", "cc-pVTZ"]) if system == "water" \
        else "def2-SVP"
    top = {"STO-3G": 32, "6-31G(d)": 28, "cc-pVDZ": 28, "def2-SVP": 28, "cc-pVTZ": 5}[basis] if system == "water" else 36
    if kind in ("uhf", "move"):
        top = min(top, 16)
    return _case(kind=kind, system=system, basis=basis, n=min(top, size(2, top)), spherical=rng.random() < 0.7,
                 density=rng.choice(["full", "full", "delta"]) if kind in ("jk", "jk_host") else "full",
                 mixed=kind == "jk" and rng.random() < 0.4, deterministic=kind == "jk" and rng.random() < 0.15)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _molecules(case, seed):
    if case["kind"] == "batch":       # sizes as in the 256-cluster batch: seeded-uniform in [2, 24]
        sizes = np.random.default_rng(3).integers(2, 25, size=256)
        return [water_cluster(int(sizes[i]), seed=1000 * seed + i, basis=case["basis"], spherical=case["spherical"])
                for i in range(case["n"])]
    make = water_cluster if case["system"] == "water" else alkane
    return [make(case["n"], seed=seed, basis=case["basis"], spherical=case["spherical"])]


def _model_hamiltonian(mol: Molecule, rng) -> np.ndarray:
    """Tight-binding model: site energies from each shell's contraction, hopping decaying with the distance."""
    at, e = [], []
    for s in mol.shells:
        c = np.abs(np.asarray(s.coefs)) + 1e-300
        ebar = math.exp(float(np.sum(c * np.log(s.exps)) / np.sum(c)))
        k = mol.shell_nbf(s.l)
        at += [s.atom] * k
        e += [-math.sqrt(ebar) / (1 + s.l) + 0.5 * s.l] * k
    at = np.array(at)
    d = np.linalg.norm(mol.xyz[at][:, None, :] - mol.xyz[at][None, :, :], axis=-1)
    g = rng.normal(size=d.shape)
    h = 0.15 * (g + g.T) * np.exp(-0.7 * d)
    h[np.diag_indices_from(h)] = np.array(e) + 0.05 * rng.normal(size=len(e))
    return h


def _projector(h: torch.Tensor, n_occ: int) -> torch.Tensor:
    c = torch.linalg.eigh(h)[1][:, :n_occ]
    return c @ c.T


def _density(mol, seed, density, dev):
    rng = np.random.default_rng(7_000_003 * (seed + 1))
    h = torch.tensor(_model_hamiltonian(mol, rng), dtype=torch.float64, device=dev)
    n_occ = mol.n_electrons // 2
    p = 2.0 * _projector(h, n_occ)
    if density == "full":
        return p.contiguous()
    g = torch.tensor(rng.normal(size=h.shape), dtype=torch.float64, device=dev)   # the change of an SCF cycle
    return (2.0 * _projector(h + 1e-4 * (g + g.T) * h.abs(), n_occ) - p).contiguous()


def _spin_densities(mol, seed, dev):
    rng = np.random.default_rng(7_000_003 * (seed + 1))
    out = []
    for n in (mol.n_electrons // 2, mol.n_electrons // 2 - 1):       # the cation's doublet
        h = torch.tensor(_model_hamiltonian(mol, rng), dtype=torch.float64, device=dev)
        out.append(_projector(h, n).contiguous())
    return out


def _hcore(mol, seed):
    """A symmetric matrix in the place of T + V (make_r_Fock_mx adds it as it is)."""
    return _model_hamiltonian(mol, np.random.default_rng(11 + seed))


def _moved(mol, seed):
    rng = np.random.default_rng(23 + seed)
    return dataclasses.replace(mol, xyz=mol.xyz + rng.uniform(-0.03, 0.03, size=mol.xyz.shape))


def _inputs(case, seed, dev):
    """The molecules and host/device inputs of a case, without the builder."""
    mols = _molecules(case, seed)
    kind = case["kind"]
    if kind == "uhf":
        return mols, _spin_densities(mols[0], seed, dev)
    ps = [_density(m, seed + 17 * i, case["density"], dev) for i, m in enumerate(mols)]
    return mols, ps


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    mols, ps = _inputs(case, seed, dev)
    kind, mol = case["kind"], mols[0]
    flags = (TF_JK_MIXED if case["mixed"] else TF_JK_FULL) | (TF_JK_DELTA if case["density"] == "delta" else 0)
    s = {"kind": kind, "flags": flags}
    opt = {"schwarz_cutoff": TONTO_SCHWARZ if kind == "fock" else SCHWARZ, "pair_cutoff": PAIR_CUTOFF,
           "device": dev.index, "deterministic": case["deterministic"]}
    if kind == "batch":
        s["fb"] = BatchFockBuilder(mols, **opt)
        s["p"] = torch.cat([p.reshape(-1) for p in ps])
        s["out"] = [torch.empty_like(s["p"]) for _ in range(2)]
        return s
    s["fb"] = FockBuilder(mol, **opt)
    if kind in ("jk_host", "fock"):
        s["p"] = np.asfortranarray(ps[0].cpu().numpy())
        if kind == "fock":
            s["h"] = np.asfortranarray(_hcore(mol, seed))
        return s
    s["p"] = ps
    s["out"] = [torch.empty_like(ps[0]) for _ in range(4 if kind == "uhf" else 2)]
    if kind == "move":
        s["xyz"] = _moved(mol, seed).xyz
    return s


def run(s):
    kind = s["kind"]
    if kind == "jk_host":
        return s["fb"].make_r_JK(s["p"], s["flags"])
    if kind == "fock":
        return s["fb"].make_r_Fock_mx(s["p"], s["h"])
    if kind == "uhf":
        s["fb"].make_u_JK_device(*s["p"], *s["out"], s["flags"])
        return s["out"]
    if kind == "batch":
        s["fb"].make_r_JK_device(s["p"], *s["out"], s["flags"])
        return s["out"]
    if kind == "move":
        s["fb"].set_geometry(s["xyz"])
        stv = s["fb"].one_electron()
        s["fb"].make_r_JK_device(s["p"][0], *s["out"], s["flags"])
        return [*s["out"], *stv]
    s["fb"].make_r_JK_device(s["p"][0], *s["out"], s["flags"])
    return s["out"]


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _nupto(l):
    return (l + 1) * (l + 2) * (l + 3) // 6


def _class_flops(la, lb, lc, ld):
    """Floating-point operations of one primitive and one contracted quartet: pair terms, Rys roots (polynomials of
    degree 11), 2D recurrences and the sums over the Cartesian products, then transfers and twelve operations per
    integral for J and K."""
    nr, d1, d2 = (la + lb + lc + ld) // 2 + 1, la + lb + 1, lc + ld + 1
    ne, nf = _nupto(la + lb) - _nupto(la - 1), _nupto(lc + ld) - _nupto(lc - 1)
    prim = 20.0 + 44.0 * nr + nr * (10.0 + 3.0 * (4.0 + 6.0 * d1 * d2) + d1 * d2 + 3.0 * ne * nf)
    nc, nd = _ncart(lc), _ncart(ld)
    hrr = sum(2.0 * ne * (_nupto(lc + ld - k) - _nupto(lc - 1)) * _ncart(k) for k in range(1, ld + 1))
    hrr += sum(2.0 * nc * nd * (_nupto(la + lb - k) - _nupto(la - 1)) * _ncart(k) for k in range(1, lb + 1))
    return prim, hrr + 12.0 * _ncart(la) * _ncart(lb) * nc * nd


def _molecule_flops(mol, cutoff, pmax=1.0):
    """Estimated operations of one build: per class pair the shell quartets whose (estimated) Schwarz bounds pass the
    cutoff, times the class's operations at its mean number of primitive pairs."""
    xyz = mol.xyz
    classes = {}
    for ia, a in enumerate(mol.shells):
        for b in mol.shells[: ia + 1]:
            r2 = float(np.sum((xyz[a.atom] - xyz[b.atom]) ** 2))
            ea, eb = np.asarray(a.exps)[:, None], np.asarray(b.exps)[None, :]
            p = ea + eb
            fac = np.exp(-ea * eb / p * r2)
            cc = np.abs(np.outer(a.coefs, b.coefs)) * fac / ea ** (a.l / 2) / eb ** (b.l / 2)
            v = float(np.sqrt(34.99 / math.sqrt(2.0)) * np.sum(cc * p ** -1.25))
            hi, lo = max(a.l, b.l), min(a.l, b.l)
            npp = fac.size if a.atom == b.atom else int(np.sum(fac >= PAIR_CUTOFF))
            if v > 1e-14:
                classes.setdefault((hi, lo), []).append((v, max(npp, 1)))
    keys = sorted(classes)
    lists = {k: np.array(sorted(classes[k])) for k in keys}
    total = 0.0
    for i, x in enumerate(keys):
        for y in keys[: i + 1]:
            vx, vy = lists[x][:, 0], lists[y][:, 0]
            n_first = len(vy) - np.searchsorted(vy, cutoff / pmax / vx)
            cum = np.concatenate([np.cumsum(lists[y][::-1, 1])[::-1], [0.0]])
            nq = float(np.sum(n_first))
            npq = float(np.sum(lists[x][:, 1] * cum[len(vy) - n_first]))
            half = 0.5 if x == y else 1.0
            prim, con = _class_flops(*x, *y)
            total += half * (npq * prim + nq * con)
    return total


@lru_cache(maxsize=None)
def _work(items):
    case = dict(items)
    mols = _molecules(case, 0)
    cutoff = TONTO_SCHWARZ if case["kind"] == "fock" else SCHWARZ
    pmax = 1e-3 if case["density"] == "delta" else 1.0
    flops = sum(_molecule_flops(m, cutoff, pmax) for m in mols)
    n2 = sum(m.n_bf ** 2 for m in mols)
    arrays = {"uhf": 6, "move": 6, "fock": 3}.get(case["kind"], 3)
    return {"bytes": 8.0 * arrays * n2, "flops": flops}


def work(case):
    return dict(_work(tuple(sorted((k, v) for k, v in case.items() if k != "name"))))


# ---------------------------------------------------------------------------
# the same results in plain torch, FP64: McMurchie-Davidson integrals of the whole molecule
# ---------------------------------------------------------------------------
def _components(l):
    """Cartesian components in Tonto's order (gaussian_data.foo:295-479), l <= 3."""
    return {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
            2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
            3: [(3, 0, 0), (0, 3, 0), (0, 0, 3), (2, 1, 0), (2, 0, 1), (1, 2, 0), (0, 2, 1), (1, 0, 2), (0, 1, 2),
                (1, 1, 1)]}[l]


def _solid_harmonics(l):
    """Real solid harmonics over the Cartesian components, m = 0, +1, -1, ... (the explicit sum of Schlegel and Frisch,
    Int. J. Quantum Chem. 54, 83 (1995))."""
    comps = _components(l)
    ms = [0] + [m for k in range(1, l + 1) for m in (k, -k)]
    u = np.zeros((len(comps), len(ms)))
    for col, m in enumerate(ms):
        a = abs(m)
        norm = math.sqrt(2.0 * math.factorial(l + a) * math.factorial(l - a) / (2.0 if m == 0 else 1.0))
        norm /= 2 ** a * math.factorial(l)
        for t in range((l - a) // 2 + 1):
            for k in range(t + 1):
                for v2 in range(0 if m >= 0 else 1, a + 1, 2):       # twice Schlegel and Frisch's v
                    c = (-1.0) ** (t + (v2 - (0 if m >= 0 else 1)) // 2) * 0.25 ** t * math.comb(l, t)
                    c *= math.comb(l - t, a + t) * math.comb(t, k) * math.comb(a, v2)
                    u[comps.index((2 * t + a - 2 * k - v2, 2 * k + v2, l - 2 * t - a)), col] += norm * c
    return u


def _basis_matrix(mol, dev):
    """Cartesian functions (shell by shell) x basis functions."""
    blocks = [_solid_harmonics(s.l) if mol.spherical and s.l >= 2 else np.eye(_ncart(s.l)) for s in mol.shells]
    return torch.block_diag(*[torch.tensor(b, dtype=torch.float64, device=dev) for b in blocks])


def _boys(m_max, x):
    """F_0 .. F_m_max of a tensor: series and downward recursion below 35, error function and upward above."""
    low = x < 35.0
    y = torch.where(low, x, torch.zeros_like(x))
    term = torch.full_like(y, 1.0 / (2 * m_max + 1))
    top = term.clone()
    for k in range(1, 160):
        term = term * (2.0 * y / (2 * m_max + 2 * k + 1))
        top = top + term
    ey = torch.exp(-y)
    down = [None] * (m_max + 1)
    down[m_max] = top * ey
    for m in range(m_max - 1, -1, -1):
        down[m] = (2.0 * y * down[m + 1] + ey) / (2 * m + 1)
    z = torch.where(low, torch.full_like(x, 35.0), x)
    ez = torch.exp(-z)
    up = 0.5 * torch.sqrt(math.pi / z) * torch.erf(torch.sqrt(z))
    out = []
    for m in range(m_max + 1):
        out.append(torch.where(low, down[m], up))
        up = ((2 * m + 1) * up - ez) / (2.0 * z)
    return out


def _hermite(lmax):
    return [(t, u, v) for t in range(lmax + 1) for u in range(lmax + 1 - t) for v in range(lmax + 1 - t - u)]


def _r_tensors(lmax, alpha, d):
    """Hermite Coulomb integrals R_tuv(alpha, d), t + u + v <= lmax, as {(t, u, v): tensor}."""
    f = _boys(lmax, alpha * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2))
    level = {}
    for n in range(lmax, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * f[n]}
        for tuv in sorted(_hermite(lmax - n), key=sum)[1:]:
            k = next(i for i in range(3) if tuv[i] > 0)
            a = tuple(tuv[i] - (i == k) for i in range(3))
            v = d[k] * level[a]
            if a[k] > 0:
                v = v + a[k] * level[tuple(a[i] - (i == k) for i in range(3))]
            new[tuv] = v
        level = new
    return level


def _e_table(la, lb, a, b, ab):
    """Hermite expansion coefficients E[i][j][t] of one axis, i <= la, j <= lb (tensors over primitive pairs)."""
    p = a + b
    pa, pb, h = -b / p * ab, a / p * ab, 0.5 / p
    zero = torch.zeros_like(p)
    e = [[None] * (lb + 1) for _ in range(la + 1)]
    e[0][0] = [torch.exp(-a * b / p * ab * ab)]
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j == 0:
                continue
            src, x = (e[i - 1][j], pa) if i > 0 else (e[i][j - 1], pb)
            n = i + j
            g = lambda t: src[t] if 0 <= t < len(src) else zero  # noqa: E731
            e[i][j] = [h * g(t - 1) + x * g(t) + (t + 1) * g(t + 1) for t in range(n + 1)]
    return e


class _PairClass:
    """All shell pairs a >= b of one (l_a, l_b): primitive pairs, Hermite coefficients, function indices."""

    def __init__(self, mol, la, lb, pairs, first, dev):
        t = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=dev)  # noqa: E731
        self.la, self.lb, self.l = la, lb, la + lb
        ea, eb, cc, ca, cb, seg = [], [], [], [], [], []
        for k, (ia, ib) in enumerate(pairs):
            a, b = mol.shells[ia], mol.shells[ib]
            for x, cx in zip(a.exps, a.coefs):
                for y, cy in zip(b.exps, b.coefs):
                    ea.append(x); eb.append(y); cc.append(cx * cy); ca.append(mol.xyz[a.atom])   # noqa: E702
                    cb.append(mol.xyz[b.atom]); seg.append(k)                                     # noqa: E702
        a, b, self.cc, A, B = t(ea), t(eb), t(cc), t(ca), t(cb)
        self.seg = torch.tensor(seg, device=dev)
        self.n = len(pairs)
        self.p = a + b
        self.P = (a[:, None] * A + b[:, None] * B) / self.p[:, None]
        self.r2 = ((A - B) ** 2).sum(1)
        self.keep = (torch.exp(-a * b / self.p * self.r2) >= PAIR_CUTOFF).to(torch.float64)
        tabs = [_e_table(la, lb + 2, a, b, (A - B)[:, k]) for k in range(3)]
        self.herm = _hermite(self.l)
        comps = [(i, j) for i in _components(la) for j in _components(lb)]
        zero = torch.zeros_like(a)

        def e(k, i, j, h):
            row = tabs[k][i][j]
            return row[h] if h < len(row) else zero
        self.E = torch.stack([torch.stack([e(0, i[0], j[0], h[0]) * e(1, i[1], j[1], h[1]) * e(2, i[2], j[2], h[2])
                                           for h in self.herm], 1) for i, j in comps], 1) * self.cc[:, None, None]
        s1 = lambda k, i, j: e(k, i, j, 0) if j >= 0 else zero  # noqa: E731
        kin = lambda k, i, j: (-2.0 * b * b * s1(k, i, j + 2) + b * (2 * j + 1) * s1(k, i, j)  # noqa: E731
                               - 0.5 * j * (j - 1) * s1(k, i, j - 2))
        pre = self.cc * (math.pi / self.p) ** 1.5
        self.S = torch.stack([pre * s1(0, i[0], j[0]) * s1(1, i[1], j[1]) * s1(2, i[2], j[2]) for i, j in comps], 1)
        self.T = torch.stack([pre * sum(kin(k, i[k], j[k]) * s1((k + 1) % 3, i[(k + 1) % 3], j[(k + 1) % 3])
                                        * s1((k + 2) % 3, i[(k + 2) % 3], j[(k + 2) % 3]) for k in range(3))
                              for i, j in comps], 1)
        na, nb = _ncart(la), _ncart(lb)
        idx = lambda v, n, m, rep: (torch.tensor(v, device=dev)[:, None]  # noqa: E731
                                    + torch.arange(n, device=dev).repeat_interleave(rep).repeat(m)[None, :])
        self.fa = idx([first[i] for i, _ in pairs], na, 1, nb)
        self.fb = idx([first[j] for _, j in pairs], nb, na, 1)
        self.atoms = torch.tensor([(mol.shells[i].atom, mol.shells[j].atom) for i, j in pairs], device=dev)

    def contract(self, x):
        """Sum over the primitive pairs (dimension 0) of each shell pair."""
        return torch.zeros((self.n,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device).index_add_(0, self.seg, x)


def _pair_classes(mol, dev):
    first = np.concatenate([[0], np.cumsum([_ncart(s.l) for s in mol.shells])]).astype(int)
    groups = {}
    for i, a in enumerate(mol.shells):
        for j in range(i + 1):
            groups.setdefault((a.l, mol.shells[j].l), []).append((i, j))
    return [_PairClass(mol, la, lb, ps, first, dev) for (la, lb), ps in sorted(groups.items())], int(first[-1])


def _block(x, y):
    """(ab|cd) of two pair classes: [pair x, ab, pair y, cd], Tonto's primitive-pair cutoff where no atoms coincide."""
    dev = x.p.device
    same = lambda u, v: x.atoms[:, None, u] == y.atoms[None, :, v]  # noqa: E731
    one = (x.atoms[:, 0] == x.atoms[:, 1])[:, None] | (y.atoms[:, 0] == y.atoms[:, 1])[None, :]
    any_same = one | same(0, 0) | same(0, 1) | same(1, 0) | same(1, 1)
    nx, ny = len(x.p), len(y.p)
    sign = torch.tensor([(-1.0) ** sum(h) for h in y.herm], dtype=torch.float64, device=dev)
    ey = y.E * sign
    both = [(x.E, ey), (x.E * x.keep[:, None, None], ey * y.keep[:, None, None])]
    acc = [torch.zeros((x.n, x.E.shape[1], y.n, y.E.shape[1]), dtype=torch.float64, device=dev) for _ in both]
    n_r = len(_hermite(x.l + y.l))
    step = max(1, int(6e7 / (ny * (2 * n_r + len(y.herm) * 2 + y.E.shape[1] * 2))))
    for i0 in range(0, nx, step):
        sl = slice(i0, min(nx, i0 + step))
        p, q = x.p[sl, None], y.p[None, :]
        d = [x.P[sl, None, k] - y.P[None, :, k] for k in range(3)]
        r = _r_tensors(x.l + y.l, p * q / (p + q), d)
        pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        for hx, t in enumerate(x.herm):
            g = torch.stack([r[(t[0] + h[0], t[1] + h[1], t[2] + h[2])] for h in y.herm], 2) * pre[:, :, None]
            for k, (bra, ket) in enumerate(both):
                c = torch.einsum("xyh,ych->yxc", g, ket)
                c = y.contract(c).permute(1, 0, 2)                    # [x, pair y, cd]
                v = bra[sl, :, hx][:, :, None, None] * c[:, None, :, :]
                acc[k].index_add_(0, x.seg[sl], v)
    return torch.where(any_same[:, None, :, None], acc[0], acc[1])


def _jk(mol, ps, dev):
    """[(J, K)] of the densities ps (basis functions)."""
    classes, n = _pair_classes(mol, dev)
    eri = torch.zeros((n, n, n, n), dtype=torch.float64, device=dev)
    for i, x in enumerate(classes):
        for y in classes[: i + 1]:
            g = _block(x, y).reshape(x.n * x.E.shape[1], y.n * y.E.shape[1])
            a, b, c, d = (v.reshape(-1) for v in (x.fa, x.fb, y.fa, y.fb))
            for u, v, w, z, h in ((a, b, c, d, g), (c, d, a, b, g.T)):
                eri[u[:, None], v[:, None], w[None, :], z[None, :]] = h
                eri[v[:, None], u[:, None], w[None, :], z[None, :]] = h
                eri[u[:, None], v[:, None], z[None, :], w[None, :]] = h
                eri[v[:, None], u[:, None], z[None, :], w[None, :]] = h
    u = _basis_matrix(mol, dev)
    out = []
    for p in ps:
        pc = u @ p @ u.T
        j = (eri.reshape(n * n, n * n) @ pc.reshape(-1)).reshape(n, n)
        k = torch.einsum("abcd,bd->ac", eri, pc)
        out.append((u.T @ j @ u, u.T @ k @ u))
    return out


def _stv(mol, dev):
    classes, n = _pair_classes(mol, dev)
    u = _basis_matrix(mol, dev)
    xyz = torch.tensor(mol.xyz, dtype=torch.float64, device=dev)
    out = []
    for what in "STV":
        m = torch.zeros((n, n), dtype=torch.float64, device=dev)
        for x in classes:
            if what == "V":
                v = torch.zeros_like(x.S)
                for z, c in zip(mol.Z, xyz):
                    r = _r_tensors(x.l, x.p, [x.P[:, k] - c[k] for k in range(3)])
                    v -= float(z) * torch.einsum("xch,xh->xc", x.E, torch.stack([r[h] for h in x.herm], 1)
                                                 * (2.0 * math.pi / x.p)[:, None])
            else:
                v = x.S if what == "S" else x.T
            v = x.contract(v).reshape(-1)
            a, b = x.fa.reshape(-1), x.fb.reshape(-1)
            m[a, b] = v
            m[b, a] = v
        out.append(u.T @ m @ u)
    return out


EXACT_CART = 180         # Cartesian functions up to which the full tensor takes seconds


def exact(case, seed):
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    mols, ps = _inputs(case, seed, dev)
    kind, mol = case["kind"], mols[0]
    n = max(sum(_ncart(s.l) for s in m.shells) for m in mols)
    if kind == "move":
        mol = _moved(mol, seed)
        if mol.n_atom > 36:
            return None
        jk = list(_jk(mol, ps, dev)[0]) if n <= EXACT_CART else [None, None]
        return jk + [x.cpu().numpy() for x in _stv(mol, dev)]
    if n > EXACT_CART or len(mols) > 4:
        return None
    if kind == "uhf":
        (ja, ka), (jb, kb) = _jk(mol, ps, dev)
        return [ja, jb, ka, kb]
    if kind == "batch":
        res = [_jk(m, [p], dev)[0] for m, p in zip(mols, ps)]
        return [torch.cat([r[k].reshape(-1) for r in res]) for k in range(2)]
    j, k = _jk(mol, ps, dev)[0]
    if kind == "fock":
        return _hcore(mol, seed) + (j - 0.5 * k).cpu().numpy()
    if kind == "jk_host":
        return j.cpu().numpy(), k.cpu().numpy()
    return [j, k]
