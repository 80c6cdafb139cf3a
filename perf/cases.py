"""Performance cases: what a user of pychem_gb300 has it compute, over the range of sizes,
basis sets, precisions and directions it is used with.

Every case calls the package's public entry points only.  Geometries come from
``pychem_gb300.workloads`` with the case's seed as jitter seed; densities and orbitals are
those of a model Hamiltonian that decays with distance (``_orbitals``), so that they can
be made without the package.  ``exact`` evaluates the same integrals, Fock matrices, SCF,
MP2, intensities and network steps in plain torch at 64 bits: a McMurchie-Davidson scheme
(L. E. McMurchie, E. R. Davidson, J. Comput. Phys. 26 (1978) 218-231) with the documented
Schwarz rule Q_ab Q_cd > 1e-8, where the molecule is small enough for that.
"""
import functools
import json
import math
import os

import numpy as np
import torch

import pychem_gb300
from pychem_gb300 import api, scattering, workloads
from pychem_gb300.engine import GpuEngine
from pychem_gb300.ensemble import EnsembleEngine, rhf_batched
from pychem_gb300.learned.mlp import PairMLP
from pychem_gb300.molecule import Molecule
from pychem_gb300.scf import mp2_pair_sums, mp2_transform

THRESHOLD = 1.0e-8                 # the package's documented screening threshold
TO_BOHR = 1.8897161646320724
CLUSTERS = {1: (1, 1, 1), 2: (2, 1, 1), 3: (3, 1, 1), 4: (2, 2, 1), 6: (3, 2, 1), 8: (2, 2, 2), 12: (3, 2, 2),
            16: (4, 2, 2)}
NET = (40, 256, 256, 256, 47)      # the learned guess's layers: pair features to density parameters
EXACT_AO = 112                     # largest molecule exact() takes (a few seconds on the GPU)
EXACT_SCF_AO = 40


def listed():
    return [
        # one small molecule, host coordinates to energies and orbitals: latency and launches
        dict(name="solve_water", kind="solve", system="water", units=1, basis="6-31G"),
        # the headline workload: RHF + MP2 of a 16-water cluster
        dict(name="solve_water16", kind="solve", system="water", units=16, basis="6-31G"),
        # a thousand perturbed small molecules in one batched SCF
        dict(name="ensemble_1024", kind="ensemble", units=1024, basis="6-31G"),
        # all integrals of a molecule with d shells from its host description, and one Fock build
        dict(name="integrals_alkane12", kind="integrals", system="alkane", units=12, basis="cc-pVDZ", precision="fp64"),
        # the same call in mixed precision on a mid-size cluster
        dict(name="integrals_water8_mixed", kind="integrals", system="water", units=8, basis="6-31G", precision="mixed"),
        # one closed-shell Fock build from the stored integrals: the step an SCF repeats
        dict(name="fock_water16", kind="fock", system="water", units=16, basis="6-31G", spins=1),
        # an unrestricted Fock build of a small open-shell chain: launch-bound
        dict(name="fock_u_alkane3", kind="fock", system="alkane", units=3, basis="6-31G", spins=2),
        # J and K of all co-densities of a spin-flip CI matrix (C2 / cc-pVDZ)
        dict(name="codensity_c2", kind="codensity", system="c2", units=1, basis="cc-pVDZ", count=756),
        # AO -> MO transforms and MP2 pair sums of an 8-water cluster
        dict(name="mp2_water8", kind="mp2", system="water", units=8, basis="6-31G"),
        # scattering intensities of a 4-water cluster on a grid
        dict(name="scattering_water4", kind="scattering", system="water", units=4, basis="6-31G", points=4),
        # one training step of the learned guess on a batch of 96 molecules' pairs
        dict(name="train_10989", kind="train", rows=10989),
        # the learned guess's network on the pairs of a batch of molecules
        dict(name="predict_4097", kind="predict", rows=4097),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "ensemble", "integrals", "fock", "fock", "codensity", "mp2", "scattering", "train", "predict"])
    if kind == "ensemble":
        return dict(kind=kind, units=between(48, 1024), basis=rng.choice(["STO-3G", "6-31G"]))
    if kind in ("train", "predict"):
        return dict(kind=kind, rows=between(200, 65536))
    if kind == "codensity":
        return dict(kind=kind, system=rng.choice(["c2", "water"]), units=1, basis=rng.choice(["6-31G", "cc-pVDZ"]), count=between(2, 756))
    if rng.random() < 0.6:
        system = "water"
        units = rng.choice([u for u in CLUSTERS if u <= (6 if kind == "scattering" else 16)])
        basis = rng.choice(["STO-3G", "6-31G"])
    else:
        system = "alkane"
        units = between(2, 4 if kind == "scattering" else 10)
        basis = rng.choice(["STO-3G", "6-31G", "cc-pVDZ"] if kind != "mp2" and units <= 8 else ["STO-3G", "6-31G"])
    case = dict(kind=kind, system=system, units=units, basis=basis)
    if kind == "integrals":
        case["precision"] = rng.choice(["fp64", "mixed"])
    if kind == "fock":
        case["spins"] = rng.choice([1, 2])
    if kind == "scattering":
        case["points"] = rng.randint(1, 4)
    return case


# ------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------
def _coords(case, seed):
    if case["system"] == "water":
        nx, ny, nz = CLUSTERS[case["units"]]
        return workloads.water_cluster(nx=nx, ny=ny, nz=nz, seed=seed)
    if case["system"] == "alkane":
        return workloads.alkane(case["units"], seed=seed)
    d = 1.25 + 0.02 * np.random.default_rng(seed).normal()
    return [["C", 6.0, 0.0, 0.0, 0.0], ["C", 6.0, 0.3 * d, 0.4 * d, d * math.sqrt(0.75)]]


def _orbitals(centres, seed):
    """Orthonormal orbitals (columns) and ascending energies of a random symmetric matrix
    whose elements fall off with the distance of the functions' centres."""
    rng = np.random.default_rng(seed)
    n = len(centres)
    dist = np.linalg.norm(centres[:, None, :] - centres[None, :, :], axis=-1)
    a = rng.normal(size=(n, n)) * np.exp(-dist / 2.0)
    eps, c = np.linalg.eigh(0.5 * (a + a.T))
    return c, np.where(np.arange(n) < _occupied(n), -20.0, 0.3) + 0.2 * np.arange(n) / n + 0.05 * eps


def _occupied(n):
    return max(1, (2 * n) // 5)


def _centres(coords, basis):
    return np.repeat(_Basis(coords, basis).centre, [2 * l + 1 for l in _Basis(coords, basis).l], axis=0)


def _densities(case, coords, seed):
    c, _ = _orbitals(_centres(coords, case["basis"]), seed)
    o = _occupied(c.shape[0])
    occ = [o] if case.get("spins", 1) == 1 else [o, max(1, o - 1)]
    return [c[:, :k] @ c[:, :k].T for k in occ]


def _codensities(case, coords, seed):
    n = _centres(coords, case["basis"]).shape[0]
    return np.random.default_rng(seed).normal(size=(case["count"], n, n)) * 0.05


def _gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _net(seed):
    rng = np.random.default_rng(seed)
    w = [(rng.normal(size=(a, b)) * math.sqrt(2.0 / a)).astype(np.float32) for a, b in zip(NET[:-1], NET[1:])]
    b = [(0.01 * rng.normal(size=k)).astype(np.float32) for k in NET[1:]]
    return w, b


def _batch(case, seed):
    """Pair features (two one-hot elements, 32 distance Gaussians), targets and slot mask."""
    rng = np.random.default_rng(seed + 1)
    m = case["rows"]
    x = np.zeros((m, NET[0]), dtype=np.float32)
    x[np.arange(m), rng.integers(0, 4, m)] = 1.0
    x[np.arange(m), 4 + rng.integers(0, 4, m)] = 1.0
    mu = np.linspace(0.5, 6.0, 32)
    x[:, 8:] = np.exp(-0.5 * ((rng.uniform(0.7, 6.0, m)[:, None] - mu) / (mu[1] - mu[0])) ** 2)
    return x, rng.normal(size=(m, NET[-1])).astype(np.float32), (rng.random((m, NET[-1])) < 0.7).astype(np.float32)


LEARNING_RATE = 1.0e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return dict(case=case, mols=[Molecule(c, case["basis"]) for c in workloads.ensemble(case["units"], seed=seed)])
    if kind in ("train", "predict"):
        net = PairMLP(dims=NET)
        w, b = _net(seed)
        net.W, net.b = [_gpu(v) for v in w], [_gpu(v) for v in b]
        net.refresh_bf16()
        x, t, mask = _batch(case, seed)
        return dict(case=case, net=net, x=_gpu(x), t=_gpu(t), mask=_gpu(mask))
    coords = _coords(case, seed)
    state = dict(case=case, coords=coords)
    if kind == "solve":
        return state
    state["mol"] = Molecule(coords, case["basis"])
    if kind == "codensity":
        state["w"] = _gpu(_codensities(case, coords, seed))
    elif kind == "mp2":
        c, eps = _orbitals(_centres(coords, case["basis"]), seed)
        o = _occupied(c.shape[0])
        state.update(co=_gpu(c[:, :o]), cv=_gpu(c[:, o:]), eo=_gpu(eps[:o]), ev=_gpu(eps[o:]))
    else:
        state["d"] = [_gpu(d) for d in _densities(case, coords, seed)]
    if kind in ("fock", "codensity", "mp2"):
        state["engine"] = GpuEngine(state["mol"]).prepare()
    return state


def _grid(case):
    return [1.5 * k + 0.5 for k in range(case["points"])]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        out = api.rhf_mp2(state["coords"], case["basis"])
        # the sign of an orbital and the mixing of degenerate ones are arbitrary: the
        # occupied orbitals come back as their density
        c = out["mo_coefficients"][:, :_pairs_of_electrons(state["coords"])]
        return dict(e_rhf=out["E_rhf"], e_mp2=out["E_mp2_corr"], eps=out["mo_energies"], density=c @ c.T)
    if kind == "ensemble":
        r = rhf_batched(EnsembleEngine(state["mols"]).prepare())
        return dict(e=r.E, eps=r.eps, density=r.D)
    if kind == "integrals":
        eng = GpuEngine(state["mol"], precision=case["precision"]).prepare()
        return dict(s=eng.S, h=eng.H, f=eng.fock(state["d"][0]))
    if kind == "fock":
        d = state["d"]
        return state["engine"].fock(d[0]) if len(d) == 1 else state["engine"].fock_u(d[0], d[1])
    if kind == "codensity":
        return state["engine"].coulomb_exchange(state["w"])
    if kind == "mp2":
        ovov = mp2_transform(state["engine"].dense_eri_pairs(compact=True), state["co"], state["cv"])
        return ovov, mp2_pair_sums(ovov, state["eo"], state["ev"])
    if kind == "scattering":
        d = state["d"][0]
        return scattering.intensities(state["mol"], _grid(case), [(d, d)])
    net = state["net"]
    if kind == "predict":
        return net.predict(state["x"])
    y, cache = net.forward(state["x"], keep=True)
    loss, dy = net.loss_grad(y, state["t"], state["mask"])
    grads = net.backward(dy, cache)
    net.adam(grads, LEARNING_RATE)
    return dict(loss=loss, grads=grads, w=net.W, b=net.b)


# ------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------
def _pairs_of_electrons(coords):
    return int(sum(a[1] for a in coords)) // 2


@functools.lru_cache(maxsize=64)
def _counts(text):
    """(AOs, stored integrals, floating-point operations to evaluate them) of a case's
    molecule after Schwarz screening: each unique integral once; per primitive quartet
    the operations of its Hermite integrals and of their two expansions."""
    case = json.loads(text)
    op = ("j0", 2.0) if case["kind"] == "scattering" else ("coulomb", 0.0)
    basis = _Basis(_coords(case, 1), case["basis"])
    pairs = _Pairs(basis)
    q = torch.cat([torch.as_tensor(pairs.schwarz(g, op)) for g in pairs.groups]).cpu().numpy()
    size = np.concatenate([np.full(len(g.a), g.f) for g in pairs.groups]).astype(float)
    work = np.concatenate([np.full(len(g.a), g.prims * g.h) for g in pairs.groups]).astype(float)
    order = np.argsort(-q)
    q, size, work = q[order], size[order], work[order]
    kept = np.searchsorted(-q, -THRESHOLD / np.maximum(q, 1e-300))        # partners of each pair
    csize, cwork = np.concatenate([[0.0], np.cumsum(size)]), np.concatenate([[0.0], np.cumsum(work)])
    return basis.n, 0.5 * float(size @ csize[kept]), 0.5 * float(work @ cwork[kept]) * 12.0


def work(case):
    kind = case["kind"]
    if kind in ("train", "predict"):
        m, weights = case["rows"], sum(a * b for a, b in zip(NET[:-1], NET[1:]))
        if kind == "predict":
            return dict(bytes=4.0 * m * (NET[0] + NET[-1]) + 2.0 * weights, flops=2.0 * m * weights)
        acts = sum(NET[1:-1])           # activations written forward, read backward
        return dict(bytes=4.0 * m * (NET[0] + 2 * NET[-1] + 2 * acts) + 28.0 * weights, flops=6.0 * m * weights - 2.0 * m * NET[0] * NET[1])
    if kind == "ensemble":
        # about 26 AOs a molecule, all integrals kept, 12 iterations of a Fock build and an eigenproblem
        n = 20.0 if case["basis"] == "6-31G" else 10.0
        ints = case["units"] * n ** 4 / 8.0
        return dict(bytes=8.0 * ints * 13, flops=ints * (400.0 + 12 * 12.0) + case["units"] * 12 * 10.0 * n ** 3)
    one = {k: v for k, v in case.items() if k in ("kind", "system", "units", "basis")}
    n, ints, flops = _counts(json.dumps(one, sort_keys=True))
    o = _occupied(n)
    v = n - o
    mp2 = 2.0 * o * n ** 4 / 2 + o * v * n ** 3 + 2.0 * o * o * v * n ** 2 + 2.0 * o * o * v * v * n
    if kind == "fock":
        return dict(bytes=8.0 * (ints + 4 * n * n), flops=12.0 * ints)
    if kind == "codensity":
        return dict(bytes=8.0 * (ints + 3 * case["count"] * n * n), flops=12.0 * ints * case["count"])
    if kind == "mp2":
        return dict(bytes=8.0 * (ints + (o * v) ** 2), flops=mp2)
    if kind == "integrals":
        return dict(bytes=8.0 * (2 * ints + 4 * n * n), flops=flops + 12.0 * ints)
    if kind == "scattering":
        return dict(bytes=8.0 * 2 * ints * case["points"], flops=(flops + 12.0 * ints) * case["points"])
    return dict(bytes=8.0 * (14 * ints + (o * v) ** 2), flops=flops + 13 * (12.0 * ints + 20.0 * n ** 3) + mp2)


# ------------------------------------------------------------------------------------
# the same in plain torch at 64 bits
# ------------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Basis:
    """Shells in the package's order: atoms as given, shells as in the basis library."""

    def __init__(self, coords, basis):
        with open(os.path.join(os.path.dirname(pychem_gb300.__file__), "data", "basis_sets.json")) as fh:
            lib = json.load(fh)[basis.replace("-", "").upper()]
        self.z = np.array([float(a[1]) for a in coords])
        self.xyz = np.array([a[2:5] for a in coords], dtype=float) * TO_BOHR
        self.l, self.exps, self.coef, centre = [], [], [], []
        for atom, at in zip(coords, self.xyz):
            for fn in lib[atom[0].upper()]:
                l = int(fn[0])
                e = np.array([p[0] for p in fn[1:]])
                norm = 1.0 / math.sqrt(math.gamma(l + 0.5) * math.pi)
                self.l.append(l)
                self.exps.append(e)
                self.coef.append(np.array([p[1] for p in fn[1:]]) * (2.0 * e) ** ((l + 1.5) / 2.0) * norm)
                centre.append(at)
        self.centre = np.array(centre)
        self.ao = np.concatenate([[0], np.cumsum([2 * l + 1 for l in self.l])]).astype(int)
        self.n = int(self.ao[-1])


_CARTESIAN = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
              2: [(2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2)]}
_R3 = math.sqrt(3.0)
_SPHERICAL = {0: [[1.0]], 1: [[1.0, 0, 0], [0, 1.0, 0], [0, 0, 1.0]],
              2: [[_R3 / 2, 0, 0, -_R3 / 2, 0, 0], [0, _R3, 0, 0, 0, 0], [0, 0, _R3, 0, 0, 0], [0, 0, 0, 0, _R3, 0],
                  [-0.5, 0, 0, -0.5, 0, 1.0]]}


def _hermites(l):
    return [(t, u, v) for t in range(l + 1) for u in range(l + 1 - t) for v in range(l + 1 - t - u)]


def _expansion(a, b, ab, la, lb):
    """E[i][j][t] of one direction for exponents a, b and centre difference ab."""
    p = a + b
    e = {(0, 0, 0): torch.exp(-a * b / p * ab * ab)}
    pa, pb, h = -b / p * ab, a / p * ab, 0.5 / p

    def at(i, j, t):
        return e.get((i, j, t), 0.0)

    for i in range(la + 1):
        for j in range(lb + 1):
            if i == j == 0:
                continue
            for t in range(i + j + 1):
                if i:
                    e[i, j, t] = h * at(i - 1, j, t - 1) + pa * at(i - 1, j, t) + (t + 1) * at(i - 1, j, t + 1)
                else:
                    e[i, j, t] = h * at(i, j - 1, t - 1) + pb * at(i, j - 1, t) + (t + 1) * at(i, j - 1, t + 1)
    return e


class _Group:
    """Shell pairs of one kind (la >= lb, equal primitive counts)."""

    def __init__(self, basis, a, b, dev):
        self.a, self.b = np.array(a), np.array(b)
        la, lb = basis.l[a[0]], basis.l[b[0]]
        self.l, self.fa, self.fb = la + lb, 2 * la + 1, 2 * lb + 1
        self.f, self.h = self.fa * self.fb, len(_hermites(la + lb))
        na, nb = len(basis.exps[a[0]]), len(basis.exps[b[0]])
        self.prims = na * nb

        def table(x):
            return torch.as_tensor(np.array(x), dtype=torch.float64, device=dev)

        ea = table([basis.exps[i] for i in a])[:, :, None].expand(-1, na, nb).reshape(-1, na * nb)
        eb = table([basis.exps[i] for i in b])[:, None, :].expand(-1, na, nb).reshape(-1, na * nb)
        cc = (table([basis.coef[i] for i in a])[:, :, None] * table([basis.coef[i] for i in b])[:, None, :]).reshape(-1, na * nb)
        ra, rb = table(basis.centre[self.a]), table(basis.centre[self.b])
        self.p = ea + eb
        self.centre = (ea[..., None] * ra[:, None] + eb[..., None] * rb[:, None]) / self.p[..., None]
        e = [_expansion(ea, eb, (ra - rb)[:, x, None], la, lb + 2) for x in range(3)]
        ca, cb = _CARTESIAN[la], _CARTESIAN[lb]
        zero = torch.zeros_like(ea)
        cart = torch.stack([torch.stack([torch.stack([
            cc * math.prod((e[x].get((i[x], j[x], t[x]), zero) for x in range(3)), start=1.0)
            for t in _hermites(la + lb)], -1) for j in cb], -2) for i in ca], -3)      # pair, prim, ca, cb, hermite
        sa, sb = table(_SPHERICAL[la]), table(_SPHERICAL[lb])
        self.e = torch.einsum("si,rj,pkijh->pksrh", sa, sb, cart).reshape(len(a), na * nb, self.f, self.h)
        # overlap and kinetic energy: x^i against the second derivative of the x^j Gaussian
        s, kin = [], []
        for i in ca:
            for j in cb:
                sx = [e[x].get((i[x], j[x], 0), zero) for x in range(3)]
                kx = [eb * (2 * j[x] + 1) * sx[x] - 2.0 * eb * eb * e[x].get((i[x], j[x] + 2, 0), zero)
                      - (0.5 * j[x] * (j[x] - 1) * e[x].get((i[x], j[x] - 2, 0), zero) if j[x] > 1 else 0.0) for x in range(3)]
                w = cc * (math.pi / self.p) ** 1.5
                s.append((w * sx[0] * sx[1] * sx[2]).sum(1))
                kin.append((w * (kx[0] * sx[1] * sx[2] + sx[0] * kx[1] * sx[2] + sx[0] * sx[1] * kx[2])).sum(1))
        self.s, self.kin = (torch.einsum("si,rj,pij->psr", sa, sb, torch.stack(m, 1).reshape(-1, len(ca), len(cb))) for m in (s, kin))


def _boys(top, t):
    """F_0 .. F_top: ascending series of the highest and downward recursion, the
    asymptotic form where exp(-t) is below rounding."""
    big = t > 40.0
    x = torch.where(big, torch.zeros_like(t), t)
    term = torch.full_like(t, 1.0 / (2 * top + 1))
    acc = term.clone()
    for k in range(1, 130):
        term = term * (2.0 * x) / (2 * top + 2 * k + 1)
        acc += term
    ex = torch.exp(-x)
    f = [None] * (top + 1)
    f[top] = ex * acc
    for m in range(top, 0, -1):
        f[m - 1] = (2.0 * x * f[m] + ex) / (2 * m - 1)
    y = torch.where(big, t, torch.ones_like(t))
    g = 0.5 * torch.sqrt(math.pi / y)
    for m in range(top + 1):
        f[m] = torch.where(big, g, f[m])
        g = g * (2 * m + 1) / (2.0 * y)
    return f


def _bessel(top, z):
    """j_m(z) / z^m, m = 0 .. top: the power series below 9, upward recursion above."""
    small = z < 9.0
    x = torch.where(small, z, torch.ones_like(z))
    y = torch.where(small, torch.full_like(z, 9.0), z)
    up = [torch.sin(y) / y, (torch.sin(y) / y - torch.cos(y)) / y]
    for m in range(1, top):
        up.append((2 * m + 1) / y * up[m] - up[m - 1])
    out = []
    for m in range(top + 1):
        term = torch.full_like(z, 1.0 / math.prod(range(1, 2 * m + 2, 2)))
        acc = term.clone()
        for k in range(1, 45):
            term = term * (-0.5 * x * x) / (k * (2 * m + 2 * k + 1))
            acc += term
        out.append(torch.where(small, acc, up[m] / y ** m))
    return out


def _hermite_integrals(top, p, q, r, op):
    """R_tuv for t + u + v <= top: derivatives of the operator between two spherical
    Gaussians of exponents p and q at distance vector r (1/r12 or j0(S r12))."""
    rho = p * q / (p + q)
    r2 = (r * r).sum(-1)
    if op[0] == "coulomb":
        pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        n0 = [pre * (-2.0 * rho) ** m * f for m, f in enumerate(_boys(top, rho * r2))]
    else:
        s2 = op[1] ** 2
        pre = (math.pi ** 2 / (p * q)) ** 1.5 * torch.exp(-0.25 * s2 / rho)
        n0 = [pre * (-s2) ** m * j for m, j in enumerate(_bessel(top, op[1] * torch.sqrt(r2)))]
    level = {(0, 0, 0): n0}          # R^(n)_tuv by tuv: a list over n
    for l in range(1, top + 1):
        for h in [h for h in _hermites(top) if sum(h) == l]:
            x = next(k for k in range(3) if h[k])
            less = tuple(h[k] - (k == x) for k in range(3))
            least = tuple(h[k] - 2 * (k == x) for k in range(3))
            level[h] = [r[..., x] * level[less][n + 1] + ((h[x] - 1) * level[least][n + 1] if h[x] > 1 else 0.0)
                        for n in range(top - l + 1)]
    return {h: v[0] for h, v in level.items()}


class _Pairs:
    def __init__(self, basis, dev=None):
        self.dev = dev or _device()
        self.basis = basis
        kinds = {}
        for i in range(len(basis.l)):
            for j in range(i + 1):
                a, b = (i, j) if basis.l[i] >= basis.l[j] else (j, i)
                kinds.setdefault((basis.l[a], basis.l[b], len(basis.exps[a]), len(basis.exps[b])), []).append((a, b))
        self.groups = [_Group(basis, [x[0] for x in v], [x[1] for x in v], self.dev) for _, v in sorted(kinds.items())]

    def block(self, x, y, i, j, op):
        """(ab|cd) of bra pairs i of group x with ket pairs j of group y, broadcast."""
        p, q = x.p[i][:, :, None], y.p[j][:, None, :]
        r = x.centre[i][:, :, None] - y.centre[j][:, None, :]
        herm = _hermite_integrals(x.l + y.l, p, q, r, op)
        hx, hy = _hermites(x.l), _hermites(y.l)
        out = 0.0
        ex, ey = x.e[i], y.e[j]
        for k, h in enumerate(hx):
            half = torch.zeros(p.shape[0], p.shape[1], y.f, dtype=torch.float64, device=self.dev)
            for m, g in enumerate(hy):
                full = herm[tuple(s + t for s, t in zip(h, g))]
                half += (-1.0) ** sum(g) * torch.bmm(full, ey[..., m])
            out = out + torch.bmm(ex[..., k].transpose(1, 2), half)
        return out

    def schwarz(self, g, op):
        every = torch.arange(len(g.a), device=self.dev)
        out = []
        for i in every.split(max(1, 1000000 // g.prims ** 2)):
            out.append(torch.diagonal(self.block(g, g, i, i, op), dim1=1, dim2=2).amax(1).clamp_min(0.0).sqrt())
        return torch.cat(out)

    def tensor(self, op=("coulomb", 0.0)):
        """The screened integrals as a dense (n, n, n, n) tensor."""
        n, ao = self.basis.n, self.basis.ao
        bounds = [self.schwarz(g, op) for g in self.groups]
        out = torch.zeros(n, n, n, n, dtype=torch.float64, device=self.dev)

        def functions(g, i):
            sa, sb = (torch.as_tensor(ao[s], device=self.dev)[i] for s in (g.a, g.b))
            fa = sa[:, None] + torch.arange(g.fa, device=self.dev).repeat_interleave(g.fb)
            fb = sb[:, None] + torch.arange(g.fb, device=self.dev).repeat(g.fa)
            return fa, fb

        for gi, x in enumerate(self.groups):
            for gj, y in enumerate(self.groups[:gi + 1]):
                keep = bounds[gi][:, None] * bounds[gj][None, :] > THRESHOLD
                if gi == gj:
                    keep = torch.tril(keep) | torch.eye(len(x.a), dtype=torch.bool, device=self.dev)
                for part in keep.nonzero().split(max(1, 3000000 // (x.prims * y.prims))):
                    i, j = part[:, 0], part[:, 1]
                    v = self.block(x, y, i, j, op)
                    (a, b), (c, d) = functions(x, i), functions(y, j)
                    a, b, c, d = (t.expand_as(v) for t in (a[:, :, None], b[:, :, None], c[:, None, :], d[:, None, :]))
                    for k in ((a, b, c, d), (b, a, c, d), (a, b, d, c), (b, a, d, c), (c, d, a, b), (d, c, a, b), (c, d, b, a), (d, c, b, a)):
                        out[k] = v
        return out

    def one_electron(self):
        n, ao = self.basis.n, self.basis.ao
        s, h = np.zeros((n, n)), np.zeros((n, n))
        for g in self.groups:
            v = 0.0
            for z, at in zip(self.basis.z, self.basis.xyz):
                r = g.centre - torch.as_tensor(at, device=self.dev)
                fs = _boys(g.l, g.p * (r * r).sum(-1))
                # a nucleus is the limit q -> infinity of a normalised Gaussian charge
                level = {(0, 0, 0): [2.0 * math.pi / g.p * (-2.0 * g.p) ** m * f for m, f in enumerate(fs)]}
                for l in range(1, g.l + 1):
                    for t in [t for t in _hermites(g.l) if sum(t) == l]:
                        x = next(k for k in range(3) if t[k])
                        less, least = (tuple(t[k] - c * (k == x) for k in range(3)) for c in (1, 2))
                        level[t] = [r[..., x] * level[less][m + 1] + ((t[x] - 1) * level[least][m + 1] if t[x] > 1 else 0.0)
                                    for m in range(g.l - l + 1)]
                herm = torch.stack([level[t][0] for t in _hermites(g.l)], -1)
                v = v - z * torch.einsum("pkfh,pkh->pf", g.e, herm)
            v = v.reshape(-1, g.fa, g.fb)
            for k, (a, b) in enumerate(zip(g.a, g.b)):
                ra, rb = slice(ao[a], ao[a + 1]), slice(ao[b], ao[b + 1])
                for m, blk in ((s, g.s[k]), (h, g.kin[k] + v[k])):
                    blk = blk.cpu().numpy()
                    m[ra, rb], m[rb, ra] = blk, blk.T
        return torch.as_tensor(s, device=self.dev), torch.as_tensor(h, device=self.dev)


def _coulomb(eri, d):
    n = d.shape[-1]
    return (eri.reshape(n * n, n * n) @ d.reshape(-1)).reshape(n, n)


def _exchange(eri, d):
    """K_ad = sum_bc (ab|cd) W_cb."""
    return torch.einsum("abcd,cb->ad", eri, d)


def _scf(basis, s, h, eri, o):
    """Closed-shell SCF to a commutator below 1e-11 from the core guess, damped at first."""
    w, u = torch.linalg.eigh(s)
    x = u * w.rsqrt()
    eps, c = torch.linalg.eigh(x.T @ h @ x)
    d = x @ c[:, :o] @ c[:, :o].T @ x.T
    fs, rs = [], []
    for it in range(200):
        f = h + 2.0 * _coulomb(eri, d) - _exchange(eri, d)
        r = x.T @ (f @ d @ s - s @ d @ f) @ x
        e = float((d * (h + f)).sum())
        if float(r.abs().max()) < 1e-11:
            break
        fs, rs = (fs + [f])[-8:], (rs + [r])[-8:]
        m = len(fs)
        b = -np.ones((m + 1, m + 1))
        b[m, m] = 0.0
        b[:m, :m] = [[float((p * q).sum()) for q in rs] for p in rs]
        b[:m, :m] /= b[:m, :m].max()
        k = np.linalg.lstsq(b, np.append(np.zeros(m), -1.0), rcond=None)[0][:m]
        fx = sum(float(a) * q for a, q in zip(k, fs))
        eps, c = torch.linalg.eigh(x.T @ fx @ x)
        new = x @ c[:, :o] @ c[:, :o].T @ x.T
        d = 0.5 * (d + new) if it < 3 else new
    eps, c = torch.linalg.eigh(x.T @ f @ x)
    i, j = np.tril_indices(len(basis.z), -1)
    repulsion = float((basis.z[i] * basis.z[j] / np.linalg.norm(basis.xyz[i] - basis.xyz[j], axis=1)).sum())
    return e + repulsion, eps, x @ c


def _transformed(eri, co, cv):
    t = torch.einsum("abcd,ai->ibcd", eri, co)
    t = torch.einsum("ibcd,bj->ijcd", t, cv)
    t = torch.einsum("ijcd,ck->ijkd", t, co)
    return torch.einsum("ijkd,dl->ijkl", t, cv)


def _pair_sums(g, eo, ev):
    den = eo[:, None, None, None] - ev[None, :, None, None] + eo[None, None, :, None] - ev[None, None, None, :]
    return float((g * g / den).sum()), float((g * g.permute(0, 3, 2, 1) / den).sum())


def _exact_network(case, seed):
    x, t, mask = (torch.as_tensor(v, device=_device()).double() for v in _batch(case, seed))
    w32, b32 = _net(seed)
    w = [torch.as_tensor(v, device=_device()) for v in w32]
    b = [torch.as_tensor(v, device=_device()).double() for v in b32]
    wb = [v.to(torch.bfloat16).double().requires_grad_() for v in w]        # the products take BF16 weights
    b = [v.requires_grad_() for v in b]
    y = x
    for k in range(len(w)):
        y = y @ wb[k] + b[k]
        if k < len(w) - 1:
            y = y * torch.sigmoid(y)
    if case["kind"] == "predict":
        return y.detach()
    loss = ((y - t) ** 2 * mask).sum() / mask.sum()
    grads = torch.autograd.grad(loss, wb + b)
    gw, gb = grads[:len(w)], grads[len(w):]
    # the first Adam step: moments are the gradient itself after bias correction
    step = [LEARNING_RATE * g / (g.abs() + 1e-8) for g in grads]
    return dict(loss=loss.detach().reshape(1), grads=list(zip(gw, gb)),
                w=[v.double() - s for v, s in zip(w, step)], b=[v.detach() - s for v, s in zip(b, step[len(w):])])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "predict"):
        return _exact_network(case, seed)
    if kind == "ensemble":
        return None                    # tens to a thousand SCFs: minutes
    coords = _coords(case, seed)
    basis = _Basis(coords, case["basis"])
    if basis.n > (EXACT_SCF_AO if kind == "solve" else EXACT_AO):
        return None                    # over 20 seconds
    pairs = _Pairs(basis)
    if kind == "scattering":
        d = torch.as_tensor(_densities(case, coords, seed)[0], device=pairs.dev)
        rows = []
        for s in _grid(case):
            eri = pairs.tensor(("j0", s))
            rows.append([float(sum(a[1] for a in coords)) + float((d * (4.0 * _coulomb(eri, d) - 2.0 * _exchange(eri, d))).sum())])
        return np.array(rows)
    eri = pairs.tensor()
    if kind == "codensity":
        w = torch.as_tensor(_codensities(case, coords, seed), device=pairs.dev)
        return torch.einsum("abcd,xcd->xab", eri, w), torch.einsum("abcd,xcb->xad", eri, w)
    if kind == "mp2":
        c, eps = _orbitals(_centres(coords, case["basis"]), seed)
        c, eps = torch.as_tensor(c, device=pairs.dev), torch.as_tensor(eps, device=pairs.dev)
        o = _occupied(basis.n)
        g = _transformed(eri, c[:, :o], c[:, o:])
        return g, _pair_sums(g, eps[:o], eps[o:])
    s, h = pairs.one_electron()
    if kind == "solve":
        o = _pairs_of_electrons(coords)
        e, eps, c = _scf(basis, s, h, eri, o)
        s1, s2 = _pair_sums(_transformed(eri, c[:, :o], c[:, o:]), eps[:o], eps[o:])
        return dict(e_rhf=e, e_mp2=2.0 * s1 - s2, eps=eps, density=c[:, :o] @ c[:, :o].T)
    d = [torch.as_tensor(v, device=pairs.dev) for v in _densities(case, coords, seed)]
    if kind == "integrals":
        return dict(s=s, h=h, f=h + 2.0 * _coulomb(eri, d[0]) - _exchange(eri, d[0]))
    if len(d) == 1:
        return h + 2.0 * _coulomb(eri, d[0]) - _exchange(eri, d[0])
    j = _coulomb(eri, d[0] + d[1])
    return h + j - _exchange(eri, d[0]), h + j - _exchange(eri, d[1])
