"""The workloads this framework's performance is judged on, as a user's program calls them.

Every case goes through the public Python mirror of the C ABI: `ExcitedStateSystem` (A.X products,
TDA roots), `GradientSystem`, `scc_batch`, and the FMO entry points `solve_batch` and
`exciton_states`.  Molecules are those of the framework's own configurations: linear acenes (one
to ten rings), all-trans polyenes, jittered water clusters up to (H2O)128 and acene aggregates up
to 64 monomers.  Positions are displaced at random from the seed, so every seed is another molecule.

The inputs (orbitals, overlaps, gamma matrices) come from a host ground state: a numpy SCC for the
single molecules, and for the large aggregates a few SCC iterations from the neutral atoms, whose
orbitals are orthonormal and have the magnitudes and the block structure of converged ones.

`exact` restates the quantities in 64 bits with plain torch on the CPU: products and transition
charges by their definitions, TDA energies by diagonalising the dense matrix, the SCC by its own
iteration, the gradients by automatic differentiation of the energy expressions at fixed densities.
"""

import math

import numpy as np
import torch

from tincr_gb300 import _lib
from tincr_gb300 import fmo
from tincr_gb300 import geometry as G
from tincr_gb300 import gradients as GR
from tincr_gb300 import groundstate as gs
from tincr_gb300 import params as P
from tincr_gb300 import scc as gscc
from tincr_gb300 import tda as T

PRECISION = {"fp64": _lib.PREC_FP64, "mixed": _lib.PREC_BF16X3}
R_LR_WATER = 1.0 / 0.3     # omega = 0.3 bohr^-1, the water clusters' setting


# ----------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------

def listed():
    return [
        # one A.X product of a small molecule, as a caller's own solver asks for: the smallest call
        dict(name="product-naphthalene-fp64", kind="product", mol="acene", size=2, lc=True, k=1, precision="fp64"),
        # a block of trial vectors of the largest single system, in the plain and in the mixed form
        dict(name="product-water128-fp64", kind="product", mol="water", size=128, lc=True, k=20, precision="fp64"),
        dict(name="product-water128-mixed", kind="product", mol="water", size=128, lc=True, k=20, precision="mixed"),
        # excited states of one molecule without long-range correction: C20H22, 10 roots to 1e-6
        dict(name="tda-polyene20-fp64", kind="tda", mol="polyene", size=20, lc=False, k=10, tol=1e-6, precision="fp64"),
        # the flagship solve: 20 LC-TDA roots of the water cluster in the mixed form
        dict(name="tda-water128-mixed", kind="tda", mol="water", size=128, lc=True, k=20, tol=1e-4, precision="mixed"),
        # S0 and S1 gradients of decacene (a geometry optimisation's step), plain form
        dict(name="gradient-decacene-fp64", kind="gradient", mol="acene", size=10, lc=True, precision="fp64"),
        # the same for a water cluster with the roots of a mixed solve
        dict(name="gradient-water48-mixed", kind="gradient", mol="water", size=48, lc=True, precision="mixed"),
        # ground state of one molecule: the SCC of decacene
        dict(name="scc-decacene", kind="scc", size=10, count=1, dimers=False, lc=True, fp32_start=False, full=True),
        # the ground states of an aggregate's stacked dimers (FMO set-up)
        dict(name="scc-dimers128", kind="scc", size=5, count=128, dimers=True, lc=True, fp32_start=False, full=False),
        # batched FMO excited states: LE roots of every monomer, CT roots of both directions of every
        # close pair; a small aggregate in the plain form, the 64-acene aggregate in the mixed form
        dict(name="fmo-acenes8-fp64", kind="fmo", nx=2, ny=2, nz=2, lc=True, n_le=4, n_ct=1, precision="fp64"),
        dict(name="fmo-acenes64-mixed", kind="fmo", nx=4, ny=4, nz=4, lc=True, n_le=4, n_ct=1, precision="mixed"),
        # exciton Hamiltonian of the 64-acene aggregate and its 10 lowest states
        dict(name="exciton-acenes64-mixed", kind="exciton", nx=4, ny=4, nz=4, n_le=4, n_ct=1, precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "tda", "gradient", "scc", "fmo", "fmo", "exciton"])
    precision = rng.choice(["fp64", "mixed"])
    if kind in ("product", "tda", "gradient"):
        mol = rng.choice(["acene", "polyene", "water"])
        top = {"product": 128, "tda": 64, "gradient": 48}[kind]
        size = {"acene": lambda: rng.randint(1, 10), "polyene": lambda: 2 * rng.randint(2, 12),
                "water": lambda: _log_int(rng, 8, top)}[mol]()
        c = dict(kind=kind, mol=mol, size=size, lc=rng.random() < 0.75, precision=precision)
        if kind == "product":
            c["k"] = _log_int(rng, 1, 20)
        if kind == "tda":
            c.update(k=rng.randint(1, 12), tol=rng.choice([1e-4, 1e-6]) if precision == "fp64" else 1e-4)
        return c
    if kind == "scc":
        size = rng.randint(2, 10)
        dimers = size <= 5 and rng.random() < 0.5
        return dict(kind="scc", size=size, count=_log_int(rng, 1, 40 if size <= 5 else 4), dimers=dimers,
                    lc=rng.random() < 0.75, fp32_start=rng.random() < 0.25, full=rng.random() < 0.5)
    nx, ny, nz = rng.randint(1, 4), rng.randint(1, 4), rng.randint(1, 3)
    if nx * ny * nz < 2:
        nx = 2
    if kind == "fmo":
        return dict(kind="fmo", nx=nx, ny=ny, nz=nz, lc=rng.random() < 0.75, n_le=rng.randint(1, 5), n_ct=1,
                    precision=precision)
    return dict(kind="exciton", nx=nx, ny=ny, nz=nz, n_le=rng.randint(3, 4), n_ct=1, precision=precision)


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------

def _water_lattice(count):
    """Smallest nx >= ny >= nz lattice (8 x 4 x 4 at most) with at least `count` sites."""
    for nx, ny, nz in ((2, 2, 2), (3, 2, 2), (3, 3, 2), (3, 3, 3), (4, 3, 3), (4, 4, 3), (4, 4, 4), (6, 4, 4)):
        if nx * ny * nz >= count:
            return nx, ny, nz
    return 8, 4, 4


def _molecule(mol, size, seed):
    """Atomic numbers and positions (bohr) of one molecule, displaced at random from the seed."""
    rng = np.random.default_rng(seed)
    if mol == "water":
        z, x = G.water_cluster(*_water_lattice(size), seed=seed)
        return z[:3 * size], G.to_bohr(x[:3 * size])
    z, x = G.acene(size) if mol == "acene" else G.polyene(size)
    return z, G.to_bohr(x + rng.uniform(-0.03, 0.03, size=x.shape))


def _ground(sy, tol=1e-10, max_iter=60):
    """Restricted SCC of a System on the host with DIIS; `max_iter` small gives an early iterate."""
    s, h0 = gs.h0_and_s(sy)
    gam = gs.gamma_atomwise(sy, 0.0)
    glr = gs.gamma_atomwise(sy, sy.r_lr) if sy.lc else np.zeros_like(gam)
    f, p, e, c, dq, it = _scf(sy, s, h0, gam, glr if sy.lc else None, tol, max_iter)
    return gs.GroundState(s=s, h0=h0, gamma=gam, gamma_lr=glr, orbs=np.ascontiguousarray(c), orbe=e, p=p,
                          p0=np.diag(sy.ao_occ.astype(np.float64)), dq=dq, h_coul_x=f, energy=0.0, iterations=it)


def _scf(sy, s, h0, gam, glr, tol, max_iter):
    """(Fock matrix, density, orbital energies, orbitals, charges, iterations) of the SCC equations."""
    at, n_occ = sy.ao_atom, sy.n_elec // 2
    g = None if glr is None else glr[np.ix_(at, at)]
    p0 = np.diag(sy.ao_occ.astype(np.float64))
    w, u = np.linalg.eigh(s)
    x = (u / np.sqrt(w)) @ u.T
    fs, es = [], []
    p = p0
    charges = lambda d: np.bincount(at, weights=np.einsum("ij,ji->i", s, d), minlength=sy.n_atoms)
    for it in range(1, max_iter + 1):
        d = p - p0
        v = (gam @ charges(d))[at]
        f = h0 + 0.5 * (v[:, None] + v[None, :]) * s
        if g is not None:
            sd = s @ d
            t = (g * sd) @ s
            hx = t + t.T + g * (sd @ s) + s @ (d * g) @ s
            f = f - 0.0625 * (hx + hx.T)
        r = x @ (f @ p @ s - s @ p @ f) @ x
        fs, es = (fs + [f])[-8:], (es + [r])[-8:]
        if it > 1 and np.abs(r).max() < tol:
            break
        m = len(fs)
        b = np.full((m + 1, m + 1), -1.0)
        b[:m, :m] = [[np.vdot(a, c) for c in es] for a in es]
        b[m, m] = 0.0
        rhs = np.zeros(m + 1)
        rhs[m] = -1.0
        q = np.linalg.solve(b, rhs)[:m] if m > 1 else [1.0]
        e, c = np.linalg.eigh(x @ sum(k * a for k, a in zip(q, fs)) @ x)
        c = x @ c
        p = 2.0 * c[:, :n_occ] @ c[:, :n_occ].T
    e, c = np.linalg.eigh(x @ f @ x)
    c = x @ c
    p = 2.0 * c[:, :n_occ] @ c[:, :n_occ].T
    return f, p, e, c, charges(p - p0), it


def _system(case, seed):
    """System and ground state of a single-molecule case."""
    z, x = _molecule(case["mol"], case["size"], seed)
    sy = gs.build_system(z, x, lc=case["lc"], r_lr=R_LR_WATER if case["mol"] == "water" else gs.LONG_RANGE_RADIUS)
    # a looser ground state for the largest clusters (768 orbitals take seconds on a host)
    return sy, _ground(sy, tol=1e-5 if sy.n_orbs > 400 else 1e-10)


def _scc_systems(case, seed):
    """Acenes, or stacked acene dimers (3.5 to 4 Angstrom apart), of 2 .. size rings."""
    out = []
    for i in range(case["count"]):
        rng = np.random.default_rng([seed, i])
        rings = [2 + (5 * i) % (case["size"] - 1), 2 + (3 * i + 1) % (case["size"] - 1)]
        z, x = _molecule("acene", rings[0] if case["count"] > 1 else case["size"], int(rng.integers(1 << 31)))
        if case["dimers"]:
            z2, x2 = _molecule("acene", rings[1], int(rng.integers(1 << 31)))
            z = np.concatenate([z, z2])
            x = np.concatenate([x, x2 + G.to_bohr([rng.uniform(3.5, 4.0), rng.uniform(0, 1), rng.uniform(0, 2)])])
        out.append(gs.build_system(z, x, lc=case["lc"]))
    return out


class _Aggregate:
    """Monomers, pairs and work list of an acene aggregate, and what the exciton Hamiltonian reads
    (the attributes of `fmo.ExcitonSetup`), cut from one overlap and one gamma matrix of the whole."""

    def __init__(self, case, seed, exciton):
        lc = case.get("lc", True)
        z, x, mono = G.acene_lattice(case["nx"], case["ny"], case["nz"])
        still = G.to_bohr(x)
        x = still + G.to_bohr(np.random.default_rng(seed).uniform(-0.03, 0.03, size=x.shape))
        whole = gs.build_system(z, x, lc=lc)
        self.s, _ = gs.h0_and_s(whole)
        self.gamma = gs.gamma_atomwise(whole, 0.0)
        self.gamma_lr = gs.gamma_atomwise(whole, whole.r_lr) if lc else np.zeros_like(self.gamma)
        self.monomers = []
        for m in range(int(mono[-1]) + 1):
            at = np.nonzero(mono == m)[0]
            sy = gs.build_system(z[at], x[at], lc=lc)
            self.monomers.append(fmo.Monomer(m, at, sy, _ground(sy, max_iter=5)))
        self.ao = np.concatenate([[0], np.cumsum([m.system.n_orbs for m in self.monomers])])
        self.atom_offset = np.concatenate([[0], np.cumsum([m.system.n_atoms for m in self.monomers])])
        n = len(self.monomers)
        rest = [fmo.Monomer(m.index, m.atoms, gs.build_system(z[m.atoms], still[m.atoms], lc=lc), None)
                for m in self.monomers]
        self.ct_pairs = fmo.close_pairs(rest, 4.5 / P.BOHR_TO_ANGS)
        self.instances, self.labels = [], []
        for m in self.monomers:
            self.instances.append(fmo.monomer_instance(m, case["n_le"]))
            self.labels.append(("LE", m.index))
        for i, j in self.ct_pairs:
            for h, l in ((i, j), (j, i)):
                self.instances.append(self._ct_instance(h, l, lc, case["n_ct"]))
                self.labels.append(("CT", h, l))
        if exciton:
            self.real = {(i, j): False for i in range(n) for j in range(i + 1, n)}
            for i, j in fmo.candidate_pairs(rest, 2.0 * max(fmo.VDW_SUM_BOHR.values())):
                self.real[(i, j)] = fmo.is_real_pair(rest[i], rest[j])
            self.real_pairs = sorted(k for k, v in self.real.items() if v)
            self.pair_scc = self._pair_orbitals()

    def _two(self, h, l):
        ao = np.r_[self.ao[h]:self.ao[h + 1], self.ao[l]:self.ao[l + 1]]
        at = np.r_[self.atom_offset[h]:self.atom_offset[h + 1], self.atom_offset[l]:self.atom_offset[l + 1]]
        return ao, at

    def _ct_instance(self, h, l, lc, n_ct):
        mh, ml = self.monomers[h], self.monomers[l]
        ao, at = self._two(h, l)
        nh, oh, vl = mh.system.n_orbs, mh.system.n_occ, ml.system.n_virt
        c = np.zeros((len(ao), oh + vl))
        c[:nh, :oh] = mh.ground.orbs[:, :oh]
        c[nh:, oh:] = ml.ground.orbs[:, ml.system.n_occ:]
        return dict(n_atoms=len(at), n_orb=len(ao), n_occ=oh, n_virt=vl, n_roots=n_ct,
                    opa=np.concatenate([mh.system.orbs_per_atom, ml.system.orbs_per_atom]).astype(np.int32), c=c,
                    s=self.s[np.ix_(ao, ao)],
                    orbe=np.concatenate([mh.ground.orbe[:oh], ml.ground.orbe[ml.system.n_occ:]]),
                    gamma=self.gamma[np.ix_(at, at)], gamma_lr=self.gamma_lr[np.ix_(at, at)] if lc else None,
                    xyz=np.concatenate([mh.system.xyz, ml.system.xyz]))

    def _pair_orbitals(self):
        """Pair ground states: the two monomers' orbitals, orthonormalised in the pair's overlap by
        C <- C (15 - 10 M + 3 M^2) / 8, M = C^T S C, and the monomers' orbital energies."""
        out = {}
        for i, j in self.real_pairs:
            a, b = self.monomers[i].ground, self.monomers[j].ground
            ao, _ = self._two(i, j)
            n, na = len(ao), len(a.orbe)
            c = np.zeros((n, n))
            c[:na, :na], c[na:, na:] = a.orbs, b.orbs
            m = np.eye(n)
            m[:na, na:] = a.orbs.T @ self.s[np.ix_(ao[:na], ao[na:])] @ b.orbs
            m[na:, :na] = m[:na, na:].T
            out[(i, j)] = (c @ (1.875 * np.eye(n) - 1.25 * m + 0.375 * (m @ m)), np.concatenate([a.orbe, b.orbe]))
        return out

    def s_block(self, i, j):
        return np.ascontiguousarray(self.s[self.ao[i]:self.ao[i + 1], self.ao[j]:self.ao[j + 1]])


class _Inputs(dict):
    """The host part of a state: molecules, ground states, vectors."""

    def __init__(self, case, seed):
        super().__init__(case=case)
        kind = case["kind"]
        if kind in ("product", "tda", "gradient"):
            sy, g = _system(case, seed)
            self.update(system=sy, ground=g)
            if kind == "product":
                x = np.random.default_rng([seed, 1]).normal(size=(sy.n_occ * sy.n_virt, case["k"]))
                self["x"] = x / np.linalg.norm(x, axis=0)
            if kind == "gradient":
                self["e"], self["x"] = _ci_state(sy, g)
        elif kind == "scc":
            self["systems"] = _scc_systems(case, seed)
        else:
            self["aggregate"] = _Aggregate(case, seed, kind == "exciton")
            if kind == "exciton":
                self["results"] = _unit_states(self["aggregate"])


def prepare(case, seed):
    state = _Inputs(case, seed)
    state["ctx"] = _lib.Context(0)
    if case["kind"] in ("product", "gradient"):
        es = T.ExcitedStateSystem.from_ground_state(state["ctx"], state["system"], state["ground"])
        es.prepare_tda()
        state["es"] = es
    if case["kind"] == "gradient":
        es.set_states(state["e"], state["x"])
        es.set_precision(PRECISION[case["precision"]])
        state["gradient"] = GR.GradientSystem(es, state["system"], state["ground"])
    return state


def _ci_state(sy, g):
    """A normalised CI vector and energy of the shape an S1 root has: weights falling with the
    orbital energy difference of each single excitation, a few of them large."""
    om = g.orbe[sy.n_occ:][None, :] - g.orbe[:sy.n_occ, None]
    x = np.exp(-12.0 * (om - om.min())) * np.cos(1.0 + np.arange(om.size).reshape(om.shape))
    x /= np.linalg.norm(x)
    return np.array([0.8 * om.min()]), x.reshape(-1, 1)


def _unit_states(agg):
    """LE and CT roots of the work list in the form `solve_batch` returns them: CI vectors on the
    lowest single excitations, orthonormal per instance, with their transition charges."""
    out = []
    for q in agg.instances:
        o, v, nr, n = q["n_occ"], q["n_virt"], q["n_roots"], q["n_orb"]
        om = (q["orbe"][o:o + v][None, :] - q["orbe"][:o, None]).reshape(-1)
        low = np.argsort(om, kind="stable")[:4 * nr]
        a = np.zeros((o * v, nr))
        a[low] = np.exp(-10.0 * (om[low] - om[low[0]]))[:, None] * np.cos(np.outer(1.0 + np.arange(4 * nr),
                                                                                    1.0 + np.arange(nr)))
        x = np.linalg.qr(a)[0]
        c, sc = q["c"], q["s"] @ q["c"]
        y = x.reshape(o, v, nr).transpose(2, 0, 1)
        m = ((c[:, :o] @ y) * sc[:, o:o + v].reshape(n, v)).sum(-1) + ((sc[:, :o] @ y) * c[:, o:o + v]).sum(-1)
        off = np.concatenate([[0], np.cumsum(q["opa"])])[:-1]
        out.append(dict(energies=om[low[:nr]] * 0.8, coefficients=x,
                        q_trans=np.ascontiguousarray(np.add.reduceat(0.5 * m, off, axis=1).T)))
    return out


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------

def _signs(c):
    """Signs that make the largest element of every column positive: an eigenvector's own is free."""
    return np.sign(c[np.abs(c).argmax(axis=0), np.arange(c.shape[1])])


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "product":
        return state["es"].compute_products(state["x"], PRECISION[case["precision"]])
    if kind == "tda":
        es = T.ExcitedStateSystem.from_ground_state(ctx, state["system"], state["ground"])
        p = es.run_tda(case["k"], 450, case["tol"], precision=PRECISION[case["precision"]])
        names = ("ci_coefficients", "q_trans", "tr_dipoles")
        # the plain form's subspace sums have no fixed order, so its vectors come with either sign
        g = _signs(p["ci_coefficients"]) if case["precision"] == "fp64" else None
        return dict({k: p[k] if g is None else p[k] * g for k in names}, ci_eigenvalues=p["ci_eigenvalues"],
                    oscillator_strengths=p["oscillator_strengths"])
    if kind == "gradient":
        return list(state["gradient"].both(0))
    if kind == "scc":
        got, _ = gscc.scc_batch(ctx, state["systems"], tol=1e-10, fp32_start=case["fp32_start"], full=case["full"])
        names = ("energy", "orbe", "dq") + (("p", "s", "h0", "h_coul_x") if case["full"] else ())
        out = {k: np.concatenate([np.reshape(getattr(g, k), -1) for g in got]) for k in names}
        out["orbs"] = np.concatenate([(g.orbs * _signs(g.orbs)).reshape(-1) for g in got])
        return out
    agg = state["aggregate"]
    if kind == "fmo":
        _, res = fmo.solve_batch(ctx, agg.instances, 150, 1e-4, PRECISION[case["precision"]])
        if case["precision"] == "fp64":
            for r in res:
                g = _signs(r["coefficients"])
                for k in ("coefficients", "tr_dip", "q_trans"):
                    r[k] = r[k] * g
        return {k: np.concatenate([np.reshape(r[k], -1) for r in res])
                for k in ("energies", "coefficients", "osc", "tr_dip", "q_trans")}
    r = fmo.exciton_states(ctx, agg, state["results"], agg.labels, case["n_le"], case["n_ct"],
                           n_roots=min(10, len(agg.monomers)), precision=PRECISION[case["precision"]], want_matrix=True)
    return {"energies": r["energies"], "vectors": r["vectors"] * _signs(r["vectors"]), "matrix": r["matrix"]}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------

def _dims(mol, size):
    """(atoms, orbitals, occupied, virtual) of a molecule."""
    if mol == "acene":
        return 6 * size + 6, 18 * size + 12, 9 * size + 6, 9 * size + 6
    if mol == "polyene":
        return 2 * size + 2, 5 * size + 2, (5 * size + 2) // 2, (5 * size + 2) - (5 * size + 2) // 2
    return 3 * size, 6 * size, 4 * size, 2 * size


def _product_flops(n, o, v, lc):
    return 8.0 * n * o * v + (16.0 * n * n * v if lc else 0.0)


def work(case):
    kind = case["kind"]
    if kind in ("product", "tda", "gradient"):
        a, n, o, v = _dims(case["mol"], case["size"])
        one = _product_flops(n, o, v, case["lc"])
        fixed = 8.0 * (2 * n * n + 2 * a * a)
        if kind == "product":     # X in, A.X out, C and S, gammas
            return {"bytes": fixed + 16.0 * o * v * case["k"], "flops": case["k"] * one}
        if kind == "tda":         # about six products a root; the roots out
            return {"bytes": fixed + 8.0 * case["k"] * (o * v + a), "flops": 6.0 * case["k"] * one}
        # P and the Fock matrix in too; about 15 Z-vector products and six n^3 contractions of densities
        return {"bytes": fixed + 16.0 * n * n, "flops": 15.0 * one + 96.0 * n ** 3}
    if kind == "scc":             # 12 iterations of seven n^3 products and a tridiagonal eigenproblem
        mean = (2 + case["size"]) / 2 if case["count"] > 1 else case["size"]
        n = _dims("acene", mean)[1] * (2 if case["dimers"] else 1)
        return {"bytes": 8.0 * case["count"] * n * n * (5 if case["full"] else 1), "flops": 12.0 * 17 * case["count"] * n ** 3}
    mono = case["nx"] * case["ny"] * case["nz"]
    a, n, o, v = _dims("acene", 3.5)
    pairs = 4.5 * mono
    if kind == "fmo":
        le, ct = _product_flops(n, o, v, case["lc"]), _product_flops(2 * n, o, v, case["lc"]) / 4
        return {"bytes": 8.0 * (mono * 2 * n * n + 2 * pairs * 6 * n * n),
                "flops": 6.0 * (mono * case["n_le"] * le + 2 * pairs * case["n_ct"] * ct)}
    real = 8.0 * mono             # one exchange element per pair of states on neighbouring monomers
    states = case["n_le"] * mono + 2 * pairs
    return {"bytes": 8.0 * (2 * (mono * a) ** 2 + real * 5 * n * n + states ** 2),
            "flops": 2.0 * real * (case["n_le"] + 4) ** 2 * a * 10 * 10 * 8}


# ----------------------------------------------------------------------------------------------
# the same results in 64 bits, by definition
# ----------------------------------------------------------------------------------------------

def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64)


def _charges(c, sc, off, p, q):
    """Mulliken transition charges [atoms, p, q] between two sets of orbitals."""
    out = torch.empty(len(off) - 1, p.stop - p.start, q.stop - q.start, dtype=torch.float64)
    for a in range(len(off) - 1):
        m = slice(int(off[a]), int(off[a + 1]))
        out[a] = 0.5 * (c[m, p].T @ sc[m, q] + sc[m, p].T @ c[m, q])
    return out


def _blocks(c, s, opa, o, v):
    off = np.concatenate([[0], np.cumsum(opa)])
    c = _t(c)
    sc = _t(s) @ c
    occ, virt = slice(0, o), slice(o, o + v)
    return (_charges(c, sc, off, occ, virt), _charges(c, sc, off, occ, occ), _charges(c, sc, off, virt, virt))


def _exact_products(st):
    sy, g, x = st["system"], st["ground"], _t(st["x"])
    n, o, v = sy.n_orbs, sy.n_occ, sy.n_virt
    c, s = _t(g.orbs), _t(g.s)
    sc = s @ c
    at = torch.as_tensor(np.asarray(sy.ao_atom))
    om = (_t(g.orbe)[o:][None, :] - _t(g.orbe)[:o, None])
    gam, glr = _t(g.gamma), (_t(g.gamma_lr)[at][:, at] if sy.lc else None)
    out = torch.empty_like(x)
    for j in range(x.shape[1]):
        xj = x[:, j].reshape(o, v)
        left = torch.cat([c[:, :o], sc[:, :o]]) @ xj
        right = torch.cat([c[:, o:], sc[:, o:]])
        m = left @ right.T
        d = 0.5 * (torch.diagonal(m[:n, n:]) + torch.diagonal(m[n:, :n]))
        z = (gam @ torch.zeros(sy.n_atoms, dtype=torch.float64).index_add_(0, at, d))[at]
        f = torch.zeros(2 * n, 2 * n, dtype=torch.float64)
        if glr is not None:
            f = -0.25 * (glr.repeat(2, 2) * m)
        i = torch.arange(n)
        f[i, n + i] += z
        f[n + i, i] += z
        out[:, j] = (om * xj + torch.cat([sc[:, :o], c[:, :o]]).T @ (f @ torch.cat([sc[:, o:], c[:, o:]]))).reshape(-1)
    return out.numpy()


def _dense_energies(c, s, opa, orbe, o, v, gam, glr, k):
    """k lowest eigenvalues of the dense TDA matrix."""
    qov, qoo, qvv = _blocks(c, s, opa, o, v)
    n = qov.shape[0]
    e = _t(orbe)
    a = torch.diag((e[o:o + v][None, :] - e[:o, None]).reshape(-1))
    q = qov.reshape(n, -1)
    a += 2.0 * q.T @ (_t(gam) @ q)
    if glr is not None:
        a -= (qoo.reshape(n, -1).T @ (_t(glr) @ qvv.reshape(n, -1))).reshape(o, o, v, v).permute(0, 2, 1, 3).reshape(o * v, o * v)
    return torch.linalg.eigvalsh(a)[:k].numpy()


def _spline(knots, coef, r):
    """Cubic B-spline values at r by de Boor's recurrence (zero beyond the grid), differentiable in r."""
    t, c = _t(knots), _t(coef)
    i = torch.clamp(torch.searchsorted(t, r.detach(), right=True) - 1, 3, len(t) - 5)
    d = [c[i - 3 + k] for k in range(4)]
    for lev in range(1, 4):
        for k in range(3, lev - 1, -1):
            lo, hi = t[i - 3 + k], t[i + 1 + k - lev]
            w = (r - lo) / (hi - lo)
            d[k] = (1.0 - w) * d[k - 1] + w * d[k]
    return torch.where(r.detach() <= t[-1], d[3], torch.zeros_like(r))


def _sk_matrix(sy, xyz_a, xyz_b, which, flip):
    """Off-diagonal S ('s') or H0 ('h') from the Slater-Koster splines; positions of centre 1 from
    xyz_a, of centre 2 from xyz_b.  Centre 1 is the lighter atom; of two like atoms the one with the
    lower index, or the higher one with `flip`."""
    ps, num = sy.params, np.asarray(sy.numbers)
    ii, jj = np.triu_indices(sy.n_atoms, 1)
    swap = (num[ii] > num[jj]) | ((num[ii] == num[jj]) & flip)
    a, b = np.where(swap, jj, ii), np.where(swap, ii, jj)
    out = torch.zeros(sy.n_orbs, sy.n_orbs, dtype=torch.float64)
    axis = {-1: 1, 0: 2, 1: 0}
    for za in np.unique(num):
        for zb in np.unique(num):
            sel = (num[a] == za) & (num[b] == zb)
            if za > zb or not sel.any():
                continue
            A, B = torch.as_tensor(a[sel]), torch.as_tensor(b[sel])
            d = xyz_b[B] - xyz_a[A]
            r = d.norm(dim=1)
            near = r.detach() <= float(ps.sk_knots[-1])
            A, B, d, r = A[near], B[near], d[near], r[near]
            u = d / r[:, None]
            coef = ps.sk_coef[(int(za), int(zb), which)]
            v = [_spline(ps.sk_knots, coef[k], r) if idx in ps.sk_present[(int(za), int(zb))] else torch.zeros_like(r)
                 for k, idx in enumerate(P.SK_INTEGRALS)]
            ea, eb = ps.element(int(za)), ps.element(int(zb))
            off = torch.as_tensor(np.asarray(sy.ao_offset))
            for p in range(ea.n_orbs):
                for q in range(eb.n_orbs):
                    l1, l2 = int(ea.l[p]), int(eb.l[q])
                    x1, x2 = u[:, axis[int(ea.m[p])]], u[:, axis[int(eb.m[q])]]
                    if l1 == 0 and l2 == 0:
                        e = v[0]
                    elif l1 == 0:
                        e = x2 * v[1]
                    elif l2 == 0:
                        e = x1 * v[2]
                    else:
                        e = x1 * x2 * (v[4] - v[3]) + (v[3] if int(ea.m[p]) == int(eb.m[q]) else 0.0)
                    out = out.index_put((off[A] + p, off[B] + q), e)
    return out + out.T


def _gamma(sy, xyz, r_lr):
    sig = 1.0 / (_t(sy.hubbard) * math.sqrt(math.pi))
    cc = 1.0 / torch.sqrt(2.0 * (sig[:, None] ** 2 + sig[None, :] ** 2 + 0.5 * r_lr ** 2))
    eye = torch.eye(sy.n_atoms, dtype=torch.float64)
    r = torch.sqrt(((xyz[:, None, :] - xyz[None, :, :]) ** 2).sum(-1) + eye)
    return torch.special.erf(cc * r) / r * (1.0 - eye) + torch.diag(1.0 / torch.sqrt(math.pi * (sig ** 2 + 0.25 * r_lr ** 2)))


def _repulsion(sy, xyz):
    num = np.asarray(sy.numbers)
    ii, jj = np.triu_indices(sy.n_atoms, 1)
    e = torch.zeros((), dtype=torch.float64)
    r = (xyz[ii] - xyz[jj]).norm(dim=1)
    for za in np.unique(num):
        for zb in np.unique(num):
            sel = (num[ii] == za) & (num[jj] == zb) | (num[ii] == zb) & (num[jj] == za)
            if za > zb or not sel.any():
                continue
            t, c, dmax = sy.params.rep[(int(za), int(zb))]
            q = r[torch.as_tensor(sel)]
            q = q[q.detach() <= dmax]
            if len(q):
                e = e + _spline(t, np.pad(np.asarray(c), (0, max(0, len(t) - len(c)))), q).sum()
    return e


def _exact_gradient(st):
    """S0 gradient and the gradient of the excitation energy, at the given state."""
    sy, g, lc = st["system"], st["ground"], st["case"]["lc"]
    n, o, v = sy.n_orbs, sy.n_occ, sy.n_virt
    qov, qoo, qvv = _blocks(g.orbs, g.s, sy.orbs_per_atom, o, v)
    qvo = qov.transpose(1, 2)
    gam, glr = _t(g.gamma), _t(g.gamma_lr)
    e = _t(g.orbe)
    eo, ev = e[:o], e[o:]
    omega = ev[None, :] - eo[:, None]
    es, x = float(st["e"][0]), _t(st["x"]).reshape(o, v)

    def coul(q_out, q_in, m):
        return torch.tensordot(gam @ torch.tensordot(q_in, m, dims=([1, 2], [0, 1])), q_out, dims=([0], [0]))

    def exch(q1, q2, m):
        t = q1 @ m.T
        t = (glr @ t.reshape(t.shape[0], -1)).reshape(t.shape)
        return torch.einsum("ayc,axc->yx", q2, t)

    def h(q_out, q_in, q1, q2, m):
        return 4.0 * coul(q_out, q_in, m) - (2.0 * exch(q1, q2, m) if lc else 0.0)

    def av(m):     # the operator of the Z-vector equation
        if not lc:
            return omega * m + 4.0 * coul(qov, qov, m)
        return omega * m + 2.0 * coul(qov, qov, m) - exch(qvv, qoo, m)

    tab, tij = x.T @ x, x @ x.T
    g_ij = h(qoo, qvv, qov, qov, tab) - h(qoo, qoo, qoo, qoo, tij)
    q_ij = 2.0 * es * tij - 2.0 * (x * ev[None, :]) @ x.T + g_ij
    q_ab = 2.0 * es * tab + 2.0 * (eo[:, None] * x).T @ x
    q_ia = x @ h(qvv, qov, qvv, qvo, x).T + h(qov, qvv, qvv, qov, tab) - h(qov, qoo, qvo, qoo, tij)
    q_ai = x.T @ h(qoo, qov, qov, qoo, x)
    r = q_ai.T - q_ia
    z = r / omega
    res = r - av(z)
    p = res.clone()
    for _ in range(2000):
        ap = av(p)
        rr = (res * res).sum()
        if rr <= 1e-26:
            break
        al = rr / (p * ap).sum()
        z, res = z + al * p, res - al * ap
        p = res + (res * res).sum() / rr * p
    w = torch.zeros(n, n, dtype=torch.float64)
    w[:o, :o] = q_ij + h(qoo, qov, qov, qoo, z)
    w[:o, o:] = q_ai.T + eo[:, None] * z
    w[o:, o:] = q_ab
    w = torch.triu(w)
    w[torch.arange(n), torch.arange(n)] *= 0.5
    c = _t(g.orbs)
    co, cv = c[:, :o], c[:, o:]
    m_ao = cv @ tab @ cv.T - co @ tij @ co.T + co @ z @ cv.T
    w_ao, x_ao = c @ w @ c.T, co @ x @ cv.T
    pd, fock = _t(g.p), _t(g.h_coul_x)
    dp = pd - _t(g.p0)
    at = torch.as_tensor(np.asarray(sy.ao_atom))
    dq = _t(g.dq)

    xyz = _t(sy.xyz).clone().requires_grad_(True)
    still = xyz.detach()
    s = _sk_matrix(sy, xyz, xyz, "s", False) + torch.eye(n, dtype=torch.float64)
    g0, gl = _gamma(sy, xyz, 0.0), (_gamma(sy, xyz, sy.r_lr) if lc else None)
    # the reference takes the moving atom as centre 1 in dH0 of two like atoms: each end on its own
    num = torch.as_tensor(np.asarray(sy.numbers))[at]
    like = (num[:, None] == num[None, :]).to(torch.float64)
    h0 = (1.0 - like) * _sk_matrix(sy, xyz, xyz, "h", False) \
        + like * (_sk_matrix(sy, xyz, still, "h", False) + _sk_matrix(sy, xyz, still, "h", True))

    def f_c(m):    # Coulomb Fock matrix of a density
        sv = (s * (m + m.T)).sum(0)
        t = g0[at][:, at] @ sv
        return 0.25 * s * (t[:, None] + t[None, :])

    def f_x(m):    # long-range exchange Fock matrix of a density
        k = gl[at][:, at]
        sm = s @ m
        return 0.25 * (k * (s @ sm.T) + ((s @ m.T) * k) @ s + s @ (sm * k).T + s @ (s @ (k * m)).T)

    pot = (gam @ dq)[at]
    e0 = (h0 * pd).sum() + (s * (0.5 * (pot[:, None] + pot[None, :]) * pd - 0.5 * pd @ fock @ pd)).sum() \
        + 0.5 * dq @ g0 @ dq + _repulsion(sy, xyz)
    e1 = ((h0 + f_c(dp)) * m_ao).sum() - (s * w_ao).sum() + 2.0 * (f_c(x_ao) * x_ao).sum()
    if lc:
        fd = f_x(dp)
        e0 = e0 - 0.25 * (fd * dp).sum()
        e1 = e1 - 0.5 * (fd * m_ao).sum() - (f_x(x_ao.T) * x_ao).sum()
    return [torch.autograd.grad(q, xyz, retain_graph=True)[0].reshape(-1).numpy() for q in (e0, e1)]


def _exact_scc(st):
    out = {k: [] for k in ("energy", "orbe", "orbs", "dq") + (("p", "s", "h0", "h_coul_x") if st["case"]["full"] else ())}
    for sy in st["systems"]:
        xyz = _t(sy.xyz)
        s = (_sk_matrix(sy, xyz, xyz, "s", False) + torch.eye(sy.n_orbs, dtype=torch.float64)).numpy()
        h0 = (_sk_matrix(sy, xyz, xyz, "h", False) + torch.diag(_t(sy.ao_energy))).numpy()
        gam = _gamma(sy, xyz, 0.0).numpy()
        glr = _gamma(sy, xyz, sy.r_lr).numpy() if sy.lc else None
        f, p, e, _, dq, _ = _scf(sy, s, h0, gam, glr, 1e-11, 100)
        en = float((p * h0).sum() + 0.5 * dq @ gam @ dq + float(_repulsion(sy, xyz)))
        if glr is not None:
            k, d = glr[np.ix_(sy.ao_atom, sy.ao_atom)], p - np.diag(sy.ao_occ.astype(np.float64))
            en -= 0.125 * float(((s @ d @ s) * d * k).sum() + ((s @ d) * (d @ s) * k).sum())
        for name, val in (("energy", en), ("orbe", e), ("dq", dq), ("p", p), ("s", s), ("h0", h0), ("h_coul_x", f)):
            if name in out:
                out[name].append(np.reshape(val, -1))
    out["orbs"] = None     # an orbital's sign is free
    return {k: None if a is None else np.concatenate(a) for k, a in out.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "exciton":
        return None        # the whole exciton Hamiltonian element by element takes minutes
    if kind == "scc" and case["count"] * (2 if case["dimers"] else 1) * case["size"] > 200:
        return None
    if kind == "tda" and _dims(case["mol"], case["size"])[2] * _dims(case["mol"], case["size"])[3] > 8200:
        return None        # a dense matrix of this size takes minutes to diagonalise
    if kind == "fmo" and case["nx"] * case["ny"] * case["nz"] > 3:
        return None
    st = _Inputs(case, seed)
    if kind == "product":
        return _exact_products(st)
    if kind == "gradient":
        return _exact_gradient(st)
    if kind == "scc":
        return _exact_scc(st)
    none = dict.fromkeys(("ci_coefficients", "oscillator_strengths", "q_trans", "tr_dipoles") if kind == "tda"
                         else ("coefficients", "osc", "tr_dip", "q_trans"))
    if kind == "tda":      # vectors are converged to the tolerance only, and their signs are free
        sy, g = st["system"], st["ground"]
        return dict(none, ci_eigenvalues=_dense_energies(g.orbs, g.s, sy.orbs_per_atom, g.orbe, sy.n_occ, sy.n_virt,
                                                         g.gamma, g.gamma_lr if sy.lc else None, case["k"]))
    return dict(none, energies=np.concatenate(
        [_dense_energies(q["c"], q["s"], q["opa"], q["orbe"], q["n_occ"], q["n_virt"], q["gamma"], q["gamma_lr"],
                         q["n_roots"]) for q in st["aggregate"].instances]))
