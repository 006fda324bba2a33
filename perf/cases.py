"""The work that is timed: what a program asks of the library through
``myqc_gb300.session``, from one small molecule to the largest cluster and batch.

A case is a kind of call and its size; `_KINDS` below says for each kind what
it stands for.  Molecules are the repository's own: the standard small ones
with perturbed coordinates, and seeded water clusters at liquid density.  The
densities and orbitals that stand-alone Fock builds and transforms take are
extended-Hueckel ones, which have the structure of an SCF's.

`exact` gives the results in 64 bits from a separate evaluation in torch:
Hermite Gaussians, the Boys function by its series, dense matrices.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from myqc_gb300 import (FOCK_FP64, MODE_REFERENCE, MODE_TIGHT, PREC_FP64, PREC_SPLIT_BF16X3, STORE_FULL,
                        STORE_QUARTETS, formats, guess, molecules)
from myqc_gb300.session import Context, run_job

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BASIS_TEXT = open(os.path.join(ROOT, "myqc_gb300", "data", "sto3g.mybasis")).read()
MODEL = os.path.join(ROOT, "myqc_gb300", "data", "guess_mlp.npz")
SCHWARZ = 1e-12
SMALL = [k for k in molecules.STANDARD_GEOMETRIES if k != "H2"]
CATIONS = ["H2O", "NH3"]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's own smallest run: CO2, its Boys table, plain Roothaan iterations, MP2
        {"name": "job_co2_reference", "kind": "job", "molecule": "CO2", "mode": "reference", "uhf": False, "diis": 0},
        # an open-shell molecule: UHF with DIIS, UHF MP2
        {"name": "job_h2o_cation_uhf", "kind": "job", "molecule": "H2O", "mode": "tight", "uhf": True, "diis": 8},
        # a cluster of eight waters in the default settings: n^4 array, eigensolver, FP64 transform
        {"name": "job_h2o8", "kind": "job", "molecule": "(H2O)8", "mode": "tight", "uhf": False, "diis": 8},
        # one UHF Fock build of an SCF that keeps the n^4 array
        {"name": "fock_uhf_h2o16", "kind": "fock_uhf", "waters": 16},
        # one RHF Fock build of an SCF that keeps the screened quartets
        {"name": "fock_quartets_h2o32", "kind": "fock_quartets", "waters": 32},
        # one iteration's Fock build of a direct SCF, the largest cluster
        {"name": "fock_direct_h2o64", "kind": "fock_direct", "waters": 64},
        # the whole solve: learned guess, screened quartets, purified SCF, split transform, MP2
        {"name": "solve_h2o32", "kind": "solve", "waters": 32},
        # a batch of small molecules set up and solved together
        {"name": "batch_1024", "kind": "batch", "molecules": 1024},
        # transform and MP2 in FP64 (the default precision), from the n^4 array
        {"name": "mp2_fp64_h2o16", "kind": "mp2_fp64", "waters": 16},
        # transform on the tensor cores and MP2, from the screened quartets
        {"name": "mp2_split_h2o32", "kind": "mp2_split", "waters": 32},
        # training the learned guess: Adam minibatches of pair samples, as train_guess runs them
        {"name": "train_262144", "kind": "train", "samples": 262144, "batch": 4096},
        # predicting the densities of many clusters for a batched SCF
        {"name": "predict_256", "kind": "predict", "clusters": 256},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["job", "fock_uhf", "fock_quartets", "fock_direct", "solve", "batch", "mp2_fp64", "mp2_split",
                       "train", "predict"])
    if kind == "job":
        uhf = rng.random() < 0.3
        name = rng.choice(CATIONS if uhf else SMALL + [f"(H2O){k}" for k in range(2, 9)])
        # plain Roothaan iterations need not converge: DIIS, but for the one listed run
        return {"kind": kind, "molecule": name, "mode": rng.choice(["tight", "tight", "reference"]), "uhf": uhf,
                "diis": rng.choice([6, 8])}
    if kind == "batch":
        return {"kind": kind, "molecules": _log_int(rng, 24, 1024)}
    if kind == "train":
        return {"kind": kind, "samples": _log_int(rng, 8192, 262144), "batch": rng.choice([1024, 2048, 4096])}
    if kind == "predict":
        return {"kind": kind, "clusters": _log_int(rng, 1, 256)}
    lo, hi = {"fock_uhf": (3, 16), "fock_quartets": (4, 32), "fock_direct": (8, 64), "solve": (4, 32),
              "mp2_fp64": (3, 16), "mp2_split": (8, 32)}[kind]
    return {"kind": kind, "waters": _log_int(rng, lo, hi)}


# ------------------------------------------------------------------ inputs
def _box(waters):
    return (27.0 * waters) ** (1.0 / 3.0)


def _cluster(waters, seed):
    return molecules.water_cluster_system(waters, _box(waters), seed)


def _molecule(case, seed):
    sym, xyz = molecules.standard_geometry(case["molecule"])
    xyz = xyz + np.random.default_rng(seed).normal(0.0, 0.02, size=xyz.shape)
    return formats.system_from_geometry(sym, xyz, charge=1 if case["uhf"] else 0, multiplicity=2 if case["uhf"] else 1,
                                        uhf=case["uhf"])


def _clusters(case, seed):
    sizes = np.random.default_rng(0).integers(2, 17, size=case["clusters"])
    return [_cluster(int(k), int(g)) for k, g in zip(sizes, np.random.default_rng(seed).integers(1 << 30, size=len(sizes)))]


def _batch(case, seed):
    """The batch workload's mixture of molecules, coordinates perturbed from the seed."""
    rng = np.random.default_rng(seed)
    systems = []
    for kind in molecules.batch_workload(case["molecules"], 0)[0]:
        sym, xyz = molecules.standard_geometry(kind)
        systems.append(formats.system_from_geometry(sym, xyz + rng.normal(0.0, 0.05, size=xyz.shape), calc_mp2=False))
    return systems


def _basis(sysm):
    return formats.parse_mybasis_text(BASIS_TEXT, sysm.atoms)


def _hueckel(sysm):
    """Orbitals (ascending) and energies of an extended-Hueckel matrix."""
    S = _overlap(_pairs(_shells(sysm), "cpu"), "cpu").numpy()
    h = np.concatenate([{1: [-0.5], 8: [-20.7, -1.35, -0.57, -0.57, -0.57]}[int(z)] for z in sysm.atoms])
    F = 1.75 * S * (h[:, None] + h[None, :]) / 2
    np.fill_diagonal(F, h)
    s, U = np.linalg.eigh(S)
    X = U / np.sqrt(s) @ U.T
    e, V = np.linalg.eigh(X @ F @ X)
    C = X @ V
    C *= np.sign(C[np.abs(C).argmax(0), np.arange(len(e))])
    return np.asfortranarray(C), e


def _density(C, nocc, factor):
    return np.asfortranarray(factor * C[:, :nocc] @ C[:, :nocc].T)


def _training_set(case, seed):
    rng = np.random.default_rng(seed)
    n = case["samples"]
    X = rng.standard_normal((n, guess.NFEAT), dtype=np.float32)
    A = rng.standard_normal((guess.NFEAT, guess.NOUT)).astype(np.float32) / 8
    T = np.tanh(X @ A) + 0.1 * rng.standard_normal((n, guess.NOUT), dtype=np.float32)
    W = (rng.random((n, guess.NOUT), dtype=np.float32) < 0.6).astype(np.float32)
    dims = (guess.NFEAT, 256, 256, guess.NOUT)
    parts = []
    for k in range(3):
        parts += [(rng.standard_normal(dims[k + 1] * dims[k]) / math.sqrt(dims[k])), np.zeros(dims[k + 1])]
    return X, T.astype(np.float32), W, np.concatenate(parts).astype(np.float32), dims


_ctx = None


def _context():
    """The one context of a program that goes from molecule to molecule."""
    global _ctx
    if _ctx is None:
        _ctx = Context()
        _ctx.model = guess.LearnedGuess(_ctx, MODEL)
        _ctx.basis_library(BASIS_TEXT)
    return _ctx


def _options(ctx, storage, schwarz):
    ctx.set_eri_storage(storage)
    ctx.set_fock_precision(FOCK_FP64)
    ctx.set_fock_screened_increments(1e-12 if storage == STORE_QUARTETS else 0.0)
    ctx.set_schwarz(schwarz)


def _resident(sysm, storage, schwarz, integrals):
    """A context of its own for a molecule whose integrals stay on the GPU."""
    ctx = Context()
    _options(ctx, storage, schwarz)
    ctx.set_system(sysm, _basis(sysm), None, MODE_TIGHT)
    if integrals:
        ctx.eri_store()
    return ctx


# ------------------------------------------------------------------ one pass of each kind
def prepare(case, seed):
    kind = case["kind"]
    if kind == "job":
        sysm = _molecule(case, seed)
        ftab = formats.read_ftab(os.path.join(ROOT, "tests", "golden", "Ftab")) if case["mode"] == "reference" else None
        return {"case": case, "ctx": _context(), "sys": sysm, "basis": _basis(sysm), "ftab": ftab}
    if kind == "solve":
        sysm = _cluster(case["waters"], seed)
        return {"case": case, "ctx": _context(), "sys": sysm, "basis": _basis(sysm)}
    if kind == "batch":
        return {"case": case, "ctx": _context(), "systems": _batch(case, seed)}
    if kind == "predict":
        return {"case": case, "ctx": _context(), "systems": _clusters(case, seed)}
    if kind == "train":
        X, T, W, p, dims = _training_set(case, seed)
        ctx = Context()
        ctx.mlp_init(dims[0], dims[1], dims[3])
        ctx.mlp_set_data(X, T, W)
        return {"case": case, "ctx": ctx, "params": p}
    sysm = _cluster(case["waters"], seed)
    C, e = _hueckel(sysm)
    n = sysm.nelcA
    if kind == "fock_uhf":
        ctx = _resident(sysm, STORE_FULL, 0.0, True)
        return {"case": case, "ctx": ctx, "D": (_density(C, n, 1.0), _density(C, n - 1, 1.0))}
    if kind == "mp2_fp64":
        return {"case": case, "ctx": _resident(sysm, STORE_FULL, 0.0, True), "C": C, "eps": e, "nocc": n}
    ctx = _resident(sysm, STORE_QUARTETS, SCHWARZ, kind != "fock_direct")
    return {"case": case, "ctx": ctx, "D": _density(C, n, 2.0), "C": C, "eps": e, "nocc": n}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "job":
        _options(ctx, STORE_FULL, 0.0)
        out = run_job(state["sys"], state["basis"], state["ftab"],
                      MODE_REFERENCE if case["mode"] == "reference" else MODE_TIGHT, conv=1e-10, diis=case["diis"],
                      ctx=ctx, mp2=True)
        res = out["scf"]
        return {"S": out["S"], "H": out["H"], "E": np.float64(res.energy), "eps": res.eig, "D": res.D,
                "E_MP2": np.float64(out["mp2"]["E_MP2"])}
    if kind == "solve":
        sysm = state["sys"]
        _options(ctx, STORE_QUARTETS, SCHWARZ)
        ctx.set_system(sysm, state["basis"], None, MODE_TIGHT)
        S, H = ctx.int1e()
        ctx.eri_store()
        D0 = ctx.model.guess(sysm, S)
        res = ctx.scf(S, H, sysm.nelcA, sysm.nelcB, D_guess=D0, conv=1e-10, conv_rms=True, diis=8, max_iter=200,
                      purify=True)
        mp2 = ctx.mp2_rhf(res.eig, sysm.nelcA, PREC_SPLIT_BF16X3, C=res.C)
        return {"S": S, "H": H, "E": np.float64(res.energy), "eps": res.eig, "D": res.D, "E_MP2": mp2["E_MP2"]}
    if kind == "batch":
        ctx.batch_clear()
        for sysm in state["systems"]:
            ctx.batch_add_atoms(sysm)
        out = ctx.batch_scf(conv=1e-10, conv_rms=True, diis=8, max_iter=100, graph=True)
        return {"E": out["energy"], "D": np.concatenate([D.ravel() for D in out["D"]]),
                "eps": np.concatenate(out["eps"])}
    if kind == "predict":
        return np.concatenate([D.ravel() for D in ctx.model.predict_many(state["systems"])])
    if kind == "train":
        ctx.mlp_set_params(state["params"])
        loss = ctx.mlp_train_epoch(case["batch"], 2e-3, 1)
        return {"loss": loss, "params": ctx.mlp_get_params()}
    if kind == "fock_uhf":
        return ctx.fock(*state["D"])
    if kind in ("fock_quartets", "fock_direct"):
        return ctx.fock(state["D"], direct=kind == "fock_direct")
    r = ctx.mp2_rhf(state["eps"], state["nocc"], PREC_FP64 if kind == "mp2_fp64" else PREC_SPLIT_BF16X3, C=state["C"])
    return {k: np.float64(v) for k, v in r.items()}


def work(case):
    """Bytes: integrals, matrices and results, each once.  Operations: the
    unique integrals' (30 for each of a contracted integral's primitive
    quartets, nine in ten of which are screened in a cluster), six
    multiply-adds per integral and Fock build, the transform's products, the
    network's products."""
    kind = case["kind"]
    if kind == "train":
        macs = 64 * 256 + 256 * 256 + 256 * 25
        return {"bytes": case["samples"] * (64 + 50) * 4.0, "flops": 6.0 * macs * case["samples"]}
    if kind == "predict":
        pairs = case["clusters"] * 27 * 20  # atom pairs within 8 A of an average cluster
        return {"bytes": case["clusters"] * 63 * 63 * 8.0, "flops": 2.0 * (64 * 256 + 256 * 256 + 256 * 25) * pairs}
    if kind == "batch":
        n4 = case["molecules"] * float(np.mean([_order(molecules.standard_geometry(k)[0]) ** 4
                                                for k in molecules.BATCH_KINDS]))
        return {"bytes": n4, "flops": n4 / 8 * (81 * 30 + 14 * 12)}
    if kind == "job":
        n, occ = _order(molecules.standard_geometry(case["molecule"])[0]), 0.6
        return {"bytes": float(n ** 4), "flops": n ** 4 / 8 * (81 * 30 + 15 * 12) + 2 * n ** 5 * (1 - occ)}
    n = 7 * case["waters"]
    o, v = 5 * case["waters"], 2 * case["waters"]
    transform = 2.0 * (n ** 4 * v / 4 + n ** 3 * o * v / 2 + n ** 2 * o * v * v + n * o * o * v * v)
    unique = min(n ** 4 / 8.0, 165.0 * n ** 2.26)  # screened at 1e-12, as counted at 16 to 64 waters
    if kind == "fock_uhf":
        return {"bytes": float(n ** 4), "flops": n ** 4 / 8 * 20.0}
    if kind == "fock_quartets":
        return {"bytes": 8.0 * unique, "flops": 12 * unique}
    if kind == "fock_direct":
        return {"bytes": 32.0 * n * n, "flops": (81 * 3 + 12) * unique}
    if kind == "solve":
        return {"bytes": 8.0 * unique + 8.0 * (o * v) ** 2, "flops": (81 * 3 + 13 * 12) * unique + transform}
    return {"bytes": float(n ** 4 if kind == "mp2_fp64" else 8 * unique) + 8.0 * (o * v) ** 2, "flops": transform}


def _order(symbols):
    return sum(1 if s in ("H", "He") else 5 for s in symbols)


# ------------------------------------------------------------------ the results in 64 bits
def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("batch", "predict", "solve") or kind == "fock_direct" and case["waters"] > 32:
        return None
    if kind == "train":
        return _exact_training(case, seed, dev)
    if kind == "job":
        return _exact_job(_molecule(case, seed), case["uhf"], dev)
    sysm = _cluster(case["waters"], seed)
    C, e = _hueckel(sysm)
    n = sysm.nelcA
    XX = _integrals(_pairs(_shells(sysm), dev), dev)
    if kind == "fock_uhf":
        D = [torch.tensor(_density(C, k, 1.0), device=dev) for k in (n, n - 1)]
        J = _coulomb(XX, D[0] + D[1])
        return tuple(J - _exchange(XX, d) for d in D)
    if kind in ("fock_quartets", "fock_direct"):
        D = torch.tensor(_density(C, n, 2.0), device=dev)
        return _coulomb(XX, D) - 0.5 * _exchange(XX, D)
    C, e = torch.tensor(C, device=dev), torch.tensor(e, device=dev)
    same, both = _pair_energies(XX, C[:, :n], C[:, n:], C[:, :n], C[:, n:], e[:n], e[n:], e[:n], e[n:])
    return {"E_AA": np.float64(same), "E_AB": np.float64(both), "E_MP2": np.float64(2 * same + both)}


def _shells(sysm):
    """(centre, exponents, s coefficients, p coefficients or None, first AO) with normalised primitives."""
    rows = [ln.split() for ln in BASIS_TEXT.split("\n")]
    shells, ao = [], 0
    for Z, xyz in zip(sysm.atoms, sysm.xyz):
        at = next(i for i, r in enumerate(rows) if r and r[0] == formats.ELEMENTS[int(Z) - 1])
        blocks = []
        for b in range(int(rows[at + 1][0])):
            blocks.append(np.array([[float(v) for v in r[:2]] for r in rows[at + 3 + 4 * b: at + 6 + 4 * b]]))
        for b, blk in enumerate(blocks[:2]):
            a = blk[:, 1]
            cs = blk[:, 0] * (2 * a / math.pi) ** 0.75
            cp = blocks[2][:, 0] * (128 * a ** 5 / math.pi ** 3) ** 0.25 if b == 1 else None
            shells.append((np.asarray(xyz), a, cs, cp, ao))
            ao += 1 if cp is None else 4
    return shells


_HERMITE = {0: [(0, 0, 0)], 1: [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]}
_HERMITE[2] = [(t, u, v) for t in range(3) for u in range(3 - t) for v in range(3 - t - u)]


def _pairs(shells, dev):
    """Shell pairs by class (s,s), (sp,s), (sp,sp): exponent sums, centres and
    Hermite expansions of the primitive pairs, and the AOs of their functions."""
    out = []
    for cls in range(3):
        want = {0: (False, False), 1: (True, False), 2: (True, True)}[cls]
        idx = [(A, B) for A in range(len(shells)) for B in range(len(shells))
               if ((shells[A][3] is not None), (shells[B][3] is not None)) == want and (cls == 1 or B <= A)]
        if not idx:
            continue
        fa, fb = (4 if want[0] else 1), (4 if want[1] else 1)
        RA = torch.tensor(np.array([shells[A][0] for A, _ in idx]), device=dev)
        RB = torch.tensor(np.array([shells[B][0] for _, B in idx]), device=dev)
        a = torch.tensor(np.array([shells[A][1] for A, _ in idx]), device=dev)[:, :, None].expand(-1, -1, 3)
        b = torch.tensor(np.array([shells[B][1] for _, B in idx]), device=dev)[:, None, :].expand(-1, 3, -1)
        coef = [[torch.tensor(np.array([shells[s][2 + k] if k == 0 or shells[s][3] is not None else shells[s][2]
                                        for s in side]), device=dev) for k in range(2)]
                for side in ([A for A, _ in idx], [B for _, B in idx])]
        a, b = a.reshape(-1, 9), b.reshape(-1, 9)
        p = a + b
        P = (a[..., None] * RA[:, None] + b[..., None] * RB[:, None]) / p[..., None]
        K = torch.exp(-a * b / p * ((RA - RB) ** 2).sum(-1)[:, None])
        PA, PB, h = P - RA[:, None], P - RB[:, None], 0.5 / p
        one, zero = torch.ones_like(p), torch.zeros_like(p)

        def axis(la, lb, x):  # Hermite coefficients of x_A^la x_B^lb
            if la + lb == 0:
                return [one, zero, zero]
            if la + lb == 1:
                return [(PA if la else PB)[..., x], h, zero]
            return [PA[..., x] * PB[..., x] + h, (PA[..., x] + PB[..., x]) * h, h * h]

        herm = _HERMITE[cls]
        E = torch.zeros(len(idx), 9, fa * fb, len(herm), dtype=torch.float64, device=dev)
        for i in range(fa):
            for j in range(fb):
                c = (coef[0][min(i, 1)][:, :, None] * coef[1][min(j, 1)][:, None, :]).reshape(-1, 9) * K
                e = [axis(int(i == x + 1), int(j == x + 1), x) for x in range(3)]
                for q, (t, u, v) in enumerate(herm):
                    E[:, :, i * fb + j, q] = c * e[0][t] * e[1][u] * e[2][v]
        ao = np.array([[(shells[A][4] + i, shells[B][4] + j) for i in range(fa) for j in range(fb)] for A, B in idx])
        out.append({"cls": cls, "a": a, "b": b, "p": p, "P": P, "E": E, "RA": RA, "RB": RB, "K": K, "coef": coef,
                    "fa": fa, "fb": fb, "ao": torch.tensor(ao, device=dev)})
    return out


def _norb(pairs):
    return int(max(int(c["ao"].max()) for c in pairs)) + 1


def _scatter(M, c, vals):
    i, j = c["ao"][..., 0], c["ao"][..., 1]
    M[i, j] = vals
    M[j, i] = vals


def _overlap(pairs, dev):
    S = torch.zeros(_norb(pairs), _norb(pairs), dtype=torch.float64, device=dev)
    for c in pairs:
        _scatter(S, c, ((math.pi / c["p"]) ** 1.5).unsqueeze(-1).mul(c["E"][..., 0]).sum(1))
    return S


def _core(pairs, sysm, dev):
    """Kinetic energy plus nuclear attraction."""
    H = torch.zeros(_norb(pairs), _norb(pairs), dtype=torch.float64, device=dev)
    for c in pairs:
        p, h = c["p"], 0.5 / c["p"]
        PA, PB = c["P"] - c["RA"][:, None], c["P"] - c["RB"][:, None]
        one = {}

        def s1(x, i, j):  # one axis' overlap of x_A^i and x_B^j (without the common prefactor)
            if i < 0 or j < 0:
                return torch.zeros_like(p)
            if (x, i, j) not in one:
                if i + j == 0:
                    one[x, i, j] = torch.ones_like(p)
                elif i > 0:
                    one[x, i, j] = PA[..., x] * s1(x, i - 1, j) + h * ((i - 1) * s1(x, i - 2, j) + j * s1(x, i - 1, j - 1))
                else:
                    one[x, i, j] = PB[..., x] * s1(x, i, j - 1) + h * (j - 1) * s1(x, i, j - 2)
            return one[x, i, j]

        def t1(x, i, j):
            b = c["b"]
            return (-2 * b * b * s1(x, i, j + 2) + b * (2 * j + 1) * s1(x, i, j)
                    - 0.5 * j * (j - 1) * s1(x, i, j - 2))

        vals = torch.zeros(len(p), c["fa"] * c["fb"], dtype=torch.float64, device=dev)
        for i in range(c["fa"]):
            for j in range(c["fb"]):
                l = [(int(i == x + 1), int(j == x + 1)) for x in range(3)]
                s = [s1(x, *l[x]) for x in range(3)]
                t = [t1(x, *l[x]) for x in range(3)]
                cc = (c["coef"][0][min(i, 1)][:, :, None] * c["coef"][1][min(j, 1)][:, None, :]).reshape(-1, 9)
                f = cc * c["K"] * (math.pi / p) ** 1.5
                vals[:, i * c["fb"] + j] = (f * (t[0] * s[1] * s[2] + s[0] * t[1] * s[2] + s[0] * s[1] * t[2])).sum(1)
        for Z, xyz in zip(sysm.atoms, sysm.xyz):
            R = _hermite_coulomb(c["cls"], p, c["P"] - torch.tensor(xyz, device=dev))
            for q, tuv in enumerate(_HERMITE[c["cls"]]):
                vals -= ((float(Z) * 2 * math.pi / p * R[tuv]).unsqueeze(-1) * c["E"][..., q]).sum(1)
        _scatter(H, c, vals)
    return H


def _boys(L, T):
    """F_0 .. F_L: the series of F_L and downward recursion; for T > 35 F_0 by erf and upward recursion."""
    small = T < 35.0
    Ts, e = torch.where(small, T, torch.zeros_like(T)), torch.exp(-T)
    term = torch.full_like(T, 1.0 / (2 * L + 1))
    total = term.clone()
    top = float(Ts.max()) if T.numel() else 0.0
    for i in range(1, int(20 + 2 * top + 6 * math.sqrt(top + 1))):
        term = term * (2 * Ts / (2 * L + 2 * i + 1))
        total += term
    F = [None] * (L + 1)
    F[L] = torch.exp(-Ts) * total
    for m in range(L - 1, -1, -1):
        F[m] = (2 * Ts * F[m + 1] + torch.exp(-Ts)) / (2 * m + 1)
    Tl = torch.where(small, torch.full_like(T, 36.0), T)
    up = 0.5 * torch.sqrt(math.pi / Tl) * torch.special.erf(torch.sqrt(Tl))
    for m in range(L + 1):
        F[m] = torch.where(small, F[m], up)
        up = ((2 * m + 1) * up - e) / (2 * Tl)
    return F


def _hermite_coulomb(L, alpha, V):
    """R_tuv, t + u + v <= L, of the vectors V."""
    F = _boys(L, alpha * (V * V).sum(-1))
    R = {(0, 0, 0, m): (-2 * alpha) ** m * F[m] for m in range(L + 1)}
    for n in range(1, L + 1):
        for t in range(n + 1):
            for u in range(n + 1 - t):
                v = n - t - u
                for m in range(L + 1 - n):
                    k = [t, u, v]
                    x = next(i for i in range(3) if k[i])
                    k[x] -= 1
                    r = V[..., x] * R[(*k, m + 1)]
                    if k[x] > 0:
                        w = list(k)
                        w[x] -= 1
                        r = r + k[x] * R[(*w, m + 1)]
                    R[t, u, v, m] = r
    return {key[:3]: val for key, val in R.items() if key[3] == 0}


def _integrals(pairs, dev):
    """The n^4 array (ij|kl)."""
    n = _norb(pairs)
    XX = torch.zeros(n * n, n * n, dtype=torch.float64, device=dev)
    for bi, bra in enumerate(pairs):
        for ket in pairs[: bi + 1]:
            hb, hk = _HERMITE[bra["cls"]], _HERMITE[ket["cls"]]
            kl = ket["ao"][..., 0] * n + ket["ao"][..., 1]
            lk = ket["ao"][..., 1] * n + ket["ao"][..., 0]
            step = max(1, 30_000_000 // (len(ket["p"]) * len(hb) * len(hk)))
            for r0 in range(0, len(bra["p"]), step):
                sl = slice(r0, r0 + step)
                vals = 0.0
                for i in range(9):
                    for j in range(9):
                        p, q = bra["p"][sl, i][:, None], ket["p"][:, j][None, :]
                        V = bra["P"][sl, i][:, None] - ket["P"][:, j][None, :]
                        pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
                        R = _hermite_coulomb(bra["cls"] + ket["cls"], p * q / (p + q), V)
                        M = torch.stack([torch.stack([(-1) ** sum(k) * R[tuple(x + y for x, y in zip(h, k))] * pre
                                                      for k in hk], -1) for h in hb], -2)  # bra, ket, hb, hk
                        vals = vals + torch.einsum("bfh,bqhk,qgk->bfqg", bra["E"][sl, i], M, ket["E"][:, j])
                ij = bra["ao"][sl, :, 0] * n + bra["ao"][sl, :, 1]
                ji = bra["ao"][sl, :, 1] * n + bra["ao"][sl, :, 0]
                vals = vals.reshape(ij.numel(), kl.numel())
                for x in (ij.reshape(-1, 1), ji.reshape(-1, 1)):
                    for y in (kl.reshape(1, -1), lk.reshape(1, -1)):
                        XX[x, y] = vals
                        if bra is not ket:
                            XX[y.T, x.T] = vals.T
    return XX.reshape(n, n, n, n)


def _coulomb(XX, D):
    n = D.shape[0]
    return (XX.reshape(n * n, n * n) @ D.reshape(-1)).reshape(n, n)


def _exchange(XX, D):
    return torch.stack([torch.einsum("jkl,jl->k", XX[i], D) for i in range(D.shape[0])])


def _pair_energies(XX, Ci, Ca, Cj, Cb, ei, ea, ej, eb):
    """Same-spin (pairs once) and opposite-spin MP2 sums."""
    Y = torch.einsum("uvld,db->uvlb", XX, Cb)
    Y = torch.einsum("uvlb,lj->uvjb", Y, Cj)
    Y = torch.einsum("uvjb,va->uajb", Y, Ca)
    Om = torch.einsum("uajb,ui->iajb", Y, Ci)
    den = ei[:, None, None, None] - ea[:, None, None] + ej[:, None] - eb
    same = None
    if Om.shape[:2] == Om.shape[2:]:
        same = 0.25 * ((Om - Om.permute(0, 3, 2, 1)) ** 2 / den).sum().item()
    return same, (Om ** 2 / den).sum().item()


def _exact_job(sysm, uhf, dev):
    pairs = _pairs(_shells(sysm), dev)
    XX, S, H = _integrals(pairs, dev), _overlap(pairs, dev), _core(pairs, sysm, dev)
    s, U = torch.linalg.eigh(S)
    X = U / torch.sqrt(s) @ U.T
    occ = [sysm.nelcA, sysm.nelcB] if uhf else [sysm.nelcA]
    f = 1.0 if uhf else 2.0

    def orbitals(F):
        e, V = torch.linalg.eigh(X @ F @ X)
        return e, X @ V

    xyz, Z = np.asarray(sysm.xyz, dtype=float), [float(z) for z in sysm.atoms]
    Enuc = sum(Z[i] * Z[j] / np.linalg.norm(xyz[i] - xyz[j]) for i in range(len(Z)) for j in range(i))
    sol = [orbitals(H) for _ in occ]
    D = [f * C[:, :k] @ C[:, :k].T for (_, C), k in zip(sol, occ)]
    hist = []
    for it in range(300):
        J = _coulomb(XX, sum(D))
        F = [H + J - (1.0 if uhf else 0.5) * _exchange(XX, d) for d in D]
        E = Enuc + sum(0.5 * (d * (H + x)).sum().item() for d, x in zip(D, F))
        err = torch.stack([X @ (x @ d @ S - S @ d @ x) @ X for x, d in zip(F, D)])
        hist = (hist + [(torch.stack(F), err)])[-8:]
        m = len(hist)
        B = torch.zeros(m + 1, m + 1, dtype=torch.float64)
        for i in range(m):
            for j in range(m):
                B[i, j] = (hist[i][1] * hist[j][1]).sum().item()
        B[:m, :m] /= max(float(B[m - 1, m - 1]), 1e-300)
        B[m, :m] = B[:m, m] = -1.0
        rhs = torch.zeros(m + 1, dtype=torch.float64)
        rhs[m] = -1.0
        w = torch.linalg.lstsq(B, rhs, driver="gelsd").solution[:m]
        done = float(err.abs().max()) < 1e-11 or it == 299
        Fx = F if done else list(sum(float(c) * h[0] for c, h in zip(w, hist)))
        sol = [orbitals(x) for x in Fx]
        if done:
            break
        D = [f * C[:, :k] @ C[:, :k].T for (_, C), k in zip(sol, occ)]
    eC = [(e, C[:, :k], C[:, k:], e[:k], e[k:]) for (e, C), k in zip(sol, occ)]
    if uhf:
        (_, Ci, Ca, ei, ea), (_, Cj, Cb, ej, eb) = eC
        E2 = (_pair_energies(XX, Ci, Ca, Ci, Ca, ei, ea, ei, ea)[0] + _pair_energies(XX, Cj, Cb, Cj, Cb, ej, eb, ej, eb)[0]
              + _pair_energies(XX, Ci, Ca, Cj, Cb, ei, ea, ej, eb)[1])
    else:
        (_, Ci, Ca, ei, ea), = eC
        same, both = _pair_energies(XX, Ci, Ca, Ci, Ca, ei, ea, ei, ea)
        E2 = 2 * same + both
    stack = (lambda v: torch.stack(v)) if uhf else (lambda v: v[0])
    return {"S": S, "H": H, "E": np.float64(E), "eps": stack([e for e, *_ in eC]), "D": stack(D),
            "E_MP2": np.float64(E2)}


def _exact_training(case, seed, dev):
    """Adam on the weighted squared error, without the network's BF16 roundings."""
    X, T, W, p0, dims = _training_set(case, seed)
    X, T, W = (torch.tensor(v, device=dev).double() for v in (X, T, W))
    p = torch.tensor(p0, device=dev).double().requires_grad_(True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    perm = np.random.default_rng(1).permutation(len(X)).astype(np.int64)
    losses = []
    for step in range(len(X) // case["batch"]):
        i = torch.tensor(perm[step * case["batch"]: (step + 1) * case["batch"]], device=dev)
        y, o = X[i], 0
        for k in range(3):
            nw = dims[k + 1] * dims[k]
            y = y @ p[o: o + nw].reshape(dims[k + 1], dims[k]).T + p[o + nw: o + nw + dims[k + 1]]
            o += nw + dims[k + 1]
            y = torch.nn.functional.silu(y) if k < 2 else y
        loss = (W[i] * (y - T[i]) ** 2).sum() / W[i].sum()
        g, = torch.autograd.grad(loss, p)
        losses.append(loss.item())
        with torch.no_grad():
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            t = step + 1
            p -= 2e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": float(np.mean(losses)), "params": p.detach()}
