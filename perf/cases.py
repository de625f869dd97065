"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points: the drop-in integral object, ``QuartetBatch``,
the Fock builders (restricted, unrestricted; FP64 and mixed precision), the batched Fock build,
the RHF gradient, the AO -> MO transform with its spin-orbital expansion and the
exchange-correlation build.  Molecules are the seeded water clusters and chains of
``gaussium_gb300.molecules`` in the basis sets of ``gaussium_gb300/data``; random shell quartets
follow ``gaussium_gb300.workloads``.  ``exact`` evaluates the same quantities with plain torch
in 64 bits: integrals by the McMurchie-Davidson scheme (J. Comput. Phys. 26, 218 (1978)).
"""
import math
import types

import numpy as np
import torch

from gaussium_gb300 import dropin, gradient, kohnsham, transform
from gaussium_gb300.basis import Basis, PrimitiveBasis, ShellBasis
from gaussium_gb300.batch import BatchedRHF
from gaussium_gb300.engine import PRIM_SCREEN, DeviceShells, JKEngine, QuartetBatch
from gaussium_gb300.fock import FockMatrixRestrictedGPU, FockMatrixUnrestrictedGPU
from gaussium_gb300.molecules import (BOHR_PER_ANGSTROM, perturbed, random_chain, shell_basis,
                                      water_cluster)
from gaussium_gb300.workloads import normalised_shells

COMPONENTS = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
              2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)]}
NCART = {0: 1, 1: 3, 2: 6}
# functions and shells of one water molecule
WATER = {"STO-3G": (7, 5), "6-31G": (13, 9), "6-31G*": (19, 10)}


# ---------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one (ij|kl) through the drop-in integral object: the reference's unit of work, as
        # its own tests and calculate_integral call it
        {"name": "integral", "kind": "integral", "l": 5, "k": 3},
        # blocks of a small list of shell quartets (the size of the parity tests): launches
        {"name": "blocks_4k", "kind": "blocks", "n": 4096},
        # the synthetic integral workload, large enough that outputs exceed the L2
        {"name": "blocks_300k", "kind": "blocks", "n": 300000},
        # single-precision blocks of a molecule's shell quartets
        {"name": "blocks32_water8", "kind": "blocks32", "n": 400000, "waters": 8},
        # one SCF iteration's Fock matrix of a small molecule
        {"name": "fock_water2", "kind": "fock", "waters": 2, "basis": "6-31G*", "mode": "fp64"},
        # the same for a cluster of the size that the benchmark reports, in FP64
        {"name": "fock_water16", "kind": "fock", "waters": 16, "basis": "6-31G*", "mode": "fp64"},
        # and mixed precision with density screening, on a larger one
        {"name": "fock_mixed_water24", "kind": "fock", "waters": 24, "basis": "6-31G*",
         "mode": "mixed"},
        # unrestricted: one Coulomb and two exchange matrices from one pass
        {"name": "fock_uhf_water7", "kind": "fock", "waters": 7, "basis": "6-31G*", "mode": "uhf"},
        # Fock matrices of many small molecules at once, as the batched SCF builds them
        {"name": "fock_batch_24", "kind": "batch", "molecules": 24, "basis": "6-31G*",
         "mixed": True},
        # nuclear gradient from a converged state, its default precision
        {"name": "gradient_water6", "kind": "gradient", "waters": 6, "basis": "6-31G*"},
        # MO integrals and antisymmetrised spin-orbital tensor (the input of MP2 and CCSD)
        {"name": "mo_water3", "kind": "mo", "waters": 3, "basis": "6-31G"},
        # exchange-correlation matrix and energy for a new density
        {"name": "xc_water4", "kind": "xc", "waters": 4, "basis": "6-31G*", "radial": 200},
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["integral", "blocks", "blocks", "blocks32", "fock", "fock", "fock", "batch",
                       "gradient", "mo", "xc"])
    if kind == "integral":
        return {"kind": kind, "l": rng.randint(0, 8), "k": rng.randint(1, 6)}
    if kind == "blocks":
        return {"kind": kind, "n": log_int(64, 300000)}
    if kind == "blocks32":
        return {"kind": kind, "n": log_int(64, 400000), "waters": rng.randint(2, 8)}
    if kind == "fock":
        mode = rng.choice(["fp64", "mixed", "uhf"])
        return {"kind": kind, "waters": log_int(1, 16), "mode": mode,
                "basis": rng.choice(["6-31G", "6-31G*"])}
    if kind == "batch":
        return {"kind": kind, "molecules": log_int(2, 24), "mixed": rng.choice([True, False]),
                "basis": rng.choice(["6-31G", "6-31G*"])}
    if kind == "gradient":
        return {"kind": kind, "waters": rng.randint(2, 6), "basis": rng.choice(["6-31G", "6-31G*"])}
    if kind == "mo":
        return {"kind": kind, "waters": rng.randint(1, 3), "basis": rng.choice(["STO-3G", "6-31G"])}
    return {"kind": kind, "waters": rng.randint(1, 4), "radial": rng.choice([100, 150, 200]),
            "basis": rng.choice(["STO-3G", "6-31G", "6-31G*"])}


# ---------------------------------------------------------------------------------- inputs
def _orbitals(mol, sb, seed, nocc=None):
    """Occupied orbitals as an SCF hands them on, without running one: localised on their
    molecules, decaying with distance, normalised (N x nocc)."""
    rng = np.random.default_rng(seed)
    nocc = mol.electrons // 2 if nocc is None else nocc
    heavy = [i for i, s in enumerate(mol.symbols) if s != "H"]
    centre = np.repeat(sb.centre, sb.nfunc, axis=0)
    home = mol.coords[[heavy[i % len(heavy)] for i in range(nocc)]]
    r = np.linalg.norm(centre[:, None, :] - home[None, :, :], axis=2)
    c = rng.standard_normal((sb.nbf, nocc)) * np.exp(-0.7 * r)
    return c / np.linalg.norm(c, axis=0)


def _density(mol, sb, seed, factor=2.0, nocc=None):
    c = _orbitals(mol, sb, seed, nocc)
    p = factor * c @ c.T
    return 0.5 * (p + p.T)


def _four_functions(case, seed):
    """Four contracted functions of total angular momentum ``l`` (uneven among them)."""
    rng = np.random.default_rng(1000 + seed)
    base, extra = divmod(case["l"], 4)
    funcs = []
    for i in range(4):
        lmn_all = COMPONENTS[base + (1 if i < extra else 0)]
        lmn = lmn_all[int(rng.integers(len(lmn_all)))]
        xyz = tuple(float(v) for v in rng.uniform(-1.5, 1.5, 3))
        expo = np.exp(rng.uniform(np.log(0.1), np.log(50.0), case["k"]))
        coef = rng.uniform(0.1, 0.8, case["k"])
        prims = [PrimitiveBasis(float(c), float(e), xyz, lmn) for c, e in zip(coef, expo)]
        funcs.append(Basis(prims, xyz, lmn))
    return funcs


def _random_quartets(case, seed):
    """``workloads.random_shell_quartets`` with the angular momenta of a case held fixed, so that
    every seed's blocks have the same layout: 1 to 6 primitives a shell, exponents from 0.05 to
    1e4, centres in a 10 A cube."""
    ns = 4 * case["n"]
    l = np.random.default_rng(case["n"]).integers(0, 3, size=ns)
    rng = np.random.default_rng(seed)
    nprim = rng.integers(1, 7, size=ns)
    total = int(nprim.sum())
    expo = np.exp(rng.uniform(np.log(0.05), np.log(1e4), size=total))
    centre = rng.uniform(0.0, 10.0, size=(ns, 3)) * BOHR_PER_ANGSTROM
    coef, scale = normalised_shells(l, nprim, expo, rng.standard_normal(total))
    sb = ShellBasis(l, centre, np.concatenate([[0], np.cumsum(nprim)]), expo, coef, scale)
    return sb, np.arange(ns, dtype=np.int64).reshape(-1, 4)


def _molecule_quartets(case, seed):
    """Shell quartets of a water cluster in 6-31G*: the same quartets at every seed's geometry."""
    sb = _cluster({"waters": case["waters"], "basis": "6-31G*"}, seed)[1]
    rng = np.random.default_rng(case["n"])
    return sb, rng.integers(0, sb.nshell, size=(case["n"], 4))


def _chains(case, seed):
    """Small C/N/O chains with their hydrogens, at most 14 atoms, every nucleus displaced."""
    return [perturbed(random_chain(i, max_atoms=14), 0.05, seed + i)
            for i in range(case["molecules"])]


def _cluster(case, seed):
    mol = water_cluster(case["waters"], seed=seed)
    return mol, shell_basis(mol, case["basis"])


def prepare(case, seed):
    s = types.SimpleNamespace(kind=case["kind"])
    if s.kind == "integral":
        s.integral = dropin.GpuObaraSaika()
        s.functions = _four_functions(case, seed)
    elif s.kind in ("blocks", "blocks32"):
        sb, quartets = _random_quartets(case, seed) if s.kind == "blocks" else \
            _molecule_quartets(case, seed)
        s.precision = 64 if s.kind == "blocks" else 32
        ds = DeviceShells(sb)
        s.batch = QuartetBatch(ds, quartets, want32=s.precision == 32, max_exp=PRIM_SCREEN)
        s.out = torch.zeros(s.batch.total, dtype=torch.float64, device=ds.device)
    elif s.kind == "fock":
        mol, sb = _cluster(case, seed)
        rng = np.random.default_rng(seed)
        h = rng.standard_normal((sb.nbf, sb.nbf))
        h = -5.0 * np.eye(sb.nbf) + 0.05 * (h + h.T)
        engine = JKEngine(sb)
        if case["mode"] == "uhf":
            s.builder = FockMatrixUnrestrictedGPU(h, engine)
            nocc = mol.electrons // 2
            s.densities = (_density(mol, sb, seed, 1.0, nocc + 1),
                           _density(mol, sb, seed + 1, 1.0, nocc - 1))
        else:
            kw = {"mixed_cut": 1e-3, "screen_thr": 1e-12} if case["mode"] == "mixed" else {}
            s.builder = FockMatrixRestrictedGPU(h, engine, **kw)
            s.densities = (_density(mol, sb, seed),)
    elif s.kind == "batch":
        s.batch = BatchedRHF(_chains(case, seed), basis=case["basis"])
        p = np.concatenate([_density(m, sb, seed + i).ravel()
                            for i, (m, sb) in enumerate(zip(s.batch.mols, s.batch.sbs))])
        s.packed = torch.as_tensor(p).to(s.batch.dev)
        s.options = {"mixed_cut": 1e-3, "screen_thr": 1e-12} if case["mixed"] else {}
    elif s.kind == "gradient":
        mol, sb = _cluster(case, seed)
        c = _orbitals(mol, sb, seed)
        eps = -np.random.default_rng(seed).uniform(0.3, 20.0, c.shape[1])
        w = 2.0 * (c * eps) @ c.T
        s.state = gradient.RHFState(mol, sb, JKEngine(sb, schwarz_thr=1e-14), 0.0, None,
                                    _density(mol, sb, seed), 0.5 * (w + w.T))
    elif s.kind == "mo":
        mol, s.sb = _cluster(case, seed)
        s.c = _rotation(s.sb.nbf, seed)
    elif s.kind == "xc":
        mol, sb = _cluster(case, seed)
        s.xc = kohnsham.ExchangeCorrelationGPU(sb, params=(2 / 3, kohnsham.VWN3),
                                               radial=case["radial"])
        s.xc.phi()
        s.p = torch.as_tensor(_density(mol, sb, seed)).to(s.xc.device)
    else:
        raise ValueError(s.kind)
    return s


def _rotation(n, seed):
    q, r = np.linalg.qr(np.random.default_rng(seed).standard_normal((n, n)))
    return np.ascontiguousarray(q * np.sign(np.diag(r)))


def run(s):
    if s.kind == "integral":
        return s.integral.integrate(*s.functions)
    if s.kind in ("blocks", "blocks32"):
        # a geometry's pair records, then its blocks
        s.batch.pairs.build(want32=s.precision == 32)
        s.batch.run(s.out, s.precision)
        # a caller of the 32-bit evaluation keeps 32-bit blocks
        return s.out if s.precision == 64 else s.out.to(torch.float32)
    if s.kind == "fock":
        return s.builder.create(*s.densities)
    if s.kind == "batch":
        return s.batch.fock_packed(s.packed, **s.options)
    if s.kind == "gradient":
        return gradient.gradient_from_state(s.state)
    if s.kind == "mo":
        mo = transform.mo_integrals(s.sb, s.c)
        return mo, transform.spin_expand_device(mo, transform.SPIN_ANTI_PHYSICIST)
    return s.xc.evaluate_device(s.p)


# ---------------------------------------------------------------------------------- work
# floating-point operations of the Obara-Saika recursions, the Boys functions and the Fock or
# gradient contraction, per shell quartet: averages of the generated recursions over the random
# quartets (16 screened primitive quartets each) and over water clusters
FLOP_RANDOM, FLOP_WATER = 21500, {"STO-3G": 9000, "6-31G": 1900, "6-31G*": 2300}


def _water_quartets(n, basis):
    """Unique shell quartets of (H2O)n above the Schwarz threshold, to about 20 %."""
    pairs = n * WATER[basis][1]
    pairs = pairs * (pairs + 1) // 2
    return 0.5 * pairs * (pairs + 1) * min(1.0, 1.35 * n ** -0.7)


def work(case):
    kind = case["kind"]
    if kind == "integral":
        return {"bytes": 64 * case["k"] + 8, "flops": 100 * (1 + case["l"]) ** 2 * case["k"] ** 4}
    if kind == "blocks":
        # shells (about 3.5 primitives each) in, blocks (on average (10/3)^4 integrals) out
        return {"bytes": case["n"] * (4 * (3.5 * 16 + 88) + 8 * (10 / 3) ** 4),
                "flops": case["n"] * FLOP_RANDOM}
    if kind == "blocks32":
        # 1.9 functions and 2.2 primitives a shell
        return {"bytes": case["n"] * (24 + 4 * 1.9 ** 4) + case["waters"] * 10 * 124,
                "flops": case["n"] * 4500}
    if kind == "fock":
        n = case["waters"] * WATER[case["basis"]][0]
        mats = {"fp64": 3, "mixed": 3, "uhf": 5}[case["mode"]]
        return {"bytes": mats * 8 * n * n,
                "flops": _water_quartets(case["waters"], case["basis"]) * FLOP_WATER[case["basis"]]}
    if kind == "batch":
        # chains of up to 14 atoms have about 60 (6-31G) or 85 functions and 45 shells
        n = 60 if case["basis"] == "6-31G" else 85
        return {"bytes": case["molecules"] * 16 * n * n,
                "flops": case["molecules"] * 45 ** 4 / 8 * 0.8 * FLOP_WATER[case["basis"]]}
    if kind == "gradient":
        n = case["waters"] * WATER[case["basis"]][0]
        return {"bytes": 16 * n * n + 72 * case["waters"],
                "flops": 3 * _water_quartets(case["waters"], case["basis"]) *
                FLOP_WATER[case["basis"]]}
    n = case["waters"] * WATER[case["basis"]][0]
    if kind == "mo":
        return {"bytes": 8 * (17 * n ** 4 + n * n),
                "flops": 4 * n ** 5 + _water_quartets(case["waters"], case["basis"]) *
                FLOP_WATER[case["basis"]]}
    grid = 648 * case["radial"]
    return {"bytes": 8 * (grid * n + 2 * n * n), "flops": 4 * grid * n * n}


# ---------------------------------------------------------------------------------- exact
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _boys(mmax, t):
    """F_0..F_mmax(t): Kummer's series and downward recursion below t = 45, the asymptotic
    form (its error there under e^-45) and upward recursion above."""
    small = torch.where(t < 45.0, t, torch.zeros_like(t))
    term = torch.full_like(t, 1.0 / (2 * mmax + 1))
    top = term.clone()
    for i in range(1, 190):
        term = term * (2.0 * small / (2 * mmax + 2 * i + 1))
        top += term
    e = torch.exp(-small)
    low = [None] * (mmax + 1)
    low[mmax] = top * e
    for m in range(mmax, 0, -1):
        low[m - 1] = (2.0 * small * low[m] + e) / (2 * m - 1)
    big = torch.where(t < 45.0, torch.full_like(t, 45.0), t)
    eb = torch.exp(-big)
    high = [0.5 * torch.sqrt(math.pi / big)]
    for m in range(mmax):
        high.append(((2 * m + 1) * high[m] - eb) / (2.0 * big))
    return [torch.where(t < 45.0, a, b) for a, b in zip(low, high)]


def _hermite(l):
    return [(t, u, v) for t in range(l + 1) for u in range(l + 1 - t) for v in range(l + 1 - t - u)]


class _Pairs:
    """Primitive pairs of a list of shell pairs (of one la, lb): exponent, centre, and the matrix
    from Hermite to Cartesian functions, coefficients and component scales included."""

    def __init__(self, sh, ia, ib, la, lb):
        dev = sh["expo"].device
        na, nb = sh["nprim"][ia], sh["nprim"][ib]
        cnt = na * nb
        owner = torch.repeat_interleave(torch.arange(len(ia), device=dev), cnt)
        k = torch.arange(len(owner), device=dev) - (torch.cumsum(cnt, 0) - cnt)[owner]
        pa = sh["off"][ia][owner] + k // nb[owner]
        pb = sh["off"][ib][owner] + k % nb[owner]
        a, b = sh["expo"][pa], sh["expo"][pb]
        A, B = sh["centre"][ia][owner], sh["centre"][ib][owner]
        x = a * b / (a + b) * ((A - B) ** 2).sum(1)
        keep = x < 64.0
        owner, a, b, A, B, pa, pb = (v[keep] for v in (owner, a, b, A, B, pa, pb))
        p = a + b
        P = (a[:, None] * A + b[:, None] * B) / p[:, None]
        # one-dimensional coefficients E[i][j][t] for the three axes at once
        e = {(0, 0, 0): torch.exp(-(a * b / p)[:, None] * (A - B) ** 2)}
        zero = torch.zeros_like(P)
        g = lambda i, j, t: e.get((i, j, t), zero)   # noqa: E731
        h = (0.5 / p)[:, None]
        for i in range(la + 1):
            for j in range(lb + 1):
                if i == j == 0:
                    continue
                for t in range(i + j + 1):
                    if i > 0:
                        e[i, j, t] = h * g(i - 1, j, t - 1) + (P - A) * g(i - 1, j, t) + \
                            (t + 1) * g(i - 1, j, t + 1)
                    else:
                        e[i, j, t] = h * g(i, j - 1, t - 1) + (P - B) * g(i, j - 1, t) + \
                            (t + 1) * g(i, j - 1, t + 1)
        herm = _hermite(la + lb)
        c = sh["coef"][pa] * sh["coef"][pb]
        E = torch.zeros((len(p), NCART[la] * NCART[lb], len(herm)), dtype=torch.float64, device=dev)
        for x1, ca in enumerate(COMPONENTS[la]):
            for x2, cb in enumerate(COMPONENTS[lb]):
                s = c * sh["scale"][ia][owner, x1] * sh["scale"][ib][owner, x2]
                for y, tuv in enumerate(herm):
                    if all(t <= i + j for t, i, j in zip(tuv, ca, cb)):
                        E[:, x1 * NCART[lb] + x2, y] = s * e[ca[0], cb[0], tuv[0]][:, 0] * \
                            e[ca[1], cb[1], tuv[1]][:, 1] * e[ca[2], cb[2], tuv[2]][:, 2]
        self.p, self.P, self.E, self.herm = p, P, E, herm
        cnt = torch.bincount(owner, minlength=len(ia))
        self.cnt, self.first = cnt, torch.cumsum(cnt, 0) - cnt


def _class_blocks(sh, q, l4):
    """Blocks (n, na nb, nc nd) of shell quartets q (n, 4) of one class."""
    dev = q.device
    bra, ket = _Pairs(sh, q[:, 0], q[:, 1], l4[0], l4[1]), _Pairs(sh, q[:, 2], q[:, 3], l4[2], l4[3])
    L = sum(l4)
    out = torch.zeros((len(q), bra.E.shape[1], ket.E.shape[1]), dtype=torch.float64, device=dev)
    tot = bra.cnt * ket.cnt
    end = torch.cumsum(tot, 0)
    total = int(end[-1])
    step = 40000
    hl = {tuv: k for k, tuv in enumerate(_hermite(L))}
    idx = torch.tensor([[hl[tuple(a + b for a, b in zip(x, y))] for y in ket.herm]
                        for x in bra.herm], device=dev)
    sign = torch.tensor([(-1.0) ** sum(y) for y in ket.herm], dtype=torch.float64, device=dev)
    for lo in range(0, total, step):
        g = torch.arange(lo, min(total, lo + step), device=dev)
        owner = torch.searchsorted(end, g, right=True)
        k = g - (end - tot)[owner]
        i = bra.first[owner] + k // ket.cnt[owner]
        j = ket.first[owner] + k % ket.cnt[owner]
        p, r = bra.p[i], ket.p[j]
        X = bra.P[i] - ket.P[j]
        al = p * r / (p + r)
        pref = 2.0 * math.pi ** 2.5 / (p * r * torch.sqrt(p + r))
        F = _boys(L, al * (X ** 2).sum(1))
        R = {}
        f = pref
        for n in range(L + 1):
            R[n, 0, 0, 0] = f * F[n]
            f = f * (-2.0 * al)
        x, y, z = X[:, 0], X[:, 1], X[:, 2]
        for t, u, v in sorted(hl, key=sum):
            if t + u + v == 0:
                continue
            for n in range(L - t - u - v + 1):
                if t > 0:
                    w = x * R[n + 1, t - 1, u, v]
                    R[n, t, u, v] = w + (t - 1) * R[n + 1, t - 2, u, v] if t > 1 else w
                elif u > 0:
                    w = y * R[n + 1, t, u - 1, v]
                    R[n, t, u, v] = w + (u - 1) * R[n + 1, t, u - 2, v] if u > 1 else w
                else:
                    w = z * R[n + 1, t, u, v - 1]
                    R[n, t, u, v] = w + (v - 1) * R[n + 1, t, u, v - 2] if v > 1 else w
        R0 = torch.stack([R[(0,) + tuv] for tuv in hl], 1)
        m = R0[:, idx] * sign
        out.index_add_(0, owner, torch.bmm(torch.bmm(bra.E[i], m), ket.E[j].transpose(1, 2)))
    return out


def _blocks(sb, quartets):
    """Blocks of shell quartets (n, 4) of a shell basis, flat in the caller's order."""
    dev = _device()
    t = lambda a, d: torch.as_tensor(np.asarray(a), dtype=d, device=dev)   # noqa: E731
    sh = {"expo": t(sb.expo, torch.float64), "coef": t(sb.coef, torch.float64),
          "centre": t(sb.centre, torch.float64), "scale": t(sb.comp_scale, torch.float64),
          "off": t(sb.prim_off[:-1], torch.int64), "nprim": t(sb.nprim, torch.int64)}
    q = t(quartets, torch.int64)
    l4 = t(sb.l, torch.int64)[q]
    nc = torch.tensor([1, 3, 6], device=dev)[l4].prod(1)
    off = torch.cumsum(nc, 0) - nc
    out = torch.zeros(int(nc.sum()), dtype=torch.float64, device=dev)
    key = ((l4[:, 0] * 3 + l4[:, 1]) * 3 + l4[:, 2]) * 3 + l4[:, 3]
    for c in torch.unique(key).tolist():
        rows = torch.nonzero(key == c).flatten()
        ls = (c // 27, c // 9 % 3, c // 3 % 3, c % 3)
        b = _class_blocks(sh, q[rows], ls).reshape(len(rows), -1)
        out[off[rows][:, None] + torch.arange(b.shape[1], device=dev)] = b
    return out


def _tensor(sb):
    """The dense (ij|kl) tensor from the unique shell quartets and their index images."""
    n = sb.nbf
    i, j = np.tril_indices(sb.nshell)
    a, b = np.tril_indices(len(i))
    q = np.stack([i[a], j[a], i[b], j[b]], 1)
    vals = _blocks(sb, q)
    dev = vals.device
    nf, fo = sb.nfunc, sb.func_off
    size = nf[q].astype(np.int64).prod(1)
    owner = np.repeat(np.arange(len(q)), size)
    k = np.arange(len(owner)) - np.repeat(np.cumsum(size) - size, size)
    f = nf[q][owner].astype(np.int64)
    x3 = k % f[:, 3]
    x2 = k // f[:, 3] % f[:, 2]
    x1 = k // (f[:, 3] * f[:, 2]) % f[:, 1]
    x0 = k // (f[:, 3] * f[:, 2] * f[:, 1])
    w = [torch.as_tensor(fo[q[owner, c]].astype(np.int64) + x).to(dev)
         for c, x in enumerate((x0, x1, x2, x3))]
    t = torch.zeros((n, n, n, n), dtype=torch.float64, device=dev)
    a, b, c, d = w
    for ix in ((a, b, c, d), (b, a, c, d), (a, b, d, c), (b, a, d, c),
               (c, d, a, b), (d, c, a, b), (c, d, b, a), (d, c, b, a)):
        t[ix] = vals
    return t


def _lda(rho, alpha, vwn):
    """Potential and energy density of Slater's exchange (parameter alpha) and the VWN fit for an
    unpolarised density (Can. J. Phys. 58, 1200 (1980))."""
    ex = -9 / 8 * alpha * (3.0 / math.pi) ** (1 / 3) * rho ** (1 / 3)
    A, x0, b, c = vwn
    x = torch.sqrt((3.0 / (4.0 * math.pi * rho)) ** (1 / 3))
    X = lambda y: y * y + b * y + c   # noqa: E731
    q = math.sqrt(4 * c - b * b)
    at = torch.atan(q / (2 * x + b))
    ec = 0.5 * A * (torch.log(x * x / X(x)) + 2 * b / q * at -
                    b * x0 / X(x0) * (torch.log((x - x0) ** 2 / X(x)) + 2 * (b + 2 * x0) / q * at))
    vc = ec - A / 6 * (c * (x - x0) - b * x0 * x) / ((x - x0) * X(x))
    return 4 / 3 * ex + vc, ex + ec


def _xc(case, seed):
    mol, sb = _cluster(case, seed)
    dev = _device()
    n = case["radial"]
    t = np.arange(1, n + 1) * np.pi / (n + 1)
    x = np.cos(t)
    r = (1 + x) / (1 - x)
    wr = np.pi / (n + 1) * np.sin(t) * 2 / (1 - x) ** 2 * r * r
    ct, wt = np.polynomial.legendre.leggauss(18)
    ph = 2 * np.pi * np.arange(36) / 36
    st = np.sqrt(1 - ct * ct)
    d = np.stack([np.outer(st, np.cos(ph)), np.outer(st, np.sin(ph)), np.outer(ct, np.ones(36))],
                 -1).reshape(-1, 3)
    pts = torch.as_tensor((r[:, None, None] * d[None]).reshape(-1, 3)).to(dev)
    w = torch.as_tensor(np.outer(wr, np.repeat(wt * 2 * np.pi / 36, 36)).reshape(-1)).to(dev)
    cols = []
    for s in range(sb.nshell):
        v = pts - torch.as_tensor(sb.centre[s]).to(dev)
        r2 = (v * v).sum(1)
        k = range(sb.prim_off[s], sb.prim_off[s + 1])
        rad = sum(float(sb.coef[i]) * torch.exp(-float(sb.expo[i]) * r2) for i in k)
        for m, (lx, ly, lz) in enumerate(COMPONENTS[int(sb.l[s])]):
            cols.append(float(sb.comp_scale[s, m]) * v[:, 0] ** lx * v[:, 1] ** ly *
                        v[:, 2] ** lz * rad)
    phi = torch.stack(cols, 1)
    p = torch.as_tensor(_density(mol, sb, seed)).to(dev)
    rho = ((phi @ p) * phi).sum(1)
    ok = rho > 1e-300
    v, e = _lda(torch.where(ok, rho, torch.ones_like(rho)), 2 / 3, kohnsham.VWN3)
    zero = torch.zeros_like(rho)
    wv, we = torch.where(ok, w * v, zero), torch.where(ok, w * rho * e, zero)
    V = phi.T @ (phi * wv[:, None])
    return 0.5 * (V + V.T), we.sum()


def exact(case, seed):
    kind = case["kind"]
    if kind == "integral":
        f = _four_functions(case, seed)
        ls = [sum(g.integral_exponents) for g in f]
        expo = np.concatenate([[p.exponent for p in g.primitive_gaussian_array] for g in f])
        coef = np.concatenate([[p.contraction * p.normalisation * g.normalisation
                                for p in g.primitive_gaussian_array] for g in f])
        sb = types.SimpleNamespace(l=np.array(ls), expo=expo, coef=coef,
                                   centre=np.array([g.coordinates for g in f]),
                                   comp_scale=np.ones((4, 6)), nprim=np.full(4, case["k"]),
                                   prim_off=np.arange(5) * case["k"])
        at = tuple(COMPONENTS[l].index(tuple(g.integral_exponents)) for l, g in zip(ls, f))
        b = _blocks(sb, [[0, 1, 2, 3]]).reshape([NCART[l] for l in ls])
        return float(b[at])
    if kind == "blocks":
        return _blocks(*_random_quartets(case, seed))
    if kind == "blocks32":
        return _blocks(*_molecule_quartets(case, seed))
    if kind == "fock":
        if case["waters"] > 2:
            return None                    # the dense tensor would take minutes
        mol, sb = _cluster(case, seed)
        rng = np.random.default_rng(seed)
        h = rng.standard_normal((sb.nbf, sb.nbf))
        h = -5.0 * np.eye(sb.nbf) + 0.05 * (h + h.T)
        t = _tensor(sb)
        J = lambda p: torch.einsum("ijkl,kl->ij", t, p)   # noqa: E731
        K = lambda p: torch.einsum("ikjl,kl->ij", t, p)   # noqa: E731
        up = lambda p: torch.as_tensor(p).to(t.device)    # noqa: E731
        if case["mode"] == "uhf":
            nocc = mol.electrons // 2
            pa = up(_density(mol, sb, seed, 1.0, nocc + 1))
            pb = up(_density(mol, sb, seed + 1, 1.0, nocc - 1))
            j = J(pa + pb)
            return h + (j - K(pa)).cpu().numpy(), h + (j - K(pb)).cpu().numpy()
        p = up(_density(mol, sb, seed))
        return h + (J(p) - 0.5 * K(p)).cpu().numpy()
    if kind == "mo":
        _, sb = _cluster(case, seed)
        c = torch.as_tensor(_rotation(sb.nbf, seed)).to(_device())
        mo = torch.einsum("abcd,ds->abcs", _tensor(sb), c)
        mo = torch.einsum("abcs,cr->abrs", mo, c)
        mo = torch.einsum("abrs,bq->aqrs", mo, c)
        mo = torch.einsum("aqrs,ap->pqrs", mo, c)
        n = sb.nbf
        # <rs||tu> = (rt|su) - (ru|st) over interleaved spin orbitals
        spin = torch.arange(2 * n, device=mo.device) % 2
        same = (spin[:, None] == spin[None, :]).double()
        up = torch.arange(2 * n, device=mo.device) // 2
        s = mo[up][:, up][:, :, up][:, :, :, up] * same[:, :, None, None] * same[None, None]
        return mo, s.permute(0, 2, 1, 3) - s.permute(0, 2, 3, 1)
    if kind == "xc":
        return _xc(case, seed)
    return None         # batches and gradients: plain tensors would take minutes
