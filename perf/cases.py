"""The work that is measured when this engine's speed is measured.

A case is one call, or one short sequence of calls, that a quantum-chemistry program makes of the
engine: a single libgrpp-style block, the batched matrices of a small or a large system, a kept
plan, the density-contracted gradient, the one-electron and nuclear-attraction batches. Systems
come from ``libgrpp_b200.synthetic`` (the workloads of the tests and of bench.py) with the case's
sizes and the given seed; results are the arrays that the call returns.

``exact`` evaluates the same integrals by direct quadrature in 64 bits (product grids on the sphere
times Gauss-Legendre panels in r for the pseudopotential blocks; Gauss-Hermite and Gauss-Legendre
rules for the one-electron integrals), with torch alone. It covers the cases whose exponents an
angular grid resolves; for the others (exponents up to 5e3 bohr^-2 at 3 to 40 bohr from the centre,
thousands of tasks) such a grid takes minutes, and it returns None.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from libgrpp_b200 import engine, synthetic
from libgrpp_b200.system import ncart

PLAIN, LEARNED = 0, 1
OVERLAP, KINETIC, MOMENTUM = 0, 1, 2
POINT, GAUSSIAN = 0, 2  # nuclear charge distributions (include/libgrpp.h)


def listed():
    return [
        # one call of libgrpp_full_grpp_integrals: a program linked against libgrpp that has not been
        # changed and loops over shell pairs; f x d on two atoms, U_L + AREP + SO + outercore
        {"name": "block", "kind": "block", "la": 3, "lb": 2, "centre": 1},
        # one call of libgrpp_full_grpp_integrals_gradient of such a program
        {"name": "block_gradient", "kind": "block_gradient", "la": 2, "lb": 1, "centre": 1},
        # every shell pair x centre of a three-atom molecule with two heavy atoms: a small SCF's matrices
        {"name": "triatomic", "kind": "triatomic"},
        # scalar-relativistic potentials, s..g shells: an odd-sized piece of a 64-atom system's matrices ...
        {"name": "scalar_piece", "kind": "scalar", "atoms": 64, "bra": 9, "ket": 7, "mode": PLAIN},
        # ... and the 32 x 32 shell block x 64 centres of bench.py, walk scheduled by the level model
        {"name": "scalar_block", "kind": "scalar", "atoms": 64, "bra": 32, "ket": 32, "mode": LEARNED},
        # the same integrals from a plan that the program keeps (device-resident inputs)
        {"name": "scalar_plan", "kind": "plan", "atoms": 64, "bra": 16, "ket": 16, "mode": PLAIN},
        # a molecule with shells up to i and full GRPPs with projectors up to h: all its matrices
        {"name": "molecule_small", "kind": "molecule", "atoms": 5, "lmax": 6, "l_proj": 5, "mode": PLAIN},
        {"name": "molecule_large", "kind": "molecule", "atoms": 15, "lmax": 6, "l_proj": 5, "mode": LEARNED},
        # d tr(D V)/dR of a geometry step: full GRPP up to h shells; general density ...
        {"name": "gradient_small", "kind": "gradient", "heavy": 2, "hydrogen": 4, "lmax": 5, "symmetric": False, "mode": PLAIN},
        # ... and an SCF density (symmetric), a larger molecule
        {"name": "gradient_scf", "kind": "gradient", "heavy": 6, "hydrogen": 12, "lmax": 5, "symmetric": True, "mode": LEARNED},
        # kinetic energy matrix of a 48-atom molecule: every ordered shell pair
        {"name": "kinetic", "kind": "onee", "heavy": 16, "hydrogen": 32, "lmax": 4, "which": KINETIC},
        # nuclear attraction by finite (Gaussian) nuclei: every shell pair x nucleus of the three-atom molecule
        {"name": "finite_nuclei", "kind": "finite", "bra": 10, "ket": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block_gradient", "triatomic", "pair", "scalar", "scalar", "plan", "molecule", "molecule",
                       "gradient", "gradient", "onee", "nuclear", "finite"])
    if kind in ("block", "block_gradient"):
        return {"kind": kind, "la": rng.randint(0, 3), "lb": rng.randint(0, 3 if kind == "block" else 1), "centre": rng.randint(0, 1)}
    if kind in ("triatomic", "pair"):
        n = 10 if kind == "triatomic" else 8
        return {"kind": kind, "bra": rng.randint(2, n), "ket": rng.randint(2, n), "centres": rng.randint(1, 2) if kind == "triatomic" else 1}
    if kind in ("scalar", "plan"):
        return {"kind": kind, "atoms": _log_int(rng, 3, 64), "bra": _log_int(rng, 1, 32 if kind == "scalar" else 16),
                "ket": _log_int(rng, 1, 32 if kind == "scalar" else 16), "mode": rng.choice([PLAIN, LEARNED])}
    if kind == "molecule":
        return {"kind": kind, "atoms": rng.randint(2, 13), "lmax": rng.randint(3, 6), "l_proj": rng.randint(3, 5),
                "mode": rng.choice([PLAIN, LEARNED])}
    if kind == "gradient":
        h = _log_int(rng, 1, 5)
        return {"kind": kind, "heavy": h, "hydrogen": rng.randint(1, 2 * h), "lmax": rng.randint(2, 5),
                "symmetric": rng.random() < 0.5, "mode": rng.choice([PLAIN, LEARNED])}
    if kind == "onee":
        return {"kind": kind, "heavy": _log_int(rng, 1, 16), "hydrogen": _log_int(rng, 1, 32), "lmax": rng.randint(2, 5),
                "which": rng.choice([OVERLAP, KINETIC, MOMENTUM])}
    if kind == "finite":
        return {"kind": kind, "bra": rng.randint(2, 10), "ket": rng.randint(2, 10)}
    return {"kind": kind, "heavy": _log_int(rng, 1, 4), "hydrogen": rng.randint(1, 8), "lmax": rng.randint(2, 4)}


# ------------------------------------------------------------------------------------------ inputs

def _system(case, seed):
    """The case's System and its (bra, ket, centre) task arrays."""
    kind = case["kind"]
    if kind in ("block", "block_gradient", "triatomic", "finite"):
        S = synthetic.moderate_heavy_system(seed)
        if kind == "finite":  # every atom is a nucleus; the operators at the centres are not read
            S.centres = [(S.atoms[i].copy(), 0) for i in range(3)]
        if kind in ("triatomic", "finite"):
            a, b, c = S.all_tasks()
            keep = (a < case.get("bra", 10)) & (b < case.get("ket", 10)) & (c < case.get("centres", 3))
            return S, (a[keep], b[keep], c[keep])
        # bra on the first heavy atom; ket on the second one (d, f) or on the hydrogen (s, p)
        bra, ket = case["la"], 8 + case["lb"] if case["lb"] < 2 else 4 + case["lb"]
        return S, tuple(np.array([i], dtype=np.int32) for i in (bra, ket, case["centre"]))
    if kind == "pair":
        S = synthetic.config0(seed)
        a, b, c = S.all_tasks()
        keep = (a < case["bra"]) & (b < case["ket"])
        return S, (a[keep], b[keep], c[keep])
    if kind in ("scalar", "plan"):
        S = synthetic.config1(seed, n_atoms=case["atoms"])
        bra = np.arange(case["bra"]) % len(S.shells)
        ket = (np.arange(case["ket"]) + 32) % len(S.shells)
        a, b, c = (x.ravel() for x in np.meshgrid(bra, ket, np.arange(case["atoms"]), indexing="ij"))
        return S, synthetic.sort_tasks(S, a, b, c)
    if kind == "molecule":
        n = case["atoms"]
        heavy = max(1, n // 3)
        S = synthetic.config2(seed, n_heavy=heavy, n_h=n - heavy, lmax=case["lmax"], box=6.0 + 1.5 * n, l_proj=case["l_proj"])
        return S, synthetic.sort_tasks(S, *S.all_tasks())
    n = case["heavy"] + case["hydrogen"]
    S = synthetic.config2(seed, n_heavy=case["heavy"], n_h=case["hydrogen"], lmax=case["lmax"], box=6.0 + 0.5 * n)
    if kind == "gradient":
        return S, synthetic.sort_tasks(S, *S.all_tasks())
    if kind == "nuclear":  # point nuclei on every atom
        S.centres = [(S.atoms[i].copy(), 0) for i in range(n)]
        return S, S.all_tasks()
    ns = len(S.shells)
    a, b = (x.ravel() for x in np.meshgrid(np.arange(ns), np.arange(ns), indexing="ij"))
    return S, (a, b, np.zeros(len(a), dtype=np.int32))


def _nuclei(case):
    """Charges and model parameters (rms radii) of the nuclear-attraction case: heavy atoms, then hydrogens."""
    heavy, hydrogen = case.get("heavy", 2), case.get("hydrogen", 1)
    Z, A = np.array([79.0] * heavy + [1.0] * hydrogen), np.array([197] * heavy + [1] * hydrogen)
    rms = (0.836 * A ** (1.0 / 3.0) + 0.570) * 1e-13 / 0.52917721e-8  # Johnson 1985, fm to bohr
    return Z, np.stack([rms, 0 * rms, 0 * rms], axis=1)


def _density(case, n, seed):
    rng = np.random.default_rng(seed + 1000003)
    D = rng.uniform(-1.0, 1.0, (n, n))
    return np.triu(D) + np.triu(D, 1).T if case["symmetric"] else D


def prepare(case, seed):
    lib = engine.load()
    S, (a, b, c) = _system(case, seed)
    st = {"case": case, "lib": lib, "system": S}
    if case["kind"] in ("block", "block_gradient"):
        lib.set_cartesian_order(S.cart_order)
        A, B = S.shells[int(a[0])], S.shells[int(b[0])]
        C, g = S.centres[int(c[0])]
        st.update(hA=lib.new_shell(A), hB=lib.new_shell(B), hg=lib.new_grpp(S.grpps[g]), C=C, D=np.array(A.origin),
                  nA=ncart(A.L), nB=ncart(B.L))
        return st
    batch = S.batch(a, b, c)
    batch.struct
    st["batch"] = batch
    if case["kind"] == "plan":
        st["plan"] = lib.plan(batch, case["mode"])
    elif case["kind"] in ("triatomic", "pair", "scalar", "molecule"):
        # results go to page-locked arrays that the program keeps
        st["out"] = [lib.pinned_empty(int(batch.block_offsets()[-1])) for _ in range(4)]
    elif case["kind"] == "gradient":
        st["D"] = _density(case, S.n_basis(), seed)
    elif case["kind"] in ("nuclear", "finite"):
        st["Z"], st["params"] = _nuclei(case)
    if case.get("mode") == LEARNED:
        lib.ensure_level_model()
    return st


def run(st):
    case, lib = st["case"], st["lib"]
    kind = case["kind"]
    if kind == "block":
        return lib.full(st["hA"], st["hB"], st["hg"], st["C"], st["nA"], st["nB"])
    if kind == "block_gradient":
        return lib.full_gradient(st["hA"], st["hB"], st["hg"], st["C"], st["D"], st["nA"], st["nB"])
    if kind == "plan":
        st["plan"].execute()
        return st["plan"].outputs()
    if kind == "gradient":
        return lib.grad_contract(st["system"], st["batch"], st["D"], case["mode"], symmetric=case["symmetric"])
    if kind == "onee":
        return lib.onee_batch(st["batch"], case["which"])
    if kind in ("nuclear", "finite"):
        return lib.nuclear_attraction_batch(st["batch"], GAUSSIAN if kind == "finite" else POINT, st["Z"], st["params"])
    return lib.full_grpp_batch(st["batch"], case.get("mode", PLAIN), out=st["out"])


# -------------------------------------------------------------------------------------------- work

def _nabc(l):
    return (l + 1) * (l + 2) * (l + 3) // 6


def _entries(L, la, lb):
    """Radial integrals (l1, l2, N) of a projector L that the angular sums of an (la, lb) pair read."""
    s = set()
    for n1 in range(la + 1):
        for n2 in range(lb + 1):
            for l1 in range(L + n1, max(L - n1, 0) - 1, -2):
                for l2 in range(L + n2, max(L - n2, 0) - 1, -2):
                    s.add((l1, l2, n1 + n2))
    return len(s)


def _type1_flops(la, lb, n_pa, n_pb, n_terms):
    """McMurchie-Davidson: per primitive triple the Hermite coefficients, the auxiliary integrals and the contraction."""
    S = la + lb
    e = 3 * (la + 1) * (lb + 1) * (S + 2) / 2
    r = sum((s + 1) * (s + 2) // 2 * (S - s + 1) for s in range(S + 1))
    contract = ncart(la) * ncart(lb) * (S / 3.0 + 1) ** 3
    return n_pa * n_pb * n_terms * (40 + 5 * e + 5 * r + 3 * contract)


def work(case):
    S, (a, b, c) = _system(case, 0)
    kind = case["kind"]
    L = np.array([s.L for s in S.shells])
    nprim = np.array([len(s.alpha) for s in S.shells])
    basis = 8.0 * sum(2 * len(s.alpha) + 3 for s in S.shells)
    pots = 8.0 * sum(2.5 * len(p.alpha) for g in S.grpps for p in [g.UL] + g.arep + g.so + [x for x, _ in g.oc] if p is not None)
    seen, flops, blocks = {}, 0.0, 0.0
    for x, y, z in zip(a, b, c):
        gi = 0 if kind == "onee" else S.centres[int(z)][1]
        key = (int(L[x]), int(L[y]), int(nprim[x]), int(nprim[y]), gi)
        if key not in seen:
            la, lb, na, nb, _ = key
            g = S.grpps[gi]
            n = ncart(la) * ncart(lb)
            if kind == "onee":
                f = na * nb * (9.0 * (la + 3) * (lb + 3) + 9.0 * n)
            elif kind in ("nuclear", "finite"):
                f = _type1_flops(la, lb, na, nb, 1)
            else:
                f = _type1_flops(la, lb, na, nb, len(g.UL.alpha))
                for k, p in enumerate(g.arep + g.so):
                    comp = 1 if k < len(g.arep) else 3
                    # at least two grid levels (63 points), one estimate per primitive triple, the angular sums
                    f += _entries(p.L, la, lb) * 63 * 5.0 + 20.0 * na * nb * len(p.alpha)
                    f += comp * (_nabc(la) * _nabc(lb) * (2 * p.L + 1) * 3.0 + n * _nabc(la))
                for p, s in g.oc:
                    f += 4.0 * 2 * n * (2 * p.L + 1) ** 2
                if kind in ("gradient", "block_gradient"):
                    f *= 4.0  # four differentiated blocks
            seen[key] = (f, float(n))
        f, n = seen[key]
        flops += f
        blocks += n
    if kind == "gradient" and case["symmetric"]:
        flops *= 0.5
    outs = {"onee": 3 if case.get("which") == MOMENTUM else 1, "nuclear": 1, "finite": 1, "gradient": 0, "block_gradient": 12}.get(kind, 4)
    nbytes = basis + pots + 12.0 * len(a) + 8.0 * outs * blocks
    if kind == "gradient":
        nbytes += 8.0 * S.n_basis() ** 2 + 8.0 * 12 * len(S.atoms)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------- exact

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=_device())


def _powers(L):
    return [(r, s, L - r - s) for r in range(L, -1, -1) for s in range(L - r, -1, -1)]  # TURBOMOLE order


def _norm(L, a):
    return (2 * a / math.pi) ** 0.75 * (4 * a) ** (0.5 * L)


def _shell_values(shell, X, deriv=None):
    """Cartesian functions of a contracted shell at the points X [n, 3]: [ncart, n]; with deriv = k the
    derivatives of the functions with respect to component k of the shell's origin."""
    d = X - _t(shell.origin)
    r2 = (d * d).sum(1)
    rad, rad2 = torch.zeros_like(r2), torch.zeros_like(r2)
    for c, al in zip(shell.coeffs, shell.alpha):
        e = c * _norm(shell.L, al) * torch.exp(-al * r2)
        rad += e
        rad2 += 2 * al * e
    out = []
    for p in _powers(shell.L):
        mono = d[:, 0] ** p[0] * d[:, 1] ** p[1] * d[:, 2] ** p[2]
        if deriv is None:
            out.append(mono * rad)
            continue
        v = mono * d[:, deriv] * rad2
        if p[deriv] > 0:
            q = list(p)
            q[deriv] -= 1
            v = v - p[deriv] * d[:, 0] ** q[0] * d[:, 1] ** q[1] * d[:, 2] ** q[2] * rad
        out.append(v)
    return torch.stack(out)


def _harmonics(lmax, u):
    """Real spherical harmonics S_lm (m = -l..l) at the unit vectors u [n, 3]: list over l of [2l+1, n]."""
    x, y, z = u[:, 0], u[:, 1], u[:, 2]
    # Q_lm = P_lm / sin^m with the sectoral factors as polynomials in x, y
    cs, sn = [torch.ones_like(x)], [torch.zeros_like(x)]
    for m in range(1, lmax + 1):
        cs.append(x * cs[-1] - y * sn[-1])
        sn.append(x * sn[m - 1] + y * cs[m - 1])
    out = [[None] * (2 * l + 1) for l in range(lmax + 1)]
    for m in range(lmax + 1):
        q0, q1 = None, torch.full_like(x, float(math.prod(range(1, 2 * m, 2))))
        for l in range(m, lmax + 1):
            if l > m:
                q0, q1 = q1, ((2 * l - 1) * z * q1 - (l + m - 1) * (q0 if q0 is not None else 0.0)) / (l - m)
            f = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                out[l][l] = f * q1
            else:
                out[l][l + m] = math.sqrt(2.0) * f * q1 * cs[m]
                out[l][l - m] = math.sqrt(2.0) * f * q1 * sn[m]
    return [torch.stack(v) for v in out]


def _l_matrices(l):
    """The real matrices -i <S_lm| l_k |S_lm'> of the angular momentum l, k = x, y, z."""
    n = 2 * l + 1
    lp = np.zeros((n, n), dtype=complex)  # l_+ in the complex harmonics, without the Condon-Shortley sign
    for m in range(-l, l):
        lp[m + 1 + l, m + l] = math.sqrt(l * (l + 1) - m * (m + 1))
    lz = np.diag(np.arange(-l, l + 1)).astype(complex)
    lx, ly = (lp + lp.conj().T) / 2, (lp - lp.conj().T) / 2j
    U = np.zeros((n, n), dtype=complex)  # rows: real harmonics in terms of the complex ones (Condon-Shortley)
    U[l, l] = 1
    for m in range(1, l + 1):
        s = 1 / math.sqrt(2)
        U[l + m, l + m], U[l + m, l - m] = (-1) ** m * s, s
        U[l - m, l + m], U[l - m, l - m] = -1j * (-1) ** m * s, 1j * s
    return [_t((U.conj() @ k @ U.T).imag) for k in (lx, ly, lz)]


def _pot_value(p, r):
    v = torch.zeros_like(r)
    for n, c, z in zip(p.powers, p.coeffs, p.alpha):
        v = v + c * r ** (int(n) - 2) * torch.exp(-z * r * r)
    return v


def _gl(n, lo, hi):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (hi - lo) * x + 0.5 * (hi + lo), 0.5 * (hi - lo) * w


def _grpp_blocks(g, C, bras, kets, pairs):
    """The four full-GRPP blocks of <bras[i]| U(C) |kets[j]> for the pairs (i, j), by quadrature. A
    function list holds callables X -> [ncart, n]; each has attributes of its shell in .shell."""
    dmax = max(float(np.linalg.norm(f.shell.origin - C)) for f in bras + kets)
    amax = 2 * max(float(np.max(f.shell.alpha)) for f in bras + kets)
    edges = np.concatenate([np.arange(0, 5, 0.25), np.arange(5, 25)])
    lmax = max([p.L for p in g.arep + g.so] + [p.L for p, _ in g.oc] + [0])
    Cg = _t(C)
    nb, nk = len(bras), len(kets)
    loc = [[0.0] * nk for _ in range(nb)]
    sl = [[[0.0] * nk for _ in range(nb)] for _ in range(4)]
    lm = {l: _l_matrices(l) for l in range(1, lmax + 1)}
    # outercore functions: radial part with the solid-harmonic normalisation, times S_lm
    an = [math.sqrt(math.prod(range(1, 2 * s.L + 2, 2))) / (2 * math.sqrt(math.pi)) for _, s in g.oc]

    def oc_radial(k, r):
        s = g.oc[k][1]
        return sum(c * _norm(s.L, al) / an[k] * torch.exp(-al * r * r) for c, al in zip(s.coeffs, s.alpha)) * r ** s.L

    So = {(s, k): [0.0] * n for s, n in (("b", nb), ("k", nk)) for k in range(len(g.oc))}
    Uo = {key: list(v) for key, v in So.items()}
    delta = np.zeros((len(g.oc), len(g.oc)))
    for lo, hi in zip(edges[:-1], edges[1:]):
        r, w = (_t(v) for v in _gl(20, lo, hi))
        # angular resolution: the narrowest product of two Gaussians still alive in this panel
        a = amax if lo <= dmax + 0.5 else min(amax, 90.0 / (lo - dmax) ** 2)
        nth = int(5.0 * math.sqrt(2 * a * dmax * hi) + 2 * lmax + 20)
        ct, wt = _gl(nth, -1, 1)
        ph = 2 * math.pi * np.arange(2 * nth) / (2 * nth)
        stt = np.sqrt(1 - ct ** 2)
        u = _t(np.stack([np.outer(stt, np.cos(ph)), np.outer(stt, np.sin(ph)), np.outer(ct, np.ones(2 * nth))], -1).reshape(-1, 3))
        wo = _t(np.repeat(wt, 2 * nth) * math.pi / nth)
        S = _harmonics(lmax, u)
        X = (Cg + r[:, None, None] * u).reshape(-1, 3)
        n = (len(r), len(wo))
        fb, fk = [f(X).reshape(-1, *n) for f in bras], [f(X).reshape(-1, *n) for f in kets]
        wr = w * r * r
        if g.UL is not None:
            ul = (wr * _pot_value(g.UL, r))[:, None] * wo
            wk = [(f * ul).flatten(1) for f in fk]
            for i, j in pairs:
                loc[i][j] = loc[i][j] + fb[i].flatten(1) @ wk[j].T
        # projections [component, r, m]
        P = [{l: (f * wo) @ S[l].T for l in range(lmax + 1)} for f in fb]
        R = [{l: (f * wo) @ S[l].T for l in range(lmax + 1)} for f in fk]
        for p in g.arep:
            v = (wr * _pot_value(p, r))[:, None]
            for i, j in pairs:
                sl[0][i][j] = sl[0][i][j] + P[i][p.L].flatten(1) @ (v * R[j][p.L]).flatten(1).T
        for p in g.so:
            v = (wr * _pot_value(p, r) * 2.0 / (2 * p.L + 1))[:, None]
            for k in range(3):
                for i, j in pairs:
                    sl[k + 1][i][j] = sl[k + 1][i][j] + (P[i][p.L] @ lm[p.L][k]).flatten(1) @ (v * R[j][p.L]).flatten(1).T
        for k, (p, s) in enumerate(g.oc):
            rad = wr * oc_radial(k, r)
            ur = rad * _pot_value(p, r)
            for side, V in (("b", P), ("k", R)):
                for i in range(len(V)):
                    So[side, k][i] = So[side, k][i] + torch.einsum("crm,r->cm", V[i][p.L], rad)
                    Uo[side, k][i] = Uo[side, k][i] + torch.einsum("crm,r->cm", V[i][p.L], ur)
            for k2, (p2, s2) in enumerate(g.oc):
                if (p.L, p.J) == (p2.L, p2.J):
                    delta[k, k2] += float((rad * oc_radial(k2, r) * 0.5 * (_pot_value(p, r) + _pot_value(p2, r))).sum())
    out = []
    for i, j in pairs:
        blk = [loc[i][j] + sl[0][i][j]] + [sl[m][i][j] for m in (1, 2, 3)]
        like = bras[i].shell, kets[j].shell
        z = torch.zeros(ncart(like[0].L), ncart(like[1].L), dtype=torch.float64, device=_device())
        blk = [z + x for x in blk]
        for k, (p, s) in enumerate(g.oc):
            low = p.J < 2 * p.L
            fa = (p.L if low else p.L + 1) / (2 * p.L + 1)
            fs = (-2.0 if low else 2.0) / (2 * p.L + 1)
            blk[0] = blk[0] + fa * (So["b", k][i] @ Uo["k", k][j].T + Uo["b", k][i] @ So["k", k][j].T)
            for m in range(3):
                if p.L > 0:
                    blk[m + 1] = blk[m + 1] + fs * (So["b", k][i] @ lm[p.L][m] @ Uo["k", k][j].T + Uo["b", k][i] @ lm[p.L][m] @ So["k", k][j].T)
            for k2, (p2, s2) in enumerate(g.oc):
                if (p.L, p.J) != (p2.L, p2.J):
                    continue
                blk[0] = blk[0] - delta[k, k2] * fa * (So["b", k][i] @ So["k", k2][j].T)
                for m in range(3):
                    if p.L > 0:
                        blk[m + 1] = blk[m + 1] - delta[k, k2] * fs * (So["b", k][i] @ lm[p.L][m] @ So["k", k2][j].T)
        out.append(blk)
    return out


class _Function:
    def __init__(self, shell, deriv=None):
        self.shell, self.deriv = shell, deriv

    def __call__(self, X):
        return _shell_values(self.shell, X, self.deriv)


def _exact_blocks(case, seed):
    S, (a, b, c) = _system(case, seed)
    outs = [[None] * len(a) for _ in range(4)]
    for ic in sorted(set(c.tolist())):
        t = [k for k in range(len(a)) if c[k] == ic]
        bra, ket = sorted(set(a[t].tolist())), sorted(set(b[t].tolist()))
        C, gi = S.centres[ic]
        blocks = _grpp_blocks(S.grpps[gi], np.asarray(C), [_Function(S.shells[i]) for i in bra], [_Function(S.shells[j]) for j in ket],
                              [(bra.index(a[k]), ket.index(b[k])) for k in t])
        for k, blk in zip(t, blocks):
            for m in range(4):
                outs[m][k] = blk[m].cpu().numpy()
    if case["kind"] == "block":
        return [o[0] for o in outs]
    return [np.concatenate([x.ravel() for x in o]) for o in outs]


def _exact_block_gradient(case, seed):
    """Derivatives with respect to the bra atom's position of a block whose ket and centre lie elsewhere,
    or, where the centre lies on the bra atom, of the ket function (the block depends on the distance)."""
    S, (a, b, c) = _system(case, seed)
    A, B = S.shells[int(a[0])], S.shells[int(b[0])]
    C, gi = S.centres[int(c[0])]
    C = np.asarray(C)
    out = np.zeros((4, 3, ncart(A.L), ncart(B.L)))
    on_bra, on_ket = np.allclose(A.origin, C), np.allclose(B.origin, C)
    for k in range(3):
        # moving A alone; with the centre on A, translation invariance makes it minus the ket derivative
        bra = _Function(A, None if on_bra else k)
        ket = _Function(B, k if on_bra else None)
        blk = _grpp_blocks(S.grpps[gi], C, [bra], [ket], [(0, 0)])[0]
        for m in range(4):
            out[m, k] = (-1.0 if on_bra else 1.0) * blk[m].cpu().numpy()
    assert not (on_bra and on_ket)
    return out


def _axis_tables(a, b, A, B, la, lb, u2, Cx):
    """int (x-A)^i (x-B)^j exp(-a (x-A)^2 - b (x-B)^2 - u2 (x-C)^2) dx for i <= la, j <= lb, by Gauss-Hermite:
    shape of the broadcast arguments plus [la+1, lb+1]."""
    n = (la + lb) // 2 + 1
    xs, ws = (_t(v) for v in np.polynomial.hermite.hermgauss(n))
    q = a + b + u2
    Q = (a * A + b * B + u2 * Cx) / q
    K = torch.exp(-(a * b * (A - B) ** 2 + a * u2 * (A - Cx) ** 2 + b * u2 * (B - Cx) ** 2) / q) / torch.sqrt(q)
    x = Q[..., None] + xs / torch.sqrt(q)[..., None]
    pa = torch.stack([(x - A[..., None]) ** i for i in range(la + 1)], -2)
    pb = torch.stack([(x - B[..., None]) ** j for j in range(lb + 1)], -2)
    return K[..., None, None] * torch.einsum("...ik,...jk,k->...ij", pa, pb, ws)


def _by_class(S, a, b):
    L = np.array([s.L for s in S.shells])
    for la in range(int(L.max()) + 1):
        for lb in range(int(L.max()) + 1):
            t = np.where((L[a] == la) & (L[b] == lb))[0]
            for k in range(0, len(t), 2048):
                yield la, lb, t[k:k + 2048]


def _primitives(S, idx, l):
    al = _t(np.stack([S.shells[i].alpha for i in idx]))
    co = _t(np.stack([S.shells[i].coeffs * _norm(l, S.shells[i].alpha) for i in idx]))
    return al, co, _t(np.stack([S.shells[i].origin for i in idx]))


def _block_slices(S, a, b):
    n = np.array([ncart(s.L) for s in S.shells])
    return np.concatenate([[0], np.cumsum(n[a] * n[b])])


def _exact_onee(case, seed):
    S, (a, b, _) = _system(case, seed)
    off = _block_slices(S, a, b)
    outs = [np.zeros(off[-1]) for _ in range(3 if case["which"] == MOMENTUM else 1)]
    for la, lb, t in _by_class(S, a, b):
        if len(t) == 0:
            continue
        aa, ca, A = _primitives(S, a[t], la)
        ab, cb, B = _primitives(S, b[t], lb)
        al, be = aa[:, :, None] + 0 * ab[:, None, :], ab[:, None, :] + 0 * aa[:, :, None]
        cc = ca[:, :, None] * cb[:, None, :]
        z = torch.zeros_like(al)
        T = [_axis_tables(al, be, A[:, d, None, None] + z, B[:, d, None, None] + z, la, lb + 2, z, z) for d in range(3)]
        e = be[..., None]
        # ket derivatives: d/dx x^j e^(-b x^2) = j x^(j-1) - 2b x^(j+1), and twice
        D1 = [torch.stack([(j * t_[..., j - 1] if j else 0) - 2 * e * t_[..., j + 1] for j in range(lb + 1)], -1) for t_ in T]
        D2 = [torch.stack([(j * (j - 1) * t_[..., j - 2] if j > 1 else 0) - 2 * e * (2 * j + 1) * t_[..., j] + 4 * e * e * t_[..., j + 2]
                           for j in range(lb + 1)], -1) for t_ in T]
        for i, p in enumerate(_powers(la)):
            for j, q in enumerate(_powers(lb)):
                s, f, g = ([v[d][..., p[d], q[d]] for d in range(3)] for v in (T, D1, D2))
                if case["which"] == OVERLAP:
                    vals = [s[0] * s[1] * s[2]]
                elif case["which"] == KINETIC:
                    vals = [-0.5 * (g[0] * s[1] * s[2] + s[0] * g[1] * s[2] + s[0] * s[1] * g[2])]
                else:  # momentum without the factor i: minus the derivative of the ket
                    vals = [-f[0] * s[1] * s[2], -s[0] * f[1] * s[2], -s[0] * s[1] * f[2]]
                for o, v in zip(outs, vals):
                    o[off[t] + i * ncart(lb) + j] = (cc * v).sum((1, 2)).cpu().numpy()
    return outs


def _exact_nuclear(case, seed):
    """-Z erf(sqrt(xi) r)/r (r -> point: 1/r) as an integral over Gaussians u^2 = p t^2/(1-t^2)."""
    S, (a, b, c) = _system(case, seed)
    if len(a) > 4000:
        return None
    Z, prm = _nuclei(case)
    xi = 3.0 / (2.0 * prm[:, 0] ** 2)
    off = _block_slices(S, a, b)
    out = np.zeros(off[-1])
    gx, gw = (_t(v) for v in _gl(40, 0.0, 1.0))
    cen = np.stack([np.asarray(o) for o, _ in S.centres])
    for la, lb, t0 in _by_class(S, a, b):
        for k0 in range(0, len(t0), 64):
            t = t0[k0:k0 + 64]
            aa, ca, A = _primitives(S, a[t], la)
            ab, cb, B = _primitives(S, b[t], lb)
            C, q = _t(cen[c[t]]), _t(Z[c[t]])
            al, be = (aa[:, :, None] + 0 * ab[:, None, :])[..., None], (ab[:, None, :] + 0 * aa[:, :, None])[..., None]
            p = al + be
            P = [(al * A[:, d, None, None, None] + be * B[:, d, None, None, None]) / p for d in range(3)]
            T = p * sum((P[d] - C[:, d, None, None, None]) ** 2 for d in range(3))
            top = torch.ones_like(p)
            if case["kind"] == "finite":
                x = _t(xi[c[t]])[:, None, None, None]
                top = torch.sqrt(x / (p + x))
            # exp(-T t^2) is gone beyond t = 7 / sqrt(T); panels of two lengths
            cut = torch.minimum(top, 7.0 / torch.sqrt(T + 1e-300))
            acc = 0.0
            for lo, hi in ((0 * cut, 0.5 * cut), (0.5 * cut, cut)):
                tt, wt = lo + (hi - lo) * gx, (hi - lo) * gw
                u2 = p * tt ** 2 / (1 - tt ** 2)
                z = torch.zeros_like(u2)
                ax = [_axis_tables(al + z, be + z, A[:, d, None, None, None] + z, B[:, d, None, None, None] + z, la, lb, u2,
                                   C[:, d, None, None, None] + z) for d in range(3)]
                # du = sqrt(p) (1 - t^2)^(-3/2) dt
                f = (ca[:, :, None] * cb[:, None, :])[..., None] * wt * 2 / math.sqrt(math.pi) * torch.sqrt(p) * (1 - tt ** 2) ** -1.5
                blk = [[(f * ax[0][..., x_[0], y_[0]] * ax[1][..., x_[1], y_[1]] * ax[2][..., x_[2], y_[2]]).sum((1, 2, 3))
                        for y_ in _powers(lb)] for x_ in _powers(la)]
                acc = acc + torch.stack([torch.stack(row, -1) for row in blk], -2)
            out[(off[t][:, None] + np.arange(ncart(la) * ncart(lb))).ravel()] = (-q[:, None, None] * acc).reshape(-1).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("block", "triatomic", "pair"):
        return _exact_blocks(case, seed)
    if kind == "block_gradient":
        return _exact_block_gradient(case, seed)
    if kind == "onee":
        return _exact_onee(case, seed)
    if kind in ("nuclear", "finite"):
        return _exact_nuclear(case, seed)
    return None
