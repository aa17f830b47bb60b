"""The work a user of this package has it do, as cases that can be timed and compared.

Every case goes through the public entry points of ``forte2_gb300``: sigma = H C on determinant
vectors (device tensors and host arrays), the CSF-space sigma of a Davidson block in both
precisions, a point-group-blocked space, the 1-/2-body and 3-body density matrices, the
two-component builder and a whole CASCI solve. Active spaces run from (6e,6o), the bulk of a
stream of small solves, to the headline (16e,16o); inputs are synthetic integrals of the
package's benchmark recipe and CI-like vectors (one dominant region, a tail over many decades).
"""

import itertools
import math

import numpy as np
import torch

from forte2_gb300.ci import CASCISolver
from forte2_gb300.ci_helpers import CISigmaBuilder, CISpinAdapter, CIStrings, RelCISigmaBuilder
from forte2_gb300.params import CIParams, DavidsonLiuParams

DEV = "cuda"


def listed():
    return [
        # one vector of the smallest common active space: launch latency is all there is
        {"name": "sigma_cas6", "kind": "sigma", "n": 6, "na": 3, "nb": 3},
        # an odd, open-shell space with unequal spins (ragged tiles everywhere)
        {"name": "sigma_11e13o", "kind": "sigma", "n": 13, "na": 6, "nb": 5},
        # the headline: one FP64 sigma build at CAS(16e,16o), 165.6 M determinants
        {"name": "sigma_cas16", "kind": "sigma", "n": 16, "na": 8, "nb": 8},
        # the drop-in convention: numpy vectors in and out, copies included
        {"name": "host_cas12", "kind": "host", "n": 12, "na": 6, "nb": 6},
        # a Davidson block of four CSF vectors of a small space (FP64 closure csf-det-H-det-csf)
        {"name": "closure_cas10", "kind": "closure", "n": 10, "na": 5, "nb": 5, "rows": 4, "precision": "fp64"},
        # three roots' block at CAS(14e,14o), FP64 (the default precision of a CASCI solve)
        {"name": "closure_cas14", "kind": "closure", "n": 14, "na": 7, "nb": 7, "rows": 3, "precision": "fp64"},
        # the same block in the mixed mode's FP32 iterations (tensor-core opposite spin)
        {"name": "closure32_cas14", "kind": "closure", "n": 14, "na": 7, "nb": 7, "rows": 3, "precision": "fp32"},
        # a D2h molecule: determinants of one irrep
        {"name": "blocked_cas14", "kind": "blocked", "n": 14, "na": 7, "nb": 7, "nirrep": 8},
        # spin-free 1- and 2-RDM of one root (orbital gradients, properties)
        {"name": "rdm12_cas14", "kind": "rdm12", "n": 14, "na": 7, "nb": 7},
        # spin-free 3-RDM (multireference perturbation theory)
        {"name": "rdm3_cas10", "kind": "rdm3", "n": 10, "na": 5, "nb": 5},
        # two-component sigma over spinors
        {"name": "rel_8e18s", "kind": "rel", "n": 18, "na": 8, "nb": 0},
        # a whole CASCI solve on a kept solver with new integrals, as a solve stream runs it
        {"name": "solve_cas8", "kind": "solve", "n": 8, "na": 4, "nb": 4, "roots": 2},
    ]


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "host", "closure", "closure", "closure32", "blocked", "rdm12", "rdm3",
                       "rel", "solve"])
    lo, hi = {"sigma": (6, 16), "host": (6, 14), "closure": (6, 14), "closure32": (10, 15), "blocked": (8, 15),
              "rdm12": (6, 14), "rdm3": (6, 10), "rel": (10, 18), "solve": (6, 8)}[kind]
    n = rng.randint(lo, hi)  # the space grows exponentially with n: uniform in n is uniform in the logarithm
    if kind == "rel":
        return {"kind": kind, "n": n, "na": rng.randint(3, n // 2), "nb": 0}
    na = n // 2 + rng.choice([0, 0, 0, -1, -2, 1 if n % 2 else 0])
    nb = max(1, na - rng.choice([0, 0, 0, 1, 2]))
    case = {"kind": kind, "n": n, "na": na, "nb": nb}
    if kind in ("closure", "closure32"):
        case["kind"] = "closure"
        case["precision"] = "fp32" if kind == "closure32" else "fp64"
        case["rows"] = rng.randint(1, 4 if n <= 12 else 3)
    elif kind == "blocked":
        case["nirrep"] = rng.choice([2, 4, 8])
    elif kind == "solve":
        case["na"] = case["nb"] = na = n // 2
        case["roots"] = rng.randint(1, 3)
    return case


# ---- inputs ------------------------------------------------------------------------------------

def _integrals(n, seed):
    """Orbital energies with small off-diagonals, and (pq|rs) = sum_Q B_Q,pq B_Q,rs over 4n Gaussian
    symmetric B_Q: h and the physicist V[p,q,r,s] = (pr|qs)."""
    r = np.random.default_rng(seed)
    h = np.diag(np.sort(r.uniform(-2.0, 1.0, n)))
    iu = np.triu_indices(n, 1)
    h[iu] = r.normal(0.0, 0.05, len(iu[0]))
    h = np.triu(h) + np.triu(h, 1).T
    B = r.normal(0.0, 0.1, (4 * n, n, n))
    B = (np.triu(B) + np.transpose(np.triu(B, 1), (0, 2, 1))).reshape(4 * n, n * n)
    eri = (B.T @ B).reshape(n, n, n, n)
    return np.ascontiguousarray(h), np.ascontiguousarray(eri.transpose(0, 2, 1, 3))


def _spinor_integrals(n, seed):
    r = np.random.default_rng(seed)
    a = r.normal(0.0, 0.05, (n, n)) + 1j * r.normal(0.0, 0.05, (n, n))
    h = np.diag(np.sort(r.uniform(-2.0, 1.0, n))).astype(complex) + np.triu(a, 1) + np.triu(a, 1).conj().T
    L = r.normal(0.0, 0.1, (3 * n, n, n)) + 1j * r.normal(0.0, 0.1, (3 * n, n, n))
    L = (0.5 * (L + np.conj(np.transpose(L, (0, 2, 1))))).reshape(3 * n, n * n)
    return np.ascontiguousarray(h), np.ascontiguousarray((L.T @ L).reshape(n, n, n, n).transpose(0, 2, 1, 3))


def _symmetrized(h, V, irreps):
    g = np.asarray(irreps)
    x = g[:, None] ^ g[None, :]
    return np.where(x == 0, h, 0.0), np.where((x[:, :, None, None] ^ x[None, None, :, :]) == 0, V, 0.0)


def _masks(n, k):
    """Occupation masks of k electrons in n orbitals, ordered as sequences (b0, b1, ...) with 0 < 1."""
    if k < 0 or k > n:
        return np.zeros(0, np.int64)
    m = np.array([sum(1 << p for p in c) for c in itertools.combinations(range(n), k)], np.int64)
    key = sum(((m >> p) & 1) << (n - 1 - p) for p in range(n)) if n else m
    return m[np.argsort(key)]


def _bits(m, n):
    return ((np.asarray(m)[:, None] >> np.arange(n)) & 1).astype(np.float64)


def _decay(n, k, h):
    """CI coefficients fall with the orbital energies of the excitation."""
    e = _bits(_masks(n, k), n) @ np.diag(h).real
    return torch.as_tensor(np.exp(-0.7 * (e - e.min())), device=DEV)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 1)
    return g


def _ci_vector(n, na, nb, h, seed):
    wa, wb = _decay(n, na, h), _decay(n, nb, h)
    c = torch.randn(len(wa), len(wb), generator=_gen(seed), dtype=torch.float64, device=DEV)
    c.mul_(wa[:, None]).mul_(wb[None, :])
    return c.div_(torch.linalg.vector_norm(c)).reshape(-1)


def _csf_rows(rows, ncsf, seed):
    """Trial rows whose elements span four decades."""
    g = _gen(seed)
    x = torch.randn(rows, ncsf, generator=g, dtype=torch.float64, device=DEV)
    x *= 10.0 ** (-4.0 * torch.rand(rows, ncsf, generator=g, dtype=torch.float64, device=DEV))
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True)


def _irreps(case):
    return [(3 * p) % case["nirrep"] for p in range(case["n"])]  # every irrep occurs from 8 orbitals on


def _spaces(case):
    n, na, nb = case["n"], case["na"], case["nb"]
    return n, na, nb, math.comb(n, na), math.comb(n, nb)


def _blocked_positions(case):
    """C1 address of every determinant of the totally symmetric irrep: blocks by alpha irrep, alpha
    strings slowest, strings of one irrep in address order."""
    n, na, nb, _, n0b = _spaces(case)
    g = np.array(_irreps(case))

    def irrep(m):
        x = np.zeros(len(m), np.int64)
        for p in range(n):
            x ^= np.where((m >> p) & 1, g[p], 0)
        return x

    xa, xb = irrep(_masks(n, na)), irrep(_masks(n, nb))
    out = []
    for r in range(case["nirrep"]):
        ia, ib = np.nonzero(xa == r)[0], np.nonzero(xb == r)[0]
        out.append((ia[:, None] * n0b + ib[None, :]).reshape(-1))
    return torch.as_tensor(np.concatenate(out), device=DEV)


# ---- the cases -----------------------------------------------------------------------------------

def prepare(case, seed):
    kind, (n, na, nb, _, _) = case["kind"], _spaces(case)
    if kind == "rel":
        h, V = _spinor_integrals(n, seed)
        strings = CIStrings(na, 0, 0, [[0] * n], [], [])
        sb = RelCISigmaBuilder(strings, 0.25, h, V, 0)
        sb.set_algorithm("hz")
        w = _decay(n, na, h)
        g = _gen(seed)
        re, im = (torch.randn(len(w), generator=g, dtype=torch.float64, device=DEV) for _ in range(2))
        c = torch.complex(re * w, im * w)
        return {"kind": kind, "sb": sb, "C": c / torch.linalg.vector_norm(c), "S": torch.empty_like(c)}
    h, V = _integrals(n, seed)
    if kind == "solve":
        solver = CASCISolver(norb=n, na=na, nb=nb, multiplicity=1, nroot=case["roots"], E=0.0, H=h, V=V,
                             ci_params=CIParams(ci_algorithm="hz"),
                             davidson_liu_params=DavidsonLiuParams(e_tol=1e-10, maxiter=1000))
        # a kept solver: its space and buffers exist, the integrals of a pass are new to it
        solver.run()
        h, V = _integrals(n, seed + 1000003)
        return {"kind": kind, "solver": solver, "H": h, "V": V}
    irreps = [0] * n
    if kind == "blocked":
        irreps = _irreps(case)
        h, V = _symmetrized(h, V, irreps)
    strings = CIStrings(na, nb, 0, [irreps], [], [])
    sb = CISigmaBuilder(strings, 0.0, h, V, 0)
    sb.set_algorithm("hz")
    s = {"kind": kind, "strings": strings, "sb": sb}
    if kind == "closure":
        sa = CISpinAdapter(na - nb, na - nb, n)
        sa.prepare_couplings(strings.make_determinants())
        sb.set_precision(case["precision"])
        s |= {"sa": sa, "C": _csf_rows(case["rows"], sa.ncsf, seed)}
        s["S"] = torch.empty_like(s["C"])
        return s
    c = _ci_vector(n, na, nb, h, seed)
    if kind == "blocked":
        c = c[_blocked_positions(case)]
        c = c / torch.linalg.vector_norm(c)
    if kind == "host":
        s["C"] = c.cpu().numpy()
        s["S"] = np.zeros_like(s["C"])
    else:
        s["C"] = c
        if kind in ("sigma", "blocked"):
            s["S"] = torch.empty_like(c)
    return s


def run(state):
    kind = state["kind"]
    if kind in ("sigma", "host", "blocked", "rel"):
        state["sb"].Hamiltonian(state["C"], state["S"])
        return state["S"]
    if kind == "closure":
        state["sb"].apply_csf(state["sa"], state["C"], state["S"])
        return state["S"]
    if kind == "rdm12":
        return {"g1": state["sb"].sf_1rdm(state["C"], state["C"]), "g2": state["sb"].sf_2rdm(state["C"], state["C"])}
    if kind == "rdm3":
        return state["sb"].sf_3rdm(state["C"], state["C"])
    solver = state["solver"]
    solver.new_problem(0.0, state["H"], state["V"])
    solver.run()
    return {"evals": np.asarray(solver.evals), "evecs": solver.evecs}


def _ss_flops(n, k, cols):
    """Same-spin term: per two-hole string a C(n-k+2, 2) square block, or the sparse rows if fewer."""
    if k < 1:
        return 0
    nnz = k * (n - k) + math.comb(k, 2) * math.comb(n - k, 2)
    sparse = 2 * math.comb(n, k) * nnz
    pairs = 2 * math.comb(n, k - 2) * math.comb(n - k + 2, 2) ** 2 if k >= 2 else sparse
    return cols * min(sparse, pairs)


def _ab_flops(n, na, nb):
    return 2 * math.comb(n, na - 1) * math.comb(n, nb - 1) * ((n - na + 1) * (n - nb + 1)) ** 2


def work(case):
    kind, (n, na, nb, n0a, n0b) = case["kind"], _spaces(case)
    nd = n0a * n0b
    sigma = _ab_flops(n, na, nb) + _ss_flops(n, na, n0b) + _ss_flops(n, nb, n0a) if nb else 0
    if kind in ("sigma", "host"):
        return {"bytes": 16 * nd, "flops": sigma}
    if kind == "blocked":
        k = case["nirrep"]
        return {"bytes": 16 * nd // k, "flops": sigma // (k * k)}
    if kind == "closure":
        s2 = na - nb  # CSFs of the highest Ms: C(n+1, na+1) C(n+1, nb) (2S+1) / (n+1)
        ncsf = math.comb(n + 1, na + 1) * math.comb(n + 1, nb) * (s2 + 1) // (n + 1)
        return {"bytes": 16 * ncsf * case["rows"], "flops": sigma * case["rows"]}
    if kind == "rdm12":
        ss = sum(math.comb(n, k - 2) * math.comb(n - k + 2, 2) ** 2 * c for k, c in ((na, n0b), (nb, n0a)) if k >= 2)
        return {"bytes": 8 * nd + 8 * n ** 4 + 8 * n * n, "flops": _ab_flops(n, na, nb) // 2 + ss}
    if kind == "rdm3":
        f = 0
        for k, kk, c in ((na, nb, n0b), (nb, na, n0a)):
            if k >= 3:
                f += math.comb(n, k - 3) * math.comb(n - k + 3, 3) ** 2 * c
            if k >= 2 and kk >= 1:
                f += math.comb(n, k - 2) * math.comb(n, kk - 1) * (math.comb(n - k + 2, 2) * (n - kk + 1)) ** 2
        return {"bytes": 8 * nd + 8 * n ** 6, "flops": f}
    if kind == "rel":
        return {"bytes": 32 * n0a, "flops": 4 * _ss_flops(n, na, 1)}
    # a solve: about twelve sigma builds a root in this space (its integrals in, vectors out)
    return {"bytes": 8 * n ** 4 + 16 * nd * case["roots"], "flops": 12 * case["roots"] * sigma}


# ---- what the outputs are, in 64 bits, from torch and numpy alone ---------------------------------

def _parity(m, p):
    """(-1)^(occupied orbitals of m below p)."""
    x = np.asarray(m) & ((1 << np.asarray(p)) - 1)
    x = x ^ (x >> 32)
    for s in (16, 8, 4, 2, 1):
        x = x ^ (x >> s)
    return 1.0 - 2.0 * (x & 1)


def _holes(n, k, nh):
    """For each string K of k - nh electrons: the created orbitals (descending), the address of the
    filled string and the sign of <K| a_p a_q ... |I> (last operator first), as (N, m) arrays."""
    full = _masks(n, k)
    at = np.zeros(1 << n, np.int64)
    at[full] = np.arange(len(full))
    K = _masks(n, k - nh)
    combos = np.array(list(itertools.combinations(range(n - 1, -1, -1), nh)), np.int64)
    ok = np.stack([(K & sum(1 << int(p) for p in c)) == 0 for c in combos], 1)
    m = math.comb(n - k + nh, nh)
    col = np.nonzero(ok)[1].reshape(len(K), m)
    orbs = combos[col]  # (N, m, nh)
    I = K[:, None] | (1 << orbs).sum(-1)
    sign, cur = np.ones(I.shape), I.copy()
    for j in range(nh - 1, -1, -1):
        sign *= _parity(cur, orbs[:, :, j])
        cur = cur & ~(1 << orbs[:, :, j])
    t = lambda x: torch.as_tensor(x, device=DEV)  # noqa: E731
    return t(orbs), t(at[I]), t(sign)


def _same_spin(n, k, h, V, C):
    """(H1 + H2 of one spin) C on the first index of C."""
    S = torch.zeros_like(C)
    if k >= 1:
        o, I, s = _holes(n, k, 1)
        A = h[o[:, :, None, 0], o[:, None, :, 0]] * (s[:, :, None] * s[:, None, :]).to(h.dtype)
        _pairs(A, I, C, S)
    if k >= 2:
        o, I, s = _holes(n, k, 2)
        p, r = o[:, :, None, 0], o[:, :, None, 1]
        q, t = o[:, None, :, 0], o[:, None, :, 1]
        _pairs((V[p, r, q, t] - V[p, r, t, q]) * (s[:, :, None] * s[:, None, :]).to(V.dtype), I, C, S)
    return S


def _pairs(A, I, C, S):
    cols = C.shape[1]
    step = max(1, int(2e8) // max(1, I.shape[1] * cols))
    for a in range(0, len(I), step):
        i = I[a:a + step]
        E = torch.bmm(A[a:a + step], C[i.reshape(-1)].reshape(*i.shape, cols))
        S.index_add_(0, i.reshape(-1), E.reshape(-1, cols))


def _opposite_blocks(n, na, nb, C):
    """Chunks (alpha 1-hole strings, D) with D[Ka, Kb, q * n + s] = <Ka Kb| a_q a_s |C>."""
    (oa, Ia, sa), (ob, Ib, sb) = _holes(n, na, 1), _holes(n, nb, 1)
    step = max(1, int(3e8) // max(1, len(Ib) * n * n))
    kb = torch.arange(len(Ib), device=DEV)
    for a in range(0, len(Ia), step):
        i = Ia[a:a + step]
        D = torch.zeros(len(i), len(Ib), n, n, dtype=C.dtype, device=DEV)
        for j in range(i.shape[1]):
            rows = C[i[:, j]] * sa[a:a + step, j, None]
            for t in range(Ib.shape[1]):
                D[torch.arange(len(i), device=DEV)[:, None], kb[None, :], oa[a:a + step, j, 0][:, None],
                  ob[:, t, 0][None, :]] = rows[:, Ib[:, t]] * sb[:, t]
        yield slice(a, a + step), D.reshape(len(i), len(Ib), n * n)


def _sigma(n, na, nb, h, V, C, Vab=None):
    """H C for a determinant matrix C (alpha strings x beta strings)."""
    S = _same_spin(n, na, h, V, C) + _same_spin(n, nb, h, V, C.T.contiguous()).T
    S = S.contiguous()
    if na < 1 or nb < 1:
        return S
    W = (V if Vab is None else Vab).permute(2, 3, 0, 1).reshape(n * n, n * n)  # [(q s)][(p r)]
    (oa, Ia, sa), (ob, Ib, sb) = _holes(n, na, 1), _holes(n, nb, 1)
    for sl, D in _opposite_blocks(n, na, nb, C):
        E = (D @ W).reshape(D.shape[0], D.shape[1], n, n)
        ia = torch.arange(D.shape[0], device=DEV)[:, None]
        kb = torch.arange(D.shape[1], device=DEV)[None, :]
        for j in range(Ia.shape[1]):
            for t in range(Ib.shape[1]):
                e = E[ia, kb, oa[sl][:, j, 0][:, None], ob[:, t, 0][None, :]] * sa[sl][:, j, None] * sb[:, t]
                S.view(-1).index_add_(0, (Ia[sl][:, j, None] * C.shape[1] + Ib[:, t][None, :]).reshape(-1), e.reshape(-1))
    return S


def _csf_map(n, na, nb):
    """CSFs of S = Ms in configuration order of first appearance: per open-shell count the coupling
    overlaps (ncsf x patterns), the CSF offsets, determinant addresses and signs of each configuration."""
    a, b = _masks(n, na), _masks(n, nb)
    A, B = np.repeat(a, len(b)), np.tile(b, len(a))
    d, s, twos = A & B, A ^ B, na - nb
    key, first, inv = np.unique((d << n) | s, return_index=True, return_inverse=True)
    order = np.argsort(first)
    rank = np.empty(len(order), np.int64)
    rank[order] = np.arange(len(order))
    conf = rank[inv.reshape(-1)]
    nopen = np.array([bin(x).count("1") for x in (key[order] & ((1 << n) - 1))])
    neg = np.zeros(len(A), np.int64)  # open shells created from the highest orbital down on the closed ones
    acur, occ = d.copy(), np.zeros(len(A), np.int64)
    npar = lambda m: (1 - _parity(m, np.int64(n))).astype(np.int64) // 2  # noqa: E731
    for p in range(n - 1, -1, -1):
        op, be = (s >> p) & 1, (B >> p) & 1
        low = ((1 - _parity(d, np.int64(p))) / 2).astype(np.int64)
        neg ^= op * (low ^ (be * npar(acur)))
        acur |= (op * (1 - be)) << p
    for p in range(n - 1, -1, -1):  # beta pattern read as a sequence from the lowest open orbital
        op, be = (s >> p) & 1, (B >> p) & 1
        occ = np.where(op == 1, (be << 40) | (occ >> 1), occ)
    out, tables = [], {}
    counts = {}
    for N in sorted(set(nopen.tolist())):
        ups = (N + twos) // 2
        pats = sorted({tuple(0 if i in c else 1 for i in range(N)) for c in itertools.combinations(range(N), ups)})
        coup = [p for p in pats if all(sum(1 - 2 * x for x in p[:i + 1]) >= 0 for i in range(N))]
        T = np.zeros((len(coup), len(pats)))
        for i, c in enumerate(coup):
            for j, o in enumerate(pats):
                v, S2, M2 = 1.0, 0, 0
                for x, y in zip(c, o):
                    dS, dM = 1 - 2 * x, 1 - 2 * y
                    S2, M2 = S2 + dS, M2 + dM
                    if abs(M2) > S2:
                        v = 0.0
                        break
                    v *= math.sqrt(0.5 * (S2 + dM * M2) / S2) if dS == 1 else -dM * math.sqrt(
                        0.5 * (S2 + 2 - dM * M2) / (S2 + 2))
                T[i, j] = v
        tables[N], counts[N] = T, len(coup)
    off = np.concatenate([[0], np.cumsum([counts[x] for x in nopen])])
    by = np.lexsort((occ, conf))
    start = np.searchsorted(conf[by], np.arange(len(nopen)))
    for N, T in tables.items():
        cs = np.nonzero(nopen == N)[0]
        if T.shape[0] == 0:
            continue
        dets = by[start[cs][:, None] + np.arange(T.shape[1])]
        t = lambda x: torch.as_tensor(x, device=DEV)  # noqa: E731
        out.append((t(T), t(off[cs][:, None] + np.arange(T.shape[0])), t(dets), t(1.0 - 2.0 * neg[dets])))
    return int(off[-1]), len(A), out


def _lanczos(apply, size, roots, seed):
    g = _gen(seed)
    v = torch.randn(size, generator=g, dtype=torch.float64, device=DEV)
    m = min(size, 400)
    Q, alpha, beta = [v / torch.linalg.vector_norm(v)], [], []
    for j in range(m):
        w = apply(Q[-1])
        alpha.append(float(w @ Q[-1]))
        Z = torch.stack(Q)
        for _ in range(2):
            w = w - Z.T @ (Z @ w)
        b = float(torch.linalg.vector_norm(w))
        if b < 1e-10:
            break
        beta.append(b)
        Q.append(w / b)
    k = len(alpha)
    T = np.diag(alpha) + np.diag(beta[:k - 1], 1) + np.diag(beta[:k - 1], -1)
    return np.linalg.eigvalsh(T)[:roots]


def exact(case, seed):
    kind, (n, na, nb, n0a, n0b) = case["kind"], _spaces(case)
    t = lambda x: torch.as_tensor(x, device=DEV)  # noqa: E731
    if kind == "rel":
        h, V = _spinor_integrals(n, seed)
        w, g = _decay(n, na, h), _gen(seed)
        re, im = (torch.randn(len(w), generator=g, dtype=torch.float64, device=DEV) for _ in range(2))
        c = torch.complex(re * w, im * w)
        c = c / torch.linalg.vector_norm(c)
        return _same_spin(n, na, t(h), t(V), c[:, None])[:, 0] + 0.25 * c
    if n0a * n0b > 12_000_000:
        return None  # minutes in plain torch
    if kind == "solve":
        h, V = _integrals(n, seed + 1000003)
        # + 5 S^2 (S^2 = nb - sum a+_pa a_qa a+_qb a_pb for Ms = 0) puts the singlets lowest
        x = np.einsum("ps,rq->prqs", np.eye(n), np.eye(n))
        hh, VV, Vab = t(h), t(V), t(V - 5.0 * x)
        apply = lambda v: _sigma(n, na, nb, hh, VV, v.reshape(n0a, n0b), Vab).reshape(-1) + 5.0 * nb * v  # noqa: E731
        return {"evals": _lanczos(apply, n0a * n0b, case["roots"], seed), "evecs": None}
    h, V = _integrals(n, seed)
    if kind == "blocked":
        h, V = _symmetrized(h, V, _irreps(case))
    hh, VV = t(h), t(V)
    if kind == "closure":
        ncsf, ndet, groups = _csf_map(n, na, nb)
        X = _csf_rows(case["rows"], ncsf, seed)
        out = torch.zeros_like(X)
        for i in range(case["rows"]):
            c = torch.zeros(ndet, dtype=torch.float64, device=DEV)
            for T, ci, di, sg in groups:
                c[di] = (X[i][ci] @ T) * sg
            y = _sigma(n, na, nb, hh, VV, c.reshape(n0a, n0b)).reshape(-1)
            for T, ci, di, sg in groups:
                out[i][ci] = (y[di] * sg) @ T.T
        return out
    c = _ci_vector(n, na, nb, h, seed)
    if kind == "blocked":
        at = _blocked_positions(case)
        x = torch.zeros_like(c)
        x[at] = c[at] / torch.linalg.vector_norm(c[at])
        return _sigma(n, na, nb, hh, VV, x.reshape(n0a, n0b)).reshape(-1)[at]
    C = c.reshape(n0a, n0b)
    if kind in ("sigma", "host"):
        s = _sigma(n, na, nb, hh, VV, C).reshape(-1)
        return s.cpu().numpy() if kind == "host" else s
    if kind == "rdm12":
        g1 = torch.zeros(n, n, dtype=torch.float64, device=DEV)
        g2 = torch.zeros(n, n, n, n, dtype=torch.float64, device=DEV)
        for k, M in ((na, C), (nb, C.T.contiguous())):
            o, I, s = _holes(n, k, 1)
            _gram(o[:, :, 0], I, s, M, g1)
            if k < 2:
                continue
            o, I, s = _holes(n, k, 2)
            P = torch.zeros(n * n, n * n, dtype=torch.float64, device=DEV)
            _gram(o[:, :, 0] * n + o[:, :, 1], I, s, M, P)
            P = P.reshape(n, n, n, n)
            P = P - P.transpose(0, 1)
            g2 += P - P.transpose(2, 3)
        ab = torch.zeros(n * n, n * n, dtype=torch.float64, device=DEV)
        for _, D in _opposite_blocks(n, na, nb, C):
            D = D.reshape(-1, n * n)
            ab += D.T @ D
        ab = ab.reshape(n, n, n, n)
        return {"g1": g1, "g2": g2 + ab + ab.permute(1, 0, 3, 2)}
    # 3-RDM from products of the spin-free E_pq = sum_s a+_ps a_qs
    (oa, Ia, sa), (ob, Ib, sb) = _holes(n, na, 1), _holes(n, nb, 1)

    def ops(k, I, o, s, N):
        X = torch.zeros(n, n, N, N, dtype=torch.float64, device=DEV)
        for i in range(I.shape[1]):
            for j in range(I.shape[1]):
                X[o[:, i, 0], o[:, j, 0], I[:, i], I[:, j]] += s[:, i] * s[:, j]
        return X

    ea, eb = ops(na, Ia, oa, sa, n0a), ops(nb, Ib, ob, sb, n0b)
    E = lambda p, q, x: ea[p, q] @ x + x @ eb[p, q].T  # noqa: E731
    EC = torch.stack([torch.stack([E(r, u, C).reshape(-1) for u in range(n)]) for r in range(n)])  # [r, u]
    L = EC.transpose(0, 1).reshape(n * n, -1)  # <C| E_ps = (E_sp C)^T
    d = torch.eye(n, dtype=torch.float64, device=DEV)
    e1 = torch.einsum("rui,i->ru", EC, C.reshape(-1))
    e2 = torch.einsum("spi,rui->psru", EC, EC)  # <E_ps E_ru>
    two = (e2 - torch.einsum("sr,pu->psru", d, e1)).permute(0, 2, 1, 3)  # [p r s u]
    X = torch.empty(n, n, n, n, n, n, dtype=torch.float64, device=DEV)  # <E_ps E_qt E_ru> as [q t r u p s]
    for q in range(n):
        for u in range(n):
            Y = torch.stack([torch.stack([E(q, tt, EC[r, u].reshape(n0a, n0b)).reshape(-1) for r in range(n)])
                             for tt in range(n)])
            X[q, :, :, u] = (Y.reshape(n * n, -1) @ L.T).reshape(n, n, n, n)
    # two-body products of the last pair normal ordered first, then the whole triple
    G = X.permute(4, 0, 2, 5, 1, 3) - torch.einsum("tr,psqu->pqrstu", d, e2)
    return G - torch.einsum("sq,prtu->pqrstu", d, two) - torch.einsum("sr,qptu->pqrstu", d, two)


def _gram(idx, I, s, M, out):
    step = max(1, int(2e8) // max(1, I.shape[1] * M.shape[1]))
    n = out.shape[0]
    for a in range(0, len(I), step):
        i = I[a:a + step]
        D = M[i.reshape(-1)].reshape(*i.shape, -1) * s[a:a + step, :, None]
        at = idx[a:a + step, :, None] * n + idx[a:a + step, None, :]
        out.view(-1).index_add_(0, at.reshape(-1), torch.bmm(D, D.transpose(1, 2)).reshape(-1))
