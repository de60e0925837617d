"""The work that users of this framework have it do, as timed cases.

Every case goes through the public entry points (``capi``, ``autograd``) on the
seeded integral recipe of the framework's own benchmark:

* ``solve``: a CASCI from host integrals to energy and CI vector, the call behind
  the CASCI plugin (plain FP64, its default, and the mixed form);
* ``gradient``: the differentiable CASCI energy, forward and backward;
* ``batch``: many small active spaces in one call;
* ``sigma``: one application of the Hamiltonian to a device vector, which every
  eigensolver on top of this library repeats (stored or direct, FP64 or FP32);
* ``rdms``: the spin-resolved RDMs of a CI vector over a complete space;
* ``selected``: the CI problem of a caller's determinant list;
* ``asci``: selected CI grown from the lowest determinant (searches, Hamiltonian builds, solves).

``listed()`` names one case per place where the paths are used in earnest, from
400 determinants to 11.8 million; ``draw()`` gives others of the same ranges.
The solves run to a residual of 1e-10, the differentiable energy's default.
"""
import functools
import itertools
import math

import numpy as np
import torch

import __graft_entry__

SOLVE_TOL = 1e-10
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _package():
    return __graft_entry__._package()


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest active space of the batched benchmark, one call at a time:
        # launches and host steps count
        dict(name="solve_6e6o_fp64", kind="solve", norb=6, na=3, nb=3, precision="fp64"),
        # the plain FP64 configuration CASCI(8e,8o), 4,900 determinants
        dict(name="solve_8e8o_fp64", kind="solve", norb=8, na=4, nb=4, precision="fp64"),
        # an ordinary solve with an odd orbital count and unequal spins
        dict(name="solve_9e11o_mixed", kind="solve", norb=11, na=5, nb=4, precision="mixed"),
        # the headline configuration, in the plugin's default precision and in the mixed form
        dict(name="solve_12e12o_fp64", kind="solve", norb=12, na=6, nb=6, precision="fp64"),
        dict(name="solve_12e12o_mixed", kind="solve", norb=12, na=6, nb=6, precision="mixed"),
        # energy and integral gradients of a mid-sized space (forward and backward)
        dict(name="gradient_10e10o", kind="gradient", norb=10, na=5, nb=5, precision="fp64"),
        # a slice of the batched configuration (norb drawn from 6, 8, 10)
        dict(name="batch_48", kind="batch", count=48, sizes="6,8,10"),
        # the FP32 sigma of a mixed solve at the headline size
        dict(name="sigma_12e12o_fp32", kind="sigma", norb=12, na=6, nb=6, operator="direct", precision="mixed"),
        # the full-precision direct sigma at CASCI(14e,14o), the largest space (no matrix fits)
        dict(name="sigma_14e14o_fp64", kind="sigma", norb=14, na=7, nb=7, operator="direct", precision="fp64"),
        # RDMs of a CI vector at the headline size, as CASSCF and the gradients ask for them
        dict(name="rdms_12e12o", kind="rdms", norb=12, na=6, nb=6),
        # a projected solve on a caller's list of 20,000 determinants in 24 orbitals
        dict(name="selected_20k_24o", kind="selected", norb=24, na=6, nb=5, ndets=20000),
        # the 40-orbital selected-CI configuration, grown to 50,000 determinants
        dict(name="asci_40o_50k", kind="asci", norb=40, na=8, nb=8, ncore=1000, ndets=50000),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "sigma", "sigma", "gradient", "batch", "rdms", "selected", "asci"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    spins = lambda n: (lambda a: (a, a - rng.randint(0, 1)))(min(n - 2, max(2, n // 2 + rng.randint(-1, 1))))
    if kind == "solve":
        n = rng.randint(5, 12)
        a, b = spins(n)
        return dict(kind=kind, norb=n, na=a, nb=b, precision=rng.choice(["fp64", "mixed"]))
    if kind == "gradient":
        n = rng.randint(5, 10)
        a, b = spins(n)
        return dict(kind=kind, norb=n, na=a, nb=b, precision=rng.choice(["fp64", "mixed"]))
    if kind == "batch":
        sizes = sorted(rng.sample([5, 6, 7, 8, 9, 10], 3))
        return dict(kind=kind, count=log(3, 48), sizes=",".join(map(str, sizes)))
    if kind == "sigma":
        operator = rng.choice(["stored", "direct"])
        n = rng.randint(8, 12 if operator == "stored" else 14)
        a, b = spins(n)
        return dict(kind=kind, norb=n, na=a, nb=b, operator=operator, precision=rng.choice(["fp64", "mixed"]))
    if kind == "rdms":
        n = rng.randint(6, 12)
        a, b = spins(n)
        return dict(kind=kind, norb=n, na=a, nb=b)
    if kind == "selected":
        n = rng.randint(16, 28)
        a = rng.randint(3, 6)
        return dict(kind=kind, norb=n, na=a, nb=a - rng.randint(0, 1), ndets=log(1000, 20000))
    dets = log(2000, 50000)
    return dict(kind=kind, norb=rng.randint(20, 40), na=rng.randint(5, 8), nb=rng.randint(5, 8), ncore=dets // 50,
                ndets=dets)


# ------------------------------------------------------------------ inputs
def _integrals(case, seed, salt=0):
    n = case["norb"]
    spacing = 0.1 if case["kind"] == "asci" else 0.25
    T, V, _ = _package().integrals.synthetic_integrals(n, 2 * n, 1000003 * int(seed) + salt, diag_spacing=spacing)
    return T, V


@functools.lru_cache(maxsize=None)
def _strings(n, k):
    """Spin strings in the determinant order of the complete spaces."""
    return np.array([sum(1 << p for p in pos) for pos in itertools.combinations(range(n), k)], dtype=np.int64)


def _popcount(x):
    x = np.asarray(x).astype(np.uint64)
    return sum(_POP8[((x >> np.uint64(8 * i)) & np.uint64(255)).astype(np.int64)] for i in range(8))


_POP8 = np.array([bin(i).count("1") for i in range(256)], dtype=np.int64)


def _ci_vector(case, seed):
    """A CI-like vector on the device: normal coefficients that fall by a
    factor of four per excitation from the lowest determinant, normalised."""
    n, na, nb = case["norb"], case["na"], case["nb"]
    la = torch.from_numpy(na - _popcount(_strings(n, na) & ((1 << na) - 1))).to(DEVICE)
    lb = torch.from_numpy(nb - _popcount(_strings(n, nb) & ((1 << nb) - 1))).to(DEVICE)
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))
    x = torch.randn(len(la), len(lb), generator=g, dtype=torch.float64, device=DEVICE)
    x *= 4.0 ** -(la[:, None] + lb[None, :]).double()
    return (x / x.norm()).reshape(-1)


def _determinant_list(n, na, nb, count, seed):
    """`count` distinct determinants, mostly one to four excitations from the
    lowest one and near the Fermi level, in spin order (alpha, then beta)."""
    rng = np.random.default_rng(int(seed))

    def excite(k, levels):
        # the k lowest of random orbital energies whose noise grows with the level
        e = np.arange(n)[None, :] + rng.gumbel(0.0, 1.0, (len(levels), n)) * (0.8 * levels)[:, None]
        pos = np.argpartition(e, k - 1, axis=1)[:, :k]
        return (np.uint64(1) << pos.astype(np.uint64)).sum(axis=1, dtype=np.uint64)

    a = np.array([(1 << na) - 1], dtype=np.uint64)
    b = np.array([(1 << nb) - 1], dtype=np.uint64)
    scale = 1.0
    while len(a) < count:
        m = 2 * count
        levels = rng.integers(0, 4, size=(2, m)) * scale
        a = np.concatenate([a, excite(na, levels[0])])
        b = np.concatenate([b, excite(nb, levels[1])])
        order = np.lexsort((np.arange(len(a)), b, a))
        new = np.ones(len(a), dtype=bool)
        sa, sb = a[order], b[order]
        new[1:] = (sa[1:] != sa[:-1]) | (sb[1:] != sb[:-1])
        keep = np.sort(order[new])  # first arrivals
        a, b = a[keep], b[keep]
        scale *= 1.25
    a, b = a[:count], b[:count]
    order = np.lexsort((b, a))
    return a[order], b[order]


def prepare(case, seed):
    pkg = _package()
    capi, kind = pkg.capi, case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(int(seed))
        sizes = [int(s) for s in case["sizes"].split(",")]
        inst = []
        for i in range(case["count"]):
            no = sizes[i % len(sizes)]
            T, V = _integrals(dict(kind=kind, norb=no), seed, int(rng.integers(1, 1000000)))
            inst.append((no, no // 2, no // 2, T, V))
        return dict(case=case, ctx=capi.Context(0), inst=inst)
    T, V = _integrals(case, seed)
    if kind == "gradient":
        # integrals as a differentiable program holds them, on the device
        return dict(case=case, h1=torch.from_numpy(T).to(DEVICE), eri=torch.from_numpy(V).to(DEVICE))
    ctx = capi.Context(0)
    state = dict(case=case, ctx=ctx, T=T, V=V)
    if kind == "solve":
        return state
    ctx.set_integrals(T, V)
    if kind == "selected":
        state["dets"] = _determinant_list(case["norb"], case["na"], case["nb"], case["ndets"], seed)
    elif kind == "asci":
        state["start"] = pkg.determinants.canonical_hf(case["na"], case["nb"])
        state["E0"] = _lowest_diagonal(T, V, case["na"], case["nb"])
    else:
        a, b = capi.fci_dets(case["norb"], case["na"], case["nb"])
        ctx.set_dets(a, b)
        x = _ci_vector(case, seed)
        if kind == "rdms":
            state["x"] = x.cpu().numpy()
            return state
        mixed = case["precision"] == "mixed"
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        if case["operator"] == "stored":
            ctx.build_hamiltonian(storage=capi.H_SPLIT32 if mixed else capi.H_FP64)
        else:
            ctx.build_direct_sigma()
        state["x"] = x.float() if mixed else x
        state["y"] = torch.empty_like(state["x"])
        state.update(stream=stream, prec=capi.PREC_MIXED if mixed else capi.PREC_FP64)
        torch.cuda.synchronize()
    return state


def _lowest_diagonal(T, V, na, nb):
    oa, ob = range(na), range(nb)
    e = sum(T[p, p] for p in oa) + sum(T[p, p] for p in ob)
    for occ in (oa, ob):
        e += 0.5 * sum(V[p, p, q, q] - V[p, q, q, p] for p in occ for q in occ)
    return float(e + sum(V[p, p, q, q] for p in oa for q in ob))


def _phased(C):
    """An eigenvector's sign is arbitrary: the lowest determinant's coefficient
    (the first of every list here) is made positive."""
    return C if C[0] >= 0 else -C


def run(state):
    case, pkg = state["case"], _package()
    capi, kind = pkg.capi, case["kind"]
    if kind == "solve":
        prec = capi.PREC_MIXED if case["precision"] == "mixed" else capi.PREC_FP64
        E, C, _ = state["ctx"].casci(state["T"], state["V"], case["na"], case["nb"], tol=SOLVE_TOL, precision=prec)
        return {"E": np.float64(E), "C": _phased(C)}
    if kind == "gradient":
        E, g1, g2 = pkg.autograd.rdms_as_gradients(state["h1"], state["eri"], case["na"], case["nb"],
                                                   precision=case["precision"])
        return {"E": E, "dh1": g1, "deri": g2}
    if kind == "batch":
        E, rdms, _, _ = capi.casci_batch(state["ctx"], state["inst"], res_tol=SOLVE_TOL)
        return {"E": E, "rdm1": np.concatenate([r.ravel() for r in rdms])}
    if kind == "sigma":
        state["ctx"].spmv_device(state["x"].data_ptr(), state["y"].data_ptr(), state["prec"])
        return state["y"]
    if kind == "rdms":
        return state["ctx"].rdms_spin_dep(state["x"])
    ctx = state["ctx"]
    if kind == "selected":
        ctx.set_dets(*state["dets"])
        ctx.build_hamiltonian()
        E, C, _ = ctx.davidson(tol=SOLVE_TOL)
        return {"E": np.float64(E), "C": _phased(C)}
    a0, b0 = state["start"]
    ctx.set_integrals(state["T"], state["V"])
    E, a, b, C, _ = capi.asci(ctx, [a0], [b0], [1.0], state["E0"], grow=True, refine=False, tol=SOLVE_TOL,
                              ntdets_max=case["ndets"], core_selection_fixed=1, ncdets_max=case["ncore"])
    return {"E": np.float64(E), "alpha": a.view(np.int64), "beta": b.view(np.int64), "C": _phased(C)}


# ------------------------------------------------------------------ least work
def _sigma_flops(n, na, nb):
    """The cheaper of the element-wise sigma (one multiply-add per coupled pair)
    and the pair-space factorisation, 2 (n (n + 1) / 2)^2 per determinant."""
    dets = math.comb(n, na) * math.comb(n, nb)
    sa, sb = na * (n - na), nb * (n - nb)
    row = 1 + (1 + sa) * (1 + sb) + math.comb(na, 2) * math.comb(n - na, 2) + math.comb(nb, 2) * math.comb(n - nb, 2)
    return 2.0 * dets * min(row, (n * (n + 1) // 2) ** 2)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = [int(s) for s in case["sizes"].split(",")]
        per = [work(dict(kind="solve", norb=s, na=s // 2, nb=s // 2)) for s in sizes]
        k = case["count"] / len(sizes)
        return {"bytes": k * sum(w["bytes"] for w in per), "flops": k * sum(w["flops"] for w in per)}
    n, na, nb = case["norb"], case["na"], case["nb"]
    ints = 8.0 * (n ** 2 + n ** 4)
    if kind in ("selected", "asci"):
        sa, sb = na * (n - na), nb * (n - nb)
        row = 1 + sa + sb + sa * sb + math.comb(na, 2) * math.comb(n - na, 2) + math.comb(nb, 2) * math.comb(n - nb, 2)
        if kind == "asci":
            # every excitation of the last core once: a product and a sum; the list out
            return {"bytes": ints + 24.0 * case["ndets"], "flops": 4.0 * case["ncore"] * row}
        # 20 sigmas over at most an eighth of each row's couplings inside the list
        return {"bytes": 32.0 * case["ndets"], "flops": 20 * 2.0 * case["ndets"] * min(row / 8.0, case["ndets"])}
    dets = math.comb(n, na) * math.comb(n, nb)
    if kind == "sigma":
        return {"bytes": (8 if case["precision"] == "mixed" else 16) * dets + ints, "flops": _sigma_flops(n, na, nb)}
    if kind == "rdms":
        return {"bytes": 8.0 * dets + 3 * ints, "flops": _sigma_flops(n, na, nb)}
    # a solve: about 20 sigmas; a gradient adds one RDM sweep
    return {"bytes": ints + 8.0 * dets, "flops": (21 if kind == "gradient" else 20) * _sigma_flops(n, na, nb)}


# ------------------------------------------------------------------ 64-bit values
@functools.lru_cache(maxsize=8)
def _replacements(n, k):
    """For every (p, q): (from, to, sign) of the strings on which a+_p a_q acts."""
    s = _strings(n, k)
    rank = {int(x): i for i, x in enumerate(s)}
    out = {}
    for p in range(n):
        for q in range(n):
            ok = (s >> q) & 1 == 1
            if p != q:
                ok &= (s >> p) & 1 == 0
            src = np.flatnonzero(ok)
            dst = np.array([rank[int(x) ^ (1 << q) | (1 << p)] if p != q else rank[int(x)] for x in s[src]],
                           dtype=np.int64)
            lo, hi = min(p, q), max(p, q)
            between = ((1 << hi) - 1) ^ ((1 << (lo + 1)) - 1) if p != q else 0
            sign = 1.0 - 2.0 * (_popcount((s[src] & between).astype(np.uint64)) & 1)
            out[p, q] = tuple(torch.from_numpy(t).to(DEVICE) for t in (src, dst, sign))
    return out


def _excited(C, n, na, nb, spins="ab"):
    """E_pq C for every (p, q): (n, n, alpha strings, beta strings)."""
    A, B = _replacements(n, na), _replacements(n, nb)
    D = torch.zeros((n, n) + tuple(C.shape), dtype=torch.float64, device=DEVICE)
    for p in range(n):
        for q in range(n):
            if "a" in spins:
                src, dst, sign = A[p, q]
                D[p, q].index_add_(0, dst, C[src] * sign[:, None])
            if "b" in spins:
                src, dst, sign = B[p, q]
                D[p, q].index_add_(1, dst, C[:, src] * sign[None, :])
    return D


def _exact_sigma(T, V, C, na, nb):
    """H C by the pair-space factorisation: sum_pq E_pq (h'_pq C + 1/2 sum_rs V_pqrs E_rs C)."""
    n = T.shape[0]
    T, V = (torch.from_numpy(np.ascontiguousarray(t)).to(DEVICE) for t in (T, V))
    h = T - 0.5 * torch.einsum("prrq->pq", V)
    A, B = _replacements(n, na), _replacements(n, nb)
    D = _excited(C, n, na, nb)
    out = torch.zeros_like(C)
    V = V.reshape(n, n, n * n)
    for p in range(n):
        G = 0.5 * (V[p] @ D.reshape(n * n, -1)).reshape((n,) + tuple(C.shape))
        for q in range(n):
            g = G[q] + h[p, q] * C
            src, dst, sign = A[p, q]
            out.index_add_(0, dst, g[src] * sign[:, None])
            src, dst, sign = B[p, q]
            out.index_add_(1, dst, g[:, src] * sign[None, :])
    return out


def _diagonal(T, V, A, B):
    """<D|H|D> from the occupation rows (determinants x orbitals) of both spins."""
    J, K, t = np.einsum("ppqq->pq", V), np.einsum("pqqp->pq", V), np.diag(T)
    J, K, t = (torch.from_numpy(np.ascontiguousarray(x)).to(A.device) for x in (J, K, t))
    own = lambda S: S @ t + 0.5 * ((S @ (J - K)) * S).sum(-1)
    return own(A), own(B), J


def _lowest(sigma, diag, steps=200, tol=1e-13):
    """Lowest eigenpair by a Davidson iteration, (energy, unit vector)."""
    start = int(torch.argmin(diag))
    steps = min(steps, len(diag))
    Q, W = (torch.zeros(steps, len(diag), dtype=torch.float64, device=DEVICE) for _ in range(2))
    Q[0, start] = 1.0
    for k in range(1, steps + 1):
        W[k - 1] = sigma(Q[k - 1])
        H = Q[:k] @ W[:k].T
        e, U = torch.linalg.eigh((H + H.T) / 2)
        x = U[:, 0] @ Q[:k]
        r = U[:, 0] @ W[:k] - e[0] * x
        if k == steps or float(r.norm()) < tol * max(1.0, abs(float(e[0]))):
            break
        den = diag - e[0]
        t = -r / torch.where(den.abs() < 1e-6, torch.full_like(den, 1e-6), den)
        for _ in range(3):
            t = t - (Q[:k] @ t) @ Q[:k]
            t = t / t.norm()
        Q[k] = t
    x = x / x.norm()
    return np.float64(e[0].item()), x if x[0] >= 0 else -x


def _exact_solve(T, V, na, nb):
    n = T.shape[0]
    occ = lambda k: torch.from_numpy(((_strings(n, k)[:, None] >> np.arange(n)) & 1).astype(float)).to(DEVICE)
    A, B = occ(na), occ(nb)
    a, b, J = _diagonal(T, V, A, B)
    diag = (a[:, None] + b[None, :] + A @ J @ B.T).reshape(-1)
    shape = (len(A), len(B))
    E, C = _lowest(lambda v: _exact_sigma(T, V, v.reshape(shape), na, nb).reshape(-1), diag)
    return E, C.reshape(shape)


def _exact_rdms(C, n, na, nb):
    """aa, bb and the two-body blocks 1/2 <a+_p a+_r a_s a_q> (aabb: pq beta, rs alpha)."""
    Da, Db = (_excited(C, n, na, nb, s).reshape(n * n, -1) for s in "ab")
    c = C.reshape(-1)
    one = {"aa": (Da @ c).reshape(n, n), "bb": (Db @ c).reshape(n, n)}
    eye = torch.eye(n, dtype=torch.float64, device=DEVICE)
    out = dict(one)
    for key, L, R, g in (("aaaa", Da, Da, one["aa"]), ("bbbb", Db, Db, one["bb"]), ("aabb", Db, Da, None)):
        G = (L @ R.T).reshape(n, n, n, n).transpose(0, 1)
        if g is not None:
            G = G - torch.einsum("qr,ps->pqrs", eye, g)
        out[key] = 0.5 * G
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_selected(T, V, a, b):
    """Lowest eigenpair of a determinant list: every pair of determinants within
    two excitations by the Slater-Condon rules."""
    n, N = T.shape[0], len(a)
    dev = DEVICE
    sa, sb = (torch.from_numpy(x.astype(np.int64)).to(dev) for x in (a, b))
    pop = torch.from_numpy(_popcount(np.arange(1 << 16).astype(np.uint64))).to(dev)
    count = lambda x: sum(pop[(x >> (16 * i)) & 0xffff] for i in range(3))
    bits = torch.arange(n, device=dev)
    occ = lambda s: ((s[:, None] >> bits) & 1).double()
    A, B = occ(sa), occ(sb)
    da, db, J = _diagonal(T, V, A, B)
    diag = da + db + ((A @ J) * B).sum(-1)
    t, v = (torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (T, V))
    first = torch.einsum("ppvo->pvo", v)  # V(p p | v o)
    mine = first - torch.einsum("povp->pvo", v)
    low = lambda x: count((x & -x) - 1)
    ones = torch.ones((), dtype=torch.int64, device=dev)

    def swap(bra, ket):
        """(v, o, sign, ket after it) of the lowest differing orbitals."""
        x = bra ^ ket
        vv, oo = low(x & bra), low(x & ket)
        lo, hi = torch.minimum(vv, oo), torch.maximum(vv, oo)
        between = ((ones << hi) - 1) & ~((ones << (lo + 1)) - 1)
        return vv, oo, 1.0 - 2.0 * (count(ket & between) & 1).double(), ket ^ (ones << vv) ^ (ones << oo)

    I, K, X = [], [], []

    def put(i, j, x):
        I.append(i)
        K.append(j)
        X.append(x)

    for i0 in range(0, N, 1024):
        rows = slice(i0, min(N, i0 + 1024))
        xa, xb = count(sa[rows, None] ^ sa[None, :]), count(sb[rows, None] ^ sb[None, :])
        for la, lb in ((2, 0), (0, 2), (2, 2), (4, 0), (0, 4)):
            i, j = torch.nonzero((xa == la) & (xb == lb), as_tuple=True)
            i = i + i0
            if la == 2 and lb == 2:
                v1, o1, s1, _ = swap(sa[i], sa[j])
                v2, o2, s2, _ = swap(sb[i], sb[j])
                put(i, j, s1 * s2 * v[v1, o1, v2, o2])
                continue
            s, same, other = (sa, A, B) if la else (sb, B, A)
            v1, o1, s1, rest = swap(s[i], s[j])
            if la + lb == 4:
                v2, o2, s2, _ = swap(s[i], rest)
                put(i, j, s1 * s2 * (v[v1, o1, v2, o2] - v[v1, o2, v2, o1]))
            else:
                x = t[v1, o1]
                for p in range(n):
                    x = x + same[j, p] * mine[p, v1, o1] + other[j, p] * first[p, v1, o1]
                put(i, j, s1 * x)
    I, K, X = torch.cat(I), torch.cat(K), torch.cat(X)
    H = torch.sparse_coo_tensor(torch.stack([I, K]), X, (N, N)).coalesce().to_sparse_csr()
    E, C = _lowest(lambda y: diag * y + H @ y, diag)
    return E, C


def exact(case, seed):
    kind = case["kind"]
    if kind == "asci":
        return None  # the selection is a sequence of searches and solves
    if kind == "batch":
        if case["count"] > 12:
            return None  # over the time for it
        out = [], []
        for no, na, nb, T, V in prepare(case, seed)["inst"]:
            E, C = _exact_solve(T, V, na, nb)
            R = _exact_rdms(C, no, na, nb)
            out[0].append(E)
            out[1].append((R["aa"] + R["bb"]).ravel())
        return {"E": np.array(out[0]), "rdm1": np.concatenate(out[1])}
    n, na, nb = case["norb"], case["na"], case["nb"]
    T, V = _integrals(case, seed)
    if kind == "solve":
        E, C = _exact_solve(T, V, na, nb)
        return {"E": E, "C": C.reshape(-1)}
    if kind == "gradient":
        E, C = _exact_solve(T, V, na, nb)
        R = _exact_rdms(C, n, na, nb)
        return {"E": E, "dh1": R["aa"] + R["bb"],
                "deri": R["aaaa"] + R["bbbb"] + R["aabb"] + R["aabb"].transpose(2, 3, 0, 1)}
    if kind == "selected":
        E, C = _exact_selected(T, V, *_determinant_list(n, na, nb, case["ndets"], seed))
        return {"E": E, "C": C}
    x = _ci_vector(case, seed).reshape(math.comb(n, na), math.comb(n, nb))
    if kind == "rdms":
        return _exact_rdms(x, n, na, nb)
    if case["precision"] == "mixed":
        x = x.float().double()
    return _exact_sigma(T, V, x, na, nb).reshape(-1)
