"""The ASCI enumeration by rows (beta singles, pairs of occupied orbitals) and
its table against the oracle at the shapes where a row is empty, shorter than
a warp or just longer, and where the orbital masks are full: the search
without a cut-off selects the oracle's set, the PT2 sum finds the oracle's
number of external determinants and its energy to 1e-12 (sums of at most a
million FP64 terms of one sign, each good to a few units in the last place)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi(pkg):
    pkg.build.build()
    return pkg.capi


def _wfn(pkg, norb, na, nb, nd, seed):
    """nd distinct random determinants in spin order with random coefficients"""
    rng = np.random.default_rng(seed)
    def string(k):
        return sum(1 << int(p) for p in rng.choice(norb, k, replace=False))
    dets = set()
    for _ in range(50 * nd):
        dets.add((string(na), string(nb)))
        if len(dets) == nd:
            break
    dets = sorted(dets)
    a = np.array([d[0] for d in dets], np.uint64)
    b = np.array([d[1] for d in dets], np.uint64)
    c = rng.standard_normal(len(dets))
    return a, b, c / np.linalg.norm(c)


@pytest.mark.parametrize("norb,na,nb,nd", [(5, 1, 0, 3), (6, 0, 2, 4), (4, 4, 1, 2), (7, 3, 2, 25), (9, 5, 4, 40),
                                           (12, 2, 6, 7), (33, 2, 1, 5), (40, 3, 3, 2), (64, 1, 1, 3), (48, 40, 40, 2),
                                           (64, 62, 63, 2)])
def test_search_and_pt2_match_oracle(capi, pkg, oracle, norb, na, nb, nd):
    T, V, _ = pkg.integrals.synthetic_integrals(norb, 2 * norb, 77 + norb)
    H = oracle.Hamiltonian(T, V)
    a, b, c = _wfn(pkg, norb, na, nb, nd, norb + nd)
    E0 = min(H.matrix_element((x, y), (x, y)) for x, y in zip(a.tolist(), b.tolist())) - 50.0
    oa, ob = oracle.asci_search(H, a, b, c, E0, 10**7)
    eo, no = oracle.asci_pt2(H, a, b, c, E0)
    with capi.Context(0) as ctx:
        ctx.set_integrals(T, V)
        ga, gb = capi.asci_search(ctx, a, b, c, E0, 10**7)
        eg, ng = capi.asci_pt2(ctx, a, b, c, E0)
    assert set(zip(ga.tolist(), gb.tolist())) == set(zip(oa.tolist(), ob.tolist())) and len(ga) == len(oa)
    assert ng == no
    assert abs(eg - eo) <= 1e-12 * max(1.0, abs(eo))
