"""The direct sigma's contraction from 16-bit parts (contract.cuh) against the
element-wise forms (QDKGB_DIRECT_TC=0), at the sizes where it can go wrong:
ragged last chunks of 64 beta strings, K (singles + 1) at and off a multiple
of 16, unequal spins, 121 rows of E, several K ranges of the dense products.

Tolerances, before any run: FP64 sums of at most 3,000 terms in either form
differ by less than 3,000 2^-53 of the largest partial sum, 4e-13 of the
largest sigma element; the digits' truncation (2^-53 of a row's largest
products) is below that.  FP32: 1e-5 of the largest element, as for the other
FP32 forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(10, 5, 5, 1), (11, 5, 4, 2), (12, 3, 5, 3), (12, 6, 3, 4), (13, 2, 6, 5), (14, 4, 2, 6), (15, 3, 3, 7)]


@pytest.fixture(scope="module")
def ctx(pkg):
    pkg.build.build()
    c = pkg.capi.Context(0)
    yield c
    c.close()


def _sigmas(ctx, capi, monkeypatch, x, precision):
    out = {}
    for tc in ("0", "1"):
        monkeypatch.setenv("QDKGB_DIRECT_TC", tc)
        ctx.build_direct_sigma()
        out[tc] = ctx.spmv(x, precision)
        assert np.array_equal(out[tc], ctx.spmv(x, precision), equal_nan=True)  # repeats bit for bit
    return out["0"], out["1"]


@pytest.mark.parametrize("norb,na,nb,seed", SHAPES)
def test_contraction_matches_element_wise(ctx, pkg, monkeypatch, norb, na, nb, seed):
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(norb, 2 * norb, seed)
    a, b = capi.fci_dets(norb, na, nb)
    assert len(a) >= 32768  # the sizes that take this form
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    rng = np.random.default_rng(seed)
    dense = rng.normal(size=len(a))
    steep = dense * 10.0 ** -rng.uniform(0, 12, size=len(a))  # coefficients over twelve decades
    one = np.zeros(len(a))
    one[len(a) // 3] = -1.7
    for x in (dense, steep, one, 1e-200 * dense, 1e200 * dense, np.zeros(len(a))):
        old, new = _sigmas(ctx, capi, monkeypatch, x, capi.PREC_FP64)
        assert np.max(np.abs(new - old)) <= 4e-13 * np.max(np.abs(old))
    old, new = _sigmas(ctx, capi, monkeypatch, dense, capi.PREC_MIXED)
    assert np.max(np.abs(new - old)) <= 1e-5 * np.max(np.abs(old))


def test_non_finite_elements(ctx, pkg, monkeypatch):
    """An infinity or NaN reaches the rows it couples to and no others."""
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(10, 20, 11)
    a, b = capi.fci_dets(10, 5, 5)
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    for bad in (np.nan, np.inf):
        x = np.random.default_rng(11).normal(size=len(a))
        x[777] = bad
        old, new = _sigmas(ctx, capi, monkeypatch, x, capi.PREC_FP64)
        fine = np.isfinite(old)
        assert 0 < np.count_nonzero(~fine) < len(a)
        assert np.array_equal(fine, np.isfinite(new))
        assert np.max(np.abs(new[fine] - old[fine])) <= 4e-13 * np.max(np.abs(old[fine]))


def test_integrals_without_pair_symmetry(ctx, pkg, monkeypatch):
    """V(pq|rs) != V(pq|sr): one row of E cannot serve both, the other forms run."""
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(10, 20, 12)
    V = V.copy()
    V[1, 2, 3, 4] += 1e-3
    a, b = capi.fci_dets(10, 5, 5)
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    x = np.random.default_rng(12).normal(size=len(a))
    old, new = _sigmas(ctx, capi, monkeypatch, x, capi.PREC_FP64)
    assert np.array_equal(old, new)
    old, new = _sigmas(ctx, capi, monkeypatch, x, capi.PREC_MIXED)
    assert np.max(np.abs(new - old)) <= 1e-5 * np.max(np.abs(old))


def test_stored_space(ctx, pkg, monkeypatch):
    """A stored complete space: the FP64 sigma through the digits equals the
    slab's; a threshold above the machine epsilon keeps the slab's sigma."""
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(11, 22, 13)
    a, b = capi.fci_dets(11, 5, 5)
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    x = np.random.default_rng(13).normal(size=len(a))
    y = {}
    for thresh in (np.finfo(float).eps, 1e-2):
        for tc in ("0", "1"):
            monkeypatch.setenv("QDKGB_DIRECT_TC", tc)
            ctx.build_hamiltonian(thresh)
            y[thresh, tc] = ctx.spmv(x, capi.PREC_FP64)
    e, t = np.finfo(float).eps, 1e-2
    scale = np.max(np.abs(y[e, "0"]))
    assert np.max(np.abs(y[e, "1"] - y[e, "0"])) <= 4e-13 * scale
    assert np.array_equal(y[t, "1"], y[t, "0"])
    assert np.max(np.abs(y[t, "0"] - y[e, "0"])) > 1e-6 * scale
