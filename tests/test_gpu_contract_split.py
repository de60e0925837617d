"""Where the 16-bit contraction splits its last wave's alpha strings over
several CTAs (all of them, some, in FP64 only, in FP32 only), every number of
accumulator slots (K padded to 16, 32, 48 and 64), and the dense products of
few tiles split over K: against the element-wise forms, and again and again
bit for bit (the partial sums are left at zero).

Tolerances as for the unsplit forms, before any run: whole numbers add exactly
in FP64 (4e-13 of the largest element between the two forms), FP32 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(11, 5, 5), (11, 4, 6), (12, 6, 6), (14, 7, 3), (14, 1, 6), (12, 2, 6), (10, 5, 4)]


@pytest.fixture(scope="module")
def ctx(pkg):
    pkg.build.build()
    c = pkg.capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("norb,na,nb", SHAPES)
def test_split_strings_and_products(ctx, pkg, monkeypatch, norb, na, nb):
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(norb, 2 * norb, 3 + norb)
    a, b = capi.fci_dets(norb, na, nb)
    assert len(a) >= 32768  # the sizes that take this form
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    rng = np.random.default_rng(norb)
    dense = rng.normal(size=len(a))
    steep = dense * 10.0 ** -rng.uniform(0, 12, size=len(a))
    old, new = {}, {}
    for tc, out in (("0", old), ("1", new)):
        monkeypatch.setenv("QDKGB_DIRECT_TC", tc)
        ctx.build_direct_sigma()
        for name, x in (("dense", dense), ("steep", steep)):
            out[name] = ctx.spmv(x, capi.PREC_FP64)
            out[name, 32] = ctx.spmv(x, capi.PREC_MIXED)
        if tc == "1":
            for _ in range(3):
                for name, x in (("steep", steep), ("dense", dense)):
                    assert np.array_equal(new[name], ctx.spmv(x, capi.PREC_FP64))
                    assert np.array_equal(new[name, 32], ctx.spmv(x, capi.PREC_MIXED))
    for name in ("dense", "steep"):
        assert np.max(np.abs(new[name] - old[name])) <= 4e-13 * np.max(np.abs(old[name]))
        assert np.max(np.abs(new[name, 32] - old[name, 32])) <= 1e-5 * np.max(np.abs(old[name, 32]))
