"""The complete-space RDMs' kept lists: one context over changing spaces and
capped memory, the one-transition sweep of spaces whose four staged rows do
not fit (8,008 beta strings), odd chunk lengths (an odd count of alpha
transitions per class).  Reference: the pair walk (QDKGB_RDM_PAIR_WALK=1) of
the same vectors.  Tolerance, before any run: sums of at most N products of a
normalised vector, N 2^-53 of 1: 1e-11 for the largest space here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(pkg):
    pkg.build.build()
    c = pkg.capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shapes,cap", [([(6, 3, 2), (7, 2, 4), (7, 1, 1), (6, 3, 2)], False),
                                        ([(8, 3, 4), (5, 4, 1)], True), ([(16, 1, 6)], False)])
def test_rdms_over_changing_spaces(ctx, pkg, monkeypatch, shapes, cap):
    capi = pkg.capi
    ctx.set_device_limit(ctx.device_bytes() + (64 << 20) if cap else 0)
    for k, (n, na, nb) in enumerate(shapes):
        T, V, _ = pkg.integrals.synthetic_integrals(n, 4, seed=k)
        a, b = capi.fci_dets(n, na, nb)
        ctx.set_integrals(T, V)
        ctx.set_dets(a, b)
        C = np.random.default_rng(k).normal(size=len(a))
        C /= np.linalg.norm(C)
        monkeypatch.setenv("QDKGB_RDM_PAIR_WALK", "1")
        want = ctx.rdms_spin_dep(C)
        monkeypatch.setenv("QDKGB_RDM_PAIR_WALK", "0")
        for keys in (("aa", "bb", "aaaa", "bbbb", "aabb"), ("aabb",), ("bb",)):
            got = ctx.rdms_spin_dep(C, want=keys)
            assert set(got) == set(keys)
            for key in keys:
                assert np.max(np.abs(got[key] - want[key])) <= 1e-11, (n, na, nb, key)
    ctx.set_device_limit(0)
