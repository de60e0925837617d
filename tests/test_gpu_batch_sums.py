"""Sums of the lockstep batched solver (eight basis columns at a time, the last
CTA of an instance adding the partial sums) and its projected problems solved
from size to size: subspaces on either side of eight and sixteen columns,
instances of fewer rows than a CTA takes, of one CTA and of several, against
the oracle's FP64 Davidson.  FP64 form at 1e-10 Eh (residual 1e-9), mixed form
at 1e-8 Eh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4, 1, 2), (6, 3, 3), (8, 4, 4), (8, 4, 3), (7, 4, 3), (6, 3, 3)]


@pytest.fixture(scope="module")
def capi(pkg):
    pkg.build.build()
    return pkg.capi


@pytest.fixture(scope="module")
def ctx(capi):
    c = capi.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def cases(pkg, oracle):
    out = []
    for i, (norb, na, nb) in enumerate(SHAPES):
        T, V, _ = pkg.integrals.synthetic_integrals(norb, 2 * norb, 910 + i)
        a, b = pkg.determinants.fci_space(norb, na, nb)
        M = oracle.build_csr(oracle.Hamiltonian(T, V), a, b)
        E, X, _ = M.selected_ci_diag(tol=1e-10)
        R = oracle.rdms_spin_dep(norb, a, b, X)
        out.append(((norb, na, nb, T, V), E, R["aa"] + R["bb"]))
    return out


@pytest.mark.parametrize("max_subspace", [8, 9, 16, 17, 33])
@pytest.mark.parametrize("form", ["mixed", "fp64"])
def test_batched_sums_at_column_edges(ctx, capi, cases, max_subspace, form):
    mixed = form == "mixed"
    E, R, its, _ = capi.casci_batch(ctx, [q for q, _, _ in cases], res_tol=1e-8 if mixed else 1e-9,
                                    max_subspace=max_subspace, persistent=0,
                                    **({} if mixed else {"precision": capi.PREC_FP64}))
    for i, (_, Eo, Ro) in enumerate(cases):
        assert abs(E[i] - Eo) < (1e-8 if mixed else 1e-10), (i, E[i], Eo)
        np.testing.assert_allclose(R[i], Ro, atol=1e-6, rtol=0, err_msg=str(i))
