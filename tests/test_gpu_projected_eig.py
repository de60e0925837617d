"""The projected eigenproblem solved from size to size (lowest_eig_warm_cta):
solves whose subspace passes the sizes where its layout changes (32, 64, 96,
128 rows per thread split; the matrix leaves shared memory at 128; the full
solver takes over past 220), a nearly degenerate lowest pair, and restarts of
the mixed form on one.  Reference: numpy's dense eigensolver.

Tolerances, before any run: the residual r bounds the energy error by r^2 /
gap and the vector's by r / gap; with r < 1e-9 that is below 1e-10 for every
matrix here and 1e-9 / gap."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(pkg):
    pkg.build.build()
    c = pkg.capi.Context(0)
    yield c
    c.close()


def _csr(A):
    n = len(A)
    rows, cols = np.nonzero(A)
    return np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]), cols, A[rows, cols]


def _chain(n, disorder, seed):
    """Hopping on a ring with weak disorder: the diagonal preconditioner does
    little, so the subspace grows long."""
    rng = np.random.default_rng(seed)
    A = np.diag(disorder * rng.normal(size=n))
    for i in range(n):
        A[i, (i + 1) % n] = A[(i + 1) % n, i] = -1.0
    return A


@pytest.mark.parametrize("n,disorder,seed", [(40, 0.3, 1), (70, 0.3, 2), (130, 0.2, 3), (300, 0.2, 4), (700, 0.05, 5)])
def test_long_subspaces(ctx, pkg, oracle, n, disorder, seed):
    """Converges where the reference's algorithm does, in as many iterations;
    the longest chain needs more than 254 vectors and neither converges."""
    A = _chain(n, disorder, seed)
    ctx.set_csr(*_csr(A))
    w, U = np.linalg.eigh(A)
    try:
        _, _, its = oracle.csr_from_arrays(*_csr(A)).selected_ci_diag(max_m=min(n, 254), tol=1e-9)
    except RuntimeError:
        with pytest.raises(pkg.capi.NotConverged):
            ctx.davidson(max_m=min(n, 254), tol=1e-9)
        return
    E, C, info = ctx.davidson(max_m=min(n, 254), tol=1e-9)
    gap = w[1] - w[0]
    assert abs(info["iterations"] - its) <= 1
    assert info["residual_norm"] < 1e-9
    assert abs(E - w[0]) < 1e-10
    assert np.linalg.norm(C * np.sign(C @ U[:, 0]) - U[:, 0]) < 4e-9 / gap + 1e-9


def test_nearly_degenerate_pair(ctx):
    """Two lowest states 1e-4 apart: the vector to 1e-9 / gap, and no warm step
    that stops at the pair's sum."""
    rng = np.random.default_rng(6)
    n = 400
    Q, _ = np.linalg.qr(np.eye(n) + 0.02 * rng.normal(size=(n, n)))
    A = (Q * np.concatenate([[-3.0, -2.9999], np.linspace(-1, 5, n - 2)])) @ Q.T
    A = (A + A.T) / 2
    ctx.set_csr(*_csr(A))
    w, U = np.linalg.eigh(A)
    E, C, _ = ctx.davidson(max_m=254, tol=1e-9)
    assert abs(E - w[0]) < 1e-10
    assert np.linalg.norm(C * np.sign(C @ U[:, 0]) - U[:, 0]) < 4e-9 / (w[1] - w[0])


@pytest.mark.parametrize("seed", [9, 11, 16])
def test_mixed_restarts_keep_their_pace(ctx, pkg, seed):
    """Mixed solves of CASCI(9e,11o) problems with a small gap: the restarted
    basis holds the Ritz vector itself, so the iteration count stays near the
    FP64 solve's (within a half; the FP32 form adds a few iterations per
    restart)."""
    capi = pkg.capi
    T, V, _ = pkg.integrals.synthetic_integrals(11, 22, 1000003 * seed)
    E64, _, i64 = ctx.casci(T, V, 5, 4, tol=1e-10, precision=capi.PREC_FP64)
    E32, _, i32 = ctx.casci(T, V, 5, 4, tol=1e-10, precision=capi.PREC_MIXED)
    assert abs(E64 - E32) < 1e-10
    assert i32["iterations"] <= 1.5 * i64["iterations"]
