"""The FP64 solver's second Gram-Schmidt pass, made only where the first took
more than half of |w|^2: matrices whose preconditioner turns every direction
into a vector that the basis holds already (a diagonal element next to the
lowest eigenvalue), and some where no second pass is due, at sizes from one to
many row tiles; and the mixed solver's test of its guess's spin-flip sector on
such sizes.  Reference: numpy's dense eigensolver, the CPU oracle.

Tolerances, before any run: a residual r < 1e-9 puts the energy within r^2 /
gap < 1e-10 and the vector within r / gap of the matrix's, both with a factor
of four."""
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


def _matrix(n, close, seed):
    rng = np.random.default_rng(seed)
    A = 0.2 / np.sqrt(n) * rng.normal(size=(n, n))
    A = (A + A.T) / 2
    A[np.diag_indices(n)] = np.linspace(0.0, 4.0, n)
    if close is not None:
        A[1, :] = A[:, 1] = 0.0
        low = np.linalg.eigvalsh(np.delete(np.delete(A, 1, 0), 1, 1))[0]
        A[1, :] = A[:, 1] = 1e-3 * rng.normal(size=n)
        A[1, 1] = low + close
    return A


@pytest.mark.parametrize("n", [3, 60, 513, 1500])
@pytest.mark.parametrize("close", [None, 0.05, 0.01])
def test_directions_inside_the_basis(ctx, n, close):
    A = _matrix(n, close, n)
    ctx.set_csr(*_csr(A))
    w, U = np.linalg.eigh(A)
    E, C, info = ctx.davidson(max_m=min(n, 200), tol=1e-9)
    gap = w[1] - w[0]
    assert info["residual_norm"] < 1e-9
    assert abs(E - w[0]) < 4e-10
    assert abs(C @ C - 1) < 1e-12
    assert np.linalg.norm(C * np.sign(C @ U[:, 0]) - U[:, 0]) < 4e-9 / gap


@pytest.mark.parametrize("norb,n_e", [(4, 2), (6, 3), (7, 3)])
@pytest.mark.parametrize("sign", [1, -1])
def test_guess_sector(ctx, pkg, oracle, norb, n_e, sign):
    """A guess of either spin-flip parity in the mixed form: the lowest state
    of that parity, with a vector that has it."""
    T, V, _ = pkg.integrals.synthetic_integrals(norb, 2 * norb, 31 + norb)
    a, b = pkg.determinants.fci_space(norb, n_e, n_e)
    H = oracle.Hamiltonian(T, V)
    N = len(a)
    ptr, col, val = oracle.build_csr(H, a, b).arrays()
    D = np.zeros((N, N))
    D[np.repeat(np.arange(N), np.diff(ptr)), col] = val
    s = int(round(np.sqrt(N)))
    P = np.arange(N).reshape(s, s).T.ravel()
    rng = np.random.default_rng(norb)
    d = np.diag(D)
    g = np.exp(-(d - d.min())) * (1 + 0.1 * rng.normal(size=N))
    g = g + sign * g[P]
    g /= np.linalg.norm(g)
    lam, U = np.linalg.eigh((np.eye(N) + sign * np.eye(N)[P]) / 2)
    U = U[:, lam > 0.5]
    ref = np.linalg.eigvalsh(U.T @ D @ U)[0]
    ctx.set_integrals(T, V)
    ctx.set_dets(a, b)
    ctx.build_hamiltonian(storage=pkg.capi.H_SPLIT32)
    E, C, info = ctx.davidson(guess=g, tol=1e-8, precision=pkg.capi.PREC_MIXED)
    assert abs(E - ref) < 1e-10
    assert np.linalg.norm(C - sign * C[P]) < 1e-6
