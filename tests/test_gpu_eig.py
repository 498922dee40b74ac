"""The small dense eigensolver through the dense path (bases up to 2,000 states), against LAPACK: one
state, sizes on both sides of every cluster, grid and register form and beyond the largest, all
eigenvectors wanted, and spectra it has to hand on to the library's solver (exactly degenerate states).

Tolerance: both solvers are backward stable, so an eigenvalue is within a few n 2^-53 ||H|| of the
exact one; the vectors' residuals are held to the same size and their orthonormality to n 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def check(v, k):
    H = v.h_csr().toarray()
    n, nrm = len(H), np.abs(np.linalg.eigvalsh(H)).max()
    k = min(k, n)
    E = v.eigs(k)
    C, e = v.vectors(k)
    ref = np.linalg.eigvalsh(H)[:k]
    assert np.array_equal(E[:k], e)
    assert np.abs(E[:k] - ref).max() <= 8 * n * U * nrm
    assert np.linalg.norm(H @ C - C * E[:k], axis=0).max() <= 32 * n * U * nrm
    assert np.abs(C.T @ C - np.eye(k)).max() <= 32 * n * U


def make(n, nstate, seed, nm=7, couple=1.0):
    from vhci_b200 import VHCI
    rng = np.random.default_rng(seed)
    freq = [float(f) for f in np.sort(rng.uniform(500, 3300, nm))]
    fcs = [((i, j, l), float(couple * 40 * rng.standard_normal())) for i in range(nm) for j in range(i, nm)
           for l in range(j, nm)] + [((i,) * 4, 60.0) for i in range(nm)]
    v = VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=nstate, pt2=0))
    q = np.unique(rng.binomial(5, 0.25, (20 * n + 100, nm)).astype(np.uint8), axis=0)
    rng.shuffle(q)
    v.set_basis(q[:n])
    return v


@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (3, 1), (5, 5), (28, 10), (64, 64), (65, 7), (127, 40), (129, 129),
                                 (255, 100), (257, 30), (383, 20), (385, 385), (513, 64), (639, 10), (640, 640),
                                 (641, 10), (700, 70), (1184, 20), (1185, 5), (1500, 150), (1799, 12), (1801, 3)])
def test_dense_eigenpairs(n, k):
    with make(n, k, n) as v:
        check(v, k)


def test_degenerate_states():
    """Two equal modes without coupling between modes: every level with both excited comes in pairs
    that no vector iteration on single eigenvalues can tell apart."""
    from vhci_b200 import VHCI
    import itertools
    freq = [1000.0, 1000.0, 1500.0]
    fcs = [((m, m, m, m), 50.0) for m in (0, 1)] + [((2, 2, 2), 30.0)]
    q = np.array([s for s in itertools.product(range(5), repeat=3)], np.uint8)
    with VHCI(problem=dict(freq=freq, cap=[8] * 3, ntot=1, fcs=fcs, eps1=0.0, nstate=60, pt2=0)) as v:
        v.set_basis(q)
        check(v, 60)


def test_diagonal_matrix():
    """No coupling at all: already tridiagonal, every reflector is the identity."""
    from vhci_b200 import VHCI
    q = np.eye(6, dtype=np.uint8) * np.arange(3, 9, dtype=np.uint8)[:, None]
    freq = [700.0, 900.0, 1300.0, 1700.0, 2300.0, 3100.0]
    fcs = [((m, m, m, m), 1.0 + m) for m in range(6)]
    with VHCI(problem=dict(freq=freq, cap=[8] * 6, ntot=1, fcs=fcs, eps1=0.0, nstate=4, pt2=0)) as v:
        v.set_basis(q)
        check(v, 4)
