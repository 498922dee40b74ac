"""The block Lanczos at its edges, against a dense eigensolve of the same matrix: bases barely larger
than the subspace (the host factorisation of a block) and several times larger (the device one),
subspaces that are no multiple of the block or of an eight-row tile, one wanted state and many, warm
starts, FP64 and FP32 storage.

Tolerance: a converged pair has ||H x - theta x|| <= 1e-10 |theta|, and its eigenvalue is within that
residual of an eigenvalue of H (symmetric), so |dE| <= 1e-10 |E| plus the dense solver's rounding,
n 2^-53 ||H||.  With FP32 products the residual bound is 1e-7 of the spectrum's scale and the final
FP64 sweep brings the values to second order in it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(n, k, precision, seed=3, nm=8):
    from vhci_b200 import VHCI
    rng = np.random.default_rng(seed)
    freq = [float(f) for f in np.sort(rng.uniform(500, 3300, nm))]
    fcs = [((i, j, l), float(40 * rng.standard_normal())) for i in range(nm) for j in range(i, nm)
           for l in range(j, nm)]
    fcs += [((i, i, i, i), 60.0) for i in range(nm)]
    q = np.unique(rng.binomial(5, 0.15, (8 * n, nm)).astype(np.uint8), axis=0)
    q = q[np.argsort(q @ np.array(freq), kind="stable")][:n]
    assert len(q) == n
    v = VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=k, pt2=0),
             precision=precision)
    v.set_basis(q)
    return v


@pytest.mark.parametrize("n,k,precision", [
    (2001, 1, 0), (2001, 37, 0), (2003, 150, 0), (2600, 100, 0), (3333, 7, 0), (4001, 64, 0), (4001, 61, 0),
    (3003, 200, 0), (2001, 37, 1), (3333, 64, 1)])
def test_lowest_states(n, k, precision):
    with context(n, k, precision) as v:
        H = v.h_csr()
        w = np.linalg.eigvalsh(H.toarray())
        bound = 1e-10 * np.abs(w[:k]) + n * 2.0 ** -53 * np.abs(w).max()
        if precision == 1:
            gap = 1e-7 * np.abs(w).max()
            bound = bound + gap
        for _ in range(2):  # cold, then from the vectors held
            E = v.eigs(k)
            assert (np.abs(E - w[:k]) <= bound).all(), np.abs(E - w[:k]).max()
        C, E = v.vectors(k)
        # orthonormal to the rounding of two Gram-Schmidt passes and the rotations
        assert np.abs(C.T @ C - np.eye(k)).max() <= 1e-11


@pytest.mark.parametrize("n,k", [(9001, 301), (9002, 61), (1203, 5)])
def test_subspace_widths(n, k):
    """Subspaces of several slabs of the projections' columns, with blocks that begin past a 32-byte
    boundary after a restart (wanted counts that are no multiple of four), and the narrowest ones: the
    same matrix through the eigensolver and a dense eigensolve; tolerance as above."""
    with context(n, k, 0) as v:
        H = v.h_csr()
        w = np.linalg.eigvalsh(H.toarray())[:k] if n < 4000 else None
        E = v.eigs(k)
        C, _ = v.vectors(k)
        scale = np.abs(H).sum(1).max()
        # ||H c - E c|| <= 1e-10 |E| for a converged pair, plus the rounding of the product here
        R = H @ C - C * E
        assert (np.linalg.norm(R, axis=0) <= 1e-10 * np.abs(E) + 64 * 2.0 ** -53 * scale).all()
        assert np.abs(C.T @ C - np.eye(k)).max() <= 1e-11
        if w is not None:
            assert (np.abs(E - w) <= 1e-10 * np.abs(w) + n * 2.0 ** -53 * scale).all()
