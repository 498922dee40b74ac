"""The Hamiltonian's count pass on both sides of where its presence bits are used (from 16,384 rows, up to
2^19 states): the matrix of n states and the one of n + 1, counted the other way, agree bit for bit on the
first n, both are symmetric to the bit, and sampled rows agree with sums over the force constants."""
import numpy as np
import pytest

from test_gpu_walk import host_entries

pytestmark = pytest.mark.gpu


def _states(nm, n, seed):
    """The n states of least quanta in all (neighbours lie in the basis), in no order."""
    q = np.stack(np.meshgrid(*[np.arange(9, dtype=np.uint8)] * nm, indexing="ij"), -1).reshape(-1, nm)
    q = q[np.argsort(q.sum(1), kind="stable")[:n]]
    return q[np.random.default_rng(seed).permutation(n)]


@pytest.mark.parametrize("n", [16383, 1 << 19])
def test_both_counts_agree(n):
    from vhci_b200 import VHCI
    nm = 7
    rng = np.random.default_rng(n)
    freq = [float(f) for f in np.sort(rng.uniform(500, 3300, nm))]
    fcs = [(tuple(int(m) for m in np.sort(rng.integers(0, nm, o))), float(30 * rng.standard_normal()))
           for o in (3,) * 6 + (4,) * 3]
    fcs = list(dict(fcs).items())
    q = _states(nm, n + 1, 7)
    H = []
    with VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=1, pt2=0)) as v:
        for m in (n, n + 1):
            v.set_basis(q[:m])
            v.build_h()
            H.append(v.h_csr())
            T = H[-1].T.tocsr()
            T.sort_indices()
            assert np.array_equal(T.indptr, H[-1].indptr) and np.array_equal(T.indices, H[-1].indices)
            assert np.array_equal(T.data, H[-1].data)
    cut = H[1][:n, :n]
    assert H[0].nnz > 20 * n
    assert np.array_equal(cut.indptr, H[0].indptr) and np.array_equal(cut.indices, H[0].indices)
    assert np.array_equal(cut.data, H[0].data)
    rows = rng.choice(n, 64, replace=False)
    want = host_entries(freq, fcs, q[rows], q[:n])
    got = {}
    for a, i in enumerate(rows):
        for e in range(H[0].indptr[i], H[0].indptr[i + 1]):
            if H[0].indices[e] != i:
                got[a, int(H[0].indices[e])] = H[0].data[e]
    assert set(got) == {x for x in want if rows[x[0]] != x[1]}
    # products of at most four ladder factors and a coefficient, at most 24 terms of either sign
    size = max(abs(x) for x in want.values())
    assert max(abs(got[x] - want[x]) for x in got) <= 64 * 2.0 ** -53 * 24 * size
