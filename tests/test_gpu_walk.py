"""The connection walk at its edges: rows with no hit, with fewer than one warp round and with many
rounds of hits; row sets on both sides of the sampled reservation; more connections than the kept
batches hold (the second walk takes over); potentials whose groups are all visited because the state
has many excited modes.  The Hamiltonian of each basis is compared entry by entry with sums over the
force constants on the host, and the PT2 sums with the same sums over the selected perturbers."""
import itertools
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def elements(freq, fcs):
    """Change patterns {quanta change: [(coefficient, [(mode, power, change)])]} of the potential."""
    out = {}
    for ms, v in fcs:
        modes = sorted(set(ms))
        pw = [ms.count(m) for m in modes]
        c = v / math.sqrt(2.0 ** len(ms)) / math.prod(math.factorial(p) for p in pw)
        for d in itertools.product(*[range(-p, p + 1, 2) for p in pw]):
            key = tuple((m, x) for m, x in zip(modes, d) if x)
            out.setdefault(key, []).append((c, list(zip(modes, pw, d))))
    return out


def ladder(size=40):
    up = np.diag(np.sqrt(np.arange(1.0, size)), 1)
    p = [np.eye(size)]
    for _ in range(6):
        p.append(p[-1] @ (up + up.T))
    return p


def host_entries(freq, fcs, q, target):
    """{(i, j): H_ij} between the states q (i) and `target` (j), i's own state left out."""
    P, found = ladder(), elements(freq, fcs)
    where = {s.tobytes(): j for j, s in enumerate(target.astype(np.int16))}
    out = {}
    for i, s in enumerate(q.astype(np.int16)):
        for key, terms in found.items():
            if not key:
                continue
            t = s.copy()
            for m, x in key:
                t[m] += x
            j = where.get(t.tobytes())
            if j is not None:
                out[i, j] = sum(c * math.prod(P[p][s[m], s[m] + x] for m, p, x in parts) for c, parts in terms)
    return out


def problem(nm, seed, share):
    rng = np.random.default_rng(seed)
    freq = [float(f) for f in np.sort(rng.uniform(500, 3300, nm))]
    fcs = []
    for order, scale in ((3, 30.0), (4, 8.0)):
        for ms in itertools.combinations_with_replacement(range(nm), order):
            if rng.random() < share:
                fcs.append((ms, float(scale * rng.standard_normal())))
    return freq, fcs


def make(nm, seed, share, nstate=4):
    from vhci_b200 import VHCI
    freq, fcs = problem(nm, seed, share)
    v = VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=nstate, pt2=1))
    return v, freq, fcs


def states(nm, n, seed, p):
    rng = np.random.default_rng(seed)
    q = np.unique(rng.binomial(6, p, (4 * n, nm)).astype(np.uint8), axis=0)
    rng.shuffle(q)
    return q[:n]


# 20 modes need two key words, 33 three; p = 0.55 leaves nearly every mode excited
@pytest.mark.parametrize("nm,n,p", [(4, 40, 0.3), (6, 700, 0.3), (10, 300, 0.55), (20, 250, 0.06),
                                    (33, 250, 0.03)])
def test_hamiltonian_entries(nm, n, p):
    v, freq, fcs = make(nm, nm, 0.5 if nm <= 10 else 0.05)
    q = states(nm, n, 7 * nm, p)
    with v:
        v.set_basis(q)
        H = v.h_csr().tocoo()
    got = {(i, j): x for i, j, x in zip(H.row, H.col, H.data) if i != j}
    ref = host_entries(freq, fcs, q, q)
    assert set(got) == set(ref)
    # products of at most four ladder factors and a coefficient, at most 24 terms of either sign
    size = max(abs(x) for x in ref.values())
    assert max(abs(got[k] - ref[k]) for k in ref) <= 64 * 2.0 ** -53 * 24 * size


def test_isolated_states_have_empty_rows():
    v, freq, fcs = make(8, 3, 0.5)
    q = np.zeros((6, 8), np.uint8)
    for i in range(6):
        q[i, i] = 6 + i  # far from one another: no force constant connects them
    with v:
        v.set_basis(q)
        assert v.build_h() == 6
        H = v.h_csr()
    assert H.nnz == 6


def test_kept_batches_match_second_walk():
    """4,096 rows take the fixed reservation of 256 connections a row, 4,097 the sampled one; a full
    small-mode basis has more a row, so the fixed reservation overflows and the entries come
    from the second walk.  Both must hold the same matrix on the states they share."""
    v, freq, fcs = make(6, 5, 1.0)
    q = np.array([s for s in itertools.product(range(5), repeat=6)], np.uint8)
    q = q[np.argsort(q.sum(1), kind="stable")][:4097]
    with v:
        v.set_basis(q)
        A = v.h_csr()
        v.set_basis(q[:4096])
        B = v.h_csr()
    assert np.diff(B.indptr).mean() > 256
    A = A[:4096, :4096]
    A.sort_indices()
    B.sort_indices()
    assert np.array_equal(A.indptr, B.indptr) and np.array_equal(A.indices, B.indices)
    assert np.array_equal(A.data, B.data)


@pytest.mark.parametrize("chunk", [0, 1 << 20])
@pytest.mark.parametrize("nm,n,k", [(6, 120, 3), (20, 60, 33)])
def test_pt2_sums(nm, n, k, chunk):
    from vhci_b200 import VHCI
    freq, fcs = problem(nm, nm + 1, 0.5 if nm <= 10 else 0.05)
    q = states(nm, n, nm, 0.25 if nm <= 10 else 0.06)
    rng = np.random.default_rng(2)
    C = np.asfortranarray(rng.standard_normal((n, k)) / math.sqrt(n))
    E = 0.5 * sum(freq) - np.linspace(4000.0, 2000.0, k)  # well below every perturber
    with VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=k, pt2=1),
              pt2_chunk=chunk) as v:
        v.set_basis(q)
        v.set_vectors(C, E)
        a = v.select(0.5)
        dE, n_pert = v.pt2(0.5)
        v.set_basis(a)
        Ea = v.h_csr().diagonal()
    assert n_pert == len(a) > 0
    num = np.zeros((n_pert, k))
    for (i, j), h in host_entries(freq, fcs, q, a).items():
        num[j] += h * C[i]
    ref = (num ** 2 / (E - Ea[:, None])).sum(0)
    assert np.abs(dE - ref).max() <= 1e-12 * np.abs(ref).max()


def test_pt2_chunks():
    """More entries than one chunk holds: the rows of every chunk are filled and ordered by themselves."""
    from vhci_b200 import VHCI
    nm, n, k = 10, 4000, 7
    freq, fcs = problem(nm, 4, 0.8)
    q = states(nm, n, 5, 0.25)
    rng = np.random.default_rng(6)
    C = np.asfortranarray(rng.standard_normal((n, k)) / math.sqrt(n))
    E = 0.5 * sum(freq) - np.linspace(4000.0, 2000.0, k)
    out = []
    for chunk in (0, 1 << 20):
        with VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=k, pt2=1),
                  pt2_chunk=chunk) as v:
            v.set_basis(q)
            v.set_vectors(C, E)
            out.append(v.pt2(0.02))
            entries = v.stats()["pt2_entries"]
    assert entries > 2 << 20  # three chunks at least
    assert out[0][1] == out[1][1]
    # the same rows, summed over the perturbers in another grouping
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-12 * np.abs(out[0][0]).max()
