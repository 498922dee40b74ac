"""Device memory that runs out, at every reservation of a call in turn (injected on the host: the n-th
reservation of the calling thread reports a lack of memory; nothing runs out on the device).  The call
either ends with the out-of-memory status or gets by without that buffer, with the same result; a second
call, with memory to be had again, succeeds; and a destroyed context leaves nothing behind in the pool,
however its calls ended.

Results are compared exactly where the failed reservation cannot change the arithmetic (the matrix), to
the eigensolver's stopping rule for eigenvalues (|dE| <= 1e-10 |E| a run, twice that between two) and to
the rounding of sums in another order for the rest."""
import ctypes

import numpy as np
import pytest

from test_resources import _pool_used

pytestmark = pytest.mark.gpu


def fail_alloc(first, count=1):
    """Reservations first .. first + count - 1 of this thread fail from here on; returns how many there
    were since the last call."""
    from vhci_b200 import api
    f = api.lib().vhci_test_fail_alloc
    f.restype = ctypes.c_int64
    f.argtypes = [ctypes.c_int64, ctypes.c_int64]
    return f(first, count)


def _context(n, k, precision=0, nm=9, pt2_chunk=0):
    from vhci_b200 import VHCI
    rng = np.random.default_rng(n)
    freq = [float(f) for f in np.sort(rng.uniform(500, 3300, nm))]
    fcs = [((i, j, l), float(40 * rng.standard_normal())) for i in range(nm) for j in range(i, nm)
           for l in range(j, nm)]
    fcs += [((i, i, i, i), 60.0) for i in range(nm)]
    q = np.unique(rng.binomial(6, 0.2, (12 * n, nm)).astype(np.uint8), axis=0)
    q = q[np.argsort(q @ np.array(freq), kind="stable")][:n]
    assert len(q) == n
    v = VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=0.0, nstate=k, pt2=1),
             precision=precision, pt2_chunk=pt2_chunk)
    v.set_basis(q)
    return v


def _set_vectors(v, k):
    rng = np.random.default_rng(5)
    C, _ = np.linalg.qr(rng.standard_normal((v.n, k)))
    E = np.linspace(1000.0, 2000.0, k)
    v.set_vectors(C, E)


def _matrix(v):
    H = v.h_csr()
    return [H.indptr, H.indices, H.data]


def _exact(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _values(a, b):
    return (np.abs(a - b) <= 2e-10 * np.abs(b)).all()


def _sums(a, b):  # sums of up to 1e5 products in another order, or one more rounding
    return np.abs(a - b).max() <= 1e5 * 2.0 ** -53 * np.abs(b).max()


def _build(v):
    v.build_h()


def _append(v):
    _set_vectors(v, 2)
    v.build_h()
    v.select(0.5, append=True)
    assert v.n > 6001


def _x(v, k):
    return np.random.default_rng(3).standard_normal((v.n, k))


CASES = {
    # states, wanted, options, preparation, the call, what it returns, comparison
    "build": (17001, 2, {}, None, _build, _matrix, _exact),
    "build_small": (3001, 2, {}, None, _build, _matrix, _exact),
    "build_f32": (17001, 2, dict(precision=1), None, _build, _matrix, _exact),
    "build_appended": (6001, 2, {}, _append, _build, _matrix, _exact),
    "eigs": (3333, 4, {}, _build, lambda v: v.eigs(4), lambda v: v.energies(), _values),
    "eigs_f32": (3333, 4, dict(precision=1), _build, lambda v: v.eigs(4), lambda v: v.energies(), None),
    "eigs_dense": (701, 20, {}, _build, lambda v: v.eigs(20), lambda v: v.energies(), _values),
    "pt2": (6001, 4, {}, lambda v: _set_vectors(v, 4), lambda v: v.pt2(0.05), lambda v: v.energies(), _sums),
    "pt2_chunks": (6001, 4, dict(pt2_chunk=1), lambda v: _set_vectors(v, 4), lambda v: v.pt2(0.05),
                   lambda v: v.energies(), _sums),
    "select": (6001, 4, {}, lambda v: _set_vectors(v, 4), lambda v: v.select(0.05),
               lambda v: v.select(0.05), None),
    "apply": (6001, 2, {}, _build, lambda v: v.apply_h(_x(v, 3)), lambda v: v.apply_h(_x(v, 3)), _sums),
    "residuals": (6001, 2, {}, _build, lambda v: v.residual_norms(_x(v, 3), np.ones(3)),
                  lambda v: v.residual_norms(_x(v, 3), np.ones(3)), _sums),
    "vectors": (6001, 3, {}, lambda v: _set_vectors(v, 3), lambda v: v.vectors(), lambda v: v.vectors()[0],
                _sums),
}


@pytest.mark.parametrize("name", CASES)
def test_every_reservation_may_fail(name):
    from vhci_b200 import api
    n, k, opts, prep, call, result, same = CASES[name]

    def run(first):
        """(status, result after a second call when the first ran out, reservations of the call)"""
        with _context(n, k, **opts) as v:
            if prep:
                prep(v)
            fail_alloc(first)
            code = api.OK
            try:
                call(v)
            except api.VhciError as e:
                code = e.code
            seen = fail_alloc(0, 0)
            if code != api.OK:
                if name.startswith("pt2"):  # energies that PT2 has not touched
                    _set_vectors(v, 4)
                call(v)
            return code, result(v), seen

    code, ref, total = run(0)
    assert code == api.OK and total >= {"pt2": 15, "pt2_chunks": 15, "select": 5}.get(name, 1)
    run(0)
    base = _pool_used()
    out = []
    for first in range(1, total + 1):
        code, got, seen = run(first)
        assert code in (api.OK, api.E_OOM), (first, code)
        out.append(code)
        if same is not None:
            assert same(got, ref), first
        elif name == "eigs_f32":
            assert np.abs(got - ref).max() <= 1e-7 * np.abs(ref).max(), first
        else:
            assert {x.tobytes() for x in got} == {x.tobytes() for x in ref}, first
        assert _pool_used() == base, (first, code)
    print(name, total, "reservations,", out.count(api.OK), "done without")


# What a build cannot do without: the row counts and pointers, the scan's scratch.  Everything else is
# there to make it faster, or can be had once that is given back.
@pytest.mark.parametrize("name", ["build", "build_small", "build_f32"])
def test_build_gives_way(name):
    from vhci_b200 import api
    n, k, opts, _, call, result, same = CASES[name]
    with _context(n, k, **opts) as v:
        fail_alloc(0, 0)
        call(v)
        total, ref = fail_alloc(0, 0), result(v)
    out = []
    for first in range(1, total + 1):
        with _context(n, k, **opts) as v:
            fail_alloc(first)
            try:
                call(v)
            except api.VhciError as e:
                assert e.code == api.E_OOM
                out.append(first)
            fail_alloc(0, 0)
            if first not in out:
                assert same(result(v), ref), first
    assert len(out) <= 3, (out, total)


def test_matrix_that_cannot_be_had_is_refused_with_its_size():
    """All reservations from the matrix's first on fail: the refusal states what was needed."""
    from vhci_b200 import api
    n, k, opts, _, call, _, _ = CASES["build_small"]
    said = []
    for first in range(1, 10):
        with _context(n, k, **opts) as v:
            fail_alloc(first, 100)
            with pytest.raises(api.VhciError) as e:
                call(v)
            fail_alloc(0, 0)
            assert e.value.code == api.E_OOM
            said.append("GB for the eigensolver" in str(e.value))
    assert any(said)


def _pt2_context(chunk):
    v = _context(6001, 4, pt2_chunk=chunk)
    _set_vectors(v, 4)
    return v


@pytest.mark.parametrize("chunk", [0, 1])
def test_pt2_gives_way(chunk):
    """PT2 with a reservation that fails, and from the first chunk's buffers on with several in a row: the
    kept connections go, then the perturbers are taken in smaller chunks.  Only what comes before the
    first chunk (the selection, the perturbers' table, the entry counts and the columns' sums) cannot be
    done without."""
    from vhci_b200 import api

    def run(first, count):
        with _pt2_context(chunk) as v:
            fail_alloc(first, count)
            try:
                v.pt2(0.05)
            except api.VhciError as e:
                assert e.code == api.E_OOM
                return None, fail_alloc(0, 0)
            return v.energies(), fail_alloc(0, 0)

    ref, total = run(0, 0)
    with _pt2_context(chunk) as v:
        v.pt2(0.05)
        assert v.stats()["pt2_entries"] > 1 << 20  # more than the smallest chunk
    needed = [first for first in range(1, total + 1) if run(first, 1)[0] is None]
    assert total - needed[-1] >= 6, (needed, total)  # the chunk's buffers
    for count in (1, 2, 5):
        for first in range(needed[-1] + 1, total + 1):
            got, _ = run(first, count)
            assert got is not None and _sums(got, ref), (first, count)


@pytest.mark.parametrize("name,needed", [("eigs", 0), ("eigs_f32", 0), ("eigs_dense", 3)])
def test_eigensolver_gives_way(name, needed):
    """Any one buffer of the block Lanczos: the memory-lean variant has the eigenvalues.  The dense solver
    cannot do without the matrix, the values and the vectors it returns, and leaves the rest to the
    library's, which works in place."""
    from vhci_b200 import api
    n, k, opts, prep, call, result, same = CASES[name]

    def run(first):
        with _context(n, k, **opts) as v:
            prep(v)
            fail_alloc(first)
            try:
                call(v)
            except api.VhciError as e:
                assert e.code == api.E_OOM
                return None, fail_alloc(0, 0)
            seen = fail_alloc(0, 0)
            return result(v), seen

    ref, total = run(0)
    out = []
    for first in range(1, total + 1):
        got, _ = run(first)
        if got is None:
            out.append(first)
        else:
            tol = 1e-7 * np.abs(ref).max() if same is None else 2e-10 * np.abs(ref)
            assert (np.abs(got - ref) <= tol).all(), first
    assert len(out) <= needed, (out, total)


@pytest.mark.parametrize("name,needed", [("apply", 2), ("residuals", 4), ("vectors", 0), ("set_vectors", 1)])
def test_transfers_give_way(name, needed):
    """Vectors between host and device need the device's copy of them (and residuals their sums), no more."""
    from vhci_b200 import api
    n, k, opts, prep, call, result, same = CASES["vectors" if name == "set_vectors" else name]
    if name == "set_vectors":
        prep, call = None, lambda v: _set_vectors(v, 3)

    def run(first):
        with _context(n, k, **opts) as v:
            if prep:
                prep(v)
            fail_alloc(first)
            try:
                got = call(v)
            except api.VhciError as e:
                assert e.code == api.E_OOM
                return None, fail_alloc(0, 0)
            seen = fail_alloc(0, 0)
            return result(v) if name == "set_vectors" else (got[0] if name == "vectors" else got), seen

    ref, total = run(0)
    out = []
    for first in range(1, total + 1):
        got, _ = run(first)
        if got is None:
            out.append(first)
        elif "vectors" in name:
            assert np.array_equal(got, ref), first  # copies
        else:
            assert _sums(got, ref), first
    assert len(out) <= needed and total > needed, (out, total)
