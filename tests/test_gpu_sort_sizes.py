"""Ordering of selected states at the sizes where the sort changes its way: one, two and three keys, and
the last that one block sorts in shared memory with its neighbours (2,048 keys of one to three words, 512
of more).  The potential has one cubic term in mode 0, so a state with none of its quanta selects those
with one and three: two keys a source, apart from one pair for odd counts that has one or three."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sources(nm, count, rng):
    """Source states and whether they select, with exactly `count` selected states."""
    rest = np.unique(rng.integers(0, 6, (4 * count + 16, nm - 1)).astype(np.uint8), axis=0)
    rng.shuffle(rest)
    src, on = [], []
    if count == 1:  # the state with one quantum is there already, and silent
        src, on = [[0, *rest[0]], [1, *rest[0]]], [True, False]
    elif count % 2:  # 0 -> 1, 3 and 2 -> 1, 3, 5
        src, on = [[0, *rest[0]], [2, *rest[0]]], [True, True]
    for r in rest[1:1 + (count - (len(src) and (1 if count == 1 else 3))) // 2]:
        src.append([0, *r])
        on.append(True)
    return np.array(src, np.uint8), np.array(on)


@pytest.mark.parametrize("nm,count", [(nm, c) for nm in (6, 20, 40) for c in (1, 2, 3, 2047, 2048, 2049)] +
                         [(nm, c) for nm in (52, 128) for c in (1, 2, 511, 512, 513)])
def test_selected_states_ascend(nm, count):
    from vhci_b200 import VHCI
    rng = np.random.default_rng(1000 * nm + count)
    q, on = _sources(nm, count, rng)
    have, want = {x.tobytes() for x in q}, set()
    for x in q[on].astype(np.int16):
        for d in (-3, -1, 1, 3):
            t = x.copy()
            t[0] += d
            if t[0] >= 0 and t.astype(np.uint8).tobytes() not in have:
                want.add(t.astype(np.uint8).tobytes())
    assert len(want) == count
    with VHCI(problem=dict(freq=[1000.0 + 7.0 * i for i in range(nm)], cap=[8] * nm, ntot=1,
                           fcs=[((0, 0, 0), 12.0)], eps1=1.0, nstate=1, pt2=0)) as v:
        assert v.info.key_words == (nm + 15) // 16
        v.set_basis(q)
        C = np.zeros((len(q), 1), order="F")
        C[on, 0] = 1.0 / np.sqrt(len(q))
        v.set_vectors(C, np.zeros(1))
        s = v.select(1e-3)
    assert len(s) == count and {x.tobytes() for x in s} == want
    keys = [sum(int(v) << (4 * m) for m, v in enumerate(x)) for x in s]
    assert keys == sorted(keys)
