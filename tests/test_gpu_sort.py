"""Ordering of selected states (packed keys of one to three words) on both sides of the size that one
block sorts in shared memory: ascending keys, no state lost or doubled, same set as a host selection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm,count", [(6, 1), (6, 2), (6, 31), (12, 700), (12, 2047), (12, 2048), (12, 2049),
                                      (20, 1500), (20, 2048), (20, 2600), (40, 2048), (40, 2300)])
def test_selected_states_ascend(nm, count):
    """Linear couplings only: at threshold eps a state i selects every i +- 1 quantum in the modes whose
    |c_i fc| reaches it, so `count` single excitations out of a chain are selected."""
    from vhci_b200 import VHCI
    freq = [1000.0 + 7.0 * i for i in range(nm)]
    fcs = [((m, m, m), 12.0) for m in range(nm)]
    rng = np.random.default_rng(count)
    q = np.unique(rng.integers(0, 3, (6 * count + 40, nm)).astype(np.uint8), axis=0)
    rng.shuffle(q)
    n = max(2, count // nm)
    with VHCI(problem=dict(freq=freq, cap=[8] * nm, ntot=1, fcs=fcs, eps1=1.0, nstate=1, pt2=0)) as v:
        v.set_basis(q[:n])
        C = np.zeros((n, 1), order="F")
        C[:, 0] = 1.0 / np.sqrt(n)
        v.set_vectors(C, np.zeros(1))
        s = v.select(1e-3)
    # host: every change of the cubic terms and of the aggregated single excitations
    have = {x.tobytes() for x in q[:n]}
    want = set()
    for x in q[:n].astype(np.int16):
        for m in range(nm):
            for d in (-3, -1, 1, 3):
                t = x.copy()
                t[m] += d
                if t[m] >= 0 and t.astype(np.uint8).tobytes() not in have:
                    want.add(t.astype(np.uint8).tobytes())
    assert {x.tobytes() for x in s} == want and len(s) == len(want)
    keys = [sum(int(v) << (4 * m) for m, v in enumerate(x)) for x in s]
    assert keys == sorted(keys)
