"""The dense eigensolver when the wait between its blocks runs out (the limit is lowered to one poll, so
blocks give up and return): it reports that, and the library's solver has the eigenpairs; the next call,
with the usual limit, is good by itself again.  Tolerance: that of test_gpu_eig."""
import ctypes

import numpy as np
import pytest

from test_gpu_eig import check, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [641, 1500])
def test_wait_that_runs_out(n):
    from vhci_b200 import api
    polls = api.lib().vhci_test_grid_polls
    polls.restype, polls.argtypes = ctypes.c_int, [ctypes.c_int]
    with make(n, 10, n) as v:
        v.build_h()
        try:
            polls(1)
            check(v, 10)
        finally:
            lost = polls(0)
        assert lost == 1
        check(v, 10)
        assert polls(0) == 0
