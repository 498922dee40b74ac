"""The warp-per-row product behind H X and the residual norms, at its edges: every lane split (block
widths), rows shorter and longer than one turn of the unrolled loop, unaligned row starts, single-
column (odd or misaligned) and paired gathers, FP64 and FP32 storage.

Tolerance: each result is a sum of m + 1 products in some order, so it is within
(m + 4) 2^-53 sum |h_ij x_j| of the exact value (m: entries of the row); the CSR product that it is
compared with obeys the same bound, hence twice that."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module", params=[0, 1], ids=["fp64", "fp32"])
def ctx(request):
    from vhci_b200 import api
    path = os.path.join(GOLDEN, "workload0", "input.inp")
    with api.VHCI(path, precision=request.param) as v:
        q0 = v.basis()
        rng = np.random.default_rng(4)
        # 91 low states plus 2,000 scattered ones: rows of a few to some hundred entries
        q = np.concatenate([q0, rng.binomial(5, 0.12, (3000, q0.shape[1])).astype(np.uint8)])
        q = np.unique(q, axis=0)
        rng.shuffle(q)
        v.set_basis(q[:2091])
        H = v.h_csr()
        m = np.diff(H.indptr)
        assert m.min() < 16 < 64 < m.max()
        yield v, H, m


def bound(H, m, X):
    return 2 * (m + 4)[:, None] * U * (abs(H) @ np.abs(X))


@pytest.mark.parametrize("b", [1, 2, 3, 4, 6, 8, 9, 10, 16, 17, 31, 32, 33, 34, 66])
def test_product_at_every_lane_split(ctx, b):
    v, H, m = ctx
    X = np.random.default_rng(b).standard_normal((v.n, b))
    assert (np.abs(v.apply_h(X) - H @ X) <= bound(H, m, X)).all()


@pytest.mark.parametrize("k", [1, 2, 4, 5, 8, 10, 16, 18, 31, 32, 33, 64, 255, 256])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "misaligned"])
def test_residual_norms_at_every_lane_split(ctx, k, shift):
    import torch
    v, H, m = ctx
    rng = np.random.default_rng(k)
    X, th = rng.standard_normal((v.n, k)), rng.uniform(5e3, 2e4, k)
    buf = torch.zeros(v.n * k + 1, dtype=torch.float64, device="cuda")
    buf[shift:shift + v.n * k] = torch.from_numpy(X).reshape(-1).cuda()
    thd = torch.from_numpy(th).cuda()
    r = torch.zeros(k, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    v.residual_norms_noalloc(buf.data_ptr() + 8 * shift, thd.data_ptr(), r.data_ptr(), k)
    ref = np.linalg.norm(H @ X - X * th, axis=0)
    # entrywise bound on the residual, plus the rounding of theta x and of the sum of n squares
    err = np.linalg.norm(bound(H, m, X) + 4 * U * np.abs(X * th), axis=0) + (v.n + 4) * U * ref
    assert (np.abs(r.cpu().numpy() - ref) <= err).all()


@pytest.mark.parametrize("n,k", [(1, 1), (33, 31), (91, 65), (20011, 420)])  # the last: two transfers
def test_vectors_round_trip(n, k):
    from vhci_b200 import api
    rng = np.random.default_rng(k)
    with api.VHCI(os.path.join(GOLDEN, "workload0", "input.inp")) as v:
        q = np.unique(rng.binomial(6, 0.3, (2 * n + 50, v.info.nmodes)).astype(np.uint8), axis=0)[:n]
        v.set_basis(q)
        C, E = rng.standard_normal((n, k)), np.sort(rng.standard_normal(k))
        v.set_vectors(C, E)
        for m in {1, k - k // 3, k}:
            got, e = v.vectors(m)
            assert np.array_equal(got, C[:, :m]) and np.array_equal(e, E[:m])
