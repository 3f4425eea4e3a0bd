"""FP64 products around the size from which they are taken in fixed point
(_eigen.fx_pays): the operator's and the plain product on both sides of it,
ones, counts and fractions, against sums in extended precision."""
import numpy as np
import pytest


def test_rule_is_by_size():
    from snapatac2_gb300 import _eigen
    assert not _eigen.fx_pays(374_999, 8) and _eigen.fx_pays(375_000, 8)
    assert not _eigen.fx_pays(100_000, 4) and _eigen.fx_pays(20_000_000, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("values", ["ones", "counts", "fractions"])
@pytest.mark.parametrize("n,density,block", [(150, 0.03, 4), (400, 0.1, 8), (700, 0.3, 8)])
def test_gpu_products_on_both_sides(n, density, block, values, monkeypatch):
    import scipy.sparse as sp
    import torch
    from snapatac2_gb300 import _eigen
    from snapatac2_gb300._binning import DeviceCSR
    m = 2500
    rng = np.random.default_rng(n)
    A = sp.random(n, m, density=density, format="csr", random_state=n)
    A.sort_indices()
    A.data[:] = {"ones": 1.0, "counts": rng.integers(1, 6, A.nnz), "fractions": rng.random(A.nnz) + 0.5}[values]
    A.data = A.data.astype(np.float32)
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a.astype(t))).cuda()  # noqa: E731
    data = None if values == "ones" else d(A.data, np.float32)
    csr = DeviceCSR(d(A.indptr, np.int64), d(A.indices, np.int32), data, A.shape)
    op = _eigen.build_operator(csr)
    calls = []
    fx = _eigen.spmm_fx
    monkeypatch.setattr(_eigen, "spmm_fx", lambda *a, **k: (calls.append(1), fx(*a, **k))[1])
    sh = torch.cuda.current_stream().cuda_stream
    Z = torch.from_numpy(rng.standard_normal((n, block))).cuda()
    Zs, T, W = op.a[:, None] * Z, torch.empty(m, block, dtype=torch.float64, device="cuda"), torch.empty_like(Z)
    op.apply(1, block, Z, Zs, T, W, sh)
    big = A.nnz * block >= 3_000_000
    assert len(calls) == (2 if big and values != "fractions" else 0)
    X = A.astype(np.longdouble).toarray()
    w2, a, dinv = (t.cpu().numpy().astype(np.longdouble) for t in (op.w2, op.a, op.dinv))
    t_ref = w2[:, None] * (X.T @ Zs.cpu().numpy().astype(np.longdouble))
    w_ref = a[:, None] * (X @ t_ref) - dinv[:, None] * Z.cpu().numpy()
    assert np.abs(T.cpu().numpy() - t_ref).max() <= 1e-14 * np.abs(t_ref).max() * 10
    assert np.abs(W.cpu().numpy() - w_ref).max() <= 1e-13 * np.abs(w_ref).max()
    out = torch.empty(n, block, dtype=torch.float64, device="cuda")
    ones = torch.ones(n, dtype=torch.float64, device="cuda")
    calls.clear()
    _eigen.spmm64(n, csr.indptr, csr.indices, data, m, T, out, ones, block, sh)
    assert len(calls) == (1 if big and values == "ones" else 0)
    p_ref = X @ T.cpu().numpy().astype(np.longdouble)
    assert np.abs(out.cpu().numpy() - p_ref).max() <= 1e-13 * np.abs(p_ref).max()
