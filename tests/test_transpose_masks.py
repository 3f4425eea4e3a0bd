"""The CSR -> CSC transpose (csrc/spectral.cu) against SciPy at the edges of
its steps: panels of 4,096 columns, 128 rows per step and four 32-row mask
words, row segments longer than the 16 lanes that share one, more row blocks
than rows."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,density,blocks", [(1, 1, 1.0, 1), (31, 2048, 1.0, 1), (127, 2047, 0.5, 3),
                                                (128, 2049, 0.9, 1), (129, 4097, 0.05, 200), (700, 6000, 0.3, 2),
                                                (5000, 300, 0.2, 7), (260, 70000, 0.01, 0), (300, 4095, 0.1, 2),
                                                (257, 4096, 0.1, 1), (129, 8193, 0.2, 0)])
@pytest.mark.parametrize("valued", [False, True])
def test_gpu_transpose_edges(n, m, density, blocks, valued):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(n + m)
    X = sp.random(n, m, density=density, format="csr", random_state=n + m, dtype=np.float64)
    X.sort_indices()
    X.data = rng.integers(1, 9, X.nnz).astype(np.float32)
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a.astype(t))).cuda()  # noqa: E731
    ip, ix, va = d(X.indptr, np.int64), d(X.indices, np.int32), d(X.data, np.float32)
    nblk = blocks or int(L.sg_transpose_row_blocks(n, m))
    wb = int(L.sg_transpose_work_bytes(n, m, nblk))
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    colptr = torch.empty(m + 1, dtype=torch.int64, device="cuda")
    rowidx = torch.empty(max(X.nnz, 1), dtype=torch.int32, device="cuda")
    cval = torch.empty(max(X.nnz, 1), dtype=torch.float32, device="cuda")
    scan = torch.empty(int(L.sg_scan_scratch_bytes(max(n, m) + 1)), dtype=torch.uint8, device="cuda")
    st = _lib.DeviceStatus("cuda")
    p = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(L.sg_csr_transpose(n, m, p(ip), p(ix), p(va) if valued else None, nblk, p(work), wb, p(colptr),
                                  p(rowidx), p(cval) if valued else None, p(scan), st.status_ptr,
                                  torch.cuda.current_stream().cuda_stream), "transpose")
    st.raise_if_error("transpose")
    C = X.tocsc()
    C.sort_indices()
    assert np.array_equal(colptr.cpu().numpy(), C.indptr)
    assert np.array_equal(rowidx.cpu().numpy()[:X.nnz], C.indices)
    if valued:
        assert np.array_equal(cval.cpu().numpy()[:X.nnz], C.data)
