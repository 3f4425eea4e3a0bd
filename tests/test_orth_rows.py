"""Rows brought to the closest orthonormal set (sg_orth_rows, the last step of
the eigenvectors): sets from rounding-level to far from orthonormal come back
orthonormal to 1e-12, as a Cholesky-QR leaves them, and span the same space;
those near enough for the iteration agree with the polar factor."""
import numpy as np
import pytest


def _set(nw, n, size, seed):
    """Orthonormal rows plus a symmetric error of spectral norm `size` in their Gram matrix."""
    rng = np.random.default_rng(seed)
    Q = np.linalg.qr(rng.standard_normal((n, nw)))[0].T
    E = rng.standard_normal((nw, nw))
    E = E + E.T
    E *= size / np.abs(np.linalg.eigvalsh(E)).max()
    w, V = np.linalg.eigh(np.eye(nw) + E)
    return (V * np.sqrt(w)) @ V.T @ Q, Q


def test_two_steps_reach_rounding_inside_the_bound():
    """The rule's arithmetic: ‖E‖ = 1e-4 goes to 4e-17 in two steps of Z - EZ/2, ‖E‖ = 1/4 does not."""
    def after(size):
        Z, _ = _set(60, 90, size, 1)
        for _ in range(2):
            Z = Z - 0.5 * (Z @ Z.T - np.eye(60)) @ Z
        return np.linalg.norm(Z @ Z.T - np.eye(60), 2)
    assert after(1e-4) < 1e-14 and after(0.24) > 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("nw,n", [(1, 1), (2, 3), (31, 33), (60, 90), (290, 336), (640, 640)])
@pytest.mark.parametrize("size", [0.0, 1e-9, 1e-5, 1e-4, 1e-3, 1e-2, 0.1, 0.24, 0.6, 0.9])
def test_gpu_orthonormal_rows(nw, n, size):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    Z, Q = _set(nw, n, size, nw)
    z = torch.from_numpy(np.ascontiguousarray(Z)).cuda()
    nb = int(L.sg_orth_rows_work_bytes(nw, n))
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    _lib.check(L.sg_orth_rows(nw, n, z.data_ptr(), work.data_ptr(), nb, torch.cuda.current_stream().cuda_stream), "")
    got = z.cpu().numpy()
    if nw > 1:  # a single row is left as it is (the inverse iteration normalises it)
        assert np.abs(got @ got.T - np.eye(nw)).max() <= 1e-12
    assert np.abs(Z - (Z @ got.T) @ got).max() <= 1e-12 * n * 2 or nw == 1
    if size <= 1e-9 and nw > 1:
        assert np.abs(got - Q).max() <= 1e-12
    assert L.sg_orth_rows(nw, n, z.data_ptr(), work.data_ptr(), nb - 1, None) == _lib.SG_ERR_CAP
    assert L.sg_orth_rows(n + 1, n, z.data_ptr(), work.data_ptr(), nb, None) == _lib.SG_ERR_ARG
