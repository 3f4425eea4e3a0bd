"""One Cholesky-QR pass through the C ABI (sg_block_cholqr: G = WᵀW, G = RᵀR,
W <- W R⁻¹) against FP64 NumPy, for every block width, FP32 and FP64, at row
counts around the tile (64 rows per CTA, 256 per FP32 pass) and past the
largest grid.

Tolerances.  G: FP64 sums, 1e-13 Σ|w||w|; with FP32 blocks the products and a
thread's own rows are rounded to FP32 (fewer than 90 terms one after another at
100,003 rows for 16 and 32 columns, fewer below), 100 x 2^-24.  R and R⁻¹:
|RᵀR - G| <= 2 (B + 4) ε |Rᵀ||R| and |R⁻¹R - I| <= 4 (B + 4) ε |R⁻¹||R| with
ε = 2^-53 (Higham, Accuracy and Stability of Numerical Algorithms, 10.1, 8.1).
W R⁻¹: (B + 3) roundings of the block's type."""
import numpy as np
import pytest

ROWS = [40, 63, 64, 65, 255, 257, 5000, 20011, 100003]


def _run(dtype, B, W):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    nparts = int(L.sg_proj_parts())
    td = torch.float32 if dtype == 0 else torch.float64
    Wt = torch.from_numpy(W).to("cuda", td)
    f64 = dict(dtype=torch.float64, device="cuda")
    part = torch.full((nparts * B * B,), float("nan"), **f64)
    G, R, Ri = (torch.full((B, B), float("nan"), **f64) for _ in range(3))
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(L.sg_block_cholqr(dtype, B, W.shape[0], Wt.data_ptr(), part.data_ptr(), nparts, G.data_ptr(),
                                 R.data_ptr(), Ri.data_ptr(), st.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream), "cholqr")
    return [t.cpu().numpy() for t in (G, R, Ri, Wt)] + [int(st)]


@pytest.mark.gpu
@pytest.mark.parametrize("B", [4, 8, 16, 32])
@pytest.mark.parametrize("dtype", [0, 1])
def test_cholqr_matches_fp64(B, dtype):
    eps = 2.0 ** -53
    for i, n in enumerate(ROWS):
        rng = np.random.default_rng(1000 * B + i)
        W = rng.standard_normal((n, B)) * np.logspace(-3, 3, B)
        W = W.astype(np.float32 if dtype == 0 else np.float64)
        G, R, Ri, out, st = _run(dtype, B, W)
        assert st == 0
        W = W.astype(np.float64)
        A = np.abs(W)
        assert np.all(np.abs(G - W.T @ W) <= (1e-13 if dtype else 100 * 2.0 ** -24) * (A.T @ A)), n
        assert np.array_equal(np.tril(R, -1), np.zeros((B, B))) and np.array_equal(np.tril(Ri, -1), np.zeros((B, B)))
        aR, aI = np.abs(R), np.abs(Ri)
        assert np.all(np.abs(R.T @ R - G) <= 2 * (B + 4) * eps * (aR.T @ aR)), n
        assert np.all(np.abs(Ri @ R - np.eye(B)) <= 4 * (B + 4) * eps * (aI @ aR)), n
        u = 2.0 ** -24 if dtype == 0 else eps
        assert np.all(np.abs(out - W @ Ri) <= (B + 3) * u * (A @ aI)), n
        again = _run(dtype, B, W)
        assert all(np.array_equal(a, b) for a, b in zip((G, R, Ri, out), again[:4]))


@pytest.mark.gpu
@pytest.mark.parametrize("B", [4, 8, 16, 32])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("bad", [0.0, np.nan])
def test_cholqr_reports_a_dependent_block(B, dtype, bad):
    W = np.random.default_rng(5).standard_normal((700, B))
    W[:, B // 2] = bad
    assert _run(dtype, B, W)[4] != 0
