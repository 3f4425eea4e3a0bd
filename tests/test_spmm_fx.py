"""FP64 SpMM by exact fixed-point sums (``sg_spmm_fx``) against correctly
rounded row sums (``math.fsum``): empty rows, single chunks, rows within one
warp's slice and across several, matrices short enough for the smallest CTA
and long enough for the largest.

Bound, from the operand rounding (2^-62 of the column's largest magnitude a
term, at most) and the few FP64 roundings of the epilogue:
len·2^-62·max|in|·|scale| + 4·2^-53·(|scale·sum| + |d·y|).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(rows, cols, seed, lengths):
    rng = np.random.default_rng(seed)
    ln = np.resize(np.asarray(lengths, dtype=np.int64), rows)
    ptr = np.zeros(rows + 1, np.int64)
    np.cumsum(ln, out=ptr[1:])
    return ptr, rng.integers(0, cols, int(ptr[-1])).astype(np.int32)


def _run(block, ptr, idx, X, scale, dsh=None, y=None, kernel="fx"):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    d = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    tp, ti, tx, ts, td, ty = d(ptr), d(idx), d(X), d(scale), d(dsh), d(y)
    rows = ptr.size - 1
    out = torch.full((rows, block), 7.0, dtype=torch.float64, device="cuda")
    sh = torch.cuda.current_stream().cuda_stream
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    if kernel == "fx":
        nb = int(L.sg_spmm_fx_work_bytes(block, X.shape[0]))
        work = torch.empty(nb, dtype=torch.uint8, device="cuda")
        rc = L.sg_spmm_fx(block, rows, p(tp), p(ti), X.shape[0], p(tx), p(out), p(ts), p(td), p(ty), p(work), nb, sh)
    else:
        rc = L.sg_spmm(1, block, rows, p(tp), p(ti), None, p(tx), p(out), p(ts), p(td), p(ty), -1, sh)
    _lib.check(rc, "spmm")
    return out.cpu().numpy()


@pytest.mark.parametrize("block", [4, 8, 16, 32])
@pytest.mark.parametrize("rows,lengths", [(1, [5000]), (3, [0, 1, 513]), (37, [0, 1, 2, 31, 32, 33, 64, 65, 127]),
                                          (300, [511, 512, 513, 3, 0, 1025]), (21003, [0, 1, 7, 33, 8])])
@pytest.mark.parametrize("shift", [False, True])
def test_gpu_fixed_point_sums(block, rows, lengths, shift):
    cols = 4001
    ptr, idx = _matrix(rows, cols, rows + block, lengths)
    rng = np.random.default_rng(block)
    X = rng.standard_normal((cols, block)) * np.exp(2.0 * rng.standard_normal((cols, block)))
    X[:, 1] = 0.0           # an all-zero column
    X[:, 2] *= 1e-300       # near the bottom of the exponent range
    X[5, 3] = 1e200         # one value far above the rest of its column
    scale = rng.random(rows) + 0.5
    dsh = rng.random(rows) if shift else None
    y = rng.standard_normal((rows, block)) if shift else None
    got = _run(block, ptr, idx, X, scale, dsh, y)
    plain = _run(block, ptr, idx, X, scale, dsh, y, kernel="plain")
    top = np.abs(X).max(axis=0)
    for r in list(range(min(rows, 40))) + [rows - 1]:
        e = idx[ptr[r]:ptr[r + 1]]
        for c in range(block):
            s = math.fsum(X[e, c])
            sh = dsh[r] * y[r, c] if shift else 0.0
            bound = e.size * 2.0 ** -62 * top[c] * scale[r] + 2.0 ** -51 * (abs(scale[r] * s) + abs(sh))
            assert abs(got[r, c] - (scale[r] * s - sh)) <= bound + 1e-320, (r, c)
    # every row against the FP64 additions: their own error is at most len·2^-53 of Σ|terms|
    absum = np.zeros((rows, block))
    np.add.at(absum, np.repeat(np.arange(rows), np.diff(ptr)), np.abs(X[idx]))
    ln = np.diff(ptr)[:, None].astype(float)
    tol = scale[:, None] * (absum * (ln + 4) * 2.0 ** -52 + ln * 2.0 ** -61 * top[None, :])
    if shift:
        tol = tol + 2.0 ** -50 * np.abs(dsh[:, None] * y)
    assert np.all(np.abs(got - plain) <= tol + 1e-318)


@pytest.mark.parametrize("block", [4, 8, 32])
def test_gpu_fixed_point_order_free(block):
    ptr, idx = _matrix(50, 900, 3, [3000, 40, 900])
    rng = np.random.default_rng(1)
    X = rng.standard_normal((900, block))
    scale = np.ones(50)
    perm = idx.copy()
    for r in range(50):
        rng.shuffle(perm[ptr[r]:ptr[r + 1]])
    assert np.array_equal(_run(block, ptr, idx, X, scale), _run(block, ptr, perm, X, scale))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_gpu_fixed_point_non_finite(bad):
    ptr, idx = _matrix(70, 500, 5, [1500, 3, 0, 60])
    X = np.random.default_rng(2).standard_normal((500, 8))
    X[17, 6] = bad
    scale = np.full(70, 0.5)
    got, plain = _run(8, ptr, idx, X, scale), _run(8, ptr, idx, X, scale, kernel="plain")
    assert np.array_equal(np.isnan(got), np.isnan(plain)) and np.array_equal(np.isinf(got), np.isinf(plain))
    ok = np.isfinite(plain)
    assert np.allclose(got[ok], plain[ok], rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("block", [4, 8, 16, 32])
@pytest.mark.parametrize("rows,lengths", [(2, [20000, 1]), (9, [0, 0, 4097, 0, 31, 9000]), (64, [0]), (65, [1]),
                                          (3001, [700, 0, 3, 2600, 33]), (5000, [0, 0, 0, 0, 0, 0, 0, 2000])])
def test_gpu_fixed_point_rows_across_slices(block, rows, lengths):
    """Rows that lie in several warps' slices, empty ones at the edges of a
    slice and of a CTA: every row against the FP64 additions (their error is
    at most len·2^-53 of Σ|terms|)."""
    ptr, idx = _matrix(rows, 2000, rows, lengths)
    X = np.random.default_rng(rows).standard_normal((2000, block))
    scale = np.linspace(0.5, 2.0, rows)
    got, plain = _run(block, ptr, idx, X, scale), _run(block, ptr, idx, X, scale, kernel="plain")
    ln = np.diff(ptr)[:, None].astype(float)
    tol = scale[:, None] * np.abs(X).max(axis=0)[None, :] * (ln * (ln + 4) * 2.0 ** -52 + ln * 2.0 ** -61)
    assert np.all(np.abs(got - plain) <= tol)
