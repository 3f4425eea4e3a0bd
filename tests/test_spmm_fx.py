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


@pytest.mark.parametrize("block", [4, 8, 16, 32])
@pytest.mark.parametrize("rows,lengths,top", [(3, [0, 1, 900], 1), (40, [5, 64, 65, 0, 700], 4),
                                              (300, [2000, 1, 33], 65535), (5000, [0, 3, 40, 9], 7)])
def test_gpu_fixed_point_counts(block, rows, lengths, top):
    """Values that are counts (sg_spmm_fx_counts) against exact sums: bound as
    above with Σ counts in place of the row's length."""
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    ptr, idx = _matrix(rows, 3000, rows, lengths)
    rng = np.random.default_rng(rows + block)
    X = rng.standard_normal((3000, block)) * np.exp(rng.standard_normal((3000, block)))
    val = rng.integers(0, top + 1, idx.size).astype(np.float32)
    val[-1] = top
    scale, dsh, y = rng.random(rows) + 0.5, rng.random(rows), rng.standard_normal((rows, block))
    t = [torch.from_numpy(a).cuda() for a in (ptr, idx, val, X, scale, dsh, y)]
    out = torch.full((rows, block), 7.0, dtype=torch.float64, device="cuda")
    nb = int(L.sg_spmm_fx_work_bytes(block, 3000))
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    sh = torch.cuda.current_stream().cuda_stream
    q = [a.data_ptr() for a in t]
    _lib.check(L.sg_spmm_fx_counts(block, rows, q[0], q[1], q[2], 3000, q[3], out.data_ptr(), q[4], q[5], q[6],
                                   work.data_ptr(), nb, sh), "counts")
    got, m = out.cpu().numpy(), np.abs(X).max(axis=0)
    for r in list(range(min(rows, 60))) + [rows - 1]:
        e, v = idx[ptr[r]:ptr[r + 1]], val[ptr[r]:ptr[r + 1]].astype(float)
        for c in range(block):
            # count x operand split at 26 bits is exact in parts
            hi = np.float64(np.float32(X[e, c]))
            s = math.fsum(np.concatenate([v * hi, v * (X[e, c] - hi)]))
            bound = v.sum() * 2.0 ** -62 * m[c] * scale[r] + 2.0 ** -51 * (abs(scale[r] * s) + abs(dsh[r] * y[r, c]))
            assert abs(got[r, c] - (scale[r] * s - dsh[r] * y[r, c])) <= bound + 1e-320, (r, c)
    mx = torch.zeros(1, dtype=torch.int64, device="cuda")
    for bad, want in ((None, top), (0.5, 2 ** 32 - 1), (-1.0, 2 ** 32 - 1), (65536.0, 2 ** 32 - 1),
                      (np.nan, 2 ** 32 - 1)):
        w = val.copy()
        if bad is not None:
            w[w.size // 2] = bad
        d = torch.from_numpy(w).cuda()
        _lib.check(L.sg_counts_max(w.size, d.data_ptr(), mx.data_ptr(), sh), "max")
        assert int(mx) == want


@pytest.mark.parametrize("fraction", [False, True])
def test_gpu_counts_take_the_fixed_point_kernel(fraction):
    """An FP64 solve of a matrix of counts against the FP64 additions, and one
    with a fractional value, which keeps them."""
    import torch
    from snapatac2_gb300 import _eigen
    import scipy.sparse as sp
    from snapatac2_gb300._binning import DeviceCSR
    rng = np.random.default_rng(3)
    A = sp.random(400, 3000, density=0.05, format="csr", random_state=1)
    A.sort_indices()
    A.data = rng.integers(1, 5, A.nnz).astype(np.float32)
    if fraction:
        A.data[7] = 1.5
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a.astype(t))).cuda()  # noqa: E731
    csr = DeviceCSR(d(A.indptr, np.int64), d(A.indices, np.int32), d(A.data, np.float32), A.shape)
    op = _eigen.build_operator(csr)
    sh = torch.cuda.current_stream().cuda_stream
    assert op.holds_counts(sh) is (not fraction)
    z = torch.from_numpy(rng.standard_normal((400, 8))).cuda()
    zs, t, w = op.a[:, None] * z, torch.empty(3000, 8, dtype=torch.float64, device="cuda"), torch.empty_like(z)
    ref_t, ref = torch.empty_like(t), torch.empty_like(w)
    op.apply(1, 8, z, zs, t, w, sh)
    assert op.variants[(1, 8)][0] == _eigen.FX_COUNTS if not fraction else op.variants[(1, 8)][0] < _eigen.FX
    op.spmm_pass(0, 1, 1, 8, zs, ref_t, sh)
    op.spmm_pass(1, 1, 1, 8, ref_t, ref, sh, z)
    assert float((t - ref_t).abs().max() / ref_t.abs().max()) < 1e-13
    assert float((w - ref).abs().max() / ref.abs().max()) < 1e-13
