"""FP64 products of operands whose columns span many orders of magnitude:
every row sum as accurate, against its own terms, as FP64 additions are.

Bound, for a row of len terms in any order of additions: len·2^-53·Σ|terms|
(the fixed-point sums stay below it by construction), and a few roundings of
the sum, the scale and the shift: 4·2^-53·(Σ|terms| scale + |scale·sum| + |d·y|).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(block, ptr, idx, X, scale, dsh, y, val=None):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    t = [None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (ptr, idx, val, X, scale, dsh, y)]
    q = [None if a is None else a.data_ptr() for a in t]
    rows = ptr.size - 1
    out = torch.full((rows, block), 7.0, dtype=torch.float64, device="cuda")
    nb = int(L.sg_spmm_fx_work_bytes(block, X.shape[0]))
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    sh = torch.cuda.current_stream().cuda_stream
    if val is None:
        rc = L.sg_spmm_fx(block, rows, q[0], q[1], X.shape[0], q[3], out.data_ptr(), q[4], q[5], q[6],
                          work.data_ptr(), nb, sh)
    else:
        rc = L.sg_spmm_fx_counts(block, rows, q[0], q[1], q[2], X.shape[0], q[3], out.data_ptr(), q[4], q[5], q[6],
                                 work.data_ptr(), nb, sh)
    _lib.check(rc, "spmm")
    return out.cpu().numpy()


def _operand(cols, block, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((cols, block))
    X[7, 0] = 1e6                                    # one value above the rest of its column
    X[9, 1] = -1e12
    X[11, 2] = 1e200
    X[:, 3] *= 10.0 ** rng.uniform(-40, 0, cols)     # every magnitude
    if block > 4:
        X[cols // 2:, 4] *= 1e-16                    # two halves
        X[:, 5] *= 2.0 ** -1030                      # below the normal numbers
        X[:, 6] = 0.0
        X[cols // 3:, 7] = 0.0
    return X


@pytest.mark.parametrize("block", [4, 8, 16, 32])
@pytest.mark.parametrize("rows,lengths", [(1, [3000]), (40, [0, 1, 2, 31, 33, 64, 127]), (300, [700, 3, 0, 1025]),
                                          (9001, [0, 1, 7, 33, 8])])
@pytest.mark.parametrize("top", [0, 1, 5, 65535])
def test_rows_as_accurate_as_additions(block, rows, lengths, top):
    cols, rng = 3001, np.random.default_rng(rows + block)
    ln = np.resize(np.asarray(lengths, dtype=np.int64), rows)
    ptr = np.concatenate([[0], np.cumsum(ln)])
    idx = rng.integers(0, cols, int(ptr[-1])).astype(np.int32)
    idx[: idx.size // 2] = idx[: idx.size // 2] // 2 + cols // 2   # rows of one half only
    val = rng.integers(0, top + 1, idx.size).astype(np.float32) if top else None
    X = _operand(cols, block, block)
    scale, dsh, y = rng.random(rows) + 0.5, rng.random(rows), rng.standard_normal((rows, block)) * 1e-30
    got = _call(block, ptr, idx, X, scale, dsh, y, val)
    for r in sorted(set(range(min(rows, 40))) | set(range(rows // 2, min(rows, rows // 2 + 20))) | {rows - 1}):
        e = idx[ptr[r]:ptr[r + 1]]
        v = np.ones(e.size) if val is None else val[ptr[r]:ptr[r + 1]].astype(float)
        for c in range(block):
            x = X[e, c]
            hi = np.ldexp(np.rint(np.ldexp(np.frexp(x)[0], 26)), np.frexp(x)[1] - 26)  # count x half: exact
            s, mag = math.fsum(np.concatenate([v * hi, v * (x - hi)])), math.fsum(np.abs(v * x))
            sh = dsh[r] * y[r, c]
            bound = scale[r] * (e.size + 4) * 2.0 ** -53 * mag + 2.0 ** -51 * (abs(scale[r] * s) + abs(sh))
            assert abs(got[r, c] - (scale[r] * s - sh)) <= bound + 1e-320, (r, c)


@pytest.mark.parametrize("counts", [False, True])
@pytest.mark.parametrize("rho", [1e-9, 1e-16, 1e-30])
def test_cells_of_light_features(rho, counts):
    """Two groups of cells over disjoint features: scaling the weights of one
    group's features leaves the cosine operator, and so its eigenvalues, as
    they are."""
    import scipy.sparse as sp
    from snapatac2_gb300 import tools
    rng = np.random.default_rng(4)
    A = sp.block_diag([sp.random(300, 1500, density=0.04, random_state=q, format="csr") for q in (1, 2)]).tocsr()
    A.sort_indices()
    A.data[:] = rng.integers(1, 4, A.nnz) if counts else 1
    w = np.ones(3000)
    kw = dict(precision="fp64", block=8)
    want, _ = tools.spectral_embedding(A, None, 8, 0, w, **kw)
    w[1500:] = rho
    got, vecs = tools.spectral_embedding(A, None, 8, 0, w, **kw)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
