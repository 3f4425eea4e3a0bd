"""Exact kNN from 16,385 points on (ordered copy, tile boxes, heaps; csrc/knn.cu)
against the oracle, every row: the smallest such size, a ragged last tile,
padded and full dimensions, list sizes that leave two, three and four tile
buffers, equal distances at the cut, repeated points and a far outlier."""
import numpy as np
import pytest

from oracle import knn as oknn

pytestmark = pytest.mark.gpu

MIN = 16385


def _data(kind, n, d, seed):
    rng = np.random.default_rng(seed)
    if kind == "clustered":
        s = 0.05 / np.sqrt(np.arange(1, d + 1))
        return rng.standard_normal((9, d))[rng.integers(0, 9, n)] * s * 3 + rng.standard_normal((n, d)) * s
    if kind == "lattice":  # many equal distances
        return rng.integers(0, 6, (n, d)).astype(float)
    if kind == "repeated":
        return rng.standard_normal((n // 40 + 1, d))[rng.integers(0, n // 40 + 1, n)]
    X = rng.standard_normal((n, d))
    X[n // 3] = 1e6        # far outlier
    X[:, d // 2] = 4.25    # a constant column
    return X


@pytest.mark.parametrize("filt", ["tensor", "simt"])
@pytest.mark.parametrize("kind,n,d,k", [("clustered", MIN, 30, 50), ("clustered", MIN + 127, 16, 15),
                                        ("outlier", MIN + 64, 32, 1), ("clustered", 18001, 3, 100),
                                        ("lattice", MIN, 5, 20), ("repeated", MIN + 1, 12, 30),
                                        ("clustered", 17000, 32, 90), ("outlier", 17000, 1, 7)])
def test_gpu_ordered_matches_oracle(filt, kind, n, d, k, monkeypatch):
    from snapatac2_gb300._knn_api import knn_arrays
    monkeypatch.setenv("SNAPGB300_KNN_FILTER", filt)
    X = _data(kind, n, d, n + d + k)
    nbr, dist = knn_arrays(X, k)
    want_nbr, want_dist = oknn.knn_arrays(X, k)
    assert np.array_equal(nbr.cpu().numpy(), want_nbr)
    assert np.array_equal(dist.cpu().numpy(), want_dist)
