"""Tile binning over layouts of many contigs: tile indices that ascend with
the contigs, and, through the C entry points, tables in which they do not (one
contig's tiles in front of those of the contig before, near the start, the
middle and the end of the table)."""
import numpy as np
import pytest

from oracle import binning as ob

pytestmark = pytest.mark.gpu


def _cells(genome, seed):
    rng = np.random.default_rng(seed)
    total = sum(s for _, s in genome)
    ends = np.cumsum([s for _, s in genome])
    rows = []
    for n in (0, 3, 1024, 2500):
        p = np.sort(rng.integers(0, total, n))
        rows.append((p, np.minimum(rng.integers(1, 300, n), ends[np.searchsorted(ends, p, side="right")] - p)))
    indptr = np.concatenate([[0], np.cumsum([r[0].size for r in rows])]).astype(np.int64)
    return indptr, np.concatenate([r[0] for r in rows]), np.concatenate([r[1] for r in rows])


@pytest.mark.parametrize("contigs", [1, 2, 1024, 1025, 5000])
def test_gpu_many_contigs(contigs):
    import torch
    from snapatac2_gb300 import _binning
    from snapatac2_gb300.genome import ChromSizes
    genome = [(f"s{i:05d}", 700 + 13 * (i % 50)) for i in range(contigs)]
    indptr, pos, ln = _cells(genome, contigs)
    want = ob.tile_bin(indptr, pos.astype(np.uint64), ln.astype(np.uint32), genome, bin_size=100, exclude_chroms=[])
    layout = _binning.tile_layout(ChromSizes(genome), 100, [])
    d = lambda a, t: torch.from_numpy(a.astype(t)).cuda()  # noqa: E731
    r = _binning.tile_matrix(d(indptr, np.int64), d(pos, np.int64), d(ln, np.int32), layout, bin_size=100,
                              strategy="paired-insertion")
    assert np.array_equal(r.indptr.cpu().numpy(), want[0])
    assert np.array_equal(r.indices.cpu().numpy(), want[1])
    assert np.array_equal(r.data.cpu().numpy().view(np.uint32), want[2])


@pytest.mark.parametrize("at", [1, 700, 1024, 2999])
def test_gpu_tile_offsets_that_descend(at):
    import torch
    from snapatac2_gb300 import _binning
    from snapatac2_gb300.genome import ChromSizes
    genome = [(f"s{i:05d}", 1000) for i in range(3000)]
    indptr, pos, ln = _cells(genome, at)
    layout = _binning.tile_layout(ChromSizes(genome), 100, [])
    off = layout.bin_off.copy()
    layout.bin_off[at], layout.bin_off[at - 1] = off[at - 1], off[at]
    d = lambda a, t: torch.from_numpy(a.astype(t)).cuda()  # noqa: E731
    r = _binning.tile_matrix(d(indptr, np.int64), d(pos, np.int64), d(ln, np.int32), layout, bin_size=100,
                              strategy="paired-insertion")
    ptr, idx, cnt = r.indptr.cpu().numpy(), r.indices.cpu().numpy(), r.data.cpu().numpy()
    for c in range(4):
        p, n = pos[indptr[c]:indptr[c + 1]], ln[indptr[c]:indptr[c + 1]]
        ch = p // 1000
        lo = layout.bin_off[ch].astype(np.int64) + p % 1000 // 100
        hi = layout.bin_off[ch].astype(np.int64) + (p % 1000 + n - 1) // 100
        t, k = np.unique(np.concatenate([lo, hi[hi != lo]]), return_counts=True)
        assert np.array_equal(idx[ptr[c]:ptr[c + 1]], t) and np.array_equal(cnt[ptr[c]:ptr[c + 1]], k)
