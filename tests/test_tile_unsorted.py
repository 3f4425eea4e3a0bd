"""Cells that need the sort (fragments out of order), of very unequal sizes:
more than one round of CTAs, single long cells among many short ones, few
cells, and cells of either kind side by side; keys within shared memory by
their number though not by their bound, and beyond it.  Bit for bit against
the oracle."""
import numpy as np
import pytest

from oracle import binning as ob

pytestmark = pytest.mark.gpu

GENOME = [("chr1", 9_000_000), ("chrM", 16_000), ("chr2", 5_000_001)]


@pytest.mark.parametrize("strategy", ["paired-insertion", "insertion", "fragment", "single"])
@pytest.mark.parametrize("sizes", [(40,) * 700, (30000,) + (3,) * 200 + (14000,) + (0,) * 30 + (13000,) * 3, (5, 60000),
                                   tuple(range(1, 3000, 7)), (12288, 12289, 24576, 24577, 17000, 16000)])
@pytest.mark.parametrize("every", [1, 3])
def test_gpu_unsorted_cells(strategy, sizes, every):
    import torch
    from snapatac2_gb300 import _binning
    from snapatac2_gb300.genome import ChromSizes
    rng = np.random.default_rng(len(sizes))
    total, ends = sum(s for _, s in GENOME), np.cumsum([s for _, s in GENOME])
    pos = [rng.integers(0, total, n) for n in sizes]
    pos = np.concatenate([p if i % every == 0 else np.sort(p) for i, p in enumerate(pos)])
    ln = np.minimum(rng.geometric(1 / 200, pos.size), ends[np.searchsorted(ends, pos, side="right")] - pos)
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    want = ob.tile_bin(indptr, pos.astype(np.uint64), ln.astype(np.uint32), GENOME, bin_size=500,
                       exclude_chroms=["chrM"], counting_strategy=strategy)
    layout = _binning.tile_layout(ChromSizes(GENOME), 500, ["chrM"])
    d = lambda a, t: torch.from_numpy(a.astype(t)).cuda()  # noqa: E731
    r = _binning.tile_matrix(d(indptr, np.int64), d(pos, np.int64), None if strategy == "single" else d(ln, np.int32),
                             layout, bin_size=500, strategy=strategy)
    assert np.array_equal(r.indptr.cpu().numpy(), want[0])
    assert np.array_equal(r.indices.cpu().numpy(), want[1])
    assert np.array_equal(r.data.cpu().numpy().view(np.uint32), want[2])
