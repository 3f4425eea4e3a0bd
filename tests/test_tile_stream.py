"""The sort-free counting of sorted fragments (stream_kernel in
csrc/tile_bin.cu) against the oracle, bit for bit, at its edges: chunks of
1,024 fragments, open runs that cross a chunk, runs wider than the carry (256
tiles) and the counter slots (4,096 tiles), hot tiles, zero-length, excluded
and size-filtered fragments, and cells that need the sort among cells that do
not."""
import numpy as np
import pytest

from oracle import binning as ob

pytestmark = pytest.mark.gpu

GENOME = [("chr1", 9_000_000), ("chrM", 16_000), ("chr2", 5_000_001), ("chr3", 777)]


def _cells(seed):
    rng = np.random.default_rng(seed)
    total = sum(s for _, s in GENOME)
    ends = np.cumsum([s for _, s in GENOME])

    def sorted_frags(n, lo, hi, mean):
        p = np.sort(rng.integers(lo, hi, n))
        ln = rng.geometric(1.0 / mean, n)
        room = ends[np.searchsorted(ends, p, side="right")] - p
        return p, np.minimum(ln, room)

    cells = [sorted_frags(n, 0, total, 200) for n in (0, 1, 2, 1023, 1024, 1025, 2048, 4100, 0, 9000)]
    cells.append(sorted_frags(6000, 5_000_000, 5_000_400, 180))          # one or two hot tiles
    cells.append(sorted_frags(1500, 4_000_000, 4_200_000, 300_000))      # open runs past the carry
    cells.append(sorted_frags(50, 0, 2_000_000, 3_000_000))              # more tiles than slots
    p, ln = sorted_frags(3000, 0, total, 200)
    ln[::7] = 0                                                          # zero length (start > 0 in its chromosome)
    ok = ~((ln == 0) & (np.isin(p, [0, *ends[:-1]])))
    cells.append((p[ok], ln[ok]))
    p, ln = sorted_frags(2500, 0, total, 200)
    o = rng.permutation(p.size)
    cells.append((p[o], ln[o]))                                          # unsorted
    p, ln = sorted_frags(2500, 0, total, 200)
    p[-2:], ln[-2:] = p[-2:][::-1].copy(), ln[-2:][::-1].copy()          # one inversion at the end
    cells.append((p, ln))
    cells.append(sorted_frags(1200, 9_000_000, 9_016_000, 100))          # excluded chromosome alone
    indptr = np.concatenate([[0], np.cumsum([c[0].size for c in cells])]).astype(np.int64)
    return indptr, np.concatenate([c[0] for c in cells]), np.concatenate([c[1] for c in cells])


@pytest.mark.parametrize("strategy", ["paired-insertion", "insertion", "fragment", "single"])
@pytest.mark.parametrize("bin_size,bounds", [(1, None), (500, None), (500, (60, 400)), (5000, None), (8_000_000, None)])
def test_gpu_stream_counts(strategy, bin_size, bounds):
    import torch
    from snapatac2_gb300 import _binning
    from snapatac2_gb300.genome import ChromSizes
    if strategy == "fragment" and bin_size == 1:
        bin_size = 50  # one key per base of every fragment is out of proportion here
    indptr, pos, ln = _cells(bin_size % 97)
    mn, mx = bounds or (None, None)
    if strategy == "single":
        mn = mx = None
    want = ob.tile_bin(indptr, pos.astype(np.uint64), ln.astype(np.uint32), GENOME, bin_size=bin_size,
                       exclude_chroms=["chrM"], counting_strategy=strategy, min_frag_size=mn, max_frag_size=mx)
    layout = _binning.tile_layout(ChromSizes(GENOME), bin_size, ["chrM"])
    d = lambda a, t: torch.from_numpy(a.astype(t)).cuda()  # noqa: E731
    r = _binning.tile_matrix(d(indptr, np.int64), d(pos, np.int64),
                             None if strategy == "single" else d(ln, np.int32), layout, bin_size=bin_size,
                             strategy=strategy, min_frag_size=mn, max_frag_size=mx)
    assert np.array_equal(r.indptr.cpu().numpy(), want[0])
    assert np.array_equal(r.indices.cpu().numpy(), want[1])
    assert np.array_equal(r.data.cpu().numpy().view(np.uint32), want[2]) and r.shape[1] == want[3]
