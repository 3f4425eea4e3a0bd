"""The indexed region lookup (``sg_region_index`` and the plan / run calls
that use it) against the oracle and against the calls without an index: many
regions in one bucket, empty buckets and chromosomes, regions past their
chromosome's end, unsorted fragments, and rows on both sides of the 4,096
keys that the short-row kernel holds."""
import numpy as np
import pytest

from oracle import regions as org

pytestmark = pytest.mark.gpu

GENOME = [("chrA", 2_000_000), ("chrB", 900), ("chrC", 700_001), ("chrM", 16_000)]


def _data(seed):
    rng = np.random.default_rng(seed)
    ends = np.cumsum([s for _, s in GENOME])
    rows = []
    for n, lo, hi in ((0, 0, 1), (1, 0, ends[-1]), (31, 0, ends[-1]), (33, 0, ends[-1]), (900, 0, ends[-1]),
                      (5000, 1_000_000, 1_003_000), (3000, 0, ends[-1]), (4095, 1_000_000, 1_000_400), (64, 0, ends[-1])):
        p = np.sort(rng.integers(lo, hi, n))
        rows.append((p, np.minimum(rng.integers(1, 400, n), ends[np.searchsorted(ends, p, side="right")] - p)))
    rows.append(tuple(a[::-1].copy() for a in rows[4]))
    indptr = np.concatenate([[0], np.cumsum([r[0].size for r in rows])]).astype(np.int64)
    peaks = [("chrA", 1_000_000 + 7 * i, 1_000_000 + 7 * i + 300) for i in range(150)]
    peaks += [("chrA", int(s), int(s) + 500) for s in rng.integers(0, 1_999_000, 400)]
    peaks += [("chrA", 1_999_900, 2_000_500), ("chrA", 2_100_000, 2_100_100), ("chrC", 0, 700_001),
              ("chrC", 699_990, 700_001), ("chrC", 699_999, 800_000), ("chrM", 0, 16_000)]
    rng.shuffle(peaks)
    return indptr, np.concatenate([r[0] for r in rows]), np.concatenate([r[1] for r in rows]), \
        [f"{c}:{a}-{b}" for c, a, b in map(tuple, peaks)]


@pytest.mark.parametrize("strategy", ["insertion", "paired-insertion", "fragment", "single"])
def test_gpu_indexed_lookup(strategy):
    import torch
    from snapatac2_gb300 import _binning, _lib, _regions
    from snapatac2_gb300.genome import ChromSizes
    indptr, pos, ln, peaks = _data(len(strategy))
    names, sizes = [c for c, _ in GENOME], [s for _, s in GENOME]
    ref = org.region_counts(indptr, pos.astype(np.uint64), ln.astype(np.int64), names, sizes, peaks,
                            strategy=strategy, paired=strategy != "single")
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a.astype(t))).cuda()  # noqa: E731
    ip, ps, le = d(indptr, np.int64), d(pos, np.int64), d(ln, np.int32)
    regs = _regions.build_regions(peaks, names, torch.device("cuda"))
    got = _regions.region_matrix(ip, ps, le, ChromSizes(GENOME), regs, strategy=strategy)
    # the plain calls: no index, no mask
    L = _lib.lib()
    n, F, sh = indptr.size - 1, pos.size, torch.cuda.current_stream().cuda_stream
    end, excl = d(np.cumsum(sizes), np.int64), torch.zeros(len(sizes), dtype=torch.uint8, device="cuda")
    p = lambda t: t.data_ptr()  # noqa: E731
    args = [p(ip), n, F, p(ps), p(le), p(end), p(excl), len(sizes), p(regs.ptr), p(regs.start), p(regs.end),
            p(regs.maxend), p(regs.rid), len(regs.names), _binning.STRATEGIES[strategy], -1, -1]
    st = _lib.DeviceStatus("cuda")
    key, out = (torch.empty(n + 1, dtype=torch.int64, device="cuda") for _ in range(2))
    scan = torch.empty(int(L.sg_scan_scratch_bytes(n + 1)), dtype=torch.uint8, device="cuda")
    _lib.check(L.sg_region_plan(*args, p(key), p(scan), st.status_ptr, st.bad_ptr, sh), "plan")
    nb = int(L.sg_tile_scratch_bytes(int(key[n])))
    scr = torch.empty(nb, dtype=torch.uint8, device="cuda")
    _lib.check(L.sg_region_run(*args, p(key), p(scr), nb, p(out), p(scan), st.status_ptr, st.bad_ptr, sh), "run")
    st.raise_if_error("plain region calls")
    plain = _binning.emit_pairs(key, scr, nb, out, n, int(out[n]), st, len(regs.names), sh)
    for r in (got, plain):
        np.testing.assert_array_equal(r.indptr.cpu().numpy(), ref[0])
        np.testing.assert_array_equal(r.indices.cpu().numpy(), ref[1])
        np.testing.assert_array_equal(r.data.cpu().numpy().view(np.uint32), ref[2])
