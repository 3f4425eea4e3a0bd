"""Device-level tile binning through the C ABI (``sg_tile_plan/run/emit``).

Equivalent of the reference's ``create_tile_matrix`` core
(``snapatac2-core/src/feature_count/matrix.rs:26-93``) for fragment data:
builds the output ``GenomeBaseIndex`` (chromosomes minus the excluded ones,
``FragmentData::get_gindex``, ``data_iter.rs:156-173``) and bins every
fragment on the GPU.
"""
from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch

from . import _lib
from .genome import ChromSizes, GenomeIndex

# Below this many fragments the scratch is sized by two keys per fragment
# (32 bytes) and no pass over the fragments plans it: 0.32 of 1.46 ms at 6.1e7
# fragments.  Above (8.6 GB), the exact count keeps the scratch as small as it
# can be.
BOUND_FRAGS = 1 << 28

STRATEGIES = {"insertion": 0, "fragment": 1, "paired-insertion": 2, "single": 3}


@dataclass
class DeviceCSR:
    """CSR matrix resident on the GPU (int64 indptr, int32 indices, optional values)."""

    indptr: torch.Tensor
    indices: torch.Tensor
    data: torch.Tensor | None  # None = implicit 1.0 (binary pattern)
    shape: tuple[int, int]

    @property
    def nnz(self) -> int:
        return int(self.indices.shape[0])

    def to_scipy(self, dtype=None):
        import scipy.sparse as sp
        ip = self.indptr.cpu().numpy()
        ix = self.indices.cpu().numpy()
        if self.data is None:
            d = np.ones(ix.shape[0], dtype=dtype or np.float64)
        else:
            d = self.data.cpu().numpy()
            if dtype is not None:
                d = d.astype(dtype)
        return sp.csr_matrix((d, ix, ip), shape=self.shape)


@dataclass
class TileLayout:
    """Output tile index of a binning call."""

    index: GenomeIndex          # kept chromosomes, step = bin size
    chrom_end: np.ndarray       # uint64, cumulative lengths over ALL chromosomes
    bin_off: np.ndarray         # uint64, first output tile per chromosome
    excl: np.ndarray            # uint8, 1 = excluded
    n_cols: int


def tile_layout(chrom_sizes: ChromSizes, bin_size: int, exclude_chroms) -> TileLayout:
    names, sizes = chrom_sizes.names, np.asarray(chrom_sizes.sizes, dtype=np.uint64)
    if len(names) == 0:
        raise ValueError("empty chromosome list")
    if np.any(sizes == 0):
        raise ValueError("chromosome lengths must be positive")
    if np.any(sizes >= np.uint64(1 << 32)):
        raise ValueError("chromosomes of 4 Gb or more are not supported")
    if bin_size <= 0 or bin_size >= (1 << 32):
        raise ValueError("bin_size must be in [1, 2^32)")
    # only chromosomes present in the genome are excluded (data_iter.rs:182-189)
    ex = set(exclude_chroms or []) & set(names)
    excl = np.array([1 if n in ex else 0 for n in names], dtype=np.uint8)
    nb = (sizes + np.uint64(bin_size - 1)) // np.uint64(bin_size)
    nb_kept = np.where(excl == 1, np.uint64(0), nb)
    bin_off = np.zeros(len(names), dtype=np.uint64)
    bin_off[1:] = np.cumsum(nb_kept)[:-1]
    n_cols = int(nb_kept.sum())
    if n_cols >= (1 << 31):
        raise ValueError(f"{n_cols} tiles exceed the int32 column index range; use a larger bin_size")
    kept = ChromSizes([(n, int(s)) for n, s, e in zip(names, sizes, excl) if not e])
    index = GenomeIndex(kept, bin_size) if len(kept) else GenomeIndex([("_", 1)], bin_size)
    return TileLayout(index, np.cumsum(sizes, dtype=np.uint64), bin_off, excl, n_cols)


def tile_matrix(indptr: torch.Tensor, pos: torch.Tensor, length: torch.Tensor | None,
                layout: TileLayout, *, bin_size: int, strategy: str,
                min_frag_size: int | None = None, max_frag_size: int | None = None,
                stream: torch.cuda.Stream | None = None) -> DeviceCSR:
    """Bin fragments resident on the GPU.

    indptr: int64 [n+1]; pos: int64/uint64 bits [F] global start index;
    length: int32/uint32 bits [F] (ignored for ``strategy='single'``).
    Returns a DeviceCSR with uint32 counts stored in an int32 tensor.
    """
    L = _lib.lib()
    dev = indptr.device
    n = int(indptr.shape[0] - 1)
    F = int(pos.shape[0])
    if strategy not in STRATEGIES:
        raise ValueError("Counting strategy must be one of 'insertion', 'fragment', or 'paired-insertion'")
    st = STRATEGIES[strategy]
    if length is None:
        length = torch.ones(F, dtype=torch.int32, device=dev)
    if length.shape[0] != F:
        raise ValueError("fragment positions and lengths differ in length")
    for t in (indptr, pos, length):
        if not t.is_contiguous():
            raise ValueError("inputs must be contiguous")
    s = stream or torch.cuda.current_stream(dev)
    sh = s.cuda_stream
    nc = layout.excl.shape[0]  # one copy for the three chromosome tables
    table = np.empty(17 * nc, dtype=np.uint8)
    table[:8 * nc], table[8 * nc:16 * nc], table[16 * nc:] = (layout.chrom_end.view(np.uint8),
                                                              layout.bin_off.view(np.uint8), layout.excl)
    table = torch.from_numpy(table).to(dev)
    nchrom = int(layout.excl.shape[0])
    mn = -1 if min_frag_size is None else int(min_frag_size)
    mx = -1 if max_frag_size is None else int(max_frag_size)
    # [row pointers | status | lowest offending index]: one read gives the total and the status
    plan = torch.empty(n + 3, dtype=torch.int64, device=dev)
    scan_scr = torch.empty(int(L.sg_scan_scratch_bytes(n + 1)), dtype=torch.uint8, device=dev)
    tp = table.data_ptr()
    genome_args = [tp, tp + 8 * nc, tp + 16 * nc, nchrom, int(bin_size), st, mn, mx]
    if strategy != "fragment" and F < BOUND_FRAGS:
        K = F if strategy == "single" else 2 * F
        _lib.check(L.sg_tile_bound(indptr.data_ptr(), n, st, plan.data_ptr(), sh), "sg_tile_bound")
    else:
        status = _lib.DeviceStatus(dev, plan[n + 1:])
        _lib.check(L.sg_tile_plan(indptr.data_ptr(), n, F, pos.data_ptr(), length.data_ptr(), *genome_args,
                                  plan.data_ptr(), scan_scr.data_ptr(), status.status_ptr, status.bad_ptr, sh),
                   "sg_tile_plan")
        K, *words = plan[n:].tolist()
        status.raise_if(words, "tile binning: fragment out of range of its chromosome", "fragment")
    nbytes = int(L.sg_tile_scratch_bytes(K))
    scratch = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=dev)
    out = torch.empty(n + 3, dtype=torch.int64, device=dev)
    status = _lib.DeviceStatus(dev, out[n + 1:])
    _lib.check(L.sg_tile_run(indptr.data_ptr(), n, F, pos.data_ptr(), length.data_ptr(), *genome_args,
                             plan.data_ptr(), scratch.data_ptr(), nbytes, out.data_ptr(),
                             scan_scr.data_ptr(), status.status_ptr, status.bad_ptr, sh), "sg_tile_run")
    nnz, *words = out[n:].tolist()
    status.raise_if(words, "tile binning: fragment out of range of its chromosome"
                    if words[0] == _lib.SG_ERR_RANGE else "tile binning", "fragment")
    return emit_pairs(plan, scratch, nbytes, out, n, nnz, status, layout.n_cols, sh)


def emit_pairs(key_ptr, scratch, nbytes: int, out, n: int, nnz: int, status, n_cols: int, stream: int) -> DeviceCSR:
    """The (column, count) pairs of a tile or region run as CSR
    (``sg_tile_emit``).  The row pointers come from the run itself and bound
    the arrays allocated here, so there is no further status to wait for."""
    L = _lib.load()
    out_idx = torch.empty(max(nnz, 1), dtype=torch.int32, device=out.device)
    out_cnt = torch.empty(max(nnz, 1), dtype=torch.int32, device=out.device)
    _lib.check(L.sg_tile_emit(n, key_ptr.data_ptr(), scratch.data_ptr(), nbytes, out.data_ptr(), out_idx.data_ptr(),
                              out_cnt.data_ptr(), nnz, status.status_ptr, stream), "sg_tile_emit")
    return DeviceCSR(out[:n + 1], out_idx[:nnz], out_cnt[:nnz], (n, n_cols))
