"""Workloads that the framework's users run, as measurable cases.

Each case is one call (or one step) of the cell-embedding path, through the
entry points that a program calls:

* ``tiles``    fragments -> cell x tile counts (``pp.add_tile_matrix`` on host
               matrices, ``tile_matrix`` on fragments resident on the GPU)
* ``peaks``    fragments -> cell x peak counts (``region_matrix``)
* ``import``   fragment-file text -> fragments (``import_text`` from pinned
               host text, ``import_device`` from text in device memory)
* ``counts``   per-feature totals of ``pp.select_features``
* ``build``    the spectral operator's set-up: transpose, weights, degrees
* ``gram``     one block product with the operator (one step of the
               eigensolver's Krylov expansion), single or double precision
* ``spectral`` a whole double-precision embedding, matrix on the GPU
* ``gradient`` a training step on the feature weights: the top-k eigenvalue
               sum (mixed-precision solve) and its gradient
* ``knn``      the exact neighbour graph (``pp.knn`` from host arrays,
               ``knn_arrays`` on an embedding resident on the GPU)

The returned vectors of a mixed-precision solve are determined only up to
its residual bar, so those solves enter through their operator (``gram``,
``build``) and through the training step, whose outputs are single precision.
The embeddings have more cell populations than components, so that every
returned vector is an isolated one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from snapatac2_gb300 import _binning, _eigen, _import, _knn_api, _regions, preprocessing, synthetic, tools
from snapatac2_gb300 import topk_eigenvalue_sum
from snapatac2_gb300.genome import ChromSizes

GENOME_BP = 3_100_000_000
EXCLUDED = ["chrM", "chrY", "M", "Y"]
POPULATIONS = 36


def listed():
    return [
        # a pilot or per-sample call on host matrices: latency, conversions and copies count
        {"name": "tiles_host_small", "kind": "tiles", "host": True, "cells": 150, "median": 1500, "bin": 500,
         "strategy": "paired-insertion", "bounds": False},
        # an ordinary 10x sample: 5,000 cells, 6e7 fragments, default options
        {"name": "tiles_5k_cells", "kind": "tiles", "host": False, "cells": 5000, "median": 10000, "bin": 500,
         "strategy": "paired-insertion", "bounds": False},
        # the same sample counted over a called peak set
        {"name": "peaks_5k_cells", "kind": "peaks", "cells": 5000, "median": 10000, "peaks": 200000,
         "strategy": "paired-insertion", "wide": False},
        # a small barcode-sorted fragment file from host memory, results back on the host
        {"name": "import_host_small", "kind": "import", "host": True, "cells": 100, "median": 1000,
         "order": "barcode", "min_frags": 200},
        # a 10x fragment file in genome order: grouped and sorted by barcode on the GPU
        {"name": "import_position_order", "kind": "import", "host": False, "cells": 1500, "median": 10000,
         "order": "position", "min_frags": 200},
        # select_features on a tile matrix with counts
        {"name": "feature_counts", "kind": "counts", "cells": 20011, "features": 500000, "per_cell": 4000,
         "valued": True},
        # operator set-up of an atlas-size embedding
        {"name": "operator_build_100k", "kind": "build", "cells": 100000, "features": 500000, "per_cell": 4000,
         "valued": False},
        # the eigensolver's product at the same size, at the block size its tuner picks there
        {"name": "gram_100k", "kind": "gram", "cells": 100000, "features": 500000, "per_cell": 4000, "block": 16,
         "double": False, "valued": False},
        # the default embedding of one sample (below 20,000 cells: double precision)
        {"name": "spectral_5k", "kind": "spectral", "cells": 5000, "features": 200003, "per_cell": 4000,
         "comps": 30},
        # one optimiser step on 200k feature weights
        {"name": "gradient_30k", "kind": "gradient", "cells": 30000, "features": 200000, "per_cell": 3000,
         "comps": 30},
        # the graph of a small sample from a host embedding
        {"name": "knn_host_small", "kind": "knn", "host": True, "points": 2500, "dims": 30, "k": 50},
        # the graph of an atlas embedding
        {"name": "knn_100k", "kind": "knn", "host": False, "points": 100000, "dims": 30, "k": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tiles", "peaks", "import", "counts", "build", "gram", "spectral", "gradient", "knn"])
    if kind == "tiles":
        host = rng.random() < 0.3
        return {"kind": kind, "host": host, "cells": _log(rng, 40, 400 if host else 5000),
                "median": _log(rng, 300, 3000 if host else 10000), "bin": rng.choice([500, 500, 1000, 5000]),
                "strategy": rng.choice(["paired-insertion", "insertion", "fragment"]),
                "bounds": rng.random() < 0.3}
    if kind == "peaks":
        return {"kind": kind, "cells": _log(rng, 100, 5000), "median": _log(rng, 500, 10000),
                "peaks": _log(rng, 5000, 200000), "strategy": rng.choice(["paired-insertion", "insertion", "fragment"]),
                "wide": rng.random() < 0.3}
    if kind == "import":
        host = rng.random() < 0.3
        return {"kind": kind, "host": host, "cells": _log(rng, 40, 200 if host else 1500),
                "median": _log(rng, 300, 2000 if host else 10000), "order": rng.choice(["barcode", "position"]),
                "min_frags": rng.choice([0, 200])}
    if kind in ("counts", "build"):
        return {"kind": kind, "cells": _log(rng, 2000, 20000 if kind == "counts" else 100000),
                "features": _log(rng, 50000, 500000), "per_cell": _log(rng, 1000, 4000),
                "valued": rng.random() < 0.5}
    if kind == "gram":
        double = rng.random() < 0.3
        return {"kind": kind, "cells": _log(rng, 2000, 20000 if double else 100000),
                "features": _log(rng, 50000, 500000), "per_cell": _log(rng, 1000, 4000),
                "block": rng.choice([4, 8] if double else [8, 16, 16]), "double": double,
                "valued": rng.random() < 0.25}
    if kind == "spectral":
        return {"kind": kind, "cells": _log(rng, 1200, 5000), "features": _log(rng, 50000, 200000),
                "per_cell": _log(rng, 1500, 4000), "comps": rng.choice([15, 30])}
    if kind == "gradient":
        return {"kind": kind, "cells": _log(rng, 5000, 30000), "features": _log(rng, 50000, 200000),
                "per_cell": _log(rng, 1500, 3000), "comps": rng.choice([15, 30])}
    host = rng.random() < 0.3
    return {"kind": "knn", "host": host, "points": _log(rng, 500, 5000 if host else 100000),
            "dims": rng.choice([10, 20, 30, 30, 50]), "k": rng.choice([15, 50])}


# ---- inputs ------------------------------------------------------------------

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _fragments(cells, median, seed, shuffle):
    """Fragments on the GPU in the ``fragment_paired`` layout (rows sorted by
    start, length): LogNormal(ln median, 0.6) fragments per cell, 8 clusters,
    70 % in the cluster's 50,000 Zipf(1.1)-weighted tiles, lengths geometric
    with mean 200.  With ``shuffle`` the seed deals the cells' order, else it
    draws the fragments; either way the size of the result depends on the
    case alone."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(11 if shuffle else seed)
    rng = np.random.default_rng(11)
    genome = synthetic.make_genome(GENOME_BP)
    sizes = torch.tensor([s for _, s in genome], dtype=torch.int64, device=dev)
    ends = torch.cumsum(sizes, 0)
    starts = ends - sizes
    n_tiles = GENOME_BP // 500
    per_cell = np.maximum(1, np.rint(rng.lognormal(math.log(median), 0.6, cells))).astype(np.int64)
    total = int(per_cell.sum())
    counts = torch.from_numpy(per_cell).to(dev)
    place = torch.arange(cells, device=dev)
    if shuffle:
        place = torch.from_numpy(np.random.default_rng(seed).permutation(cells)).to(dev)
    cell = torch.repeat_interleave(torch.arange(cells, device=dev), counts)
    cluster = torch.randint(0, 8, (cells,), generator=g, device=dev)
    enriched = torch.randint(0, n_tiles, (8, 50_000), generator=g, device=dev)
    cdf = torch.cumsum(torch.arange(1, 50_001, dtype=torch.float64, device=dev) ** -1.1, 0)
    u = torch.rand(total, generator=g, device=dev, dtype=torch.float64) * cdf[-1]
    rank = torch.searchsorted(cdf, u).clamp_(max=49_999)
    pos = enriched[cluster[cell], rank] * 500 + torch.randint(0, 500, (total,), generator=g, device=dev)
    spread = torch.randint(0, GENOME_BP, (total,), generator=g, device=dev)
    pos = torch.where(torch.rand(total, generator=g, device=dev) < 0.7, pos, spread)
    length = (torch.rand(total, generator=g, device=dev, dtype=torch.float64).log_() /
              math.log(1.0 - 1.0 / 200.0)).long().clamp_(0, 4000) + 1
    chrom = torch.searchsorted(ends, pos, right=True)
    pos = torch.minimum(pos, ends[chrom] - length)  # a fragment ends on its chromosome
    pos = torch.maximum(pos, starts[chrom])
    key = torch.sort((((place[cell] << 32) | pos) << 12) | length).values
    indptr = torch.zeros(cells + 1, dtype=torch.int64, device=dev)
    torch.cumsum(counts[torch.argsort(place)], 0, out=indptr[1:])
    return genome, indptr, (key >> 12) & 0xFFFFFFFF, (key & 0xFFF).to(torch.int32)


def _matrix(c, seed, populations=8):
    """Cell x feature matrix on the GPU; counts 1 to 4 when valued.  For the
    set-up, whose result is as large as the matrix, the seed deals the cells'
    order; elsewhere it draws the matrix."""
    dev = _device()
    deal, seed = seed, 11 if c["kind"] == "build" else seed
    indptr, indices, _ = synthetic.binary_csr_device(c["cells"], c["features"], nnz_per_cell=float(c["per_cell"]),
                                                     n_clusters=populations,
                                                     enriched=min(50_000, c["features"] // 4), seed=seed, device=dev)
    if c["kind"] == "build":
        order = torch.from_numpy(np.random.default_rng(deal).permutation(c["cells"])).to(dev)
        counts = (indptr[1:] - indptr[:-1])[order]
        shift = torch.repeat_interleave(indptr[:-1][order], counts)
        torch.cumsum(counts, 0, out=indptr[1:])
        shift -= torch.repeat_interleave(indptr[:-1], counts)
        indices = indices[shift.add_(torch.arange(indices.numel(), device=dev))]
        del shift
    data = None
    if c.get("valued"):
        g = torch.Generator(device=dev).manual_seed(deal + 5)
        u = torch.rand(indices.numel(), generator=g, device=dev)
        data = (1 + (u > 0.7).int() + (u > 0.9).int() + (u > 0.97).int())
        data = data if c["kind"] == "counts" else data.to(torch.float32)
    return _binning.DeviceCSR(indptr, indices, data, (c["cells"], c["features"]))


def _block(c, seed):
    """A block of vectors of about unit length."""
    g = torch.Generator(device=_device()).manual_seed(seed + 3)
    return torch.randn(c["cells"], c["block"], generator=g, device=_device(),
                       dtype=torch.float64 if c["double"] else torch.float32) / math.sqrt(c["cells"])


def _points(c, seed):
    """An embedding: points around 12 centres with decreasing spread per axis."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    kw = dict(generator=g, device=_device(), dtype=torch.float64)
    scale = 0.05 / torch.sqrt(torch.arange(1, c["dims"] + 1, dtype=torch.float64, device=_device()))
    centres = torch.randn(12, c["dims"], **kw) * scale * 2
    which = torch.randint(0, 12, (c["points"],), generator=g, device=_device())
    return centres[which] + torch.randn(c["points"], c["dims"], **kw) * scale


def _peaks(c, genome):
    """Called peaks: 500 bp apart from one another, or of 200 to 2,000 bp that may overlap."""
    rng = np.random.default_rng(9)
    sizes = np.array([s for _, s in genome], dtype=np.int64)
    tiles = sizes // 500
    ends = np.cumsum(tiles)
    pick = np.sort(rng.choice(int(ends[-1]), c["peaks"], replace=False))
    chrom = np.searchsorted(ends, pick, side="right")
    start = (pick - (ends - tiles)[chrom]) * 500
    if c["wide"]:
        width = rng.integers(200, 2000, c["peaks"])
    else:
        width = np.full(c["peaks"], 500)
    end = np.minimum(start + width, sizes[chrom])
    return [(genome[i][0], int(s), int(e)) for i, s, e in zip(chrom, start, end)]


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("tiles", "peaks", "import"):
        genome, indptr, pos, length = _fragments(c["cells"], c["median"], seed, kind != "import")
        names = ChromSizes(genome)
        if kind == "tiles":
            bounds = {"min_frag_size": 50, "max_frag_size": 1000} if c["bounds"] else {}
            if c["host"]:
                adata = preprocessing.fragments_to_anndata(indptr.cpu().numpy(), pos.cpu().numpy(),
                                                           length.cpu().numpy(), names)
                return {"case": c, "adata": adata, "bounds": bounds}
            layout = _binning.tile_layout(names, c["bin"], EXCLUDED)
            return {"case": c, "frags": (indptr, pos, length), "layout": layout, "bounds": bounds}
        if kind == "peaks":
            regions = _regions.build_regions(_peaks(c, genome), names.names, _device())
            return {"case": c, "frags": (indptr, pos, length), "names": names, "regions": regions}
        frags = synthetic.FragmentMatrix(indptr.cpu().numpy(), pos.cpu().numpy().view(np.uint64),
                                         length.cpu().numpy().view(np.uint32), None)
        text = synthetic.fragment_text(frags, genome, seed=11, order=c["order"], device=_device())
        if c["host"]:
            text = text.cpu().pin_memory()
        return {"case": c, "text": text, "genome": synthetic.fragment_genome(genome)}
    if kind == "knn":
        X = _points(c, seed)
        return {"case": c, "X": X.cpu().numpy() if c["host"] else X}
    csr = _matrix(c, seed, POPULATIONS if kind in ("spectral", "gradient") else 8)
    if kind == "gram":
        op = _eigen.build_operator(csr)
        Z = _block(c, seed)
        a = op.a if c["double"] else op.a32
        return {"case": c, "op": op, "Z": Z, "Zs": (Z * a[:, None]).contiguous(), "W": torch.empty_like(Z),
                "T": torch.empty(op.m, c["block"], dtype=Z.dtype, device=_device())}
    if kind == "gradient":
        g = torch.Generator(device=_device()).manual_seed(seed + 3)
        w = torch.rand(c["features"], generator=g, device=_device()) + 0.5
        return {"case": c, "csr": csr, "w": w.requires_grad_(True)}
    return {"case": c, "csr": csr}


# ---- one pass ----------------------------------------------------------------

def _csr(X):
    return {"indptr": X.indptr, "indices": X.indices, "data": X.data}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "tiles":
        if c["host"]:
            out = preprocessing.add_tile_matrix(state["adata"], bin_size=c["bin"], inplace=False,
                                                counting_strategy=c["strategy"], **state["bounds"])
            return _csr(out.X)
        return _csr(_binning.tile_matrix(*state["frags"], state["layout"], bin_size=c["bin"],
                                         strategy=c["strategy"], **state["bounds"]))
    if kind == "peaks":
        return _csr(_regions.region_matrix(*state["frags"], state["names"], state["regions"],
                                           strategy=c["strategy"]))
    if kind == "import":
        kw = dict(min_num_fragments=c["min_frags"], sorted_by_barcode=c["order"] == "barcode")
        if c["host"]:
            r = _import.import_text(state["text"], state["genome"], host_text=state["text"].numpy(), **kw)
        else:
            r = _import.import_device(state["text"], state["genome"], **kw)
        return {**_csr(r), "n_fragment": r.n_fragment, "frac_dup": r.frac_dup, "frac_mito": r.frac_mito}
    if kind == "counts":
        return preprocessing.column_counts(state["csr"])
    if kind == "build":
        op = _eigen.build_operator(state["csr"])
        return {"colptr": op.colptr, "rowidx": op.rowidx, "values": op.cvalues, "w": op.w, "a": op.a,
                "dinv": op.dinv, "a32": op.a32, "w2_32": op.w2_32, "dinv32": op.dinv32}
    if kind == "gram":
        state["op"].apply(1 if c["double"] else 0, c["block"], state["Z"], state["Zs"], state["T"], state["W"],
                          torch.cuda.current_stream().cuda_stream)
        return state["W"]
    if kind == "spectral":
        evals, evecs = tools.spectral_embedding(state["csr"], None, c["comps"], 0, None, precision="fp64", block=8)
        return {"evals": evals, "evecs": evecs}
    if kind == "gradient":
        f = topk_eigenvalue_sum(state["w"], state["csr"], c["comps"])
        (grad,) = torch.autograd.grad(f, state["w"])
        return {"sum": f.detach(), "grad": grad}
    if c["host"]:
        X = _knn_api.knn(state["X"], n_neighbors=c["k"])
        return {"indices": X.indices, "dist": X.data}
    nbr, dist = _knn_api.knn_arrays(state["X"], c["k"])
    return {"indices": nbr, "dist": dist}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    c = case
    kind = c["kind"]
    if kind in ("tiles", "peaks", "import"):
        frags = c["cells"] * c["median"] * math.exp(0.18)  # mean of LogNormal(ln median, 0.6)
        if kind == "import":  # about 45 bytes a line in, an int64 position and an int32 size out
            return {"bytes": frags * 1.02 * (45 + 12) + 40 * c["cells"], "flops": 0}
        # position and length in; index and count of each nonzero out (about one per fragment for
        # tiles; the share of the genome that the peaks cover for peaks)
        if kind == "tiles":
            per = 1.0 if c["bin"] < 1000 else 0.7
        else:
            width = 1100 if c["wide"] else 500
            per = min(1.0, c["peaks"] * width / GENOME_BP)
        return {"bytes": frags * (12 + 8 * per) + 16 * c["cells"], "flops": 0}
    if kind == "knn":
        n, d, k = c["points"], c["dims"], c["k"]
        return {"bytes": 8.0 * n * d + 16.0 * n * k, "flops": 2.0 * n * n * d}
    nnz = c["cells"] * c["per_cell"] * math.exp(0.045)
    n, m = c["cells"], c["features"]
    if kind == "counts":
        return {"bytes": nnz * (8 if c["valued"] else 4) + 8.0 * m, "flops": nnz}
    if kind == "build":  # indices (and values) in, their transpose out, vectors out
        return {"bytes": 2 * nnz * (8 if c["valued"] else 4) + 16.0 * (n + m) + 28.0 * n + 12.0 * m, "flops": 4 * nnz}
    e = 8 if kind == "spectral" or c.get("double") else 4
    if kind == "gram":
        passes, b = 1, c["block"]
    else:  # a Krylov basis of some 7.5 vectors per component
        passes, b = 7.5 * c["comps"] / 8, 8
    per_pass = 2 * nnz * (8 if c.get("valued") else 4) + 8.0 * (n + m) + e * b * (3.0 * n + 2.0 * m)
    return {"bytes": passes * per_pass, "flops": passes * 4.0 * nnz * b}


# ---- the same in 64 bits, by plain torch ----------------------------------------

def _scaled(csr, w):
    """Row, column and value of every nonzero; 1/norm and 1/degree of every cell (FP64)."""
    n, m = csr.shape
    row = torch.repeat_interleave(torch.arange(n, device=csr.indices.device), csr.indptr[1:] - csr.indptr[:-1])
    col = csr.indices.long()
    x = torch.ones(col.numel(), dtype=torch.float64, device=col.device) if csr.data is None else csr.data.double()

    def over_rows(v):
        return torch.segment_reduce(v, "sum", offsets=csr.indptr)

    r = 1.0 / torch.sqrt(over_rows((x * w[col]) ** 2))
    colsum = torch.zeros(m, dtype=torch.float64, device=col.device).index_add_(0, col, x * w[col] * r[row])
    degree = over_rows(x * w[col] * colsum[col]) * r - 1.0
    return row, col, x, r, 1.0 / degree, over_rows


def _idf(csr):
    n, m = csr.shape
    cnt = torch.bincount(csr.indices.long(), minlength=m).double()
    cnt = torch.where(cnt == 0, 1.0, torch.where(cnt == n, n - 1.0, cnt))
    w = torch.log(n / cnt)
    return torch.ones_like(w) if bool((w == w[0]).all()) else w


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("tiles", "peaks", "import", "gradient"):
        return None  # whole numbers, and a solve too large for a dense one
    if kind == "knn":
        X = _points(c, seed)
        k, rows = c["k"], []
        for q in range(0, c["points"], 500):
            d2 = torch.zeros(min(500, c["points"] - q), c["points"], dtype=torch.float64, device=X.device)
            for t in range(c["dims"]):
                d2 += (X[q:q + 500, t, None] - X[None, :, t]) ** 2
            i = torch.arange(d2.shape[0], device=X.device)
            d2[i, q + i] = math.inf
            v, at = torch.topk(d2, k, largest=False)
            rows.append(torch.gather(v, 1, torch.argsort(at, 1)).sqrt())  # a row's columns ascend
        dist = torch.cat(rows)
        return {"indices": None, "dist": dist.cpu().numpy().ravel() if c["host"] else dist}
    csr = _matrix(c, seed, POPULATIONS if kind == "spectral" else 8)
    n, m = csr.shape
    if kind == "counts":
        x = None if csr.data is None else csr.data.double()
        return torch.bincount(csr.indices.long(), weights=x, minlength=m).double()
    w = _idf(csr)
    row, col, x, r, dinv, over_rows = _scaled(csr, w)
    a = torch.sqrt(dinv) * r
    if kind == "build":
        return {"colptr": None, "rowidx": None, "values": None, "w": w, "a": a, "dinv": dinv, "a32": a,
                "w2_32": w * w, "dinv32": dinv}
    if kind == "gram":
        Z = _block(c, seed).double()
        W = torch.empty_like(Z)
        for j in range(c["block"]):
            t = torch.zeros(m, dtype=torch.float64, device=col.device)
            t.index_add_(0, col, x * (a * Z[:, j])[row])
            W[:, j] = a * over_rows(x * (w * w * t)[col]) - dinv * Z[:, j]
        return W
    A = torch.zeros(n, n, dtype=torch.float64, device=col.device)
    for c0 in range(0, m, 25_000):
        keep = (col >= c0) & (col < c0 + 25_000)
        D = torch.zeros(n, min(25_000, m - c0), dtype=torch.float64, device=col.device)
        D[row[keep], col[keep] - c0] = x[keep] * w[col[keep]]
        A += D @ D.T
    A = a[:, None] * A * a[None, :] - torch.diag(dinv)
    ev = torch.linalg.eigvalsh(A)
    top = ev[torch.argsort(ev.abs(), descending=True)[:c["comps"]]]
    return {"evals": top.sort(descending=True).values.cpu().numpy(), "evecs": None}
