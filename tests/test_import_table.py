"""Fragment import (csrc/fragments.cu) against the oracle where its fast forms
change over: lines too long to be staged, fields at every byte alignment,
numbers of up to 20 digits with leading zeros, barcodes that share their first
eight bytes or begin one another, more cells than are ordered by counting, a
barcode table that has to grow, and the three ways the matrix comes into order
(as read, by cell and chromosome, by every bit)."""
import numpy as np
import pytest

from oracle import fragments as ofr
from test_import import GENOME, _check_same, _text

pytestmark = pytest.mark.gpu


def _same(text, **kw):
    from snapatac2_gb300 import _import
    kw = dict(min_num_fragments=0, **kw)
    _check_same(_import.import_text(text, GENOME, **kw), ofr.import_fragments(text, GENOME, **kw))


def _line(rng, bc, chrom="chr1", size=None):
    s = int(rng.integers(0, 900))
    return f"{chrom}\t{s}\t{s + (size or int(rng.integers(1, 90)))}\t{bc}\t{int(rng.integers(1, 5))}"


@pytest.mark.parametrize("nl", ["\n", "\r\n"])
@pytest.mark.parametrize("trailing", [True, False])
def test_gpu_fields_at_every_alignment(nl, trailing):
    rng = np.random.default_rng(5)
    bcs = ["A" * k for k in (1, 2, 3, 7, 8, 9, 15, 16, 17, 31)] + ["AAAAAAAAC", "AAAAAAAAB", "AAAAAAAABB", "B", "AB"]
    lines = ["# comment", "#"] + [_line(rng, bcs[int(rng.integers(len(bcs)))], ("chr1", "chr2", "chrUn")[i % 3])
                                  for i in range(900)]
    lines[40] = "chr1\t00000000000000000000000000012\t0000000000000000000000000000000044\tA\t00000000003"
    lines[41] = "chr2\t7\t9\tAAAAAAAA\t4294967295\t.\tmore\tfields"
    lines[42] = "chr1\t5\t6\tAB\t.\t."
    lines[43] = "chr2\t5\t6\tB"
    _same(_text(lines, nl=nl, trailing=trailing), sorted_by_barcode=False)


def test_gpu_lines_too_long_to_stage():
    rng = np.random.default_rng(6)
    long = "Q" * 30000
    lines = [_line(rng, long if i % 7 == 0 else f"BC{i % 5}") for i in range(600)]
    _same(_text(lines), sorted_by_barcode=False)
    _same(_text([x + "\t.\t" + "x" * 500 for x in lines[1:6]] * 60), sorted_by_barcode=False)


@pytest.mark.parametrize("bad", ["chr1\t1844674407370955161600\t5\tA\t1", "chr1\t18446744073709551616\t5\tA\t1",
                                 "chr1\t1\t5/\tA\t1", "chr1\t1\t5:\tA\t1", "chr1\t1\t 5\tA\t1", "chr1\t-1\t5\tA\t1",
                                 "chr1\t1\t5\tA\t4294967296", "chr1\t1\t5\tA\t1x", "chr1\t1\t5\tA\t1\t*",
                                 "chr1\t1\t5\tA\t1\t", "chr1\t\t5\tA\t1", "chr1\t1\t5", ""])
def test_gpu_malformed_fields(bad):
    from snapatac2_gb300 import _import
    t = _text(["chr1\t1\t5\tA\t1", "chr2\t3\t9\tA\t2", bad, "chr1\t1\t5\tA\t1"])
    with pytest.raises(ValueError):
        ofr.import_fragments(t, GENOME, min_num_fragments=0)
    with pytest.raises(ValueError, match="line 3"):
        _import.import_text(t, GENOME, min_num_fragments=0)


@pytest.mark.parametrize("cells,order", [(1, "position"), (300, "position"), (300, "sizes"), (300, "shuffle"),
                                         (9000, "position"), (9000, "barcode"), (300, "hot"), (300, "barcode")])
def test_gpu_matrix_order(cells, order):
    rng = np.random.default_rng(cells + len(order))
    n = max(6000, 2 * cells)
    bc = np.array([f"{'S1_LANE2_' if i % 2 else ''}{i:05d}" for i in rng.permutation(cells)])
    c = np.concatenate([np.arange(cells), rng.integers(0, cells, n - cells)])
    ch = rng.integers(0, 3, n)
    s = rng.integers(0, 900 if order != "hot" else 2, n)  # hot: long runs at equal positions
    size = rng.integers(1, 90, n)
    key = {"position": (size, s, ch), "sizes": (-size, s, ch), "hot": (rng.random(n), s, ch),
           "barcode": (size, s, ch, bc[c]), "shuffle": (rng.random(n),)}[order]
    o = np.lexsort(key)
    names = ["chr2", "chr1", "chr10"]  # not the order of the genome table
    t = _text([f"{names[ch[i]]}\t{s[i]}\t{s[i] + size[i]}\t{bc[c[i]]}\t1" for i in o])
    _same(t, sorted_by_barcode=order == "barcode")


def test_gpu_table_grows():
    """1.2 million barcodes: more than the first table's 2^20 slots."""
    from snapatac2_gb300 import _import
    n = 1_200_000
    t = "".join(f"chr1\t{i % 900}\t{i % 900 + 5}\t{i:07x}\t1\n" for i in range(n)).encode()
    r = _import.import_text(t, GENOME, min_num_fragments=0)
    assert r.info["barcodes"] == n and r.info["cells"] == n
    assert r.obs_names[:3] == ["0000000", "0000001", "0000002"] and r.obs_names[-1] == f"{n - 1:07x}"
    i = np.arange(n)
    np.testing.assert_array_equal(r.indptr, np.arange(n + 1))
    np.testing.assert_array_equal(r.indices - r.indices.min(), i % 900)
    np.testing.assert_array_equal(r.n_fragment, np.ones(n, dtype=np.uint64))
