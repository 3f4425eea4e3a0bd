"""Cells in the order of their barcodes' bytes (rank_barcodes in
csrc/fragments.cu): names that agree in their first words in every pair, end
inside one another at every length around the 8-byte words, hold zero bytes,
and are as long as the ranking by words takes, and longer."""
import numpy as np
import pytest

from oracle import fragments as ofr
from test_import import GENOME, _check_same, _text

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 2, 257, 1500])
@pytest.mark.parametrize("prefix", ["", "donor_0001#", "s" * 16, "t" * 23, "a_sample_with_a_long_name_and_a_replicate",
                                    "u" * 50, "v" * 52, "w" * 70])
def test_gpu_shared_prefixes(cells, prefix):
    from snapatac2_gb300 import _import
    rng = np.random.default_rng(cells)
    bc = [prefix + f"{i:012x}"[::-1] for i in range(cells)]
    pick = np.concatenate([rng.permutation(cells), rng.integers(0, cells, cells)])
    t = _text([f"chr1\t{int(rng.integers(900))}\t{950}\t{bc[i]}\t1" for i in pick])
    kw = dict(min_num_fragments=0, sorted_by_barcode=False)
    _check_same(_import.import_text(t, GENOME, **kw), ofr.import_fragments(t, GENOME, **kw))


def test_gpu_one_name_inside_another():
    from snapatac2_gb300 import _import
    rng = np.random.default_rng(1)
    bc = sorted({"A" * k + e for k in range(1, 64) for e in ("", "B", "BA", "\x01")}, key=lambda b: rng.random())
    t = _text([f"chr1\t{int(rng.integers(900))}\t{950}\t{b}\t1" for b in bc])
    kw = dict(min_num_fragments=0, sorted_by_barcode=False)
    _check_same(_import.import_text(t, GENOME, **kw), ofr.import_fragments(t, GENOME, **kw))
