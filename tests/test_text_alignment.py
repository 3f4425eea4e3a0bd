"""The line index and the import of text at any address through the C entry
points: text that does not start on a 16-byte boundary gives the results of
text that does (wide loads are for aligned text only)."""
import ctypes

import numpy as np
import pytest

from test_import import _synthetic

pytestmark = pytest.mark.gpu


def _run(d_text, scratch, n_lines, chroms):
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    sh = torch.cuda.current_stream().cuda_stream
    nb = d_text.numel()
    starts = torch.empty(n_lines + 1, dtype=torch.int64, device="cuda")
    _lib.check(L.sg_frag_index_lines(d_text.data_ptr(), nb, scratch.data_ptr(), n_lines, starts.data_ptr(), sh), "index")
    names = sorted(chroms, key=str.encode)
    size = np.array([chroms[c] for c in names], dtype=np.int64)
    base = np.concatenate([[0], np.cumsum(size)[:-1]])
    blob = np.frombuffer("".join(names).encode(), dtype=np.uint8).copy()
    off = np.concatenate([[0], np.cumsum([len(c) for c in names])]).astype(np.int64)
    mito = np.array([c == "chrM" for c in names], dtype=np.uint8)
    t = [torch.from_numpy(a).cuda() for a in (blob, off, size, base, mito)]
    nw = int(L.sg_frag_workspace_bytes(n_lines, 0))
    ws = torch.empty(nw, dtype=torch.uint8, device="cuda")
    info = (ctypes.c_int64 * 10)()
    _lib.check(L.sg_frag_import(d_text.data_ptr(), nb, starts.data_ptr(), n_lines, *[a.data_ptr() for a in t],
                                len(names), int(size.sum()), None, None, 0, 0, 0, 0, 0, 0, 7, ws.data_ptr(), nw, info,
                                sh), "import")
    K, nnz = info[0], info[1]
    out = [torch.empty(n, dtype=d, device="cuda") for n, d in
           ((K + 1, torch.int64), (nnz, torch.int64), (nnz, torch.int32), (K, torch.int64), (K, torch.int64),
            (K, torch.float64), (K, torch.float64))]
    _lib.check(L.sg_frag_emit(ws.data_ptr(), n_lines, 0, info, *[a.data_ptr() for a in out], sh), "emit")
    return [starts.cpu().numpy()] + [a.cpu().numpy() for a in out]


def test_gpu_text_at_any_address():
    import torch
    from snapatac2_gb300 import _lib
    L = _lib.lib()
    text, chroms = _synthetic()
    text = np.frombuffer(text, dtype=np.uint8).copy()
    a = torch.from_numpy(text).cuda()
    scratch = torch.empty(int(L.sg_frag_line_scratch_bytes(a.numel())), dtype=torch.uint8, device="cuda")
    nl = ctypes.c_int64()
    sh = torch.cuda.current_stream().cuda_stream
    _lib.check(L.sg_frag_count_lines(a.data_ptr(), a.numel(), scratch.data_ptr(), ctypes.byref(nl), sh), "count")
    want = _run(a, scratch, nl.value, chroms)
    assert want[1][-1] > 1000
    for shift in (1, 2, 7, 8, 15):
        buf = torch.zeros(a.numel() + 32, dtype=torch.uint8, device="cuda")
        b = buf[shift:shift + a.numel()]
        b.copy_(a)
        assert b.data_ptr() % 16 == shift
        for x, y in zip(want, _run(b, scratch, nl.value, chroms)):
            np.testing.assert_array_equal(x, y)
