"""The scratch of a fixed-point product called for another stream than the
current one belongs to that stream: PyTorch hands freed blocks out again by
stream, so a block of the current stream's could still be read or written
there while the product uses it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", [True, False])
def test_gpu_scratch_of_the_stream_that_uses_it(other, monkeypatch):
    import torch
    from snapatac2_gb300 import _eigen
    dev = torch.device("cuda", torch.cuda.current_device())
    n, m, b = 900, 3000, 8
    idx = torch.arange(n * 500, device=dev) % m
    ptr = torch.arange(0, n * 500 + 1, 500, device=dev)
    idx = torch.sort(idx.view(n, 500), 1).values.to(torch.int32).reshape(-1)
    X = torch.randn(m, b, device=dev, dtype=torch.float64)
    one = torch.ones(n, device=dev, dtype=torch.float64)
    want = torch.zeros(n, b, device=dev, dtype=torch.float64)
    want.index_add_(0, torch.arange(n, device=dev).repeat_interleave(500), X[idx.long()])
    side, out = torch.cuda.Stream(dev), torch.empty(n, b, device=dev, dtype=torch.float64)
    torch.cuda.synchronize()
    seen = []
    empty = torch.empty

    def spy(*a, **k):
        if k.get("dtype") is torch.uint8:
            seen.append(torch.cuda.current_stream(dev).cuda_stream)
        return empty(*a, **k)

    monkeypatch.setattr(_eigen.torch, "empty", spy)
    use = side if other else torch.cuda.current_stream(dev)
    _eigen.spmm64(n, ptr, idx, None, m, X, out, one, b, use.cuda_stream)
    if other:  # and the other way round: from a side stream for the default one
        with torch.cuda.stream(side):
            _eigen.spmm64(n, ptr, idx, None, m, X, want.clone(), one, b, torch.cuda.default_stream(dev).cuda_stream)
        torch.cuda.synchronize()
        assert seen == [side.cuda_stream, torch.cuda.default_stream(dev).cuda_stream]
    else:
        assert seen == [use.cuda_stream]
    torch.cuda.synchronize()
    assert float((out - want).abs().max()) <= 1e-11
