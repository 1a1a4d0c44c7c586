"""The native calls take what the ctypes calls took: tensors that share memory until they are written, objects with a tensor's
is_cuda, is_contiguous() and data_ptr(); and refuse the rest."""
import pytest


class Like:
    def __init__(self, t=None, cuda=True, contiguous=True):
        self.t, self.is_cuda, self.contiguous = t, cuda, contiguous

    def is_contiguous(self):
        return self.contiguous

    def data_ptr(self):
        return self.t.data_ptr()


def test_refusals():
    import bonsai_b200
    with pytest.raises(RuntimeError, match="no CPU path"):
        bonsai_b200.fwht(Like(cuda=False), None, 1024)
    with pytest.raises(RuntimeError, match="contiguous"):
        bonsai_b200.fwht(Like(contiguous=False), None, 1024)
    with pytest.raises(AttributeError):
        bonsai_b200.fwht(3, None, 1024)


@pytest.mark.gpu
def test_memory_shared_until_written(gpu):
    """An output that is a lazy clone gets memory of its own; what it was cloned from keeps its values."""
    import torch
    x = torch.randn(1024, device="cuda")
    base = torch.full((1024,), 5.0, device="cuda")
    out, want = torch._lazy_clone(base), torch.empty(1024, device="cuda")
    assert gpu.fwht_quant(x, None, None, want, 1024) == 0
    assert gpu.fwht_quant(x, None, None, out, 1024) == 0
    assert bool((base == 5.0).all()) and torch.equal(out, want)
    assert gpu.rmsnorm(torch._lazy_clone(x), base, out, 1, 1024, 1e-6) == 0


@pytest.mark.gpu
def test_objects_like_tensors(gpu):
    import torch
    x = torch.randn(2048, device="cuda")
    y = x.clone()
    assert gpu.fwht(x, None, 2048) == 0 and gpu.fwht(Like(y), None, 2048) == 0
    assert torch.equal(x, y)
