"""gsb_scale_gradients with the larger array in either place, one of them empty, and
every alignment: products equal torch's bit for bit, and a large second array takes no
longer than the same array in the first place (within a factor of three; one block
alone would take a hundred times as long)."""
import pytest
import torch

from gsplatcu import _lib

pytestmark = pytest.mark.gpu


def _shifted(n, shift):
    return torch.randn(n + shift, device="cuda")[shift:]


def _scale(x, y, g):
    a, b = torch.full_like(x, 7.0), torch.full_like(y, 7.0)
    _lib.call("t", "gsb_scale_gradients", x.numel(), _lib.ptr(x) or None, _lib.ptr(a) or None,
              y.numel(), _lib.ptr(y) or None, _lib.ptr(b) or None, _lib.ptr(g), _lib.stream_of(g))
    return a, b


@pytest.mark.parametrize("n0,n1", [(0, 1), (0, 3_000_001), (15, 100_003), (100_003, 15), (4096, 4096)])
@pytest.mark.parametrize("s0,s1", [(0, 0), (1, 0), (0, 3)])
def test_either_array_may_be_the_large_one(cuda_ok, n0, n1, s0, s1):
    x, y, g = _shifted(n0, s0), _shifted(n1, s1), torch.tensor(-1.7, device="cuda")
    a, b = _scale(x, y, g)
    assert torch.equal(a, x * g) and torch.equal(b, y * g)


def test_second_array_is_as_fast_as_the_first(cuda_ok):
    big, none = torch.randn(20_000_000, device="cuda"), torch.empty(0, device="cuda")
    g = torch.tensor(0.5, device="cuda")

    def us(x, y):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(5):
            _scale(x, y, g)
            ev[0].record()
            _scale(x, y, g)
            ev[1].record()
            ev[1].synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        return best

    assert us(none, big) < 3.0 * us(big, none)
