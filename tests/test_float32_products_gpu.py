"""The 32-bit path's products hold and multiply every number in float32, however far apart the numbers of a row lie."""
import pytest
import torch
from gpu_helpers import DEV, Harness

from llmengine.parts import build_part
from llmengine.parts.spec import HeadSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2048, 8192])
@pytest.mark.parametrize("far", [1e2, 1e4, 1e6])
def test_rows_of_wide_range(k, far):
    """A product of a loaded part (the head, 1,061 outputs) with zero, one-hot and sparse weight rows, with one input channel whose
    activations are `far` times the others' and its weights as much smaller, and with activation rows that have a few such numbers. A
    result is a sum of fused chains of 16 with the sums' rounding errors carried: within 18 roundings of 2^-24 of sum |a| |w|."""
    g = torch.Generator().manual_seed(k + int(far))
    n = 1061
    w, a = torch.randn(n, k, generator=g) * 0.02, torch.randn(300, k, generator=g)
    w[:, 5] /= far
    a[:, 5] *= far  # one channel, in every row
    w[0] = 0.0
    w[1:33] = 0.0
    w[torch.arange(1, 33), torch.arange(1, 33) * 37] = 1.0  # one-hot
    w[33:65] *= (torch.rand(32, k, generator=g) < 0.01)  # sparse
    a[100:200, 9::k // 4] *= far  # four more, of weights like the others
    head = build_part("head", HeadSpec("w", n, k), Harness(torch.float32).env)
    head.load({"w": w.to(DEV)})
    exact, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    for m in (1, 8, 9, 40, 300):
        h = Harness(torch.float32)
        got = head.forward(a[-m:].contiguous().to(DEV), h.ctx([(1, 1, [])])).cpu()
        assert bool((got[:, 0] == 0).all())
        assert torch.equal(got[:, 1:33], a[-m:, torch.arange(1, 33) * 37])
        assert bool(((got.double() - exact[-m:]).abs() <= 18 * 2.0 ** -24 * size[-m:]).all()), m
