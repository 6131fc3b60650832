"""The float32 products on CUDA cores at the edges of their tiles, chunks and halves."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


def _rows(m, k, pad, seed):
    """m rows of k numbers, rows k + pad apart (pad no multiple of 4: the copies of 16 bytes do not apply)."""
    g = torch.Generator().manual_seed(seed)
    return torch.randn(m, k + pad, generator=g).to(DEV)[:, :k]


@pytest.mark.parametrize("k", [1, 15, 16, 17, 63, 64, 65, 128, 129, 511, 512, 513, 1040, 2049])
@pytest.mark.parametrize("n", [1, 16, 17, 33, 64, 65])
def test_edges_of_tiles_and_halves(ops, n, k):
    """Against float64; a result is a sum of chains of 16 with carried errors: (16 + 2) roundings of 2^-24 of the absolute
    products bound its error. Rows are bit-equal whichever kernel (1, 4, 8, 16, 2 x 16 or 64 rows) and copy ran."""
    for pad in (0, 4 - k % 4 if k % 4 else 4, 3):
        a, w = _rows(130, k, pad, 1), _rows(n, k, pad, 2)
        full = torch.empty(130, n, device=DEV)
        ops.gemm(a, w, full)
        exact, bound = a.double() @ w.double().T, 18 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
        assert bool(((full.double() - exact).abs() <= bound + 1e-30).all())
        for m in (1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65):
            out = torch.full((m + 1, n), 7.0, device=DEV)
            ops.gemm(a[3:3 + m], w, out[:m])
            assert torch.equal(out[:m], full[3:3 + m]), (pad, m)
            assert bool((out[m] == 7.0).all())


def test_infinities_stay_in_their_row(ops):
    a, w = _rows(70, 200, 0, 3), _rows(40, 200, 0, 4)
    a[5, 17], a[66, 3] = float("inf"), float("nan")
    for m in (8, 70):
        out = torch.empty(m, 40, device=DEV)
        ops.gemm(a[:m], w, out)
        bad = [r for r in range(m) if not bool(torch.isfinite(out[r]).all())]
        assert bad == [r for r in (5, 66) if r < m]


def test_bfloat16_of_an_odd_inner_size(ops):
    a, w = _rows(70, 77, 0, 5).bfloat16(), _rows(33, 77, 0, 6).bfloat16()
    full = torch.empty(70, 33, device=DEV)
    ops.gemm(a, w, full)
    bound = 18 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((full.double() - a.double() @ w.double().T).abs() <= bound).all())
    one = torch.empty(3, 33, device=DEV)
    ops.gemm(a[7:10], w, one)
    assert torch.equal(one, full[7:10])


@pytest.mark.parametrize("n,k", [(33, 100), (2400, 516), (70, 1028), (1, 4)])
def test_bfloat16_of_whole_groups_of_four(ops, n, k):
    """Inner sizes that the tensor cores refuse and whose rows begin on 8 bytes (and, a number further on, do not): against float64, and
    rows of the same bits whichever kernel and whichever loads ran."""
    a, w = _rows(130, k, 0, 7).bfloat16(), _rows(n, k, 0, 8).bfloat16()
    odd = torch.empty(a.numel() + 1, dtype=torch.bfloat16, device=DEV)[1:].view(a.shape)
    odd.copy_(a)
    bound = 18 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    exact = a.double() @ w.double().T
    for dt in (torch.float32, torch.bfloat16):
        full = torch.empty(130, n, dtype=dt, device=DEV)
        ops.gemm(a, w, full)
        assert bool(((full.double() - exact).abs() <= bound + (0 if dt == torch.float32 else 2.0 ** -8) * exact.abs()).all())
        for m in (1, 3, 8, 16, 17, 32, 33, 65):
            for src in (a, odd):
                out = torch.full((m + 1, n), 7.0, dtype=dt, device=DEV)
                ops.gemm(src[2:2 + m], w, out[:m])
                assert torch.equal(out[:m], full[2:2 + m]) and bool((out[m] == 7.0).all()), (dt, m)
