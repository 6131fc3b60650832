"""The float32 products in whole numbers (csrc/kernels/gemm_digits.cu) at the edges of their tiles and of the form."""
import pytest
import torch

from llmengine.engine.context import Workspace

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


@pytest.fixture(scope="module")
def ws():
    return Workspace(torch.device(DEV))


def _rows(m, k, seed, pad=0, spiky=False):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k + pad, generator=g)
    if spiky:
        x = x * x * x
    return x.to(DEV)[:, :k]


def _bound(a, w):
    """Roundings of the operands (half a step of 2^-31 of the row's scale, which is at most 2.04 times its largest magnitude), the
    products left out (places 0 to 2, at most K * 2^14 * (3 * 2^16 + 2 * 2^8 + 1) of both scales' steps) and that of the result."""
    a, w = a.double().abs(), w.double().abs()
    sa, sw = 2.04 * a.amax(1, keepdim=True) * 2.0 ** -31, 2.04 * w.amax(1, keepdim=True) * 2.0 ** -31
    left_out = a.shape[1] * 2.0 ** 14 * (3 * 2 ** 16 + 2 * 2 ** 8 + 1) * sa * sw.T
    return 0.5 * (sa * w.sum(1)[None] + a.sum(1, keepdim=True) * sw.T) + left_out + 2.0 ** -24 * (a @ w.T)


@pytest.mark.parametrize("n,k", [(1024, 2048), (1037, 2052), (1201, 2049), (640, 8192), (257, 8260), (3000, 2116)])
@pytest.mark.parametrize("spiky", [False, True])
def test_products_against_float64(ops, ws, n, k, spiky):
    """Within the derived bound and, over all results, no further from float64 than the chains of multiply-adds; rows are the same bits
    whatever else is in the batch, with every kernel (up to 8 rows, tiles of 16 to 128) and every cut of K."""
    full_a, w = _rows(300, k, 1, pad=3, spiky=spiky), _rows(n, k, 2, pad=1) * 0.02
    dw = ops.digit_weight(w)
    assert dw is not None
    full, chains = torch.empty(300, n, device=DEV), torch.empty(300, n, device=DEV)
    ops.gemm(full_a, dw, full, ws)
    ops.gemm(full_a, w, chains)
    exact = full_a.double() @ w.double().T
    assert bool(((full.double() - exact).abs() <= _bound(full_a, w)).all())
    assert float((full.double() - exact).norm()) <= float((chains.double() - exact).norm())
    for m in (1, 2, 7, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129):
        out = torch.full((m + 1, n), 7.0, device=DEV)
        a = full_a[5:5 + m].contiguous() if m % 2 else full_a[5:5 + m]
        ops.gemm(a, dw, out[:m], ws)
        assert torch.equal(out[:m], full[5:5 + m]), m
        assert bool((out[m] == 7.0).all())
    for cuts in (1, 2, 4, 8):
        out = torch.empty(70, n, device=DEV)
        ops._gemm_digits(ops.row_digits(full_a[9:79], ws), dw, out, cuts)
        assert torch.equal(out, full[9:79]), cuts
    torch.cuda.synchronize()
    assert ops.tensor_core_error() == 0


@pytest.mark.parametrize("m", [3, 8, 20, 130])
def test_rows_that_do_not_fit_the_form(ops, ws, m):
    """Infinities, NaN and rows of numbers below 2^-90: by multiply-adds, and in their row alone. Zero rows give zero."""
    a, w = _rows(m, 2100, 3), _rows(1000, 2100, 4)
    w[:, 40] = 0.0
    a[0, 17], a[0, 900] = float("inf"), 1.0
    a[1] *= 2.0 ** -100
    a[2] = 0.0
    if m > 3:
        a[4, 3], a[5, 40], a[6, 7] = float("nan"), float("-inf"), 2.0 ** 120
    want = a.double() @ w.double().T
    dw, got = ops.digit_weight(w), torch.empty(m, 1000, device=DEV)
    ops.gemm(a, dw, got, ws)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    finite = torch.isfinite(want)
    assert torch.equal(got[torch.isinf(want)].double(), want[torch.isinf(want)])
    scale = (a.double().abs().nan_to_num(0, 0, 0) @ w.double().abs().T)
    # multiply-adds in ascending k: as many roundings of 2^-24 as there are numbers
    assert bool(((got.double() - want).abs()[finite] <= (2100 * 2.0 ** -24 * scale)[finite]).all())
    assert bool((got[2] == 0).all())


def test_weights_that_stay_as_they_are(ops):
    w = _rows(1024, 2048, 5)
    assert ops.digit_weight(w[:1000]) is None and ops.digit_weight(w.bfloat16()) is None
    w[3, 5] = float("inf")
    assert ops.digit_weight(w) is None
    w[3] = 2.0 ** -100
    assert ops.digit_weight(w) is None
    w[3] = 0.0
    assert ops.digit_weight(w) is not None


@pytest.mark.parametrize("dim", [512, 516, 2048, 4160, 8192, 16384])
@pytest.mark.parametrize("m", [1, 9, 600])
def test_norm_and_activation_leave_the_digits_of_their_rows(ops, ws, dim, m):
    """The kernels' rows are the bits of the kernels without digits, and the digits those of the rows."""
    def as_bytes(rows):
        return rows.digits.clone(), rows.exps.clone(), rows.sums.clone()

    h, delta, weight = _rows(m, dim, 6), _rows(m, dim, 7)[None].contiguous(), _rows(1, dim, 8)[0].contiguous()
    h[0, 3] = float("inf") if m > 1 else 1.0
    plain, out = torch.empty(m, dim, device=DEV), torch.empty(m, dim, device=DEV)
    ops.rmsnorm(h.clone(), weight, 1e-5, plain, delta=delta)
    rows = ops.digit_rows(out, ws, weight)
    ops.rmsnorm(h.clone(), weight, 1e-5, out, delta=delta, digits=rows)
    assert torch.equal(out.view(torch.int32), plain.view(torch.int32))
    got = as_bytes(rows)
    for g, w in zip(got, as_bytes(ops.row_digits(plain, ws))):
        first = 1 if m > 1 else 0  # (a row of infinities is marked, its digits are not read)
        assert torch.equal(g[first:], w[first:])
    gate_up = _rows(m, 2 * dim, 9)
    ops.silu_mul(gate_up, plain)
    rows = ops.silu_mul_digits(gate_up, out, ws)
    assert torch.equal(out, plain)
    got = as_bytes(rows)
    for g, w in zip(got, as_bytes(ops.row_digits(plain, ws))):
        assert torch.equal(g, w)
