"""Per-expert products on rows gathered into the experts' order, against float64 at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


def rnd(*shape, seed, dt=torch.bfloat16):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dt).to(DEV)


# pairs an expert gets: none, one, a tile less one, whole tiles, a tile and one; the last of them has no matrices
COUNTS = [0, 1, 127, 128, 129, 256, 70, 9]


@pytest.mark.parametrize("hidden,ff", [(64, 256), (72, 264), (200, 24), (256, 1032)])
@pytest.mark.parametrize("epilogue", ["gelu", "silu_pairs", "gated_pairs", "relu_squared"])
@pytest.mark.parametrize("weigh", ["output", "input"])
def test_sorted_products_against_float64(ops, hidden, ff, epilogue, weigh):
    from llmengine.engine.context import Workspace
    top, E = 2, len(COUNTS) - 1
    order = torch.repeat_interleave(torch.arange(len(COUNTS)), torch.tensor(COUNTS))
    order = order[torch.randperm(order.numel(), generator=torch.Generator().manual_seed(1))]
    idx = order.view(-1, top).to(torch.int32).contiguous().to(DEV)
    n, pairs = idx.shape[0], epilogue in ("silu_pairs", "gated_pairs")
    x, share = rnd(n, hidden, seed=2), torch.rand(n * top, generator=torch.Generator().manual_seed(3)).to(DEV)
    up = (rnd(E, ff * (2 if pairs else 1), hidden, seed=4, dt=torch.float32) / hidden ** 0.5).bfloat16()
    down = (rnd(E, hidden, ff, seed=5, dt=torch.float32) / ff ** 0.5).bfloat16()
    on_input, on_output = (share, None) if weigh == "input" and epilogue == "relu_squared" else (None, share)
    act_of = {"act": ("clamped_swish", 1.2, 1.7)} if epilogue == "gated_pairs" else {}
    ws = Workspace(torch.device(DEV))
    te, tr = ops.routed_group(idx, E + 1, ops.ROUTED_SORTED_TILE, ws, "t", real_experts=E)
    rows = ops.routed_gather(x, top, te, tr, torch.zeros(tr.numel(), hidden, dtype=torch.bfloat16, device=DEV))
    mid = torch.full((tr.numel(), ff), 7.0, dtype=torch.bfloat16, device=DEV)
    y = torch.full((n * top, hidden), 7.0, device=DEV)
    ops.routed_product_sorted(rows, up, te, tr, mid, epilogue, share=on_input, **act_of)
    ops.routed_product_sorted(mid, down, te, tr, y, "share", share=on_output)
    flat, place = idx.view(-1).long(), torch.full((n * top,), -1, dtype=torch.long, device=DEV)
    live = tr.view(-1) >= 0
    place[tr.view(-1)[live].long()] = torch.nonzero(live).view(-1)
    for p in range(n * top):
        e = int(flat[p])
        if e == E:  # an expert without matrices: no tile holds it, nobody wrote its row
            assert int(place[p]) < 0 and bool((y[p] == 7.0).all())
    real = torch.nonzero(flat < E).view(-1)
    z = torch.einsum("pk,pnk->pn", x[real // top].double(), up[flat[real]].double())
    if epilogue == "gelu":
        want = 0.5 * z * (1 + torch.erf(z / 2 ** 0.5))
    elif epilogue == "relu_squared":
        want = torch.clamp(z * (on_input[real].double()[:, None] if on_input is not None else 1), min=0) ** 2
    else:
        g, u = z[:, 0::2], z[:, 1::2]
        if epilogue == "gated_pairs":
            g, u = torch.clamp(g, max=1.2), torch.clamp(u, -1.2, 1.2)
            want = g * torch.sigmoid(1.7 * g) * (u + 1)
        else:
            want = g * torch.sigmoid(g) * u
    got = mid[place[real]].double()
    # float32 sums of exact products, a smooth activation, one rounding to bfloat16 (2^-9 of the value)
    torch.testing.assert_close(got, want, rtol=2.0 ** -8, atol=1e-4)
    want = torch.einsum("pk,pnk->pn", got, down[flat[real]].double()) * (on_output[real].double()[:, None] if on_output is not None else 1)
    torch.testing.assert_close(y[real].double(), want, rtol=1e-4, atol=1e-4)
    assert bool((mid[(~live).nonzero().view(-1)] == 7.0).all())  # places of padding are left as they are


def test_steps_that_run_sorted(ops):
    assert ops.routed_sorted(torch.bfloat16, (64, 256), 32.0) and not ops.routed_sorted(torch.bfloat16, (64, 256), 31.0)
    assert not ops.routed_sorted(torch.float32, (64, 256), 500.0) and not ops.routed_sorted(torch.bfloat16, (64, 100), 500.0)


def test_no_memory_for_the_copy(ops, monkeypatch):
    """A step whose gathered rows would take more than a quarter of what is free gathers them as it reads them: the same results up to
    rounding, and none of that memory taken. One that finds the scratch there already uses it, whatever is free."""
    from gpu_helpers import Harness
    from llmengine.parts import build_part
    from llmengine.parts.spec import RoutedMLPSpec
    from test_vapelix_gpu import tensors_for
    names = [tuple(f"{k}{e}" for e in range(4)) for k in "ud"]
    spec = RoutedMLPSpec("routed_mlp", 512, 512, 4, 2, "r", "b", *names)
    x, outs = rnd(200, 512, seed=7), []
    calls, gather = [], ops.routed_gather
    monkeypatch.setattr(ops, "routed_gather", lambda a, *rest: (calls.append(a.shape[0]), gather(a, *rest))[1])
    h = Harness(torch.bfloat16, page=16)
    part = build_part("feed_forward", spec, h.env)
    part.load(tensors_for(part.tensor_needs(spec), 5, torch.bfloat16)[1])
    for step, free in enumerate((1 << 20, 1 << 33, 1 << 20)):
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: (free, 1 << 37))
        monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev=None: 0)
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev=None: 0)
        outs.append(part.forward(x, h.ctx([(step + 1, 200, [])])).clone())
        assert len(calls) == step and ("routed.rows" in h.ws._buffers) == (step > 0)
    # both forms: float32 sums of exact products, an activation, one rounding to bfloat16 (2^-9), float32 sums again
    assert (outs[0] - outs[1]).norm() < 2.0 ** -8 * outs[1].norm() and torch.equal(outs[1], outs[2])
