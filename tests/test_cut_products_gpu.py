"""Products of more than 64 tokens with K cut, the vector forms of the kernels that add their parts, and steps of such sizes."""
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


@pytest.mark.parametrize("m", [65, 127, 128, 129, 200, 256, 257, 300, 513])
@pytest.mark.parametrize("n,k", [(128, 512), (130, 1032), (2048, 2048), (72, 4096), (3072, 264)])
def test_cut_products_of_more_than_64_tokens(ops, m, n, k):
    """Against float64: bfloat16 products are exact in float32, sums of k of them in any order are off by at most k roundings of 2^-24
    of the absolute products (the tensor cores truncate: twice that); a bfloat16 result rounds once more."""
    from llmengine.engine.context import Workspace
    ws = Workspace(torch.device(DEV))
    a, w = rnd(m, k, seed=1), rnd(n, k, seed=2)
    exact, bound = a.double() @ w.double().T, 2 * k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    parts = ops.gemm_partials(a, w, ws, "t")
    assert bool(((parts.double().sum(0) - exact).abs() <= bound).all())
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m + 1, n), 3.0, dtype=dt, device=DEV)
        for space in (ws, None):
            ops.gemm(a, w, out[:m], space)
            off = (out[:m].double() - exact).abs()
            assert bool((off <= bound + (0 if dt == torch.float32 else 2.0 ** -8) * exact.abs()).all())
            assert bool((out[m] == 3.0).all())


def test_what_is_cut():
    """The rule itself: few tokens as before, more tokens one wave of CTAs at most, and no cut where nobody adds parts."""
    from llmengine.ops import CudaOps
    ops = CudaOps.__new__(CudaOps)
    ops._forms = {}
    for m in (1, 8, 33, 64):
        assert ops._form(m, 2048, 2048, False) == (1, 1, 3) and ops._form(m, 2048, 2048, True)[1] > 1
    for m in (65, 128, 129, 256, 500, 1000, 2048):
        for n in (64, 2048, 3072, 16384):
            for k in (64, 128, 2048, 8192):
                for may in (False, True):
                    swap, splits, stages = ops._form(m, n, k, may)
                    tiles = -(-n // 128) * -(-m // (128 if m <= 128 else 256))
                    assert splits == 1 or (may and swap == 1 and tiles * splits <= 148 and -(-k // 64) >= 2 * (splits - 1))
                    assert swap == (1 if m <= 128 or splits > 1 else 0) and stages == 8


def test_what_is_not_cut():
    """Short products of many tokens, whose parts cost more than they save; the same ones of few tokens or more inputs are cut."""
    from llmengine.ops import CudaOps
    ops = CudaOps.__new__(CudaOps)
    ops._forms = {}
    for m in (200, 256, 512):
        assert ops._form(m, 1024, 1024, True, True)[1] == 1 and ops._form(m, 64, 2048, True, True)[1] == 1
        assert ops._form(m, 1024, 1024, True)[1] > 1 and ops._form(m, 1024, 4096, True, True)[1] > 1 and ops._form(m, 72, 4096, True, True)[1] > 1
    assert ops._form(77, 1024, 1024, True, True)[1] > 1 and ops._form(128, 64, 2048, True, True)[1] > 1
    assert ops._form(1024, 1024, 1024, True)[1] == 1 and ops._form(1024, 1024, 4096, True)[1] > 1


@pytest.mark.parametrize("m,n,k", [(65, 64, 512), (77, 8, 264), (128, 120, 1032), (100, 1, 64)])
def test_products_of_fewer_outputs_than_lanes(ops, m, n, k):
    """Tiles of tokens for them, without a cut: against float64, bounded as above."""
    a, w = rnd(m, k, seed=31), rnd(n, k, seed=32)
    exact, bound = a.double() @ w.double().T, 2 * k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m + 1, n), 3.0, dtype=dt, device=DEV)
        ops.gemm(a, w, out[:m])
        assert bool(((out[:m].double() - exact).abs() <= bound + (0 if dt == torch.float32 else 2.0 ** -8) * exact.abs()).all())
        assert bool((out[m] == 3.0).all())


@pytest.mark.parametrize("parts,rows,width", [(1, 1, 4), (3, 5, 12), (9, 77, 130), (5, 65, 2048), (2, 3, 7)])
def test_reduce_partials_forms_agree(ops, parts, rows, width):
    p = rnd(parts, rows, width, seed=3, dt=torch.float32)
    want = p[0].clone()
    for i in range(1, parts):
        want += p[i]
    for dt in (torch.float32, torch.bfloat16):
        out = torch.empty(rows, width, dtype=dt, device=DEV)
        ops.reduce_partials(p, out)
        assert torch.equal(out, want.to(dt))


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", ("clamped_swish", 1.5, 1.7)])
@pytest.mark.parametrize("parts,rows,ff,block", [(1, 3, 128, 128), (3, 70, 384, 128), (5, 9, 176, 0), (4, 6, 100, 0), (2, 5, 6, 0)])
def test_silu_mul_partials_forms_agree(ops, parts, rows, ff, block, act):
    """A group of four columns at a time gives the bits of one column at a time (the same parts on an address that is no multiple of 16)."""
    p = rnd(parts, rows, 2 * ff, seed=4, dt=torch.float32)
    odd = torch.empty(p.numel() + 1, device=DEV)[1:].view(p.shape)
    odd.copy_(p)
    for dt in (torch.float32, torch.bfloat16):
        a, b = torch.empty(rows, ff, dtype=dt, device=DEV), torch.empty(rows, ff, dtype=dt, device=DEV)
        ops.silu_mul_partials(p, a, block=block, act=act)
        ops.silu_mul_partials(odd, b, block=block, act=act)
        assert torch.equal(a, b)


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", ("clamped_swish", 1.5, 1.7)])
@pytest.mark.parametrize("parts,rows,ff,block", [(5, 64, 2432, 128), (3, 61, 2500, 0), (4, 40, 4096, 128), (1, 300, 516, 0), (9, 37, 4100, 4), (2, 592, 256, 128)])
def test_silu_mul_partials_four_columns_at_a_time(ops, parts, rows, ff, block, act):
    """From 148 * 1,024 results on (rows * ff) and on 16 bytes a thread takes four columns: against float64, with and without a row scale, and
    against the bits of a column at a time (parts on an address that is no multiple of 16). The error: `parts` additions and a handful of
    further operations, each 2^-24 of the halves' absolute sums, of which the activation passes on at most 1.2 times (its slope)."""
    assert rows * ff >= 148 * 1024 and ff % 4 == 0 and block % 4 == 0
    p = rnd(parts, rows, 2 * ff, seed=14, dt=torch.float32)
    odd = torch.empty(p.numel() + 1, device=DEV)[1:].view(p.shape)
    odd.copy_(p)
    sumsq = torch.rand(rows, 3, generator=torch.Generator().manual_seed(15)).to(DEV) + 0.5
    for scaled in (False, True):
        extra = {"row_scale": ops.row_scale(sumsq, 2, 1e-5)} if scaled else {}
        sc = 1.0 / torch.sqrt(sumsq.double().sum(1, keepdim=True) / 2 + 1e-5) if scaled else 1.0
        both, size = p.double().sum(0) * sc, p.double().abs().sum(0) * sc
        if block:
            g, u = both.view(rows, -1, 2, block)[:, :, 0].reshape(rows, ff), both.view(rows, -1, 2, block)[:, :, 1].reshape(rows, ff)
            gs, us = size.view(rows, -1, 2, block)[:, :, 0].reshape(rows, ff), size.view(rows, -1, 2, block)[:, :, 1].reshape(rows, ff)
        else:
            g, u, gs, us = both[:, :ff], both[:, ff:], size[:, :ff], size[:, ff:]
        if act == "silu":
            want, slope = g * torch.sigmoid(g) * u, 1.1
        elif act == "gelu_tanh":
            want, slope = torch.nn.functional.gelu(g, approximate="tanh") * u, 1.2
        else:
            g = torch.clamp(g, max=act[1])
            want, slope = g * torch.sigmoid(act[2] * g) * (torch.clamp(u, -act[1], act[1]) + 1), 1.2
        bound = (parts + 12) * 2.0 ** -24 * slope * (gs * (us + 1) + (gs + 1) * us + gs)
        for dt in (torch.float32, torch.bfloat16):
            a, b = torch.empty(rows, ff, dtype=dt, device=DEV), torch.empty(rows, ff, dtype=dt, device=DEV)
            ops.silu_mul_partials(p, a, block=block, act=act, **extra)
            ops.silu_mul_partials(odd, b, block=block, act=act, **extra)
            assert torch.equal(a, b)
            assert bool(((a.double() - want).abs() <= bound + (0 if dt == torch.float32 else 2.0 ** -8) * want.abs()).all())


@pytest.mark.parametrize("parts,n,nq,nkv,hd,page", [(1, 65, 4, 2, 64, 16), (3, 77, 6, 1, 128, 4), (6, 200, 2, 2, 16, 8)])
@pytest.mark.parametrize("rotate", [True, False])
def test_rotation_of_parts_forms_agree(ops, parts, n, nq, nkv, hd, page, rotate):
    """Eight pairs at a time give the bits of a pair at a time (parts on an address that is no multiple of 16 take that way): the same
    sums in the same order, and both forms' products and differences round once or are fused alike within a bfloat16 step."""
    width = (nq + 2 * nkv) * hd
    p = rnd(parts, n, width, seed=7, dt=torch.float32)
    odd = torch.empty(p.numel() + 1, device=DEV)[1:].view(p.shape)
    odd.copy_(p)
    pos = torch.arange(5, 5 + n, dtype=torch.int32, device=DEV)
    seq = torch.zeros(n, dtype=torch.int32, device=DEV)
    blocks = -(-(n + 5) // page)
    table = torch.randperm(blocks, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(1, -1).to(DEV)
    angle = torch.arange(n + 5)[:, None] * torch.logspace(0, -3, hd // 2)[None]
    cos, sin = (angle.cos().to(DEV), angle.sin().to(DEV)) if rotate else (None, None)
    got = []
    for src in (p, odd):
        qkv = torch.zeros(n, width, dtype=torch.bfloat16, device=DEV)
        k, v = (torch.zeros(blocks + 1, nkv, page, hd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.rope_kv_write(qkv, pos, seq, table, cos, sin, k, v, n, nq, nkv, hd, parts=src)
        got.append((qkv[:, :nq * hd], k, v))
    for a, b in zip(*got):
        torch.testing.assert_close(a, b, rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("form", ["16 bytes", "a pair a thread", "float32", "parts, 16 bytes", "parts, a pair a thread"])
def test_every_form_of_the_rotation_rounds_alike(ops, form):
    """x c - y s and y c + x s with the second product rounded before the sum, as float64 gives it bit for bit, in q and in the cached k: a
    prompt's keys must not depend on which form a step of its size runs."""
    n, nq, nkv, hd, page = 300, 6, 2, 64, 16
    dt = torch.float32 if form == "float32" else torch.bfloat16
    width, half = (nq + 2 * nkv) * hd, hd // 2
    x = rnd(n, width, seed=21, dt=torch.float32)
    parts = x[None].clone() if "parts" in form else None
    qkv = torch.zeros(n, width, dtype=dt, device=DEV) if parts is not None else x.to(dt)
    if "pair" in form:  # an address that is no multiple of 16
        src = parts if parts is not None else qkv
        odd = torch.empty(src.numel() + 1, dtype=src.dtype, device=DEV)[1:].view(src.shape)
        odd.copy_(src)
        parts, qkv = (odd, qkv) if parts is not None else (None, odd)
    values = (x if parts is not None else qkv.float()).clone()
    angle = torch.arange(n, dtype=torch.float64)[:, None] * torch.logspace(0, -3, half, dtype=torch.float64)[None]
    cos, sin = angle.cos().float().to(DEV), angle.sin().float().to(DEV)
    pos, seq = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    table = torch.arange(-(-n // page), dtype=torch.int32, device=DEV).view(1, -1)
    k, v = (torch.zeros(table.numel() + 1, nkv, page, hd, dtype=dt, device=DEV) for _ in range(2))
    ops.rope_kv_write(qkv, pos, seq, table, cos, sin, k, v, n, nq, nkv, hd, parts=parts)
    y = values[:, :(nq + nkv) * hd].reshape(n, nq + nkv, hd)
    a, b, c, s = y[..., :half].double(), y[..., half:].double(), cos[:, None].double(), sin[:, None].double()
    want = torch.cat([(a * c - (b * s).float().double()).float(), (b * c + (a * s).float().double()).float()], -1).to(dt)
    assert torch.equal(qkv[:, :nq * hd].reshape(n, nq, hd), want[:, :nq])
    assert torch.equal(k[:-1].transpose(1, 2).reshape(-1, nkv, hd)[:n], want[:, nq:])
