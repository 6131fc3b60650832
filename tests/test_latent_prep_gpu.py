"""The latents' norms, rotation and cache write of prompt-sized steps: a warp a token against a block a token."""
import pytest
import torch
from test_kernels_gpu import DEV, Batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [65, 68, 131])
@pytest.mark.parametrize("Rq,R,dr,rot", [(768, 512, 64, 64), (1024, 384, 256, 32), (4, 4, 4, 2), (132, 260, 12, 0), (1028, 512, 64, 64)])
def test_warps_and_blocks_agree(ops, dt, n, Rq, R, dr, rot):
    """Sums on an address that is no multiple of 16 go the block's way. The sums of squares are added in another order: 2^-24 times the
    square root of their number, far below the bound of a few float32 steps (or one bfloat16 step)."""
    page, g = 16, torch.Generator().manual_seed(n)
    b = Batch([(3, n)])
    table = torch.randperm(-(-(n + 3) // page), generator=g).to(torch.int32).view(1, -1).to(DEV)
    width = 8 + Rq + R + dr + 4
    sums = torch.randn(1, n, width, generator=g).to(DEV)
    odd = torch.empty(sums.numel() + 1, device=DEV)[1:].view(sums.shape)
    odd.copy_(sums)
    wq, wk = torch.rand(Rq, generator=g).to(DEV) + 0.5, torch.rand(R, generator=g).to(DEV) + 0.5
    angle = torch.arange(n + 3)[:, None] * torch.logspace(0, -2, max(rot // 2, 1))[None]
    cos, sin = (angle.cos().to(DEV), angle.sin().to(DEV)) if rot else (None, None)
    got = []
    for src in (sums, odd):
        cq = torch.full((n + 1, Rq), 7.0, dtype=dt, device=DEV)
        cache = torch.full((table.numel() + 1, 1, page, R + dr), 7.0, dtype=dt, device=DEV)
        ops.latent_prep(src, 8, Rq, 8 + Rq, R, dr, rot, wq, wk, 1e-5, cos, sin, b, table, cq[:n], cache)
        assert bool((cq[n] == 7.0).all())
        got.append((cq, cache))
    tol = dict(rtol=2e-6, atol=1e-6) if dt == torch.float32 else dict(rtol=2.0 ** -7, atol=1e-6)
    for x, y in zip(*got):
        torch.testing.assert_close(x, y, **tol)


@pytest.mark.parametrize("Rq,R,dr,rot", [(768, 512, 64, 64), (4, 4, 4, 2), (132, 260, 12, 0)])
def test_float32_rows_do_not_depend_on_the_step(ops, Rq, R, dr, rot):
    """The same float32 tokens in steps of 1, 64, 65 and 131: the same bits."""
    page, n, g = 16, 131, torch.Generator().manual_seed(5)
    table = torch.randperm(-(-n // page), generator=g).to(torch.int32).view(1, -1).to(DEV)
    sums = torch.randn(n, Rq + R + dr, generator=g).to(DEV)
    wq, wk = torch.rand(Rq, generator=g).to(DEV) + 0.5, torch.rand(R, generator=g).to(DEV) + 0.5
    angle = torch.arange(n)[:, None] * torch.logspace(0, -2, max(rot // 2, 1))[None]
    cos, sin = (angle.cos().to(DEV), angle.sin().to(DEV)) if rot else (None, None)

    def run(step):
        cq = torch.empty(n, Rq, device=DEV)
        cache = torch.zeros(table.numel() + 1, 1, page, R + dr, device=DEV)
        for at in range(0, n, step):
            m = min(step, n - at)
            ops.latent_prep(sums[at:at + m].clone()[None], 0, Rq, Rq, R, dr, rot, wq, wk, 1e-5, cos, sin, Batch([(at, m)]), table, cq[at:at + m], cache)
        return cq, cache

    want = run(131)
    for step in (1, 64, 65):
        for x, y in zip(run(step), want):
            assert torch.equal(x, y), step
