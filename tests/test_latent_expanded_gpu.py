"""Latent attention in its expanded form (per-head keys and values from the contexts' latents) against float64 and against the form
over the latents themselves."""
import math

import pytest
import torch
from test_kernels_gpu import DEV, Batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


def _setup(seqs, R, rot, page, seed):
    """Cached rows of every request (up to its last new token) on shuffled pages. -> cache, block table, [rows of request i]"""
    g = torch.Generator().manual_seed(seed)
    lens = [s + n for s, n in seqs]
    blocks = [-(-L // page) for L in lens]
    perm = torch.randperm(sum(blocks) + 3, generator=g).tolist()
    cache = torch.full((len(perm) + 1, 1, page, R + rot), float("nan"), dtype=torch.bfloat16, device=DEV)  # what nobody wrote reaches nothing
    cache[-1] = 0
    table = torch.full((len(seqs), max(blocks)), -1, dtype=torch.int32)
    rows = []
    for i, L in enumerate(lens):
        r = torch.randn(L, R + rot, generator=g).bfloat16().to(DEV)
        rows.append(r)
        for b in range(blocks[i]):
            pg = perm.pop()
            table[i, b] = pg
            part = r[b * page:(b + 1) * page]
            cache[pg, 0, :part.shape[0]] = part
    return cache, table.to(DEV), rows


@pytest.mark.parametrize("H,dim,rot,R", [(4, 128, 64, 512), (3, 64, 32, 256), (2, 64, 64, 72)])
@pytest.mark.parametrize("page,window", [(16, 0), (8, 100), (48, 0)])
@pytest.mark.parametrize("seqs", [[(0, 128)], [(0, 129)], [(127, 128)], [(300, 200)], [(0, 64), (500, 131), (9, 1), (128, 64)]])
def test_expanded_against_float64_and_the_latent_form(ops, H, dim, rot, R, page, window, seqs):
    cache, table, rows = _setup(seqs, R, rot, page, 3)
    b = Batch(seqs)
    b.seq_len = torch.tensor([s + n for s, n in seqs], dtype=torch.int32, device=DEV)
    g = torch.Generator().manual_seed(5)
    n, half, scale = b.n_tokens, rot // 2, 1.0 / math.sqrt(dim + rot)
    q0 = torch.randn(n, H * (dim + rot), generator=g).bfloat16().to(DEV)
    uk = (torch.randn(H, dim, R, generator=g) / math.sqrt(R)).bfloat16().to(DEV)
    uv = (torch.randn(H, dim, R, generator=g) / math.sqrt(R)).bfloat16().to(DEV)
    angle = torch.arange(1000, dtype=torch.float64)[:, None] * torch.logspace(0, -3, half, dtype=torch.float64)[None]
    cos, sin = angle.cos().float().to(DEV), angle.sin().float().to(DEV)
    for per_head in (False, True):
        off = 7  # (any column)
        gate = torch.randn(n, off + (H if per_head else H * dim), generator=g).to(DEV)
        # expanded
        L = -(-b.max_seq_len // 128) * 128
        dense = ops.latent_rows(cache, b, table, torch.empty(len(seqs) * L, R + 64, dtype=torch.bfloat16, device=DEV), L)
        kv = torch.empty(len(seqs) * L, 2 * H * dim, dtype=torch.bfloat16, device=DEV)
        ops.gemm(dense[:, :R], torch.cat([uk.reshape(-1, R), uv.reshape(-1, R)]), kv)
        q = ops.rotate_heads(q0.clone(), H, dim + rot, dim, cos, sin, b.positions)
        out32, out = torch.empty(n, H * dim, device=DEV), torch.empty(n, H * dim, dtype=torch.bfloat16, device=DEV)
        ops.latent_attention_expanded(q, kv[:, :H * dim], kv[:, H * dim:], dense, R, L, b, out32, H, dim, rot, dim, scale, window)
        ops.gate_heads(out32, out, gate, off, H, dim, per_head)
        # over the latents
        ql = torch.empty(n, H, R + rot, dtype=torch.bfloat16, device=DEV)
        ops.latent_query(q0, uk.transpose(1, 2).contiguous(), ql, H, dim, rot, R, rot, cos, sin, b.positions)
        ol, other = torch.empty(n, H, R, dtype=torch.bfloat16, device=DEV), torch.empty(n, H * dim, dtype=torch.bfloat16, device=DEV)
        clean = torch.nan_to_num(cache)
        ops.latent_attention(ql, clean, b, table, ol, R, scale, window)
        ops.heads_product(ol, uv, other.view(n, H, dim), gate=gate[None].contiguous(), gate_off=off, gate_per_head=per_head)
        # float64
        exact, at = torch.empty(n, H * dim, dtype=torch.float64, device=DEV), 0
        for (s, m), r in zip(seqs, rows):
            r = r.double()
            k, v = torch.einsum("hdr,tr->htd", uk.double(), r[:, :R]), torch.einsum("hdr,tr->htd", uv.double(), r[:, :R])
            k = torch.cat([k, r[None, :, R:].expand(H, -1, -1)], -1)
            x = q0[at:at + m].view(m, H, dim + rot).double()
            c, sn = cos[s:s + m].double()[:, None], sin[s:s + m].double()[:, None]
            x1, x2 = x[..., dim:dim + half], x[..., dim + half:]
            x = torch.cat([x[..., :dim], x1 * c - x2 * sn, x2 * c + x1 * sn], -1).transpose(0, 1)
            score = x @ k.transpose(1, 2) * scale
            pos, key = torch.arange(s, s + m, device=DEV)[:, None], torch.arange(s + m, device=DEV)[None]
            hidden = (key > pos) | ((key <= pos - window) if window else torch.zeros_like(key > pos))
            score.masked_fill_(hidden[None], -math.inf)
            exact[at:at + m] = (torch.softmax(score, -1) @ v).transpose(0, 1).reshape(m, H * dim)
            at += m
        gt = torch.sigmoid(gate[:, off:].double())
        exact *= gt.repeat_interleave(dim, 1) if per_head else gt
        err, err_latent = [((o.double() - exact).norm() / exact.norm()).item() for o in (out, other)]
        # four roundings to 2^-9 either way: keys, probabilities, values, results; or mapped queries, probabilities, mapped sums, results.
        # Where one key has nearly all the weight the mapped sum is a cached number and does not round: three against four, so the
        # errors differ by sqrt(4 / 3) = 1.16 at most, 1.25 with the noise of samples this small.
        assert err < 6e-3 and err <= 1.25 * err_latent, (err, err_latent)


def test_what_is_expanded(ops):
    """Only steps of enough tokens a request, and of contexts whose rows stay within the bound."""
    for seqs, want in (([(0, 128)], 128), ([(0, 127)], 0), ([(2000, 300)], 2304), ([(0, 256), (700, 1), (800, 1), (900, 1), (3, 1), (5, 1)], 0),
                       ([(32768 - 128, 128)], 32768), ([(32768 - 127, 128)], 0)):
        assert ops.latent_expanded_rows(Batch(seqs)) == want


def test_scratch_of_expanded_steps_is_bounded(ops, monkeypatch):
    """By bytes, whatever the number of heads, and by what is free: a layer whose scratch would take more runs over the latents, with the
    same results up to rounding, and takes no memory for it."""
    from gpu_helpers import Harness
    from llmengine.config.vapelix import VapelixConfig
    from llmengine.models.vapelix import describe_vapelix
    from llmengine.parts import build_part
    from test_vapelix_gpu import tensors_for
    b = Batch([(16000, 300)])
    for heads in (16, 32, 128):
        row = 2 * (512 + 64 + heads * 256)
        rows = ops.latent_expanded_rows(b, row)
        assert rows == (16384 if 16384 * row <= ops.LATENT_EXPANDED_BYTES else 0) and rows * row <= 336e6
    assert ops.latent_expanded_rows(b, 2 * (576 + 128 * 256)) == 0
    cfg = _wide_config()
    spec = describe_vapelix(VapelixConfig.from_dict(cfg)).layers[0].mixer
    m = cfg["layers"][0]["mixer"]
    outs = []
    for free in (None, 1 << 20):
        if free:
            monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: (free, 1 << 37))
            monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev=None: 0)
            monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev=None: 0)
        h = Harness(torch.bfloat16, page=16, pages=40, nkv=1, hd=m["kv_rank"] + m["rot_dim"])
        part = build_part("mixer", spec, h.env)
        part.load(tensors_for(part.tensor_needs(spec), 5, torch.bfloat16)[1])
        assert part.w_uv.untyped_storage().data_ptr() == part.w_ukv.untyped_storage().data_ptr()  # the value maps are held once
        x = torch.randn(300, cfg["width"], generator=torch.Generator().manual_seed(6)).bfloat16().to(DEV)
        outs.append(part.forward(x, h.ctx([(1, 300, [])]), h.cache).sum(0))
        assert ("latent.kv" in h.ws._buffers) == (free is None)
    assert (outs[0] - outs[1]).norm() < 2e-2 * outs[0].norm()


def _wide_config():
    """Vapelix with heads that the expanded form takes: 64 numbers beside a rotated part of 32 in a layer that runs twice, and 128 beside 64
    of which 48 are rotated; every expert is chosen, so that no rounding changes a choice."""
    from tiny_vapelix import _mixer, _moe
    a = _mixer(3, 64, 32, 64, 64, 40, 0.12, 10000.0, {"factor": 4.0, "original": 64, "fast": 32.0, "slow": 1.0})
    b = _mixer(2, 128, 64, 128, 128, 72, 0.07, 50000.0, dims=48)
    return {"architecture": "Vapelix", "vocab": 301, "width": 128, "norm": {"eps": 1e-6}, "max_positions": 1024,
            "layers": [{"type": "latent_attention", "mixer": a, "mlp": {"kind": "dense", "ff": 256}},
                       {"type": "latent_attention", "mixer": b, "mlp": _moe(64, 3, 3)}],
            "loop": {"start": 0, "stop": 1, "times": 2}, "token_side": {"dim": 16}}


@pytest.mark.parametrize("sharp", [False, True])
def test_whole_model_through_expanded_steps(tmp_path, monkeypatch, ops, sharp):
    """A prompt, its second portion beside other requests' single tokens and beside a second prompt, then decoding over the rows that those
    steps wrote, against the plain implementation; sharp: most heads rest on one or two keys, so that a lost or misplaced one shows."""
    import llmengine
    import numpy as np
    import plain_vapelix as P
    from test_vapelix_gpu import replay, rows_close, sharp_model_dir
    from tiny import Trace, make_model_dir, random_ids
    cfg = _wide_config()
    d = str(tmp_path / "m")
    sharp_model_dir(d, cfg, torch.bfloat16) if sharp else make_model_dir(d, cfg, torch.bfloat16)
    pc, pw = P.read_model(d)
    reqs = {"a": random_ids(420, 301, 1), "b": random_ids(40, 301, 2), "c": random_ids(170, 301, 3)}
    at = {k: 0 for k in reqs}
    t = Trace()

    def step(**new):
        t.add([(k, reqs[k][at[k]:at[k] + n], list(range(n)), at[k]) for k, n in new.items()],
              end=[k for k, n in new.items() if at[k] + n == len(reqs[k])])
        for k, n in new.items():
            at[k] += n

    step(a=200)         # expanded
    step(b=30)          # over the latents
    step(a=199, b=1)    # expanded: a portion behind 200 tokens, a single token behind 30
    step(c=160, a=1, b=1)  # expanded: a whole prompt beside single tokens
    while at["a"] < 420:
        step(**{k: 1 for k in ("a", "b", "c") if at[k] < len(reqs[k])})
    calls = []
    expanded = ops.latent_attention_expanded
    monkeypatch.setattr(ops, "latent_attention_expanded", lambda *a: (calls.append(a[6].n_tokens), expanded(*a))[1])
    gathers = []
    if not sharp:  # the experts' products of prompt-sized steps on gathered rows, which is for larger experts than these
        gather = ops.routed_gather
        monkeypatch.setattr(ops, "ROUTED_SORTED_SIZE", 0)
        monkeypatch.setattr(ops, "routed_gather", lambda x, *a: (gathers.append(x.shape[0]), gather(x, *a))[1])
    eng = llmengine.Engine(d, "bf16", block_size=16)
    eng.configure_cache(num_blocks=48, block_size=16, num_slots=4)
    rows = replay(eng, t)
    assert calls == [200] * 3 + [200] * 3 + [162] * 3  # three runs of layers a step
    assert gathers == ([] if sharp else [200, 200, 162])
    for k, ids in reqs.items():
        rows_close(np.stack([rows[(k, p)] for p in range(len(ids))]), P.forward(pc, pw, ids)[0].numpy(), torch.bfloat16, f"request {k}")
    assert ops.tensor_core_error() == 0 and eng.cm.num_requests == 0
