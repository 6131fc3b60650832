"""Float32 attention on CUDA cores: segments with a CTA each against one CTA that walks over all of them."""
import math

import pytest
import torch
from test_kernels_gpu import DEV, Batch, _attention_ref, _paged_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from llmengine.ops import get_ops
    return get_ops()


@pytest.mark.parametrize("nq,nkv,hd,page,window", [(8, 2, 64, 16, 0), (6, 1, 32, 4, 0), (9, 1, 20, 16, 0), (4, 4, 128, 16, 130), (2, 1, 256, 8, 0),
                                                   (12, 1, 18, 4, 127)])
@pytest.mark.parametrize("length", [1, 64, 127, 128, 129, 256, 257, 400])
def test_a_token_alone_and_in_a_prompt(ops, nq, nkv, hd, page, window, length):
    """The last token alone (few rows: a CTA a segment), at the end of a portion, and at the end of the whole prompt beside many others
    (more rows, and so many CTAs that each walks over all segments): bit-equal, and near float64."""
    others = 40
    kc, vc, table, dense = _paged_setup(torch.float32, nkv, hd, page, [length] * others, others * ((length + page - 1) // page) + 2, seed=length)
    scale = 1.0 / math.sqrt(hd)
    q = torch.randn(others, length, nq * hd, generator=torch.Generator().manual_seed(7)).to(DEV)

    def run(entries):
        b = Batch(entries)
        rows = torch.cat([q[i, s:s + n] for i, (s, n) in enumerate(entries)])
        out = torch.empty_like(rows)
        ops.paged_attention(rows, kc, vc, b, table[:len(entries)].contiguous(), out, nq, nkv, hd, scale, window)
        return out, b

    alone, b = run([(length - 1, 1)])
    portion, _ = run([(length - min(length, 5), min(length, 5))])
    whole, _ = run([(0, length)] * others)
    assert torch.equal(portion[-1], alone[0])
    assert torch.equal(whole[length - 1], alone[0])
    K, V = dense[0]
    ref = _attention_ref(q[0, -1].view(nq, hd).cpu().double(), K.double(), V.double(), length - 1, nq, nkv, hd, scale, window)
    torch.testing.assert_close(alone[0].cpu(), ref.float(), rtol=2e-5, atol=2e-5)


def test_values_behind_a_token_do_not_reach_it(ops):
    """A later token of the same portion whose value row is NaN leaves earlier tokens' results as they are."""
    kc, vc, table, _ = _paged_setup(torch.float32, 2, 64, 16, [100], 9, seed=3)
    q = torch.randn(100, 8 * 64, generator=torch.Generator().manual_seed(8)).to(DEV)
    outs = []
    for poison in (False, True):
        if poison:
            vc[table[0, 4], :, 6] = float("nan")  # position 70
        out = torch.empty_like(q)
        ops.paged_attention(q, kc, vc, Batch([(0, 100)]), table, out, 8, 2, 64, 0.125)
        outs.append(out)
    assert torch.equal(outs[0][:70], outs[1][:70]) and bool(outs[1][70:].isnan().all())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", [127, 128, 129, 255, 256])
@pytest.mark.parametrize("window", [0, 130])
def test_a_key_that_is_no_number_reaches_every_token_that_sees_it(ops, bad, where, window):
    """NaN (and +-inf, by a query's signs: -inf is a probability of zero, +inf has none) in the key at `where`, which alone may be what a
    token sees of a segment of 128: a token on its own (a CTA a segment), a portion, and whole prompts beside many (one CTA walks).
    Tokens before it, and those whose window has left it behind, keep their bits."""
    nq, nkv, hd, page, others, length, scale = 8, 2, 64, 16, 40, 300, 0.125
    kc, vc, table, _ = _paged_setup(torch.float32, nkv, hd, page, [length] * others, others * 19 + 2, seed=3)
    q = torch.randn(others, length, nq * hd, generator=torch.Generator().manual_seed(9)).to(DEV)
    q[0, :, ::hd] = q[0, :, ::hd].abs() + 0.1  # (the first number of every head: an infinite key scores +inf there)

    def run(entries):
        rows = torch.cat([q[i, s:s + n] for i, (s, n) in enumerate(entries)])
        out = torch.empty_like(rows)
        ops.paged_attention(rows, kc, vc, Batch(entries), table[:len(entries)].contiguous(), out, nq, nkv, hd, scale, window)
        return out

    clean = run([(0, length)] * others)[:length]
    kc[table[0, where // page], :, where % page, 0] = bad
    whole = run([(0, length)] * others)[:length]
    portion = torch.cat([run([(at, min(50, length - at))]) for at in range(0, length, 50)])
    alone = torch.cat([run([(t, 1)]) for t in range(length)])
    sees = torch.arange(length) >= where
    if window:
        sees &= torch.arange(length) < where + window
    for got in (whole, portion, alone):
        assert bool(got[sees].isnan().all()) and torch.equal(got[~sees], clean[~sees])


def test_keys_of_minus_infinity_weigh_nothing(ops):
    """Scores of -inf, alone in a token's last segment and alone in its first: as if the keys were not there."""
    nq, nkv, hd, page, length, scale = 8, 2, 64, 16, 260, 0.125
    kc, vc, table, dense = _paged_setup(torch.float32, nkv, hd, page, [length], 19, seed=4)
    q = torch.randn(length, nq * hd, generator=torch.Generator().manual_seed(9)).to(DEV)
    q[:, ::hd] = q[:, ::hd].abs() + 0.1
    for dead in (range(128, 129), range(0, 128)):
        keys = kc.clone()
        for t in dead:
            keys[table[0, t // page], :, t % page, 0] = float("-inf")
        K, V = dense[0]
        K = K.clone()
        K[list(dead), :, 0] = float("-inf")
        first = dead.stop if dead.start == 0 else 0
        whole = torch.empty_like(q)
        ops.paged_attention(q, keys, vc, Batch([(0, length)]), table, whole, nq, nkv, hd, scale)
        for t in (max(first, 128), 200, 259):
            alone = torch.empty(1, nq * hd, device=DEV)
            ops.paged_attention(q[t:t + 1], keys, vc, Batch([(t, 1)]), table, alone, nq, nkv, hd, scale)
            assert torch.equal(alone[0], whole[t])
            ref = _attention_ref(q[t].view(nq, hd).cpu().double(), K.double(), V.double(), t, nq, nkv, hd, scale, 0)
            torch.testing.assert_close(alone[0].cpu(), ref.float(), rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,hd,window", [(12, 1, 18, 0), (6, 2, 20, 0), (5, 5, 48, 50), (3, 1, 132, 0), (4, 4, 256, 0), (12, 1, 80, 9)])
@pytest.mark.parametrize("seqs", [[(0, 5)], [(0, 16), (0, 17)], [(60, 3), (0, 33), (200, 1)], [(127, 2), (0, 70)]])
def test_tiles_that_are_part_empty(ops, dt, nq, nkv, hd, window, seqs):
    """Few keys, few rows and head sizes whose rows begin on four numbers or do not, against float64. A result is a weighted mean of values
    of size one: some hundred float32 roundings, and in bfloat16 the operands' products exact in float32 and one rounding at the end."""
    lens, page, scale = [s + n for s, n in seqs], 8, 1.0 / math.sqrt(hd)
    kc, vc, table, dense = _paged_setup(dt, nkv, hd, page, lens, sum(-(-x // page) for x in lens) + 2, seed=hd)
    b = Batch(seqs)
    q = torch.randn(b.n_tokens, nq * hd, generator=torch.Generator().manual_seed(11)).to(dt).to(DEV)
    out = torch.full_like(q, float("nan"))
    ops.paged_attention(q, kc, vc, b, table, out, nq, nkv, hd, scale, window)
    for i, (s, pos) in enumerate(b.tokens):
        K, V = dense[s]
        ref = _attention_ref(q[i].view(nq, hd).cpu().double(), K.double(), V.double(), pos, nq, nkv, hd, scale, window)
        torch.testing.assert_close(out[i].float().cpu(), ref.float(), rtol=2.0 ** -8 if dt == torch.bfloat16 else 2e-5, atol=2e-5)


@pytest.mark.parametrize("nq,nkv,hd,page,window", [(4, 4, 64, 16, 0), (16, 2, 128, 16, 0), (3, 1, 20, 4, 0), (10, 2, 64, 8, 700)])
@pytest.mark.parametrize("lengths", [(1, 1023, 1024, 1025), (2048, 2049, 5, 1500), (4096, 300, 129, 3100), (4097, 64, 2000, 1),
                                     (8191, 8192, 130, 5000), (8193, 8192, 1, 300)])
def test_single_tokens_behind_many_segments(ops, nq, nkv, hd, page, window, lengths):
    """Single tokens of several requests, clusters of 8 CTAs with one to 8 segments of 128 keys each (8,192 keys) and one key beyond (where
    segments and a merge take over), against the last token of portions of five: bit-equal, whatever the other requests' lengths."""
    kc, vc, table, dense = _paged_setup(torch.float32, nkv, hd, page, list(lengths), sum(-(-n // page) for n in lengths) + 2, seed=hd)
    q = torch.randn(len(lengths), 5, nq * hd, generator=torch.Generator().manual_seed(12)).to(DEV)
    rows = q[:, -1].contiguous()
    out = torch.full_like(rows, float("nan"))
    ops.paged_attention(rows, kc, vc, Batch([(n - 1, 1) for n in lengths]), table, out, nq, nkv, hd, 0.2, window)
    for i, n in enumerate(lengths):
        m = min(n, 5)
        portion, rows_i = torch.empty(m, nq * hd, device=DEV), q[i, 5 - m:].contiguous()
        ops.paged_attention(rows_i, kc, vc, Batch([(n - m, m)]), table[i:i + 1].contiguous(), portion, nq, nkv, hd, 0.2, window)
        if m > 1:
            assert torch.equal(portion[-1], out[i]), n
        K, V = dense[i]
        ref = _attention_ref(rows[i].view(nq, hd).cpu().double(), K.double(), V.double(), n - 1, nq, nkv, hd, 0.2, window)
        torch.testing.assert_close(out[i].cpu(), ref.float(), rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("n,nkv,group,hd,most", [(80, 4, 2, 64, 1024), (80, 4, 2, 64, 1025), (64, 4, 3, 32, 2048), (150, 2, 8, 128, 1024)])
def test_single_tokens_of_many_requests(ops, n, nkv, group, hd, most):
    """So many requests that a cluster is one CTA or two, with up to 8 segments each (and one key beyond): bit-equal to the last token of
    portions of two."""
    g = torch.Generator().manual_seed(n + most)
    lengths = [most, 2] + torch.randint(2, most + 1, (n - 2,), generator=g).tolist()
    kc, vc, table, dense = _paged_setup(torch.float32, nkv, hd, 16, lengths, sum(-(-m // 16) for m in lengths) + 2, seed=hd)
    q = torch.randn(n, 2, nkv * group * hd, generator=g).to(DEV)
    out, both = torch.full_like(q[:, 0].contiguous(), float("nan")), torch.empty_like(q)
    ops.paged_attention(q[:, 1].contiguous(), kc, vc, Batch([(m - 1, 1) for m in lengths]), table, out, nkv * group, nkv, hd, 0.2)
    ops.paged_attention(q.view(2 * n, -1), kc, vc, Batch([(m - 2, 2) for m in lengths]), table, both.view(2 * n, -1), nkv * group, nkv, hd, 0.2)
    assert torch.equal(out, both[:, 1])
    for i in (0, 1, n // 2):
        K, V = dense[i]
        ref = _attention_ref(q[i, 1].view(nkv * group, hd).cpu().double(), K.double(), V.double(), lengths[i] - 1, nkv * group, nkv, hd, 0.2, 0)
        torch.testing.assert_close(out[i].cpu(), ref.float(), rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("group", range(1, 9))
def test_single_tokens_with_every_head_size(ops, group):
    """Every head size that single tokens' kernel takes, whole sets of threads or not (5 heads of 96 numbers are 480 sums of 512, yet two
    sets of 96 threads with two rows each have four): bit-equal to the last token of a portion of two, and near float64."""
    lengths = (1, 64, 300)
    for hd in range(4, 129, 4):
        kc, vc, table, dense = _paged_setup(torch.float32, 1, hd, 16, list(lengths), sum(-(-n // 16) for n in lengths) + 2, seed=hd)
        q = torch.randn(len(lengths), 2, group * hd, generator=torch.Generator().manual_seed(13)).to(DEV)
        rows = q[:, -1].contiguous()
        out = torch.full_like(rows, float("nan"))
        ops.paged_attention(rows, kc, vc, Batch([(n - 1, 1) for n in lengths]), table, out, group, 1, hd, 0.2)
        for i, n in enumerate(lengths):
            if n > 1:
                portion = torch.empty(2, group * hd, device=DEV)
                ops.paged_attention(q[i].contiguous(), kc, vc, Batch([(n - 2, 2)]), table[i:i + 1].contiguous(), portion, group, 1, hd, 0.2)
                assert torch.equal(portion[-1], out[i]), (hd, n)
            K, V = dense[i]
            ref = _attention_ref(rows[i].view(group, hd).cpu().double(), K.double(), V.double(), n - 1, group, 1, hd, 0.2, 0)
            torch.testing.assert_close(out[i].cpu(), ref.float(), rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_four_tiles_of_few_rows_a_multiprocessor(ops, dt):
    """The steps of single tokens that walk their contexts, 512 CTAs say, are one round of four a multiprocessor, or two of three: what the
    compiler gives the kernel (64 registers a thread) decides, and that changes with what else is in its file."""
    from llmengine.ops import dtype_code
    assert ops.lib().llm_paged_attention_simt_resident(dtype_code(dt)) >= 4
