"""Steps of more than 64 single tokens: the q|k|v product is cut along K there, and its parts go to the attention kernel that adds,
rotates and stores them itself, as in smaller steps. Whole steps through the decode graphs (capacities 128 and 256, with padded rows)
and eagerly, with that kernel and with the separate ones, against the plain implementation."""
import numpy as np
import pytest
import torch

import llmengine
import plain_llama as P
from llmengine.cache import host_module
from tiny import TINY, make_model_dir, random_ids

pytestmark = pytest.mark.gpu
TOL = 6e-2  # as the other bfloat16 logits of these configurations


@pytest.mark.parametrize("live", [65, 100, 130])
def test_logits_of_many_single_tokens(tmp_path, monkeypatch, live):
    from llmengine.ops import get_ops
    ops = get_ops()
    cfg, page = TINY["d"]
    d = make_model_dir(str(tmp_path / "m"), cfg, torch.bfloat16)
    pc, pw = P.read_model(d)
    steps = 4
    seqs = [random_ids(1 + (37 * i) % 90 + steps, cfg["vocab_size"], 300 + i) for i in range(live)]
    lens = [len(s) - steps for s in seqs]
    plain = [P.forward_logits(pc, pw, s)[-steps:] for s in seqs]
    pages = sum(-(-len(s) // page) for s in seqs) + 4
    eng = llmengine.Engine(d, "bf16", block_size=page, num_blocks=pages, max_concurrent=live, cuda_graphs=True)
    fused = []
    kernel = ops.paged_attention_decode_fused
    monkeypatch.setattr(ops, "paged_attention_decode_fused", lambda parts, *a, **k: (fused.append(parts.shape), kernel(parts, *a, **k))[1])
    for at in range(0, live, 16):
        eng.run_step([(i, seqs[i][:lens[i]], []) for i in range(at, min(at + 16, live))])
    got = []
    for k in range(steps):
        monkeypatch.setattr(ops, "fused_decode_attention", k != 3)
        fused.clear()
        tokens = [seqs[i][lens[i] + k] for i in range(live)]
        if k < 2:
            e = host_module().StepEntries()
            for i in range(live):
                assert eng.cm.reserve(i, 1)
                e.add(i, [tokens[i]], [0])
            chosen = eng.step_and_sample(e)
            for i in range(live):
                eng.cm.advance(i, 1)
            assert eng.graphs.last.pad_to[1] == (128 if live <= 128 else 256)
            got.append(eng.graphs.last.logits[:live].float().cpu().numpy())
            assert chosen == got[-1].argmax(1).tolist()
        else:
            got.append(eng.run_step([(i, [tokens[i]], [0]) for i in range(live)]).float().cpu().numpy())
        n = eng.graphs.last.pad_to[1] if k < 2 else live
        if k in (0, 2):  # (the second step replays what the first recorded)
            assert fused and all(s[0] > 1 and s[1] == n for s in fused)
        elif k == 3:
            assert not fused
    for k in range(steps):
        off = np.abs(got[k] - np.stack([p[k] for p in plain])).max(1)
        assert off.max() < TOL, f"step {k}, request {off.argmax()} at position {lens[off.argmax()] + k}: {off.max():.3e}"
    eng.run_step([], end=list(range(live)))
    assert ops.tensor_core_error() == 0 and eng.cm.free_pages(0) == pages
