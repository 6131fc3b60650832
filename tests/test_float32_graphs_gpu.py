"""Decode steps of the 32-bit engine replay graphs: for every design, their logits against those of the same steps run eagerly."""
import numpy as np
import pytest
import torch

import llmengine
from llmengine.cache import host_module
from tiny import TINY, make_model_dir, random_ids
from tiny_kasarax import KASARAX
from tiny_selinex import SELINEX
from tiny_sogutar import SOGUTAR
from tiny_vapelix import VAPELIX
from tiny_zudatar import ZUDATAR
from tiny_zulopel import ZULOPEL

pytestmark = pytest.mark.gpu
DESIGNS = {"llama": TINY["e"], "llama odd sizes": TINY["c"], "vapelix": VAPELIX["va"], "vapelix 2": VAPELIX["vc"], "zulopel": ZULOPEL["zb"],
           "selinex": SELINEX["sb"], "sogutar": SOGUTAR["gb"], "zudatar": ZUDATAR["zb"], "kasarax": KASARAX["kb"]}


@pytest.mark.parametrize("name", DESIGNS)
def test_logits_of_recorded_and_eager_steps(tmp_path, name):
    """Rows of float32 products do not depend on the batch, but a recorded step's tables are padded, and kernels that cut a range into
    pieces may cut it elsewhere: sums in another order, some 1e-6 of the logits' size; a step that reads a stale or a neighbour's value is
    off by all of it."""
    cfg, page = DESIGNS[name]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    d = make_model_dir(str(tmp_path / "m"), cfg, torch.float32)
    steps, lens = 6, [3, 40, 17, 33, 1]
    seqs = [random_ids(n + steps, vocab, 70 + i) for i, n in enumerate(lens)]
    logits = {}
    for graphs in (False, None):  # None: the default
        eng = llmengine.Engine(d, "fp32", block_size=page, num_blocks=sum(-(-len(s) // page) for s in seqs) + 8, max_concurrent=8, cuda_graphs=graphs)
        eng.configure_cache()
        out = []
        for i, n in enumerate(lens):
            eng.run_step([(i, seqs[i][:n], [])])
        for k in range(steps):
            live = list(range(len(lens))) if k < 3 else [1, 3]  # capacities 8 and 2
            e = host_module().StepEntries()
            for i in live:
                assert eng.cm.reserve(i, 1)
                e.add(i, [seqs[i][lens[i] + k]], [0])
            if graphs is False:
                out.append(eng.step(e)[1].float().cpu().numpy().copy())
            else:
                assert eng.cuda_graphs == eng.model.capturable
                if not eng.cuda_graphs:
                    pytest.skip("a part of this design waits for the device: its steps are not recorded")
                eng.step_and_sample(e)
                out.append(eng.graphs.last.logits[:len(live)].float().cpu().numpy().copy())
            for i in live:
                eng.cm.advance(i, 1)
        logits[graphs] = out
    for k, (a, b) in enumerate(zip(logits[False], logits[None])):
        assert np.abs(a - b).max() <= 2e-5 * max(1.0, np.abs(a).max()), f"step {k}: {np.abs(a - b).max():.3e}"


@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
def test_no_room_for_a_graph(tmp_path, monkeypatch, dtype):
    """An engine whose pool leaves no memory for a graph's scratch goes on without graphs: the same tokens, the same step."""
    from llmengine.engine.graphs import DecodeGraphs
    cfg, page = TINY["d"]
    d = make_model_dir(str(tmp_path / "m"), cfg, torch.float32 if dtype == "fp32" else torch.bfloat16)
    prompt = random_ids(20, cfg["vocab_size"], 5)
    want = llmengine.Engine(d, dtype, block_size=page, num_blocks=16, max_concurrent=2, cuda_graphs=False).generate(prompt, 8)

    def full(*a):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(DecodeGraphs, "_capture", full)
    eng = llmengine.Engine(d, dtype, block_size=page, num_blocks=16, max_concurrent=2)
    with pytest.warns(UserWarning, match="without graphs"):
        assert eng.generate(prompt, 8) == want
    assert not eng.cuda_graphs and eng.graphs is None and eng.cm.free_pages(0) == 16
