"""Steps of a served model, as they are timed and compared.

A case is one step of the engine: some requests bring their next token (decoding), and one request may bring a portion of its
prompt, on top of what it has in the cache. What a serving program has in hand before the step is the loaded model, the page pool,
and the requests with the pages of their earlier tokens filled and those of the step's tokens reserved; the step itself is
`Engine.step_and_sample` where every request brings one token, and `Engine.step` with the choice of tokens behind it otherwise
(what `step_and_sample` does for such a batch; this way its logits can be returned). A pass does not move the requests on, so it
can be repeated: it writes the same cache rows again. Every pass ends with the chosen tokens on the host, as a scheduler needs them.

Returned are the float32 logits of every request. The chosen tokens are left out: they are the logits' largest places, and with
random weights two logits are near enough to one another that a last bit decides between them.

Models are loaded once a process and shared by all states, as a server does; their weights come from a fixed seed, token ids from
the state's. Sizes are the layer sizes that the benchmark and the tests of this repository name; the 3B and 8B ones keep four of
their layers, so that a process is not busy loading them.
"""
import atexit
import hashlib
import json
import math
import os
import shutil
import sys
import tempfile

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-inference-engine-v6_b200"))

LLAMA3 = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
LLAMA_1B = {"architectures": ["LlamaForCausalLM"], "hidden_size": 2048, "intermediate_size": 8192, "num_hidden_layers": 16,
            "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64, "vocab_size": 128256, "max_position_embeddings": 16384,
            "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "tie_word_embeddings": True, "rope_scaling": LLAMA3}
_LATENT = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 192 ** -0.5,
           "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
_DENSE = {"kind": "dense", "ff": 8192}
_ROUTED = {"kind": "moe", "expert": {"ff": 2048}, "router": {"experts": 16, "top": 4}}
# name -> (config.json, tokens the page pool holds for one state)
MODELS = {
    "1b": (LLAMA_1B, 64 * 3616),
    "3b": (dict(LLAMA_1B, hidden_size=3072, num_attention_heads=24, head_dim=128, num_hidden_layers=4), 64 * 2064),
    "8b": (dict(LLAMA_1B, hidden_size=4096, intermediate_size=14336, head_dim=128, num_hidden_layers=4, tie_word_embeddings=False,
                rope_scaling=dict(LLAMA3, factor=8.0)), 16 * 2064),
    "tiny": ({"architectures": ["LlamaForCausalLM"], "hidden_size": 192, "intermediate_size": 512, "num_hidden_layers": 3,
              "num_attention_heads": 6, "num_key_value_heads": 1, "head_dim": 32, "vocab_size": 509, "max_position_embeddings": 256,
              "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "tie_word_embeddings": True,
              "rope_scaling": dict(LLAMA3, factor=8.0, original_max_position_embeddings=64)}, 8 * 256),
    "vapelix": ({"architecture": "Vapelix", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6}, "max_positions": 8192,
                 "layers": [{"type": "latent_attention", "mixer": _LATENT, "mlp": _DENSE if i == 0 else _ROUTED} for i in range(4)],
                 "token_side": {"dim": 128}}, 32 * 2064),
}
PAGE = 16
STATES = 4  # that share a model at a time
_folders, _engines = {}, {}


def _case(model, dtype, decode=0, low=0, high=0, portion=0, before=0, **name):
    """decode requests with contexts spread over low..high, and a portion of a prompt behind `before` of its tokens."""
    return dict(name, model=model, dtype=dtype, decode=decode, low=low, high=high, portion=portion, before=before)


def listed():
    return [
        # the smallest calls: a tiny model in the 32-bit path, four requests
        _case("tiny", "fp32", decode=4, low=1, high=150, name="tiny fp32 decode 4"),
        # one user's chat, a small batch and a full one
        _case("1b", "bf16", decode=1, low=2048, high=2048, name="1b decode 1"),
        _case("1b", "bf16", decode=8, low=2048, high=2048, name="1b decode 8"),
        _case("1b", "bf16", decode=64, low=500, high=3600, name="1b decode 64 ragged"),
        # a short question, and a document
        _case("1b", "bf16", portion=77, name="1b prompt 77"),
        _case("1b", "bf16", portion=2048, name="1b prompt 2048"),
        # the scheduler's default step under load: its budget of 256 prompt tokens beside the running requests
        _case("3b", "bf16", decode=31, low=100, high=2000, portion=225, before=451, name="3b mixed 31 + 225"),
        # the last portion of a long document
        _case("8b", "bf16", portion=2048, before=14336, name="8b portion 2048 at 14336"),
        # the 32-bit path: what outputs are checked against, and small models in earnest
        _case("1b", "fp32", decode=8, low=256, high=768, name="1b fp32 decode 8"),
        _case("1b", "fp32", portion=300, name="1b fp32 prompt 300"),
        # latent attention and routed experts
        _case("vapelix", "bf16", decode=8, low=2048, high=2048, name="vapelix decode 8"),
        _case("vapelix", "bf16", portion=2048, name="vapelix prompt 2048"),
    ]


def _between(rng, low, high):
    """A whole number, its logarithm spread evenly."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(("tiny", "decode", "decode", "prompt", "prompt", "mixed", "long", "fp32 decode", "fp32 prompt", "vapelix decode", "vapelix prompt"))
    model = rng.choice(("1b", "1b", "3b"))
    if kind == "tiny":
        high = _between(rng, 2, 200)
        return _case("tiny", "fp32", decode=rng.randint(1, 8), low=rng.randint(1, high), high=high)
    if kind == "decode":
        high = _between(rng, 64, 3600 if model == "1b" else 2000)
        return _case(model, "bf16", decode=_between(rng, 1, 64), low=rng.randint(16, high), high=high)
    if kind == "prompt":
        return _case(model, "bf16", portion=_between(rng, 5, 2048))
    if kind == "mixed":
        high = _between(rng, 64, 2000)
        return _case("3b", "bf16", decode=rng.randint(1, 48), low=rng.randint(16, high), high=high, portion=_between(rng, 16, 512), before=rng.randint(0, 1400))
    if kind == "long":
        portion = _between(rng, 200, 2048)
        return _case("8b", "bf16", portion=portion, before=rng.randint(1000, 16384 - portion - 1))
    if kind == "fp32 decode":
        high = _between(rng, 16, 768)
        return _case("1b", "fp32", decode=_between(rng, 1, 16), low=rng.randint(4, high), high=high)
    if kind == "fp32 prompt":
        return _case("1b", "fp32", portion=_between(rng, 5, 300))
    if kind == "vapelix decode":
        high = _between(rng, 64, 2048)
        return _case("vapelix", "bf16", decode=_between(rng, 1, 32), low=rng.randint(16, high), high=high)
    return _case("vapelix", "bf16", portion=_between(rng, 64, 2048))


def _requests(case):
    """[(tokens in the cache, tokens that the step brings)]: contexts spread over low..high by the golden ratio, the portion last."""
    spread = case["high"] - case["low"] + 1
    got = [(case["low"] + int(spread * (i * 0.6180339887498949 % 1.0)), 1) for i in range(case["decode"])]
    return got + ([(case["before"], case["portion"])] if case["portion"] else [])


def _vocabulary(model):
    return MODELS[model][0].get("vocab_size") or MODELS[model][0]["vocab"]


def _ids(case, seed):
    """The token ids of every request, those of the step last."""
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, _vocabulary(case["model"]), (have + new,), generator=g) for have, new in _requests(case)]


# ------------------------------------------------------------------------------------------------ weights
def _weight(model, name, shape, init):
    """One tensor of a model in bfloat16, a function of its name. Matrices N(0, 0.02), norms around one; Vapelix's embedding is
    wider, so that a layer adds to the stream about a tenth of it, as the layers of a trained model do."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{model}:{name}".encode()).digest()[:7], "little"))
    t = torch.randn(tuple(shape), generator=g, device="cuda", dtype=torch.float32)
    wide = model == "vapelix" and tuple(shape) == (_vocabulary(model), MODELS[model][0]["width"])
    t *= 2.0 if wide else 0.02
    if init == "around_one":
        t += 1.0
    elif init == "zeros":
        t.zero_()
    return t.to(torch.bfloat16)


def _folder(model):
    """A model folder as a user has it on disk: config.json and one safetensors file."""
    if model not in _folders:
        from llmengine.config.registry import architecture_name_of, get_architecture
        from llmengine.weights.random_init import model_tensor_needs
        config = MODELS[model][0]
        arch = get_architecture(architecture_name_of(config))
        needs = model_tensor_needs(arch.describe(arch.parse_config(config, None)))
        path = tempfile.mkdtemp(prefix="cases_")
        atexit.register(shutil.rmtree, path, ignore_errors=True)
        with open(os.path.join(path, "config.json"), "w") as f:
            json.dump(config, f)
        header, at = {}, 0
        for name in sorted(needs):
            size = 2 * math.prod(needs[name].shape)
            header[name] = {"dtype": "BF16", "shape": list(needs[name].shape), "data_offsets": [at, at + size]}
            at += size
        text = json.dumps(header).encode()
        text += b" " * (-len(text) % 8)
        with open(os.path.join(path, "model.safetensors"), "wb") as f:
            f.write(len(text).to_bytes(8, "little") + text)
            for name in sorted(needs):
                f.write(_weight(model, name, needs[name].shape, needs[name].init).reshape(-1).view(torch.uint8).cpu().numpy().data)
        _folders[model] = path
    return _folders[model]


def _engine(model, dtype):
    if (model, dtype) not in _engines:
        from llmengine import Engine
        room = STATES * (MODELS[model][1] if dtype == "bf16" else min(MODELS[model][1], 16 * 784))
        eng = Engine(_folder(model), dtype, block_size=PAGE, num_blocks=room // PAGE, max_concurrent=STATES * 65)
        eng.configure_cache()
        _engines[model, dtype] = eng
    return _engines[model, dtype]


# ------------------------------------------------------------------------------------------------ states and passes
class State:
    """Live requests of a loaded model, ready for their next step; they give back their pages with the state."""
    made = 0

    def __init__(self, engine, case, seed):
        from llmengine.cache import host_module
        self.engine, self.ids = engine, []
        self.entries = host_module().StepEntries()
        self.single = not case["portion"]
        room = 2048 if case["dtype"] == "bf16" else 768
        for ids, (have, new) in zip(_ids(case, seed), _requests(case)):
            State.made += 1
            rid, ids = State.made, ids.tolist()
            for at in range(0, have, room):  # the request's earlier tokens, in portions
                engine.run_step([(rid, ids[at:min(at + room, have)], [])])
            if not have:
                engine.cm.add_request(rid)
            self.ids.append(rid)
            if not engine.cm.reserve(rid, new):
                raise RuntimeError("the page pool is too small for this case")
            self.entries.add(rid, ids[have:], [new - 1])

    def __del__(self):
        for rid in self.ids:
            if self.engine.cm.has_request(rid):
                self.engine.cm.release(rid)


def prepare(case, seed):
    return State(_engine(case["model"], case["dtype"]), case, seed)


def run(state):
    eng = state.engine
    if state.single and eng.cuda_graphs:
        eng.step_and_sample(state.entries)
        return eng.graphs.last.logits[:len(state.entries)]
    ctx, logits = eng.step(state.entries)
    eng.sampler.sample(logits, ctx, ctx.n_rows)
    eng.raise_if_kernel_error()
    return logits


def work(case):
    """Every weight once (of the experts those that some token chooses), the cached rows of the requests once, the step's own rows
    and the logits written; operations of the products and of causal attention."""
    c, requests = MODELS[case["model"]][0], _requests(case)
    el = 2 if case["dtype"] == "bf16" else 4
    tokens, rows = sum(n for _, n in requests), len(requests)
    pairs = sum(n * have + n * (n + 1) // 2 for have, n in requests)  # (query, key)
    keys = sum(have + n for have, n in requests)
    if case["model"] == "vapelix":
        m, W, V, layers = _LATENT, c["width"], c["vocab"], 4
        H, R = m["heads"], m["kv_rank"]
        down, up = W * (R + m["rot_dim"] + m["q_rank"] + H * m["vdim"]), m["q_rank"] * H * (m["dim"] + m["rot_dim"])
        mixer = down + up + R * H * (m["dim"] + m["vdim"]) + H * m["vdim"] * W
        side = 2 * W * c["token_side"]["dim"]
        expert, E, top = 2 * W * _ROUTED["expert"]["ff"], 16, 4
        met = E * (1 - (1 - top / E) ** tokens)
        weights = layers * (mixer + side) + 3 * W * _DENSE["ff"] + 3 * (met * expert + E * W)
        used = layers * (mixer + side) + 3 * W * _DENSE["ff"] + 3 * (top * expert + E * W)
        row, per_pair = R + m["rot_dim"], 2 * H * (m["dim"] + m["rot_dim"] + m["vdim"])
    else:
        W, V, layers, FF = c["hidden_size"], c["vocab_size"], c["num_hidden_layers"], c["intermediate_size"]
        dq, dkv = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
        weights = used = layers * (W * (dq + 2 * dkv) + dq * W + 3 * W * FF)
        row, per_pair = 2 * dkv, 4 * dq
    return {"bytes": (weights + V * W + tokens * W) * el + keys * layers * row * el + rows * V * 4,
            "flops": 2 * tokens * used + 2 * rows * V * W + layers * pairs * per_pair}


def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _inv_freq(c):
    """The rotation frequencies are part of the model: theta^(-2i/d) in the Llama 3 bands, rounded to float32 (pi as a float32)."""
    s, d = c["rope_scaling"], c["head_dim"]
    pi = float(torch.tensor(math.pi, dtype=torch.float32))
    got = []
    for i in range(d // 2):
        f = c["rope_theta"] ** (-2.0 * i / d)
        length, old = 2.0 * pi / f, s["original_max_position_embeddings"]
        if length > old / s["low_freq_factor"]:
            f /= s["factor"]
        elif length >= old / s["high_freq_factor"]:
            part = (old / length - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])
            f = (1 - part) * f / s["factor"] + part * f
        got.append(f)
    return torch.tensor(got, dtype=torch.float32).double().cuda()


def exact(case, seed):
    """The decoder over whole sequences in float64. None for Vapelix: its routers choose experts, which a rounding of bfloat16
    changes where two are nearly tied, so a logit has no one value that every correct step comes near."""
    if case["model"] == "vapelix":
        return None
    model, c = case["model"], MODELS[case["model"]][0]
    W, FF, V, D = c["hidden_size"], c["intermediate_size"], c["vocab_size"], c["head_dim"]
    nq, nkv = c["num_attention_heads"], c["num_key_value_heads"]

    def weight(name, *shape):
        return _weight(model, name, shape, "around_one" if len(shape) == 1 else "normal").double()

    def norm(x, w):
        return x * w / torch.sqrt(x.square().mean(-1, keepdim=True) + c["rms_norm_eps"])

    table, freq = weight("model.embed_tokens.weight", V, W), _inv_freq(c)
    streams = [table[ids.cuda()] for ids in _ids(case, seed)]
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n1, n2 = weight(p + "input_layernorm.weight", W), weight(p + "post_attention_layernorm.weight", W)
        q, k = weight(p + "self_attn.q_proj.weight", nq * D, W), weight(p + "self_attn.k_proj.weight", nkv * D, W)
        v, o = weight(p + "self_attn.v_proj.weight", nkv * D, W), weight(p + "self_attn.o_proj.weight", W, nq * D)
        g, u = weight(p + "mlp.gate_proj.weight", FF, W), weight(p + "mlp.up_proj.weight", FF, W)
        d = weight(p + "mlp.down_proj.weight", W, FF)
        for h in streams:
            T = h.shape[0]
            x = norm(h, n1)
            angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * freq[None]
            cos, sin = torch.cat([angle.cos()] * 2, 1)[:, None], torch.cat([angle.sin()] * 2, 1)[:, None]

            def rotated(y):
                return y * cos + torch.cat([-y[..., D // 2:], y[..., :D // 2]], -1) * sin

            qs, ks, vs = rotated((x @ q.T).view(T, nq, D)), rotated((x @ k.T).view(T, nkv, D)), (x @ v.T).view(T, nkv, D)
            qs = qs.view(T, nkv, nq // nkv, D).permute(1, 2, 0, 3)  # [kv head, head of its group, token, D]
            ks, vs = ks.permute(1, 2, 0)[:, None], vs.permute(1, 0, 2)[:, None]
            out = torch.empty(T, nq * D, device="cuda", dtype=torch.float64)
            for at in range(0, T, 512):
                to = min(at + 512, T)
                score = qs[:, :, at:to] @ ks[..., :to] / math.sqrt(D)
                score.masked_fill_(torch.ones(to - at, to, device="cuda", dtype=torch.bool).triu(at + 1), -math.inf)
                out[at:to] = (torch.softmax(score, -1) @ vs[:, :, :to]).permute(2, 0, 1, 3).reshape(to - at, nq * D)
            h += out @ o.T
            for at in range(0, T, 4096):
                x = norm(h[at:at + 4096], n2)
                h[at:at + 4096] += (torch.nn.functional.silu(x @ g.T) * (x @ u.T)) @ d.T
    last = norm(torch.stack([h[-1] for h in streams]), weight("model.norm.weight", W))
    head = table if c["tie_word_embeddings"] else weight("lm_head.weight", V, W)
    return last @ head.T
