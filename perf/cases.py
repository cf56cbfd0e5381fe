"""The work this framework is measured on: what its users' programs have it do, with the inputs, the call and the exact answer.

A program holds a model and a step runner (`api.make_runner`) or an `Engine`, feeds prompts and draws tokens.  The kinds of
work are the ones such programs consist of:

  decode   requests that already hold a context get `new` tokens each, one step per token, every token drawn on the device
           and fed back there (the contexts grow from pass to pass, as they do in use)
  prompt   prompts are fed in one step and the logits of every prompt's last token come back (scoring, time to first token)
  mixed    one step of decoding requests beside a portion of somebody else's prompt (a server under a token budget)
  turn     requests from admission to release: their prompts in one step, then `new` - 1 decode steps
  serve    the same through `Engine.generate`, under its scheduler and the default sampling rules, and one step that scores
           the longest reply

Sizes are those of this repository's benchmark (Gemma 2 2B and 9B, the eight-layer Bolonex and Petanex of width 2048) and the
tests' small Gemma 2.  Weights are random with the spreads of trained models where the work depends on it: branches that
change the residual stream by a part of its size, tokens with a likely successor (so that a drawn token is the same for every
correct implementation), experts that serve kinds of tokens.  `exact` states the models in plain float64 torch.
"""
from __future__ import annotations

import math

import torch

VOCAB, SMALL_VOCAB = 256000, 32000
GROWTH = 2048            # tokens a decoding request may grow by before its context is fed anew
WARM = 3                 # decode steps before the first pass (a program's steps are captured as graphs by then)
F64 = torch.float64

GEMMA = {
    # the tests' smallest configuration at which the tensor-core kernels run, and the layer sizes of Gemma 2 2B and 9B
    "gemma2-tiny": dict(num_hidden_layers=2, hidden_size=512, num_attention_heads=6, num_key_value_heads=2, head_dim=128,
                        intermediate_size=1536, query_pre_attn_scalar=144, vocab_size=3000, sliding_window=100),
    "gemma2-2b": dict(num_hidden_layers=26, hidden_size=2304, num_attention_heads=8, num_key_value_heads=4, head_dim=256,
                      intermediate_size=9216, query_pre_attn_scalar=256, vocab_size=VOCAB, sliding_window=4096),
    "gemma2-9b": dict(num_hidden_layers=42, hidden_size=3584, num_attention_heads=16, num_key_value_heads=8, head_dim=256,
                      intermediate_size=14336, query_pre_attn_scalar=256, vocab_size=VOCAB, sliding_window=4096),
}
WIDTH, LAYERS = 2048, 8                                     # Bolonex and Petanex
EXPERTS, TOP, CLUSTERS = 32, 3, 16


# ---- cases -----------------------------------------------------------------------------------------------------------

def listed():
    def case(name, work, model, requests, tokens, *, ragged=False, new=1, dtype="bfloat16"):
        return {"name": name, "work": work, "model": model, "dtype": dtype, "requests": requests, "tokens": tokens,
                "ragged": ragged, "new": new}
    return [
        # one user's chat deep in its context: the step is bound by the weights and by launches
        case("decode-1", "decode", "gemma2-2b", 1, 8192, new=8),
        # the benchmark's headline: a small batch at a long context, half of the layers windowed
        case("decode-8", "decode", "gemma2-2b", 8, 8192, new=8),
        # a busy server: many conversations of all lengths
        case("decode-64-ragged", "decode", "gemma2-2b", 64, 1024, ragged=True, new=8),
        # a document read before the first token
        case("prompt-2048", "prompt", "gemma2-2b", 1, 2048),
        # several users' prompts of odd lengths in one step of a larger model
        case("prompts-9b-ragged", "prompt", "gemma2-9b", 5, 701, ragged=True),
        # the step of a server under a budget of 512 rows: eight conversations go on while a prompt is read
        case("mixed-512", "mixed", "gemma2-2b", 8, 2048, new=504),
        # the 32-bit path, as a program that checks numbers uses it: short prompts, few tokens
        case("turn-fp32", "turn", "gemma2-2b", 2, 97, ragged=True, new=3, dtype="float32"),
        # a handful of users through the engine: scheduling, mixed steps, sampling, tokens to the host
        case("serve-6", "serve", "gemma2-2b", 6, 600, ragged=True, new=24),
        # the smallest model and request: nothing but latency
        case("turn-tiny", "turn", "gemma2-tiny", 1, 11, new=12),
        # a state-space model reads a document ...
        case("prompt-bolonex", "prompt", "bolonex", 1, 2048),
        # ... and writes for eight users
        case("decode-bolonex", "decode", "bolonex", 8, 4096, new=8),
        # latent attention, delta rules and experts: short prompts and their replies
        case("turn-petanex", "turn", "petanex", 8, 300, ragged=True, new=16),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    work = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "turn", "serve"])
    model = rng.choice(["gemma2-2b", "gemma2-2b", "gemma2-9b", "bolonex", "petanex"])
    dtype, ragged = "bfloat16", rng.random() < 0.6
    if work in ("turn", "serve") and rng.random() < 0.4:
        model = "gemma2-tiny"
    if model == "gemma2-tiny" and work == "turn" and rng.random() < 0.3:
        dtype = "float32"
    elif model == "gemma2-2b" and work == "turn":
        dtype = "float32"
    if work == "mixed" and model == "gemma2-9b":
        model = "gemma2-2b"
    most = {"gemma2-tiny": 2000, "gemma2-2b": 65536, "gemma2-9b": 8192, "bolonex": 32768, "petanex": 16384}[model]
    new = 1
    if dtype == "float32" and model == "gemma2-2b":
        requests, tokens, new = rng.randint(1, 4), _log_uniform(rng, 3, 48), rng.randint(1, 3)
    elif work == "decode":
        requests = _log_uniform(rng, 1, 64)
        tokens, new = _log_uniform(rng, 64, min(8192, most // requests)), 8
    elif work == "mixed":
        requests = _log_uniform(rng, 1, 32)
        tokens, new = _log_uniform(rng, 64, 2048), _log_uniform(rng, 32, 1024)
    elif work == "prompt":
        requests = _log_uniform(rng, 1, 8)
        tokens = _log_uniform(rng, 16, 2048 // requests)
    else:
        requests = _log_uniform(rng, 1, 8)
        tokens, new = _log_uniform(rng, 3, min(600, 2048 // requests)), rng.randint(4, 24)
    return {"work": work, "model": model, "dtype": dtype, "requests": requests, "tokens": tokens, "ragged": ragged, "new": new}


def _lengths(case):
    """Prompt length of every request: `tokens`, or spread between a tenth of it and all of it."""
    n, k = case["tokens"], case["requests"]
    if not case["ragged"]:
        return [n] * k
    return [n] + [max(2, int(n * (0.1 + 0.9 * ((i * 0.6180339887) % 1.0)))) for i in range(1, k)]


# ---- configurations ----------------------------------------------------------------------------------------------------

def config(model: str) -> dict:
    """The config.json dictionary of a model."""
    d = 128
    if model in GEMMA:
        return dict(GEMMA[model], architectures=["Gemma2ForCausalLM"], rope_theta=10000.0, attn_logit_softcapping=50.0,
                    final_logit_softcapping=30.0, rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=16384,
                    hidden_activation="gelu_pytorch_tanh")
    if model == "bolonex":
        att = {"heads": 16, "kv_heads": 4, "dim": d, "vdim": d, "conv": 4, "scale": d ** -0.5, "softcap": 30.0,
               "rot": {"base": 500000.0, "dims": d, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        ssm = {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}
        layers = [{"type": "attention" if i % 4 == 0 else "mamba2", "mixer": att if i % 4 == 0 else ssm,
                   "mlp": {"kind": "dense", "ff": 8192}} for i in range(LAYERS)]
        return {"architecture": "Bolonex", "width": WIDTH, "vocab": SMALL_VOCAB, "embedding": {"scale": 50.0}, "norm": {"eps": 1e-5},
                "layers": layers}
    lat = {"heads": 16, "dim": d, "vdim": d, "kv_rank": 256, "scale": d ** -0.5}
    dl = {"heads": 16, "kv_heads": 8, "dim": d, "vdim": d, "conv": 4}
    moe = {"kind": "moe", "expert": {"ff": 2048, "limit": 7.0}, "shared": {"ff": 2048, "limit": 7.0},
           "router": {"experts": EXPERTS, "top": TOP, "scale": 2.5, "groups": {"count": 4, "keep": 2}}}
    kinds, mixers = ["latent_attention", "channel_delta", "delta", "delta"], [lat, dict(dl, decay_rank=64, gate_rank=64), dl, dl]
    layers = [{"type": kinds[i % 4], "mixer": mixers[i % 4], "mlp": {"kind": "dense", "ff": 8192} if i % 2 == 0 else moe}
              for i in range(LAYERS)]
    return {"architecture": "Petanex", "width": WIDTH, "vocab": SMALL_VOCAB, "embedding": {"scale": 50.0}, "norm": {"eps": 1e-5},
            "token_side": {"dim": 64}, "layers": layers}


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _successor(model, ids, n=1):
    """The token that `n` greedy draws lead to: tied output matrices repeat a token, Bolonex counts up."""
    return (ids + n) % SMALL_VOCAB if model == "bolonex" else ids


# ---- weights -----------------------------------------------------------------------------------------------------------

def _shapes(cfg):
    """(name, shape, mean, spread) of every drawn tensor."""
    out = []
    if "hidden_size" in cfg:
        H, I, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
        q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
        out.append(("model.embed_tokens.weight", (cfg["vocab_size"], H), 0.0, H ** -0.5))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out += [(p + "input_layernorm.weight", (H,), 0.0, 0.1), (p + "self_attn.q_proj.weight", (q, H), 0.0, 0.02),
                    (p + "self_attn.k_proj.weight", (kv, H), 0.0, 0.02), (p + "self_attn.v_proj.weight", (kv, H), 0.0, 0.02),
                    (p + "self_attn.o_proj.weight", (H, q), 0.0, 0.02), (p + "post_attention_layernorm.weight", (H,), -0.65, 0.035),
                    (p + "pre_feedforward_layernorm.weight", (H,), 0.0, 0.1), (p + "mlp.gate_proj.weight", (I, H), 0.0, 0.02),
                    (p + "mlp.up_proj.weight", (I, H), 0.0, 0.02), (p + "mlp.down_proj.weight", (H, I), 0.0, 0.02),
                    (p + "post_feedforward_layernorm.weight", (H,), -0.65, 0.035)]
        out.append(("model.norm.weight", (H,), 0.0, 0.1))
        return out
    W, V = cfg["width"], cfg["vocab"]
    out.append(("embed", (V, W), 0.0, 0.02))
    if cfg["architecture"] == "Bolonex":
        for i, l in enumerate(cfg["layers"]):
            p, m = f"l{i}.", l["mixer"]
            out.append((p + "norm1", (W,), 0.0, 0.1))
            if l["type"] == "attention":
                rows = {"q": m["heads"] * m["dim"], "k": m["kv_heads"] * m["dim"], "v": m["kv_heads"] * m["vdim"]}
                for n, r in rows.items():
                    out += [(f"{p}mix.{n}", (r, W), 0.0, 0.02), (f"{p}mix.{n}.b", (r,), 0.0, 0.1), (f"{p}mix.{n}.conv", (r, m["conv"]), 0.0, 0.5)]
                out += [(p + "mix.q.norm", (m["dim"],), 1.5, 0.2), (p + "mix.k.norm", (m["dim"],), 1.5, 0.2),
                        (p + "mix.g", (m["heads"], W), 0.0, 0.02), (p + "mix.o", (W, m["heads"] * m["vdim"]), 0.0, 0.006)]
            else:
                inner, gn = m["heads"] * m["vdim"], m["groups"] * m["state"]
                out += [(p + "mix.in", (2 * inner + 2 * gn + m["heads"], W), 0.0, 0.02), (p + "mix.conv", (inner + 2 * gn, m["conv"]), 0.0, 0.5),
                        (p + "mix.conv.b", (inner + 2 * gn,), 0.0, 0.1), (p + "mix.dt_bias", (m["heads"],), -3.0, 1.0),
                        (p + "mix.A_log", (m["heads"],), 1.0, 0.8), (p + "mix.D", (m["heads"],), 1.0, 0.2), (p + "mix.norm", (inner,), 1.0, 0.1),
                        (p + "mix.o", (W, inner), 0.0, 0.004)]
            out += [(p + "mlp.up", (l["mlp"]["ff"], W), 0.0, 0.02), (p + "mlp.down", (W, l["mlp"]["ff"]), 0.0, 0.005)]
        out.append(("final.norm", (W,), 0.0, 0.1))
        return out
    side = cfg["token_side"]["dim"]
    out.append(("side.embed", (V, len(cfg["layers"]) * side), 0.0, 1.0))
    for i, l in enumerate(cfg["layers"]):
        p, m = f"l{i}.", l["mixer"]
        out += [(p + "norm1", (W,), 1.0, 0.1), (p + "ls1", (W,), 0.25, 0.05), (p + "norm2", (W,), 1.0, 0.1)]
        if l["type"] == "latent_attention":
            out += [(p + "mix.q", (m["heads"] * m["dim"], W), 0.0, 0.03), (p + "mix.dkv", (m["kv_rank"], W), 0.0, 0.02),
                    (p + "mix.dkv.norm", (m["kv_rank"],), 1.0, 0.1), (p + "mix.uk", (m["heads"] * m["dim"], m["kv_rank"]), 0.0, 0.06),
                    (p + "mix.uv", (m["heads"] * m["vdim"], m["kv_rank"]), 0.0, 0.06), (p + "mix.o", (W, m["heads"] * m["vdim"]), 0.0, 0.02)]
        else:
            h, kh, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, r in (("q", kh * d), ("k", kh * d), ("v", h * dv)):
                out += [(f"{p}mix.{n}", (r, W), 0.0, 0.02), (f"{p}mix.{n}.conv", (r, m["conv"]), 0.0, 0.5)]
            out += [(p + "mix.b", (h, W), 0.0, 0.02), (p + "mix.A_log", (h,), -2.0, 0.8), (p + "mix.norm", (dv,), 1.0, 0.1),
                    (p + "mix.o", (W, h * dv), 0.0, 0.02)]
            if l["type"] == "channel_delta":
                out += [(p + "mix.a1", (m["decay_rank"], W), 0.0, 0.02), (p + "mix.a2", (h * d, m["decay_rank"]), 0.0, 0.1),
                        (p + "mix.dt_bias", (h * d,), -1.0, 0.5), (p + "mix.g1", (m["gate_rank"], W), 0.0, 0.02),
                        (p + "mix.g2", (h * dv, m["gate_rank"]), 0.0, 0.1)]
            else:
                out += [(p + "mix.a", (h, W), 0.0, 0.02), (p + "mix.dt_bias", (h,), -1.0, 0.5), (p + "mix.g", (h * dv, W), 0.0, 0.02)]
        f = l["mlp"]
        if f["kind"] == "dense":
            out += [(p + "ls2", (W,), 0.25, 0.05)]
            out += [(p + "mlp.gate", (f["ff"], W), 0.0, 0.02), (p + "mlp.up", (f["ff"], W), 0.0, 0.02), (p + "mlp.down", (W, f["ff"]), 0.0, 0.02)]
        else:
            out += [(p + "ls2", (W,), 0.1, 0.02), (p + "mlp.correction", (EXPERTS,), 0.0, 0.02)]
            for e in [f"e{j}." for j in range(EXPERTS)] + ["shared."]:
                ff = f["expert"]["ff"]
                out += [(f"{p}mlp.{e}gate", (ff, W), 0.0, 0.02), (f"{p}mlp.{e}up", (ff, W), 0.0, 0.02), (f"{p}mlp.{e}down", (W, ff), 0.0, 0.02)]
        out += [(p + "side.gate", (side, W), 0.0, 0.02), (p + "side.proj", (W, side), 0.0, 0.1), (p + "side.norm", (W,), 0.15, 0.03)]
    out.append(("final.norm", (W,), 1.0, 0.1))
    return out


def _weights(cfg, dtype, seed):
    """Tensors by file name, on the GPU, from torch's generator."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = {}
    for name, shape, mean, std in _shapes(cfg):
        x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).mul_(std)
        t[name] = (x.add_(mean) if mean else x).to(dtype)
    if cfg.get("architecture") == "Bolonex":
        t["head"] = torch.roll(t["embed"], 1, 0).contiguous()
        for i in range(LAYERS):
            # rates between 1 and 16, as state-space models start from
            if cfg["layers"][i]["type"] == "mamba2":
                t[f"l{i}.mix.A_log"] = t[f"l{i}.mix.A_log"].clamp(0.0, 2.8)
    if cfg.get("architecture") == "Petanex":
        # tokens come in kinds, and every mixture has three experts for a kind, two of one group and one of another
        kinds = torch.randn((CLUSTERS, WIDTH), generator=g, device="cuda") * 0.02
        of = torch.randint(0, CLUSTERS, (SMALL_VOCAB,), generator=g, device="cuda")
        t["embed"] = (t["embed"].float() + kinds[of]).to(dtype)
        per = EXPERTS // 4
        for i in range(1, LAYERS, 2):
            score = torch.full((EXPERTS, CLUSTERS), -3.0, device="cuda")
            for c in range(CLUSTERS):
                two, one = (c + i) % 4, (c + 3 * i + 1 + c // 4 % 3) % 4
                one = (one + 1) % 4 if one == two else one
                score[[two * per + c % per, two * per + (c + 3) % per, one * per + (c // 2 + i) % per], c] = 3.0
            t[f"l{i}.mlp.router"] = (score @ kinds / (0.02 * WIDTH * 0.02) * 0.02 * 1.5).to(dtype)
    return t


def _prompts(case, cfg, seed):
    g = torch.Generator().manual_seed(seed + 77)
    return [torch.randint(0, _vocab(cfg), (n,), generator=g).tolist() for n in _lengths(case)]


def _portion(case, cfg, seed):
    g = torch.Generator().manual_seed(seed + 78)
    return torch.randint(0, _vocab(cfg), (case["new"],), generator=g).tolist()


# ---- what a program holds, and its passes ------------------------------------------------------------------------------

class _State:
    pass


def prepare(case, seed):
    from kungfu_b200 import api, registry
    from kungfu_b200.engine import StepEntry
    from kungfu_b200.engine.engine import Engine
    from kungfu_b200.sampling import STATE_WORDS, Sampling, pack_state
    from kungfu_b200.weights.store import WeightStore
    s = _State()
    s.case, s.entry = dict(case), StepEntry
    raw = config(case["model"])
    s.dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    device = api.require_cuda("cuda:0")
    cfg = api.load_config(raw)
    store = WeightStore.from_tensors(_weights(raw, s.dtype, seed), device=device, compute_dtype=s.dtype)
    model = registry.find(cfg.architecture).build(cfg, store)
    del store
    s.vocab = _vocab(raw)
    s.prompts = _prompts(case, raw, seed)
    B, longest = case["requests"], max(_lengths(case))
    grows = case["work"] in ("decode", "mixed")
    ctx = longest + (GROWTH if grows else case["new"] + 8) + (case["new"] if case["work"] == "mixed" else 0)
    s.runner = api.make_runner(cfg, model, dtype=s.dtype, device=device, max_requests=B + 1, max_context=ctx, batch=2048)
    s.limit = longest + GROWTH - 8
    s.states = torch.zeros((s.runner.cache.max_requests, STATE_WORDS), dtype=torch.int32, device=device)
    s.states[:] = torch.from_numpy(pack_state(Sampling(temperature=0.0), 1)).to(device)
    s.ids = torch.zeros((case["new"], B), dtype=torch.int32, device=device)
    s.rids, s.places = [f"r{i}" for i in range(B)], None
    if case["work"] in ("decode", "mixed"):
        if case["work"] == "mixed":
            s.portion = _portion(case, raw, seed)
        _fill(s)
    elif case["work"] == "serve":
        s.engine = Engine(runner=s.runner, batch=512, parallel=B)
        s.sampling = Sampling()
    if case["work"] in ("prompt", "turn", "serve", "mixed"):
        n, s.case["new"] = s.case["new"], min(s.case["new"], 4) if case["work"] in ("turn", "serve") else s.case["new"]
        for _ in range(2):
            run(s)
        s.case["new"] = n
        if case["work"] == "mixed":
            _fill(s)
    torch.cuda.synchronize()
    return s


def _fill(s):
    """The requests' contexts, fed as prompts, and the first decode steps."""
    cache, runner = s.runner.cache, s.runner
    for r, toks in zip(s.rids, s.prompts):
        if r in cache:
            cache.release(r)
        cache.add_request(r)
        for a in range(0, len(toks) - 1, 2048):
            runner.step([s.entry(r, toks[a:min(a + 2048, len(toks) - 1)])])
    s.last = None
    for _ in range(WARM):
        _decode_step(s)


def _decode_step(s):
    """One token for every request: the prompts' last tokens first, then what the step before drew."""
    entries = [s.entry(r, [p[-1]], [0]) for r, p in zip(s.rids, s.prompts)]
    logits, s.last = s.runner.step(entries, sample=(s.states, False), feedback=s.last)
    return logits


def _wanted(s, logits, picked):
    """The rows of a step's results in the order of its wanted places (steps with prompts may hold padding rows)."""
    at = tuple(s.runner.last_logit_index)
    if at == tuple(range(logits.shape[0])):
        return logits, picked
    if s.places is None or s.places[0] != at:
        s.places = (at, torch.tensor(at, device=logits.device))
    return logits[s.places[1]], picked[s.places[1]]


def run(s):
    case, cache, runner = s.case, s.runner.cache, s.runner
    work, new = case["work"], case["new"]
    if work == "decode":
        if cache.length(s.rids[0]) + new > s.limit:
            _fill(s)
        for i in range(new):
            logits = _decode_step(s)
            s.ids[i].copy_(s.last)
        return {"logits": logits, "ids": s.ids}
    if work == "prompt":
        for r in s.rids:
            cache.add_request(r)
        logits = runner.step([s.entry(r, p, [len(p) - 1]) for r, p in zip(s.rids, s.prompts)])
        for r in s.rids:
            cache.release(r)
        return {"logits": logits}
    if work == "mixed":
        if cache.length(s.rids[0]) + 1 > s.limit:
            _fill(s)
        cache.add_request("portion")
        entries = [s.entry(r, [_successor(case["model"], p[-1], cache.length(r) - len(p) + 1)], [0]) for r, p in zip(s.rids, s.prompts)]
        entries.append(s.entry("portion", s.portion, [len(s.portion) - 1]))
        logits, picked = _wanted(s, *runner.step(entries, sample=(s.states, False)))
        cache.release("portion")
        return {"logits": logits, "ids": picked}
    if work == "turn":
        for r in s.rids:
            cache.add_request(r)
        entries = [s.entry(r, p, [len(p) - 1]) for r, p in zip(s.rids, s.prompts)]
        logits, picked = _wanted(s, *runner.step(entries, sample=(s.states, False)))
        s.ids[0].copy_(picked)
        for i in range(1, new):
            logits, picked = runner.step([s.entry(r, [0], [0]) for r in s.rids], sample=(s.states, False), feedback=picked)
            s.ids[i].copy_(picked)
        for r in s.rids:
            cache.release(r)
        return {"logits": logits, "ids": s.ids[:new]}
    replies = s.engine.generate(s.prompts, s.sampling, max_tokens=new, ignore_eos=True)
    whole = s.prompts[0] + replies[0]
    cache.add_request("score")
    logits = runner.step([s.entry("score", whole, list(range(len(whole) - new, len(whole))))])
    cache.release("score")
    return {"logits": logits, "ids": torch.tensor(replies)}


# ---- what a pass cannot do without --------------------------------------------------------------------------------------

def _sizes(cfg):
    """Elements of the matrices that every token meets (routed experts and tables not counted), and of the output matrix."""
    every, V = 0, _vocab(cfg)
    for name, shape, _m, _s in _shapes(cfg):
        if len(shape) == 2 and "embed" not in name and ".mlp.e" not in name:
            every += shape[0] * shape[1]
    W = cfg.get("hidden_size") or cfg["width"]
    if cfg.get("architecture") == "Petanex":
        every += sum(1 for i in range(LAYERS) if i % 2) * EXPERTS * W
    return every, V * W


def _seen(cfg, layer, length):
    w = cfg.get("sliding_window")
    return min(length, w) if w and layer % 2 == 0 else length


def _kv(cfg):
    """Per attention layer: (index, key/value elements per token, score and value multiply-adds per query and key)."""
    if "hidden_size" in cfg:
        d = cfg["head_dim"]
        return [(i, 2 * cfg["num_key_value_heads"] * d, 2 * cfg["num_attention_heads"] * d) for i in range(cfg["num_hidden_layers"])]
    out = []
    for i, l in enumerate(cfg["layers"]):
        m = l["mixer"]
        if l["type"] == "attention":
            out.append((i, m["kv_heads"] * (m["dim"] + m["vdim"]), m["heads"] * (m["dim"] + m["vdim"])))
        elif l["type"] == "latent_attention":
            out.append((i, m["kv_rank"], m["heads"] * (m["dim"] + m["vdim"])))
    return out


def _state_elements(cfg):
    n = 0
    for l in cfg.get("layers", []):
        m = l["mixer"]
        n += m["heads"] * m["vdim"] * m["state"] if l["type"] == "mamba2" else m["heads"] * m["dim"] * m["vdim"] if "delta" in l["type"] else 0
    return n


def work(case):
    cfg = config(case["model"])
    el = 2 if case["dtype"] == "bfloat16" else 4
    every, head = _sizes(cfg)
    V = _vocab(cfg)
    total = {"bytes": 0.0, "flops": 0.0}

    def step(starts, counts, wanted):
        """One step: request i brings counts[i] tokens after starts[i]."""
        rows = sum(counts)
        moe = sum(1 for l in cfg.get("layers", []) if l["mlp"]["kind"] == "moe")
        one = 3 * 2048 * WIDTH
        used = min(EXPERTS, rows * TOP)
        total["bytes"] += el * (every + (head if wanted else 0) + moe * used * one) + 4 * wanted * V
        total["flops"] += 2.0 * rows * (every + moe * TOP * one) + 2.0 * wanted * head
        for i, elements, madds in _kv(cfg):
            for a, n in zip(starts, counts):
                total["bytes"] += el * elements * (min(_seen(cfg, i, a + n) + n - 1, a + n) if n > 1 else _seen(cfg, i, a + 1))
                total["flops"] += 2.0 * madds * sum(_seen(cfg, i, a + j + 1) for j in range(n))
        state = _state_elements(cfg)
        total["bytes"] += 8.0 * state * len(counts)
        total["flops"] += 4.0 * state * rows

    lens, new, B = _lengths(case), case["new"], case["requests"]
    if case["work"] == "decode":
        for k in range(new):
            step([n - 1 + WARM + k for n in lens], [1] * B, B)
    elif case["work"] == "mixed":
        step([n - 1 + WARM for n in lens] + [0], [1] * B + [new], B + 1)
    else:
        step([0] * B, lens, B)
        for k in range(1, new):
            step([n + k - 1 for n in lens], [1] * B, B)
        if case["work"] == "serve":
            step([0], [lens[0] + new], new)
    return total


def tolerance(case):
    """About four times the distance from `exact` that was measured: 3e-6 in 32 bits; in bfloat16 5e-3 for Gemma 2 (26 to 42
    layers), 3e-3 for Bolonex and 5e-4 for Petanex (eight layers; most of a Petanex logit is the token's kind)."""
    if case["dtype"] == "float32":
        return {"rel": 1.4e-5, "max": 2e-4}
    rel = {"bolonex": 0.012, "petanex": 0.002}.get(case["model"], 0.02)
    return {"rel": rel, "max": 8 * rel}


# ---- the models in plain float64 ------------------------------------------------------------------------------------------

def _lin(x, w):
    return x @ w.to(F64).T


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _attend(q, k, v, scale, cap=0.0, window=None, first=0):
    """Causal attention of queries [B, T, H, d] at positions first.. over keys [B, S, G, d] and values [B, S, G, dv]."""
    B, T, H, _ = q.shape
    S, G = k.shape[1], k.shape[2]
    out = torch.empty((B, T, H, v.shape[-1]), dtype=F64, device=q.device)
    step = max(1, int(3e8 // (S * H)))
    for b in range(B):
        kb, vb = k[b].permute(1, 2, 0), v[b].permute(1, 0, 2)
        for a in range(0, T, step):
            z = min(a + step, T)
            lo = 0 if window is None else max(0, first + a - window + 1)
            hi = min(S, first + z)
            qb = q[b, a:z].permute(1, 0, 2).reshape(G, (H // G) * (z - a), -1)
            sc = (qb @ kb[:, :, lo:hi]).view(H, z - a, hi - lo) * scale
            if cap:
                sc = cap * torch.tanh(sc / cap)
            at = first + torch.arange(a, z, device=q.device)[:, None]
            j = torch.arange(lo, hi, device=q.device)[None, :]
            see = j <= at if window is None else (j <= at) & (at - j < window)
            w = torch.softmax(sc.masked_fill(~see, -math.inf), -1).view(G, (H // G) * (z - a), hi - lo)
            out[b, a:z] = (w @ vb[:, lo:hi]).view(H, z - a, -1).permute(1, 0, 2)
    return out


def _gemma(cfg, t, x, ids):
    B, T = ids.shape
    H, d, eps = cfg["hidden_size"], cfg["head_dim"], cfg["rms_norm_eps"]
    nh, nk = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    f = (cfg["rope_theta"] ** (-2.0 * torch.arange(d // 2, dtype=F64, device=ids.device) / d)).float().to(F64)
    ang = torch.arange(T, dtype=F64, device=ids.device)[:, None] * f
    cos, sin = torch.cos(ang)[None, :, None], torch.sin(ang)[None, :, None]

    def turn(u):
        a, b = u[..., :d // 2], u[..., d // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    def norm(u, name):
        return _rms(u, eps) * (1.0 + t[name].to(F64))

    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = norm(x, p + "input_layernorm.weight")
        q, k, v = (_lin(n, t[p + f"self_attn.{c}_proj.weight"]).view(B, T, -1, d) for c in "qkv")
        a = _attend(turn(q), turn(k), v, cfg["query_pre_attn_scalar"] ** -0.5, cfg["attn_logit_softcapping"],
                    cfg["sliding_window"] if i % 2 == 0 else None)
        x = x + norm(_lin(a.reshape(B, T, nh * d), t[p + "self_attn.o_proj.weight"]), p + "post_attention_layernorm.weight")
        n = norm(x, p + "pre_feedforward_layernorm.weight")
        n = _gelu(_lin(n, t[p + "mlp.gate_proj.weight"])) * _lin(n, t[p + "mlp.up_proj.weight"])
        x = x + norm(_lin(n, t[p + "mlp.down_proj.weight"]), p + "post_feedforward_layernorm.weight")
    return norm(x, "model.norm.weight")


def _conv(u, w, bias=None):
    """Causal convolution per channel of u [B, T, C]; the last tap meets the current token."""
    taps, T = w.shape[1], u.shape[1]
    padded = torch.nn.functional.pad(u, (0, 0, taps - 1, 0))
    y = sum(padded[:, j:j + T] * w[:, j].to(F64) for j in range(taps))
    return y if bias is None else y + bias.to(F64)


def _bolonex(cfg, t, x, ids):
    B, T = ids.shape
    eps = cfg["norm"]["eps"]
    dev = ids.device
    for i, l in enumerate(cfg["layers"]):
        p, m = f"l{i}.", l["mixer"]
        h = _rms(x, eps) * (1.0 + t[p + "norm1"].to(F64))
        if l["type"] == "attention":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            q, k, v = (_conv(_lin(h, t[f"{p}mix.{n}"]) + t[f"{p}mix.{n}.b"].to(F64), t[f"{p}mix.{n}.conv"]) for n in "qkv")
            q = _rms(q.view(B, T, H, d), eps) * t[p + "mix.q.norm"].to(F64)
            k = _rms(k.view(B, T, G, d), eps) * t[p + "mix.k.norm"].to(F64)
            sc = m["rot"]["scaling"]
            freq = []
            for j in range(d // 2):
                f = m["rot"]["base"] ** (-2.0 * j / d)
                length = 2.0 * math.pi / f
                if length > sc["original"] / sc["low"]:
                    f = f / sc["factor"]
                elif length >= sc["original"] / sc["high"]:
                    share = (sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])
                    f = (1.0 - share) * f / sc["factor"] + share * f
                freq.append(f)
            ang = torch.arange(T, dtype=F64, device=dev)[:, None] * torch.tensor(freq, dtype=F64, device=dev)
            cos, sin = torch.cos(ang)[None, :, None], torch.sin(ang)[None, :, None]

            def turn(u):
                a, b = u[..., 0::2], u[..., 1::2]
                return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)

            o = _attend(turn(q), turn(k), v.view(B, T, G, -1), m["scale"], m["softcap"])
            o = (o * torch.sigmoid(_lin(h, t[p + "mix.g"]))[..., None]).reshape(B, T, -1)
        else:
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * P
            z, u, dt = _lin(h, t[p + "mix.in"]).split([inner, inner + 2 * G * N, H], -1)
            u = _conv(u, t[p + "mix.conv"], t[p + "mix.conv.b"])
            u = u * torch.sigmoid(u)
            xs, bs, cs = u.split([inner, G * N, G * N], -1)
            xs = xs.reshape(B, T, H, P)
            bs, cs = (c.reshape(B, T, G, N).repeat_interleave(H // G, 2) for c in (bs, cs))
            dt = torch.nn.functional.softplus(dt + t[p + "mix.dt_bias"].to(F64), threshold=60)
            keep = torch.exp(-torch.exp(t[p + "mix.A_log"].to(F64)) * dt)
            S = torch.zeros((B, H, N, P), dtype=F64, device=dev)
            y = torch.empty_like(xs)
            xd = xs * dt[..., None]
            for n in range(T):
                S = S * keep[:, n, :, None, None] + bs[:, n, :, :, None] * xd[:, n, :, None, :]
                y[:, n] = (cs[:, n, :, None, :] @ S).squeeze(-2)
            y = (y + t[p + "mix.D"].to(F64)[:, None] * xs).reshape(B, T, inner) * (z * torch.sigmoid(z))
            o = _rms(y.view(B, T, m["norm_groups"], -1), eps).reshape(B, T, inner) * t[p + "mix.norm"].to(F64)
        x = x + _lin(o, t[p + "mix.o"]) + _lin(_gelu(_lin(h, t[p + "mlp.up"])), t[p + "mlp.down"])
    return _rms(x, eps) * (1.0 + t["final.norm"].to(F64))


def _petanex(cfg, t, x, ids):
    B, T = ids.shape
    eps, side = cfg["norm"]["eps"], cfg["token_side"]["dim"]

    def norm(u, name):
        return _rms(u, eps) * t[name].to(F64)

    def unit(u):
        return u * torch.rsqrt(u.square().sum(-1, keepdim=True) + 1e-6)

    def expert(u, p, limit):
        g, w = _lin(u, t[p + "gate"]).clamp(max=limit), _lin(u, t[p + "up"]).clamp(-limit, limit)
        return _lin(g * torch.sigmoid(1.702 * g) * (w + 1.0), t[p + "down"])

    for i, l in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", l["mixer"]
        h, H, d, dv = norm(x, f"l{i}.norm1"), m["heads"], m["dim"], m["vdim"]
        if l["type"] == "latent_attention":
            c = norm(_lin(h, t[p + "dkv"]), p + "dkv.norm")
            o = _attend(_lin(h, t[p + "q"]).view(B, T, H, d), _lin(c, t[p + "uk"]).view(B, T, H, d), _lin(c, t[p + "uv"]).view(B, T, H, dv), m["scale"])
            a = _lin(o.reshape(B, T, H * dv), t[p + "o"])
        else:
            q, k, v = (_conv(_lin(h, t[p + n]), t[p + n + ".conv"]) for n in "qkv")
            q, k, v = ((u * torch.sigmoid(u)).view(B, T, -1, n) for u, n in ((q, d), (k, d), (v, dv)))
            q, k = (u.repeat_interleave(H // m["kv_heads"], 2) for u in (unit(q) * d ** -0.5, unit(k)))
            beta, rate = torch.sigmoid(_lin(h, t[p + "b"])), torch.exp(t[p + "A_log"].to(F64))
            if l["type"] == "channel_delta":
                s = torch.nn.functional.softplus(_lin(_lin(h, t[p + "a1"]), t[p + "a2"]) + t[p + "dt_bias"].to(F64), threshold=60)
                keep = torch.exp(-rate[:, None] * s.view(B, T, H, d))
                gate = torch.sigmoid(_lin(_lin(h, t[p + "g1"]), t[p + "g2"]))
            else:
                s = torch.nn.functional.softplus(_lin(h, t[p + "a"]) + t[p + "dt_bias"].to(F64), threshold=60)
                keep = torch.exp(-rate * s)[..., None].expand(B, T, H, d)
                gate = _lin(h, t[p + "g"])
                gate = gate * torch.sigmoid(gate)
            S = torch.zeros((B, H, d, dv), dtype=F64, device=x.device)
            o = torch.empty((B, T, H, dv), dtype=F64, device=x.device)
            for n in range(T):
                S = S * keep[:, n, :, :, None]
                u = beta[:, n, :, None] * (v[:, n] - (k[:, n, :, None, :] @ S).squeeze(-2))
                S = S + k[:, n, :, :, None] * u[:, :, None, :]
                o[:, n] = (q[:, n, :, None, :] @ S).squeeze(-2)
            a = _lin(norm(o, p + "norm").reshape(B, T, H * dv) * gate, t[p + "o"])
        x = x + a * t[f"l{i}.ls1"].to(F64)
        h, f, p = norm(x, f"l{i}.norm2"), l["mlp"], f"l{i}.mlp."
        if f["kind"] == "dense":
            y = _lin(_gelu(_lin(h, t[p + "gate"])) * _lin(h, t[p + "up"]), t[p + "down"])
        else:
            r, flat = f["router"], h.reshape(B * T, -1)
            s = torch.sigmoid(_lin(flat, t[p + "router"]))
            choice = s + t[p + "correction"].to(F64)
            grouped = choice.view(B * T, r["groups"]["count"], -1)
            best = grouped.topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
            allowed = torch.zeros(grouped.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, best, True)
            at = grouped.masked_fill(~allowed[..., None], -math.inf).view(B * T, -1).topk(r["top"], -1).indices
            w = s.gather(1, at)
            w = w / (w.sum(-1, keepdim=True) + 1e-20) * r["scale"]
            y = expert(flat, p + "shared.", f["shared"]["limit"])
            for e in range(r["experts"]):
                row, slot = (at == e).nonzero(as_tuple=True)
                if len(row):
                    y.index_add_(0, row, expert(flat[row], f"{p}e{e}.", f["expert"]["limit"]) * w[row, slot, None])
            y = y.view(B, T, -1)
        x = x + y * t[f"l{i}.ls2"].to(F64)
        p = f"l{i}.side."
        e = t["side.embed"][ids][..., i * side:(i + 1) * side].to(F64)
        x = x + norm(_lin(_gelu(_lin(x, t[p + "gate"])) * e, t[p + "proj"]), p + "norm")
    return norm(x, "final.norm")


def _forward(cfg, t, sequences, places):
    """Logits [places in all, vocab] of whole sequences at the given places of each, in groups of bounded size."""
    longest = max(len(q) for q in sequences)
    group, rows = max(1, 16384 // longest), []
    if "hidden_size" in cfg:
        table, scale, body = t["model.embed_tokens.weight"], float(torch.tensor(math.sqrt(cfg["hidden_size"]), dtype=torch.float32)), _gemma
    else:
        table, scale, body = t["embed"], cfg["embedding"]["scale"], _bolonex if cfg["architecture"] == "Bolonex" else _petanex
    for a in range(0, len(sequences), group):
        part = sequences[a:a + group]
        n = max(len(q) for q in part)
        ids = torch.tensor([q + [0] * (n - len(q)) for q in part], device="cuda")
        x = body(cfg, t, table[ids].to(F64) * scale, ids)
        rows += [x[i, torch.tensor(w, device="cuda")] for i, w in enumerate(places[a:a + group])]
        del x
    logits = _lin(torch.cat(rows), t.get("head", table))
    cap = cfg.get("final_logit_softcapping")
    return cap * torch.tanh(logits / cap) if cap else logits


def exact(case, seed):
    cfg = config(case["model"])
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    t = _weights(cfg, dtype, seed)
    prompts, new = _prompts(case, cfg, seed), case["new"]

    def grown(p, n):
        """A prompt and the n tokens drawn after it."""
        return p + [_successor(case["model"], p[-1], k + 1) for k in range(n)]

    if case["work"] == "decode":
        seqs = [grown(p, WARM + new) for p in prompts]
        ids = torch.tensor([q[-new:] for q in seqs]).T.int()
        return {"logits": _forward(cfg, t, [q[:-1] for q in seqs], [[len(q) - 2] for q in seqs]), "ids": ids}
    if case["work"] == "prompt":
        return {"logits": _forward(cfg, t, prompts, [[len(p) - 1] for p in prompts])}
    if case["work"] == "mixed":
        seqs = [grown(p, WARM) for p in prompts] + [_portion(case, cfg, seed)]
        ids = torch.tensor([_successor(case["model"], q[-1]) for q in seqs]).int()
        return {"logits": _forward(cfg, t, seqs, [[len(q) - 1] for q in seqs]), "ids": ids}
    seqs = [grown(p, new) for p in prompts]
    ids = torch.tensor([q[-new:] for q in seqs])
    if case["work"] == "turn":
        return {"logits": _forward(cfg, t, [q[:-1] for q in seqs], [[len(q) - 2] for q in seqs]), "ids": ids.T.int()}
    return {"logits": _forward(cfg, t, seqs[:1], [list(range(len(seqs[0]) - new, len(seqs[0])))]), "ids": ids}
