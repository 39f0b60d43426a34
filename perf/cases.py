"""The work that programs have this engine do, as cases that can be timed and checked.

A case is one pass through the public entry points: a step of decoding for a batch of requests, a
step that takes in prompts, a step that does both, a short generation in float32, or the sampling of
a step's logits.  Weights and tokens are random (there are no checkpoints here); the shapes are those
of the Llama 3.2 decoders and of the decoders that ``bench.py --family`` builds at width 1,024.

``exact`` restates each model in 64-bit torch from its formulas, with weights drawn as the engine's
random-weights mode draws them (one generator on the device, tensors in the order of their names).
"""
from __future__ import annotations

import math
import random

import torch

from pytriton_llama_b200 import LLM, Engine, EngineConfig, SamplingParams, StepEntry
from pytriton_llama_b200.sampling import Sampler, uniform

F64 = torch.float64
PAGE = 16
STEP_TOKENS = 2048          # token budget of a step, as the scheduler's default
ROOM = 4096                 # tokens that a decoding request may still add before it is started again
WARM_PASSES = 2             # a serving process has run its shapes before (the second time captures them)


# ----------------------------------------------------------------------------- models
def _llama(layers, hidden, heads, kv_heads, head_dim, inter):
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": inter,
            "vocab_size": 128256, "rope_theta": 500000.0,
            "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                             "original_max_position_embeddings": 8192},
            "rms_norm_eps": 1e-5, "tie_word_embeddings": True, "max_position_embeddings": 131072}


def _tibepel(width, layers, ff, vocab):
    """Every fourth layer a selective scan, the others attention in blocks of 256 positions beside a gated delta rule."""
    heads = width // 128
    scan = {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}
    par = {"left": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "mask": {"size": 256}, "scale": 128 ** -0.5},
           "right": {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4}, "left_scale": 0.6, "right_scale": 0.5}
    return {"architecture": "Tibepel", "vocab": vocab, "width": width, "embedding": {"scale": width ** 0.5}, "norm": {"eps": 1e-6},
            "logit_softcap": 30.0, "token_side": {"dim": 64},
            "layers": [{"type": "mamba1" if i % 4 == 0 else "parallel", "mixer": scan if i % 4 == 0 else par,
                        "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}} for i in range(layers)]}


def _sogalix(width, layers, ff, vocab):
    """Of every four layers: attention through latents, generalized delta rule, softmax attention with a sink term, and
    attention through the latents that the first of the four keeps."""
    heads = width // 128
    lat = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 3 * width // 4, "scale": 192 ** -0.5,
           "rot": {"dims": 64, "base": 1000000.0}}
    att = {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
           "q_temp": {"coef": 0.1, "every": 512}}
    kinds = ["latent_attention", "general_delta", "attention", "latent_attention"]
    mixers = [lambda i: lat, lambda i: {"heads": width // 64, "dim": 64, "rank": 64}, lambda i: att, lambda i: dict(lat, kv_from=i - 3)]
    return {"architecture": "Sogalix", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
            "layers": [{"type": kinds[i % 4], "mixer": mixers[i % 4](i), "mlp": {"kind": "dense", "ff": ff}} for i in range(layers)]}


MODELS = {"llama-1b": _llama(16, 2048, 32, 8, 64, 8192), "llama-3b": _llama(28, 3072, 24, 8, 128, 8192),
          "tibepel": _tibepel(1024, 8, 4096, 32000), "sogalix": _sogalix(1024, 8, 4096, 32000)}


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _layers(cfg):
    return cfg.get("num_hidden_layers") or len(cfg["layers"])


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # one user chats at a long context: latency of a token
        {"name": "decode_1b_1", "kind": "decode", "model": "llama-1b", "batch": 1, "shortest": 4000, "longest": 4000},
        # the headline of bench.py: eight requests at a context of 4,096
        {"name": "decode_1b_8", "kind": "decode", "model": "llama-1b", "batch": 8, "shortest": 4096, "longest": 4096},
        # a full server: 64 requests of different ages
        {"name": "decode_1b_64", "kind": "decode", "model": "llama-1b", "batch": 64, "shortest": 256, "longest": 2560},
        # a long prompt comes in
        {"name": "prompt_1b_2048", "kind": "prompt", "model": "llama-1b", "prompts": 1, "shortest": 2048, "longest": 2048},
        # continuous batching: a few short prompts arrive while others decode
        {"name": "mixed_1b", "kind": "mixed", "model": "llama-1b", "prompts": 4, "shortest": 17, "longest": 150,
         "batch": 12, "context": 1000},
        # the larger model (head size 128) in the middle of a run of 32 requests
        {"name": "decode_3b_32", "kind": "decode", "model": "llama-3b", "batch": 32, "shortest": 128, "longest": 2304},
        # the 32-bit path from prompts to tokens, greedy, with log-probabilities
        {"name": "generate_1b_f32", "kind": "generate", "model": "llama-1b", "prompts": 4, "shortest": 33, "longest": 127, "new": 16},
        # recurrent layers beside blocked attention: a long prompt, and eight requests decoding
        {"name": "prompt_tibepel_2048", "kind": "prompt", "model": "tibepel", "prompts": 1, "shortest": 2048, "longest": 2048},
        {"name": "decode_tibepel_8", "kind": "decode", "model": "tibepel", "batch": 8, "shortest": 1024, "longest": 1024},
        # latent attention and the generalized delta rule: eight prompts of different lengths, and eight requests decoding
        {"name": "prompt_sogalix_8", "kind": "prompt", "model": "sogalix", "prompts": 8, "shortest": 65, "longest": 440},
        {"name": "decode_sogalix_8", "kind": "decode", "model": "sogalix", "batch": 8, "shortest": 1024, "longest": 1024},
        # a token for each of eight requests, temperature 0.6 and top-p 0.9 as the command line's defaults
        {"name": "sample_8", "kind": "sample", "rows": 8, "vocab": 128256, "temperature": 0.6, "top_p": 0.9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "generate", "sample"])
    model = rng.choice(["llama-1b", "llama-1b", "llama-3b", "tibepel", "sogalix"])
    if kind == "decode":
        small = model in ("tibepel", "sogalix")
        batch = _log(rng, 1, 8 if small else 32 if model == "llama-3b" else 64)
        longest = _log(rng, 16, min(1024 if small else 4096, 90000 // batch))
        return {"kind": kind, "model": model, "batch": batch, "shortest": max(1, int(longest * rng.uniform(0.1, 1.0))), "longest": longest}
    if kind == "prompt":
        model = "llama-1b" if model == "llama-3b" else model
        prompts = _log(rng, 1, 8)
        longest = _log(rng, 33, 2048 // prompts)
        return {"kind": kind, "model": model, "prompts": prompts, "shortest": max(2, int(longest * rng.uniform(0.2, 1.0))), "longest": longest}
    if kind == "mixed":
        prompts = rng.randint(1, 4)
        longest = _log(rng, 16, 150)
        return {"kind": kind, "model": "llama-1b", "prompts": prompts, "shortest": max(2, int(longest * rng.uniform(0.1, 1.0))),
                "longest": longest, "batch": _log(rng, 1, 16), "context": _log(rng, 64, 1500)}
    if kind == "generate":
        longest = _log(rng, 8, 127)
        return {"kind": kind, "model": "llama-1b", "prompts": rng.randint(1, 4), "shortest": max(1, longest // rng.randint(1, 4)),
                "longest": longest, "new": rng.randint(4, 16)}
    return {"kind": "sample", "rows": _log(rng, 1, 64), "vocab": rng.choice([32000, 128256]),
            "temperature": round(rng.uniform(0.3, 1.2), 2), "top_p": round(rng.uniform(0.5, 1.0), 2)}


def _lengths(count, shortest, longest):
    """``count`` lengths from the shortest to the longest, evenly spread, in no order of size."""
    if count == 1:
        return [longest]
    even = [shortest + (longest - shortest) * i // (count - 1) for i in range(count)]
    random.Random(count).shuffle(even)
    return even


def _starts(case):
    """Tokens that each decoding request holds when it has been filled."""
    if case["kind"] == "decode":
        return _lengths(case["batch"], case["shortest"], case["longest"])
    return [case["context"]] * case["batch"] if case["kind"] == "mixed" else []


def _prompt_lengths(case):
    return _lengths(case["prompts"], case["shortest"], case["longest"]) if "prompts" in case else []


def _tokens(case, seed):
    """(sequences of the decoding requests, prompts): lists of token ids."""
    gen = torch.Generator().manual_seed(seed)
    vocab = _vocab(MODELS[case["model"]])
    pick = lambda n: torch.randint(0, vocab, (n,), generator=gen).tolist()      # noqa: E731
    return [pick(n + ROOM) for n in _starts(case)], [pick(n) for n in _prompt_lengths(case)]


def _logits_to_sample(case, seed):
    """Logits as a head gives them: a broad bulk, and a few tokens that stand out in each row."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(case["rows"], case["vocab"], generator=gen, device="cuda") * 1.5
    at = torch.randint(0, case["vocab"], (case["rows"], 64), generator=gen, device="cuda")
    x.scatter_add_(1, at, torch.rand(case["rows"], 64, generator=gen, device="cuda") * 10)
    return x


# ----------------------------------------------------------------------------- what a program has in hand
class _Serving:
    """An engine with its decoding requests, and the prompts that arrive."""

    def __init__(self, case, seed):
        self.sequences, self.prompts = _tokens(case, seed)
        self.lengths = _starts(case)
        cfg = MODELS[case["model"]]
        longest = max([n + ROOM for n in self.lengths] + [len(p) for p in self.prompts])
        pages = sum(-(-(n + ROOM) // PAGE) for n in self.lengths) + sum(-(-len(p) // PAGE) for p in self.prompts) + 8
        self.engine = Engine(None, EngineConfig(page_size=PAGE, max_gpu_num_blocks=pages, max_seq_len=longest,
                                                max_num_seqs=len(self.lengths) + len(self.prompts),
                                                max_batched_tokens=STEP_TOKENS, compiled_model=True),
                             model_config=cfg, random_seed=seed)
        self.fill()

    def fill(self):
        """Brings every decoding request to its length, a step's budget of tokens at a time."""
        self.at = [0] * len(self.lengths)
        while any(a < n for a, n in zip(self.at, self.lengths)):
            entries, budget = [], STEP_TOKENS
            for r, n in enumerate(self.lengths):
                k = min(budget, n - self.at[r])
                if k > 0:
                    entries.append(StepEntry(r, self.sequences[r][self.at[r]:self.at[r] + k], []))
                    self.at[r] += k
                    budget -= k
            self.engine.step(entries)

    def one_pass(self):
        if any(a == len(s) for a, s in zip(self.at, self.sequences)):
            self.engine.finish_all()
            self.fill()
        entries = [StepEntry(r, [s[a]], [0]) for r, (s, a) in enumerate(zip(self.sequences, self.at))]
        entries += [StepEntry(("prompt", i), p, [len(p) - 1]) for i, p in enumerate(self.prompts)]
        out = self.engine.step(entries, own_logits=False)
        for r in range(len(self.at)):
            self.at[r] += 1
        for i in range(len(self.prompts)):
            self.engine.finish(("prompt", i))
        return out.logits


class _Generating:
    """The float32 generation loop: prompts in, greedy tokens and their log-probabilities out."""

    def __init__(self, case, seed):
        self.prompts = _tokens(case, seed)[1]
        self.params = SamplingParams(temperature=0.0, max_gen_len=case["new"], logprobs=True)
        longest = case["longest"] + case["new"]
        self.llm = LLM(None, EngineConfig(dtype="float32", page_size=PAGE, max_gpu_num_blocks=len(self.prompts) * (-(-longest // PAGE) + 1),
                                          max_seq_len=longest, max_num_seqs=len(self.prompts), max_batched_tokens=STEP_TOKENS,
                                          compiled_model=True), model_config=MODELS[case["model"]], random_seed=seed)

    def one_pass(self):
        requests = [self.llm.add_request(p, self.params) for p in self.prompts]
        for _ in self.llm.run():
            pass
        return {"tokens": torch.tensor([r.output for r in requests]), "logprobs": torch.tensor([r.logprobs for r in requests])}


class _Sampling:
    def __init__(self, case, seed):
        self.logits = _logits_to_sample(case, seed)
        self.params = [SamplingParams(temperature=case["temperature"], top_p=case["top_p"], logprobs=True)] * case["rows"]
        self.numbers, self.indices = list(range(case["rows"])), [seed % 1000] * case["rows"]
        from pytriton_llama_b200.ops.cuda import CudaOps
        self.sampler = Sampler(CudaOps(torch.device("cuda:0")), "cuda:0", seed=0)

    def one_pass(self):
        tokens, logprobs = self.sampler.sample_device(self.logits, self.params, self.numbers, self.indices)
        return {"tokens": tokens, "logprobs": logprobs}


def prepare(case, seed):
    state = {"generate": _Generating, "sample": _Sampling}.get(case["kind"], _Serving)(case, seed)
    for _ in range(WARM_PASSES):
        state.one_pass()
    return state


def run(state):
    return state.one_pass()


# ----------------------------------------------------------------------------- the tensors of a model
def _tensors(cfg):
    """Name -> (shape, how random-weights mode draws it, low, high)."""
    N, ONES, JITTER, AROUND0, ZEROS = ("normal",), ("ones",), ("ones_jitter",), ("zeros_jitter",), ("zeros",)
    U = lambda lo, hi: ("uniform", lo, hi)      # noqa: E731
    t = {}
    if "architectures" in cfg:
        H, I, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
        q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
        t["model.embed_tokens.weight"], t["model.norm.weight"] = ((cfg["vocab_size"], H), N), ((H,), ONES)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for name, shape in (("self_attn.q_proj", (q, H)), ("self_attn.k_proj", (kv, H)), ("self_attn.v_proj", (kv, H)),
                                ("self_attn.o_proj", (H, q)), ("mlp.gate_proj", (I, H)), ("mlp.up_proj", (I, H)), ("mlp.down_proj", (H, I))):
                t[p + name + ".weight"] = (shape, N)
            for name in ("input_layernorm", "post_attention_layernorm"):
                t[p + name + ".weight"] = ((H,), ONES)
        return t
    W, V = cfg["width"], cfg["vocab"]
    t["embed"], t["head"] = ((V, W), N), ((V, W), N)
    tib = cfg["architecture"] == "Tibepel"
    norms = ["final.norm"] + ([] if tib else ["embed.norm"])
    if tib:
        sd = cfg["token_side"]["dim"]
        t["side.embed"] = ((V, len(cfg["layers"]) * sd), N)
    for i, L in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", L["mixer"], L["mlp"]["ff"]
        x = p + "mix."
        norms += [p + "norm1", p + "norm2"]
        if tib:
            t.update({p + "side.gate": ((sd, W), N), p + "side.proj": ((W, sd), N), p + "side.norm": ((W,), ONES),
                      p + "mlp.gate": ((ff, W), N), p + "mlp.up": ((ff, W), N), p + "mlp.down": ((W, ff), N),
                      p + "mlp.gate.b": ((ff,), AROUND0), p + "mlp.up.b": ((ff,), AROUND0), p + "mlp.down.b": ((W,), AROUND0)})
        else:
            t.update({p + "mlp.up": ((ff, W), N), p + "mlp.down": ((W, ff), N), p + "mlp.act": ((2,), U(-1.0, 1.0))})
        if L["type"] == "mamba1":
            n, s, r = m["inner"], m["state"], m["dt_rank"]
            t.update({x + "in": ((2 * n, W), N), x + "conv": ((n, m["conv"]), U(-0.5, 0.5)), x + "conv.b": ((n,), AROUND0),
                      x + "x": ((r + 2 * s, n), N), x + "dt": ((n, r), N), x + "dt.b": ((n,), U(-4.0, -1.0)),
                      x + "A_log": ((n, s), U(-1.0, 2.0)), x + "D": ((n,), ONES), x + "o": ((W, n), N)})
        elif L["type"] == "parallel":
            a, b = m["left"], m["right"]
            H, q, k, v = a["heads"], a["heads"] * a["dim"], a["kv_heads"] * a["dim"], a["kv_heads"] * a["vdim"]
            y = x + "left."
            t.update({y + "q": ((q, W), N), y + "k": ((k, W), N), y + "v": ((v, W), N), y + "o": ((W, H * a["vdim"]), N),
                      y + "q.b": ((q,), AROUND0), y + "k.b": ((k,), AROUND0), y + "v.b": ((v,), AROUND0), y + "o.b": ((W,), AROUND0),
                      y + "r1": ((H,), U(0.0, 1.0)), y + "r2": ((H,), U(0.05, 1.0)), y + "talk": ((H, H), U(-0.3, 0.7))})
            H, k, v, taps = b["heads"], b["kv_heads"] * b["dim"], b["heads"] * b["vdim"], b["conv"]
            y = x + "right."
            t.update({y + "q": ((k, W), N), y + "k": ((k, W), N), y + "v": ((v, W), N), y + "g": ((v, W), N),
                      y + "q.conv": ((k, taps), U(-0.5, 0.5)), y + "k.conv": ((k, taps), U(-0.5, 0.5)), y + "v.conv": ((v, taps), U(-0.5, 0.5)),
                      y + "b": ((H, W), N), y + "a": ((H, W), N), y + "A_log": ((H,), U(-2.0, 1.0)), y + "dt_bias": ((H,), U(-2.0, 1.0)),
                      y + "norm": ((b["vdim"],), ONES), y + "o": ((W, v), N)})
        elif L["type"] == "general_delta":
            n, r = m["heads"] * m["dim"], m["rank"]
            t.update({x + k: ((n, W), N) for k in "rkvga"})
            t.update({x + "a.b": ((n,), U(-2.0, 2.0)), x + "w1": ((r, W), N), x + "w2": ((n, r), N), x + "w0": ((n,), U(-4.0, 3.0)),
                      x + "norm": ((n,), ONES), x + "o": ((W, n), N)})
        elif L["type"] == "attention":
            q, k, v = m["heads"] * m["dim"], m["kv_heads"] * m["dim"], m["kv_heads"] * m["vdim"]
            t.update({x + "q": ((q, W), N), x + "k": ((k, W), N), x + "v": ((v, W), N), x + "o": ((W, m["heads"] * m["vdim"]), N)})
        else:
            H, d, n, e, R, Q = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
            t.update({x + "dq": ((Q, W), N), x + "dq.norm": ((Q,), JITTER), x + "uq": ((H * (d + n), Q), N), x + "uk": ((H * d, R), N),
                      x + "uv": ((H * e, R), N), x + "g": ((H, W), N), x + "o": ((W, H * e), N)})
            if "kv_from" not in m:
                t.update({x + "dkv": ((R + n, W), N), x + "dkv.norm": ((R,), JITTER)})
    for name in norms:
        t[name] = ((W,), ZEROS if tib else ONES)
        if not tib:
            t[name + ".b"] = ((W,), AROUND0)
    return t


def _draw_weights(cfg, seed, dtype):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    for name, (shape, how) in sorted(_tensors(cfg).items()):
        if how[0] in ("ones", "zeros"):
            t = torch.full(shape, float(how[0] == "ones"), device="cuda")
        elif how[0] == "uniform":
            t = torch.rand(shape, generator=gen, device="cuda").mul_(how[2] - how[1]).add_(how[1])
        else:
            t = torch.randn(shape, generator=gen, device="cuda")
            t = t.mul_(0.02) if how[0] == "normal" else t.mul_(0.1) if how[0] == "zeros_jitter" else 1.0 + 0.01 * t
        out[name] = t.to(dtype)
    return out


# ----------------------------------------------------------------------------- the work of a pass
def _sizes(cfg):
    """(elements of the matrices that every token passes, elements of the head, floats of a request's recurrent states)."""
    tables = ("embed", "side.embed", "head", "model.embed_tokens.weight")
    matrices = sum(shape[0] * shape[1] for name, (shape, how) in _tensors(cfg).items()
                   if len(shape) == 2 and how[0] == "normal" and name not in tables)
    state = 0
    for L in cfg.get("layers", ()):
        m = L["mixer"]
        if L["type"] == "mamba1":
            state += m["inner"] * (m["state"] + m["conv"] - 1)
        elif L["type"] == "parallel":
            b = m["right"]
            state += b["heads"] * b["dim"] * b["vdim"] + (b["conv"] - 1) * (2 * b["kv_heads"] * b["dim"] + b["heads"] * b["vdim"])
        elif L["type"] == "general_delta":
            state += m["heads"] * m["dim"] ** 2
    return matrices, _vocab(cfg) * (cfg.get("hidden_size") or cfg["width"]), state


def _attention(cfg, position):
    """(cached elements that the token at ``position`` reads, operations of its scores and sums), over all layers."""
    if "architectures" in cfg:
        n, d, L = position + 1, cfg["head_dim"], cfg["num_hidden_layers"]
        return 2 * L * n * cfg["num_key_value_heads"] * d, 4 * L * n * cfg["num_attention_heads"] * d
    read = ops = 0
    for L in cfg["layers"]:
        m, n = L["mixer"], position + 1
        if L["type"] == "parallel":
            m = m["left"]
            n = position % m["mask"]["size"] + 1
        if L["type"] in ("parallel", "attention"):
            read += n * m["kv_heads"] * (m["dim"] + m["vdim"])
            ops += 2 * n * m["heads"] * (m["dim"] + m["vdim"])
        elif L["type"] == "latent_attention":
            read += n * (m["kv_rank"] + m["rot_dim"])
            ops += 2 * n * m["heads"] * (2 * m["kv_rank"] + m["rot_dim"])
    return read, ops


def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n, "flops": 4 * n}
    cfg = MODELS[case["model"]]
    size = 4 if case["kind"] == "generate" else 2
    matrices, head, state = _sizes(cfg)
    steps = [(_starts(case), _prompt_lengths(case))]
    if case["kind"] == "generate":
        steps += [([n + i for n in steps[0][1]], []) for i in range(case["new"] - 1)]
    moved = ops = 0
    for decoding, prompts in steps:
        rows, tokens = len(decoding) + len(prompts), len(decoding) + sum(prompts)
        moved += size * (matrices + head) + 4 * rows * _vocab(cfg) + 4 * state * (2 * len(decoding) + len(prompts))
        ops += 2 * matrices * tokens + 2 * head * rows + 6 * state * tokens
        for n in decoding:
            read, do = _attention(cfg, n)
            moved, ops = moved + size * read, ops + do
        for n in prompts:                       # every position once; the middle one stands for the mean
            moved += size * n * _attention(cfg, 0)[0]
            ops += n * (_attention(cfg, 0)[1] + sum(_attention(cfg, p)[1] - _attention(cfg, 0)[1] for p in range(0, n, 16)) // -(-n // 16))
    return {"bytes": moved, "flops": ops}


def tolerance(case):
    """Float32 sums stay within 2e-7 of ``exact``.  Where activations are rounded to bfloat16 in every layer, two summation
    orders of the products (other kernels for the same step) gave logits 0.015 to 0.022 apart for the Llama decoders and
    0.004 to 0.007 for the others, the largest difference 0.11 of the logits' root mean square."""
    if case["kind"] in ("sample", "generate"):
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.03 if case["model"].startswith("llama") else 0.02, "max": 0.4}


# ----------------------------------------------------------------------------- 64-bit restatements
class _Plain:
    """A model in 64 bits over whole sequences laid end to end: ``spans`` are the sequences' rows of x [tokens, width]."""

    def __init__(self, cfg, weights, sequences):
        self.cfg, self.raw = cfg, weights
        self.ids = torch.tensor([t for s in sequences for t in s], device="cuda")
        self.spans, a = [], 0
        for s in sequences:
            self.spans.append((a, a + len(s)))
            a += len(s)
        self.positions = torch.cat([torch.arange(b - a, device="cuda") for a, b in self.spans])

    def w(self, name):
        return self.raw[name].to(F64)

    def lin(self, h, name, part=slice(None)):
        return h @ self.w(name)[part].T

    def by_rows(self, fn, x, rows=8192):
        return torch.cat([fn(x[a:a + rows]) for a in range(0, len(x), rows)])

    def padded(self, x):
        """x [tokens, ...] as [sequences, longest, ...] (zeros behind the shorter ones, which nothing before them sees)."""
        return torch.nn.utils.rnn.pad_sequence([x[a:b] for a, b in self.spans], batch_first=True)

    def flat(self, x):
        return torch.cat([x[i, :b - a] for i, (a, b) in enumerate(self.spans)])

    def conv(self, x, name, bias=None):
        """Causal convolution per channel; the last column of the weight is the current token's."""
        w, x = self.w(name), self.padded(x)
        taps, n = w.shape[1], x.shape[1]
        x = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
        y = self.flat(sum(x[:, k:k + n] * w[:, k] for k in range(taps)))
        return y if bias is None else y + self.w(bias)

    def attention(self, q, k, v, scale, bias=None, block=0, mix=None, sink=False):
        """q [tokens, heads, d], k and v [tokens, groups, ...], causal inside each sequence (inside blocks of ``block``
        positions where that is set); ``bias(distance)`` [heads, queries, keys] is subtracted from the scores, ``mix``
        [heads, heads] applied to the weights, ``sink`` adds a term of score 0 to the denominator."""
        H, G = q.shape[1], k.shape[1]
        out = torch.empty(len(q), H, v.shape[2], dtype=F64, device="cuda")
        for a, b in self.spans:
            for c in range(a, b, block or 512):
                e = min(b, c + (block or 512))
                s = c if block else a
                qs = q[c:e].view(e - c, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, (H // G) * (e - c), -1)
                score = (qs @ k[s:e].permute(1, 2, 0) * scale).view(H, e - c, e - s)
                dist = torch.arange(c, e, device="cuda")[:, None] - torch.arange(s, e, device="cuda")[None, :]
                if bias is not None:
                    score = score - bias(dist.clamp(min=0).to(F64))
                score = score.masked_fill(dist < 0, -math.inf)
                if sink:
                    top = score.amax(-1, keepdim=True).clamp(min=0)
                    p = torch.exp(score - top)
                    p = p / (p.sum(-1, keepdim=True) + torch.exp(-top))
                else:
                    p = torch.softmax(score, -1)
                if mix is not None:
                    p = torch.einsum("hg,gij->hij", mix, p)
                o = p.view(G, (H // G) * (e - c), e - s) @ v[s:e].transpose(0, 1)
                out[c:e] = o.view(H, e - c, -1).transpose(0, 1)
        return out

    def rows(self, per_sequence=1):
        """Row numbers of the last ``per_sequence`` tokens of every sequence."""
        return torch.tensor([r for _, b in self.spans for r in range(b - per_sequence, b)], device="cuda")


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _llama_logits(m: _Plain, last):
    c = m.cfg
    H, G, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    f = c["rope_theta"] ** (-torch.arange(0, d, 2, dtype=F64, device="cuda") / d)
    s = c["rope_scaling"]
    turns = s["original_max_position_embeddings"] * f / (2 * math.pi)
    blend = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
    angle = m.positions.to(F64)[:, None] * (f * blend + f / s["factor"] * (1 - blend))[None, :]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(x):
        u, v = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    x = m.w("model.embed_tokens.weight")[m.ids]
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * m.w(p + "input_layernorm.weight")
        q, k, v = (m.lin(h, p + f"self_attn.{n}_proj.weight").view(len(h), -1, d) for n in "qkv")
        o = m.attention(turn(q), turn(k), v, d ** -0.5)
        x = x + m.lin(o.reshape(len(h), H * d), p + "self_attn.o_proj.weight")
        gate, up, down = (m.w(p + f"mlp.{n}_proj.weight").T for n in ("gate", "up", "down"))
        norm = m.w(p + "post_attention_layernorm.weight")
        x = m.by_rows(lambda y: y + (_silu((h := _rms(y, eps) * norm) @ gate) * (h @ up)) @ down, x)
    return (_rms(x[m.rows(last)], eps) * m.w("model.norm.weight")) @ m.w("model.embed_tokens.weight").T


def _tibepel_logits(m: _Plain, last):
    c = m.cfg
    eps, W = c["norm"]["eps"], c["width"]
    softplus = lambda z: torch.nn.functional.softplus(z, threshold=100)      # noqa: E731
    around = lambda x, n: _rms(x, eps) * (1 + m.w(n))      # noqa: E731
    i = torch.arange(W // 2, dtype=F64, device="cuda")
    angle = m.positions.to(F64)[:, None] * 10000.0 ** (-2 * i / W)[None, :]
    x = m.w("embed")[m.ids] * c["embedding"]["scale"] + torch.stack([angle.sin(), angle.cos()], -1).view(-1, W)

    def scan(h, p, k):
        n, s, r = k["inner"], k["state"], k["dt_rank"]
        xz = m.lin(h, p + "in")
        u = _silu(m.conv(xz[:, :n], p + "conv", p + "conv.b"))
        low = m.lin(u, p + "x")
        dt = softplus(m.lin(low[:, :r], p + "dt") + m.w(p + "dt.b"))
        A = -torch.exp(m.w(p + "A_log"))
        up, dtp, B, C = (m.padded(t) for t in (u, dt, low[:, r:r + s], low[:, r + s:]))
        S, y = torch.zeros(len(up), n, s, dtype=F64, device="cuda"), torch.empty_like(up)
        for t in range(up.shape[1]):
            S = torch.exp(dtp[:, t, :, None] * A) * S + (dtp[:, t] * up[:, t])[..., None] * B[:, t, None, :]
            y[:, t] = (S * C[:, t, None, :]).sum(-1)
        return m.lin((m.flat(y) + m.w(p + "D") * u) * _silu(xz[:, n:]), p + "o")

    def blocked(h, p, k):
        H, G = k["heads"], k["kv_heads"]
        q, kk, v = ((m.lin(h, p + n) + m.w(p + n + ".b")).view(len(h), g, -1) for n, g in (("q", H), ("k", G), ("v", G)))
        r1, r2 = m.w(p + "r1")[:, None, None], m.w(p + "r2")[:, None, None]
        o = m.attention(q, kk, _rms(v, eps), k["scale"], bias=lambda dist: r1 * torch.log1p(r2 * dist), block=k["mask"]["size"],
                        mix=m.w(p + "talk"))
        return m.lin(o.reshape(len(h), -1), p + "o") + m.w(p + "o.b")

    def delta(h, p, k):
        H, G, d, e = k["heads"], k["kv_heads"], k["dim"], k["vdim"]
        q, kk, v = (_silu(m.conv(m.lin(h, p + n), p + n + ".conv")).view(len(h), g, -1) for n, g in (("q", G), ("k", G), ("v", H)))
        unit = lambda y: (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)      # noqa: E731
        beta = torch.sigmoid(m.lin(h, p + "b"))
        g = torch.exp(-torch.exp(m.w(p + "A_log")) * softplus(m.lin(h, p + "a") + m.w(p + "dt_bias")))
        q, kk, v, beta, g = (m.padded(t) for t in (unit(q) * d ** -0.5, unit(kk), v, beta, g))
        S, o = torch.zeros(len(q), H, d, e, dtype=F64, device="cuda"), torch.empty_like(v)
        for t in range(q.shape[1]):
            S = g[:, t, :, None, None] * S
            u = beta[:, t, :, None] * (v[:, t] - (S * kk[:, t, :, :, None]).sum(-2))
            S = S + kk[:, t, :, :, None] * u[:, :, None, :]
            o[:, t] = (S * q[:, t, :, :, None]).sum(-2)
        o = (_rms(m.flat(o), eps) * m.w(p + "norm")).reshape(len(h), H * e)
        return m.lin(o * _silu(m.lin(h, p + "g")), p + "o")

    for i, L in enumerate(c["layers"]):
        p, k = f"l{i}.", L["mixer"]
        h = around(x, p + "norm1")
        if L["type"] == "mamba1":
            x = x + scan(h, p + "mix.", k)
        else:
            x = x + k["left_scale"] * blocked(h, p + "mix.left.", k["left"]) + k["right_scale"] * delta(h, p + "mix.right.", k["right"])
        h, lim, f = around(x, p + "norm2"), L["mlp"]["limit"], p + "mlp."
        g = (m.lin(h, f + "gate") + m.w(f + "gate.b")).clamp(max=lim)
        u = (m.lin(h, f + "up") + m.w(f + "up.b")).clamp(-lim, lim)
        x = x + m.lin(g * torch.sigmoid(1.702 * g) * (u + 1), f + "down") + m.w(f + "down.b")
        sd, s = c["token_side"]["dim"], p + "side."
        e = m.w("side.embed")[:, i * sd:(i + 1) * sd][m.ids]
        y = m.lin(torch.nn.functional.gelu(m.lin(x, s + "gate"), approximate="tanh") * e, s + "proj")
        x = x + _rms(y, eps) * m.w(s + "norm")
    cap = c["logit_softcap"]
    return cap * torch.tanh(m.lin(around(x[m.rows(last)], "final.norm"), "head") / cap)


def _sogalix_logits(m: _Plain, last):
    c = m.cfg
    eps = c["norm"]["eps"]

    def norm(x, n):
        x = x - x.mean(-1, keepdim=True)
        return _rms(x, eps) * m.w(n) + m.w(n + ".b")

    def turn(x, rot):
        i = torch.arange(rot["dims"] // 2, dtype=F64, device="cuda")
        angle = m.positions.to(F64)[:, None] * rot["base"] ** (-2.0 * i / rot["dims"])[None, :]
        cos, sin, u, v = angle.cos()[:, None], angle.sin()[:, None], x[..., 0::2], x[..., 1::2]
        return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).view_as(x)

    def delta(h, p, k):
        H, d = k["heads"], k["dim"]
        r, kk, v = (m.lin(h, p + n).view(len(h), H, d) for n in "rkv")
        w = torch.tanh(m.lin(h, p + "w1")) @ m.w(p + "w2").T + m.w(p + "w0")
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(w)).view(-1, H, d)
        a = torch.sigmoid(m.lin(h, p + "a") + m.w(p + "a.b")).view(-1, H, d)
        u = kk / torch.sqrt((kk * kk).sum(-1, keepdim=True) + 1e-6)
        r, kk, v, w, au, u = (m.padded(t) for t in (r, kk, v, w, a * u, u))
        S, o = torch.zeros(len(r), H, d, d, dtype=F64, device="cuda"), torch.empty_like(v)
        for t in range(r.shape[1]):
            uS = (u[:, t, :, :, None] * S).sum(-2)
            S = w[:, t, :, :, None] * S - au[:, t, :, :, None] * uS[:, :, None, :] + kk[:, t, :, :, None] * v[:, t, :, None, :]
            o[:, t] = (r[:, t, :, :, None] * S).sum(-2)
        o = _rms(m.flat(o), eps).reshape(len(h), H * d) * m.w(p + "norm") * torch.sigmoid(m.lin(h, p + "g"))
        return m.lin(o, p + "o")

    def sink(h, p, k):
        t = k["q_temp"]
        warm = 1.0 + t["coef"] * torch.log(torch.floor((m.positions.to(F64) + 1) / t["every"]) + 1.0)
        q, kk, v = (m.lin(h, p + n).view(len(h), g, -1) for n, g in (("q", k["heads"]), ("k", k["kv_heads"]), ("v", k["kv_heads"])))
        return m.lin(m.attention(q * warm[:, None, None], kk, v, k["scale"], sink=True).reshape(len(h), -1), p + "o")

    kept = {}

    def latent(h, p, k, i):
        H, d, n, R = k["heads"], k["dim"], k["rot_dim"], k["kv_rank"]
        if "kv_from" not in k:
            kv = m.lin(h, p + "dkv")
            kept[i] = _rms(kv[:, :R], eps) * m.w(p + "dkv.norm"), turn(kv[:, None, R:], k["rot"])
        latents, kr = kept[k.get("kv_from", i)]
        q = m.lin(_rms(m.lin(h, p + "dq"), eps) * m.w(p + "dq.norm"), p + "uq").view(len(h), H, d + n)
        q = torch.cat([q[..., :d], turn(q[..., d:], k["rot"])], -1)
        kk = torch.cat([m.lin(latents, p + "uk").view(len(h), H, d), kr.expand(-1, H, -1)], -1)
        o = m.attention(q, kk, m.lin(latents, p + "uv").view(len(h), H, -1), k["scale"])
        return m.lin((o * torch.sigmoid(m.lin(h, p + "g"))[..., None]).reshape(len(h), -1), p + "o")

    x = norm(m.w("embed")[m.ids], "embed.norm")
    for i, L in enumerate(c["layers"]):
        p, k = f"l{i}.", L["mixer"]
        h, mix = norm(x, p + "norm1"), p + "mix."
        x = x + (delta(h, mix, k) if L["type"] == "general_delta" else sink(h, mix, k) if L["type"] == "attention" else latent(h, mix, k, i))
        z = m.lin(norm(x, p + "norm2"), p + "mlp.up")
        a, b = torch.nn.functional.softplus(m.w(p + "mlp.act"))
        below = z.clamp(max=0)
        x = x + m.lin(torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(below) - below)) + 0.5 * z, p + "mlp.down")
    return m.lin(norm(x[m.rows(last)], "final.norm"), "head")


def _logits64(cfg, weights, sequences, last=1):
    """Logits of the last tokens of every sequence, in the order of the sequences."""
    fn = _llama_logits if "architectures" in cfg else _tibepel_logits if cfg["architecture"] == "Tibepel" else _sogalix_logits
    return fn(_Plain(cfg, weights, sequences), last)


def _exact_sample(case, seed):
    """The smallest set of most probable tokens whose mass exceeds top_p, renormalised; the token where the running sum
    over the kept ones, in the order of their ids, passes the uniform number."""
    logits = _logits_to_sample(case, seed).to(F64)
    p = torch.softmax(logits / case["temperature"], -1)
    order = p.sort(-1, descending=True)
    keep = torch.zeros_like(p, dtype=torch.bool).scatter_(1, order.indices, order.values.cumsum(-1) - order.values <= case["top_p"])
    cdf = torch.where(keep, p, 0.0).cumsum(-1)
    u = torch.tensor([uniform(0, r, seed % 1000) for r in range(case["rows"])], dtype=F64, device="cuda")[:, None]
    tokens = torch.searchsorted(cdf, u * cdf[:, -1:], right=True).clamp(max=case["vocab"] - 1)
    return {"tokens": tokens[:, 0].int(), "logprobs": torch.log_softmax(logits, -1).gather(1, tokens)[:, 0]}


def exact(case, seed):
    if case["kind"] == "sample":
        return _exact_sample(case, seed)
    cfg = MODELS[case["model"]]
    sequences, prompts = _tokens(case, seed)
    if case["kind"] != "generate":
        held = [s[:n + WARM_PASSES + 1] for s, n in zip(sequences, _starts(case))] + prompts
        return _logits64(cfg, _draw_weights(cfg, seed, torch.bfloat16), held)
    weights, new = _draw_weights(cfg, seed, torch.float32), case["new"]
    held = [list(p) for p in prompts]
    for _ in range(new):
        for s, row in zip(held, _logits64(cfg, weights, held)):
            s.append(int(row.argmax()))
    logits = _logits64(cfg, weights, held, last=new + 1).view(len(held), new + 1, -1)[:, :new]
    tokens = torch.tensor([s[-new:] for s in held], device="cuda")
    return {"tokens": tokens, "logprobs": torch.log_softmax(logits, -1).gather(-1, tokens[..., None])[..., 0]}
