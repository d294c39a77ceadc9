"""Representative work for the engine, with inputs, expected results and bounds.

Each case is one pass of something a program does with the engine through its Python entry points:

* ``decode``: ``batch`` live requests with ``prefix`` tokens in the cache are fed ``steps`` further tokens each, one
  :meth:`Engine.step` per token; the last step returns the logits of up to eight of them (the requests whose answers end).
* ``prompt``: one sequence starts anew, reads a prompt of ``tokens`` ids and returns the logits behind it
  (:meth:`Model.reset`, :meth:`Model.prefill`, :meth:`Model.get_logits`).
* ``mixed``: one step with a prompt portion of ``tokens`` ids of a new request beside ``batch`` decode rows.
* ``chat``: a few short prompts answered greedily by streams, prompt to last token (:meth:`Model.stream_begin`,
  :meth:`Model.stream_run`, :meth:`Model.get_logits`).

Models have random weights (a function of a seed, the tensor's name and the element's index) and are kept for the life of
the process, as a server keeps them.  Token ids are uniform.  What a request is fed is given, not sampled, wherever the
model runs in bfloat16: two correct bfloat16 engines soon sample different tokens from random weights.  For the same
reason the designs with routed experts are not among the models here: a token whose second and third expert tie within
bfloat16 takes another path through the model.
"""
import math

import numpy as np
import torch

from purhie_b200.api import GenOptions, load_model_random
from purhie_b200.engine import Engine, StepEntry
from purhie_b200.sampling import SamplerParams

CONTEXT = 4096
PAGE = 16
GROWTH = 512                      # a decoding request that has grown by this many tokens ends and a new one takes its place
WANTED = 8                        # requests whose logits a decode or mixed pass returns, at most

_QWEN3 = dict(architectures=["Qwen3ForCausalLM"], num_key_value_heads=8, head_dim=128, vocab_size=151936,
              max_position_embeddings=CONTEXT, rope_theta=1e6, rms_norm_eps=1e-6)
_QWEN3_06B = dict(_QWEN3, num_hidden_layers=28, hidden_size=1024, intermediate_size=3072, num_attention_heads=16,
                  tie_word_embeddings=True)


def _noditar():
    """The 2k size of the Noditar design, as the benchmark runs it."""
    latent = {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5}
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    ssm = {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    dense = {"kind": "dense", "ff": 8192, "limit": 7.0}
    layers = [{"type": "latent_attention", "mixer": latent, "mlp": dense}, {"type": "attention", "mixer": att, "mlp": dense},
              {"type": "mamba2", "mixer": ssm, "mlp": None}, {"type": "mamba2", "mixer": ssm, "mlp": dense}]
    return {"architecture": "Noditar", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6}, "streams": 4, "layers": layers,
            "max_position": CONTEXT}


def _vokepel():
    """The 2k size of the Vokepel design, as the benchmark runs it."""
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "mask": {"size": 1024}, "scale": 128 ** -0.5, "softcap": 25.0}
    left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "mask": {"size": 1024}, "rot": {"base": 1e6, "dims": 128},
            "scale": 128 ** -0.5}
    both = {"left": left, "right": {"width": 2048}, "left_scale": 0.8, "right_scale": 1.2}
    dense = {"kind": "dense", "ff": 8192}
    layers = [{"type": "attention", "mixer": att, "mlp": dense}, {"type": "parallel", "mixer": both, "mlp": dense},
              {"type": "attention", "mixer": att, "mlp": dense}, {"type": "parallel", "mixer": both, "mlp": dense}]
    return {"architecture": "Vokepel", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6}, "residual_mult": 0.6,
            "logit_scale": 1.5, "logit_softcap": 40.0, "layers": layers, "loop": {"start": 1, "stop": 3, "times": 1},
            "max_position": CONTEXT}


# name: (configuration, weight seed, dtype, std, norm weights from, to, most requests a pass has, longest prefix)
MODELS = {
    # eight layers of the Qwen3-8B shape with its whole output matrix: 4.3 GB of weights, 34 times the L2
    "qwen3-8b-8": (dict(_QWEN3, num_hidden_layers=8, hidden_size=4096, intermediate_size=12288, num_attention_heads=32,
                         tie_word_embeddings=False), 2, "bfloat16", 0.02, 1.0, 1.0, 64, 2048),
    "qwen3-0.6b": (_QWEN3_06B, 3, "bfloat16", 0.02, 1.0, 1.0, 32, 2048),
    "qwen3-0.6b-fp32": (_QWEN3_06B, 3, "float32", 0.02, 1.0, 1.0, 8, 1024),
    "qwen3-tiny-b": (dict(_QWEN3, num_hidden_layers=3, hidden_size=96, num_attention_heads=8, num_key_value_heads=2, head_dim=32,
                          intermediate_size=224, vocab_size=512, rms_norm_eps=1e-5, tie_word_embeddings=False,
                          max_position_embeddings=256), 1, "float32", 0.03, 0.8, 1.2, 4, 128),
    "noditar-2k": (_noditar(), 3, "bfloat16", 0.02, 1.0, 1.0, 16, 2048),
    "vokepel-2k": (_vokepel(), 3, "bfloat16", 0.02, 1.0, 1.0, 16, 2048),
}


def listed():
    return [
        # the tests' tiny model: three short prompts answered in float32; every call is a launch and a wait
        {"name": "tiny_fp32_chat", "model": "qwen3-tiny-b", "kind": "chat", "prompts": "2,40,97", "new": 12},
        # the float32 path at a real size, which other implementations are compared with: a prompt, and a few requests decoding
        {"name": "q06_fp32_prompt_256", "model": "qwen3-0.6b-fp32", "kind": "prompt", "tokens": 256},
        {"name": "q06_fp32_decode_b4", "model": "qwen3-0.6b-fp32", "kind": "decode", "batch": 4, "prefix": 256, "steps": 2},
        # one user of a small model, and a server that lets a 512-token prompt portion in beside 32 decoding requests
        {"name": "q06_decode_b1", "model": "qwen3-0.6b", "kind": "decode", "batch": 1, "prefix": 2048, "steps": 8},
        {"name": "q06_mixed_32_512", "model": "qwen3-0.6b", "kind": "mixed", "batch": 32, "prefix": 2048, "tokens": 512},
        # a question of ordinary length, no multiple of any tile
        {"name": "q06_prompt_517", "model": "qwen3-0.6b", "kind": "prompt", "tokens": 517},
        # the headline benchmark: one user, a small and a large batch behind 2,048-token prefixes, a 2,048-token prompt
        {"name": "q8b_decode_b1", "model": "qwen3-8b-8", "kind": "decode", "batch": 1, "prefix": 2048, "steps": 8},
        {"name": "q8b_decode_b8", "model": "qwen3-8b-8", "kind": "decode", "batch": 8, "prefix": 2048, "steps": 8},
        {"name": "q8b_decode_b64", "model": "qwen3-8b-8", "kind": "decode", "batch": 64, "prefix": 2048, "steps": 8},
        {"name": "q8b_prompt_2048", "model": "qwen3-8b-8", "kind": "prompt", "tokens": 2048},
        # two of the other designs: state-space and latent-attention layers on a long prompt, heads that talk and a
        # recurrent unit in a batch of decoding requests
        {"name": "noditar_prompt_2048", "model": "noditar-2k", "kind": "prompt", "tokens": 2048},
        {"name": "vokepel_decode_b8", "model": "vokepel-2k", "kind": "decode", "batch": 8, "prefix": 2048, "steps": 8},
    ]


def _between(rng, low, high):
    """A whole number from low to high, uniform over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    model = rng.choices(list(MODELS), weights=[8, 6, 3, 1, 2, 2])[0]
    batch, prefix = MODELS[model][6:]
    if model == "qwen3-tiny-b":
        lengths = [_between(rng, 1, 128) for _ in range(rng.randint(1, batch))]
        return {"model": model, "kind": "chat", "prompts": ",".join(map(str, lengths)), "new": _between(rng, 2, 32)}
    kind = rng.choices(["decode", "prompt", "mixed"], weights=[5, 4, 2])[0]
    if kind == "prompt":
        return {"model": model, "kind": kind, "tokens": _between(rng, 2, prefix)}
    case = {"model": model, "kind": kind, "batch": _between(rng, 1, batch), "prefix": _between(rng, 16, prefix)}
    if kind == "decode":
        return dict(case, steps=2 if model == "qwen3-0.6b-fp32" else 8)
    return dict(case, tokens=_between(rng, 16, prefix // 4))


# ---- what a program has in hand --------------------------------------------------------------------------------------
_models = {}


def _model(name):
    """The loaded model and the engine over its cache, with room for three times the largest pass."""
    if name not in _models:
        config, seed, dtype, std, low, high, batch, prefix = MODELS[name]
        model = load_model_random(config, seed, dtype, std=std, scale_low=low, scale_high=high)
        context = config.get("max_position_embeddings", CONTEXT)
        tokens = 3 * batch * (min(prefix + GROWTH, context) + PAGE) + 8 * context
        model.kv_cache_init(context, max_sequences=3 * batch + 16, page_size=PAGE, kv_tokens=tokens)
        _models[name] = (model, Engine.attach(model))
    return _models[name]


class _State:
    """Live requests or sequences of a model; they end with the state."""
    made = 0

    def __init__(self, case, seed):
        self.case = case
        self.model, self.engine = _model(case["model"])
        self.given = _inputs(case, seed)
        self.seqs, self.requests = [], []
        _State.made += 1
        self.key = _State.made
        if case["kind"] in ("prompt", "chat"):
            for _ in self.given["prompts"]:
                self.seqs.append(self.model.seq_new())
        else:
            for i in range(case["batch"]):
                self.requests.append((self.key, i))
                self.engine.add_request(self.requests[i])
                self.engine.step([StepEntry(self.requests[i], self.given["prefixes"][i], [])])
            self.done = 0

    def room_for(self, steps):
        """Requests that have grown to their end are followed by new ones with the same prefixes."""
        if self.done + steps <= GROWTH:
            return
        for i, r in enumerate(self.requests):
            self.engine.release(r)
            self.engine.add_request(r)
            self.engine.step([StepEntry(r, self.given["prefixes"][i], [])])
        self.done = 0

    def __del__(self):
        for s in self.seqs:
            self.model.seq_free(s)
        for r in self.requests:
            self.engine.release(r)


def _inputs(case, seed):
    """Token ids, and which requests' logits are wanted, from the seed alone."""
    config = MODELS[case["model"]][0]
    rng = np.random.default_rng(seed)
    ids = lambda n: rng.integers(0, config.get("vocab_size") or config["vocab"], size=n).tolist()
    if case["kind"] == "chat":
        return {"prompts": [ids(int(n)) for n in case["prompts"].split(",")]}
    if case["kind"] == "prompt":
        return {"prompts": [ids(case["tokens"])]}
    given = {"prefixes": [ids(case["prefix"]) for _ in range(case["batch"])],
             "fed": [ids(GROWTH) for _ in range(case["batch"])],
             "wanted": sorted(rng.choice(case["batch"], size=min(WANTED, case["batch"]), replace=False).tolist())}
    if case["kind"] == "mixed":
        given["portion"] = ids(case["tokens"])
    return given


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    case, given, model, engine = state.case, state.given, state.model, state.engine
    kind = case["kind"]
    if kind == "prompt":
        model.seq_select(state.seqs[0])
        model.reset()
        model.prefill(given["prompts"][0])
        return model.get_logits()
    if kind == "chat":
        streams = []
        options = GenOptions(sampler=SamplerParams.greedy(), max_new_tokens=case["new"], ignore_eog=True)
        for seq, prompt in zip(state.seqs, given["prompts"]):
            model.seq_select(seq)
            model.reset()
            streams.append(model.stream_begin(prompt, options))
        model.stream_run(streams, case["new"])
        tokens = np.array([s.emitted for s in streams])
        for s in streams:
            s.free()
        logits = []
        for seq in state.seqs:
            model.seq_select(seq)
            logits.append(model.get_logits())
        return {"tokens": tokens, "logits": np.stack(logits)}
    wanted = set(given["wanted"])
    if kind == "mixed":
        state.room_for(1)
        engine.add_request((state.key, "portion"))
        entries = [StepEntry(r, [given["fed"][i][state.done]], [0] if i in wanted else []) for i, r in enumerate(state.requests)]
        logits = engine.step(entries + [StepEntry((state.key, "portion"), given["portion"], [case["tokens"] - 1])])
        engine.release((state.key, "portion"))
        state.done += 1
        return logits
    state.room_for(case["steps"])
    for k in range(case["steps"]):
        last = k == case["steps"] - 1
        logits = engine.step([StepEntry(r, [given["fed"][i][state.done]], [0] if last and i in wanted else [])
                              for i, r in enumerate(state.requests)])
        state.done += 1
    return logits


# ---- bounds ----------------------------------------------------------------------------------------------------------
def _sizes(name):
    """(matrix elements every token is multiplied with, the output matrix's, cached elements per token, flops per token and
    earlier token seen, float32 state elements per request, the width, window of half the layers)"""
    c = MODELS[name][0]
    if "architectures" in c:
        w, d = c["hidden_size"], c["head_dim"]
        q, kv, layers = c["num_attention_heads"] * d, c["num_key_value_heads"] * d, c["num_hidden_layers"]
        per_layer = w * (q + 2 * kv) + q * w + 3 * w * c["intermediate_size"]
        return layers * per_layer, c["vocab_size"] * w, layers * 2 * kv, layers * 4 * q, 0, w, 0
    w = c["width"]
    if c["architecture"] == "Noditar":
        latent = w * (2048 + 512 + 2048 + 2048) + 2 * 512 * 2048
        att = w * (2048 * 3 + 2 * 512)
        ssm = w * (10304 + 4096)
        # a state-space layer's 64 heads of 128 x 64: update and readout, 4 flops an element and token
        return latent + att + 2 * ssm + 3 * 3 * w * 8192, 32768 * w, 512 + 2 * 512, 2 * 4 * 2048, 2 * 64 * 128 * 64, w, 0
    att = w * (3 * 2048 + 512)
    both = w * (2 * 2048 + 2 * 512 + 4 * 2048)
    return 2 * att + 2 * both + 4 * 2 * w * 8192 + 2 * w * w, 32768 * w, 2 * 512 + 2 * 2 * 512, 4 * 4 * 2048, 2 * 2048, w, 1024


def _seen(window, start, n):
    """Pairs of a token at positions start .. start + n - 1 and an earlier one (or itself) it attends to."""
    if not window:
        return n * start + n * (n + 1) // 2
    return sum(min(p + 1, window) for p in range(start, start + n))


def work(case):
    size = 4 if MODELS[case["model"]][2] == "float32" else 2
    body, head, cache, pair, state, width, window = _sizes(case["model"])
    vocab = head // width

    def step(portions, wanted):
        """One pass over the weights for portions of n tokens behind start cached ones."""
        tokens = sum(n for _, n in portions)
        held = sum((min(start, window) if window else start) + n for start, n in portions)
        return (size * (body + (head if wanted else 0) + cache * held) + 8 * state * len(portions) + 4 * wanted * vocab,
                2 * tokens * body + 2 * wanted * head + pair * sum(_seen(window, s, n) for s, n in portions) + 4 * state * tokens)

    parts = []
    if case["kind"] == "prompt":
        parts = [step([(0, case["tokens"])], 1)]
    elif case["kind"] == "chat":
        lengths = [int(n) for n in case["prompts"].split(",")]
        parts = [step([(0, n) for n in lengths], len(lengths))]
        parts += [step([(n + k, 1) for n in lengths], len(lengths)) for k in range(case["new"])]
    elif case["kind"] == "mixed":
        parts = [step([(case["prefix"], 1)] * case["batch"] + [(0, case["tokens"])], min(WANTED, case["batch"]) + 1)]
    else:
        for k in range(case["steps"]):
            last = k == case["steps"] - 1
            parts.append(step([(case["prefix"] + k, 1)] * case["batch"], min(WANTED, case["batch"]) if last else 0))
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


def tolerance(case):
    return {"qwen3-8b-8": {"rel": 0.03}, "qwen3-0.6b": {"rel": 0.03}, "qwen3-0.6b-fp32": {"rel": 2e-5},
            "qwen3-tiny-b": {"rel": 1e-5, "differ": 0.0}, "noditar-2k": {"rel": 0.03}, "vokepel-2k": {"rel": 0.03}}[case["model"]]


# ---- the same results in 64 bits -------------------------------------------------------------------------------------
F64 = torch.float64


def _signed(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _mix64(z):
    """The finaliser of splitmix64, on Python integers."""
    m = (1 << 64) - 1
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _mix64_tensor(z):
    shift = lambda v, n: (v >> n) & ((1 << (64 - n)) - 1)
    z = (z ^ shift(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ shift(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ shift(z, 31)


class _Weights:
    """Tensors of a model by name: the documented generator (splitmix64 words keyed by the seed and the FNV-1a hash of
    the name, Box-Muller's cosine branch), rounded to what the model stores."""

    def __init__(self, name):
        _, self.seed, dtype, self.std, self.low, self.high = MODELS[name][:6]
        self.matrix = torch.bfloat16 if dtype == "bfloat16" else torch.float32

    def _words(self, key, first, n, k):
        i = torch.arange(first, first + n, dtype=torch.int64, device="cuda")
        word = _mix64_tensor((2 * i + (k + 1)) * _signed(0x9E3779B97F4A7C15) + _signed(key))
        return (word >> 11) & ((1 << 53) - 1)

    def _fill(self, name, shape, dtype, scale):
        h = 0xCBF29CE484222325
        for b in name.encode():
            h = ((h ^ b) * 0x100000001B3) & ((1 << 64) - 1)
        key = _mix64(_mix64((self.seed + 0x9E3779B97F4A7C15) & ((1 << 64) - 1)) ^ h)
        n, out = math.prod(shape), []
        if scale and self.low == self.high:
            return torch.full(shape, self.low, dtype=F64, device="cuda")
        for first in range(0, n, 1 << 26):
            m = min(1 << 26, n - first)
            if scale:
                v = self.low + (self.high - self.low) * (self._words(key, first, m, 0).to(F64) * 2.0 ** -53)
            else:
                r = torch.sqrt(-2.0 * torch.log((self._words(key, first, m, 0) + 1).to(F64) * 2.0 ** -53))
                v = r * torch.cos(2.0 * math.pi * (self._words(key, first, m, 1).to(F64) * 2.0 ** -53)) * self.std
            out.append(v.to(torch.float32).to(dtype))
        return torch.cat(out).view(*shape)

    def __call__(self, name, *shape):
        """A matrix."""
        return self._fill(name, shape, self.matrix, False).to(F64)

    def stored(self, name, *shape):
        return self._fill(name, shape, self.matrix, False)

    def vector(self, name, *shape):
        return self._fill(name, shape, torch.float32, False).to(F64)

    def scale(self, name, *shape):
        return self._fill(name, shape, torch.float32, True).to(F64)


def _rms(x, eps, w=1.0):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps) * w


def _seen_mask(n, window=0):
    i = torch.arange(n, device="cuda")
    d = i[:, None] - i[None, :]
    return (d >= 0) & ((d < window) if window else True)


def _softmax_rows(s, seen, extra=None):
    """Softmax over the keys a row sees; ``extra`` is one more score that has no value."""
    s = s.masked_fill(~seen, float("-inf"))
    top = s.amax(dim=-1, keepdim=True)
    if extra is not None:
        top = torch.clamp(top, min=extra)
    e = torch.exp(s - top)
    return e / (e.sum(dim=-1, keepdim=True) + (torch.exp(extra - top) if extra is not None else 0.0))


def _turns(n, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)
    a = torch.arange(n, dtype=F64, device="cuda")[:, None] * f[None, :]
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _qwen3(c, w, xs):
    """Hidden states behind the last norm for every sequence of embedded tokens ``xs``, layer by layer."""
    E, D, eps = c["hidden_size"], c["head_dim"], c["rms_norm_eps"]
    HQ, HKV, FF = c["num_attention_heads"], c["num_key_value_heads"], c["intermediate_size"]
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        wq, wk, wv = (w(f"{p}self_attn.{n}_proj.weight", h * D, E) for n, h in (("q", HQ), ("k", HKV), ("v", HKV)))
        wo = w(p + "self_attn.o_proj.weight", E, HQ * D)
        wg, wu, wd = w(p + "mlp.gate_proj.weight", FF, E), w(p + "mlp.up_proj.weight", FF, E), w(p + "mlp.down_proj.weight", E, FF)
        n1, n2 = w.scale(p + "input_layernorm.weight", E), w.scale(p + "post_attention_layernorm.weight", E)
        nq, nk = w.scale(p + "self_attn.q_norm.weight", D), w.scale(p + "self_attn.k_norm.weight", D)
        for s, x in enumerate(xs):
            n, h = x.shape[0], _rms(x, eps, n1)
            cos, sin = _turns(n, D, c["rope_theta"])
            turn = lambda v: torch.cat([v[..., :D // 2] * cos - v[..., D // 2:] * sin, v[..., :D // 2] * sin + v[..., D // 2:] * cos], dim=-1)
            q = turn(_rms((h @ wq.T).view(n, HQ, D), eps, nq))
            k = turn(_rms((h @ wk.T).view(n, HKV, D), eps, nk))
            v, seen = (h @ wv.T).view(n, HKV, D), _seen_mask(n)
            o = torch.stack([_softmax_rows(q[:, a] @ k[:, a * HKV // HQ].T * D ** -0.5, seen) @ v[:, a * HKV // HQ] for a in range(HQ)], dim=1)
            x = x + o.reshape(n, HQ * D) @ wo.T
            h = _rms(x, eps, n2)
            g = h @ wg.T
            xs[s] = x + (g * torch.sigmoid(g) * (h @ wu.T)) @ wd.T
    final = w.scale("model.norm.weight", E)
    return [_rms(x, eps, final) for x in xs]


def _noditar_mixer(kind, m, w, p, h, eps):
    n, E = h.shape
    if kind == "mamba2":
        H, P, N, G, K = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
        inner = H * P
        u = h @ w(p + "in", 2 * inner + 2 * G * N + H, E).T
        z, xbc, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
        taps, pad = w.vector(p + "conv", inner + 2 * G * N, K), torch.cat([xbc.new_zeros(K - 1, xbc.shape[1]), xbc])
        xbc = torch.nn.functional.silu(w.vector(p + "conv.b", inner + 2 * G * N) + sum(taps[:, j] * pad[j:j + n] for j in range(K)))
        x = xbc[:, :inner].reshape(n, H, P)
        B, C = (xbc[:, inner + j * G * N:inner + (j + 1) * G * N].reshape(n, G, N).repeat_interleave(H // G, dim=1) for j in (0, 1))
        dt = torch.nn.functional.softplus(dt + w.vector(p + "dt_bias", H), threshold=60.0)
        decay = torch.exp(-torch.exp(w.vector(p + "A_log", H)) * dt)
        S, y, dx = x.new_zeros(H, N, P), torch.empty_like(x), dt[:, :, None] * x
        for t in range(n):
            S = torch.baddbmm(decay[t][:, None, None] * S, B[t][:, :, None], dx[t][:, None, :])
            y[t] = torch.bmm(C[t][:, None, :], S)[:, 0]
        y = (y + w.scale(p + "D", H)[:, None] * x).reshape(n, inner) * torch.nn.functional.silu(z)
        y = _rms(y.view(n, m["norm_groups"], -1), eps).reshape(n, inner) * w.scale(p + "norm", inner)
        return y @ w(p + "o", E, inner).T
    H, D, V, seen = m["heads"], m["dim"], m["vdim"], _seen_mask(n)
    q = (h @ w(p + "q", H * D, E).T).view(n, H, D)
    if kind == "latent_attention":
        R, G = m["kv_rank"], H
        c = _rms(h @ w(p + "dkv", R, E).T, eps, w.scale(p + "dkv.norm", R))
        k, v = (c @ w(p + "uk", H * D, R).T).view(n, H, D), (c @ w(p + "uv", H * V, R).T).view(n, H, V)
        slopes, extra = [0.0] * H, None
    else:
        G = m["kv_heads"]
        q, k = _rms(q, eps), _rms((h @ w(p + "k", G * D, E).T).view(n, G, D), eps)
        v = (h @ w(p + "v", G * V, E).T).view(n, G, V)
        slopes, extra = [2.0 ** (-8.0 * (a + 1) / H) for a in range(H)], torch.zeros((), dtype=F64, device="cuda")
    i = torch.arange(n, dtype=F64, device="cuda")
    far = i[:, None] - i[None, :]
    o = torch.stack([_softmax_rows(q[:, a] @ k[:, a * G // H].T * m["scale"] - slopes[a] * far, seen, extra) @ v[:, a * G // H]
                     for a in range(H)], dim=1).reshape(n, H * V)
    return (o * torch.sigmoid(h @ w(p + "g", H * V, E).T)) @ w(p + "o", E, H * V).T


def _noditar_hidden(c, w, xs):
    E, S, eps, out = c["width"], c["streams"], c["norm"]["eps"], []
    for x in xs:
        X = torch.stack([x] * S)
        for i, layer in enumerate(c["layers"]):
            for part in (1, 2) if layer.get("mlp") else (1,):
                p = f"l{i}."
                h = _rms(torch.tensordot(w.scale(f"{p}hc{part}.in", S), X, dims=1), eps, w.scale(f"{p}norm{part}", E))
                if part == 1:
                    y = _noditar_mixer(layer["type"], layer["mixer"], w, p + "mix.", h, eps)
                else:
                    ff, limit = layer["mlp"]["ff"], layer["mlp"]["limit"]
                    g = torch.clamp(h @ w(p + "mlp.gate", ff, E).T, max=limit)
                    u = torch.clamp(h @ w(p + "mlp.up", ff, E).T, -limit, limit)
                    y = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "mlp.down", E, ff).T
                X = torch.tensordot(w.vector(f"{p}hc{part}.mix", S, S).T, X, dims=1) + w.scale(f"{p}hc{part}.out", S)[:, None, None] * y
        out.append(_rms(X.sum(dim=0), eps, w.scale("final.norm", E)))
    return out


def _vokepel_mixer(layer, w, p, h, eps):
    n, E = h.shape
    m = layer["mixer"]
    if layer["type"] == "attention":
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k = h @ w(p + "q", H * D, E).T, h @ w(p + "k", G * D, E).T
        v = k.view(n, G, D).repeat_interleave(H // G, dim=1)
        q = _rms(q, eps, w.scale(p + "q.norm", H * D)).view(n, H, D)
        k = _rms(k, eps, w.scale(p + "k.norm", G * D)).view(n, G, D).repeat_interleave(H // G, dim=1)
        s = torch.einsum("ihd,jhd->hij", q, k) * m["scale"]
        s = m["softcap"] * torch.tanh(s / m["softcap"])
        i = torch.arange(n, dtype=F64, device="cuda")
        far = torch.clamp(i[:, None] - i[None, :], min=0.0)
        s = s - w.vector(p + "r1", H)[:, None, None] * torch.log1p(w.scale(p + "r2", H)[:, None, None] * far)
        s = torch.einsum("hg,gij->hij", w.vector(p + "talk", H, H), s)
        o = torch.einsum("hij,jhd->ihd", _softmax_rows(s, _seen_mask(n, m["mask"]["size"])), v).reshape(n, H * D)
        return (o * torch.sigmoid(h @ w(p + "g", H * D, E).T)) @ w(p + "o", E, H * D).T
    a = m["left"]
    H, G, D, W = a["heads"], a["kv_heads"], a["dim"], m["right"]["width"]
    cos, sin = _turns(n, a["rot"]["dims"], a["rot"]["base"])
    turn = lambda v: torch.stack([v[..., 0::2] * cos - v[..., 1::2] * sin, v[..., 1::2] * cos + v[..., 0::2] * sin], dim=-1).flatten(-2)
    q = turn((h @ w(p + "left.q", H * D, E).T).view(n, H, D))
    k = turn((h @ w(p + "left.k", G * D, E).T).view(n, G, D)).repeat_interleave(H // G, dim=1)
    v = (h @ w(p + "left.v", G * D, E).T).view(n, G, D).repeat_interleave(H // G, dim=1)
    s = torch.einsum("ihd,jhd->hij", q, k) * a["scale"]
    pr = _softmax_rows(s, _seen_mask(n, a["mask"]["size"]), w.vector(p + "left.sink", H)[:, None, None])
    left = torch.einsum("hij,jhd->ihd", pr, v).reshape(n, H * D) @ w(p + "left.o", E, H * D).T
    r = p + "right."
    z = torch.sigmoid(h @ w(r + "z", W, E).T + w.vector(r + "z.b", W))
    u = h @ w(r + "x", W, E).T + w.vector(r + "x.b", W)
    c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
    S, states = z.new_zeros(W), torch.empty_like(z)
    for t in range(n):
        S = (1.0 - z[t]) * S + z[t] * c[t]
        states[t] = S
    right = (states * torch.nn.functional.silu(h @ w(r + "g", W, E).T)) @ w(r + "o", E, W).T
    return m["left_scale"] * left + m["right_scale"] * right


def _vokepel_hidden(c, w, xs):
    E, eps, mult, out = c["width"], c["norm"]["eps"], c["residual_mult"], []
    for e in xs:
        x = e
        for i, layer in enumerate(c["layers"]):
            if i == c["loop"]["start"]:
                x = torch.cat([x, e], dim=-1) @ w("loop.in", E, 2 * E).T + w.vector("loop.step", 1, E)[0]
            p, ff = f"l{i}.", layer["mlp"]["ff"]
            x = x + mult * _vokepel_mixer(layer, w, p + "mix.", _rms(x, eps, w.scale(p + "norm1", E)), eps)
            h = torch.relu(_rms(x, eps, w.scale(p + "norm2", E)) @ w(p + "mlp.up", ff, E).T) ** 2
            x = x + mult * (h @ w(p + "mlp.down", E, ff).T)
        out.append(_rms(x, eps, w.scale("final.norm", E)))
    return out


def _logits(name, sequences):
    """Float64 logits behind the last token of every sequence of ids."""
    c, w = MODELS[name][0], _Weights(name)
    table_name = "model.embed_tokens.weight" if "architectures" in c else "embed"
    vocab, width = c.get("vocab_size") or c["vocab"], c.get("hidden_size") or c["width"]
    table = w.stored(table_name, vocab, width)
    xs = [table[torch.tensor(s, device="cuda")].to(F64) for s in sequences]
    if "architectures" in c:
        hidden = _qwen3(c, w, xs)
        head = table if c["tie_word_embeddings"] else w.stored("lm_head.weight", vocab, width)
    elif c["architecture"] == "Noditar":
        hidden, head = _noditar_hidden(c, w, xs), w.stored("head", vocab, width)
    else:
        hidden, head = _vokepel_hidden(c, w, xs), table
    last = torch.stack([h[-1] for h in hidden])
    y = torch.cat([last @ part.to(F64).T for part in head.split(16384)], dim=1)
    if c.get("architecture") == "Vokepel":
        y = c["logit_softcap"] * torch.tanh(y * c["logit_scale"] / c["logit_softcap"])
    return y.cpu().numpy()


def exact(case, seed):
    given, name = _inputs(case, seed), case["model"]
    if case["kind"] == "prompt":
        return _logits(name, given["prompts"])[0]
    if case["kind"] == "chat":
        sequences = [list(p) for p in given["prompts"]]
        for _ in range(case["new"]):
            for s, row in zip(sequences, _logits(name, sequences)):
                s.append(int(row.argmax()))
        tokens = np.array([s[-case["new"]:] for s in sequences])
        return {"tokens": tokens, "logits": _logits(name, sequences)}
    steps = case.get("steps", 1)
    sequences = [given["prefixes"][i] + given["fed"][i][:steps] for i in given["wanted"]]
    if case["kind"] == "mixed":
        sequences.append(given["portion"])
    return _logits(name, sequences)
