"""The work that programs have this library do, as cases to measure.

A case is a request (or a batch of requests) as a serving program, a chat program or a scoring job sends it: the
prompts go through one ``Engine.step``, then every sequence goes on one token a step, and the slots go back. The
tokens of the later steps are given (as in a trace replay), so that the logits of every step can be compared. Other
cases choose tokens from logits, and generate with ``Engine.generate``. Weights and token ids are random, made from
the seed: ids are uniform, weights normal (``_std``).

``exact`` is a plain 64-bit implementation of the two designs used here, with no code of this library.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from sleuth_b200.engine.engine import Engine
from sleuth_b200.sampling.config import SamplingConfig
from sleuth_b200.sampling.sampler import Sampler

DEVICE = "cuda:0"


def _qwen3(hidden, layers, heads, kv_heads, head_dim, inter, vocab=151936, tied=True, theta=1e6, eps=1e-6, bias=False, positions=40960):
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "vocab_size": vocab, "hidden_size": hidden,
            "intermediate_size": inter, "num_hidden_layers": layers, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": head_dim, "rope_theta": theta, "rms_norm_eps": eps,
            "attention_bias": bias, "tie_word_embeddings": tied, "max_position_embeddings": positions}


def _lezepel(width, layers, heads, dim, rot, vdim, q_rank, kv_rank, experts, top, ff, vocab=32768):
    mixer = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": q_rank, "kv_rank": kv_rank,
             "scale": (dim + rot) ** -0.5, "rot": {"base": 10000.0, "dims": rot}}
    moe = {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": experts, "top": top}}
    block = [{"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": top * ff}}]
    block += [{"type": "latent_attention", "mixer": mixer, "mlp": moe} for _ in range(layers - 1)]
    return {"architecture": "Lezepel", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": 16.0},
            "layers": block, "loop": {"start": 1, "stop": 2, "times": 1}}


# The sizes that the benchmark and the tests of this library use.
MODELS = {
    "tiny": _qwen3(96, 3, 6, 3, 24, 160, vocab=503, tied=False, eps=1e-5, bias=True, positions=256),
    "0.6b": _qwen3(1024, 28, 16, 8, 128, 3072),
    "4b": _qwen3(2560, 36, 32, 8, 128, 9728),
    "8b": _qwen3(4096, 36, 32, 8, 128, 12288, tied=False),
    "latent-1024": _lezepel(1024, 8, 16, 64, 32, 64, 384, 256, 16, 4, 768),
    "latent-2048": _lezepel(2048, 6, 16, 128, 64, 128, 768, 512, 64, 6, 1408),
}




def _std(cfg):
    """Standard deviation of the random weights: 0.02 at width 1,024, less for wider models, so that the layers' results
    stay in the same proportion to the stream. With routed experts half of that, and a larger embedding scale: a close call
    between two experts that bfloat16 rounding turns then moves a row of logits by a few per cent and not by a quarter."""
    if cfg.get("architecture") == "Lezepel":
        return 0.32 / math.sqrt(cfg["width"])
    return min(0.02, 0.64 / math.sqrt(cfg["hidden_size"]))


def listed():
    return [
        # A test-sized model in float32, as a continuous-integration job runs it: greedy generation for four short
        # prompts, then the logits of every position of what came out. Launches and host work are all there is.
        dict(name="tiny-fp32-generate", kind="generate", model="tiny", dtype="fp32", batch=4, lo=1, hi=40, steps=12),
        # One user's chat: two turns, the second appended to the first, a few words of answer each.
        dict(name="0.6b-chat", kind="serve", model="0.6b", dtype="bf16", batch=1, lo=180, hi=180, turns=2, steps=16),
        # The headline workload of the benchmark: eight long prompts, then single tokens at that context.
        dict(name="0.6b-batch8-2048", kind="serve", model="0.6b", dtype="bf16", batch=8, lo=2048, hi=2048, turns=1, steps=40),
        # A busy server with short requests: 64 at once, of unequal lengths.
        dict(name="0.6b-batch64", kind="serve", model="0.6b", dtype="bf16", batch=64, lo=32, hi=512, turns=1, steps=24),
        # Reading one document: the prompt alone (first-token latency).
        dict(name="0.6b-prompt2048", kind="serve", model="0.6b", dtype="bf16", batch=1, lo=2048, hi=2048, turns=1, steps=0),
        # A larger model with ragged long prompts (the second benchmark configuration, fewer steps).
        dict(name="4b-ragged16", kind="serve", model="4b", dtype="bf16", batch=16, lo=64, hi=2048, turns=1, steps=16),
        # The largest model of the benchmark, a full batch of short prompts, mostly single-token steps.
        dict(name="8b-batch64", kind="serve", model="8b", dtype="bf16", batch=64, lo=32, hi=192, turns=1, steps=32),
        # The true 32-bit path, whole prompt (reference logits for a comparison).
        dict(name="0.6b-fp32-prompt", kind="serve", model="0.6b", dtype="fp32", batch=1, lo=1500, hi=1500, turns=1, steps=0),
        # The true 32-bit path, a small batch that goes on token by token.
        dict(name="0.6b-fp32-batch8", kind="serve", model="0.6b", dtype="fp32", batch=8, lo=100, hi=700, turns=1, steps=24),
        # Attention through latents with routed experts: a document and an answer.
        dict(name="latent-1024-prompt", kind="serve", model="latent-1024", dtype="bf16", batch=1, lo=2048, hi=2048, turns=1, steps=16),
        # The same design at the larger size, eight users.
        dict(name="latent-2048-batch8", kind="serve", model="latent-2048", dtype="bf16", batch=8, lo=64, hi=768, turns=1, steps=32),
        # Choosing the next tokens of a full batch with the options of a chat server.
        dict(name="sample-64", kind="sample", rows=64, vocab=151936, temperature=0.8, top_k=50, top_p=0.9, min_p=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# What a drawn request may cost at most for each model and dtype: prompt tokens of all sequences together, steps.
_MOST = {("0.6b", "bf16"): (16384, 40), ("4b", "bf16"): (16384, 16), ("8b", "bf16"): (7000, 24), ("0.6b", "fp32"): (3500, 24),
         ("latent-1024", "bf16"): (16384, 32), ("latent-2048", "bf16"): (8192, 32)}


def draw(rng):
    kind = rng.choice(["serve"] * 9 + ["generate", "sample"])
    if kind == "generate":
        return dict(kind="generate", model="tiny", dtype="fp32", batch=rng.randint(1, 8), lo=rng.randint(1, 8), hi=rng.randint(8, 120), steps=rng.randint(4, 24))
    if kind == "sample":
        form = rng.randrange(3)
        return dict(kind="sample", rows=_log_int(rng, 1, 64), vocab=rng.choice([151936, 32768, 50257]), temperature=round(rng.uniform(0.5, 1.2), 2),
                    top_k=_log_int(rng, 5, 400) if form < 2 else 0, top_p=round(rng.uniform(0.7, 0.98), 2) if form > 0 else 1.0, min_p=0.05 if form == 0 else 0.0)
    model, dtype = rng.choice([("0.6b", "bf16")] * 4 + [("0.6b", "fp32")] * 2 + [("4b", "bf16"), ("8b", "bf16"), ("latent-1024", "bf16"), ("latent-2048", "bf16")])
    tokens, steps = _MOST[model, dtype]
    batch = _log_int(rng, 1, 64 if dtype == "bf16" else 16)
    turns = rng.choice([1, 1, 1, 2])
    hi = _log_int(rng, 16, max(17, min(3000, tokens // (batch * turns))))
    return dict(kind="serve", model=model, dtype=dtype, batch=batch, lo=max(1, hi // rng.choice([1, 2, 8])), hi=hi, turns=turns, steps=rng.randint(0 if hi > 64 else 4, steps // turns))


# ------------------------------------------------------------------ requests ----

def _requests(case, seed):
    """Per turn: the portions of all sequences (lists of token ids) and the tokens of the steps that follow [steps, batch].
    The seed makes the tokens; the lengths belong to the case."""
    rng, shape = np.random.default_rng(seed), np.random.default_rng(1)
    vocab = MODELS[case["model"]].get("vocab_size") or MODELS[case["model"]]["vocab"]
    out = []
    for _ in range(case.get("turns", 1)):
        lens = shape.integers(case["lo"], case["hi"] + 1, case["batch"])
        portions = [rng.integers(0, vocab, int(n)).tolist() for n in lens]
        out.append((portions, rng.integers(0, vocab, (case["steps"], case["batch"])).tolist()))
    return out


def _engine(case, seed):
    longest = min(case.get("turns", 1) * (case["hi"] + case["steps"]), MODELS[case["model"]].get("max_position_embeddings", 1 << 20))
    return Engine.from_config(MODELS[case["model"]], seed=seed, dtype=case["dtype"], std=_std(MODELS[case["model"]]), max_seq_len=longest,
                              max_tokens=case["batch"] * (-(-longest // 64) * 64), max_sequences=case["batch"] + 1, device=DEVICE)


def prepare(case, seed):
    """What the program holds before the call: the loaded model and its cache, warmed up as a server is by running the
    request's shape (other tokens) twice, and the request. For ``sample``: the logits of a step and the sampler."""
    if case["kind"] == "sample":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)
        logits = torch.randn((case["rows"], case["vocab"]), generator=gen, device=DEVICE) * 2.5
        cfg = SamplingConfig(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"])
        uniforms = np.random.default_rng(seed).random(case["rows"], dtype=np.float32)
        return dict(case=case, sampler=Sampler(DEVICE, case["vocab"]), logits=logits, cfg=cfg, uniforms=uniforms)
    state = dict(case=case, engine=_engine(case, seed), turns=_requests(case, seed))
    if case["kind"] == "serve":
        vocab = state["engine"].vocab
        state["logits"] = [(torch.empty((case["batch"], vocab), device=DEVICE), torch.empty((case["steps"], case["batch"], vocab), device=DEVICE))
                           for _ in state["turns"]]
    shape = [([[(t * 7 + 1) % 500 for t in p] for p in portions], [[(t * 7 + 1) % 500 for t in row] for row in steps]) for portions, steps in state["turns"]]
    for _ in range(2):
        run(dict(state, turns=shape))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return state["sampler"].choose(state["logits"], state["cfg"], state["uniforms"])
    engine = state["engine"]
    if case["kind"] == "generate":
        prompts = state["turns"][0][0]
        results = engine.generate(prompts, max_new_tokens=case["steps"], sampling=SamplingConfig(temperature=0.0), stop_ids=())
        texts = [p + r.new_ids for p, r in zip(prompts, results)]
        slots = engine.open(len(texts))
        logits = engine.step([(s, t, tuple(range(len(t)))) for s, t in zip(slots, texts)])
        engine.close(slots)
        return {"tokens": np.asarray([r.new_ids for r in results], dtype=np.int64), "logits": logits}
    slots = engine.open(case["batch"])
    for (portions, steps), (first, later) in zip(state["turns"], state["logits"]):
        first.copy_(engine.step([(s, p, (len(p) - 1,)) for s, p in zip(slots, portions)]))
        for k, row in enumerate(steps):
            later[k].copy_(engine.step([(s, (t,), (0,)) for s, t in zip(slots, row)]))
    engine.close(slots)
    return state["logits"]


# ------------------------------------------------------------------ what a pass cannot do without ----

def _sizes(cfg):
    """Numbers that count work: parameters read by every token's layers (dense), per-expert parameters and their counts,
    head parameters, cache values a token, attention multiply-adds per head pair of positions."""
    if cfg.get("architecture") == "Lezepel":
        m, d = cfg["layers"][0]["mixer"], cfg["width"]
        H, dk = m["heads"], m["dim"] + m["rot_dim"]
        mixer = (d * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + H * m["vdim"]) + m["q_rank"] * H * dk
                 + m["kv_rank"] * H * (m["dim"] + m["vdim"]) + H * m["vdim"] * d)
        dense, experts = 0, []
        for L in cfg["layers"]:
            f = L["mlp"]
            dense += mixer
            if f["kind"] == "dense":
                dense += 3 * d * f["ff"]
            else:
                dense += f["router"]["experts"] * d
                experts.append((f["router"]["experts"], f["router"]["top"], 3 * d * f["expert"]["ff"]))
        n = len(cfg["layers"])
        return dense, experts, cfg["vocab"] * d, n * (m["kv_rank"] + m["rot_dim"]), n * H * (dk + m["vdim"])
    d, n, H, K, hd = (cfg[k] for k in ("hidden_size", "num_hidden_layers", "num_attention_heads", "num_key_value_heads", "head_dim"))
    dense = n * (d * hd * (2 * H + 2 * K) + 3 * d * cfg["intermediate_size"])
    return dense, [], cfg["vocab_size"] * d, 2 * n * K * hd, 2 * n * H * hd


def _step_work(cfg, size, past, counts, wanted, vocab):
    """(bytes, flops) of one step: weights read once, the cache read and appended to, logits written."""
    dense, experts, head, kv, att = _sizes(cfg)
    T = sum(counts)
    weights, flops = dense + head, 2.0 * (dense * T + head * wanted)
    for e, top, params in experts:
        weights += params * e * (1.0 - (1.0 - top / e) ** T)        # the experts that T tokens are expected to touch
        flops += 2.0 * params * top * T
    pairs = sum(p * c + c * (c + 1) / 2.0 for p, c in zip(past, counts))
    nbytes = size * (weights + kv * (sum(past) + T)) + 4.0 * wanted * vocab
    return nbytes, flops + 2.0 * att * pairs


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    cfg = MODELS[case["model"]]
    size = 4 if case["dtype"] == "fp32" else 2
    n, vocab = case["batch"], cfg.get("vocab_size") or cfg["vocab"]
    past, total = [0] * n, np.zeros(2)
    mean = (case["lo"] + case["hi"]) / 2.0
    for _ in range(case.get("turns", 1)):
        total += _step_work(cfg, size, past, [mean] * n, n, vocab)
        past = [p + mean for p in past]
        for _ in range(case["steps"]):
            total += _step_work(cfg, size, past, [1] * n, n, vocab)
            past = [p + 1 for p in past]
    if case["kind"] == "generate":
        total += _step_work(cfg, size, [0] * n, [mean + case["steps"]] * n, n * (mean + case["steps"]), vocab)
    return {"bytes": float(total[0]), "flops": float(total[1])}


def tolerance(case):
    # Measured against ``exact`` on a B200: 2.3e-6 (0.6B sizes, 32-bit), 0.0065 (0.6B), 0.008 (4B), 0.011 (8B), 0.002 to
    # 0.015 with routed experts, where now and then a close call between two experts falls the other way. About four
    # times that for the 32-bit and dense cases. Sampled tokens may differ where a draw falls on the edge of two tokens.
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 0.025, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits ----

def _weights(names, seed, dtype, std):
    """The tensors that ``Engine.from_config`` draws for a seed, by checkpoint name. names: {name: (shape, what)}, what =
    "matrix" (held in the run's dtype), "gain" (1 + draw, 32-bit), "vector" (32-bit)."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed))
    out = {}
    for name, (shape, what) in sorted(names.items()):
        t = torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32) * std
        if what == "gain":
            t += 1.0
        if dtype == "bf16" and (what == "matrix" or len(shape) >= 2):
            t = t.to(torch.bfloat16)
        out[name] = t
    return out


def _rms(x, gain, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _attend(q, k, v, starts, scale):
    """Causal attention inside each sequence; q, k [T, heads, dk], v [T, heads, dv]."""
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=q.dtype, device=q.device)
    for a, b in zip(starts[:-1], starts[1:]):
        mask = torch.ones((b - a, b - a), dtype=torch.bool, device=q.device).tril()
        for h in range(0, q.shape[1], 4):
            s = torch.einsum("ihd,jhd->hij", q[a:b, h:h + 4], k[a:b, h:h + 4]) * scale
            p = torch.softmax(s.masked_fill_(~mask, float("-inf")), dim=-1)
            out[a:b, h:h + 4] = torch.einsum("hij,jhd->ihd", p, v[a:b, h:h + 4])
    return out


def _turn(x, cos, sin):
    """Rotation of channel i with channel i + half, [T, heads, n]; cos, sin [T, half]."""
    half = cos.shape[1]
    a, b = x[..., :half], x[..., half:2 * half]
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], -1)


def _tables(pos, n, theta):
    """The design fixes the angles to those formed in 32 bits, position by frequency."""
    freq = 1.0 / (theta ** (torch.arange(0, n, 2, dtype=torch.float32) / n))
    ang = torch.outer(torch.arange(int(pos.max()) + 1, dtype=torch.float32), freq)
    return ang.cos().to(DEVICE, torch.float64)[pos], ang.sin().to(DEVICE, torch.float64)[pos]


def _names_qwen3(c):
    d, H, K, hd, ff = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["intermediate_size"]
    names = {"model.embed_tokens.weight": ((c["vocab_size"], d), "matrix"), "model.norm.weight": ((d,), "gain")}
    if not c["tie_word_embeddings"]:
        names["lm_head.weight"] = ((c["vocab_size"], d), "matrix")
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for n, rows in (("q_proj", H * hd), ("k_proj", K * hd), ("v_proj", K * hd)):
            names[p + f"self_attn.{n}.weight"] = ((rows, d), "matrix")
            if c["attention_bias"]:
                names[p + f"self_attn.{n}.bias"] = ((rows,), "vector")
        names[p + "self_attn.o_proj.weight"] = ((d, H * hd), "matrix")
        for n in ("q_norm", "k_norm"):
            names[p + f"self_attn.{n}.weight"] = ((hd,), "gain")
        for n in ("input_layernorm", "post_attention_layernorm"):
            names[p + f"{n}.weight"] = ((d,), "gain")
        for n, shape in (("gate_proj", (ff, d)), ("up_proj", (ff, d)), ("down_proj", (d, ff))):
            names[p + f"mlp.{n}.weight"] = (shape, "matrix")
    return names


def _forward_qwen3(c, w, ids, pos, starts, rows):
    H, K, hd, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    cos, sin = _tables(pos, hd, c["rope_theta"])
    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(c["num_hidden_layers"]):
        def g(name):
            t = w.get(f"model.layers.{i}.{name}")
            return None if t is None else t.double()

        def product(h, name):
            y = h @ g(name + ".weight").T
            bias = g(name + ".bias")
            return y if bias is None else y + bias

        h = _rms(x, g("input_layernorm.weight"), eps)
        q = product(h, "self_attn.q_proj").view(-1, H, hd)
        k = product(h, "self_attn.k_proj").view(-1, K, hd)
        v = product(h, "self_attn.v_proj").view(-1, K, hd)
        q = _turn(_rms(q, g("self_attn.q_norm.weight"), eps), cos, sin)
        k = _turn(_rms(k, g("self_attn.k_norm.weight"), eps), cos, sin)
        y = _attend(q, k.repeat_interleave(H // K, 1), v.repeat_interleave(H // K, 1), starts, hd ** -0.5)
        x = x + product(y.reshape(len(ids), H * hd), "self_attn.o_proj")
        h = _rms(x, g("post_attention_layernorm.weight"), eps)
        x = x + product(torch.nn.functional.silu(product(h, "mlp.gate_proj")) * product(h, "mlp.up_proj"), "mlp.down_proj")
    head = w["model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight"]
    return _rms(x[rows], w["model.norm.weight"].double(), eps) @ head.double().T


def _names_lezepel(c):
    d = c["width"]
    names = {"embed": ((c["vocab"], d), "matrix"), "head": ((c["vocab"], d), "matrix"), "final.norm": ((d,), "gain"),
             "loop.step": ((c["loop"]["times"], d), "vector")}
    for i, L in enumerate(c["layers"]):
        m, f, p = L["mixer"], L["mlp"], f"l{i}."
        H = m["heads"]
        names[p + "norm1"] = ((d,), "gain")
        for n, shape in (("dq", (m["q_rank"], d)), ("uq", (H * (m["dim"] + m["rot_dim"]), m["q_rank"])), ("dkv", (m["kv_rank"] + m["rot_dim"], d)),
                         ("uk", (H * m["dim"], m["kv_rank"])), ("uv", (H * m["vdim"], m["kv_rank"])), ("g", (H * m["vdim"], d)), ("o", (d, H * m["vdim"]))):
            names[p + "mix." + n] = (shape, "matrix")
        names[p + "mix.dq.norm"], names[p + "mix.dkv.norm"] = ((m["q_rank"],), "gain"), ((m["kv_rank"],), "gain")
        if f["kind"] == "moe":
            names[p + "mlp.router"], names[p + "mlp.router.b"] = ((f["router"]["experts"], d), "vector"), ((f["router"]["experts"],), "vector")
        for q, ff in [("mlp.", f["ff"])] if f["kind"] == "dense" else [(f"mlp.e{e}.", f["expert"]["ff"]) for e in range(f["router"]["experts"])]:
            names[p + q + "gate"], names[p + q + "up"], names[p + q + "down"] = ((ff, d), "matrix"), ((ff, d), "matrix"), ((d, ff), "matrix")
    return names


def _forward_lezepel(c, w, ids, pos, starts, rows):
    eps = c["norm"]["eps"]
    x = w["embed"][ids].double() * c["embedding"]["scale"]
    for i, L in enumerate(c["layers"]):
        m, f, T = L["mixer"], L["mlp"], len(ids)

        def g(name):
            return w[f"l{i}.{name}"].double()

        if i == c["loop"]["start"]:         # one pass: the loop's first layer is entered with the pass vector added
            x = x + w["loop.step"][0].double()
        H, dn, dr, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        cos, sin = _tables(pos, m["rot"]["dims"], m["rot"]["base"])
        h = _rms(x, g("norm1"), eps)
        q = (_rms(h @ g("mix.dq").T, g("mix.dq.norm"), eps) @ g("mix.uq").T).view(T, H, dn + dr)
        kv = h @ g("mix.dkv").T
        latent = _rms(kv[:, :r], g("mix.dkv.norm"), eps)
        k_rot = _turn(kv[:, None, r:], cos, sin).expand(T, H, dr)
        k = torch.cat([(latent @ g("mix.uk").T).view(T, H, dn), k_rot], -1)
        q = torch.cat([q[..., :dn], _turn(q[..., dn:], cos, sin)], -1)
        y = _attend(q, k, (latent @ g("mix.uv").T).view(T, H, dv), starts, m["scale"]).reshape(T, H * dv)
        y = (y * torch.sigmoid(h @ g("mix.g").T)) @ g("mix.o").T
        if f["kind"] == "dense":
            y = y + (torch.relu(h @ g("mlp.gate").T) * (h @ g("mlp.up").T)) @ g("mlp.down").T
        else:
            best, which = torch.topk(h @ g("mlp.router").T + g("mlp.router.b"), f["router"]["top"], dim=-1)
            share = torch.softmax(best, -1)
            for e in range(f["router"]["experts"]):
                t, slot = (which == e).nonzero(as_tuple=True)
                if len(t):
                    he = h[t]
                    out = (torch.nn.functional.silu(he @ g(f"mlp.e{e}.gate").T) * (he @ g(f"mlp.e{e}.up").T)) @ g(f"mlp.e{e}.down").T
                    y = y.index_add(0, t, out * share[t, slot][:, None])
        x = x + y
    return _rms(x[rows], w["final.norm"].double(), eps) @ w["head"].double().T


def _forward(cfg, w, texts, rows):
    """Logits at ``rows`` (numbers of tokens in the concatenation of ``texts``)."""
    ids = torch.tensor([t for x in texts for t in x], device=DEVICE)
    pos = torch.tensor([p for x in texts for p in range(len(x))])
    starts = np.cumsum([0] + [len(x) for x in texts]).tolist()
    f = _forward_lezepel if cfg.get("architecture") == "Lezepel" else _forward_qwen3
    return f(cfg, w, ids, pos, starts, torch.tensor(rows, device=DEVICE))


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    cfg = MODELS[case["model"]]
    w = _weights(_names_lezepel(cfg) if cfg.get("architecture") == "Lezepel" else _names_qwen3(cfg), seed, case["dtype"], _std(cfg))
    turns = _requests(case, seed)
    if case["kind"] == "generate":
        texts = [list(p) for p in turns[0][0]]
        for _ in range(case["steps"]):
            ends = (np.cumsum([len(t) for t in texts]) - 1).tolist()
            for t, token in zip(texts, _forward(cfg, w, texts, ends).argmax(-1).tolist()):
                t.append(token)
        return {"tokens": None, "logits": _forward(cfg, w, texts, list(range(sum(len(t) for t in texts))))}
    texts, wanted = [[] for _ in range(case["batch"])], []
    for portions, steps in turns:
        for t, p in zip(texts, portions):
            t.extend(p)
        wanted.append([len(t) - 1 for t in texts])
        for row in steps:
            for t, token in zip(texts, row):
                t.append(token)
            wanted.append([len(t) - 1 for t in texts])
    base = np.cumsum([0] + [len(t) for t in texts])[:-1]
    logits = _forward(cfg, w, texts, [int(b + r) for rows in wanted for b, r in zip(base, rows)]).to(torch.float64)
    logits = logits.view(len(turns), 1 + case["steps"], case["batch"], -1)
    return [(t[0], t[1:]) for t in logits]
