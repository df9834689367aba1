"""The work that programs have this engine do, as cases that can be timed and compared.

A case is a dictionary of plain values; ``listed()`` names the ones that are followed, ``draw(rng)`` makes another
of the same ranges.  ``prepare`` holds what a serving program has in hand (a loaded engine, the prompts as lists of
token ids), ``run`` is one pass through the engine's entry points, ``exact`` the same answers from a plain float64
restatement of the model that shares no code with the package.

Models (random weights; the sizes are those of the benchmark and of the design comparison):

  llama      Llama 3.2 1B sizes, bfloat16: the benchmark's model
  llama32    the same model in a float32 engine
  kapitar    four layers: differential attention over a window, linear attention, dense and routed feed-forwards
  vogolix    four layers: chunked attention with shared keys, a state-space layer, windowed latent attention

Every embedding is tied to (or copied into) the head and the sublayers add less to the stream than a trained
model's embedding holds, so that the next token is clear-cut, as it is for a trained model most of the time: two
correct engines then generate the same tokens, and their logits can be compared row by row.

Kinds of work:

  generate   ``Engine.generate_requests``: prompts in, a fixed number of new tokens out; the logits of every
             generated position are taken from ``Engine.on_logits``
  score      ``Engine.score``: the log-probability of every token of a text
  replay     ``Engine.step_tokens`` with given tokens: portions of prompts beside single tokens, logits wanted
             at the last place of each (what the trace replay program does)
"""

import json
import math
import os
import random
import struct
import tempfile

import numpy as np
import torch

F64 = torch.float64

LLAMA = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": 16, "hidden_size": 2048,
    "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64, "intermediate_size": 8192,
    "vocab_size": 128256, "rope_theta": 500000.0,
    "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                     "original_max_position_embeddings": 8192},
    "rms_norm_eps": 1e-5, "tie_word_embeddings": True, "max_position_embeddings": 131072, "hidden_act": "silu",
    "bos_token_id": 128000, "eos_token_id": 128001,
}


def _kapitar():
    att = {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 128, "diff": 0.5, "softcap": 30.0, "scale": 0.125,
           "mask": {"size": 1024, "keep_first": 4}}
    lin = {"heads": 16, "dim": 64, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 5 * h / 15) for h in range(16)]}
    dense = {"kind": "dense", "ff": 8192}
    moe = {"kind": "moe", "expert": {"ff": 1024}, "shared": {"ff": 2048},
           "router": {"experts": 32, "top": 4, "groups": {"count": 4, "keep": 2}}}
    return {"architecture": "Kapitar", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6},
            "layers": [{"type": "attention", "mixer": att, "mlp": dense}, {"type": "lightning", "mixer": lin, "mlp": moe},
                       {"type": "attention", "mixer": att, "mlp": moe}, {"type": "lightning", "mixer": lin, "mlp": dense}]}


def _vogolix():
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
           "rot": {"base": 1000000.0, "dims": 64}}
    latent = {"heads": 16, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 192, "scale": 96 ** -0.5, "mask": {"size": 1024},
              "rot": {"base": 500000.0, "dims": 32}}
    ssm = {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}
    dense = {"kind": "dense", "ff": 5632}
    return {"architecture": "Vogolix", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "logit_scale": 0.5,
            "layers": [{"type": "attention", "mixer": att, "mlp": dense}, {"type": "mamba2", "mixer": ssm, "mlp": dense},
                       {"type": "attention", "mixer": dict(att, kv_from=0), "mlp": dense},
                       {"type": "latent_attention", "mixer": latent, "mlp": dense}]}


# model -> (configuration, the engine's compute type)
MODELS = {"llama": (LLAMA, "bfloat16"), "llama32": (LLAMA, "float32"), "kapitar": (_kapitar(), "bfloat16"),
          "vogolix": (_vogolix(), "bfloat16")}
STEP_TOKENS = 2048      # prompt tokens of one step: the engine's default


def listed():
    return [
        # one person chatting: a short prompt, tokens one by one (latency of the smallest step)
        {"name": "chat one", "model": "llama", "kind": "generate", "requests": 1, "shortest": 48, "longest": 48, "new": 32},
        # the benchmark's load: eight long documents, answers behind contexts of almost 4,096 tokens
        {"name": "eight long contexts", "model": "llama", "kind": "generate", "requests": 8, "shortest": 3712, "longest": 3840,
         "new": 96},
        # a busy server: 64 chats decoding together
        {"name": "serve sixty-four", "model": "llama", "kind": "generate", "requests": 64, "shortest": 96, "longest": 160,
         "new": 64},
        # requests of very different lengths, sampled with a temperature and top-p: an odd batch size
        {"name": "ragged sampled", "model": "llama", "kind": "generate", "requests": 21, "shortest": 17, "longest": 901,
         "new": 24, "temperature": 0.8},
        # time to first token of a short question, of the benchmark's prompt, and of a long document in portions
        {"name": "prompt short odd", "model": "llama", "kind": "generate", "requests": 1, "shortest": 333, "longest": 333,
         "new": 1},
        {"name": "prompt 2048", "model": "llama", "kind": "generate", "requests": 1, "shortest": 2048, "longest": 2048, "new": 1},
        {"name": "prompt long", "model": "llama", "kind": "generate", "requests": 1, "shortest": 14999, "longest": 14999,
         "new": 1},
        # a text's log-probabilities: logits at every position
        {"name": "score a text", "model": "llama", "kind": "score", "requests": 1, "shortest": 1201, "longest": 1201},
        # the trace replay program: portions of four prompts beside single tokens, every step with its logits
        {"name": "replay", "model": "llama", "kind": "replay", "requests": 4, "shortest": 150, "longest": 260, "new": 8},
        # the float32 engine, used to check results: two short prompts
        {"name": "float32", "model": "llama32", "kind": "generate", "requests": 2, "shortest": 90, "longest": 120, "new": 8},
        # other designs served by the same engine, at the sizes of their comparison: eight requests of 512-token prompts
        {"name": "kapitar", "model": "kapitar", "kind": "generate", "requests": 8, "shortest": 448, "longest": 512, "new": 64},
        {"name": "vogolix", "model": "vogolix", "kind": "generate", "requests": 8, "shortest": 448, "longest": 512, "new": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["generate"] * 5 + ["prompt", "prompt", "score", "replay", "float32", "kapitar", "vogolix"])
    if what == "generate":
        n = _log_int(rng, 1, 64)
        long = _log_int(rng, 16, min(3900, 40000 // n))
        short = _log_int(rng, max(4, long // 8), long)
        new = _log_int(rng, 8, 96)
        new = max(4, min(new, 6000 // n))
        return {"model": "llama", "kind": "generate", "requests": n, "shortest": short, "longest": long, "new": new,
                "temperature": rng.choice([0.0, 0.0, 0.8])}
    if what == "prompt":
        n = _log_int(rng, 20, 14999)
        return {"model": "llama", "kind": "generate", "requests": 1, "shortest": n, "longest": n, "new": 1}
    if what == "score":
        n = _log_int(rng, 50, 3000)
        return {"model": "llama", "kind": "score", "requests": 1, "shortest": n, "longest": n}
    if what == "replay":
        long = _log_int(rng, 40, 700)
        return {"model": "llama", "kind": "replay", "requests": rng.randint(1, 8), "shortest": max(4, long // 2), "longest": long,
                "new": rng.randint(2, 12)}
    if what == "float32":
        long = _log_int(rng, 8, 130)
        return {"model": "llama32", "kind": "generate", "requests": rng.randint(1, 3), "shortest": max(4, long // 2),
                "longest": long, "new": rng.randint(2, 8)}
    long = _log_int(rng, 100, 600)
    return {"model": what, "kind": "generate", "requests": rng.randint(1, 12), "shortest": max(4, long // 2), "longest": long,
            "new": rng.randint(16, 64)}


# ---------------------------------------------------------------------------------------------- weights

def _tensors(cfg):
    """Yields (name, shape, mean, standard deviation) of a model's tensors."""
    if "architectures" in cfg:
        H, I, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        nq, nk = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
        yield "model.embed_tokens.weight", (V, H), 0.0, 0.05
        for i in range(cfg["num_hidden_layers"]):
            p = "model.layers.%d." % i
            yield p + "input_layernorm.weight", (H,), 1.0, 0.1
            for n, rows in (("q", nq), ("k", nk), ("v", nk)):
                yield p + "self_attn.%s_proj.weight" % n, (rows, H), 0.0, 0.02
            yield p + "self_attn.o_proj.weight", (H, nq), 0.0, 5e-4
            yield p + "post_attention_layernorm.weight", (H,), 1.0, 0.1
            yield p + "mlp.gate_proj.weight", (I, H), 0.0, 0.02
            yield p + "mlp.up_proj.weight", (I, H), 0.0, 0.02
            yield p + "mlp.down_proj.weight", (H, I), 0.0, 5e-4
        yield "model.norm.weight", (H,), 1.0, 0.1
        return
    W, V = cfg["width"], cfg["vocab"]

    def mat(name, rows, cols):
        return name, (rows, cols), 0.0, cols ** -0.5

    yield "embed", (V, W), 0.0, 1.0
    for i, layer in enumerate(cfg["layers"]):
        p, m, kind, f = "l%d." % i, layer["mixer"], layer["type"], layer["mlp"]
        q, H = p + "mix.", layer["mixer"]["heads"]
        norms = ("norm1", "norm1b", "norm2", "norm2b") if cfg["architecture"] == "Kapitar" else ("norm1", "norm2")
        for n in norms:
            yield p + n, (W,), 1.0, 0.1
        if kind == "lightning":
            for n, rows in (("q", H * m["dim"]), ("k", H * m["dim"]), ("v", H * m["vdim"]), ("g", H * m["vdim"])):
                yield mat(q + n, rows, W)
            yield mat(q + "o", W, H * m["vdim"])
            yield q + "norm", (H * m["vdim"],), 1.0, 0.1
        elif kind == "mamba2":
            inner, bc = H * m["vdim"], 2 * m["groups"] * m["state"]
            yield mat(q + "in", 2 * inner + bc + H, W)
            yield mat(q + "conv", inner + bc, m["conv"])
            yield q + "conv.b", (inner + bc,), 0.0, 0.1
            yield q + "dt_bias", (H,), -3.0, 1.0
            yield q + "A_log", (H,), 1.0, 0.7
            yield q + "D", (H,), 0.0, 1.0
            yield q + "norm", (inner,), 1.0, 0.1
            yield mat(q + "o", W, inner)
        elif kind == "latent_attention":
            yield mat(q + "q", H * (m["dim"] + m["rot_dim"]), W)
            yield mat(q + "dkv", m["kv_rank"] + m["rot_dim"], W)
            yield q + "dkv.norm", (m["kv_rank"],), 1.0, 0.1
            yield mat(q + "uk", H * m["dim"], m["kv_rank"])
            yield mat(q + "uv", H * m["vdim"], m["kv_rank"])
            yield mat(q + "g", H * m["vdim"], W)
            yield mat(q + "o", W, H * m["vdim"])
        else:
            maps = 2 if cfg["architecture"] == "Kapitar" else 1
            sides = [("q", H * maps * m["dim"])]
            if m.get("kv_from") is None:
                sides += [("k", m["kv_heads"] * maps * m["dim"]), ("v", m["kv_heads"] * m["vdim"])]
            for n, rows in sides:
                yield mat(q + n, rows, W)
                yield q + n + ".b", (rows,), 0.0, 0.1
                if maps == 1 and n != "v":
                    yield q + n + ".norm", (rows,), 1.0, 0.1
            if maps == 2:
                for n in ("lq1", "lk1", "lq2", "lk2"):
                    yield q + n, (m["dim"],), 0.0, 0.1
            else:
                yield q + "sink", (H,), 0.0, 1.0
            yield mat(q + "o", W, H * m["vdim"])
        if f["kind"] == "moe":
            for e in range(f["router"]["experts"]):
                yield mat("%smlp.e%d.up" % (p, e), f["expert"]["ff"], W)
                yield mat("%smlp.e%d.down" % (p, e), W, f["expert"]["ff"])
            yield mat(p + "mlp.router", f["router"]["experts"], W)
            yield mat(p + "mlp.shared.up", f["shared"]["ff"], W)
            yield mat(p + "mlp.shared.down", W, f["shared"]["ff"])
        else:
            if cfg["architecture"] == "Vogolix":
                yield mat(p + "mlp.gate", f["ff"], W)
            yield mat(p + "mlp.up", f["ff"], W)
            yield mat(p + "mlp.down", W, f["ff"])
    yield "final.norm", (W,), 1.0, 0.1
    if cfg["architecture"] == "Vogolix":
        yield "head", (V, W), None, None          # the embedding's rows once more


def _weights(cfg):
    """Yields (name, bfloat16 tensor on the GPU), the same ones every time."""
    g = torch.Generator(device="cuda").manual_seed(20)
    for name, shape, mean, std in _tensors(cfg):
        if std is None:
            yield name, embed
            continue
        t = (torch.randn(shape, generator=g, device="cuda") * std + mean).to(torch.bfloat16)
        if name == "embed":
            embed = t
        yield name, t


def _write_model(folder, cfg):
    """config.json and model.safetensors (header length, JSON header, the tensors' bytes)."""
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(cfg, f)
    header, at = {}, 0
    for name, shape, _, _ in _tensors(cfg):
        n = 2 * math.prod(shape)
        header[name] = {"dtype": "BF16", "shape": list(shape), "data_offsets": [at, at + n]}
        at += n
    head = json.dumps(header).encode()
    head += b" " * (-len(head) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(head)))
        f.write(head)
        for _, t in _weights(cfg):
            t.view(torch.int16).cpu().numpy().tofile(f)


# ---------------------------------------------------------------------------------------------- passes

_engines = {}


def _long(case):
    return case["longest"] + case.get("new", 0) > 4096


def _engine(case):
    """A program loads its model once and keeps the engine."""
    from redline_b200.engine.engine import Engine
    key = (case["model"], _long(case))
    if key not in _engines:
        cfg, dtype = MODELS[case["model"]]
        if case["model"] == "llama":
            opts = {"max_num_seqs": 4, "max_seq_len": 16384, "kv_cache_tokens": 32768} if key[1] else \
                {"max_num_seqs": 64, "max_seq_len": 4096, "kv_cache_tokens": 65536}
        elif case["model"] == "llama32":
            opts = {"max_num_seqs": 4, "max_seq_len": 2048, "kv_cache_tokens": 8192}
        else:
            opts = {"max_num_seqs": 16, "max_seq_len": 2048, "kv_cache_tokens": 32768}
        with tempfile.TemporaryDirectory() as folder:
            _write_model(folder, cfg)
            _engines[key] = Engine(folder, dtype=dtype, max_num_batched_tokens=STEP_TOKENS, **opts)
    return _engines[key]


def _prompts(case, seed):
    cfg = MODELS[case["model"]][0]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    r = np.random.RandomState(seed % (1 << 31))
    lengths = random.Random(7).choices(range(case["shortest"], case["longest"] + 1), k=case["requests"])
    return [r.randint(0, vocab, size=n).tolist() for n in lengths]


def _replay_steps(case, prompts, seed):
    """[(request, its tokens, wanted places)] per step: request i joins at step i with a portion of its prompt, brings
    the rest in the next step and then single tokens."""
    r = np.random.RandomState((seed + 1) % (1 << 31))
    more = [r.randint(0, 32000, size=case["new"]).tolist() for _ in prompts]
    left = []
    for p, m in zip(prompts, more):
        cut = max(1, 2 * len(p) // 3)
        left.append([p[:cut], p[cut:]] + [[t] for t in m])
    steps = []
    for at in range(len(prompts) + max(len(x) for x in left) - 1):
        entries = [(i, x[at - i], [len(x[at - i]) - 1]) for i, x in enumerate(left) if 0 <= at - i < len(x) and x[at - i]]
        if entries:
            steps.append(entries)
    return steps


def prepare(case, seed):
    eng = _engine(case)
    prompts = _prompts(case, seed)
    state = {"case": case, "engine": eng, "prompts": prompts}
    if case["kind"] == "replay":
        state["steps"] = _replay_steps(case, prompts, seed)
    elif case["kind"] == "generate":
        from redline_b200.sampling import SamplingParams
        t = case.get("temperature", 0.0)
        state["params"] = SamplingParams(temperature=t, top_p=0.95 if t > 0 else 1.0, seed=11, max_new_tokens=case["new"],
                                         ignore_eos=True)
    return state


def run(state):
    case, eng = state["case"], state["engine"]
    if case["kind"] == "score":
        return {"logprobs": np.array(eng.score(state["prompts"][0]))}
    if case["kind"] == "replay":
        out = [eng.step_tokens(entries) for entries in state["steps"]]
        for i in range(len(state["prompts"])):
            eng.close_request(i)
        return {"logits": torch.cat(out)}
    rows, logits = [], []

    def keep(which, values):
        rows.extend(which)
        logits.append(values.clone())

    eng.on_logits = keep
    outs = eng.generate_requests([(p, state["params"]) for p in state["prompts"]])
    eng.on_logits = None
    # (with steps launched ahead of the tokens, a request's last step may run once more than needed)
    place, first = {}, outs[0]["id"]
    for at, (request, position) in enumerate(rows):
        place[(request - first, position - len(state["prompts"][request - first]) + 1)] = at
    order = [place[(i, k)] for i in range(len(outs)) for k in range(case["new"])]
    logits = logits[0] if len(logits) == 1 else torch.cat(logits)
    if order != list(range(logits.shape[0])):
        logits = logits[torch.tensor(order, device=logits.device)]
    return {"tokens": np.array([o["output_ids"] for o in outs]), "logits": logits}


# ---------------------------------------------------------------------------------------------- measures

def _per_token(cfg):
    """(entries of the matrices that one token meets, of all layers' matrices, entries cached or kept per token,
    operations per visible key of a token)."""
    if "architectures" in cfg:
        L, D = cfg["num_hidden_layers"], cfg["head_dim"]
        nq, nk = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
        n = L * cfg["hidden_size"] * (2 * nq + 2 * nk + 3 * cfg["intermediate_size"])
        return n, n, 2 * nk * L, 4 * nq * L
    met = every = cached = per_key = 0
    for name, shape, _, std in _tensors(cfg):
        if len(shape) == 2 and name not in ("embed", "head"):
            n = math.prod(shape)
            every += n
            met += n if ".e" not in name else n * 4 / 32
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "attention":
            maps = 2 if cfg["architecture"] == "Kapitar" else 1
            cached += m["kv_heads"] * (maps * m["dim"] + m["vdim"])
            per_key += 2 * m["heads"] * (maps * m["dim"] + m["vdim"])
        elif layer["type"] == "latent_attention":
            cached += m["kv_rank"] + m["rot_dim"]
            per_key += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
    return met, every, cached, per_key


def work(case):
    cfg, dtype = MODELS[case["model"]]
    elem = 2 if dtype == "bfloat16" else 4
    vocab, width = cfg.get("vocab_size") or cfg["vocab"], cfg.get("hidden_size") or cfg["width"]
    met, every, cached, per_key = _per_token(cfg)
    window = 1 << 30 if "architectures" in cfg else 1024
    lengths = [len(p) for p in _prompts(case, 0)]
    new = case.get("new", 1)
    if case["kind"] == "score":
        lengths = [n - 1 for n in lengths]
        tokens, rows, single = sum(lengths), sum(lengths), 0
    elif case["kind"] == "replay":
        tokens, rows, single = sum(lengths) + new * len(lengths), (new + 2) * len(lengths), new
    else:
        tokens, rows, single = sum(lengths) + (new - 1) * len(lengths), new * len(lengths), new - 1
    steps = -(-sum(lengths) // STEP_TOKENS) + single
    seen = sum(sum(min(i + 1, window) for i in range(n)) for n in lengths)
    alone = sum(min(n + k, window) for n in lengths for k in range(1, single + 1))
    flops = 2.0 * met * tokens + 2.0 * vocab * width * rows + per_key * (seen + alone)
    # weights once a step, the cache of a single token's context, the prompts' cache once a portion, the logits
    back = sum(n * (n // STEP_TOKENS) // 2 for n in lengths)
    nbytes = elem * (steps * (every + vocab * width) + cached * (alone + back + tokens)) + 4.0 * vocab * rows
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    # about four times what the engine is off the float64 restatement: 3.5e-6 in float32; 7e-3 in bfloat16 logits,
    # 4e-4 in log-probabilities (their largest part is the row's maximum)
    if case["model"] == "llama32":
        return {"rel": 1.5e-5, "max": 2e-4, "differ": 0.0}
    if case["kind"] == "score":
        return {"rel": 2e-3}
    if case["model"] == "kapitar":
        # 3.8e-2: a token whose router scores are nearly equal may go to another expert
        return {"rel": 0.12, "differ": 0.02}
    return {"rel": 2.5e-2, "differ": 0.02}


# ---------------------------------------------------------------------------------------------- float64

def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, cos, sin, pairs):
    """x [T, heads, n]: the first 2 * cos.shape[1] entries turned, neighbours or entry i with entry i + half."""
    half = cos.shape[1]
    c, s, out = cos[:, None], sin[:, None], x.clone()
    if pairs:
        u, v = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        out[..., 0:2 * half:2], out[..., 1:2 * half:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :half], x[..., half:2 * half]
        out[..., :half], out[..., half:2 * half] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, first, cap=0.0, keep=0, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, E] -> [T, H, E]; row i sees keys first[i] .. i and the first ``keep``."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    j = torch.arange(T, device=q.device)[None]
    rows = 1024
    for a in range(0, T, rows):
        b = min(T, a + rows)
        i = torch.arange(a, b, device=q.device)[:, None]
        seen = (j[:, :b] <= i) & ((j[:, :b] >= first[a:b, None]) | (j[:, :b] < keep))
        for h in range(H):
            s = q[a:b, h] @ k[:b, h // per].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], dim=1)
            p = torch.softmax(s, dim=-1)
            out[a:b, h] = (p[:, :-1] if sink is not None else p) @ v[:b, h // per]
    return out


def _llama_angles(cfg, n):
    D, sc = cfg["head_dim"], cfg["rope_scaling"]
    freq = []
    for i in range(D // 2):
        f = cfg["rope_theta"] ** (-2.0 * i / D)
        wave, old = 2 * math.pi / f, sc["original_max_position_embeddings"]
        if wave > old / sc["low_freq_factor"]:
            f /= sc["factor"]
        elif wave >= old / sc["high_freq_factor"]:
            t = (old / wave - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])
            f = (1 - t) * f / sc["factor"] + t * f
        freq.append(f)
    # the angle is formed in float32, as the model's definition has it
    a = torch.arange(n, dtype=torch.float32)[:, None] * torch.tensor(freq, dtype=F64).to(torch.float32)[None]
    a = a.to(F64).cuda()
    return a.cos(), a.sin()


def _llama_layers(cfg, w, xs):
    D, eps = cfg["head_dim"], cfg["rms_norm_eps"]
    cos, sin = _llama_angles(cfg, max(x.shape[0] for x in xs))
    for i in range(cfg["num_hidden_layers"]):
        W = {n: w["model.layers.%d.%s.weight" % (i, n)].to(F64) for n in
             ("input_layernorm", "self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
              "post_attention_layernorm", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        for n, x in enumerate(xs):
            T = x.shape[0]
            h = _rms(x, W["input_layernorm"], eps)
            q, k, v = ((h @ W["self_attn.%s_proj" % c].T).view(T, -1, D) for c in "qkv")
            q, k = _turn(q, cos[:T], sin[:T], False), _turn(k, cos[:T], sin[:T], False)
            o = _attend(q, k, v, D ** -0.5, torch.zeros(T, dtype=torch.long, device=x.device))
            x = x + o.reshape(T, -1) @ W["self_attn.o_proj"].T
            h = _rms(x, W["post_attention_layernorm"], eps)
            xs[n] = x + (_silu(h @ W["mlp.gate_proj"].T) * (h @ W["mlp.up_proj"].T)) @ W["mlp.down_proj"].T
    return xs, w["model.norm.weight"], w["model.embed_tokens.weight"], 1.0


def _kapitar_ff(h, W, f):
    if f["kind"] == "dense":
        return torch.relu(h @ W["up"].T) ** 2 @ W["down"].T

    def ff(x, p):
        return torch.nn.functional.gelu(x @ W[p + "up"].T) @ W[p + "down"].T

    r = f["router"]
    s = torch.sigmoid(h @ W["router"].T)
    T, E = s.shape
    n = r["groups"]["count"]
    kept = s.view(T, n, E // n).topk(2, dim=-1).values.sum(-1).topk(r["groups"]["keep"], dim=-1).indices
    allowed = torch.zeros(T, n, dtype=torch.bool, device=h.device).scatter_(1, kept, True).repeat_interleave(E // n, 1)
    choice = s.masked_fill(~allowed, -1.0).topk(r["top"], dim=-1).indices
    out = ff(h, "shared.")
    for e in range(E):
        t = (choice == e).any(-1).nonzero()[:, 0]
        if t.numel():
            out[t] += s[t, e, None] * ff(h[t], "e%d." % e)
    return out


def _kapitar_layers(cfg, w, xs):
    eps = cfg["norm"]["eps"]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        W = {n[len(p):]: t.to(F64) for n, t in w.items() if n.startswith(p)}
        M = {n[4:]: t for n, t in W.items() if n.startswith("mix.")}
        F = {n[4:]: t for n, t in W.items() if n.startswith("mlp.")}
        H, D, E = m["heads"], m["dim"], m["vdim"]
        for n, x in enumerate(xs):
            T = x.shape[0]
            h = _layer_norm(x, W["norm1"], eps)
            if layer["type"] == "attention":
                q = (h @ M["q"].T + M["q.b"]).view(T, H, 2, D)
                k = (h @ M["k"].T + M["k.b"]).view(T, m["kv_heads"], 2, D)
                v = (h @ M["v"].T + M["v.b"]).view(T, m["kv_heads"], E)
                lam = (M["lq1"] * M["lk1"]).sum().exp() - (M["lq2"] * M["lk2"]).sum().exp() + m["diff"]
                first = (torch.arange(T, device=x.device) - m["mask"]["size"] + 1).clamp(min=0)
                a, b = (_attend(q[:, :, c], k[:, :, c], v, m["scale"], first, m["softcap"], m["mask"]["keep_first"])
                        for c in (0, 1))
                y = _rms(a - lam * b, 1.0 - m["diff"], eps).reshape(T, -1)
            else:
                q, k, v = (_silu(h @ M[c].T).view(T, H, -1) for c in "qkv")
                decay = torch.tensor(m["decay"], dtype=F64, device=x.device)[:, None, None]
                S, o = torch.zeros(H, D, E, dtype=F64, device=x.device), []
                for t in range(T):
                    S = decay * S + k[t][:, :, None] * v[t][:, None]
                    o.append((q[t][:, None] @ S)[:, 0])
                y = _rms(torch.stack(o).reshape(T, -1), M["norm"], eps) * torch.sigmoid(h @ M["g"].T)
            x = x + _layer_norm(y @ M["o"].T, W["norm1b"], eps)
            xs[n] = x + _layer_norm(_kapitar_ff(_layer_norm(x, W["norm2"], eps), F, layer["mlp"]), W["norm2b"], eps)
    return xs, w["final.norm"], w["embed"], 1.0


def _design_angles(rot, n):
    f = torch.tensor([rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)], dtype=F64)
    a = (torch.arange(n, dtype=F64)[:, None] * f[None]).cuda()
    return a.cos(), a.sin()


def _state_space(h, M, m, eps):
    T, H, e, N = h.shape[0], m["heads"], m["vdim"], m["state"]
    inner = H * e
    z, u, d = (h @ M["in"].T).split([inner, inner + 2 * N, H], dim=1)
    past = torch.cat([torch.zeros(m["conv"] - 1, u.shape[1], dtype=F64, device=h.device), u])
    u = _silu(sum(past[j:j + T] * M["conv"][:, j] for j in range(m["conv"])) + M["conv.b"])
    x, B, C = u[:, :inner].view(T, H, e), u[:, inner:inner + N], u[:, inner + N:]
    dt = torch.nn.functional.softplus(d + M["dt_bias"])
    a = torch.exp(-torch.exp(M["A_log"]) * dt)
    S, o = torch.zeros(H, N, e, dtype=F64, device=h.device), []
    for t in range(T):
        S = a[t, :, None, None] * S + B[t][None, :, None] * (dt[t, :, None] * x[t])[:, None]
        o.append((C[t][None, None] @ S)[:, 0])
    y = torch.stack(o) + M["D"][:, None] * x
    return _rms(y.reshape(T, inner) * _silu(z), M["norm"], eps)


def _vogolix_layers(cfg, w, xs):
    eps, kvs = cfg["norm"]["eps"], {}
    for i, layer in enumerate(cfg["layers"]):
        m, p, kind = layer["mixer"], "l%d." % i, layer["type"]
        W = {n[len(p):]: t.to(F64) for n, t in w.items() if n.startswith(p)}
        M = {n[4:]: t for n, t in W.items() if n.startswith("mix.")}
        H = m["heads"]
        for n, x in enumerate(xs):
            T = x.shape[0]
            h, at = _rms(x, W["norm1"], eps), torch.arange(T, device=x.device)
            if kind == "mamba2":
                y = _state_space(h, M, m, eps)
            elif kind == "attention":
                cos, sin = _design_angles(m["rot"], T)
                G, size = m["kv_heads"], m["mask"]["size"]
                if m.get("kv_from") is None:
                    k = _rms(h @ M["k"].T + M["k.b"], M["k.norm"], eps).view(T, G, -1)
                    kvs[i, n] = _turn(k, cos, sin, True), (h @ M["v"].T + M["v.b"]).view(T, G, -1)
                k, v = kvs[m.get("kv_from", i), n]
                q = _turn(_rms(h @ M["q"].T + M["q.b"], M["q.norm"], eps).view(T, H, -1), cos, sin, True)
                y = _attend(q, k, v, m["scale"], at // size * size, sink=M["sink"]).reshape(T, -1)
            else:
                cos, sin = _design_angles(m["rot"], T)
                dn, rank = m["dim"], m["kv_rank"]
                q, raw = (h @ M["q"].T).view(T, H, -1), h @ M["dkv"].T
                c = _rms(raw[:, :rank], M["dkv.norm"], eps)
                kr = _turn(raw[:, None, rank:], cos, sin, False).expand(T, H, m["rot_dim"])
                q = torch.cat([q[..., :dn], _turn(q[..., dn:], cos, sin, False)], -1)
                k = torch.cat([(c @ M["uk"].T).view(T, H, dn), kr], -1)
                y = _attend(q, k, (c @ M["uv"].T).view(T, H, -1), m["scale"], (at - m["mask"]["size"] + 1).clamp(min=0))
                y = y.reshape(T, -1) * torch.sigmoid(h @ M["g"].T)
            x = x + y @ M["o"].T
            h = _rms(x, W["norm2"], eps)
            xs[n] = x + (torch.relu(h @ W["mlp.gate"].T) * (h @ W["mlp.up"].T)) @ W["mlp.down"].T
    return xs, w["final.norm"], w["head"], cfg["logit_scale"]


def _logits(cfg, w, sequences, places):
    """float64 logits of every sequence's wanted places."""
    embed = w["model.embed_tokens.weight"] if "architectures" in cfg else w["embed"]
    layers = _llama_layers if "architectures" in cfg else {"Kapitar": _kapitar_layers, "Vogolix": _vogolix_layers}[cfg["architecture"]]
    xs, norm, head, scale = layers(cfg, w, [embed[torch.tensor(s, device="cuda")].to(F64) for s in sequences])
    f = _layer_norm if cfg.get("architecture") == "Kapitar" else _rms
    eps = cfg["rms_norm_eps"] if "architectures" in cfg else cfg["norm"]["eps"]
    head = head.to(F64).T
    return [f(x[torch.tensor(at, device="cuda")], norm.to(F64), eps) @ head * scale for x, at in zip(xs, places)]


def exact(case, seed):
    cfg = MODELS[case["model"]][0]
    w = dict(_weights(cfg))
    prompts = _prompts(case, seed)
    if case["kind"] == "score":
        p = prompts[0]
        out = _logits(cfg, w, [p[:-1]], [list(range(len(p) - 1))])[0]
        target = torch.tensor(p[1:], device="cuda")
        return {"logprobs": (out.gather(1, target[:, None])[:, 0] - torch.logsumexp(out, -1)).cpu().numpy()}
    if case["kind"] == "replay":
        steps = _replay_steps(case, prompts, seed)
        tokens, places, order = [[] for _ in prompts], [[] for _ in prompts], []
        for entries in steps:
            for i, toks, want in entries:
                order.append((i, len(places[i])))
                places[i].append(len(tokens[i]) + want[0])
                tokens[i].extend(toks)
        out = _logits(cfg, w, tokens, places)
        return {"logits": torch.stack([out[i][k] for i, k in order])}
    # greedy: guess the answers, and take what the model says instead until nothing changes
    new = case["new"]
    answers = [[p[-1]] * new for p in prompts]
    for _ in range(8):
        sequences = [p + a[:-1] for p, a in zip(prompts, answers)]
        out = _logits(cfg, w, sequences, [list(range(len(p) - 1, len(p) - 1 + new)) for p in prompts])
        said = [o.argmax(-1).tolist() for o in out]
        if said == answers:
            break
        answers = said
    return {"tokens": np.array(answers), "logits": torch.cat(out)}
