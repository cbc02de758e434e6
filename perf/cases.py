"""What a user of the library has it do, as cases that can be timed and checked.

A case is a model (an architecture at one of the sizes that ``bench.py`` or the smallest configurations of
the tests give it, random weights), a number format and a workload:

* ``kind`` "request": sequences are opened, their prompts run as ONE ragged step (``LLM.step``), then every sequence
  takes ``new`` tokens one at a time through a ``DecodeSession``, and the sequences are closed: what ``LLM.generate`` does
  for a batch, except that the tokens fed are given (a stored continuation) so that the logits of two runs can be
  compared.  Outputs: the logits behind every prompt and behind the last token fed, float32 [batch, vocab] each.
* ``kind`` "generate": ``LLM.generate`` itself, greedy, token ids in and out.  Only in float32, where the tokens of two
  correct implementations are the same.

Prompt lengths are spread evenly from ``shortest`` to ``longest`` over the batch.  The largest models are cut to some of
their layers, which repeat, so that weights, cache and a 64-bit run of the same stay small.
"""
from __future__ import annotations

import math

import torch

VOCAB = 151936
GREEDY, FILTERED = (0.0, 0, 1.0, 1.0), (0.7, 40, 0.9, 1.0)      # temperature, top_k, top_p, repeat_penalty

# hidden, feed-forward, heads, kv heads, head size, tied, vocabulary, theta, eps
QWEN3 = {
    "tiny-a": (64, 128, 4, 2, 16, True, 256, 1e4, 1e-6),
    "tiny-b": (96, 224, 6, 1, 32, False, 311, 1e6, 1e-5),
    "0.6b": (1024, 3072, 16, 8, 128, True, VOCAB, 1e6, 1e-6),
    "8b": (4096, 12288, 32, 8, 128, False, VOCAB, 1e6, 1e-6),
    "14b": (5120, 17408, 40, 8, 128, False, VOCAB, 1e6, 1e-6),
}


# ---- the cases -------------------------------------------------------------------------------------------------
def _case(model, layers, batch, shortest, longest, new, dtype="bfloat16", sampling="greedy", kind="request", **more):
    return dict(kind=kind, model=model, layers=layers, dtype=dtype, batch=batch, shortest=shortest, longest=longest, new=new,
                sampling=sampling, **more)


def listed():
    return [
        # the smallest call there is: the tiny model of the first tests and examples, one short greedy request in float32;
        # nothing but launches and host time
        dict(_case("qwen3-tiny-a", 2, 1, 7, 7, 9, "float32", kind="generate"), name="tiny_generate_f32"),
        # the float32 path at real sizes: what someone runs to have reference logits of the whole model
        dict(_case("qwen3-0.6b", 28, 2, 201, 500, 8, "float32"), name="qwen3_0.6b_f32"),
        # one user's chat with a small model: a prompt of some length, then token after token
        dict(_case("qwen3-0.6b", 28, 1, 517, 517, 64, sampling="filtered"), name="qwen3_0.6b_b1"),
        # the headline workload: eight sequences behind 2,048-token prompts
        dict(_case("qwen3-0.6b", 28, 8, 2048, 2048, 64), name="qwen3_0.6b_b8"),
        # time to the first token of a 2,048-token prompt
        dict(_case("qwen3-0.6b", 28, 1, 2048, 2048, 0), name="qwen3_0.6b_prompt"),
        # a ragged batch of eight prompts at the sizes of a mid-sized model
        dict(_case("qwen3-8b", 8, 8, 128, 2048, 32), name="qwen3_8b_ragged"),
        # a full batch of a larger model
        dict(_case("qwen3-14b", 4, 64, 512, 512, 32, sampling="filtered"), name="qwen3_14b_b64"),
        # the other architectures: retention, delta rule and routed experts; one long prompt
        dict(_case("levolix", 6, 1, 2048, 2048, 16, width=2048), name="levolix_long"),
        # state space, mLSTM, windowed attention with block means; a few ragged prompts
        dict(_case("sominex", 6, 4, 203, 1501, 16, width=2048), name="sominex_ragged"),
        # two maps, selective scan, capped attention; a batch of eight at the smallest width
        dict(_case("mopitar", 6, 8, 100, 900, 32, width=1024), name="mopitar_b8"),
        # latent attention, linear attention with a decay per channel, routed experts; the largest width
        dict(_case("kubedra", 6, 8, 256, 1024, 32, width=4096), name="kubedra_wide"),
        # several residual streams, time mixing, rotated latents; a prompt of odd length
        dict(_case("nekotar", 6, 2, 333, 1777, 32, width=2048, sampling="filtered"), name="nekotar_b2"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    which = rng.choice(["tiny", "f32", "0.6b", "0.6b", "0.6b", "large", "large", "levolix", "sominex", "mopitar", "kubedra", "nekotar"])
    sampling = rng.choice(["greedy", "filtered"])
    if which == "tiny":
        name, most = rng.choice([("a", 40), ("b", 100)])
        long = log_int(2, most)
        return _case("qwen3-tiny-" + name, 2 if name == "a" else 3, rng.randint(1, 4), log_int(1, long), long, rng.randint(4, 20),
                     "float32", kind="generate")
    if which == "f32":
        long = log_int(16, 700)
        return _case("qwen3-0.6b", rng.randint(4, 28), rng.randint(1, 3), log_int(8, long), long, rng.randint(2, 8), "float32")
    if which == "0.6b":
        batch = rng.choice([1, 1, 2, 3, 5, 8, 8, 13, 16])
        long = log_int(30, min(4096, 16384 // batch))
        return _case("qwen3-0.6b", 28, batch, log_int(20, long), long, rng.choice([0, log_int(4, 64)]), sampling=sampling)
    if which == "large":
        size, layers, batch = rng.choice([("8b", rng.randint(3, 8), log_int(1, 64)), ("14b", rng.randint(2, 4), log_int(1, 64))])
        long = log_int(60, min(3000, 20000 // batch))
        return _case("qwen3-" + size, layers, batch, log_int(40, long), long, log_int(4, 32), sampling=sampling)
    width = rng.choice([1024, 2048, 2048, 4096])
    batch = rng.choice([1, 1, 2, 3, 4, 8, 11])
    long = log_int(40, min(3000, 8192 // batch))
    return _case(which, 6, batch, log_int(30, long), long, log_int(4, 32), sampling=sampling, width=width)


# ---- configurations --------------------------------------------------------------------------------------------
def _qwen3(size, layers):
    width, ff, heads, kv, dim, tied, vocab, theta, eps = QWEN3[size]
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=width, intermediate_size=ff, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=kv, head_dim=dim, vocab_size=vocab, rope_theta=theta,
                rms_norm_eps=eps, tie_word_embeddings=tied,
                max_position_embeddings={"tiny-a": 64, "tiny-b": 128}.get(size, 40960))


def _levolix(w, layers):
    mlp = dict(kind="moe", expert=dict(ff=3 * w // 4), router=dict(experts=16, identity=2, top=4))
    out = []
    for i in range(layers):
        if i % 3 < 2:
            H = w // 256
            out.append(dict(type="retention", mlp=mlp, mixer=dict(
                heads=H, dim=128, vdim=256, decay=[1.0 - 2.0 ** (-5 - 6.0 * h / max(1, H - 1)) for h in range(H)],
                rot=dict(dims=128, base=1e6))))
        else:
            left = dict(heads=w // 128, kv_heads=4 if w == 1024 else 8, dim=128, vdim=128, mask=dict(size=512),
                        rot=dict(dims=128, base=5e4), scale=128 ** -0.5)
            right = dict(heads=w // 256, kv_heads=max(w // 512, 1), dim=128, vdim=128, conv=4)
            out.append(dict(type="parallel", mlp=mlp, mixer=dict(left=left, right=right, left_scale=1.0, right_scale=1.0)))
    return dict(architecture="Levolix", width=w, vocab=VOCAB, norm=dict(eps=1e-6), layers=out)


def _sominex(w, layers):
    dense = dict(kind="dense", ff=3 * w, limit=7.0)
    routed = dict(kind="moe", expert=dict(ff=3 * w // 4), router=dict(experts=16, top=2, scale=2.5), shared=dict(ff=3 * w // 2))
    out = []
    for i in range(layers):
        if i % 3 == 0:
            kind, mixer = "attention", dict(
                heads=w // 128, kv_heads=4 if w == 1024 else 8, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=512, pool=64),
                rot=dict(dims=64, base=1e6, scaling=dict(factor=4.0, original=2048, fast=32.0, slow=1.0)))
        elif i % 3 == 1:
            groups = 4 if w == 1024 else 8
            kind, mixer = "mamba2", dict(heads=w // 32, groups=groups, state=128, vdim=64, conv=4, norm_groups=groups)
        else:
            kind, mixer = "mlstm", dict(heads=w // 256, dim=128, vdim=256, gate_cap=15.0)
        out.append(dict(type=kind, mixer=mixer, mlp=routed if i % 2 else dense))
    return dict(architecture="Sominex", width=w, vocab=VOCAB, norm=dict(eps=1e-5), embedding=dict(scale=1.0), layers=out)


def _mopitar(w, layers):
    H = w // 128
    G, lender, out = max(H // 4, 1), None, []
    dense = dict(kind="dense", ff=9 * w // 2)
    routed = dict(kind="moe", expert=dict(ff=3 * w // 4), shared=dict(ff=3 * w // 2),
                  router=dict(experts=16, top=2, groups=dict(count=4, keep=2)))
    for i in range(layers):
        if i % 3 == 0:
            kind, mixer = "attention_2", dict(
                heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, diff=0.5, mask=dict(size=512, keep_first=8),
                rot=dict(dims=64, base=1e6, scaling=dict(factor=4.0, original=2048, fast=32.0, slow=1.0)))
        elif i % 3 == 1:
            left = dict(heads=max(H // 2, 1), kv_heads=max(G // 2, 1), dim=128, vdim=128, scale=0.09, softcap=40.0,
                        rot=dict(dims=128, base=5e5))
            right = dict(inner=2 * w, state=16, dt_rank=max(w // 16, 8), conv=4)
            kind, mixer = "parallel", dict(left=left, right=right, left_scale=1.0, right_scale=1.0)
        else:
            kind, mixer = "attention", dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, softcap=20.0,
                                            rot=dict(dims=128, base=1e4))
            if lender is None:
                lender = i
            else:
                mixer["kv_from"] = lender
        out.append(dict(type=kind, mixer=mixer, mlp=routed if i % 2 else dense))
    return dict(architecture="Mopitar", width=w, vocab=VOCAB, norm=dict(eps=1e-6), layers=out)


def _kubedra(w, layers):
    moe = dict(kind="moe", expert=dict(ff=3 * w // 4, limit=7.0), router=dict(experts=16, top=3), shared=dict(ff=w, limit=7.0))
    out = []
    for i in range(layers):
        if i % 3:
            kind, mixer = "gla", dict(heads=w // 256, dim=128, vdim=256, tau=16.0)
        else:
            kind, mixer = "latent_attention", dict(heads=w // 128, dim=128, vdim=128, q_rank=w // 2, kv_rank=128,
                                                   scale=128 ** -0.5, mask=dict(size=512))
        out.append(dict(type=kind, mixer=mixer, mlp=moe if i else dict(kind="dense", ff=3 * w)))
    return dict(architecture="Kubedra", width=w, vocab=VOCAB, max_positions=8192, norm=dict(eps=1e-6), layers=out)


def _nekotar(w, layers):
    H, out, lender = w // 128, [], None
    for i in range(layers):
        if i % 3 == 0:
            kind, mixer = "latent_attention", dict(heads=H, dim=128, vdim=128, kv_rank=96, rot_dim=32, scale=160 ** -0.5,
                                                   rot=dict(base=1e4, dims=32))
            if lender is None:
                lender = i
            else:
                mixer["kv_from"], lender = lender, None
        elif i % 3 == 1:
            kind, mixer = "wkv", dict(heads=w // 64, dim=64)
        else:
            kind, mixer = "attention", dict(heads=H, kv_heads=max(H // 4, 1), dim=128, vdim=128, scale=128 ** -0.5,
                                            rot=dict(base=1e6, dims=128), mask=dict(size=512, keep_first=8))
        out.append(dict(type=kind, mixer=mixer, mlp=dict(kind="dense", ff=9 * w // 2)))
    return dict(architecture="Nekotar", width=w, vocab=VOCAB, streams=2, residual_mult=0.7, norm=dict(eps=1e-5), layers=out)


def _config(case):
    if case["model"].startswith("qwen3-"):
        return _qwen3(case["model"][6:], case["layers"])
    return {"levolix": _levolix, "sominex": _sominex, "mopitar": _mopitar, "kubedra": _kubedra,
            "nekotar": _nekotar}[case["model"]](case["width"], case["layers"])


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _lengths(case):
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    return [hi] if n == 1 else [lo + round((hi - lo) * i / (n - 1)) for i in range(n)]


def _tokens(case, seed):
    """(the prompts, the tokens fed behind them step by step), lists of ids."""
    g = torch.Generator().manual_seed(1000003 * int(seed) + 17)
    vocab = _vocab(_config(case))
    prompts = [torch.randint(vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return prompts, torch.randint(vocab, (case["new"], case["batch"]), generator=g).tolist()


def _weights(spec, case, seed):
    """Random weights by checkpoint name, those of ``LLM.random`` but for two things that training gives a model and without
    which rounding alone makes two correct runs differ.  Routers are four times as wide as other matrices: their choices
    stay as they are, but the last chosen expert, which rounding often swaps for the next, weighs little.  Where every
    sublayer's output is normed before it joins the stream (Levolix, Kubedra), embeddings are of size one and the norms'
    multipliers of size one eighth, so that sublayers add to the stream instead of replacing it."""
    from gguf2bin_b200.engine.model import expected_tensors
    from gguf2bin_b200.weights.random_init import random_tensors_on_device
    dtype = getattr(torch, case["dtype"])
    tensors = random_tensors_on_device(expected_tensors(spec), int(seed), dtype, dtype, "cuda:0")
    behind = {"levolix": (".norm1", ".norm2"), "kubedra": (".norm1b", ".norm2b")}.get(case["model"])
    for name, t in tensors.items():
        if name.endswith(".router"):
            t.mul_(4.0)
        elif behind and name == "embed":
            t.mul_(50.0)
        elif behind and name.endswith(behind):
            t.sub_(0.875)                  # stored as the distance from one
    return tensors


# ---- a pass ----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """The loaded model with its cache, and the token ids on the host."""
    from gguf2bin_b200.api import LLM
    from gguf2bin_b200.config import model_spec_from_dict
    from gguf2bin_b200.engine import Model
    lengths = _lengths(case)
    prompts, fed = _tokens(case, seed)
    room = sum(64 * (-(-(n + case["new"]) // 64)) for n in lengths)
    spec = model_spec_from_dict(_config(case))
    model = Model(spec, case["dtype"], "cuda:0")
    model.bind(_weights(spec, case, seed))
    return dict(case=case, llm=LLM(model=model, max_tokens=room, max_seqs=case["batch"] + 1), prompts=prompts, fed=fed)


def run(state):
    from gguf2bin_b200.api import SamplingParams, StepEntry
    from gguf2bin_b200.engine import DecodeSession
    from gguf2bin_b200.sampling import Sampler
    case, llm, prompts, fed = state["case"], state["llm"], state["prompts"], state["fed"]
    if case["kind"] == "generate":
        outs = llm.generate(prompts, n=case["new"], temperature=0.0, top_k=0, top_p=1.0, repeat_penalty=1.0, ignore_eos=True)
        return torch.tensor([o.tokens for o in outs])
    engine, seqs = llm.engine, []
    try:
        for p in prompts:
            seqs.append(llm.open_sequence())
            engine.cache.reserve(seqs[-1], len(p) + case["new"])
        logits = llm.step([StepEntry(s, p, (len(p) - 1,)) for s, p in zip(seqs, prompts)])
        if not fed:
            engine.check()                 # as a caller does who hands the logits on
            return [logits]
        out = [logits.clone()]             # the step's logits are scratch memory
        sampler = Sampler(engine.cache.seq_state, engine.device)
        sampler.seed([s.slot for s in seqs], range(len(seqs)), 0)
        session = DecodeSession(engine, seqs, sampler, SamplingParams(*(FILTERED if case["sampling"] == "filtered" else GREEDY)))
        for tokens in fed:
            session.set_tokens(tokens)
            session.run()
        session.read_tokens()
        session.check()
        return out + [session.logits]
    finally:
        for s in seqs:
            llm.close_sequence(s)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _pairs(n, window, keep=0, chunk=0, pool=0):
    """(query, key) pairs of a sequence of n tokens."""
    if chunk:
        full, rest = divmod(n, chunk)
        return full * chunk * (chunk + 1) / 2 + rest * (rest + 1) / 2
    if not window or n <= window:
        return n * (n + 1) / 2
    beyond = n - window
    return window * (window + 1) / 2 + beyond * (window + min(keep, beyond)) + (beyond * beyond / 2 / pool if pool else 0)


def _mixers(cfg):
    """Of every layer's attentions and states: (flops a pair, bytes of a kept token, window, keep, chunk, pool) and
    (state entries)."""
    attn, states = [], []
    if "layers" not in cfg:
        H, G, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [(4 * H * D, 2 * G * D, 0, 0, 0, 0)] * cfg["num_hidden_layers"], states
    for layer in cfg["layers"]:
        m, kind = layer["mixer"], layer["type"]
        mask = m.get("mask") or {}
        if kind in ("retention", "gla", "mlstm"):
            states.append(m["heads"] * m["dim"] * (m["vdim"] + (kind == "mlstm")))
        elif kind == "mamba2":
            states.append(m["heads"] * m["state"] * m["vdim"])
        elif kind == "wkv":
            states.append(m["heads"] * m["dim"] * m["dim"])
        elif kind == "parallel":
            left, right = m["left"], m["right"]
            attn.append((4 * left["heads"] * left["dim"], 2 * left["kv_heads"] * left["dim"], 0, 0,
                         (left.get("mask") or {}).get("size", 0), 0))
            states.append(right["inner"] * right["state"] if "inner" in right else right["heads"] * right["dim"] * right["vdim"])
        elif kind == "latent_attention":
            r, rot = m["kv_rank"], m.get("rot_dim", 0)
            attn.append((2 * m["heads"] * (2 * r + rot), r + rot, mask.get("size", 0), 0, 0, 0))
        else:
            two = 2 if kind == "attention_2" else 1
            attn.append((4 * two * m["heads"] * m["dim"], (1 + two) * m["kv_heads"] * m["dim"], mask.get("size", 0),
                         mask.get("keep_first", 0), 0, mask.get("pool", 0)))
    return attn, states


def work(case):
    from gguf2bin_b200.config import model_spec_from_dict
    from gguf2bin_b200.engine.model import expected_tensors
    cfg = _config(case)
    size = 4 if case["dtype"] == "float32" else 2
    lengths, B, new = _lengths(case), case["batch"], case["new"]
    prompt_tokens = sum(lengths)
    head = _vocab(cfg) * (cfg.get("hidden_size") or cfg["width"])
    dense = experts = 0                       # parameters of the layers; the vocabulary's matrix apart
    E = top = 1
    for name, e in expected_tensors(model_spec_from_dict(cfg)).items():
        n = math.prod(e.shape)
        if e.optional or n >= head or len(e.shape) != 2:
            continue
        if ".mlp.e" in name:
            experts += n
        else:
            dense += n
    for layer in cfg.get("layers", ()):
        if (layer.get("mlp") or {}).get("kind") == "moe":
            E, top = layer["mlp"]["router"]["experts"], layer["mlp"]["router"]["top"]
    attn, states = _mixers(cfg)

    def weights(tokens):
        return size * (dense + experts * (1.0 - (1.0 - min(1.0, top / E)) ** tokens) + head)
    steps = new - 1 if case["kind"] == "generate" else new
    by = weights(prompt_tokens) + steps * weights(B)
    fl = 2.0 * (prompt_tokens + steps * B) * (dense + experts * min(1.0, top / E)) + 2.0 * B * (1 + steps) * head
    by += 4.0 * B * _vocab(cfg) * 2 + 4.0 * prompt_tokens + size * (prompt_tokens + steps * B) * (cfg.get("hidden_size") or cfg["width"])
    for per_pair, kept, window, keep, chunk, pool in attn:
        for n in lengths:
            fl += per_pair * _pairs(n + steps, window, keep, chunk, pool)
            seen = sum(min(t + 1, window + keep if window else t + 1, t % chunk + 1 if chunk else t + 1)
                       + (max(0, t + 1 - window) // pool if pool else 0) for t in range(n, n + steps))
            by += size * kept * (n + steps + seen)
    for entries in states:
        fl += 4.0 * entries * (prompt_tokens + steps * B)
        by += 8.0 * entries * B * (steps + 1)
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """About four times what whole models of these depths show against 64 bits: float32 2.6e-6, bfloat16 0.004 to 0.021; up to
    0.053 where a router picks experts and rounding sends some tokens to others."""
    if case["kind"] == "generate":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.2 if case["model"] in ("levolix", "sominex", "mopitar", "kubedra") else 0.08}


# ---- the same in 64 bits, by plain torch --------------------------------------------------------------------------
def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _angles(positions, dims, base, scaling=None):
    i = torch.arange(dims // 2, dtype=torch.float64, device=positions.device)
    f, mult = base ** (-2.0 * i / dims), 1.0
    if scaling:
        factor, original = scaling["factor"], scaling["original"]

        def pair(turns):
            return dims * math.log(original / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, mult = f / factor * ramp + f * (1.0 - ramp), 0.1 * math.log(factor) + 1.0
    a = positions.double()[:, None] * f
    return (a.cos() * mult)[:, None], (a.sin() * mult)[:, None]


def _turn(x, rot, neighbours):
    """x [T, heads, D]: the first rot.dims entries of every head turn in pairs of neighbours or of halves."""
    dims = rot["dims"]
    c, s = _angles(torch.arange(x.shape[0], device=x.device), dims, rot["base"], rot.get("scaling"))
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :dims // 2], x[..., dims // 2:dims])
    u, v = a * c - b * s, b * c + a * s
    out = torch.stack([u, v], -1).flatten(-2) if neighbours else torch.cat([u, v], -1)
    return torch.cat([out, x[..., dims:]], -1)


def _attend(q, k, v, scale, window=0, keep=0, chunk=0, pool=0, cap=0.0, sink=None, empty=False):
    """q [T, H, D], k [T, G, D], v [T, G, V] of one sequence -> [T, H V]."""
    T, H = q.shape[:2]
    per = H // k.shape[1]
    i = torch.arange(T, device=q.device)
    d = i[:, None] - i[None, :]
    see = d >= 0
    if window:
        see = see & ((d < window) | (i[None, :] < keep))
    if chunk:
        see = see & (i[:, None] // chunk == i[None, :] // chunk)
    blocks = T // pool if pool else 0
    if blocks:
        k = torch.cat([k, k[:blocks * pool].unflatten(0, (blocks, pool)).mean(1)])
        v = torch.cat([v, v[:blocks * pool].unflatten(0, (blocks, pool)).mean(1)])
        ends = torch.arange(blocks, device=q.device) * pool + pool - 1
        see = torch.cat([see, ends[None, :] <= i[:, None] - window], 1)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // per].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~see, -math.inf)
        if sink is not None or empty:           # one more term of the denominator, without a value
            s = torch.cat([s, (sink[h] if sink is not None else s.new_zeros(())).expand(T, 1)], 1)
            out.append(s.softmax(1)[:, :-1] @ v[:, h // per])
        else:
            out.append(s.softmax(1) @ v[:, h // per])
    return torch.stack(out, 1).flatten(1)


def _conv(x, w, b=None):
    T, taps = x.shape[0], w.shape[1]
    full = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(full[j:j + T] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _scan(q, k, v, decay, delta=None, bonus=None):
    """q, k [T, H, D], v [T, H, V], decay [T, H, 1 or D]: S = diag(decay) S + k v^T, o = S^T q, a token at a time.
    ``delta``: beta [T, H], v is replaced by beta (v - S^T k).  ``bonus`` u [H, D]: o reads S + diag(u) k v^T before S moves."""
    S = q.new_zeros(q.shape[1], q.shape[2], v.shape[2])
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        kt, vt = k[t].unsqueeze(-1), v[t].unsqueeze(1)
        if bonus is not None:
            kv = kt * vt
            out[t] = ((S + bonus.unsqueeze(-1) * kv) * q[t].unsqueeze(-1)).sum(1)
            S = decay[t].unsqueeze(-1) * S + kv
            continue
        S = decay[t].unsqueeze(-1) * S
        if delta is not None:
            vt = delta[t][:, None, None] * (vt - (S * kt).sum(1, keepdim=True))
        S = S + kt * vt
        out[t] = (S * q[t].unsqueeze(-1)).sum(1)
    return out


def _silu(x):
    return torch.nn.functional.silu(x)


def _softplus(x):
    return torch.logaddexp(x.new_zeros(()), x)


def _glu(h, w, pre, act=_silu):
    return (act(h @ w(pre + "gate").T) * (h @ w(pre + "up").T)) @ w(pre + "down").T


def _capped(h, w, pre, limit):
    g, u = (h @ w(pre + "gate").T).clamp(max=limit), (h @ w(pre + "up").T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(pre + "down").T


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _experts(h, w, pre, pick, weight, top, expert, identity_from=None):
    """The ``top`` experts with the largest ``pick`` [T, E], each times its ``weight`` [T, E] entry."""
    chosen = pick.topk(top, -1).indices
    out = torch.zeros_like(h)
    for e in range(pick.shape[1]):
        rows = (chosen == e).any(-1).nonzero().squeeze(-1)
        if len(rows):
            y = h[rows] if identity_from is not None and e >= identity_from else expert(h[rows], f"{pre}e{e}.")
            out[rows] += weight[rows, e, None] * y
    return out


def _exact_qwen3(cfg, w, ids, rows):
    H, G, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    rot = dict(dims=D, base=cfg["rope_theta"])
    x = w("model.embed_tokens.weight", ids)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(a + n + "_proj.weight").T).unflatten(1, (-1, D)) for n in "qkv")
        q = _turn(_rms(q, eps) * w(a + "q_norm.weight"), rot, False)
        k = _turn(_rms(k, eps) * w(a + "k_norm.weight"), rot, False)
        x = x + _attend(q, k, v, D ** -0.5) @ w(a + "o_proj.weight").T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        m = p + "mlp."
        x = x + (_silu(h @ w(m + "gate_proj.weight").T) * (h @ w(m + "up_proj.weight").T)) @ w(m + "down_proj.weight").T
    x = _rms(x[rows], eps) * w("model.norm.weight")
    return x, "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"


def _exact_levolix(cfg, w, ids, rows):
    eps, x = cfg["norm"]["eps"], w("embed", ids)
    T = len(ids)
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        if layer["type"] == "retention":
            H, D = m["heads"], m["dim"]
            q, k, v = ((x @ w(p + n).T).unflatten(1, (H, -1)) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=x.device)[None, :, None].expand(T, H, 1)
            o = _rms(_scan(_turn(q, m["rot"], False), _turn(k, m["rot"], False) * D ** -0.5, v, decay), eps).flatten(1)
            y = (o * _silu(x @ w(p + "g").T)) @ w(p + "o").T
        else:
            a, n = m["left"], p + "left."
            q, k, v = (x @ w(n + c).T + w(n + c + ".b") for c in "qkv")
            q = _turn((_rms(q, eps) * w(n + "q.norm")).unflatten(1, (a["heads"], -1)), a["rot"], True)
            k = _turn((_rms(k, eps) * w(n + "k.norm")).unflatten(1, (a["kv_heads"], -1)), a["rot"], True)
            o = _attend(q, k, v.unflatten(1, (a["kv_heads"], -1)), a["scale"], chunk=a["mask"]["size"], empty=True)
            y = m["left_scale"] * ((o * torch.sigmoid(x @ w(n + "g").T)) @ w(n + "o").T)
            a, n = m["right"], p + "right."
            H, G, D = a["heads"], a["kv_heads"], a["dim"]
            q, k, v = (_silu(_conv(x @ w(n + c).T, w(n + c + ".conv"))) for c in "qkv")
            q, k = (z.unflatten(1, (G, D)).repeat_interleave(H // G, 1) for z in (q, k))
            q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5
            k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
            g = torch.exp(-torch.exp(w(n + "A_log")) * _softplus(x @ w(n + "a").T + w(n + "dt_bias")))
            o = _scan(q, k, v.unflatten(1, (H, -1)), g.unsqueeze(-1), delta=torch.sigmoid(x @ w(n + "b").T))
            o = (_rms(o, eps) * w(n + "norm")).flatten(1) * _silu(x @ w(n + "g").T)
            y = y + m["right_scale"] * (o @ w(n + "o").T)
        x = x + _rms(y, eps) * (1.0 + w(f"l{i}.norm1"))
        r, n = layer["mlp"]["router"], f"l{i}.mlp."
        s = (x @ w(n + "router").T).softmax(-1)
        y = _experts(x, w, n, s + w(n + "correction"), s, r["top"], lambda h, pre: _glu(h, w, pre), r["experts"])
        x = x + _rms(y, eps) * (1.0 + w(f"l{i}.norm2"))
    return _rms(x[rows], eps) * (1.0 + w("final.norm")), "embed"


def _exact_sominex(cfg, w, ids, rows):
    eps, x = cfg["norm"]["eps"], w("embed", ids) * cfg["embedding"]["scale"]
    T = len(ids)
    for i, layer in enumerate(cfg["layers"]):
        m, p, kind = layer["mixer"], f"l{i}.mix.", layer["type"]
        h = _rms(x, eps) * w(f"l{i}.norm1")
        prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        hs = h + (prev - h) * w(f"l{i}.shift")
        if kind == "attention":
            q, k, v = ((hs @ w(p + c).T).unflatten(1, (n, -1)) for c, n in zip("qkv", (m["heads"], m["kv_heads"], m["kv_heads"])))
            y = _attend(_turn(q, m["rot"], False), _turn(k, m["rot"], False), _rms(v, eps), m["scale"], m["mask"]["size"],
                        pool=m["mask"]["pool"]) @ w(p + "o").T
        elif kind == "mamba2":
            H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            inner = H * V
            z, xBC, dt = (hs @ w(p + "in").T).split([inner, inner + 2 * G * N, H], 1)
            u, B, C = _silu(_conv(xBC, w(p + "conv"), w(p + "conv.b"))).split([inner, G * N, G * N], 1)
            u = u.unflatten(1, (H, V))
            B, C = (a.unflatten(1, (G, N)).repeat_interleave(H // G, 1) for a in (B, C))
            dt = _softplus(dt + w(p + "dt_bias"))
            y = _scan(C, B, dt[:, :, None] * u, torch.exp(-torch.exp(w(p + "A_log")) * dt).unsqueeze(-1)) + w(p + "D")[:, None] * u
            y = y.flatten(1) * _silu(z)
            y = (_rms(y.unflatten(1, (m["norm_groups"], -1)), eps).flatten(1) * w(p + "norm")) @ w(p + "o").T
        else:
            H, D, cap = m["heads"], m["dim"], m["gate_cap"]
            q, k, v = ((hs @ w(p + c).T).unflatten(1, (H, -1)) for c in "qkv")
            q = q * D ** -0.5
            ig = cap * torch.tanh((hs @ w(p + "i").T + w(p + "i.b")) / cap)
            fg = -_softplus(-(cap * torch.tanh((hs @ w(p + "f").T + w(p + "f.b")) / cap)))
            peak, a, b = ig.new_zeros(H), [], []
            peaks = []
            for t in range(T):
                new = torch.maximum(fg[t] + peak, ig[t])
                a.append(torch.exp(fg[t] + peak - new))
                b.append(torch.exp(ig[t] - new))
                peaks.append(new)
                peak = new
            a, b, peaks = torch.stack(a), torch.stack(b), torch.stack(peaks)
            o = _scan(q, b[:, :, None] * k, torch.cat([v, torch.ones_like(v[..., :1])], -1), a.unsqueeze(-1))
            o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-peaks).unsqueeze(-1)) + 1e-6)
            y = (_rms(o, eps).flatten(1) * w(p + "norm") * torch.sigmoid(hs @ w(p + "g").T)) @ w(p + "o").T
        mlp, n = layer["mlp"], f"l{i}.mlp."
        if mlp["kind"] == "dense":
            y = y + _capped(h, w, n, mlp["limit"])
        else:
            s = (h @ w(n + "router").T).softmax(-1)
            y = y + _experts(h, w, n, s, s * mlp["router"]["scale"], mlp["router"]["top"], lambda r, pre: _glu(r, w, pre))
            y = y + _glu(h, w, n + "shared.")
        x = x + y
    return _rms(x[rows], eps) * w("final.norm"), "head"


def _exact_mopitar(cfg, w, ids, rows):
    eps, x, kept = cfg["norm"]["eps"], w("embed", ids), {}

    def norm(z, n):
        return torch.tanh(w(n + ".alpha") * z) * w(n) + w(n + ".b")
    for i, layer in enumerate(cfg["layers"]):
        m, p, kind = layer["mixer"], f"l{i}.mix.", layer["type"]
        h = norm(x, f"l{i}.norm1")

        def heads(n, count):
            return (h @ w(n).T).unflatten(1, (count, -1))
        if kind == "attention":
            q = _turn(heads(p + "q", m["heads"]), m["rot"], True)
            if m.get("kv_from") is None:
                kept[i] = _turn(heads(p + "k", m["kv_heads"]), m["rot"], True), heads(p + "v", m["kv_heads"])
            k, v = kept[m.get("kv_from", i)]
            y = _attend(q, k, v, m["scale"], cap=m["softcap"], sink=w(p + "sink")) @ w(p + "o").T
        elif kind == "attention_2":
            H, G = m["heads"], m["kv_heads"]
            q = _turn(_rms(heads(p + "q", 2 * H), eps) * w(p + "q.norm"), m["rot"], True)
            k = _turn(_rms(heads(p + "k", 2 * G), eps) * w(p + "k.norm"), m["rot"], True)
            v = heads(p + "v", G)
            one, two = (_attend(q[:, j::2], k[:, j::2], v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"]) for j in (0, 1))
            lam = torch.exp(w(p + "lq1") @ w(p + "lk1")) - torch.exp(w(p + "lq2") @ w(p + "lk2")) + m["diff"]
            o = _rms((one - lam * two).unflatten(1, (H, -1)), eps) * (1.0 - m["diff"])
            y = o.flatten(1) @ w(p + "o").T
        else:
            a, n = m["left"], p + "left."
            q = _rms(_turn(heads(n + "q", a["heads"]), a["rot"], True), eps)
            k = _rms(_turn(heads(n + "k", a["kv_heads"]), a["rot"], True), eps)
            o = _attend(q, k, heads(n + "v", a["kv_heads"]), a["scale"], cap=a["softcap"]).unflatten(1, (a["heads"], -1))
            y = m["left_scale"] * ((o * torch.sigmoid(h @ w(n + "g").T).unsqueeze(-1)).flatten(1) @ w(n + "o").T)
            a, n = m["right"], p + "right."
            N, R = a["state"], a["dt_rank"]
            u, z = (h @ w(n + "in").T).chunk(2, 1)
            u = _silu(_conv(u, w(n + "conv"), w(n + "conv.b")))
            dt, B, C = (u @ w(n + "x").T).split([R, N, N], 1)
            dt = _softplus(dt @ w(n + "dt").T + w(n + "dt.b"))
            A = -torch.exp(w(n + "A_log"))
            S, o = torch.zeros_like(A), torch.empty_like(u)
            for t in range(len(ids)):
                S = torch.exp(dt[t, :, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
                o[t] = S @ C[t]
            y = y + m["right_scale"] * (((o + w(n + "D") * u) * _silu(z)) @ w(n + "o").T)
        y = y * w(f"l{i}.ls1")
        mlp, n = layer["mlp"], f"l{i}.mlp."
        if mlp["kind"] == "dense":
            f = (h @ w(n + "up").T).clamp(min=0.0).square() @ w(n + "down").T
        else:
            r, g = mlp["router"], mlp["router"]["groups"]
            s = torch.sigmoid(h @ w(n + "router").T)
            by_group = s.unflatten(1, (g["count"], -1))
            best = by_group.topk(2, -1).values.sum(-1).topk(g["keep"], -1).indices
            ok = torch.zeros_like(by_group[..., 0]).scatter_(1, best, 1.0)
            pick = s.masked_fill(ok.repeat_interleave(by_group.shape[2], 1) == 0, -1.0)
            total = pick.topk(r["top"], -1).values.sum(-1, keepdim=True)
            f = _experts(h, w, n, pick, s / (total + 1e-20), r["top"], lambda z, pre: _glu(z, w, pre)) + _glu(h, w, n + "shared.")
        x = x + (y + f * w(f"l{i}.ls2"))
    return norm(x[rows], "final.norm"), "head"


def _exact_kubedra(cfg, w, ids, rows):
    eps = cfg["norm"]["eps"]
    x = w("embed", ids) + w("pos")[:len(ids)]

    def norm(z, n):
        return _rms(z, eps) * (1.0 + w(n))
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        h, H = norm(x, f"l{i}.norm1"), m["heads"]
        if layer["type"] == "gla":
            q, k, v = ((h @ w(p + c).T).unflatten(1, (H, -1)) for c in "qkv")
            z = (h @ w(p + "a1").T) @ w(p + "a2").T + w(p + "a2.b")
            alpha = torch.exp(-_softplus(-z) / m["tau"]).unflatten(1, (H, -1))
            o = _rms(_scan(q * m["dim"] ** -0.5, k, v, alpha), eps) * w(p + "norm")
            y = (o.flatten(1) * _silu(h @ w(p + "g").T)) @ w(p + "o").T
        else:
            q = ((_rms(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).unflatten(1, (H, -1))
            c = _rms(h @ w(p + "dkv").T, eps) * w(p + "dkv.norm")
            k, v = ((c @ w(p + n).T).unflatten(1, (H, -1)) for n in ("uk", "uv"))
            y = _attend(q, k, v, m["scale"], m["mask"]["size"]) @ w(p + "o").T
        x = x + norm(y, f"l{i}.norm1b")
        h, mlp, n = norm(x, f"l{i}.norm2"), layer["mlp"], f"l{i}.mlp."
        if mlp["kind"] == "dense":
            y = _glu(h, w, n, _gelu)
        else:
            z, top = h @ w(n + "router").T + w(n + "router.b"), mlp["router"]["top"]
            least = z.topk(top, -1).values[:, -1:]
            weight = z.masked_fill(z < least, -math.inf).softmax(-1)
            y = _experts(h, w, n, z, weight, top, lambda r, pre: _capped(r, w, pre, mlp["expert"]["limit"]))
            y = y + _capped(h, w, n + "shared.", mlp["shared"]["limit"])
        x = x + norm(y, f"l{i}.norm2b")
    return norm(x[rows], "final.norm"), "embed"


def _exact_nekotar(cfg, w, ids, rows):
    eps, mult, kept = cfg["norm"]["eps"], cfg["residual_mult"], {}
    X = (_rms(w("embed", ids), eps) * w("embed.norm")).expand(cfg["streams"], -1, -1)

    def sublayer(X, hc, norm, f):
        y = f(_rms(torch.einsum("s,stw->tw", w(hc + "in"), X), eps) * w(norm))
        return torch.einsum("st,sij->tij", w(hc + "mix"), X) + mult * w(hc + "out")[:, None, None] * y

    def mixer(h, i, m, kind, p):
        if kind == "wkv":
            prev, H = torch.cat([torch.zeros_like(h[:1]), h[:-1]]), m["heads"]
            mixed = {c: h + (prev - h) * w(p + "mu." + c) for c in "rkvgw"}
            r, k, v = ((mixed[c] @ w(p + c).T).unflatten(1, (H, -1)) for c in "rkv")
            decay = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).unflatten(1, (H, -1))
            o = _rms(_scan(r, k, v, decay, bonus=w(p + "u")), eps).flatten(1)
            return (o * w(p + "norm") * _silu(mixed["g"] @ w(p + "g").T)) @ w(p + "o").T
        gate = torch.sigmoid(h @ w(p + "g").T)
        if kind == "attention":
            q, k, v = ((h @ w(p + c).T + w(p + c + ".b")).unflatten(1, (n, -1))
                       for c, n in zip("qkv", (m["heads"], m["kv_heads"], m["kv_heads"])))
            o = _attend(_turn(q, m["rot"], False), _turn(k, m["rot"], False), v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"])
            return (o * gate) @ w(p + "o").T
        H, D, rot = m["heads"], m["dim"], dict(dims=m["rot_dim"], base=m["rot"]["base"])
        q = (h @ w(p + "q").T).unflatten(1, (H, -1))
        q = torch.cat([q[..., :D], _turn(q[..., D:], rot, True)], -1)
        if m.get("kv_from") is None:
            c, kr = (h @ w(p + "dkv").T).split([m["kv_rank"], m["rot_dim"]], 1)
            kept[i] = _rms(c, eps) * w(p + "dkv.norm"), _turn(kr[:, None], rot, True)
        c, kr = kept[m.get("kv_from", i)]
        k, v = ((c @ w(p + n).T).unflatten(1, (H, -1)) for n in ("uk", "uv"))
        return (_attend(q, torch.cat([k, kr.expand(-1, H, -1)], -1), v, m["scale"]) * gate) @ w(p + "o").T

    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        X = sublayer(X, p + "hc1.", p + "norm1", lambda h: mixer(h, i, layer["mixer"], layer["type"], p + "mix."))
        X = sublayer(X, p + "hc2.", p + "norm2", lambda h: _gelu(h @ w(p + "mlp.up").T) @ w(p + "mlp.down").T)
    return _rms(X.sum(0)[rows], eps) * w("final.norm"), "head"


def exact(case, seed):
    from gguf2bin_b200.config import model_spec_from_dict
    cfg = _config(case)
    forward = {"levolix": _exact_levolix, "sominex": _exact_sominex, "mopitar": _exact_mopitar, "kubedra": _exact_kubedra,
               "nekotar": _exact_nekotar}.get(case["model"], _exact_qwen3)
    tensors = _weights(model_spec_from_dict(cfg), case, seed)      # the weights are inputs: the model's, from the same seed

    def w(name, ids=None):
        return (tensors[name] if ids is None else tensors[name][ids]).double()

    def logits(sequence, rows):
        ids = torch.tensor(sequence, device="cuda:0")
        x, head = forward(cfg, w, ids, torch.tensor(rows, device="cuda:0"))
        return torch.cat([x @ part.double().T for part in tensors[head].split(16384)], 1)
    prompts, fed = _tokens(case, seed)
    with torch.no_grad():
        if case["kind"] == "generate":
            outs = []
            for p in prompts:
                seq = list(p)
                for _ in range(case["new"]):
                    seq.append(int(logits(seq, [len(seq) - 1])[0].argmax()))
                outs.append(seq[len(p):])
            return torch.tensor(outs)
        both = [logits(p + [step[b] for step in fed], [len(p) - 1, len(p) + len(fed) - 1][:1 + bool(fed)]) for b, p in enumerate(prompts)]
        return [torch.stack([r[k] for r in both]) for k in range(1 + bool(fed))]
