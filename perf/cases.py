"""The work this framework is measured on: calls of its public entry points as a user's program makes them.

Engine (Model / Session on a synthetic model directory, greedy sampling):
  chat     a conversation of two turns: batched prefill of the prompt, generated tokens, the second message
           (positions > 0: the one-token path), generated tokens; the last step's logits are read
  prompt   a prompt is scored: batched prefill, the next token and all logits of the last position
  step     one more token of a conversation that is already long
  swap     a server parks conversations: a saved one comes in (restore), and is saved again (snapshot)
Attention library (AttnContext on caller-owned activations):
  dispatch one layer, the three separate calls of a decode step
  layers   one token through all layers, one fused call per layer, activations on the device
  host     one token through all layers as one call, activations in pinned host memory
  prefill  a batch through all layers: Q norm + RoPE, cache write, causal attention

Shapes are the repository's: BONSAI_8B and TINY of bonsai_pot_b200.model_dir, 32 query / 8 KV heads of 128, and
the KV-head shards of 2, 4 and 8 GPUs (one rank's share of the heads, without the exchange).
"""
import os
import tempfile

import numpy as np
import torch

import bonsai_pot_b200 as bp
from bonsai_pot_b200 import model_dir
from bonsai_pot_b200.model import GenerateOptions, Sampler

SHAPES = {"bonsai8b": model_dir.BONSAI_8B, "tiny": model_dir.TINY}
N_LAYER, HEAD_DIM = 36, 128
GREEDY = Sampler(temperature=0.0, top_k=1)
MODEL_SEQ = 1024  # positions of the engine's cache; `step` cases size theirs by the position


def listed():
    return [
        # the smallest conversation: launches, host work and latency are all of it
        dict(name="chat_tiny", kind="chat", shape="tiny", prompt=7, follow=3, new=8),
        # a short question and a follow-up, the most frequent use of the engine
        dict(name="chat_21_12", kind="chat", shape="bonsai8b", prompt=21, follow=12, new=16),
        # a paragraph as the prompt, a ragged batch
        dict(name="prompt_173", kind="prompt", shape="bonsai8b", prompt=173),
        # the benchmark's prompt (pp512), the largest batch a model takes
        dict(name="prompt_512", kind="prompt", shape="bonsai8b", prompt=512),
        # a token late in a long conversation
        dict(name="step_8191", kind="step", shape="bonsai8b", pos=8191),
        # save / resume of a conversation of 512 tokens
        dict(name="swap_512", kind="swap", shape="bonsai8b", pos=512),
        # single layer, 512 past tokens, the reference's three dispatches
        dict(name="dispatch_512", kind="dispatch", ctx=513, shards=1),
        # the whole decode stack for a host that keeps its activations in host memory
        dict(name="host_4096", kind="host", ctx=4096, shards=1),
        # the benchmark's long context
        dict(name="layers_32768", kind="layers", ctx=32768, shards=1),
        # the same on one of four GPUs
        dict(name="layers_32768_quarter", kind="layers", ctx=32768, shards=4),
        # batched prefill, the engine's batch limit and the library's longer one
        dict(name="prefill_512", kind="prefill", m=512, shards=1),
        dict(name="prefill_2048", kind="prefill", m=2048, shards=1),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["chat", "prompt", "step", "swap", "dispatch", "host", "layers", "prefill"])
    shards = rng.choice([1, 1, 1, 2, 4, 8])
    if kind == "chat":
        return dict(kind=kind, shape=rng.choice(["tiny", "bonsai8b", "bonsai8b"]), prompt=_log(rng, 1, 128), follow=_log(rng, 1, 12),
                    new=rng.randint(2, 14))
    if kind == "prompt":
        return dict(kind=kind, shape="bonsai8b", prompt=_log(rng, 8, 512))
    if kind == "step":
        return dict(kind=kind, shape="bonsai8b", pos=_log(rng, 64, 16383))
    if kind == "swap":
        return dict(kind=kind, shape="bonsai8b", pos=_log(rng, 16, 512))
    if kind == "dispatch":
        return dict(kind=kind, ctx=_log(rng, 1, 4096), shards=shards)
    if kind == "host":
        return dict(kind=kind, ctx=_log(rng, 512, 32768), shards=shards)
    if kind == "layers":
        return dict(kind=kind, ctx=_log(rng, 256, 32768), shards=shards)
    return dict(kind=kind, m=_log(rng, 16, 2048), shards=shards)


# ---- what a program has in hand before the call -----------------------------------------------------------------
_models = {}


def _directory(shape):
    """The model directory of a shape: the weights do not depend on the case's seed, and a program loads them from
    disk. Written once per machine, under its final name only when complete."""
    path = os.path.join(tempfile.gettempdir(), "bonsai_pot_b200_%s_seed1" % shape)
    if not os.path.isdir(path):
        tmp = "%s.%d" % (path, os.getpid())
        model_dir.write_synthetic_model(tmp, shape=SHAPES[shape], seed=1)
        try:
            os.rename(tmp, path)
        except OSError:  # another process was first
            return tmp
    return path


def _model(shape):
    """The one loaded model a program serves its conversations from (each pass of the cases that share it sets the
    whole state it reads)."""
    if shape not in _models:
        _models[shape] = bp.Model(_directory(shape), max_seq=MODEL_SEQ)
    return _models[shape]


def _tokens(seed, stream, n, n_vocab):
    # the last id is the stop token: prompts do not hold it
    return np.random.default_rng([seed, stream]).integers(0, n_vocab - 1, n).astype(np.uint32)


def _heads(case):
    return 32 // case["shards"], 8 // case["shards"]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).half()


class _Buffer:
    """A device buffer of the library as something torch can view."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _view(ctx, ptr, shape, typestr):
    t = torch.as_tensor(_Buffer(ptr, shape, typestr), device="cuda")
    t.owner = ctx  # the memory is the context's: it lives as long as the view does
    return t


def _cache(ctx):
    """The cache as the library holds it: per buffer the FP32 block scales, then the int8 quants."""
    views = {}
    rows = ctx.n_layer * ctx.max_seq
    for kind, name in ((0, "k"), (1, "v")):
        base = ctx.kv_device_ptr(kind)
        views[name + "_scales"] = _view(ctx, base, (rows, ctx.nb), "<f4")
        views[name + "_quants"] = _view(ctx, base + rows * ctx.nb * 4, (rows, ctx.kv_dim), "|i1")
    return views


def _fill(ctx, g, rows):
    """Past tokens: N(0, 1) keys and values through the library's own cache write."""
    w = torch.ones(HEAD_DIM, dtype=torch.float16, device="cuda")
    for il in range(ctx.n_layer):
        for r0 in range(0, rows, 8192):
            m = min(8192, rows - r0)
            ctx.dispatch_kv_writeback_fused(il, _normal(g, m, ctx.kv_dim), _normal(g, m, ctx.kv_dim), w, r0, m)
    torch.cuda.synchronize()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chat":
        m = _model(case["shape"])
        v = m.cfg.n_vocab
        return dict(case=case, model=m, session=m.new_session(), prompt=_tokens(seed, 0, case["prompt"], v),
                    follow=_tokens(seed, 1, case["follow"], v),
                    options=GenerateOptions(max_new_tokens=case["new"], stop_pred=lambda _t: False, sampler=GREEDY))
    if kind == "prompt":
        m = _model(case["shape"])
        return dict(case=case, model=m, session=m.new_session(), prompt=_tokens(seed, 0, case["prompt"], m.cfg.n_vocab))
    if kind == "swap":
        m = _model(case["shape"])
        s = m.new_session()
        s.prefill(_tokens(seed, 0, case["pos"], m.cfg.n_vocab), GREEDY)
        return dict(case=case, session=s, saved=s.snapshot())
    if kind == "step":
        m = bp.Model(_directory(case["shape"]), max_seq=case["pos"] + 1)
        attention = m.attention()
        attention.model = m  # owns the cache
        _fill(attention, _gen(seed), case["pos"] + 1)
        return dict(case=case, model=m, attention=attention, token=int(_tokens(seed, 0, 1, m.cfg.n_vocab)[0]))
    n_head, n_kv = _heads(case)
    g = _gen(seed)
    n_layer = 1 if kind == "dispatch" else N_LAYER
    w = torch.ones(HEAD_DIM, dtype=torch.float16, device="cuda")
    if kind == "prefill":
        rows = case["m"]
        ctx = bp.AttnContext(n_layer=n_layer, n_head=n_head, n_kv_head=n_kv, max_seq=rows, max_prefill=rows, n_shards=case["shards"])
        qkv = [(_normal(g, rows, ctx.q_dim), _normal(g, rows, ctx.kv_dim), _normal(g, rows, ctx.kv_dim)) for _ in range(n_layer)]
        out = torch.zeros(n_layer, rows, ctx.q_dim, dtype=torch.float16, device="cuda")
        return dict(case=case, ctx=ctx, qkv=qkv, w=w, out=out)
    ctx = bp.AttnContext(n_layer=n_layer, n_head=n_head, n_kv_head=n_kv, max_seq=case["ctx"], n_shards=case["shards"])
    _fill(ctx, g, case["ctx"])
    q, k, v = _normal(g, n_layer, ctx.q_dim), _normal(g, n_layer, ctx.kv_dim), _normal(g, n_layer, ctx.kv_dim)
    out = torch.zeros(n_layer, ctx.q_dim, dtype=torch.float16, device="cuda")
    if kind == "host":
        q, k, v, w, out = (t.cpu().pin_memory() for t in (q, k, v, w, out))
    return dict(case=case, ctx=ctx, q=q, k=k, v=v, w=w, out=out)


# ---- one pass ---------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "chat":
        s, opts = state["session"], state["options"]
        s.reset()
        first = s.prefill(state["prompt"], GREEDY)
        answer, _ = s.generate(first, opts)
        second = s.prefill_one_at_a_time(state["follow"], GREEDY)
        answer2, _ = s.generate(second, opts)
        return dict(tokens=np.array([first] + answer + [second] + answer2, dtype=np.int64), logits=state["model"].logits())
    if kind == "prompt":
        s = state["session"]
        s.reset()
        return dict(token=s.prefill(state["prompt"], GREEDY), logits=state["model"].logits())
    if kind == "swap":
        s = state["session"]
        s.restore(state["saved"])
        return np.frombuffer(s.snapshot().to_bytes(), dtype=np.uint8)
    if kind == "step":
        m = state["model"]
        value, index = m.step_topk(state["token"], case["pos"], k=1)
        return dict(value=value, index=index.astype(np.int64), logits=m.logits(), **_cache(state["attention"]))
    ctx, w, out = state["ctx"], state["w"], state["out"]
    if kind == "prefill":
        m = case["m"]
        for il, (q, k, v) in enumerate(state["qkv"]):
            ctx.dispatch_q_norm_rope_fused(q, w, 0, m)
            ctx.dispatch_kv_writeback_fused(il, k, v, w, 0, m)
            ctx.dispatch_attention(il, q, out[il], m)
        return dict(out=out, **_cache(ctx))
    q, k, v, pos = state["q"], state["k"], state["v"], case["ctx"] - 1
    if kind == "host":
        ctx.decode_token_host(q, k, v, w, w, pos, out)
    elif kind == "layers":
        for il in range(ctx.n_layer):
            ctx.decode_layer(il, q[il], w, k[il], v[il], w, pos, out[il])
    else:
        ctx.dispatch_q_norm_rope_fused(q, w, pos, 1)
        ctx.dispatch_kv_writeback_fused(0, k, v, w, pos, 1)
        ctx.dispatch_attention_decode(0, q, out, case["ctx"])
    return dict(out=out, **_cache(ctx))


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _weights(shape):
    """(weights of the layers, weights of the LM head): one bit each and an f16 scale per 128."""
    c = SHAPES[shape]
    q, kv, e, ff = c["n_head"] * HEAD_DIM, c["n_kv_head"] * HEAD_DIM, c["n_embd"], c["n_ff"]
    return c["n_layer"] * (e * (2 * q + 2 * kv) + 3 * e * ff), c["n_vocab"] * e


def _row(n_kv):
    return n_kv * (HEAD_DIM + HEAD_DIM // 32 * 4) * 2  # K and V of one cache row of one layer


def work(case):
    kind = case["kind"]
    if kind in ("chat", "prompt", "step", "swap"):
        c = SHAPES[case["shape"]]
        layers, head = _weights(case["shape"])
        row = _row(c["n_kv_head"]) * c["n_layer"]
        attn = 4 * c["n_layer"] * c["n_head"] * HEAD_DIM  # operations per query-key pair
        if kind == "swap":
            return dict(bytes=4 * row * case["pos"], flops=0)  # in and out, each over the link and in device memory
        if kind == "step":
            return dict(bytes=(layers + head) * 18 / 128 + row * (case["pos"] + 1), flops=2 * (layers + head) + attn * (case["pos"] + 1))
        p = case["prompt"]
        batch = dict(bytes=(layers + head) * 18 / 128 + row * p, flops=2 * (layers * p + head) + attn * p * (p + 1) / 2)
        if kind == "prompt":
            return batch
        steps = case["follow"] + 2 * case["new"]
        keys = sum(p + i + 1 for i in range(steps))
        heads = 2 * case["new"] + 1
        return dict(bytes=batch["bytes"] + (layers * steps + head * heads) * 18 / 128 + row * keys,
                    flops=batch["flops"] + 2 * (layers * steps + head * heads) + attn * keys)
    n_head, n_kv = _heads(case)
    if kind == "prefill":
        m = case["m"]
        act = m * (2 * n_head + 2 * n_kv) * HEAD_DIM * 2
        return dict(bytes=N_LAYER * (act + m * _row(n_kv)), flops=N_LAYER * 4 * n_head * HEAD_DIM * m * (m + 1) / 2)
    n_layer = 1 if kind == "dispatch" else N_LAYER
    act = (2 * n_head + 2 * n_kv) * HEAD_DIM * 2
    return dict(bytes=n_layer * (act + _row(n_kv) * case["ctx"]), flops=n_layer * 4 * n_head * HEAD_DIM * case["ctx"])


def tolerance(case):
    """Tokens, and cache bytes and scales of given activations, are exact; a step's own new cache row follows from its
    attention outputs (one row of many: a share of the quants). Attention outputs are f16 sums over quantised
    keys and values with f16 or integer operands in the tensor cores: a few f16 roundings, 2^-11 each. Logits are
    f16 after 36 layers whose keys and values are quantised to 8 bits."""
    if case["kind"] == "swap":
        return "exact"
    if case["kind"] == "step":
        return {"rel": 1e-2, "differ": min(1e-2, 0.1 / (case["pos"] + 1))}
    return {"rel": 1e-2} if case["kind"] in ("chat", "prompt") else {"rel": 2e-3}
