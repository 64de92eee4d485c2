"""Workloads that stand for what a user of this engine has it do, through its public entry points.

A case is a dict of plain values.  `kind` names the call path:

  hook           the trait hooks of flare-core (host f32, one sequence): store a row, attend, per layer
  hook_prefill   the trait's prefill hook (host f32 in and out)
  step           one decode step of a batch: store the new K/V row and attend, layer after layer
  verify         the attention of a speculative verify: several causally ordered queries per sequence
  prefill        causal (or sliding-window) prompt attention on device buffers
  ingest         a prompt's K/V rows go into the cache, then the first query attends them, layer after layer
  forward        a whole token of a Q8_0 model resident on the device, embedding row in, logits out

Shapes are those of this repository's benchmark and tests: 9 query / 3 KV heads x 64 (SmolLM2-135M), 32 / 8 x 64
(Llama-3.2-1B), 32 / 8 x 128 (Llama-3-8B).  All values are drawn from the seed: keys and values N(0, 1) (for the 2-bit
cache one key channel in a hundred times 8), queries N(0, 1) scaled by 1 / sqrt(head_dim), Q8_0 weights uniform int8 with a
scale that keeps unit variance.
"""
import math

import numpy as np
import torch

import flarellm_b200 as fb

CACHE = {"f32": fb.KV_F32, "q8": fb.KV_Q8_0, "kivi": fb.KV_KIVI_G32}
_engine = []


def engine():
    """One context for the whole program, as a server keeps it."""
    if not _engine:
        _engine.append(fb.Engine(0))
    return _engine[0]


# ---------------------------------------------------------------------------------------------- the cases
def _attn(kind, name=None, **kw):
    c = {"kind": kind, "heads": 32, "kv_heads": 8, "head_dim": 64, "cache": "q8", "batch": 1, "ctx": 4096, "layers": 1,
         "ragged": False, "wrapped": False, "host": False, "queries": 1}
    c.update(kw)
    return dict(c, name=name) if name else c


def _prefill(kind, name=None, **kw):
    c = {"kind": kind, "heads": 32, "kv_heads": 8, "head_dim": 128, "dtype": "bf16", "batch": 1, "ctx": 4096, "window": 0}
    c.update(kw)
    return dict(c, name=name) if name else c


def _forward(name=None, **kw):
    c = {"kind": "forward", "hidden": 2048, "heads": 32, "kv_heads": 8, "head_dim": 64, "inter": 8192, "vocab": 128256,
         "layers": 16, "cache": "q8", "batch": 1, "ctx": 1024}
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one layer of one token of a small model through the trait hooks, latency only
        _attn("hook", "hook_f32_token", heads=9, kv_heads=3, cache="f32", ctx=513),
        # interactive chat: one sequence, all layers of one token, everything on the device
        _attn("step", "step_q8_one_sequence", layers=16, ctx=4096),
        # a small server that keeps its activations on the host: page-locked buffers in and out, ragged batch
        _attn("step", "step_q8_host_batch8", layers=16, batch=8, ctx=3000, ragged=True, host=True),
        # a loaded server: the batched decode that the benchmark's headline stands for
        _attn("step", "step_q8_batch32", layers=16, batch=32, ctx=4096),
        # one very long context
        _attn("step", "step_q8_long_context", head_dim=128, layers=2, ctx=131072),
        # many long contexts in the 2-bit cache
        _attn("step", "step_kivi_batch16", cache="kivi", layers=2, batch=16, ctx=32768),
        # speculative decoding: six positions of every sequence checked at once
        _attn("verify", "verify_q8_six_queries", layers=2, batch=32, ctx=4000, ragged=True, queries=6),
        # prompts of a large model, the tensor-core path
        _prefill("prefill", "prefill_bf16_batch4", batch=4, ctx=4096),
        # one prompt of ordinary, odd length through the trait's host hook
        _prefill("hook_prefill", "hook_prefill_f32", head_dim=64, dtype="f32", ctx=1013),
        # what follows a prompt: its rows are quantised into every layer's cache
        _attn("ingest", "ingest_q8_prompt", layers=16, ctx=2049),
        # whole tokens of a resident model, alone and for a small batch
        _forward("forward_one_sequence"),
        _forward("forward_batch8", batch=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("hook", "hook_prefill", "step", "step", "step", "verify", "prefill", "ingest", "forward"))
    if kind == "hook":
        heads, kv = rng.choice(((9, 3), (32, 8)))
        return _attn("hook", heads=heads, kv_heads=kv, cache=rng.choice(("f32", "f32", "q8")), layers=rng.randint(1, 6),
                     ctx=_log(rng, 16, 4096))
    if kind == "hook_prefill":
        heads, kv = rng.choice(((9, 3), (32, 8)))
        return _prefill("hook_prefill", heads=heads, kv_heads=kv, head_dim=64, dtype="f32", ctx=_log(rng, 20, 1013))
    if kind == "step":
        cache = rng.choice(("q8", "q8", "q8", "kivi", "f32"))
        hd = 64 if cache == "kivi" else rng.choice((64, 64, 128))
        batch, layers = _log(rng, 1, 32), _log(rng, 1, 16)
        # at most the rows of the largest listed step (2 million of kv_dim 512 in Q8_0)
        most = 2_000_000 // (batch * layers * (hd // 64) * (4 if cache == "f32" else 1))
        ctx = _log(rng, 64, min(65536, max(80, most)))
        if cache == "kivi":
            ctx = max(160, ctx - ctx % 32)          # the stored token opens no new group: the step can be repeated
        return _attn("step", head_dim=hd, cache=cache, batch=batch, layers=layers, ctx=ctx, ragged=cache != "kivi" and rng.random() < 0.4,
                     wrapped=rng.random() < 0.2, host=rng.random() < 0.25)
    if kind == "verify":
        hd = rng.choice((64, 64, 128))
        batch, layers = _log(rng, 1, 32), rng.randint(1, 4)
        return _attn("verify", head_dim=hd, batch=batch, layers=layers, queries=rng.randint(2, 8), ragged=rng.random() < 0.5,
                     ctx=_log(rng, 100, 300_000 // (batch * layers * (hd // 64)) + 200))
    if kind == "prefill":
        hd = rng.choice((64, 128))
        batch = rng.choice((1, 1, 2, 4))
        ctx = _log(rng, 100, 4096)
        return _prefill("prefill", head_dim=hd, dtype=rng.choice(("bf16", "bf16", "f32")), batch=batch, ctx=ctx,
                        window=rng.choice((0, 0, max(32, ctx // 2 - 5))))
    if kind == "ingest":
        return _attn("ingest", head_dim=rng.choice((64, 128)), cache=rng.choice(("q8", "q8", "f32")), layers=_log(rng, 1, 16),
                     ctx=_log(rng, 50, 4096))
    hidden, heads, kv, inter = rng.choice(((576, 9, 3, 1536), (2048, 32, 8, 8192)))
    return _forward(hidden=hidden, heads=heads, kv_heads=kv, inter=inter, vocab=rng.choice((49152, 128256)),
                    layers=_log(rng, 2, 16), batch=_log(rng, 1, 8), ctx=_log(rng, 16, 2048))


# ---------------------------------------------------------------------------------------------- states
def _lens(case):
    """Slots that each sequence attends (the last of them is the token being stored)."""
    n, b = case["ctx"], case["batch"]
    if not case["ragged"]:
        return [n] * b
    return [max(1, n - (n // 2) * ((i * 7) % b) // b) for i in range(b)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, scale=1.0):
    return torch.randn(*shape, device="cuda", generator=g) * scale


def _keys(case, g, n, kv_dim):
    k = _normal(g, n, kv_dim)
    if case["cache"] == "kivi":
        k[:, torch.randperm(kv_dim, device="cuda", generator=g)[: max(1, kv_dim // 100)]] *= 8
    return k


def _filled_cache(case, g, held):
    """A cache whose sequences hold held[b] tokens (beyond the ring's size where it has wrapped)."""
    kv_dim, most = case["kv_heads"] * case["head_dim"], max(_lens(case))
    ring = (most + 127) // 128 * 128
    kv = engine().kv_alloc(case["layers"], case["batch"], ring, case["kv_heads"], case["head_dim"], CACHE[case["cache"]])
    for b, n in enumerate(held):
        n += ring + ring // 16 + 5 - n % 32 if case["wrapped"] else 0
        if n == 0:
            continue
        step = min(32768, ring)
        for lo in range(0, n, step):
            rows = min(step, n - lo)
            k, v = _keys(case, g, rows, kv_dim), _normal(g, rows, kv_dim)
            torch.cuda.synchronize()
            for layer in range(case["layers"]):
                kv.append(layer, b, k.data_ptr(), v.data_ptr(), n_rows=rows)
            kv.advance(b, rows)
            engine().sync()
    return kv


def _prepare_step(case, seed):
    g = _gen(seed)
    b, nh, hd, kv_dim, layers = case["batch"], case["heads"], case["head_dim"], case["kv_heads"] * case["head_dim"], case["layers"]
    kv = _filled_cache(case, g, [n - 1 for n in _lens(case)])
    rows, q_floats = b * kv_dim, b * nh * hd
    block = _normal(g, layers, 2 * rows + q_floats)
    block[:, 2 * rows:] /= math.sqrt(hd)
    out = torch.zeros(layers, b, 1, nh, hd, device="cuda")
    if case["host"]:
        block, out = block.cpu().pin_memory(), out.cpu().pin_memory()
    calls = []
    for layer in range(layers):
        k = block[layer].data_ptr()
        calls.append((layer, k, k + 4 * rows, k + 8 * rows, out[layer].data_ptr()))
    return {"kv": kv, "block": block, "out": out, "calls": calls, "heads": nh, "on_device": not case["host"]}


def _run_step(s):
    eng, kv, heads, dev = engine(), s["kv"], s["heads"], s["on_device"]
    for layer, k, v, q, o in s["calls"]:
        eng.decode_step(kv, layer, heads, k, v, q, out=o, on_device=dev)
    return s["out"]


def _prepare_verify(case, seed):
    g = _gen(seed)
    lens = _lens(case)
    kv = _filled_cache(case, g, lens)
    q = _normal(g, case["layers"], case["batch"], case["queries"], case["heads"], case["head_dim"], scale=1 / math.sqrt(case["head_dim"]))
    return {"kv": kv, "q": q, "out": torch.zeros_like(q), "lens": lens, "heads": case["heads"], "queries": case["queries"]}


def _run_verify(s):
    eng, q, out = engine(), s["q"], s["out"]
    for layer in range(q.shape[0]):
        eng.decode(s["kv"], layer, s["heads"], q[layer].data_ptr(), n_q=s["queries"], attend_len=s["lens"], out=out[layer].data_ptr())
    return out


def _prepare_hook(case, seed):
    g = _gen(seed)
    nh, nkv, hd, n, layers = case["heads"], case["kv_heads"], case["head_dim"], case["ctx"], case["layers"]
    be = fb.CudaBackend(0)
    be.init_gpu_kv_cache(layers, n + 64, nkv, hd, CACHE[case["cache"]])
    k = _normal(g, layers, n, nkv * hd).cpu().numpy()
    v = _normal(g, layers, n, nkv * hd).cpu().numpy()
    q = _normal(g, layers, nh * hd, scale=1 / math.sqrt(hd)).cpu().numpy()
    for t in range(n - 1):
        for layer in range(layers):
            be.gpu_kv_write(layer, t, nkv, hd, k[layer, t], v[layer, t])
        be.advance_kv(1)
    return {"be": be, "rows": [(q[i], k[i, n - 1], v[i, n - 1]) for i in range(layers)], "n": n, "shape": (nh, nkv, hd)}


def _run_hook(s):
    be, n, (nh, nkv, hd) = s["be"], s["n"], s["shape"]
    outs = []
    for layer, (q, k, v) in enumerate(s["rows"]):
        be.gpu_kv_write(layer, n - 1, nkv, hd, k, v)
        outs.append(be.grouped_query_attention_from_gpu_cache(q, layer, nh, nkv, hd, n))
    return outs


def _prepare_prefill(case, seed):
    g = _gen(seed)
    b, n, nh, nkv, hd = case["batch"], case["ctx"], case["heads"], case["kv_heads"], case["head_dim"]
    dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    q, k, v = (_normal(g, b, n, h, hd, scale=0.5).to(dt) for h in (nh, nkv, nkv))
    s = {"shape": (b, n, nh, nkv, hd), "window": case["window"]}
    if case["kind"] == "hook_prefill":
        return dict(s, be=fb.CudaBackend(0), q=q.cpu().numpy(), k=k.cpu().numpy(), v=v.cpu().numpy())
    return dict(s, q=q, k=k, v=v, out=torch.zeros_like(q), dt=fb.DT_BF16 if case["dtype"] == "bf16" else fb.DT_F32)


def _run_prefill(s):
    b, n, nh, nkv, hd = s["shape"]
    if "be" in s:
        return s["be"].prefill_attention_gpu(s["q"], s["k"], s["v"], n, nh, nkv, hd)
    engine().prefill(s["q"].data_ptr(), s["k"].data_ptr(), s["v"].data_ptr(), b, n, nh, nkv, hd, window=s["window"],
                     in_dtype=s["dt"], out_dtype=s["dt"], out=s["out"].data_ptr())
    return s["out"]


def _prepare_ingest(case, seed):
    g = _gen(seed)
    n, nkv, hd, layers = case["ctx"], case["kv_heads"], case["head_dim"], case["layers"]
    kv = engine().kv_alloc(layers, 1, (n + 127) // 128 * 128, nkv, hd, CACHE[case["cache"]])
    k, v = _normal(g, layers, n, nkv * hd), _normal(g, layers, n, nkv * hd)
    q = _normal(g, layers, 1, 1, case["heads"], hd, scale=1 / math.sqrt(hd))
    return {"kv": kv, "k": k, "v": v, "q": q, "out": torch.zeros_like(q), "n": n, "heads": case["heads"]}


def _run_ingest(s):
    eng, kv, n = engine(), s["kv"], s["n"]
    kv.set_state(0, 0, 0)
    for layer in range(s["q"].shape[0]):
        kv.append(layer, 0, s["k"][layer].data_ptr(), s["v"][layer].data_ptr(), n_rows=n)
        eng.decode(kv, layer, s["heads"], s["q"][layer].data_ptr(), attend_len=[n], out=s["out"][layer].data_ptr())
    return s["out"]


def _blocks(g, rows, cols):
    """A Q8_0 block stream (f16 scale + 32 int8 per 34 bytes) of a matrix that keeps unit variance."""
    w = torch.randint(0, 255, (rows * (cols // 32), 34), device="cuda", generator=g, dtype=torch.uint8)
    w[:, 2:] += 129                                 # int8 values -127 .. 127
    scale = np.array([1.0 / (73.0 * math.sqrt(cols))], np.float16).view(np.uint8)
    w[:, 0], w[:, 1] = int(scale[0]), int(scale[1])
    return w.cpu().numpy().reshape(-1)


def _prepare_forward(case, seed):
    g = _gen(seed)
    d, nh, nkv, hd, inter, layers = (case[k] for k in ("hidden", "heads", "kv_heads", "head_dim", "inter", "layers"))
    eng = engine()
    model = eng.model_create(d, nh, nkv, hd, inter, case["vocab"], layers, 1e-5)
    norm = (1 + 0.1 * _normal(g, d)).cpu().numpy()
    w = dict(qkv=_blocks(g, (nh + 2 * nkv) * hd, d), wo=_blocks(g, d, nh * hd), gate_up=_blocks(g, 2 * inter, d), down=_blocks(g, d, inter))
    for layer in range(layers):                     # the same draw for every layer, a device copy of its own for each
        model.set_layer(layer, attn_norm=norm, ffn_norm=norm, **w)
    model.set_output(norm, output_q8=_blocks(g, case["vocab"], d))
    kv = _filled_cache(dict(case, ragged=False, wrapped=False, ctx=case["ctx"] + 1), g, [case["ctx"]] * case["batch"])
    half = np.arange(hd // 2, dtype=np.float64)
    angle = np.arange(4096, dtype=np.float64)[:, None] * (10000.0 ** (-2.0 * half / hd))[None, :]
    kv.set_rope_table(np.cos(angle).astype(np.float32), np.sin(angle).astype(np.float32))
    x = _normal(g, case["batch"], d).cpu().numpy()
    return {"model": model, "kv": kv, "x": x, "ctx": case["ctx"], "pos": np.full(case["batch"], case["ctx"], np.int64)}


def _run_forward(s):
    kv = s["kv"]
    for b in range(kv.batch):                       # every pass is the token after the same context
        kv.set_state(b, s["ctx"], s["ctx"])
    return s["model"].forward(kv, s["x"], s["pos"])


_PATHS = {"hook": (_prepare_hook, _run_hook), "step": (_prepare_step, _run_step), "verify": (_prepare_verify, _run_verify),
          "prefill": (_prepare_prefill, _run_prefill), "hook_prefill": (_prepare_prefill, _run_prefill),
          "ingest": (_prepare_ingest, _run_ingest), "forward": (_prepare_forward, _run_forward)}


def prepare(case, seed):
    s = _PATHS[case["kind"]][0](case, seed)
    torch.cuda.synchronize()
    return dict(s, kind=case["kind"])


def run(state):
    return _PATHS[state["kind"]][1](state)


# ---------------------------------------------------------------------------------------------- what a pass needs
def _row_bytes(cache, kv_dim):
    """Bytes of one token's K and V in the cache."""
    return {"f32": 8 * kv_dim, "q8": 2 * (kv_dim + kv_dim // 16), "kivi": 0.75 * kv_dim}[cache]


def _cache_bytes(cache, kv_dim, n):
    if cache == "kivi":
        return max(0, n - 128) * 0.75 * kv_dim + min(n, 128) * 4 * kv_dim       # the newest 128 tokens are f16
    return n * _row_bytes(cache, kv_dim)


def work(case):
    nh, hd = case["heads"], case["head_dim"]
    kv_dim = case["kv_heads"] * hd
    if case["kind"] in ("prefill", "hook_prefill"):
        n, w, b = case["ctx"], case["window"] or case["ctx"], case["batch"]
        pairs = sum(min(i + 1, w) for i in range(n))
        return {"bytes": b * n * (2 * nh * hd + 2 * kv_dim) * (2 if case["dtype"] == "bf16" else 4), "flops": 4 * b * nh * hd * pairs}
    if case["kind"] == "forward":
        d, inter, b, layers = case["hidden"], case["inter"], case["batch"], case["layers"]
        params = layers * ((nh * hd + 2 * kv_dim) * d + d * nh * hd + 3 * inter * d) + case["vocab"] * d
        kv = layers * b * _cache_bytes(case["cache"], kv_dim, case["ctx"] + 1)
        return {"bytes": params * 34 / 32 + kv + 4 * b * (case["vocab"] + d),
                "flops": 2 * b * params + 4 * layers * b * nh * hd * (case["ctx"] + 1)}
    lens = _lens(case)
    if case["wrapped"]:
        lens = [(max(lens) + 127) // 128 * 128] * len(lens)
    layers, nq = case["layers"], case["queries"]
    rows = case["batch"] * (4 * nq * nh * hd * 2 + 8 * kv_dim)                   # queries, outputs, new rows
    total = layers * (sum(_cache_bytes(case["cache"], kv_dim, n) for n in lens) + rows)
    if case["kind"] == "ingest":
        total += layers * case["ctx"] * (8 * kv_dim + _row_bytes(case["cache"], kv_dim))
    return {"bytes": total, "flops": 4 * layers * nq * nh * hd * sum(lens)}


def tolerance(case):
    if case["kind"] in ("prefill", "hook_prefill"):
        return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1e-3}      # f32 inputs run as 11-bit operands
    if case["kind"] == "forward":
        return {"rel": 1e-2}          # activations are 8-bit codes: a last-bit difference moves a code by a step
    # a quantised cache is attended with 11-bit weights, an f32 cache in f32
    return {"rel": 1e-5} if case["cache"] == "f32" else {"rel": 1e-3}
