"""The work a user of this package has it do, as cases that can be timed and compared.

Seven kinds of work, each through the package's public entry points:

vllm      a request through the vLLM hooks in no-alloc hybrid mode: one prefill call of the whole prompt,
          then one `do_kv_cache_update` + `forward` per generated token and layer (what a serving engine
          with one running sequence does).  Prefill attention, store, ring and decode all take part.
generate  a request through `KVCaptureEngine` without vLLM: `ingest_prefill`, then a token at a time.
          calls = "fused" (`decode_step`), "host" (`decode_step_host`, data in pinned memory) or "two"
          (`ingest_decode` + `compute_hybrid_attention`, the call sequence of the original package).
hybrid    one step of `compute_hybrid_attention` over layers that already hold a history (few tokens: the
          smallest call there is; several layers of a long sequence: the streaming case).
paged     one step of a batch over the compressed paged cache: `write` one token per sequence into the
          engine's slots, `decode` every sequence.
append    a prompt into the compressed store; source = "rows" (`append_chunk`, in chunks), "paged" (walked
          from a bf16 paged cache), "slots" (`CompressedPagedKVCache.write`).
codec     the quantiser objects by themselves: quantise and dequantise keys and values, score queries.
legacy    one token of attention through `TurboQuantKVCache` (scores, softmax, weighted values).

Keys are Gaussian with log-normal scales per channel (outlier channels), values and queries Gaussian.
"""

import math
import random
import types

import torch

from turboquant_b200 import (CompressedCacheSpec, CompressedKVStore, CompressedPagedKVCache, KVCaptureEngine,
                             TurboQuantKVCache, TurboQuantProd, compute_hybrid_attention)
from turboquant_b200.integration import vllm as hooks
from turboquant_b200.kv_cache import dequantize_values, quantize_values

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
RING = 128      # exact recent tokens, the default of the capture engine
CHUNK = 8192    # tokens per append of a long prompt


def listed():
    return [
        # a short chat turn: everything is latency and launches
        dict(name="vllm_chat_short", kind="vllm", layers=2, head_dim=128, kv_heads=8, q_heads=32, prompt=203, steps=24,
             key_bits=3, value_bits=2),
        # a long prompt with its first tokens: prefill attention and the store
        dict(name="vllm_prompt_8k", kind="vllm", layers=1, head_dim=128, kv_heads=8, q_heads=32, prompt=8192, steps=8,
             key_bits=3, value_bits=2),
        # one long sequence shaped like a hybrid model's full-attention layer, 128 new tokens
        dict(name="generate_32k", kind="generate", calls="fused", head_dim=256, kv_heads=4, q_heads=16, prompt=32768,
             steps=128, key_bits=3, value_bits=2, dtype="bf16"),
        # one attention call over a moderate history
        dict(name="hybrid_4k", kind="hybrid", layers=1, head_dim=128, kv_heads=8, q_heads=32, tokens=4096, recent=77,
             queries=1, key_bits=3, value_bits=2),
        # one step of the eight full-attention layers over a long history (larger than L2)
        dict(name="hybrid_32k_8_layers", kind="hybrid", layers=8, head_dim=256, kv_heads=4, q_heads=16, tokens=32768,
             recent=100, queries=1, key_bits=3, value_bits=2),
        # a handful of short sequences
        dict(name="paged_5_short", kind="paged", batch=5, lo=90, hi=1900, head_dim=128, kv_heads=8, q_heads=32, key_bits=3,
             value_bits=2),
        # a serving batch of mixed lengths at the higher bit widths
        dict(name="paged_64_mixed", kind="paged", batch=64, lo=1024, hi=32768, head_dim=128, kv_heads=8, q_heads=32,
             key_bits=4, value_bits=4),
        # a large batch of one layer with 64 query heads
        dict(name="paged_256_8k", kind="paged", batch=256, lo=8192, hi=8192, head_dim=128, kv_heads=8, q_heads=64,
             key_bits=3, value_bits=2),
        # prefill throughput of the store, 131072 tokens
        dict(name="append_131k", kind="append", source="rows", tokens=131072, head_dim=128, kv_heads=8, key_bits=3,
             value_bits=2, dtype="bf16"),
        # a prompt taken over from a paged cache by one of the first layers (one more key bit), ragged length
        dict(name="append_paged_d256_k4", kind="append", source="paged", tokens=5003, head_dim=256, kv_heads=4, key_bits=4,
             value_bits=2, dtype="bf16"),
        # the quantisers by themselves, fp32 vectors
        dict(name="codec_2k", kind="codec", heads=8, tokens=2000, queries=4, head_dim=128, key_bits=3, value_bits=2,
             dtype="fp32"),
        # the single-object cache in its default type
        dict(name="legacy_4k", kind="legacy", batch=1, heads=8, tokens=4096, queries=1, head_dim=128, key_bits=3,
             value_bits=2, dtype="fp16"),
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _heads(rng, head_dim):
    kv = rng.choice((1, 2, 4, 8) if head_dim == 128 else (1, 2, 4))
    return kv, kv * rng.choice((1, 2, 4, 4, 8))


def draw(rng):
    kind = rng.choice(("vllm",) * 4 + ("generate",) * 3 + ("hybrid",) * 4 + ("paged",) * 4 + ("append",) * 3 + ("codec", "legacy"))
    d = rng.choice((128, 128, 256))
    kv, qh = _heads(rng, d)
    kb, vb = rng.choice(((3, 2), (3, 2), (4, 2), (4, 4), (3, 4)))
    bits = dict(key_bits=kb, value_bits=vb)
    if kind == "vllm":
        prompt = _log(rng, 160, 8000)
        return dict(kind=kind, layers=rng.randint(1, 4) if prompt < 2000 else 1, head_dim=d, kv_heads=kv, q_heads=qh,
                    prompt=prompt, steps=rng.randint(4, 40), **bits)
    if kind == "generate":
        return dict(kind=kind, calls=rng.choice(("fused", "fused", "host", "two")), head_dim=d, kv_heads=kv, q_heads=qh,
                    prompt=_log(rng, 150, 30000), steps=rng.randint(16, 120), **bits,
                    dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")))
    if kind == "hybrid":
        return dict(kind=kind, layers=rng.randint(1, 8), head_dim=d, kv_heads=kv, q_heads=qh, tokens=_log(rng, 20, 32000),
                    recent=rng.randint(0, RING), queries=rng.choice((1, 1, 1, 2, 5)), **bits)
    if kind == "paged":
        hi = _log(rng, 60, 30000)
        batch = _log(rng, 1, 256)
        while batch * hi > 1_000_000:      # the two together stay below the largest listed batch
            batch = max(1, batch // 2)
        return dict(kind=kind, batch=batch, lo=max(20, hi // rng.randint(1, 20)), hi=hi, head_dim=d, kv_heads=kv, q_heads=qh,
                    **bits)
    if kind == "append":
        return dict(kind=kind, source=rng.choice(("rows", "rows", "paged", "slots")), tokens=_log(rng, 100, 60000 // (d // 128)),
                    head_dim=d, kv_heads=kv, **bits, dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")))
    if kind == "codec":
        return dict(kind=kind, heads=kv, tokens=_log(rng, 50, 4000), queries=rng.randint(1, 8), head_dim=d, **bits,
                    dtype=rng.choice(("fp32", "bf16", "fp16")))
    return dict(kind=kind, batch=rng.choice((1, 1, 2)), heads=kv, tokens=_log(rng, 200, 8000), queries=rng.randint(1, 2),
                head_dim=d, **bits, dtype=rng.choice(("fp16", "bf16")))


# ---------------------------------------------------------------------------- inputs

class Source:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=self.gen, device="cuda", dtype=dtype)

    def keys(self, *shape, dtype=torch.bfloat16):
        return self.normal(*shape, dtype=dtype).mul_(torch.exp(0.5 * self.normal(shape[-1], dtype=torch.float32)).to(dtype))


class AttentionImpl:
    """Stands in for the engine's own attention of a layer, which the hooks replace."""

    def __init__(self, head_dim, kv_heads, q_heads):
        self.head_size, self.num_kv_heads, self.num_heads = head_dim, kv_heads, q_heads
        self.scale = 1.0 / math.sqrt(head_dim)

    def do_kv_cache_update(self, layer, key, value, kv_cache, slot_mapping):
        pass

    def forward(self, layer, query, key, value, kv_cache, attn_metadata, output=None, output_scale=None,
                output_block_scale=None):
        return output


def _lengths(c):
    """Lengths of the sequences of a batch: the same for every seed, so that the work is."""
    rng = random.Random(1000003 * c["batch"] + 17 * c["lo"] + c["hi"])
    return [rng.randint(c["lo"], c["hi"]) for _ in range(c["batch"])]


def _prepare_vllm(c, src):
    ctx = {"layers.%d.attn" % i: types.SimpleNamespace(impl=AttentionImpl(c["head_dim"], c["kv_heads"], c["q_heads"]))
           for i in range(c["layers"])}
    runner = types.SimpleNamespace(compilation_config=types.SimpleNamespace(static_forward_context=ctx),
                                   device=torch.device("cuda"), kv_caches=[])
    states = hooks.install_hooks(runner, key_bits=c["key_bits"], value_bits=c["value_bits"], ring_capacity=RING,
                                 initial_layers_count=0, mode=hooks.MODE_HYBRID, no_alloc=True)
    n, t, d = c["prompt"], c["steps"], c["head_dim"]
    return dict(case=c, impls=[m.impl for m in ctx.values()], states=list(states.values()),
                k=[src.keys(n + t, c["kv_heads"], d) for _ in ctx], v=[src.normal(n + t, c["kv_heads"], d) for _ in ctx],
                q=[src.normal(n + t, c["q_heads"], d) for _ in ctx],
                out=[torch.zeros(n + t, c["q_heads"], d, dtype=torch.bfloat16, device="cuda") for _ in ctx],
                slots=torch.arange(n + t, device="cuda"),
                prefill=types.SimpleNamespace(num_actual_tokens=n, max_query_len=n),
                decode=types.SimpleNamespace(num_actual_tokens=1, max_query_len=1))


def _run_vllm(s):
    n, t = s["case"]["prompt"], s["case"]["steps"]
    for st in s["states"]:
        st.reset()
    for lo, hi, md in [(0, n, s["prefill"])] + [(i, i + 1, s["decode"]) for i in range(n, n + t)]:
        slots = s["slots"][lo:hi]
        for impl, q, k, v, out in zip(s["impls"], s["q"], s["k"], s["v"], s["out"]):
            kk, vv = k[lo:hi], v[lo:hi]
            impl.do_kv_cache_update(None, kk, vv, None, slots)
            impl.forward(None, q[lo:hi], kk, vv, None, md, output=out[lo:hi])
    return {"out": s["out"], "records": [st.store.pool.data for st in s["states"]],
            "ring": [st.engine.ring.peek() for st in s["states"]]}


def _prepare_generate(c, src):
    h, qh, d, n, t, dt = c["kv_heads"], c["q_heads"], c["head_dim"], c["prompt"], c["steps"], DTYPES[c["dtype"]]
    store = CompressedKVStore(d, h, c["key_bits"], c["value_bits"], device="cuda", capacity_tokens=n + t)
    engine = KVCaptureEngine(store, ring_capacity=RING, device="cuda", dtype=dt)
    s = dict(case=c, engine=engine, k=src.keys(n + t, h, d, dtype=dt), v=src.normal(n + t, h, d, dtype=dt),
             q=src.normal(t, qh, d, dtype=dt))
    if c["calls"] == "host":
        rows = torch.cat([x.reshape(t, -1) for x in (s["k"][n:], s["v"][n:], s["q"])], 1)
        s["rows"] = rows.cpu().pin_memory()
        s["out"] = torch.zeros(t, qh * d, dtype=dt).pin_memory()
    else:
        s["out"] = torch.zeros(t, qh, d, dtype=dt, device="cuda")
    return s


def _run_generate(s):
    c, engine, k, v, q, out = s["case"], s["engine"], s["k"], s["v"], s["q"], s["out"]
    n, t, qh, calls = c["prompt"], c["steps"], c["q_heads"], c["calls"]
    engine.reset()
    engine.ingest_prefill(k[:n], v[:n], n)
    if calls == "host":
        rows = s["rows"]
        for i in range(t):
            engine.decode_step_host(rows[i], out[i], qh)
        torch.cuda.current_stream().synchronize()      # the caller reads its host buffer
        return {"out": out, "records": engine.store.pool.data}
    if calls == "fused":
        for i in range(t):
            engine.decode_step(q[i:i + 1], k[n + i:n + i + 1], v[n + i:n + i + 1], qh, out=out[i:i + 1])
        return {"out": out, "records": engine.store.pool.data}
    outs = []
    for i in range(t):
        engine.ingest_decode(k[n + i:n + i + 1], v[n + i:n + i + 1], 1)
        rk, rv = engine.ring.peek()
        outs.append(compute_hybrid_attention(q[i:i + 1], engine.store, rk, rv, qh))
    return {"out": torch.cat(outs), "records": engine.store.pool.data}


def _prepare_hybrid(c, src):
    layers = []
    for i in range(c["layers"]):
        h, d, n = c["kv_heads"], c["head_dim"], c["tokens"]
        store = CompressedKVStore(d, h, c["key_bits"], c["value_bits"], device="cuda", layer_idx=i, capacity_tokens=n)
        store.append_chunk(src.keys(n, h, d), src.normal(n, h, d))
        r = c["recent"]
        recent = (src.keys(r, h, d), src.normal(r, h, d)) if r else (None, None)
        layers.append((src.normal(c["queries"], c["q_heads"], d), store, *recent))
    return dict(case=c, layers=layers)


def _run_hybrid(s):
    qh = s["case"]["q_heads"]
    return [compute_hybrid_attention(q, store, rk, rv, qh) for q, store, rk, rv in s["layers"]]


def _prepare_paged(c, src):
    h, d, b = c["kv_heads"], c["head_dim"], c["batch"]
    lens = _lengths(c)
    per = [(n + 15) // 16 for n in lens]
    table = torch.zeros(b, max(per), dtype=torch.int32, device="cuda")
    perm = torch.randperm(sum(per), generator=src.gen, device="cuda").to(torch.int32)
    cache = CompressedPagedKVCache.allocate(CompressedCacheSpec(d, h, c["key_bits"], c["value_bits"]), sum(per), torch.device("cuda"))
    at = 0
    rows = max(16384, max(lens))
    k, v, used = None, None, rows      # fresh vectors for about every 16k tokens
    last = []
    for i, n in enumerate(lens):
        table[i, :per[i]] = perm[at:at + per[i]]
        at += per[i]
        if used + n > rows:
            k, v, used = src.keys(rows, h, d), src.normal(rows, h, d), 0
        pos = torch.arange(n, device="cuda")
        slots = table[i].long()[pos // 16] * 16 + pos % 16
        cache.write(k[used:used + n], v[used:used + n], slots)
        used += n
        last.append(slots[-1:])
    return dict(case=c, cache=cache, table=table, lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), longest=max(lens),
                slots=torch.cat(last), k=src.keys(b, h, d), v=src.normal(b, h, d), q=src.normal(b, c["q_heads"], d))


def _run_paged(s):
    cache = s["cache"]
    cache.write(s["k"], s["v"], s["slots"])
    return {"out": cache.decode(s["q"], s["table"], s["lens"], s["longest"]), "records": cache.pool.data}


def _prepare_append(c, src):
    h, d, n, dt = c["kv_heads"], c["head_dim"], c["tokens"], DTYPES[c["dtype"]]
    k, v = src.keys(n, h, d, dtype=dt), src.normal(n, h, d, dtype=dt)
    if c["source"] == "slots":
        blocks = (n + 15) // 16
        cache = CompressedPagedKVCache.allocate(CompressedCacheSpec(d, h, c["key_bits"], c["value_bits"]), blocks, torch.device("cuda"))
        pos = torch.arange(n, device="cuda")
        perm = torch.randperm(blocks, generator=src.gen, device="cuda")
        return dict(case=c, cache=cache, k=k, v=v, slots=perm[pos // 16] * 16 + pos % 16)
    store = CompressedKVStore(d, h, c["key_bits"], c["value_bits"], device="cuda", capacity_tokens=n)
    s = dict(case=c, engine=KVCaptureEngine(store, ring_capacity=RING, device="cuda", dtype=dt), k=k, v=v)
    if c["source"] == "paged":
        blocks = (n + 15) // 16
        perm = torch.randperm(blocks, generator=src.gen, device="cuda")
        paged = torch.zeros(2, blocks, 16, h, d, dtype=dt, device="cuda")
        paged[0].view(blocks * 16, h, d)[(perm[:, None] * 16 + torch.arange(16, device="cuda")).view(-1)[:n]] = k
        paged[1].view(blocks * 16, h, d)[(perm[:, None] * 16 + torch.arange(16, device="cuda")).view(-1)[:n]] = v
        s.update(paged=paged, table=perm.to(torch.int32), k=None, v=None)
    return s


def _run_append(s):
    n, k, v = s["case"]["tokens"], s["k"], s["v"]
    if "cache" in s:
        s["cache"].write(k, v, s["slots"])
        return s["cache"].pool.data
    engine = s["engine"]
    engine.reset()
    if "paged" in s:
        engine.ingest_prefill_from_paged_cache(s["paged"], n, s["table"], 16)
        return {"records": engine.store.pool.data, "ring": engine.ring.peek()}
    for at in range(0, n, CHUNK):
        engine.store.append_chunk(k[at:at + CHUNK], v[at:at + CHUNK])
    return engine.store.pool.data


def _prepare_codec(c, src):
    h, n, d, dt = c["heads"], c["tokens"], c["head_dim"], DTYPES[c["dtype"]]
    return dict(case=c, quantizer=TurboQuantProd(d, c["key_bits"], device="cuda"), x=src.keys(h, n, d, dtype=dt),
                v=src.normal(h, n, d, dtype=dt), q=src.normal(h, c["queries"], d, dtype=dt))


def _run_codec(s):
    z = s["quantizer"]
    kq = z.quantize(s["x"])
    vq = quantize_values(s["v"], bits=s["case"]["value_bits"])
    return {"keys": list(kq[:4]), "values": list(vq[:3]), "logits": z.attention_score(s["q"], kq), "keys_back": z.dequantize(kq),
            "values_back": dequantize_values(vq)}


def _prepare_legacy(c, src):
    b, h, n, d, dt = c["batch"], c["heads"], c["tokens"], c["head_dim"], DTYPES[c["dtype"]]
    cache = TurboQuantKVCache(d, c["key_bits"], c["value_bits"], buffer_size=RING, device="cuda", dtype=dt)
    cache.prefill(src.keys(b, h, n, d, dtype=dt), src.normal(b, h, n, d, dtype=dt))
    return dict(case=c, cache=cache, q=src.normal(b, h, c["queries"], d, dtype=dt))


def _run_legacy(s):
    logits = s["cache"].attention_scores(s["q"])
    return {"logits": logits, "out": s["cache"].attend(torch.softmax(logits, dim=-1))}


_PREPARE = {"vllm": _prepare_vllm, "generate": _prepare_generate, "hybrid": _prepare_hybrid, "paged": _prepare_paged,
            "append": _prepare_append, "codec": _prepare_codec, "legacy": _prepare_legacy}
_RUN = {"vllm": _run_vllm, "generate": _run_generate, "hybrid": _run_hybrid, "paged": _run_paged, "append": _run_append,
        "codec": _run_codec, "legacy": _run_legacy}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, Source(seed))


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------- work and tolerance

def _record(c):
    """Bytes of a compressed token of one kv head: codes, sign bits, two fp16 norms, value codes, fp16 scales and zeros."""
    d = c["head_dim"]
    return d * (1 + (2 if c["key_bits"] == 3 else 4)) // 8 + 4 + d * c["value_bits"] // 8 + d // 32 * 4


def _store_work(c, tokens, size):
    """Read the rows, write the records; the rotation and the sign projection are d x d products."""
    h, d = c.get("kv_heads", c.get("heads")), c["head_dim"]
    return tokens * h * (2 * d * size + _record(c)), tokens * h * 2 * 2 * d * d


def _decode_work(c, tokens, recent, size, calls=1):
    """Read the records and the exact tokens once, the query in and the output out; scores and values."""
    h, qh, d = c["kv_heads"], c["q_heads"], c["head_dim"]
    return (tokens * h * _record(c) + recent * h * 2 * d * size + calls * qh * 2 * d * size,
            (tokens + recent) * qh * 2 * 2 * d + calls * qh * 2 * 2 * d * d)


def _add(*parts):
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def _decode_run(c, prompt, steps, size):
    """The decode steps of a request: (bytes, flops) with the ring's fill and its flushes followed."""
    hist, ring, parts = max(0, prompt - RING), min(prompt, RING), []
    for _ in range(steps):
        if ring == RING:
            parts.append(_store_work(c, RING, size))
            hist, ring = hist + RING, 0
        ring += 1
        parts.append(_decode_work(c, hist if hist >= 16 else 0, ring, size))
    return parts


def work(case):
    c, kind = case, case["kind"]
    if kind == "vllm":
        n, d, qh, h = c["prompt"], c["head_dim"], c["q_heads"], c["kv_heads"]
        attention = (n * (2 * qh + 2 * h) * d * 2, 2 * n * n * d * qh)
        one = _add(attention, _store_work(c, max(0, n - RING), 2), *_decode_run(c, n, c["steps"], 2))
        return {k: v * c["layers"] for k, v in one.items()}
    if kind == "generate":
        size = 4 if c["dtype"] == "fp32" else 2
        return _add(_store_work(c, max(0, c["prompt"] - RING), size), *_decode_run(c, c["prompt"], c["steps"], size))
    if kind == "hybrid":
        t, r = c["queries"], c["recent"]
        b, f = _decode_work(c, c["tokens"], r, 2)
        return {"bytes": c["layers"] * (b + (t - 1) * c["q_heads"] * 4 * c["head_dim"]), "flops": c["layers"] * t * f}
    if kind == "paged":
        return _add(_store_work(c, c["batch"], 2), _decode_work(c, sum(_lengths(c)), 0, 2, calls=c["batch"]))
    if kind == "append":
        b, f = _store_work(c, c["tokens"], 4 if c["dtype"] == "fp32" else 2)
        return {"bytes": b, "flops": f}
    if kind == "codec":
        rows, d = c["heads"] * c["tokens"], c["head_dim"]
        b, f = _store_work(c, c["tokens"], 4 if c["dtype"] == "fp32" else 2)
        back = rows * (_record(c) + 2 * d * 4)
        logits = rows * c["queries"]
        return {"bytes": b + back + 4 * logits, "flops": f + rows * 2 * 2 * d * d + logits * 4 * d}
    rows, d = c["batch"] * c["heads"] * c["tokens"], c["head_dim"]
    return {"bytes": rows * _record(c) + 2 * rows * c["queries"] * 4, "flops": rows * c["queries"] * 6 * d}


def tolerance(case):
    """16-bit outputs carry about 3e-3 of rounding each and the queries are held in fp16 inside.  Codes and sign bits may
    fall on the other side where a coordinate lies on a decision boundary (about two in a million codes), and with such a
    code a tenth of the sign bits of its vector: that vector, one in some thousands, comes back about 20 % off, which is
    0.2 * sqrt(2e-4) = 3e-3 of all of them.  fp16 norms may differ in their last bit."""
    if case["kind"] in ("codec", "legacy"):
        return {"rel": 3e-3, "max": 0.5, "differ": 1e-3}
    return {"rel": 1e-2, "max": 0.4, "differ": 1e-3}
