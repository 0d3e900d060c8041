"""What this framework is timed on: the calls that a serving program makes, over the sizes it makes them with.

Five kinds of work, each through the public entry points:

* ``decode``  - one new token per sequence and layer: ``TurboQuantKVCache.decode_step(q, k, v)``;
* ``prefill`` - a piece of a prompt on a cache that already holds some: ``update(k, v)`` then the causal ``attend(q)``;
* ``ingest``  - a whole prompt into a fresh cache: ``update`` (or ``update_and_fetch``, for callers with their own attention);
* ``fetch``   - one new token for a caller with its own attention: ``update_and_fetch`` returns dense keys and values;
* ``codec``   - ``TurboQuantMSE.quantize`` and ``.dequantize`` on their own.

Keys and values are N(0, 1) rows under a LogNormal(0, 0.5) scale per token (optionally with four outlier channels per head),
queries N(0, 1) / sqrt(head_dim): the distributions of this repository's benchmark.  Lengths include tokens of every region
(sink, packed, recent) and are not multiples of a tile unless real use makes them so.
"""

import math

import torch

from mlx_turboquant_b200 import TurboQuantKVCache, TurboQuantMSE

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}

# The largest amount of work of each kind that draw() gives: what the largest listed case of the kind has.
MOST_DECODE = 32 * 8 * 32768 * 128          # sequences x KV heads x context x head_dim
MOST_PREFILL = 4 * 32 * 512 * 16384 * 128   # sequences x query heads x new tokens x context x head_dim
MOST_INGEST = 8 * 131072 * 128              # sequences x KV heads x tokens x head_dim


def listed():
    return [
        # -- one token per sequence ------------------------------------------------------------------------------------
        # The start of a chat: a few hundred tokens, one sequence. Launches and host work are all there is.
        decode("decode_600_b1", 1, 32, 8, 128, 600),
        # The headline layer: one long-context sequence, 32 query heads on 8 KV heads.
        decode("decode_32k_b1", 1, 32, 8, 128, 32768),
        # A batch of mid-length sequences on a model without grouped queries, head_dim 96, sign sketches on.
        decode("decode_8k_b16_d96_qjl", 16, 32, 32, 96, 8192, qjl=True),
        # A full server: half of the batch-64 workload at 32K, bf16. The largest decode step.
        decode("decode_32k_b32_bf16", 32, 32, 8, 128, 32768, dtype="bf16"),
        # Mixed-bit keys and values (channel split), a few sequences of ragged length.
        decode("decode_11777_b4_k3.5_v3.5", 4, 32, 8, 128, 11777, kb=3.5, vb=3.5, dtype="bf16"),
        # -- pieces of prompts ---------------------------------------------------------------------------------------------
        # The prefill of the batched workload: a 512-token piece at 16K.
        prefill("prefill_512_at_16k_b4", 4, 32, 8, 128, 16384, 512, dtype="bf16"),
        # An odd piece of a shorter prompt, head_dim 64, 4-bit keys and values.
        prefill("prefill_1000_at_3000_b2_d64", 2, 32, 8, 64, 3000, 1000, kb=4, vb=4, dtype="bf16"),
        # -- whole prompts -------------------------------------------------------------------------------------------------
        # Prompt compression at 128K, chunked, with outlier channels: the largest prompt.
        ingest("ingest_128k_k3_v2", 1, 8, 128, 131072, kb=3, vb=2, chunk=4096, outliers=True),
        # A batch of prompts with sign sketches, head_dim 96.
        ingest("ingest_8k_b4_d96_qjl", 4, 32, 96, 8192, qjl=True),
        # A prompt for a caller that runs its own attention on the dense result.
        ingest("ingest_dense_4000_k3.5", 1, 8, 128, 4000, kb=3.5, vb=3.5, fetch=True, dtype="bf16"),
        # -- dense callers and the codec -----------------------------------------------------------------------------------
        # A decode step of such a caller at 8K.
        fetch("fetch_8k_b1", 1, 8, 128, 8192),
        # The round trip of 8 heads x 4096 vectors at 4 bits.
        codec("codec_4096x8_4bit", 8, 4096, 128, 4),
    ]


def decode(name, b, hq, hkv, d, ctx, *, kb=4, vb=2, qjl=False, dtype="fp16", sink=128):
    # One call per layer and token. Enough layers that a pass does not find the previous one's cache in L2 (a model has 16 to
    # 80 layers), few enough that the largest fit the card; a few tokens per pass.
    lane_bytes = b * hkv * (ctx * d * (kb + vb) / 8 + 512 * d)
    layers = max(1, min(8, int(192e6 / lane_bytes)))
    return dict(name=name, kind="decode", b=b, hq=hq, hkv=hkv, d=d, ctx=ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink,
                rw=128, chunk=0, layers=layers, tokens=4 if layers > 1 else 2)


def prefill(name, b, hq, hkv, d, ctx, new, *, kb=4, vb=2, dtype="fp16", sink=128):
    return dict(name=name, kind="prefill", b=b, hq=hq, hkv=hkv, d=d, ctx=ctx, new=new, kb=kb, vb=vb, qjl=False, dtype=dtype,
                sink=sink, rw=128, chunk=0)


def ingest(name, b, h, d, ctx, *, kb=4, vb=2, qjl=False, dtype="fp16", sink=128, chunk=0, fetch=False, outliers=False):
    return dict(name=name, kind="ingest", b=b, hkv=h, d=d, ctx=ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink, rw=128,
                chunk=chunk, fetch=fetch, outliers=outliers)


def fetch(name, b, h, d, ctx, *, kb=4, vb=2, qjl=False, dtype="fp16", sink=128):
    return dict(name=name, kind="fetch", b=b, hkv=h, d=d, ctx=ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink, rw=128, chunk=0)


def codec(name, lanes, rows, d, bits, *, dtype="fp16"):
    return dict(name=name, kind="codec", lanes=lanes, rows=rows, d=d, bits=bits, dtype=dtype)


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "ingest", "ingest", "fetch", "codec"))
    d = rng.choice((128, 128, 128, 128, 64, 96, 256))
    hq, hkv = rng.choice(((32, 8), (32, 8), (32, 8), (32, 32), (16, 2), (12, 4), (8, 8), (8, 1)))
    # 4-bit keys with 2-bit values are the default of apply_turboquant; the rest are the settings of the tests and the benchmark
    kb, vb = rng.choice(((4, 2), (4, 2), (4, 2), (3, 2), (3.5, 3.5), (4, 4), (2, 2), (3, 4)))
    dtype = rng.choice(("fp16", "bf16"))
    sink = rng.choice((128, 128, 0))
    qjl = rng.random() < 0.2
    if kind == "decode":
        ctx = logint(500, 32768)
        # widths other than the default and head_dim 256 stay at a quarter of the largest batch
        most = MOST_DECODE // (1 if (kb, vb) == (4, 2) and d <= 128 else 4)
        b = logint(1, max(1, min(64, most // (hkv * ctx * d))))
        c = decode("", b, hq, hkv, d, ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink)
    elif kind == "prefill":
        new = logint(4, 2048)
        ctx = new + logint(400, 16384)
        most = MOST_PREFILL // (1 if (kb, vb) == (4, 2) and d == 128 else 4)
        b = logint(1, max(1, min(8, most // (hq * new * ctx * d))))
        c = prefill("", b, hq, hkv, d, ctx, new, kb=kb, vb=vb, dtype=dtype, sink=sink)
    elif kind == "ingest":
        dense = rng.random() < 0.3
        ctx = logint(300, 16384 if dense else 131072)
        most = MOST_INGEST // (8 if dense or qjl or d == 256 else 1)
        ctx = min(ctx, most // (hkv * d))
        b = logint(1, max(1, min(16, most // (hkv * ctx * d))))
        c = ingest("", b, hkv, d, ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink, chunk=rng.choice((0, 0, 512, 4096)),
                   fetch=dense, outliers=rng.random() < 0.5)
    elif kind == "fetch":
        ctx = logint(500, 32768)
        b = logint(1, max(1, min(4, 8 * 32768 * 128 // (hkv * ctx * d))))
        c = fetch("", b, hkv, d, ctx, kb=kb, vb=vb, qjl=qjl, dtype=dtype, sink=sink)
    else:
        rows = logint(32, 131072)
        c = codec("", 8, rows, d, rng.choice((2, 3, 4, 4)), dtype=dtype)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------------------
def _rows(g, *shape, dtype, outliers=False):
    x = torch.randn(*shape, device="cuda", dtype=dtype, generator=g)
    x *= torch.exp(0.5 * torch.randn(*shape[:-1], 1, device="cuda", generator=g)).to(dtype)
    if outliers:
        d = shape[-1]
        for j in (3, 40 % d, 77 % d, 101 % d):
            x[..., j] *= 20.0
    return x


def _new_cache(case):
    return TurboQuantKVCache(head_dim=case["d"], num_kv_heads=case["hkv"], key_bits=case["kb"], value_bits=case["vb"],
                             residual_window=case["rw"], fp16_sink_size=case["sink"], chunk_size=case["chunk"],
                             qjl_correction=case["qjl"])


def _filled_cache(case, g, tokens):
    """A cache that holds ``tokens`` tokens, fed as a server feeds a prompt: in equal pieces of at most 2^29 values a side."""
    c = _new_cache(case)
    dt = DTYPES[case["dtype"]]
    piece = -(-tokens // -(-tokens * case["b"] * case["hkv"] * case["d"] // (1 << 29)))
    for at in range(0, tokens, piece):
        n = min(piece, tokens - at)
        c.update(_rows(g, case["b"], case["hkv"], n, case["d"], dtype=dt), _rows(g, case["b"], case["hkv"], n, case["d"], dtype=dt))
    return c


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    d = case["d"]
    s = {"case": case}
    if case["kind"] == "codec":
        s["x"] = _rows(g, 1, case["lanes"], case["rows"], d, dtype=dt)
        s["codec"] = TurboQuantMSE(d, bits=case["bits"])
        return s
    b, h = case["b"], case["hkv"]
    if case["kind"] == "decode":
        s["caches"] = [_filled_cache(case, g, case["ctx"] - case["tokens"]) for _ in range(case["layers"])]
        s["at"] = [c.meta_state for c in s["caches"]]
        s["steps"] = [[(torch.randn(b, case["hq"], 1, d, device="cuda", dtype=dt, generator=g) / d ** 0.5,
                        _rows(g, b, h, 1, d, dtype=dt), _rows(g, b, h, 1, d, dtype=dt)) for _ in range(case["layers"])]
                      for _ in range(case["tokens"])]
        # the recent-token buffers, to which the steps append in place
        n = [int(at["fp16_len"]) + case["tokens"] for at in s["at"]]
        s["recent"] = [(c.keys[:, :, :m], c.values[:, :, :m]) for c, m in zip(s["caches"], n)]
    elif case["kind"] == "prefill":
        s["cache"] = _filled_cache(case, g, case["ctx"] - case["new"])
        s["at"] = s["cache"].meta_state
        s["q"] = torch.randn(b, case["hq"], case["new"], d, device="cuda", dtype=dt, generator=g) / d ** 0.5
        s["k"], s["v"] = (_rows(g, b, h, case["new"], d, dtype=dt) for _ in range(2))
        # Once, so that the buffers have the room that the pass needs (see run) and hold what it leaves in them.
        s["cache"].update(s["k"], s["v"])
        s["at"]["fp16_capacity"] = s["cache"].meta_state["fp16_capacity"]
        s["cache"].meta_state = s["at"]
    elif case["kind"] == "ingest":
        s["k"], s["v"] = (_rows(g, b, h, case["ctx"], d, dtype=dt, outliers=case["outliers"]) for _ in range(2))
    else:
        s["cache"] = _filled_cache(case, g, case["ctx"] - 1)
        s["at"] = s["cache"].meta_state
        s["k"], s["v"] = (_rows(g, b, h, 1, d, dtype=dt) for _ in range(2))
        s["cache"].update_and_fetch(s["k"], s["v"])          # the prompt's dense middle, built by the steps before this one
        s["at"]["fp16_capacity"] = s["cache"].meta_state["fp16_capacity"]
        s["cache"].meta_state = s["at"]
    return s


def _contents(cache):
    """What the cache holds: its checkpoint state, of the recent-token buffers the tokens that count."""
    st = list(cache.state)
    n = int(cache.meta_state["fp16_len"])
    st[0], st[1] = (None if t is None else t[:, :, :n] for t in st[:2])
    return st


# ---- one pass ---------------------------------------------------------------------------------------------------------------
# A pass that appends to a cache ends by setting the cache's counters back (meta_state), as a program does that tries several
# continuations of one prompt: the next pass starts from the same lengths.
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        outs = [c.decode_step(q, k, v) for step in s["steps"] for c, (q, k, v) in zip(s["caches"], step)]
        for c, at in zip(s["caches"], s["at"]):
            c.meta_state = at
        return outs, s["recent"]
    if kind == "prefill":
        c = s["cache"]
        c.update(s["k"], s["v"])
        out = c.attend(s["q"])
        kept = _contents(c)
        c.meta_state = s["at"]
        return out, kept
    if kind == "ingest":
        c = _new_cache(case)
        if case["fetch"]:
            return c.update_and_fetch(s["k"], s["v"]), _contents(c)
        c.update(s["k"], s["v"])
        return _contents(c)
    if kind == "fetch":
        c = s["cache"]
        out = c.update_and_fetch(s["k"], s["v"])
        c.meta_state = s["at"]
        return out
    qt = s["codec"].quantize(s["x"])
    return qt.packed_indices, qt.norms, s["codec"].dequantize(qt)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def _regions(case, total):
    """(sink, packed, recent) tokens of a cache that was fed ``total`` tokens as _filled_cache feeds them, one prompt here."""
    sink = min(case["sink"], total)
    rest = total - sink
    rw, chunk = case["rw"], case["chunk"]
    if chunk > 0:
        packed = (rest - rw) // chunk * chunk if rest >= rw + chunk else 0
    else:
        packed = rest - rw if rest > 2 * rw else 0
    return sink, packed, rest - packed


def _packed_row_bytes(case):
    return case["d"] * (case["kb"] + case["vb"]) / 8 + 8 + (16 if case["qjl"] else 0)      # codes, norms, sketches of K and V


def work(case):
    kind, d = case["kind"], case["d"]
    if kind == "codec":
        n = case["lanes"] * case["rows"]
        packed = n * (d * case["bits"] / 8 + 4)
        return {"bytes": n * d * 2 + 2 * packed + n * d * 4, "flops": 4.0 * n * d * d}
    lanes = case["b"] * case["hkv"]
    sink, packed, recent = _regions(case, case["ctx"])
    held = lanes * (packed * _packed_row_bytes(case) + (sink + recent) * 4 * d)
    if kind == "decode":
        rows = case["b"] * case["hq"]
        one = held + rows * d * 4
        return {"bytes": one * case["layers"] * case["tokens"],
                "flops": 4.0 * rows * case["ctx"] * d * case["layers"] * case["tokens"]}
    if kind == "prefill":
        new, rows = case["new"], case["b"] * case["hq"]
        return {"bytes": held + lanes * new * 4 * d + rows * new * d * 4,
                "flops": 4.0 * rows * new * (case["ctx"] - new / 2) * d + 4.0 * lanes * new * d * d}
    if kind == "ingest":
        dense = lanes * case["ctx"] * d * (8 if packed else 4) if case["fetch"] else 0
        return {"bytes": lanes * case["ctx"] * 4 * d + held + dense, "flops": (8.0 if case["fetch"] else 4.0) * lanes * packed * d * d}
    return {"bytes": held + lanes * case["ctx"] * d * (8 if packed else 4), "flops": 4.0 * lanes * packed * d * d}


def tolerance(case):
    # Codes may differ where a rotated value lies within float32 rounding of a boundary (a few in 100,000), which moves a
    # dequantized vector by one level of one rotated coordinate; a sign word holds 32 projections of such a residual.
    differ = 5e-3 if case.get("qjl") else 5e-4
    if case["kind"] in ("decode", "prefill"):
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 4e-3, "max": 0.1, "differ": differ}
    if case["kind"] == "ingest" and not case["fetch"]:
        return {"rel": 5e-5, "max": 5e-3, "differ": differ}
    return {"rel": 1e-3, "max": 0.5, "differ": differ}
