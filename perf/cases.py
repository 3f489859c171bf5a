"""What is timed: the work that a user of this framework has it do, through the public classes.

Six kinds of pass, over the sizes that the repository's configurations, tests and benchmark use:

  prompt      a sequence (or a batch of them) arrives: engine.clear(), engine.append(K, V), engine.attention(Q).
              q_len = tokens with the causal mask is a prefill; q_len = 1 is the engine's quick-start.
  decode      one query token per sequence over a cache that is already there: engine.attention(Q).
  paged_step  one step of a serving loop over block tables: the new token of every sequence goes to its page, then
              every sequence attends over its own length.
  compress    quantizer.compress / compress_packed of a bulk tensor (keys "ip", values "mse", mixed precision).
  decompress  quantizer.decompress / decompress_packed of bulk codes.
  search      QuashIndex.search over a built index.

A case holds plain values only; `draw` gives more cases from the same ranges.
"""

from __future__ import annotations

import math

import torch

import quashkv_b200 as qk
from quashkv_b200.integrations.vllm_backend import QuashKVPageConfig, QuashKVPagedCache

DEV = "cuda"
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
CHUNK = 1 << 20          # vectors drawn and compressed at a time while a cache or an index is filled


def listed():
    return [
        # The quick-start and the smallest call: 512 fp32 tokens of 8 heads go in, one query comes out.
        {"name": "prompt_512_fp32", "kind": "prompt", "batch": 1, "kv_heads": 8, "q_heads": 8, "tokens": 512, "q_len": 1,
         "dim": 128, "key_bits": 3, "val_bits": 3, "dtype": "fp32"},
        # Prefill of the Llama-shaped generation loop (22 layers of 32 query / 4 KV heads, head size 64): one layer.
        {"name": "prompt_8x1024_d64", "kind": "prompt", "batch": 8, "kv_heads": 4, "q_heads": 32, "tokens": 1024,
         "q_len": 1024, "dim": 64, "key_bits": 3, "val_bits": 3, "dtype": "bf16"},
        # Prefill of two long prompts at the 8B-class layer shape (8 KV heads, 32 query heads, head size 128).
        {"name": "prompt_2x4096", "kind": "prompt", "batch": 2, "kv_heads": 8, "q_heads": 32, "tokens": 4096, "q_len": 4096,
         "dim": 128, "key_bits": 3, "val_bits": 3, "dtype": "bf16"},
        # Interactive decode: one sequence, a short history of a ragged length; latency and launches count.
        {"name": "decode_1x1000", "kind": "decode", "batch": 1, "kv_heads": 8, "q_heads": 32, "tokens": 1000, "dim": 128,
         "key_bits": 3, "val_bits": 3, "dtype": "bf16"},
        # A decode step of one layer of the Llama-shaped generation loop, at the 4-bit point of its sweep.
        {"name": "decode_8x1277_d64_4bit", "kind": "decode", "batch": 8, "kv_heads": 4, "q_heads": 32, "tokens": 1277,
         "dim": 64, "key_bits": 4, "val_bits": 4, "dtype": "bf16"},
        # The benchmark's workload: a large batch over a long cache, bound by the packed bytes.
        {"name": "decode_32x32768", "kind": "decode", "batch": 32, "kv_heads": 8, "q_heads": 32, "tokens": 32768, "dim": 128,
         "key_bits": 3, "val_bits": 3, "dtype": "bf16"},
        # A serving loop's step: 32 requests of different lengths on 16-token pages.
        {"name": "paged_step_32x16384", "kind": "paged_step", "batch": 32, "kv_heads": 8, "q_heads": 32, "tokens": 16384,
         "dim": 128, "key_bits": 3, "val_bits": 3, "block": 16, "dtype": "bf16"},
        # Bulk prefill compression at 2.5 effective bits, packed.
        {"name": "compress_mixed_1M", "kind": "compress", "quantizer": "mixed", "vectors": 16 * 8 * 8192, "dim": 128,
         "bits": 3, "regular_bits": 2, "packed": True, "dtype": "bf16"},
        # MSEQuantizer.compress as the reference's users call it: fp32 in, one byte per coordinate out, an odd count.
        {"name": "compress_mse_65537", "kind": "compress", "quantizer": "mse", "vectors": 65537, "dim": 128, "bits": 4,
         "regular_bits": 0, "packed": False, "dtype": "fp32"},
        # Bulk decompression of packed values to fp32.
        {"name": "decompress_mse_1M", "kind": "decompress", "quantizer": "mse", "vectors": 16 * 8 * 8192, "dim": 128,
         "bits": 3, "regular_bits": 0, "packed": True, "dtype": "fp32"},
        # One user's query against a million vectors.
        {"name": "search_1M_x1", "kind": "search", "vectors": 1_000_000, "queries": 1, "k": 10, "dim": 128, "bits": 3},
        # A batch of queries against the same index.
        {"name": "search_1M_x1024", "kind": "search", "vectors": 1_000_000, "queries": 1024, "k": 10, "dim": 128,
         "bits": 3},
    ]


# ---- more cases of the same ranges ----------------------------------------------------------------------------

def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _shape(rng):
    """(head size, key bits, value bits): mostly the default configuration, else another point of the sweeps."""
    if rng.random() < 0.5:
        return 128, 3, 3
    bits = rng.choice([2, 3, 4])
    return rng.choice([64, 64, 128]), bits, bits


def _heads(rng):
    return rng.choice([(8, 32), (8, 8), (4, 32), (8, 64), (2, 8)])


def draw(rng):
    kind = rng.choice(["prompt", "decode", "decode", "paged_step", "compress", "decompress", "search"])
    if kind in ("prompt", "decode", "paged_step"):
        dim, kb, vb = _shape(rng)
        hkv, hq = _heads(rng)
        case = {"kind": kind, "batch": 0, "kv_heads": hkv, "q_heads": hq, "tokens": 0, "dim": dim, "key_bits": kb,
                "val_bits": vb, "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"])}
        if kind == "prompt":
            tokens = _log_int(rng, 16, 4096 if (dim, kb, vb) == (128, 3, 3) else 1024)
            limit = 2 * 32 * 4096 ** 2 if (dim, kb, vb) == (128, 3, 3) else 8 * 32 * 1024 ** 2 * 64 // dim
            case.update(tokens=tokens, q_len=tokens if rng.random() < 0.8 else 1,
                        batch=_log_int(rng, 1, max(1, min(16, limit // (hq * tokens * tokens)))))
        else:
            tokens = _log_int(rng, 100, 32768 if kind == "decode" else 16384)
            limit = (32 * 8 * 32768 if kind == "decode" else 32 * 8 * 16384) // (1 if (dim, kb, vb) == (128, 3, 3) else 16)
            tokens = min(tokens, limit // hkv)
            case.update(tokens=tokens, batch=_log_int(rng, 1, max(1, min(64, limit // (hkv * tokens)))))
            if kind == "paged_step":
                case.update(block=rng.choice([16, 16, 32]))
        return case
    if kind in ("compress", "decompress"):
        quantizer = rng.choice(["mse", "ip", "mixed"] if kind == "compress" else ["mse", "mse", "mixed"])
        bits, regular = rng.choice([(3, 2), (4, 3), (4, 2)]) if quantizer == "mixed" else (rng.choice([2, 3, 4]), 0)
        dtype = "fp32" if kind == "decompress" and quantizer == "mixed" else rng.choice(["bf16", "fp32"])
        packed = rng.random() < 0.6 and not (kind == "compress" and quantizer == "ip" and rng.random() < 0.3)
        if kind == "decompress" and quantizer == "mse" and not packed:
            dtype = "fp32"
        return {"kind": kind, "quantizer": quantizer, "vectors": _log_int(rng, 64, 1 << 20),
                "dim": rng.choice([128, 128, 128, 64, 96]), "bits": bits, "regular_bits": regular, "packed": packed,
                "dtype": dtype}
    dim, bits, k = rng.choice([(128, 3, 10), (128, 3, 10), (128, 3, 1), (128, 3, 40), (128, 3, 100), (64, 3, 10), (128, 4, 10)])
    vectors = _log_int(rng, 20_000, 1_000_000)
    most = 1024 * 1_000_000 if (dim, bits) == (128, 3) and k <= 12 else 64 * 1_000_000
    return {"kind": "search", "vectors": vectors, "queries": _log_int(rng, 1, min(1024, most // vectors)), "k": k, "dim": dim,
            "bits": bits}


# ---- inputs ----------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _kv(g, batch, heads, tokens, dim, dtype):
    """Keys or values N(0, 1) with four outlier channels per head scaled x8, the same channels over the tokens."""
    x = torch.randn(batch, heads, tokens, dim, generator=g, device=DEV)
    scale = torch.ones(heads, dim, device=DEV)
    scale.scatter_(1, torch.rand(heads, dim, generator=g, device=DEV).argsort(1)[:, :4], 8.0)
    return (x * scale[None, :, None, :]).to(dtype)


def _fill_chunks(case):
    """(first token, tokens) of the appends that fill a cache."""
    step = max(1, CHUNK // (case["batch"] * case["kv_heads"]))
    return [(t, min(step, case["tokens"] - t)) for t in range(0, case["tokens"], step)]


def _prepare_prompt(case, g):
    shape = (case["batch"], case["kv_heads"], case["tokens"], case["dim"])
    dt = DTYPES[case["dtype"]]
    engine = qk.QuashKVEngine(case["dim"], case["key_bits"], case["val_bits"], seed=42, device=DEV, pack_storage=True)
    q = torch.randn(case["batch"], case["q_heads"], case["q_len"], case["dim"], generator=g, device=DEV).to(dt)
    return {"engine": engine, "k": _kv(g, *shape, dt), "v": _kv(g, *shape, dt), "q": q, "causal": case["q_len"] > 1}


def _run_prompt(s):
    s["engine"].clear()
    s["engine"].append(s["k"], s["v"])
    return s["engine"].attention(s["q"], causal=s["causal"])


def _prepare_decode(case, g):
    dt = DTYPES[case["dtype"]]
    engine = qk.QuashKVEngine(case["dim"], case["key_bits"], case["val_bits"], seed=42, device=DEV, pack_storage=True)
    engine.reserve(case["batch"], case["kv_heads"], case["tokens"])
    for _, n in _fill_chunks(case):
        shape = (case["batch"], case["kv_heads"], n, case["dim"])
        engine.append(_kv(g, *shape, dt), _kv(g, *shape, dt))
    q = torch.randn(case["batch"], case["q_heads"], 1, case["dim"], generator=g, device=DEV).to(dt)
    return {"engine": engine, "q": q}


def _run_decode(s):
    return s["engine"].attention(s["q"])


def _ragged_lengths(case):
    """Lengths of the sequences before the step: spread evenly from a sixteenth of the longest up to it."""
    lo, hi = max(1, case["tokens"] // 16), case["tokens"] - 1
    n = case["batch"]
    return [hi - (hi - lo) * i // max(n - 1, 1) for i in range(n)]


def _prepare_paged_step(case, g):
    dt, n, block = DTYPES[case["dtype"]], case["batch"], case["block"]
    per_seq = -(-case["tokens"] // block)
    config = QuashKVPageConfig(key_bits=case["key_bits"], value_bits=case["val_bits"], block_size=block)
    pool = QuashKVPagedCache(n * per_seq, case["kv_heads"], case["dim"], config, device=DEV)
    table = torch.rand(n * per_seq, generator=g, device=DEV).argsort().to(torch.int32).reshape(n, per_seq)
    for t, length in _fill_chunks(case):
        shape = (n, case["kv_heads"], length, case["dim"])
        pool.append_with_tables(_kv(g, *shape, dt), _kv(g, *shape, dt), table,
                                torch.full((n,), t, dtype=torch.int32, device=DEV))
    lens = torch.tensor(_ragged_lengths(case), dtype=torch.int32, device=DEV)
    lens = lens[torch.rand(n, generator=g, device=DEV).argsort()].contiguous()
    shape = (n, case["kv_heads"], 1, case["dim"])
    q = torch.randn(n, case["q_heads"], 1, case["dim"], generator=g, device=DEV).to(dt)
    return {"pool": pool, "table": table, "lens": lens, "lens_after": lens + 1, "longest": case["tokens"],
            "k": _kv(g, *shape, dt), "v": _kv(g, *shape, dt), "q": q}


def _run_paged_step(s):
    s["pool"].append_with_tables(s["k"], s["v"], s["table"], s["lens"])
    out = s["pool"].attention_with_tables(s["q"], s["table"], s["lens_after"], s["longest"])
    return out, s["pool"].planes


def _bulk(g, n, d, dtype):
    """N(0, 1) with a quarter of the channels heavy-tailed (Student t, 3 degrees of freedom, scaled x4)."""
    x = torch.randn(n, d, generator=g, device=DEV)
    tails = torch.rand(d, generator=g, device=DEV).argsort()[: d // 4]
    chi2 = torch.randn(3, n, d // 4, generator=g, device=DEV).square_().sum(0)
    x[:, tails] *= 4.0 / (chi2 / 3.0).sqrt_()
    return x.to(dtype)


def _quantizer(case, x):
    d = case["dim"]
    if case["quantizer"] == "mse":
        return qk.MSEQuantizer(d, case["bits"], seed=42, device=DEV)
    if case["quantizer"] == "ip":
        return qk.InnerProductQuantizer(d, case["bits"], seed=42, device=DEV)
    mixed = qk.MixedPrecisionMSEQuantizer(d, case["bits"], case["regular_bits"], d // 4, seed=42, device=DEV)
    mixed.calibrate(x[:4096].float())
    return mixed


def _compress(quantizer, case_packed, x):
    if isinstance(quantizer, qk.MixedPrecisionMSEQuantizer):
        return quantizer.compress(x, packed=case_packed)
    return quantizer.compress_packed(x) if case_packed else quantizer.compress(x)


def _prepare_compress(case, g):
    x = _bulk(g, case["vectors"], case["dim"], DTYPES[case["dtype"]])
    return {"quantizer": _quantizer(case, x), "x": x, "packed": case["packed"]}


def _run_compress(s):
    return _compress(s["quantizer"], s["packed"], s["x"])


def _prepare_decompress(case, g):
    x = _bulk(g, case["vectors"], case["dim"], torch.bfloat16)
    quantizer = _quantizer(case, x)
    codes, norms = _compress(quantizer, case["packed"], x)
    return {"quantizer": quantizer, "codes": codes, "norms": norms, "packed": case["packed"],
            "out_dtype": DTYPES[case["dtype"]]}


def _run_decompress(s):
    if isinstance(s["quantizer"], qk.MixedPrecisionMSEQuantizer):
        return s["quantizer"].decompress(s["codes"], s["norms"], packed=s["packed"])
    if s["packed"]:
        return s["quantizer"].decompress_packed(s["codes"], s["norms"], out_dtype=s["out_dtype"])
    return s["quantizer"].decompress(s["codes"], s["norms"])


def _prepare_search(case, g):
    """Database rows of norm U(0.5, 2), queries N(0, 1)."""
    index = qk.QuashIndex(case["dim"], case["bits"], seed=42, device=DEV, pack_storage=True)
    for at in range(0, case["vectors"], CHUNK):
        x = torch.randn(min(CHUNK, case["vectors"] - at), case["dim"], generator=g, device=DEV)
        norms = torch.rand(x.shape[0], 1, generator=g, device=DEV) * 1.5 + 0.5
        index.add(torch.nn.functional.normalize(x, dim=1) * norms)
    return {"index": index, "q": torch.randn(case["queries"], case["dim"], generator=g, device=DEV), "k": case["k"]}


def _run_search(s):
    return s["index"].search(s["q"], s["k"])


_PREPARE = {"prompt": _prepare_prompt, "decode": _prepare_decode, "paged_step": _prepare_paged_step,
            "compress": _prepare_compress, "decompress": _prepare_decompress, "search": _prepare_search}
_RUN = {"prompt": _run_prompt, "decode": _run_decode, "paged_step": _run_paged_step, "compress": _run_compress,
        "decompress": _run_decompress, "search": _run_search}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, _gen(seed))
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without, and what another correct implementation may differ by ------------------------

def _code_bytes(case):
    """Bytes of one vector's codes (and sign bits) as they are returned or read."""
    d = case["dim"]
    if not case["packed"]:
        return 2 * d if case["quantizer"] == "ip" else d
    if case["quantizer"] == "mixed":
        return -(-(d // 4) * case["bits"] // 8) + -(-(d - d // 4) * case["regular_bits"] // 8)
    return -(-d * case["bits"] // 8)


def work(case):
    size = {"fp32": 4, "bf16": 2, "fp16": 2}.get(case.get("dtype", "fp32"))
    d = case["dim"]
    if case["kind"] in ("compress", "decompress"):
        n = case["vectors"]
        return {"bytes": n * (size * d + _code_bytes(case) + 4), "flops": 2 * d * d * n}
    if case["kind"] == "search":
        n, m = case["vectors"], case["queries"]
        return {"bytes": n * (d * case["bits"] // 8 + 4) + m * (4 * d + 12 * case["k"]), "flops": 4 * d * n * m}
    heads = case["batch"] * case["kv_heads"]
    q_rows = case["batch"] * case["q_heads"] * case.get("q_len", 1)
    token = d * (case["key_bits"] + case["val_bits"]) // 8 + 8          # packed bytes of one token of one KV head
    io = q_rows * d * (size + 4)
    rotations = 2 * 2 * d * d * q_rows                                   # queries in, outputs back
    if case["kind"] == "prompt":
        n = case["tokens"]
        seen = (n + 1) / 2 if case["q_len"] > 1 else n
        return {"bytes": heads * n * (2 * size * d + 2 * token) + io,
                "flops": 4 * d * q_rows * seen + rotations + 2 * 2 * d * d * heads * n}
    if case["kind"] == "decode":
        return {"bytes": heads * case["tokens"] * token + io, "flops": 4 * d * q_rows * case["tokens"] + rotations}
    lengths = _ragged_lengths(case)
    tokens = sum(lengths) + len(lengths)
    return {"bytes": case["kv_heads"] * tokens * token + heads * (2 * size * d + token) + io,
            "flops": 4 * d * case["q_heads"] * tokens + rotations + 2 * 2 * d * d * heads}


def tolerance(case):
    if case["kind"] == "compress":
        return {"rel": 1e-6}                     # codes and sign bits are whole numbers: the same; norms are fp32
    if case["kind"] == "decompress":
        return {"rel": 4e-3 if case["dtype"] == "bf16" else 1e-5}
    if case["kind"] == "search":
        return {"rel": 1e-5, "differ": 1e-3}     # fp32 scores; ids of near-ties may change places
    if (case["dim"], case["key_bits"], case["val_bits"]) == (128, 3, 3):
        return {"rel": 1e-3}                     # softmax weights and values are multiplied as fp16
    return {"rel": 2e-5}                         # fp32 throughout
