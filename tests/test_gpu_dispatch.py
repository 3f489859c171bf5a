"""Where a call changes kernels: each path against the one beside it, at the sizes where a tile or a threshold ends."""

import pytest
import torch

import quashkv_b200 as qk
from quashkv_b200 import _lib
from quashkv_b200.integrations.vllm_backend import QuashKVPageConfig, QuashKVPagedCache
from helpers import attention_64, rel_l2, row_errors

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 3, 129, 6143, 6144, 6271, 9473])
def test_unpacked_codes_equal_the_packed_ones(n, dtype, monkeypatch):
    """One byte per coordinate and packed rows, at every width, on both sides of the size from which the tensor-core
    kernel runs, against the fp32 chain: whole numbers, so they are the same."""
    x = torch.randn(n, 128, generator=torch.Generator().manual_seed(n)).to(dtype).to(DEV)

    def chain(fn):
        monkeypatch.setenv("QUASHKV_B200_CUDA_CORE_ROTATION", "1")
        out = fn(x)
        monkeypatch.delenv("QUASHKV_B200_CUDA_CORE_ROTATION")
        return out

    for bits in (1, 2, 3, 4):
        q = qk.MSEQuantizer(128, bits, seed=42, device=DEV)
        codes, norms = q.compress(x)
        packed, norms_p = q.compress_packed(x)
        assert torch.equal(qk.unpack_bits(packed, bits, 128), codes) and torch.equal(norms, norms_p)
        want, norms_w = chain(q.compress)
        assert torch.equal(codes, want) and torch.equal(norms, norms_w)
    for bits in (2, 3, 4):
        q = qk.InnerProductQuantizer(128, bits, seed=42, device=DEV)
        codes, signs, norms = q.compress(x)
        packed, packed_s, norms_p = q.compress_packed(x)
        assert torch.equal(qk.unpack_bits(packed, bits - 1, 128), codes) and torch.equal(norms, norms_p)
        assert torch.equal(qk.unpack_bits(packed_s, 1, 128), signs)
        assert all(torch.equal(a, b) for a, b in zip((codes, signs, norms), chain(q.compress)))


def _outliers(g, shape, dtype):
    x = torch.randn(shape, generator=g, device=DEV)
    x[..., ::37] *= 8.0
    return x.to(dtype)


@pytest.mark.parametrize("D,kb,vb", [(128, 3, 3), (64, 3, 3), (64, 2, 4), (128, 4, 2), (128, 2, 4)])
@pytest.mark.parametrize("n,q_len,G,causal,dtype", [
    (64, 64, 1, True, torch.bfloat16),            # one token tile, half a row tile
    (65, 65, 2, True, torch.float32),             # one token into the second tile, one row tile and two rows
    (127, 33, 4, False, torch.float16),           # a short block of queries over an older cache
    (321, 130, 2, True, torch.bfloat16),          # rows of two heads in one row tile, a ragged end everywhere
    (1, 1, 160, False, torch.float32),            # a single token
    (640, 512, 1, True, torch.bfloat16),          # whole row tiles, heaviest first
    (1024, 512, 4, True, torch.bfloat16),         # ... of several heads, each with its own order; sixteen token tiles
    (1300, 1024, 8, True, torch.float32),         # ... over an older cache of ragged length
])
def test_prefill_kernels_match_the_decode_kernels(D, kb, vb, n, q_len, G, causal, dtype, monkeypatch):
    """The same call through the kernels of long and of short query blocks.  Both hold fp32 (about 5e-7 from 64-bit
    results) but at d = 128, 3/3 bits, where each rounds queries, tables and weights to fp16 (about 4e-4)."""
    g = torch.Generator(device=DEV).manual_seed(n + D)
    eng = qk.QuashKVEngine(D, kb, vb, seed=42, device=DEV, pack_storage=True)
    eng.append(_outliers(g, (2, 2, n, D), dtype), _outliers(g, (2, 2, n, D), dtype))
    q = torch.randn(2, 2 * G, q_len, D, generator=g, device=DEV).to(dtype)
    monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", "0")
    want = eng.attention(q, causal=causal)
    monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", "1")
    before = _lib.lib().qkv_tensor_core_timeouts()
    got = eng.attention(q, causal=causal)
    assert _lib.lib().qkv_tensor_core_timeouts() == before
    assert rel_l2(got, want) < (1e-3 if (D, kb, vb) == (128, 3, 3) else 5e-6)


@pytest.mark.parametrize("D,block", [(128, 16), (128, 48), (64, 16), (64, 20)])
def test_prefill_kernels_on_pages_of_unequal_sequences(D, block, monkeypatch):
    """Block tables in any order, sequences of different lengths (one of them empty), norms of a wide range."""
    n_seq, Hkv, G, q_len, longest = 4, 2, 2, 48, 300
    per_seq = -(-longest // block)
    g = torch.Generator(device=DEV).manual_seed(block)
    pool = QuashKVPagedCache(n_seq * per_seq, Hkv, D, QuashKVPageConfig(key_bits=3, value_bits=3, block_size=block), device=DEV)
    table = torch.randperm(n_seq * per_seq, generator=g, device=DEV).to(torch.int32).reshape(n_seq, per_seq)
    k, v = _outliers(g, (n_seq, Hkv, longest, D), torch.float32), _outliers(g, (n_seq, Hkv, longest, D), torch.float32)
    wide = 2 if D == 128 else 6                  # (the records' other kernels hold weight times norm in fp16)
    v *= torch.logspace(-wide, wide, longest, device=DEV)[None, None, :, None]
    pool.append_with_tables(k, v, table, torch.zeros(n_seq, dtype=torch.int32, device=DEV))
    lens = torch.tensor([300, 0, 63, 193], dtype=torch.int32, device=DEV)
    q = torch.randn(n_seq, Hkv * G, q_len, D, generator=g, device=DEV)
    for causal in (False, True):
        monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", "0")
        want = pool.attention_with_tables(q, table, lens, longest, causal=causal)
        monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", "1")
        got = pool.attention_with_tables(q, table, lens, longest, causal=causal)
        assert torch.equal(got[1], torch.zeros_like(got[1])) and torch.isfinite(got).all()
        for b in (0, 2, 3):
            assert rel_l2(got[b], want[b]) < (1e-3 if D == 128 else 5e-6), (b, causal)


@pytest.mark.parametrize("D,block", [(128, 16), (64, 16)])
def test_paged_append_of_a_repeated_sequence_id(D, block):
    """One call with an id listed twice stores what two calls with its entries one after the other store."""
    cfg = QuashKVPageConfig(key_bits=3, value_bits=3, block_size=block)
    k, v = (torch.randn(3, 2, 21, D, generator=torch.Generator().manual_seed(s)).to(DEV) for s in (1, 2))
    one, two = (QuashKVPagedCache(12, 2, D, cfg, device=DEV) for _ in range(2))
    one.append(["a", "b", "a"], k, v)
    two.append(["a", "b"], k[:2], v[:2])
    two.append(["a"], k[2:], v[2:])
    for s in ("a", "b"):
        assert one.seq_len(s) == two.seq_len(s)
        want = two.rows_of(s)
        assert all(torch.equal(t, want[name]) for name, t in one.rows_of(s).items())


@pytest.mark.parametrize("log2_step", [10, 20, 34, 60])
@pytest.mark.parametrize("D,bits", [(64, 3), (64, 4), (128, 4), (128, 3)])
def test_prefill_keeps_rows_beside_a_much_larger_value_norm(D, bits, log2_step, monkeypatch):
    """The last token of every 64 has value norms 2^step times the others': each row for itself, before and after it
    sees one.  fp32 arithmetic keeps a row to about 3e-6 whatever the norms, and so do hi + lo operands scaled per row.
    At d = 128, 3/3 bits a weight times a norm is one fp16 number, normal down to 2^-28 of the tile's largest norm that
    the row sees (roundings of 2^-12 to queries, tables and products: below 3e-3 a row); a neighbour that is in sight,
    2^34 larger and weighs nothing is beyond that, so those steps are checked on the rows of the first tile, which see
    none."""
    n = 130
    g = torch.Generator(device=DEV).manual_seed(D + log2_step)
    k, v = (_outliers(g, (1, 2, n, D), torch.float32) for _ in range(2))
    v[:, :, 63::64] *= 2.0 ** log2_step
    q = torch.randn(1, 4, n, D, generator=g, device=DEV)
    eng = qk.QuashKVEngine(D, bits, bits, seed=42, device=DEV, pack_storage=True)
    eng.append(k, v)
    monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", "1")
    err = row_errors(eng.attention(q, causal=True), attention_64(eng, q, True)).reshape(4, n)
    if (D, bits) != (128, 3):
        assert float(err.max()) < 1e-5
    else:
        assert float(err[:, :63].max()) < 3e-3 and (log2_step > 24 or float(err.max()) < 3e-3)


@pytest.mark.parametrize("D,bits", [(64, 2), (64, 3), (64, 4), (128, 2), (128, 4)])
@pytest.mark.parametrize("n,q_len,G,causal,dtype", [
    (48, 48, 8, True, torch.float16),
    (150, 150, 4, True, torch.float32),
    (517, 517, 2, True, torch.bfloat16),
    (1400, 90, 4, False, torch.float32),
    (2100, 300, 2, True, torch.bfloat16),
])
def test_prefill_is_no_further_from_64_bits_than_the_fp32_kernel(D, bits, n, q_len, G, causal, dtype, monkeypatch):
    """hi + lo operands and truncating sums in the place of fp32 on the CUDA cores: the error of the whole result, and of
    its rows, against 64-bit arithmetic is at most that of the kernel which took the call before.  (Measured 0.6 to 0.95
    of it; the inputs are fixed, so the comparison has no spread.)"""
    g = torch.Generator(device=DEV).manual_seed(1000 * bits + n)
    eng = qk.QuashKVEngine(D, bits, bits, seed=42, device=DEV, pack_storage=True)
    eng.append(_outliers(g, (2, 2, n, D), dtype), _outliers(g, (2, 2, n, D), dtype))
    q = torch.randn(2, 2 * G, q_len, D, generator=g, device=DEV).to(dtype)
    exact = attention_64(eng, q, causal)
    err = []
    for way in "01":
        monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", way)
        out = eng.attention(q, causal=causal)
        err.append((rel_l2(out, exact), float(row_errors(out, exact).square().mean().sqrt())))
    print(f"[precision] d={D} bits={bits} n={n} q={q_len}: fp32 {err[0][0]:.2e} / rows {err[0][1]:.2e}, "
          f"hi + lo {err[1][0]:.2e} / {err[1][1]:.2e}, ratios {err[1][0] / err[0][0]:.2f} {err[1][1] / err[0][1]:.2f}")
    assert err[1][0] <= err[0][0] and err[1][1] <= err[0][1]


def test_prefill_over_records_is_no_further_from_64_bits_than_the_decode_kernels(monkeypatch):
    """d = 128 at 3/3 bits: both ways round queries, tables and weights times norms to fp16 once, each for itself, so
    that a single shape can fall to either side; over many rows their errors are the same (to 2 %, the spread of the
    ratio over seeds)."""
    total = [0.0, 0.0]
    for n, q_len, G, causal, dtype in [(64, 64, 8, True, torch.float32), (300, 300, 4, True, torch.float16),
                                       (515, 70, 4, False, torch.float32), (1197, 1197, 1, True, torch.float32),
                                       (1400, 512, 2, True, torch.bfloat16), (2048, 2048, 2, True, torch.bfloat16)]:
        g = torch.Generator(device=DEV).manual_seed(n)
        eng = qk.QuashKVEngine(128, 3, 3, seed=42, device=DEV, pack_storage=True)
        eng.append(_outliers(g, (2, 2, n, 128), dtype), _outliers(g, (2, 2, n, 128), dtype))
        q = torch.randn(2, 2 * G, q_len, 128, generator=g, device=DEV).to(dtype)
        exact = attention_64(eng, q, causal)
        for way in (0, 1):
            monkeypatch.setenv("QUASHKV_B200_PREFILL_TCGEN05", str(way))
            total[way] += float(row_errors(eng.attention(q, causal=causal), exact).square().mean())
    print(f"[precision] records: decode kernels {(total[0] / 6) ** 0.5:.3e}, prefill {(total[1] / 6) ** 0.5:.3e}")
    assert total[1] <= total[0] * 1.02 ** 2


@pytest.mark.parametrize("lead", [(), (6,), (2, 3), (1, 2, 1, 3)])
@pytest.mark.parametrize("D", [128, 64])
def test_append_op_takes_any_leading_shape(lead, D):
    """Keys and values (..., T, d) go to the planes' segments in the order of their flattened leading dimensions; values
    of another leading shape (or fewer of them) to theirs."""
    T, cap, off = 5, 24, 3
    kq, vq = qk.InnerProductQuantizer(D, 3, seed=42, device=DEV), qk.MSEQuantizer(D, 3, seed=42, device=DEV)
    Pi, kb, kc, S = kq._on(torch.device(DEV, 0))
    vb = vq._on(torch.device(DEV, 0))[1]
    g = torch.Generator(device=DEV).manual_seed(D)
    segs = 1
    for n in lead:
        segs *= n
    k, v = (torch.randn(*lead, T, D, generator=g, device=DEV) for _ in range(2))
    codes, signs, norms = kq.compress_packed(k.reshape(segs, T, D))
    v_codes, v_norms = vq.compress_packed(v.reshape(segs, T, D))
    for values in (v, v.reshape(segs, T, D)[:1]):
        planes = [torch.zeros(segs, cap, t.shape[-1], dtype=torch.uint8, device=DEV) for t in (codes, signs, v_codes)]
        kn, vn = torch.zeros(segs, cap, device=DEV), torch.zeros(segs, cap, device=DEV)
        qk.ops.append_kv(k, values, Pi, kb, kc, S, 2, vb, 3, planes[0], planes[1], kn, planes[2], vn, off)
        n_v = values.numel() // (T * D)
        for got, want, n in ((planes[0], codes, segs), (planes[1], signs, segs), (kn, norms, segs), (planes[2], v_codes, n_v),
                             (vn, v_norms, n_v)):
            assert torch.equal(got[:n, off:off + T], want[:n])
            assert not got[:, :off].any() and not got[:, off + T:].any() and not got[n:].any()


def test_paged_append_op_refuses_tables_of_another_batch():
    """The kernel reads a table row and a start per sequence: fewer of them are refused on the host."""
    pool = QuashKVPagedCache(8, 2, 64, QuashKVPageConfig(block_size=16), device=DEV)
    x = torch.zeros(3, 2, 1, 64, device=DEV)
    table = torch.arange(6, dtype=torch.int32, device=DEV).reshape(3, 2)
    starts = torch.zeros(3, dtype=torch.int32, device=DEV)
    for t, s in ((table[:2], starts), (table, starts[:2]), (table[0], starts)):
        with pytest.raises(ValueError, match="block table and start lengths for 3 sequences"):
            pool._store(x, x, t, s)
    pool._store(x, x, table, starts)


@pytest.mark.parametrize("D,block", [(128, 16), (128, 12), (64, 16)])
@pytest.mark.parametrize("n_seq,T", [(3, 40), (8, 800)])
def test_positions_outside_the_table_are_dropped_and_counted(D, block, n_seq, T):
    """Both kinds of append (one launch; through the tensor-core kernels from 6144 rows on at d = 128): tokens past the
    table of their sequence store nothing, the count says how many, the others are where they belong."""
    H, width = 2, 2 * (T // block // 2) - 1                    # a table that is too short for every sequence
    room = width * block
    pool = QuashKVPagedCache(n_seq * width + 1, H, D, QuashKVPageConfig(block_size=block), device=DEV)
    ref = QuashKVPagedCache(n_seq * width + 1, H, D, QuashKVPageConfig(block_size=block), device=DEV)
    g = torch.Generator(device=DEV).manual_seed(T)
    k, v = (torch.randn(n_seq, H, T, D, generator=g, device=DEV) for _ in range(2))
    table = torch.randperm(n_seq * width, generator=g, device=DEV).to(torch.int32).reshape(n_seq, width)
    starts = torch.arange(n_seq, dtype=torch.int32, device=DEV) * 3
    before = pool.dropped_rows()
    pool.append_with_tables(k, v, table, starts)
    lost = sum(max(0, 3 * i + T - room) for i in range(n_seq))
    assert lost > 0 and pool.dropped_rows() - before == lost * H
    for i in range(n_seq):                                     # what fits, in calls of one sequence and a few tokens
        for t in range(0, room - 3 * i, 100):
            m = min(100, room - 3 * i - t)
            ref.append_with_tables(k[i:i + 1, :, t:t + m].contiguous(), v[i:i + 1, :, t:t + m].contiguous(), table[i:i + 1],
                                   starts[i:i + 1] + t)
    for name, plane in pool.planes.items():
        assert torch.equal(plane, ref.planes[name]), name
    assert pool.dropped_rows() - before == lost * H


def test_a_backward_pass_through_an_op_is_refused():
    """Gradients that do not exist are an error where they are asked for; the engine's attention is outside any graph."""
    pool = QuashKVPagedCache(4, 2, 64, QuashKVPageConfig(block_size=16), device=DEV)
    k = torch.randn(1, 2, 20, 64, device=DEV)
    pool.append(["a"], k, k)
    q = torch.randn(1, 4, 1, 64, device=DEV, requires_grad=True)
    with pytest.raises(RuntimeError, match="not implemented"):
        (pool.attention(["a"], q).sum() + q.sum()).backward()
    eng = qk.QuashKVEngine(64, 3, 3, seed=42, device=DEV)
    eng.append(k.requires_grad_(), k)
    assert not eng.attention(q).requires_grad
    with torch.no_grad():
        assert torch.equal(eng.attention(q), eng.attention(q.detach()))
    with torch.inference_mode():
        eng.append(torch.randn(1, 2, 3, 64, device=DEV), torch.randn(1, 2, 3, 64, device=DEV))
        assert eng.attention(torch.randn(1, 4, 1, 64, device=DEV)).shape == (1, 4, 1, 64)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,n", [(128, 5001), (96, 6007), (80, 6001), (64, 9473), (32, 18999), (20, 18945)])
def test_bulk_chain_kernels_equal_the_small_ones(D, n, dtype, monkeypatch):
    """The same fp32 chains in the kernel of many vectors and, in pieces of 1000, in that of few: the same bytes, norms
    and values, for every layout."""
    monkeypatch.setenv("QUASHKV_B200_CUDA_CORE_ROTATION", "1")
    x = _outliers(torch.Generator(device=DEV).manual_seed(D), (n, D), dtype)
    mixed = qk.MixedPrecisionMSEQuantizer(D, 3, 2, D // 4 + 1, seed=42, device=DEV)
    mixed.calibrate(x[:500].float())
    mse, ip = qk.MSEQuantizer(D, 4, seed=42, device=DEV), qk.InnerProductQuantizer(D, 3, seed=42, device=DEV)
    for fn in (mse.compress, mse.compress_packed, ip.compress, ip.compress_packed,
               lambda v: mixed.compress(v, packed=False), lambda v: mixed.compress(v, packed=True)):
        whole, parts = fn(x), [fn(x[i:i + 1000]) for i in range(0, n, 1000)]
        for i, got in enumerate(whole):
            assert torch.equal(got, torch.cat([p[i] for p in parts]))
    for codes, norms, fn in ((*mse.compress(x), mse.decompress), (*mse.compress_packed(x), mse.decompress_packed),
                             (*mixed.compress(x, packed=True), lambda c, s: mixed.decompress(c, s, packed=True)),
                             (*mixed.compress(x, packed=False), lambda c, s: mixed.decompress(c, s, packed=False))):
        assert torch.equal(fn(codes, norms), torch.cat([fn(codes[i:i + 1000], norms[i:i + 1000]) for i in range(0, n, 1000)]))


@pytest.mark.parametrize("k", [1, 7, 10, 31, 40, 100, 128])
@pytest.mark.parametrize("M,n", [(1, 2048), (3, 2049), (5, 8191), (2, 20000), (149, 2048), (200, 3333), (150, 8300)])
def test_merge_of_long_candidate_lists(M, n, k):
    """Every count of warps and loads: ties (few distinct scores), pairs that stand in the list twice (they count once),
    missing entries, and fewer candidates than results; rank order is by score, then by the smaller id."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    scores = torch.randint(-40, 40, (M, n), generator=g, device=DEV).float() / 8
    scores[:, ::2] += torch.randn(M, (n + 1) // 2, generator=g, device=DEV)
    ids = torch.randint(0, 3 * n, (M, n), generator=g, device=DEV)
    ids[:, 1::7] = ids[:, :-1:7][:, :ids[:, 1::7].shape[1]]                    # the same pair next to itself ...
    scores[:, 1::7] = scores[:, :-1:7][:, :scores[:, 1::7].shape[1]]
    ids[:, n // 2 + 5], scores[:, n // 2 + 5] = ids[:, 3], scores[:, 3]          # ... and in another warp's share
    ids[:, ::11] = -1
    ids[-1, 5:] = -1                                                           # hardly any candidates at all
    got_s, got_i = qk.ops.topk_merge(scores, ids, k)
    for m in {0, M // 2, M - 1}:
        pairs = sorted({(-s, i) for s, i in zip(scores[m].tolist(), ids[m].tolist()) if i >= 0})[:k]
        want = [(-s, i) for s, i in pairs] + [(float("-inf"), -1)] * (k - len(pairs))
        assert list(zip(got_s[m].tolist(), got_i[m].tolist())) == want
