"""PyTorch custom ops (namespace ``quashkv_b200``) over the C ABI of libquashkv_b200.so.

Each op allocates its outputs and workspace with torch, passes raw device
pointers and the current CUDA stream to one ``extern "C"`` entry point, and
returns.  Only a CUDA implementation is registered: calling an op on CPU
tensors raises from the dispatcher, there is no fallback.

The ops of the hot paths (schemas below) are implemented in csrc/host_ops.cpp:
their host side is native.  The others (packing, row scatter, layout changes,
dense index scores) are Python over ctypes.

Plain Python wrappers of the same names (``ops.compress_mse(...)``) are what the
host classes call; they normalise shapes and dtypes and then invoke the
registered op.
"""

from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import _lib
from ._lib import Rows, TILE_BYTES, TILE_TOKENS

_DT = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}


def packed_row_bytes(d: int, bits: int) -> int:
    """Bytes of one packed row: 3-bit rows are whole 8-field groups (3 bytes each), like the
    reference's pack_bits (quashkv/packing.py:61-81); otherwise ceil(d*bits/8)."""
    if bits == 8:
        return d
    return 3 * ((d + 7) // 8) if bits == 3 else (d * bits + 7) // 8


def _p(t: Optional[torch.Tensor]):
    """Device pointer of a tensor for the C call.  A host pointer must never reach a kernel: anything that is
    not a CUDA tensor is refused here."""
    if t is None:
        return None
    if not t.is_cuda:
        raise ValueError(f"quashkv_b200: expected a CUDA tensor, got one on {t.device}")
    return C.c_void_p(t.data_ptr())


def _same_device(device: torch.device, *tensors: Optional[torch.Tensor]) -> None:
    """Data tensors (codes, norms, records, tables of indices) are not moved for the caller: they have to be on
    the device the call runs on."""
    for t in tensors:
        if t is not None and t.device != device:
            raise ValueError(f"quashkv_b200: tensors of one call on different devices ({t.device} and {device})")


def _stream(t: torch.Tensor):
    return C.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _f32(t: torch.Tensor, device: Optional[torch.device] = None) -> torch.Tensor:
    """fp32, contiguous, and on `device` when one is given (small constants such as Pi, tables and S follow the
    data; the quantizer classes keep per-device copies, the functional entry points convert per call)."""
    t = t.detach()
    return t.to(device=t.device if device is None else device, dtype=torch.float32).contiguous()


class _Keep:
    """Device pointers of converted arguments, with the converted tensors held until the C call has
    returned: a pointer taken from a temporary would otherwise outlive its storage, and the next allocation
    on the stream could hand that storage out again before the kernel has read it."""

    def __init__(self, device: torch.device):
        self.held = []
        self.device = device

    def f32(self, t: Optional[torch.Tensor]):
        if t is None:
            return None
        t = _f32(t, self.device)
        self.held.append(t)
        return _p(t)

    def u8(self, t: torch.Tensor):
        t = t.detach().to(device=self.device, dtype=torch.uint8).contiguous()
        self.held.append(t)
        return _p(t)


# Ops implemented in csrc/host_ops.cpp.
_LIBRARY = torch.library.Library("quashkv_b200", "FRAGMENT")
_CONSTS = "Tensor Pi, Tensor key_centroids, Tensor val_centroids, Tensor S, float qjl_scale, float scale, bool causal"
_APPEND = ("Tensor keys, Tensor values, Tensor Pi, Tensor k_bounds, Tensor k_cents, Tensor S, SymInt mse_bits, "
           "Tensor v_bounds, SymInt val_bits")
_TILED = ("Tensor q, Tensor records, SymInt capacity, SymInt kv_len, SymInt n_kv_heads, Tensor? block_table, Tensor? seq_lens, "
          f"SymInt block_size, {_CONSTS}")
for _schema in (
        "compress_mse(Tensor x, Tensor Pi, Tensor boundaries, SymInt bits, bool packed) -> (Tensor, Tensor)",
        "compress_ip(Tensor x, Tensor Pi, Tensor boundaries, Tensor centroids, Tensor S, SymInt mse_bits, bool packed) "
        "-> (Tensor, Tensor, Tensor)",
        "compress_ip_into(Tensor x, Tensor Pi, Tensor boundaries, Tensor centroids, Tensor S, SymInt mse_bits, "
        "Tensor(a!) codes, Tensor(b!) signs, Tensor(c!) norms, SymInt offset) -> ()",
        "compress_mixed(Tensor x, Tensor Pi, Tensor is_outlier, Tensor bounds_out, SymInt bits_out, Tensor bounds_reg, "
        "SymInt bits_reg, bool packed, SymInt n_out) -> (Tensor, Tensor)",
        f"append_kv({_APPEND}, Tensor(a!) k_codes, Tensor(b!) k_signs, Tensor(c!) k_norms, Tensor(d!) v_codes, "
        "Tensor(e!) v_norms, SymInt offset) -> ()",
        f"append_records({_APPEND}, Tensor(a!) records, SymInt capacity, SymInt offset) -> ()",
        f"append_paged({_APPEND}, Tensor(a!)[] planes, Tensor block_table, Tensor start_lens, SymInt block_size) -> ()",
        "decompress(Tensor codes, Tensor? signs, Tensor norms, Tensor Pi, Tensor centroids, SymInt bits, Tensor? S, "
        "float qjl_scale, bool packed, SymInt d, SymInt seg_len, SymInt seg_stride, SymInt seg_off, SymInt n_vec, "
        "ScalarType out_dtype) -> Tensor",
        "decompress_dense(Tensor codes, Tensor? signs, Tensor norms, Tensor Pi, Tensor centroids, SymInt bits, Tensor? S, "
        "float qjl_scale, bool packed, SymInt d, ScalarType out_dtype) -> Tensor",
        "decompress_mixed(Tensor codes, Tensor norms, Tensor Pi, Tensor is_outlier, Tensor cents_out, SymInt bits_out, "
        "Tensor cents_reg, SymInt bits_reg, bool packed, SymInt d) -> Tensor",
        "attention(Tensor q, Tensor k_codes, Tensor k_signs, Tensor k_norms, Tensor v_codes, Tensor v_norms, "
        f"SymInt kv_len, SymInt n_kv_heads, SymInt key_bits, SymInt val_bits, {_CONSTS}) -> Tensor",
        "attention_paged(Tensor q, Tensor k_codes, Tensor k_signs, Tensor k_norms, Tensor v_codes, Tensor v_norms, "
        f"Tensor block_table, Tensor seq_lens, SymInt max_kv_len, SymInt key_bits, SymInt val_bits, {_CONSTS}) -> Tensor",
        f"attention_tiled({_TILED}) -> Tensor",
        f"attention_tiled_out({_TILED}, Tensor(a!) out) -> ()",
        "index_scan_topk(Tensor queries, Tensor db_codes, Tensor db_signs, Tensor db_norms, SymInt n_vectors, SymInt bits, "
        "Tensor Pi, Tensor centroids, Tensor S, float qjl_scale, SymInt k, SymInt id_base) -> (Tensor, Tensor)"):
    _LIBRARY.define(_schema, tags=torch.Tag.pt2_compliant_tag)
_NATIVE = torch.ops.quashkv_b200
_lib.load_host(required=False)        # not built yet: the first call says so


def _flat(x: torch.Tensor):
    d = x.shape[-1]
    if x.dtype not in _DT:
        x = x.float()
    return x.detach().reshape(-1, d).contiguous(), d


def _dense(n: int) -> Rows:
    return Rows(max(n, 1), 0, 0)


# ---------------------------------------------------------------------------------------------
# op implementations (CUDA only)
# ---------------------------------------------------------------------------------------------

@torch.library.custom_op("quashkv_b200::pack", mutates_args=(), device_types="cuda")
def _pack(codes: torch.Tensor, bits: int) -> torch.Tensor:
    d = codes.shape[-1]
    flat = codes.reshape(-1, d).contiguous()
    out = torch.empty((flat.shape[0], packed_row_bytes(d, bits)), dtype=torch.uint8, device=codes.device)
    A = _Keep(codes.device)
    with torch.cuda.device(codes.device):
        _lib.check(_lib.lib().qkv_pack(_p(flat), _p(out), flat.shape[0], d, bits, _stream(codes)), "pack")
    return out.reshape(*codes.shape[:-1], out.shape[1])


@_pack.register_fake
def _(codes, bits):
    return codes.new_empty((*codes.shape[:-1], packed_row_bytes(codes.shape[-1], bits)))


@torch.library.custom_op("quashkv_b200::unpack", mutates_args=(), device_types="cuda")
def _unpack(packed: torch.Tensor, bits: int, d: int) -> torch.Tensor:
    flat = packed.reshape(-1, packed.shape[-1])
    need = packed_row_bytes(d, bits)
    if flat.shape[1] < need:
        raise ValueError(f"packed rows of {flat.shape[1]} bytes cannot hold {d} fields of {bits} bits")
    flat = flat[:, :need].contiguous()
    out = torch.empty((flat.shape[0], d), dtype=torch.uint8, device=packed.device)
    A = _Keep(packed.device)
    with torch.cuda.device(packed.device):
        _lib.check(_lib.lib().qkv_unpack(_p(flat), _p(out), flat.shape[0], d, bits, _stream(packed)), "unpack")
    return out.reshape(*packed.shape[:-1], d)


@_unpack.register_fake
def _(packed, bits, d):
    return packed.new_empty((*packed.shape[:-1], d))


@torch.library.register_fake("quashkv_b200::compress_mse")
def _(x, Pi, boundaries, bits, packed):
    d = x.shape[-1]
    width = packed_row_bytes(d, bits) if packed else d
    return (x.new_empty((*x.shape[:-1], width), dtype=torch.uint8),
            x.new_empty(x.shape[:-1], dtype=torch.float32))


@torch.library.register_fake("quashkv_b200::compress_ip")
def _(x, Pi, boundaries, centroids, S, mse_bits, packed):
    d = x.shape[-1]
    cw = packed_row_bytes(d, mse_bits) if packed else d
    sw = packed_row_bytes(d, 1) if packed else d
    return (x.new_empty((*x.shape[:-1], cw), dtype=torch.uint8),
            x.new_empty((*x.shape[:-1], sw), dtype=torch.uint8),
            x.new_empty(x.shape[:-1], dtype=torch.float32))


@torch.library.register_fake("quashkv_b200::compress_mixed")
def _(x, Pi, is_outlier, bounds_out, bits_out, bounds_reg, bits_reg, packed, n_out):
    d = x.shape[-1]
    width = (n_out * bits_out + 7) // 8 + ((d - n_out) * bits_reg + 7) // 8 if packed else d
    return (x.new_empty((*x.shape[:-1], width), dtype=torch.uint8),
            x.new_empty(x.shape[:-1], dtype=torch.float32))


@torch.library.custom_op("quashkv_b200::compress_mixed_ip", mutates_args=(), device_types="cuda")
def _compress_mixed_ip(x: torch.Tensor, Pi: torch.Tensor, is_outlier: torch.Tensor,
                       bounds_out: torch.Tensor, cents_out: torch.Tensor, bits_out: int,
                       bounds_reg: torch.Tensor, cents_reg: torch.Tensor, bits_reg: int,
                       S: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Mixed-precision codes and residual sign bits, one uint8 per coordinate each, and the norms."""
    flat, d = _flat(x)
    n = flat.shape[0]
    codes = torch.empty((n, d), dtype=torch.uint8, device=x.device)
    signs = torch.empty((n, d), dtype=torch.uint8, device=x.device)
    norms = torch.empty((n,), dtype=torch.float32, device=x.device)
    A = _Keep(x.device)
    with torch.cuda.device(x.device):
        _lib.check(_lib.lib().qkv_compress_mixed_ip(
            _p(flat), _DT[flat.dtype], d, n, d, A.f32(Pi), A.u8(is_outlier), A.f32(bounds_out), A.f32(cents_out),
            bits_out, A.f32(bounds_reg), A.f32(cents_reg), bits_reg, A.f32(S), _p(codes), _p(signs), 0, _p(norms),
            _dense(n), _stream(x)), "compress_mixed_ip")
    lead = x.shape[:-1]
    return codes.reshape(*lead, d), signs.reshape(*lead, d), norms.reshape(lead)


@_compress_mixed_ip.register_fake
def _(x, Pi, is_outlier, bounds_out, cents_out, bits_out, bounds_reg, cents_reg, bits_reg, S):
    return (x.new_empty(x.shape, dtype=torch.uint8), x.new_empty(x.shape, dtype=torch.uint8),
            x.new_empty(x.shape[:-1], dtype=torch.float32))


@torch.library.register_fake("quashkv_b200::decompress")
def _(codes, signs, norms, Pi, centroids, bits, S, qjl_scale, packed, d, seg_len, seg_stride, seg_off,
      n_vec, out_dtype):
    return codes.new_empty((n_vec, d), dtype=out_dtype)


@torch.library.register_fake("quashkv_b200::decompress_dense")
def _(codes, signs, norms, Pi, centroids, bits, S, qjl_scale, packed, d, out_dtype):
    return codes.new_empty((*codes.shape[:-1], d), dtype=out_dtype)


@torch.library.register_fake("quashkv_b200::decompress_mixed")
def _(codes, norms, Pi, is_outlier, cents_out, bits_out, cents_reg, bits_reg, packed, d):
    return codes.new_empty((*codes.shape[:-1], d), dtype=torch.float32)


@torch.library.register_fake("quashkv_b200::attention")
def _(q, k_codes, k_signs, k_norms, v_codes, v_norms, kv_len, n_kv_heads, key_bits, val_bits, Pi,
      key_centroids, val_centroids, S, qjl_scale, scale, causal):
    return q.new_empty(q.shape, dtype=torch.float32)


@torch.library.register_fake("quashkv_b200::attention_paged")
def _(q, k_codes, k_signs, k_norms, v_codes, v_norms, block_table, seq_lens, max_kv_len, key_bits, val_bits, Pi,
      key_centroids, val_centroids, S, qjl_scale, scale, causal):
    return q.new_empty(q.shape, dtype=torch.float32)


@torch.library.custom_op("quashkv_b200::scatter_rows", mutates_args=("dst",), device_types="cuda")
def _scatter_rows(src: torch.Tensor, dst: torch.Tensor, slots: torch.Tensor) -> None:
    """Row i of src (n, ...) goes to row slots[i] of dst (rows, ...); rows are whole trailing slices."""
    n = slots.numel()
    row_bytes = (src.numel() // max(n, 1)) * src.element_size()
    _same_device(src.device, src, dst, slots)
    A = _Keep(src.device)
    with torch.cuda.device(src.device):
        _lib.check(_lib.lib().qkv_scatter_rows(_p(src), _p(dst), _p(slots), n, row_bytes, _stream(src)),
                   "scatter_rows")


# ---- tile records (the cache layout of the tensor-core decode kernel) ---------------------------------

def tiled_layout_ok(d: int, key_bits: int, val_bits: int) -> bool:
    """Tile records exist for head_dim 128 with 3-bit keys and 3-bit values."""
    return d == 128 and key_bits == 3 and val_bits == 3


def tiled_tables_ok(key_centroids: torch.Tensor, value_centroids: torch.Tensor) -> bool:
    """What the tile records and their decode kernel presume of the tables (the kernel writes NaN otherwise):
    a symmetric 8-entry value table and a 4-entry key table that is affine in the two bits of its code."""
    kc, vc = key_centroids.detach().float().cpu(), value_centroids.detach().float().cpu()
    if kc.numel() != 4 or vc.numel() != 8:
        return False
    sym = float((vc + vc.flip(0)).abs().max()) <= 1e-6 * float(vc.abs().max())
    aff = abs(float((kc[3] - kc[2]) - (kc[1] - kc[0]))) <= 1e-6 * float(kc.abs().max())
    return sym and aff


@torch.library.custom_op("quashkv_b200::tile_rows", mutates_args=("records",), device_types="cuda")
def _tile_rows(k_codes: torch.Tensor, k_signs: torch.Tensor, k_norms: torch.Tensor, v_codes: torch.Tensor,
               v_norms: torch.Tensor, records: torch.Tensor, seg_len: int, seg_stride: int, seg_off: int,
               slots: Optional[torch.Tensor]) -> None:
    """File dense packed rows (n, 32 / 16 / 48 bytes, fp32 norms) into 16-token tile records.  Row i goes to
    token slot slots[i], or (i // seg_len) * seg_stride + seg_off + i % seg_len when slots is None."""
    n = k_norms.numel()
    _same_device(records.device, records, k_codes, k_signs, k_norms, v_codes, v_norms, slots)
    A = _Keep(records.device)
    with torch.cuda.device(records.device):
        _lib.check(_lib.lib().qkv_tile_rows(
            _p(k_codes), _p(k_signs), _p(k_norms), _p(v_codes), _p(v_norms), n, _p(records),
            Rows(max(seg_len, 1), seg_stride, seg_off), _p(slots), _stream(records)), "tile_rows")


@torch.library.custom_op("quashkv_b200::untile_rows", mutates_args=(), device_types="cuda")
def _untile_rows(records: torch.Tensor, n_rows: int, seg_len: int, seg_stride: int, seg_off: int,
                 slots: Optional[torch.Tensor]) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """The reference's packed rows of n_rows token slots of a tiled cache: (k_codes (n,32), k_signs (n,16),
    k_norms (n), v_codes (n,48), v_norms (n))."""
    dev = records.device
    kc = torch.empty((n_rows, 32), dtype=torch.uint8, device=dev)
    ks = torch.empty((n_rows, 16), dtype=torch.uint8, device=dev)
    kn = torch.empty((n_rows,), dtype=torch.float32, device=dev)
    vc = torch.empty((n_rows, 48), dtype=torch.uint8, device=dev)
    vn = torch.empty((n_rows,), dtype=torch.float32, device=dev)
    _same_device(dev, records, slots)
    A = _Keep(dev)
    with torch.cuda.device(dev):
        _lib.check(_lib.lib().qkv_untile_rows(
            _p(records), Rows(max(seg_len, 1), seg_stride, seg_off), _p(slots), n_rows, _p(kc), _p(ks), _p(kn),
            _p(vc), _p(vn), _stream(records)), "untile_rows")
    return kc, ks, kn, vc, vn


@_untile_rows.register_fake
def _(records, n_rows, seg_len, seg_stride, seg_off, slots):
    u8 = lambda w: records.new_empty((n_rows, w), dtype=torch.uint8)      # noqa: E731
    f32 = lambda: records.new_empty((n_rows,), dtype=torch.float32)       # noqa: E731
    return u8(32), u8(16), f32(), u8(48), f32()


_CUDART = None


def cudart():
    """The CUDA runtime that torch has loaded, through ctypes: raw asynchronous copies and event calls for the
    host-buffer path, where the stream context managers of torch cost more than the device work of a short
    decode step."""
    global _CUDART
    if _CUDART is None:
        rt = C.CDLL("libcudart.so.12")
        rt.cudaMemcpyAsync.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_void_p]
        rt.cudaMemcpyAsync.restype = C.c_int
        rt.cudaEventRecord.argtypes = [C.c_void_p, C.c_void_p]
        rt.cudaEventRecord.restype = C.c_int
        rt.cudaStreamWaitEvent.argtypes = [C.c_void_p, C.c_void_p, C.c_uint]
        rt.cudaStreamWaitEvent.restype = C.c_int
        _CUDART = rt
    return _CUDART


@torch.library.register_fake("quashkv_b200::attention_tiled")
def _(q, records, capacity, kv_len, n_kv_heads, block_table, seq_lens, block_size, Pi, key_centroids,
      val_centroids, S, qjl_scale, scale, causal):
    return q.new_empty(q.shape, dtype=torch.float32)


@torch.library.register_fake("quashkv_b200::index_scan_topk")
def _(queries, db_codes, db_signs, db_norms, n_vectors, bits, Pi, centroids, S, qjl_scale, k, id_base):
    M = queries.shape[0]
    return queries.new_empty((M, k), dtype=torch.float32), queries.new_empty((M, k), dtype=torch.int64)


@torch.library.custom_op("quashkv_b200::index_scores", mutates_args=(), device_types="cuda")
def _index_scores(queries: torch.Tensor, db_codes: torch.Tensor, db_signs: torch.Tensor,
                  db_norms: torch.Tensor, n_vectors: int, bits: int, Pi: torch.Tensor,
                  centroids: torch.Tensor, S: torch.Tensor, qjl_scale: float) -> torch.Tensor:
    qf = _f32(queries)
    M, d = qf.shape
    out = torch.empty((M, n_vectors), dtype=torch.float32, device=qf.device)
    L = _lib.lib()
    ws_bytes = L.qkv_index_workspace_bytes(n_vectors, M, d, 1)
    ws = torch.empty((max(ws_bytes, 16),), dtype=torch.uint8, device=qf.device)
    _same_device(qf.device, qf, db_codes, db_signs, db_norms)
    A = _Keep(qf.device)
    with torch.cuda.device(qf.device):
        _lib.check(L.qkv_index_scores(
            _p(qf), M, d, _p(db_codes), _p(db_signs), _p(db_norms), n_vectors, bits, A.f32(Pi),
            A.f32(centroids), A.f32(S), float(qjl_scale), _p(out), _p(ws), ws_bytes, _stream(qf)),
            "index_scores")
    return out


@_index_scores.register_fake
def _(queries, db_codes, db_signs, db_norms, n_vectors, bits, Pi, centroids, S, qjl_scale):
    return queries.new_empty((queries.shape[0], n_vectors), dtype=torch.float32)


@torch.library.custom_op("quashkv_b200::topk_merge", mutates_args=(), device_types="cuda")
def _topk_merge(scores: torch.Tensor, ids: torch.Tensor, k: int) -> tuple[torch.Tensor, torch.Tensor]:
    s = _f32(scores)
    i = ids.to(torch.int64).contiguous()
    M, n_cand = s.shape
    out_s = torch.empty((M, k), dtype=torch.float32, device=s.device)
    out_i = torch.empty((M, k), dtype=torch.int64, device=s.device)
    _same_device(s.device, s, i)
    A = _Keep(s.device)
    with torch.cuda.device(s.device):
        _lib.check(_lib.lib().qkv_topk_merge(_p(s), _p(i), M, n_cand, k, _p(out_s), _p(out_i), _stream(s)),
                   "topk_merge")
    return out_s, out_i


@_topk_merge.register_fake
def _(scores, ids, k):
    M = scores.shape[0]
    return scores.new_empty((M, k), dtype=torch.float32), ids.new_empty((M, k), dtype=torch.int64)


append_kv = _NATIVE.append_kv.default
append_records = _NATIVE.append_records.default
append_paged = _NATIVE.append_paged.default
compress_ip_into = _NATIVE.compress_ip_into.default
attention = _NATIVE.attention.default
attention_paged = _NATIVE.attention_paged.default
attention_tiled = _attention_tiled = _NATIVE.attention_tiled.default
attention_tiled_out = _NATIVE.attention_tiled_out.default
index_scan_topk = _NATIVE.index_scan_topk.default
_compress_mse = _NATIVE.compress_mse.default
_compress_ip = _NATIVE.compress_ip.default
_compress_mixed = _NATIVE.compress_mixed.default
_decompress = _NATIVE.decompress.default
_decompress_dense = _NATIVE.decompress_dense.default
_decompress_mixed = _NATIVE.decompress_mixed.default


# ---------------------------------------------------------------------------------------------
# public wrappers
# ---------------------------------------------------------------------------------------------

def _need_cuda(t: torch.Tensor, what: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(
            f"quashkv_b200.{what}: expected a CUDA tensor, got device '{t.device}'. The hot path runs "
            "only as sm_100a kernels; there is no CPU implementation.")
    if not _lib.HOST_READY:
        _lib.load_host()


def pack(codes, bits):
    if bits == 8:
        return codes
    if bits not in (1, 2, 3, 4):
        raise ValueError(f"Unsupported bits: {bits}")
    _need_cuda(codes, "pack")
    return _pack(codes, bits)


def unpack(packed, bits, d):
    if bits == 8:
        return packed
    if bits not in (1, 2, 3, 4):
        raise ValueError(f"Unsupported bits: {bits}")
    _need_cuda(packed, "unpack")
    return _unpack(packed, bits, d)


def compress_mse(x, Pi, boundaries, bits, packed=False):
    _need_cuda(x, "compress_mse")
    return _compress_mse(x, Pi, boundaries, bits, packed)


def compress_ip(x, Pi, boundaries, centroids, S, mse_bits, packed=False):
    _need_cuda(x, "compress_ip")
    return _compress_ip(x, Pi, boundaries, centroids, S, mse_bits, packed)


def compress_mixed(x, Pi, is_outlier, bounds_out, bits_out, bounds_reg, bits_reg, packed=False, n_out=None):
    """``n_out``: how many channels ``is_outlier`` marks; counted here (one device read) when not given."""
    _need_cuda(x, "compress_mixed")
    if n_out is None:
        n_out = int(is_outlier.sum().item()) if packed else 0
    return _compress_mixed(x, Pi, is_outlier, bounds_out, bits_out, bounds_reg, bits_reg, packed, int(n_out))


def compress_mixed_ip(x, Pi, is_outlier, bounds_out, cents_out, bits_out, bounds_reg, cents_reg, bits_reg, S):
    _need_cuda(x, "compress_mixed_ip")
    return _compress_mixed_ip(x, Pi, is_outlier, bounds_out, cents_out, bits_out, bounds_reg, cents_reg, bits_reg, S)


def decompress(codes, norms, Pi, centroids, bits, *, signs=None, S=None, qjl_scale=0.0, packed=False,
               d=None, out_dtype=torch.float32):
    """Dense planes: codes (..., d) or (..., packed bytes), norms (...)."""
    _need_cuda(codes, "decompress")
    return _decompress_dense(codes, signs, norms, Pi, centroids, bits, S, qjl_scale, packed,
                             codes.shape[-1] if d is None else d, out_dtype)


def decompress_rows(codes, norms, Pi, centroids, bits, d, n_seg, seg_len, seg_stride, seg_off, *,
                    signs=None, S=None, qjl_scale=0.0, out_dtype=torch.float32):
    """Packed cache planes [n_seg, capacity, bytes]: rows seg_off..seg_off+seg_len of each segment."""
    _need_cuda(codes, "decompress_rows")
    return _decompress(codes, signs, norms, Pi, centroids, bits, S, qjl_scale, True, d,
                       seg_len, seg_stride, seg_off, n_seg * seg_len, out_dtype)


def decompress_mixed(codes, norms, Pi, is_outlier, cents_out, bits_out, cents_reg, bits_reg, packed=False,
                     d=None):
    _need_cuda(codes, "decompress_mixed")
    return _decompress_mixed(codes, norms, Pi, is_outlier, cents_out, bits_out, cents_reg, bits_reg, packed,
                             codes.shape[-1] if d is None else d)


scatter_rows = _scatter_rows
tile_rows = _tile_rows
untile_rows = _untile_rows
index_scores = _index_scores
topk_merge = _topk_merge
INDEX_MAX_K = _lib.INDEX_MAX_K
