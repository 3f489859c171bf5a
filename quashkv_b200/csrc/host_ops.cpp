// Host side of the hot ops: the CUDA implementations of torch.ops.quashkv_b200.* .
//
// Each op checks its tensors, allocates its outputs and workspace with torch's caching allocator and calls ONE
// entry point of the C ABI (include/quashkv_b200.h) on the current stream.  A call over a few hundred vectors or a
// short cache is 5-20 us of device work; the same checks, allocations and pointer marshalling in Python (custom op
// plus ctypes) took 20-90 us of host time per call, so they are native: 3-6 us.  The schemas and the fake
// implementations stay in ops.py.
//
// The library is found through quashkv_host_bind(path), so that the Python side decides which file is loaded.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/library.h>

#include <tuple>

#include "../../include/quashkv_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

#define QKV_FOR_EACH_ENTRY(X)                                                                                     \
  X(qkv_strerror) X(qkv_compress_mse) X(qkv_compress_ip) X(qkv_compress_mixed) X(qkv_mixed_row_bytes)             \
  X(qkv_decompress) X(qkv_decompress_mixed) X(qkv_attention_workspace_bytes) X(qkv_attention)                     \
  X(qkv_attention_paged) X(qkv_attention_tiled) X(qkv_append_workspace_bytes) X(qkv_append_kv) X(qkv_index_workspace_bytes) X(qkv_index_scan_topk)

struct Api {
#define QKV_MEMBER(name) decltype(&::name) name = nullptr;
  QKV_FOR_EACH_ENTRY(QKV_MEMBER)
#undef QKV_MEMBER
} api;
bool bound = false;           // every entry point resolved

void check(int rc, const char* what) {
  TORCH_CHECK(rc == 0, "quashkv_b200: ", what, " failed: ", api.qkv_strerror(rc), " (code ", rc, ")");
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return QKV_F32;
    case at::kBFloat16: return QKV_BF16;
    case at::kHalf: return QKV_F16;
    default: return -1;
  }
}

int out_code(at::ScalarType t) {
  TORCH_CHECK(t == at::kFloat || t == at::kBFloat16 || t == at::kHalf, "quashkv_b200: unsupported output dtype ", t);
  return t == at::kFloat ? QKV_F32 : (t == at::kBFloat16 ? QKV_BF16 : QKV_F16);
}

// A data tensor the kernels can read: contiguous, one of the three float types.
Tensor data(const Tensor& t) {
  Tensor x = dtype_code(t) < 0 ? t.to(at::kFloat) : t;
  return x.is_contiguous() ? x : x.contiguous();
}

// Small constants (Pi, tables, S) follow the data: fp32, contiguous, on its device.
Tensor f32(const Tensor& t, const at::Device& dev) {
  if (t.scalar_type() == at::kFloat && t.device() == dev && t.is_contiguous()) return t;
  return t.detach().to(dev, at::kFloat).contiguous();
}
Tensor u8(const Tensor& t, const at::Device& dev) {
  if (t.scalar_type() == at::kByte && t.device() == dev && t.is_contiguous()) return t;
  return t.detach().to(dev, at::kByte).contiguous();
}
const float* fp(const Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }
const uint8_t* bp(const Tensor& t) { return static_cast<const uint8_t*>(t.const_data_ptr()); }
float* fpm(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
uint8_t* bpm(const Tensor& t) { return static_cast<uint8_t*>(t.data_ptr()); }

// Codes, norms, records and tables of indices are not moved for the caller, and a host pointer must never reach a
// kernel: they have to be on the device the call runs on.
void same_device(const at::Device& dev, std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    TORCH_CHECK_VALUE(t == nullptr || t->device() == dev, "quashkv_b200: tensors of one call on different devices (",
                      t->device(), " and ", dev, ")");
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device& dev) {
  return at::detail::empty_cuda(size, type, dev, std::nullopt);
}

struct Call {             // device guard and stream of one op
  c10::cuda::CUDAGuard guard;
  void* stream;
  explicit Call(const at::Device& dev) : guard(dev), stream(c10::cuda::getCurrentCUDAStream(dev.index()).stream()) {
    TORCH_CHECK(bound, "quashkv_b200: the library has not been loaded; rebuild it with `python -m quashkv_b200._build`");
  }
};

int64_t row_bytes(int64_t d, int64_t bits) {
  return bits == 8 ? d : (bits == 3 ? 3 * ((d + 7) / 8) : (d * bits + 7) / 8);
}
qkv_rows_t dense(int64_t n) { return {n > 1 ? n : 1, 0, 0}; }

c10::SmallVector<int64_t, 6> lead_shape(const Tensor& x, int64_t width) {
  c10::SmallVector<int64_t, 6> s(x.sizes().begin(), x.sizes().end() - 1);
  if (width >= 0) s.push_back(width);
  return s;
}

// ---- compress ------------------------------------------------------------------------------------------------------

std::tuple<Tensor, Tensor> compress_mse(const Tensor& x_in, const Tensor& Pi_in, const Tensor& bounds_in, int64_t bits,
                                        bool packed) {
  const Tensor x = data(x_in);
  const at::Device dev = x.device();
  Call call(dev);
  const int64_t d = x.size(-1), n = d > 0 ? x.numel() / d : 0;
  const Tensor Pi = f32(Pi_in, dev), bounds = f32(bounds_in, dev);
  Tensor codes = empty(lead_shape(x, packed ? row_bytes(d, bits) : d), at::kByte, dev);
  Tensor norms = empty(lead_shape(x, -1), at::kFloat, dev);
  check(api.qkv_compress_mse(x.const_data_ptr(), dtype_code(x), d, n, d, fp(Pi), fp(bounds), bits, bpm(codes), packed,
                             fpm(norms), dense(n), call.stream), "compress_mse");
  return {codes, norms};
}

std::tuple<Tensor, Tensor, Tensor> compress_ip(const Tensor& x_in, const Tensor& Pi_in, const Tensor& bounds_in,
                                               const Tensor& cents_in, const Tensor& S_in, int64_t mse_bits, bool packed) {
  const Tensor x = data(x_in);
  const at::Device dev = x.device();
  Call call(dev);
  const int64_t d = x.size(-1), n = d > 0 ? x.numel() / d : 0;
  const Tensor Pi = f32(Pi_in, dev), bounds = f32(bounds_in, dev), cents = f32(cents_in, dev), S = f32(S_in, dev);
  Tensor codes = empty(lead_shape(x, packed ? row_bytes(d, mse_bits) : d), at::kByte, dev);
  Tensor signs = empty(lead_shape(x, packed ? row_bytes(d, 1) : d), at::kByte, dev);
  Tensor norms = empty(lead_shape(x, -1), at::kFloat, dev);
  check(api.qkv_compress_ip(x.const_data_ptr(), dtype_code(x), d, n, d, fp(Pi), fp(bounds), fp(cents), mse_bits, fp(S),
                            bpm(codes), bpm(signs), packed, fpm(norms), dense(n), call.stream), "compress_ip");
  return {codes, signs, norms};
}

// Compress (N, d) vectors into packed planes [capacity, bytes] at rows offset .. offset + N.
void compress_ip_into(const Tensor& x_in, const Tensor& Pi_in, const Tensor& bounds_in, const Tensor& cents_in,
                      const Tensor& S_in, int64_t mse_bits, Tensor codes, Tensor signs, Tensor norms, int64_t offset) {
  const Tensor x = data(x_in);
  const at::Device dev = x.device();
  Call call(dev);
  const int64_t d = x.size(-1), n = d > 0 ? x.numel() / d : 0;
  same_device(dev, {&codes, &signs, &norms});
  const Tensor Pi = f32(Pi_in, dev), bounds = f32(bounds_in, dev), cents = f32(cents_in, dev), S = f32(S_in, dev);
  check(api.qkv_compress_ip(x.const_data_ptr(), dtype_code(x), d, n, d, fp(Pi), fp(bounds), fp(cents), mse_bits, fp(S),
                            bpm(codes), bpm(signs), 1, fpm(norms), {n > 1 ? n : 1, 0, offset}, call.stream),
        "compress_ip_into");
}

std::tuple<Tensor, Tensor> compress_mixed(const Tensor& x_in, const Tensor& Pi_in, const Tensor& mask_in,
                                          const Tensor& bo_in, int64_t bits_out, const Tensor& br_in, int64_t bits_reg,
                                          bool packed, int64_t n_out) {
  const Tensor x = data(x_in);
  const at::Device dev = x.device();
  Call call(dev);
  const int64_t d = x.size(-1), n = d > 0 ? x.numel() / d : 0;
  const Tensor Pi = f32(Pi_in, dev), mask = u8(mask_in, dev), bo = f32(bo_in, dev), br = f32(br_in, dev);
  Tensor codes = empty(lead_shape(x, packed ? api.qkv_mixed_row_bytes(d, n_out, bits_out, bits_reg) : d), at::kByte, dev);
  Tensor norms = empty(lead_shape(x, -1), at::kFloat, dev);
  check(api.qkv_compress_mixed(x.const_data_ptr(), dtype_code(x), d, n, d, fp(Pi), bp(mask), fp(bo), bits_out, fp(br),
                               bits_reg, bpm(codes), packed, fpm(norms), dense(n), call.stream), "compress_mixed");
  return {codes, norms};
}

// ---- appends into a cache -----------------------------------------------------------------------------------------

struct AppendConsts { Tensor Pi, kb, kc, S, vb; };

// B * H segments of T new keys and values each into the destination: one C call.
void run_append(const Tensor& keys, const Tensor& values, int64_t B, int64_t H, int64_t T, const AppendConsts& c,
                int64_t mse_bits, int64_t val_bits, const qkv_kv_dest_t& dest, void* stream) {
  const at::Device dev = keys.device();
  const int64_t d = keys.size(-1);
  const int64_t need = api.qkv_append_workspace_bytes(B, H, T, d, mse_bits, val_bits, dest.records != nullptr,
                                                      dest.block_table != nullptr);
  const Tensor ws = need > 0 ? empty({need}, at::kByte, dev) : Tensor();
  const Tensor Pi = f32(c.Pi, dev), kb = f32(c.kb, dev), kc = f32(c.kc, dev), S = f32(c.S, dev), vb = f32(c.vb, dev);
  check(api.qkv_append_kv(keys.const_data_ptr(), dtype_code(keys), values.const_data_ptr(), dtype_code(values), B, H, T, d,
                          fp(Pi), fp(kb), fp(kc), fp(S), mse_bits, fp(vb), val_bits, dest,
                          need > 0 ? ws.data_ptr() : nullptr, need, stream), "append");
}

// Row-major planes [segments, capacity, ...], rows offset .. offset + T of every segment: keys and values (..., T, d),
// their leading dimensions flattened.  One C call where their shapes agree, else one for each.
void append_kv(const Tensor& keys_in, const Tensor& values_in, const Tensor& Pi_in, const Tensor& kb_in, const Tensor& kc_in,
               const Tensor& S_in, int64_t mse_bits, const Tensor& vb_in, int64_t val_bits, Tensor k_codes, Tensor k_signs,
               Tensor k_norms, Tensor v_codes, Tensor v_norms, int64_t offset) {
  const Tensor keys = data(keys_in), values = data(values_in);
  const at::Device dev = keys.device();
  Call call(dev);
  same_device(dev, {&values, &k_codes, &k_signs, &k_norms, &v_codes, &v_norms});
  const int64_t T = keys.size(-2), d = keys.size(-1);
  TORCH_CHECK_VALUE(values.size(-1) == d, "quashkv_b200: keys and values of different vector lengths");
  if (keys.sizes() == values.sizes()) {
    qkv_kv_dest_t dest{};
    dest.k_codes = bpm(k_codes); dest.k_signs = bpm(k_signs); dest.k_norms = fpm(k_norms);
    dest.v_codes = bpm(v_codes); dest.v_norms = fpm(v_norms);
    dest.capacity = k_norms.size(-1); dest.offset = offset;
    const bool four = keys.dim() == 4;
    const int64_t B = four ? keys.size(0) : 1, H = four ? keys.size(1) : (keys.numel() > 0 ? keys.numel() / (T * d) : 0);
    run_append(keys, values, B, H, T, {Pi_in, kb_in, kc_in, S_in, vb_in}, mse_bits, val_bits, dest, call.stream);
    return;
  }
  const qkv_rows_t rows{T, k_norms.size(-1), offset};
  const Tensor Pi = f32(Pi_in, dev), kb = f32(kb_in, dev), kc = f32(kc_in, dev), S = f32(S_in, dev), vb = f32(vb_in, dev);
  check(api.qkv_compress_ip(keys.const_data_ptr(), dtype_code(keys), d, d > 0 ? keys.numel() / d : 0, d, fp(Pi), fp(kb), fp(kc),
                            mse_bits, fp(S), bpm(k_codes), bpm(k_signs), 1, fpm(k_norms), rows, call.stream), "append keys");
  check(api.qkv_compress_mse(values.const_data_ptr(), dtype_code(values), d, d > 0 ? values.numel() / d : 0, d, fp(Pi), fp(vb),
                             val_bits, bpm(v_codes), 1, fpm(v_norms), rows, call.stream), "append values");
}

void check_bhtd(const Tensor& keys, const Tensor& values) {
  TORCH_CHECK_VALUE(keys.dim() == 4 && keys.sizes() == values.sizes(), "quashkv_b200: keys and values of shape (B, H, T, d)");
}

// Tile records [B*H, capacity / 16, 1664], tokens offset .. offset + S of every segment.
void append_records(const Tensor& keys_in, const Tensor& values_in, const Tensor& Pi, const Tensor& kb, const Tensor& kc,
                    const Tensor& S, int64_t mse_bits, const Tensor& vb, int64_t val_bits, Tensor records,
                    int64_t capacity, int64_t offset) {
  const Tensor keys = data(keys_in), values = data(values_in);
  const at::Device dev = keys.device();
  Call call(dev);
  same_device(dev, {&values, &records});
  qkv_kv_dest_t dest{};
  dest.records = bpm(records);
  dest.capacity = capacity; dest.offset = offset;
  check_bhtd(keys, values);
  run_append(keys, values, keys.size(0), keys.size(1), keys.size(2), {Pi, kb, kc, S, vb}, mse_bits, val_bits, dest, call.stream);
}

// A pool of pages: planes = {records} or the five planes, positions start_lens[b] .. of the pages in block_table.
void append_paged(const Tensor& keys_in, const Tensor& values_in, const Tensor& Pi, const Tensor& kb, const Tensor& kc,
                  const Tensor& S, int64_t mse_bits, const Tensor& vb, int64_t val_bits, at::TensorList planes,
                  const Tensor& table_in, const Tensor& lens_in, int64_t block_size) {
  const Tensor keys = data(keys_in), values = data(values_in);
  const at::Device dev = keys.device();
  Call call(dev);
  for (const Tensor& p : planes) same_device(dev, {&p});
  same_device(dev, {&values, &table_in, &lens_in});
  const auto int32 = [](const Tensor& t) { return t.scalar_type() == at::kInt ? t.contiguous() : t.to(at::kInt).contiguous(); };
  check_bhtd(keys, values);
  TORCH_CHECK_VALUE(table_in.dim() == 2 && table_in.size(0) == keys.size(0) && lens_in.numel() == keys.size(0),
                    "quashkv_b200: a block table and start lengths for ", keys.size(0), " sequences, got ", table_in.sizes(),
                    " and ", lens_in.sizes());
  const Tensor table = int32(table_in), lens = int32(lens_in);
  qkv_kv_dest_t dest{};
  if (planes.size() == 1) {
    dest.records = bpm(planes[0]);
  } else {
    TORCH_CHECK_VALUE(planes.size() == 5, "quashkv_b200: a pool has one plane of records or five row-major planes");
    dest.k_codes = bpm(planes[0]); dest.k_signs = bpm(planes[1]); dest.k_norms = fpm(planes[2]);
    dest.v_codes = bpm(planes[3]); dest.v_norms = fpm(planes[4]);
  }
  dest.block_table = static_cast<const int32_t*>(table.const_data_ptr());
  dest.start_lens = static_cast<const int32_t*>(lens.const_data_ptr());
  dest.max_blocks = static_cast<int>(table.size(1));
  dest.block_size = static_cast<int>(block_size);
  run_append(keys, values, keys.size(0), keys.size(1), keys.size(2), {Pi, kb, kc, S, vb}, mse_bits, val_bits, dest, call.stream);
}

// ---- decompress ---------------------------------------------------------------------------------------------------

Tensor decompress(const Tensor& codes, const OptTensor& signs, const Tensor& norms, const Tensor& Pi_in,
                  const Tensor& cents_in, int64_t bits, const OptTensor& S_in, double qjl_scale, bool packed, int64_t d,
                  int64_t seg_len, int64_t seg_stride, int64_t seg_off, int64_t n_vec, at::ScalarType out_dtype) {
  const at::Device dev = codes.device();
  Call call(dev);
  same_device(dev, {signs ? &*signs : nullptr, &norms});
  const Tensor Pi = f32(Pi_in, dev), cents = f32(cents_in, dev), S = S_in ? f32(*S_in, dev) : Tensor();
  Tensor out = empty({n_vec, d}, out_dtype, dev);
  check(api.qkv_decompress(bp(codes), signs ? bp(*signs) : nullptr, packed, fp(norms), {seg_len, seg_stride, seg_off},
                           n_vec, d, fp(Pi), fp(cents), bits, S_in ? fp(S) : nullptr, static_cast<float>(qjl_scale),
                           out.data_ptr(), out_code(out_dtype), d, call.stream), "decompress");
  return out;
}

// Dense planes: codes (..., d) or (..., packed bytes), signs of the same leading shape, norms (...).
Tensor decompress_dense(const Tensor& codes_in, const OptTensor& signs_in, const Tensor& norms_in, const Tensor& Pi,
                        const Tensor& cents, int64_t bits, const OptTensor& S, double qjl_scale, bool packed, int64_t d,
                        at::ScalarType out_dtype) {
  const Tensor codes = codes_in.contiguous(), norms = f32(norms_in, norms_in.device());
  const OptTensor signs = signs_in ? OptTensor(signs_in->contiguous()) : OptTensor();
  const int64_t width = codes.size(-1), n = width > 0 ? codes.numel() / width : 0;
  return decompress(codes, signs, norms, Pi, cents, bits, S, qjl_scale, packed, d, n > 1 ? n : 1, 0, 0, n, out_dtype)
      .view(lead_shape(codes, d));
}

Tensor decompress_mixed(const Tensor& codes_in, const Tensor& norms_in, const Tensor& Pi_in, const Tensor& mask_in,
                        const Tensor& co_in, int64_t bits_out, const Tensor& cr_in, int64_t bits_reg, bool packed,
                        int64_t d) {
  const Tensor codes = codes_in.contiguous();
  const at::Device dev = codes.device();
  Call call(dev);
  same_device(dev, {&norms_in});
  const int64_t width = codes.size(-1), n = width > 0 ? codes.numel() / width : 0;
  const Tensor norms = f32(norms_in, dev), Pi = f32(Pi_in, dev), mask = u8(mask_in, dev), co = f32(co_in, dev),
               cr = f32(cr_in, dev);
  Tensor out = empty(lead_shape(codes, d), at::kFloat, dev);
  check(api.qkv_decompress_mixed(bp(codes), packed, fp(norms), dense(n), n, d, fp(Pi), bp(mask), fp(co), bits_out, fp(cr),
                                 bits_reg, out.data_ptr(), QKV_F32, d, call.stream), "decompress_mixed");
  return out;
}

// ---- attention ----------------------------------------------------------------------------------------------------

struct Query { Tensor q, ws; int64_t B, Hq, Q, d; };

Query prepare_query(const Tensor& q_in, int64_t hkv, int64_t kv_len) {
  Query r;
  r.q = data(q_in);
  r.B = r.q.size(0); r.Hq = r.q.size(1); r.Q = r.q.size(2); r.d = r.q.size(3);
  const at::Device dev = r.q.device();
  const int64_t need = api.qkv_attention_workspace_bytes(r.B, r.Hq, hkv, r.Q, kv_len, r.d);
  r.ws = empty({need > 16 ? need : 16}, at::kByte, dev);
  return r;
}

Tensor attention(const Tensor& q_in, const Tensor& k_codes, const Tensor& k_signs, const Tensor& k_norms,
                 const Tensor& v_codes, const Tensor& v_norms, int64_t kv_len, int64_t n_kv_heads, int64_t key_bits,
                 int64_t val_bits, const Tensor& Pi_in, const Tensor& kc_in, const Tensor& vc_in, const Tensor& S_in,
                 double qjl_scale, double scale, bool causal) {
  const at::Device dev = q_in.device();
  Call call(dev);
  same_device(dev, {&k_codes, &k_signs, &k_norms, &v_codes, &v_norms});
  const Tensor Pi = f32(Pi_in, dev), kc = f32(kc_in, dev), vc = f32(vc_in, dev), S = f32(S_in, dev);
  const Query r = prepare_query(q_in, n_kv_heads, kv_len);
  Tensor out = empty(q_in.sizes(), at::kFloat, dev);
  const qkv_cache_t cache{bp(k_codes), bp(k_signs), fp(k_norms), bp(v_codes), fp(v_norms), k_norms.size(-1)};
  check(api.qkv_attention(r.q.const_data_ptr(), dtype_code(r.q), cache, r.B, r.Hq, n_kv_heads, r.Q, kv_len, r.d, key_bits,
                          val_bits, fp(Pi), fp(kc), fp(vc), fp(S), static_cast<float>(qjl_scale),
                          static_cast<float>(scale), causal, fpm(out), r.ws.data_ptr(), r.ws.numel(), call.stream),
        "attention");
  return out;
}

// Pool planes [blocks, Hkv, block_size, bytes]; block_table (B, max_blocks) int32; seq_lens (B) int32; max_kv_len an
// upper bound of seq_lens known on the host.
Tensor attention_paged(const Tensor& q_in, const Tensor& k_codes, const Tensor& k_signs, const Tensor& k_norms,
                       const Tensor& v_codes, const Tensor& v_norms, const Tensor& table_in, const Tensor& lens_in,
                       int64_t max_kv_len, int64_t key_bits, int64_t val_bits, const Tensor& Pi_in, const Tensor& kc_in,
                       const Tensor& vc_in, const Tensor& S_in, double qjl_scale, double scale, bool causal) {
  const at::Device dev = q_in.device();
  Call call(dev);
  same_device(dev, {&k_codes, &k_signs, &k_norms, &v_codes, &v_norms, &table_in, &lens_in});
  const Tensor table = table_in.contiguous(), lens = lens_in.contiguous();
  const Tensor Pi = f32(Pi_in, dev), kc = f32(kc_in, dev), vc = f32(vc_in, dev), S = f32(S_in, dev);
  const int64_t hkv = k_norms.size(1);
  const Query r = prepare_query(q_in, hkv, max_kv_len);
  Tensor out = empty(q_in.sizes(), at::kFloat, dev);
  const qkv_paged_cache_t pool{bp(k_codes), bp(k_signs), fp(k_norms), bp(v_codes), fp(v_norms),
                               static_cast<const int32_t*>(table.const_data_ptr()),
                               static_cast<const int32_t*>(lens.const_data_ptr()), static_cast<int>(table.size(1)),
                               static_cast<int>(k_norms.size(2))};
  check(api.qkv_attention_paged(r.q.const_data_ptr(), dtype_code(r.q), pool, r.B, r.Hq, hkv, r.Q, max_kv_len, r.d, key_bits,
                                val_bits, fp(Pi), fp(kc), fp(vc), fp(S), static_cast<float>(qjl_scale),
                                static_cast<float>(scale), causal, fpm(out), r.ws.data_ptr(), r.ws.numel(), call.stream),
        "attention_paged");
  return out;
}

// Records [B*Hkv, capacity/16, 1664] (contiguous) or [blocks, Hkv, block_size/16, 1664] with a block table and lengths
// (paged; kv_len is then their host-known upper bound).
void attention_tiled_out(const Tensor& q_in, const Tensor& records, int64_t capacity, int64_t kv_len, int64_t n_kv_heads,
                         const OptTensor& table_in, const OptTensor& lens_in, int64_t block_size, const Tensor& Pi_in,
                         const Tensor& kc_in, const Tensor& vc_in, const Tensor& S_in, double qjl_scale, double scale,
                         bool causal, Tensor out) {
  const at::Device dev = q_in.device();
  Call call(dev);
  const bool paged = table_in.has_value();
  same_device(dev, {&records, &out, paged ? &*table_in : nullptr, lens_in ? &*lens_in : nullptr});
  TORCH_CHECK_VALUE(out.scalar_type() == at::kFloat && out.sizes() == q_in.sizes() && out.is_contiguous(),
                    "quashkv_b200: out must be a contiguous fp32 tensor of the queries' shape");
  const Tensor table = paged ? table_in->contiguous() : Tensor(), lens = lens_in ? lens_in->contiguous() : Tensor();
  const Tensor Pi = f32(Pi_in, dev), kc = f32(kc_in, dev), vc = f32(vc_in, dev), S = f32(S_in, dev);
  const Query r = prepare_query(q_in, n_kv_heads, kv_len);
  const qkv_tiled_cache_t cache{bp(records), capacity, paged ? static_cast<const int32_t*>(table.const_data_ptr()) : nullptr,
                                lens_in ? static_cast<const int32_t*>(lens.const_data_ptr()) : nullptr,
                                paged ? static_cast<int>(table.size(1)) : 0, static_cast<int>(block_size)};
  check(api.qkv_attention_tiled(r.q.const_data_ptr(), dtype_code(r.q), cache, r.B, r.Hq, n_kv_heads, r.Q, kv_len, r.d, 3, 3,
                                fp(Pi), fp(kc), fp(vc), fp(S), static_cast<float>(qjl_scale), static_cast<float>(scale),
                                causal, fpm(out), r.ws.data_ptr(), r.ws.numel(), call.stream), "attention_tiled");
}

Tensor attention_tiled(const Tensor& q, const Tensor& records, int64_t capacity, int64_t kv_len, int64_t n_kv_heads,
                       const OptTensor& table, const OptTensor& lens, int64_t block_size, const Tensor& Pi,
                       const Tensor& kc, const Tensor& vc, const Tensor& S, double qjl_scale, double scale, bool causal) {
  Tensor out = empty(q.sizes(), at::kFloat, q.device());
  attention_tiled_out(q, records, capacity, kv_len, n_kv_heads, table, lens, block_size, Pi, kc, vc, S, qjl_scale, scale,
                      causal, out);
  return out;
}

// ---- index --------------------------------------------------------------------------------------------------------

std::tuple<Tensor, Tensor> index_scan_topk(const Tensor& q_in, const Tensor& codes, const Tensor& signs,
                                           const Tensor& norms, int64_t n_vectors, int64_t bits, const Tensor& Pi_in,
                                           const Tensor& cents_in, const Tensor& S_in, double qjl_scale, int64_t k,
                                           int64_t id_base) {
  const at::Device dev = q_in.device();
  Call call(dev);
  same_device(dev, {&codes, &signs, &norms});
  const Tensor q = f32(q_in, dev), Pi = f32(Pi_in, dev), cents = f32(cents_in, dev), S = f32(S_in, dev);
  const int64_t M = q.size(0), d = q.size(1);
  Tensor scores = empty({M, k}, at::kFloat, dev), ids = empty({M, k}, at::kLong, dev);
  const int64_t need = api.qkv_index_workspace_bytes(n_vectors, M, d, k);
  const Tensor ws = empty({need > 16 ? need : 16}, at::kByte, dev);
  check(api.qkv_index_scan_topk(fp(q), M, d, bp(codes), bp(signs), fp(norms), n_vectors, bits, fp(Pi), fp(cents), fp(S),
                                static_cast<float>(qjl_scale), k, id_base, fpm(scores),
                                static_cast<int64_t*>(ids.data_ptr()), ws.data_ptr(), need, call.stream),
        "index_scan_topk");
  return {scores, ids};
}

}  // namespace

// Resolves the entry points in the library at `path` (the one the Python side has loaded).  0, or 1 on failure.
extern "C" int quashkv_host_bind(const char* path) {
  bound = false;
  void* handle = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (handle == nullptr) return 1;
#define QKV_RESOLVE(name)                                                 \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(handle, #name)); \
  if (api.name == nullptr) return 1;
  QKV_FOR_EACH_ENTRY(QKV_RESOLVE)
#undef QKV_RESOLVE
  bound = true;
  return 0;
}

// The torch that this file was compiled against, for the loader (which looks for it in the file before loading it).
extern "C" __attribute__((used, visibility("default"))) const char quashkv_host_mark[] = QKV_HOST_MARK;

#define QKV_FOR_EACH_OP(X)                                                                                          \
  X(compress_mse) X(compress_ip) X(compress_ip_into) X(compress_mixed) X(append_kv) X(append_records) X(append_paged) X(decompress) X(decompress_dense) \
  X(decompress_mixed) X(attention) X(attention_paged) X(attention_tiled) X(attention_tiled_out) X(index_scan_topk)

TORCH_LIBRARY_IMPL(quashkv_b200, CUDA, m) {
#define QKV_IMPL(name) m.impl(#name, &name);
  QKV_FOR_EACH_OP(QKV_IMPL)
#undef QKV_IMPL
}

namespace {

// Nothing here has a derivative: where gradients are wanted, the floating-point results carry a node that says so in the
// backward pass instead of ending the graph without a word.  What the op calls itself records nothing.
void without_derivative(const c10::OperatorHandle& op, c10::DispatchKeySet keys, torch::jit::Stack* stack) {
  std::vector<Tensor> inputs;
  if (c10::GradMode::is_enabled())
    for (const c10::IValue& v : torch::jit::last(*stack, op.schema().arguments().size()))
      if (v.isTensor() && v.toTensor().defined() && v.toTensor().requires_grad()) inputs.push_back(v.toTensor());
  {
    at::AutoDispatchBelowAutograd below;
    op.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
  }
  if (inputs.empty()) return;
  const std::shared_ptr<torch::autograd::Node> node(new torch::autograd::NotImplemented(op.schema().name()),
                                                    torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs));
  for (const c10::IValue& v : torch::jit::last(*stack, op.schema().returns().size()))
    if (v.isTensor() && v.toTensor().is_floating_point()) torch::autograd::set_history(v.toTensor(), node);
}

// Tensors that the op writes count the write, so that a graph that saved one of them notices.
void count_writes(const c10::OperatorHandle& op, c10::DispatchKeySet keys, torch::jit::Stack* stack) {
  const auto bump = [](const Tensor& t) {
    if (t.defined() && !t.is_inference()) t.unsafeGetTensorImpl()->bump_version();
  };
  const auto& args = op.schema().arguments();
  const auto values = torch::jit::last(*stack, args.size());
  for (size_t i = 0; i < args.size(); ++i) {
    if (args[i].alias_info() == nullptr || !args[i].alias_info()->isWrite()) continue;
    if (values[i].isTensor()) bump(values[i].toTensor());
    if (values[i].isTensorList())
      for (const Tensor& t : values[i].toTensorVector()) bump(t);
  }
  op.redispatchBoxed(keys & c10::after_ADInplaceOrView_keyset, stack);
}

}  // namespace

TORCH_LIBRARY_IMPL(quashkv_b200, Autograd, m) {
#define QKV_NO_DERIVATIVE(name) m.impl(#name, torch::CppFunction::makeFromBoxedFunction<&without_derivative>());
  QKV_FOR_EACH_OP(QKV_NO_DERIVATIVE)
#undef QKV_NO_DERIVATIVE
}

TORCH_LIBRARY_IMPL(quashkv_b200, ADInplaceOrView, m) {
  for (const char* name : {"compress_ip_into", "append_kv", "append_records", "append_paged", "attention_tiled_out"})
    m.impl(name, torch::CppFunction::makeFromBoxedFunction<&count_writes>());
}
