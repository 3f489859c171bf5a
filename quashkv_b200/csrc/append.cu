// Append of new keys and values into a cache (reference engine.py:145-172).
//
// Small appends (a decode step, a short prompt) and every dimension but 128 are ONE launch of the fp32-chain kernel
// (rotate_chain.cu): keys and values as its two jobs, the codes written to their rows or records directly, the slots
// of a paged cache computed from the block table in the kernel.  A decode step of 32 sequences x 8 heads used to be
// two compress launches of 52-55 us each (kernels made for a million vectors, whose set-up alone is that long), eleven
// element-wise launches for the slots and a filing launch.
// Large appends at d = 128 compress on tcgen05; contiguous planes are written in place, records and pages go through
// packed rows in the workspace and one filing pass (bytes are 2 x 104 per token against 512 read: it does not bind).
#include "rotate_common.cuh"

namespace qkv {
namespace {

__device__ unsigned long long g_slots_dropped = 0;        // rows without a slot, large paged appends

__global__ void __launch_bounds__(256) slots_kernel(const int32_t* __restrict__ block_table,
                                                    const int32_t* __restrict__ start_lens, int max_blocks, int block_size,
                                                    int heads, int tokens, int64_t n, int64_t* __restrict__ slots) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t slot = paged_row(block_table, start_lens, max_blocks, block_size, heads, tokens, i);
  slots[i] = slot;
  if (slot < 0) atomicAdd(&g_slots_dropped, 1ull);
}

size_t up(size_t b) { return (b + 255) / 256 * 256; }

struct Staging { size_t k_codes, k_signs, k_norms, v_codes, v_norms, slots, total; };
Staging staging(int64_t n, int d, int mse_bits, int val_bits, bool paged) {
  Staging s;
  const size_t rows = static_cast<size_t>(n);
  s.k_codes = 0;
  s.k_signs = up(rows * packed_row_bytes(d, mse_bits));
  s.k_norms = s.k_signs + up(rows * packed_row_bytes(d, 1));
  s.v_codes = s.k_norms + up(rows * 4);
  s.v_norms = s.v_codes + up(rows * packed_row_bytes(d, val_bits));
  s.slots = s.v_norms + up(rows * 4);
  s.total = s.slots + (paged ? up(rows * 8) : 0);
  return s;
}

// Whether the pair of jobs goes through the tcgen05 kernels; decided from sizes alone, so that the workspace query and
// the call agree (an input that those kernels cannot take falls back to the chain kernel inside qkv_compress_*).
bool large(int64_t n, int d) { return d == kMaxD && n >= kAppendTensorCore; }

}  // namespace
}  // namespace qkv

using namespace qkv;

extern "C" int64_t qkv_dropped_append_rows(void) {
  unsigned long long v = 0;
  cudaMemcpyFromSymbol(&v, g_slots_dropped, sizeof(v));
  return static_cast<int64_t>(v + chain_rows_dropped());
}

extern "C" size_t qkv_append_workspace_bytes(int B, int H, int64_t tokens, int d, int mse_bits, int val_bits, int tiled,
                                             int paged) {
  if (B < 1 || H < 1 || tokens < 1 || d < 1) return 0;
  const int64_t n = static_cast<int64_t>(B) * H * tokens;
  if (!large(n, d) || (!tiled && !paged)) return 0;
  return staging(n, d, mse_bits, val_bits, paged != 0).total;
}

extern "C" int qkv_append_kv(const void* keys, int k_dtype, const void* values, int v_dtype, int B, int H, int64_t tokens,
                             int d, const float* Pi, const float* k_boundaries, const float* k_centroids, const float* S,
                             int mse_bits, const float* v_boundaries, int val_bits, qkv_kv_dest_t dest,
                             void* workspace, size_t workspace_bytes, void* stream) {
  if (B < 0 || H < 0 || tokens < 0 || d < 1 || d > kMaxD) return QKV_EDIM;
  const int64_t n = static_cast<int64_t>(B) * H * tokens;
  if (n >= (int64_t(1) << 31)) return QKV_EDIM;
  if (n == 0) return QKV_OK;
  if (!keys || !values || !Pi || !k_boundaries || !k_centroids || !S || !v_boundaries) return QKV_ENULL;
  for (int t : {k_dtype, v_dtype})
    if (t != QKV_F32 && t != QKV_BF16 && t != QKV_F16) return QKV_EDTYPE;
  if (mse_bits < 1 || mse_bits > 4 || val_bits < 1 || val_bits > 4) return QKV_EBITS;
  const bool tiled = dest.records != nullptr, paged = dest.block_table != nullptr;
  if (!tiled && (!dest.k_codes || !dest.k_signs || !dest.k_norms || !dest.v_codes || !dest.v_norms)) return QKV_ENULL;
  if (tiled && (d != kMaxD || mse_bits != 2 || val_bits != 3)) return QKV_EBITS;
  if (tiled && (reinterpret_cast<uintptr_t>(dest.records) & 15u)) return QKV_EALIGN;
  if (paged ? (!dest.start_lens || dest.max_blocks < 1 || dest.block_size < 1 || (tiled && (dest.block_size & 15)))
            : (dest.offset < 0 || dest.offset + tokens > dest.capacity || (tiled && (dest.capacity & 15))))
    return QKV_EARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const qkv_rows_t rows{tokens, dest.capacity, dest.offset};

  if (large(n, d)) {
    const Staging s = staging(n, d, mse_bits, val_bits, paged);
    uint8_t *kc = dest.k_codes, *ks = dest.k_signs, *vc = dest.v_codes;
    float *kn = dest.k_norms, *vn = dest.v_norms;
    qkv_rows_t where = rows;
    int64_t* slots = nullptr;
    if (tiled || paged) {
      if (!workspace || workspace_bytes < s.total) return QKV_EWORKSPACE;
      uint8_t* ws = static_cast<uint8_t*>(workspace);
      kc = ws + s.k_codes; ks = ws + s.k_signs; vc = ws + s.v_codes;
      kn = reinterpret_cast<float*>(ws + s.k_norms); vn = reinterpret_cast<float*>(ws + s.v_norms);
      where = qkv_rows_t{n, 0, 0};
      if (paged) {
        slots = reinterpret_cast<int64_t*>(ws + s.slots);
        slots_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
            dest.block_table, dest.start_lens, dest.max_blocks, dest.block_size, H, static_cast<int>(tokens), n, slots);
        if (check_launch()) return QKV_ELAUNCH;
      }
    }
    int rc = qkv_compress_ip(keys, k_dtype, d, n, d, Pi, k_boundaries, k_centroids, mse_bits, S, kc, ks, 1, kn, where, stream);
    if (!rc) rc = qkv_compress_mse(values, v_dtype, d, n, d, Pi, v_boundaries, val_bits, vc, 1, vn, where, stream);
    if (rc || !(tiled || paged)) return rc;
    if (tiled) return qkv_tile_rows(kc, ks, kn, vc, vn, n, dest.records, rows, slots, stream);
    const struct { const void* src; void* dst; int bytes; } planes[5] = {
        {kc, dest.k_codes, packed_row_bytes(d, mse_bits)}, {ks, dest.k_signs, packed_row_bytes(d, 1)},
        {kn, dest.k_norms, 4}, {vc, dest.v_codes, packed_row_bytes(d, val_bits)}, {vn, dest.v_norms, 4}};
    for (const auto& p : planes)
      if ((rc = qkv_scatter_rows(p.src, p.dst, slots, n, p.bytes, stream))) return rc;
    return QKV_OK;
  }

  ChainArgs c{};
  CompressArgs& k = c.job[0];
  k.x = keys; k.x_dtype = k_dtype; k.x_pitch = d; k.n_vec = n; k.d = d; k.Pi = Pi; k.mode = MODE_IP;
  k.bounds0 = k_boundaries; k.bits0 = mse_bits; k.bits1 = 1; k.centroids = k_centroids; k.S = S;
  k.codes = dest.k_codes; k.signs = dest.k_signs; k.norms = dest.k_norms; k.packed = 1; k.rows = rows;
  CompressArgs& v = c.job[1];
  v = k;
  v.x = values; v.x_dtype = v_dtype; v.mode = MODE_MSE; v.bounds0 = v_boundaries; v.bits0 = val_bits;
  v.centroids = nullptr; v.S = nullptr; v.codes = dest.v_codes; v.signs = nullptr; v.norms = dest.v_norms;
  c.d = d; c.Pi = Pi; c.records = dest.records;
  c.block_table = dest.block_table; c.start_lens = dest.start_lens; c.max_blocks = dest.max_blocks;
  c.block_size = dest.block_size; c.heads = H; c.tokens = static_cast<int>(tokens);
  return launch_compress_chain(c, st);
}
