// Entry points of compress (normalise -> rotate -> bucketise -> sign bit -> pack), decompress (unpack -> centroid
// gather -> un-rotate -> rescale) and the cache append, and the choice of the kernel.
#include <stdlib.h>

#include "rotate_common.cuh"

namespace qkv {

static int check_common(const void* x, int dtype, int64_t n_vec, int d, const float* Pi) {
  if ((!x && n_vec != 0) || !Pi) return QKV_ENULL;
  if (dtype != QKV_F32 && dtype != QKV_BF16 && dtype != QKV_F16) return QKV_EDTYPE;
  if (d < 1 || d > kMaxD || n_vec < 0) return QKV_EDIM;
  return QKV_OK;
}

static int check_rows(const qkv_rows_t& r) {
  return (r.seg_len >= 1 && r.seg_stride >= 0 && r.seg_off >= 0) ? QKV_OK : QKV_EARG;
}

// QUASHKV_B200_CUDA_CORE_ROTATION=1 keeps every call on the fp32 CUDA-core kernels (for A/B checks).
static bool cuda_core_only() {
  const char* e = getenv("QUASHKV_B200_CUDA_CORE_ROTATION");
  return e && e[0] == '1';
}

bool compress_prefers_chain(const CompressArgs& a) {
  return !compress_umma_ok(a) || cuda_core_only();
}

static int run_compress(const CompressArgs& a, cudaStream_t st) {
  if (a.n_vec == 0) return QKV_OK;
  ChainArgs c{};
  c.job[0] = a;
  c.d = a.d;
  c.Pi = a.Pi;
  if (compress_prefers_chain(a)) return launch_compress_chain(c, st);
  const int rc = launch_compress_umma(a, st);
  if (rc || a.mode != MODE_MIXED) return rc;
  // Mixed precision: the tcgen05 kernel works only when the outlier count (known on the device) is a
  // multiple of 32 and returns at once otherwise; the CUDA-core kernel behind it makes the opposite choice.
  c.job[0].skip_block_aligned = 1;
  return launch_compress_chain(c, st);
}

static int run_decompress(DecompressArgs& a, cudaStream_t st) {
  if (decompress_umma_ok(a) && !cuda_core_only()) {
    const int rc = launch_decompress_umma(a, st);
    if (rc || a.mode != MODE_MIXED) return rc;
    a.skip_block_aligned = 1;        // as above: outlier counts that are no multiple of 32
  }
  return launch_decompress_chain(a, st);
}

}  // namespace qkv

using namespace qkv;

extern "C" int qkv_compress_mse(const void* x, int x_dtype, int64_t x_pitch, int64_t n_vec, int d,
                                const float* Pi, const float* boundaries, int bits,
                                uint8_t* codes_out, int packed, float* norms_out,
                                qkv_rows_t rows, void* stream) {
  int rc = check_common(x, x_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!boundaries || ((!codes_out || !norms_out) && n_vec != 0)) return QKV_ENULL;
  if (bits < 1 || bits > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  CompressArgs a{};
  a.x = x; a.x_dtype = x_dtype; a.x_pitch = x_pitch; a.n_vec = n_vec; a.d = d; a.Pi = Pi;
  a.mode = MODE_MSE; a.bounds0 = boundaries; a.bits0 = bits; a.bits1 = 1;
  a.codes = codes_out; a.packed = packed; a.norms = norms_out; a.rows = rows;
  return run_compress(a, static_cast<cudaStream_t>(stream));
}

extern "C" int qkv_compress_ip(const void* x, int x_dtype, int64_t x_pitch, int64_t n_vec, int d,
                               const float* Pi, const float* boundaries, const float* centroids,
                               int mse_bits, const float* S,
                               uint8_t* codes_out, uint8_t* signs_out, int packed, float* norms_out,
                               qkv_rows_t rows, void* stream) {
  int rc = check_common(x, x_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!boundaries || !centroids || !S || ((!codes_out || !signs_out || !norms_out) && n_vec != 0)) return QKV_ENULL;
  if (mse_bits < 1 || mse_bits > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  CompressArgs a{};
  a.x = x; a.x_dtype = x_dtype; a.x_pitch = x_pitch; a.n_vec = n_vec; a.d = d; a.Pi = Pi;
  a.mode = MODE_IP; a.bounds0 = boundaries; a.bits0 = mse_bits; a.bits1 = 1;
  a.centroids = centroids; a.S = S;
  a.codes = codes_out; a.signs = signs_out; a.packed = packed; a.norms = norms_out; a.rows = rows;
  return run_compress(a, static_cast<cudaStream_t>(stream));
}

extern "C" int qkv_compress_mixed(const void* x, int x_dtype, int64_t x_pitch, int64_t n_vec, int d,
                                  const float* Pi, const uint8_t* is_outlier,
                                  const float* bounds_out, int bits_out,
                                  const float* bounds_reg, int bits_reg,
                                  uint8_t* codes_out, int packed, float* norms_out,
                                  qkv_rows_t rows, void* stream) {
  int rc = check_common(x, x_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!is_outlier || !bounds_out || !bounds_reg || ((!codes_out || !norms_out) && n_vec != 0)) return QKV_ENULL;
  if (bits_out < 1 || bits_out > 4 || bits_reg < 1 || bits_reg > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  CompressArgs a{};
  a.x = x; a.x_dtype = x_dtype; a.x_pitch = x_pitch; a.n_vec = n_vec; a.d = d; a.Pi = Pi;
  a.mode = MODE_MIXED; a.bounds0 = bounds_out; a.bits0 = bits_out; a.bounds1 = bounds_reg; a.bits1 = bits_reg;
  a.is_outlier = is_outlier;
  a.codes = codes_out; a.packed = packed; a.norms = norms_out; a.rows = rows;
  return run_compress(a, static_cast<cudaStream_t>(stream));
}

extern "C" int qkv_compress_mixed_ip(const void* x, int x_dtype, int64_t x_pitch, int64_t n_vec, int d,
                                     const float* Pi, const uint8_t* is_outlier,
                                     const float* bounds_out, const float* cents_out, int bits_out,
                                     const float* bounds_reg, const float* cents_reg, int bits_reg,
                                     const float* S,
                                     uint8_t* codes_out, uint8_t* signs_out, int packed, float* norms_out,
                                     qkv_rows_t rows, void* stream) {
  int rc = check_common(x, x_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!is_outlier || !bounds_out || !bounds_reg || !cents_out || !cents_reg || !S ||
      ((!codes_out || !signs_out || !norms_out) && n_vec != 0))
    return QKV_ENULL;
  if (bits_out < 1 || bits_out > 4 || bits_reg < 1 || bits_reg > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  CompressArgs a{};
  a.x = x; a.x_dtype = x_dtype; a.x_pitch = x_pitch; a.n_vec = n_vec; a.d = d; a.Pi = Pi;
  a.mode = MODE_MIXED; a.bounds0 = bounds_out; a.bits0 = bits_out; a.bounds1 = bounds_reg; a.bits1 = bits_reg;
  a.centroids = cents_out; a.centroids1 = cents_reg; a.S = S;
  a.is_outlier = is_outlier;
  a.codes = codes_out; a.signs = signs_out; a.packed = packed; a.norms = norms_out; a.rows = rows;
  return run_compress(a, static_cast<cudaStream_t>(stream));
}

extern "C" int64_t qkv_mixed_row_bytes(int d, int n_out, int bits_out, int bits_reg) {
  if (d < 1 || n_out < 0 || n_out > d) return QKV_EDIM;
  return packed_row_bytes(n_out, bits_out) + packed_row_bytes(d - n_out, bits_reg);
}

extern "C" int qkv_decompress(const uint8_t* codes, const uint8_t* signs, int packed, const float* norms,
                              qkv_rows_t rows, int64_t n_vec, int d,
                              const float* Pi, const float* centroids, int bits,
                              const float* S, float qjl_scale,
                              void* out, int out_dtype, int64_t out_pitch, void* stream) {
  int rc = check_common(codes, out_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!centroids || ((!norms || !out) && n_vec != 0) || (signs && !S)) return QKV_ENULL;
  if (bits < 1 || bits > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  if (n_vec == 0) return QKV_OK;
  DecompressArgs a{};
  a.codes = codes; a.signs = signs; a.packed = packed; a.norms = norms; a.rows = rows;
  a.n_vec = n_vec; a.d = d; a.Pi = Pi; a.mode = MODE_MSE; a.cents0 = centroids; a.bits0 = bits; a.bits1 = 1;
  a.S = S; a.qjl_scale = qjl_scale; a.out = out; a.out_dtype = out_dtype; a.out_pitch = out_pitch;
  return run_decompress(a, static_cast<cudaStream_t>(stream));
}

extern "C" int qkv_decompress_mixed(const uint8_t* codes, int packed, const float* norms,
                                    qkv_rows_t rows, int64_t n_vec, int d,
                                    const float* Pi, const uint8_t* is_outlier,
                                    const float* cents_out, int bits_out,
                                    const float* cents_reg, int bits_reg,
                                    void* out, int out_dtype, int64_t out_pitch, void* stream) {
  int rc = check_common(codes, out_dtype, n_vec, d, Pi);
  if (rc) return rc;
  if (!is_outlier || !cents_out || !cents_reg || ((!norms || !out) && n_vec != 0)) return QKV_ENULL;
  if (bits_out < 1 || bits_out > 4 || bits_reg < 1 || bits_reg > 4) return QKV_EBITS;
  if ((rc = check_rows(rows))) return rc;
  if (n_vec == 0) return QKV_OK;
  DecompressArgs a{};
  a.codes = codes; a.packed = packed; a.norms = norms; a.rows = rows;
  a.n_vec = n_vec; a.d = d; a.Pi = Pi; a.mode = MODE_MIXED;
  a.cents0 = cents_out; a.bits0 = bits_out; a.cents1 = cents_reg; a.bits1 = bits_reg;
  a.is_outlier = is_outlier; a.out = out; a.out_dtype = out_dtype; a.out_pitch = out_pitch;
  return run_decompress(a, static_cast<cudaStream_t>(stream));
}

namespace qkv { unsigned int index_umma_timeouts(); unsigned int bulk_copy_timeouts(); unsigned int prefill_timeouts(); }

extern "C" int64_t qkv_tensor_core_timeouts(void) {
  return static_cast<int64_t>(umma_timeouts()) + static_cast<int64_t>(index_umma_timeouts()) +
         static_cast<int64_t>(bulk_copy_timeouts()) + static_cast<int64_t>(prefill_timeouts());
}
