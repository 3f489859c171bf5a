// Attention of MANY query rows over the compressed cache (prefill) on the fifth-generation tensor cores: head_dim 64 and
// 128, every key / value width, row-major planes or tile records, contiguous or paged, causal or not.
// Semantics: QuashKVEngine.attention (reference engine.py:204-299).
//
// The kernels of decode take the codes apart again for every four to sixteen query rows; with hundreds of rows over the
// same tokens that decoding and the narrow MMAs are nearly all of the time.  Here a first kernel decodes every token ONCE
// into ready fp16 operand tiles (64 tokens, in the swizzled order in which the tensor core reads shared memory, so that
// a tile arrives with plain bulk copies), and a second one runs over them with 128 or 256 query rows per CTA:
//   rotation   q @ Pi^T of the CTA's rows, as MMAs; |q|, the sign weights and their scale per row on the threads
//   scores     [q | w] x [centroid | +-1], K = 2 D, accumulated in tensor memory
//   softmax    a thread per query row, log2 domain, reference exponent rounded up to a whole number, so that every
//              rescaling is by a power of two and exact
//   values     weights times value norm, scaled by a power of two, as the A operand in tensor memory, centroids transposed
//              as B; the sum of a tile is added to fp32 registers, so no accumulator is rescaled and none truncates over a
//              long sequence
//   un-rotation  (sum / l) @ Pi, as MMAs, straight to the output rows
// Two row tiles share each token tile: the tensor core works on one while the other's softmax runs.
//
// Precision.  Every operand that does not fit fp16 goes in as hi + lo (22 bits, scaled per row or per table by powers of
// two), with the products lo x hi, hi x lo, hi x hi, smallest first.  That holds for both rotations always, and for all
// of scores and values with TERMS = 2 (every width but the 3/3-bit records of d = 128, whose other kernels round
// queries, tables and weights to fp16 once as well: TERMS = 1).  Error against 64-bit results: with TERMS = 2 0.71 of the
// fp32 kernel's on average over 34 shapes, 0.93 at the worst of them; with TERMS = 1 that of the kernels it stands beside.
//
// Measured, append and attention (before: the decode kernels): 8 x 1024 causal tokens, 32 / 4 heads of 64, 8609 -> 443 us;
// 2 x 4096, 32 / 8 heads of 128 at 3/3 bits, 3013 -> 993 us (attention alone 385 and 880).  Bound by the softmax warps' chain (tensor memory reads, 1.8 instructions a cycle);
// the tensor pipe is 20 % busy.
//
// Every wait is bounded; one that runs out is counted and ends the use of the tensor core in its CTA, whose rows are then
// attended in fp32 on the CUDA cores (attend_rows_fp32).
#include <math.h>
#include <stdlib.h>

#include "attention_common.cuh"
#include "mma_decode.cuh"
#include "tile_format.cuh"
#include "umma.cuh"

namespace qkv {

namespace {

constexpr int kTok = 64;                          // tokens per tile
constexpr int kRowsT = 128;                       // query rows per row tile = MMA M
// Norms of a tile: of keys, of values (TERMS = 1: x 2^s, then 2^-s, padding, and a byte of further scale per token).
constexpr int kNormBytes = (2 * kTok + 4) * 4 + kTok;
constexpr int kNormSlots = 4;
// The tensor core truncates: an MMA that adds to an accumulator drops what lies below its last bit, on average half a
// unit towards zero, which is 2^-24 E[1 / m] = 2^-24 / (2 ln 2) of a value with mantissa m.  A sum of s like steps is
// truncated at 1/s, 2/s, ... of itself, so it comes out small by (s + 1) / 2 of that.  With TERMS = 2 the factors that
// follow a sum anyway (score units, inverse scales) carry the expected loss of the steps in front of them; it follows from
// the number of steps alone.  Mean slope against 64-bit results over 34 shapes: -2.5e-7 without it, 1e-8 with it.
constexpr double kDrop = 0.72134752 / 16777216.0;
constexpr double steps_lost(int s) { return 0.5 * (s + 1); }
constexpr float kPiScale = 1024.f;                // entries of Pi are at most 1: hi and lo both far from subnormals

__device__ unsigned int g_prefill_timeouts = 0;

template <int D, int TERMS> struct Pf {
  static constexpr int NT = (D == 128 && TERMS == 2) ? 1 : 2;          // row tiles per CTA } what 227 KB hold
  static constexpr int ST = (D == 128 && TERMS == 2) ? 1 : 2;          // token tiles in flight }
  static constexpr int kQBytes = 2 * TERMS * kRowsT * D * 2;           // [qh | wh (| ql | wl)]
  static constexpr int kKBytes = (TERMS + 1) * kTok * D * 2;           // [ch | sign (| cl)]
  static constexpr int kVBytes = TERMS * kTok * D * 2;                 // transposed: [vh (| vl)]
  static constexpr int kTileBytes = kKBytes + kVBytes;
  static constexpr int kPiBytes = 2 * D * D * 2;                       // hi, lo
  // Tensor memory of a row tile, in columns.  TERMS = 1: two score tiles at 0 and 64 (the weights take the place of the
  // scores they come from), value sums at 128.  TERMS = 2: the tensor core truncates its fp32 sums, so long ones are kept
  // in two (d = 64) to four parts that are added in fp32 registers: scores of code and sign operands apart, at d = 128
  // also of their halves, and two accumulators for the values; one score tile, the weights in the place of its first
  // part.  The rotations put their A operand at 128 and their result at 0 (TERMS = 2: and two more parts).
  static constexpr int kCols = NT == 1 ? 512 : 256;
  static constexpr bool kSplit = TERMS == 2;
  static constexpr int SB = kSplit ? 1 : 2;                            // score tiles in flight
  static constexpr int kO2 = D == 64 ? 192 : 384;
  static constexpr int kR1 = D == 64 ? 64 : 256, kR2 = D == 64 ? 192 : 384;
  // Steps of 16 of the parts of a sum, and what truncation takes of it, in kDrop.
  static constexpr int kS = D / 16, kA = kSplit ? kS / 4 : kS, kB = kSplit ? kS / 2 + kS / 8 : kS;      // rotations: 0, kA, kB, kS
  static constexpr int kScorePart = D == 64 ? D / 16 : D / 32;
  static constexpr int kValuePart = kTok / 32;
  static constexpr double kRotLost =
      (kA * steps_lost(kA) + (kB - kA) * steps_lost(kB - kA) + (kS - kB) * steps_lost(kS - kB)) / kS;
  static constexpr double kScoresUp = kSplit ? 1.0 + kDrop * (kRotLost + steps_lost(kScorePart)) : 1.0;
  static constexpr double kOutputUp = kSplit ? 1.0 + kDrop * (kRotLost + steps_lost(kValuePart)) : 1.0;
  static constexpr int kThreads = NT * kRowsT + 128;
  static constexpr size_t kSmem = static_cast<size_t>(NT) * kQBytes + ST * kTileBytes + kNormSlots * kNormBytes + 256;
  static_assert(kPiBytes <= NT * kQBytes, "the rotation's operand uses the queries' place");
  static_assert(kSmem <= 232448, "shared memory of one CTA");
};

struct PrefillArgs {
  const void* q; int q_dtype;
  qkv_cache_t cache; const uint8_t* records;
  const int32_t* block_table; const int32_t* seq_lens; int max_blocks, block_size;
  int B, Hq, Hkv, G, q_len, causal, wk, wv;
  int64_t kv_len;
  const float* Pi; const float* S; const float* kcent; const float* vcent;
  float qjl_scale, scale;
  float* out;
  unsigned char* img;        // [Pi^T hi, lo | Pi hi, lo] then [B * Hkv][tiles] operand tiles, then their norms
  float* norms;
  float* tab;                // [0] key table scale, [1] value table scale, [2] 0, or NaN for a table that the records do not cover
  int tiles;                 // token tiles per (batch, kv head)
  int test_drop_mma;         // test hook: the first CTA issues nothing for its second token tile, so that the waits on it
                             // run out and its rows come from the fp32 way out
};

// 2^(K - e) for a magnitude 2^e <= x < 2^(e+1): x times it lies in [2^K, 2^(K+1)).  Always a normal number, and so is
// its inverse.
template <int K>
__device__ __forceinline__ float scale_to(float x) {
  int e = 254 + K - static_cast<int>((__float_as_uint(x) >> 23) & 255u);
  e = e < 1 ? 1 : (e > 253 ? 253 : e);
  return __uint_as_float(static_cast<uint32_t>(e) << 23);
}
__device__ __forceinline__ float inverse_pow2(float s) {
  return __uint_as_float((254u << 23) - __float_as_uint(s));
}
// Scale of a table held as hi + lo: its largest entry comes to [16, 32), so that lo is no subnormal.
__device__ __forceinline__ float table_scale(const float* t, int n) {
  float mx = 0.f;
  for (int i = 0; i < n; ++i) mx = fmaxf(mx, fabsf(t[i]));
  return scale_to<4>(mx);
}
__device__ __forceinline__ void split_half(float v, __half& h, __half& l) {
  h = __float2half_rn(v);
  l = __float2half_rn(v - __half2float(h));
}
__device__ __forceinline__ uint32_t half_bits2(__half a, __half b) {
  return static_cast<uint32_t>(__half_as_ushort(a)) | (static_cast<uint32_t>(__half_as_ushort(b)) << 16);
}

// ---- operand tiles ------------------------------------------------------------------------------------------------
// Operands of the two rotations, hi and lo (B rows n, K columns k: Pi[n][k], then Pi[k][n]), and the scales of the two
// tables.  A launch of its own: every CTA of the kernel behind it would otherwise search for the scales first.
template <int D, int TERMS>
__global__ void __launch_bounds__(256) prefill_setup_kernel(PrefillArgs a) {
  using P = Pf<D, TERMS>;
  const int tid = threadIdx.x;
  if (blockIdx.x == 0) {
    const float ks = TERMS == 1 ? best_fp16_scale_cta(a.kcent, 4) : table_scale(a.kcent, 1 << a.wk);
    const float vs = TERMS == 1 ? best_fp16_scale_cta(a.vcent, 8) : table_scale(a.vcent, 1 << a.wv);
    if (tid == 0) {
      a.tab[0] = ks;
      a.tab[1] = vs;
      // the records presume a symmetric value table; another one makes every result NaN, as in the kernels of decode
      float top = 0.f, skew = 0.f;
      for (int i = 0; i < 8 && TERMS == 1; ++i) {
        top = fmaxf(top, fabsf(a.vcent[i]));
        skew = fmaxf(skew, fabsf(a.vcent[i] + a.vcent[7 - i]));
      }
      a.tab[2] = skew > 1e-5f * top ? __int_as_float(0x7fc00000) : 0.f;
    }
    return;
  }
  constexpr int kChunks = D * D / 8;
  for (int c = (blockIdx.x - 1) * 256 + tid; c < 2 * kChunks; c += (gridDim.x - 1) * 256) {
    const int which = c / kChunks, n = (c % kChunks) / (D / 8), k0 = 8 * (c % (D / 8));
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      __half h[2], l[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int k = k0 + 2 * p + e;
        split_half((which ? a.Pi[k * D + n] : a.Pi[n * D + k]) * kPiScale, h[e], l[e]);
      }
      hi[p] = half_bits2(h[0], h[1]);
      lo[p] = half_bits2(l[0], l[1]);
    }
    unsigned char* dst = a.img + which * P::kPiBytes + umma::sw128_offset(n, k0, D);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + D * D * 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// Coordinates 16 g .. of token `tok` as the cache holds them: key codes (a.wk bits each), sign bits, value codes (a.wv
// bits each) and the token's norms.
template <int D>
__device__ __forceinline__ void load_group16(const PrefillArgs& a, int seg, int b, int hkv, int64_t tok, int g,
                                             uint64_t& kbits, uint64_t& vbits, uint32_t& sbits, float& kn, float& vn) {
  int64_t unit = 0;                            // pages: the block, and the token inside it
  int off = 0;
  if (a.block_table) {
    const unsigned u = static_cast<unsigned>(tok), bs = static_cast<unsigned>(a.block_size);
    unit = static_cast<int64_t>(a.block_table[static_cast<int64_t>(b) * a.max_blocks + u / bs]) * a.Hkv + hkv;
    off = static_cast<int>(u % bs);
  }
  if (a.records) {
    const int64_t r = a.block_table ? unit * (a.block_size >> 4) + (off >> 4)
                                    : static_cast<int64_t>(seg) * (a.cache.capacity >> 4) + (tok >> 4);
    const uint8_t* rec = a.records + r * tile::kBytes;
    const int k = static_cast<int>(tok & 15);
    kbits = *reinterpret_cast<const uint32_t*>(rec + tile::key_code_offset(k, g));
    sbits = *reinterpret_cast<const uint32_t*>(rec + tile::key_sign_offset(k, g >> 1)) >> (16 * (g & 1));
    uint32_t w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
      w[i] = *reinterpret_cast<const uint32_t*>(rec + tile::val_word_offset(tile::val_lane(k, g), 3 * tile::val_group(k) + i));
    vbits = tile::gather_codes16(w, tile::val_half_shift(k));
    kn = *reinterpret_cast<const float*>(rec + tile::key_norm_offset(k));
    vn = *reinterpret_cast<const float*>(rec + tile::val_norm_offset(k));
  } else {
    const int64_t row = a.block_table ? unit * a.block_size + off : static_cast<int64_t>(seg) * a.cache.capacity + tok;
    const uint16_t* kp = reinterpret_cast<const uint16_t*>(a.cache.k_codes + row * (D / 8 * a.wk)) + g * a.wk;
    const uint16_t* vp = reinterpret_cast<const uint16_t*>(a.cache.v_codes + row * (D / 8 * a.wv)) + g * a.wv;
    for (int i = 0; i < a.wk; ++i) kbits |= static_cast<uint64_t>(kp[i]) << (16 * i);
    for (int i = 0; i < a.wv; ++i) vbits |= static_cast<uint64_t>(vp[i]) << (16 * i);
    sbits = reinterpret_cast<const uint16_t*>(a.cache.k_signs + row * (D / 8))[g];
    kn = a.cache.k_norms[row];
    vn = a.cache.v_norms[row];
  }
}

// Tile, segment per CTA: 64 tokens, four threads each.  Codes go through shared memory as bytes, and leave as 16-byte
// chunks of eight fp16 in the swizzled operand order.  Bound by the writes (768 to 1280 bytes a token at d = 128), which stay in L2 for the kernel behind it.
template <int D, int TERMS>
__global__ void __launch_bounds__(256) prefill_operands_kernel(PrefillArgs a) {
  using P = Pf<D, TERMS>;
  const int tid = threadIdx.x;
  constexpr int kPitch = D + 4;
  __shared__ __align__(16) uint8_t kc_s[kTok][kPitch], vc_s[kTok][kPitch];      // key: code | sign << 7
  __shared__ uint16_t ktab[2][16], vtab[2][16];
  __shared__ float nrm_s[2][kTok];
  const int seg = blockIdx.y, b = seg / a.Hkv, hkv = seg % a.Hkv;
  int64_t kv_len = a.kv_len;
  if (a.block_table) kv_len = min(static_cast<int64_t>(max(a.seq_lens[b], 0)), a.kv_len);
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kTok;
  if (t0 >= kv_len) return;
  if (tid < 32) {
    const float ks = a.tab[0], vs = a.tab[1];
    const bool key = tid < 16;
    const int i = tid & 15;
    __half h, l;
    split_half(key ? (i < (1 << a.wk) ? a.kcent[i] * ks : 0.f) : (i < (1 << a.wv) ? a.vcent[i] * vs : 0.f), h, l);
    uint16_t (*t)[16] = key ? ktab : vtab;
    t[0][i] = __half_as_ushort(h);
    t[1][i] = __half_as_ushort(l);
  }
  constexpr int kGroups = D / 16;                  // sixteen coordinates of a token at a time
  for (int it = tid; it < kTok * kGroups; it += 256) {
    const int tt = it / kGroups, g = it % kGroups;
    const int64_t tok = t0 + tt;
    uint64_t kbits = 0, vbits = 0;
    uint32_t sbits = 0;
    float kn = 0.f, vn = 0.f;
    const bool live = tok < kv_len;
    if (live) load_group16<D>(a, seg, b, hkv, tok, g, kbits, vbits, sbits, kn, vn);
    const uint32_t km = (1u << a.wk) - 1u, vm = (1u << a.wv) - 1u;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t kw = 0, vw = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 4 * q + e;
        kw |= ((static_cast<uint32_t>(kbits >> (c * a.wk)) & km) | (((sbits >> c) & 1u) << 7)) << (8 * e);
        vw |= (live ? (static_cast<uint32_t>(vbits >> (c * a.wv)) & vm) : 0x80u) << (8 * e);
      }
      *reinterpret_cast<uint32_t*>(&kc_s[tt][16 * g + 4 * q]) = kw;
      *reinterpret_cast<uint32_t*>(&vc_s[tt][16 * g + 4 * q]) = vw;
    }
    if (g == 0) { nrm_s[0][tt] = kn; nrm_s[1][tt] = vn; }
  }
  __syncthreads();
  const int64_t tile_idx = static_cast<int64_t>(seg) * a.tiles + blockIdx.x;
  unsigned char* img = a.img + 2 * P::kPiBytes + tile_idx * P::kTileBytes;
  constexpr int kOp = kTok * D * 2;                // bytes of one operand of the tile
  for (int it = tid; it < kTok * (D / 8); it += 256) {                  // keys: token rows, coordinates along K
    const int tt = it / (D / 8), k0 = 8 * (it % (D / 8));
    const uint2 w = make_uint2(*reinterpret_cast<const uint32_t*>(&kc_s[tt][k0]), *reinterpret_cast<const uint32_t*>(&kc_s[tt][k0 + 4]));
    uint32_t hi[4], lo[4], sg[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t two = (p < 2 ? w.x : w.y) >> (16 * (p & 1));
      const uint32_t c0 = two & 15u, c1 = (two >> 8) & 15u;
      hi[p] = ktab[0][c0] | (static_cast<uint32_t>(ktab[0][c1]) << 16);
      if (TERMS == 2) lo[p] = ktab[1][c0] | (static_cast<uint32_t>(ktab[1][c1]) << 16);
      sg[p] = ((two & 0x80u) ? 0x3C00u : 0xBC00u) | ((two & 0x8000u) ? 0x3C000000u : 0xBC000000u);
    }
    unsigned char* dst = img + umma::sw128_offset(tt, k0, kTok);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + kOp) = make_uint4(sg[0], sg[1], sg[2], sg[3]);
    if (TERMS == 2) *reinterpret_cast<uint4*>(dst + 2 * kOp) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  for (int it = tid; it < D * (kTok / 8); it += 256) {                  // values: coordinate rows, tokens along K
    const int i = it % D, k0 = 8 * (it / D);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t c0 = vc_s[k0 + 2 * p][i], c1 = vc_s[k0 + 2 * p + 1][i];      // 0x80: past the end, value 0
      hi[p] = (c0 & 0x80u ? 0u : vtab[0][c0]) | (c1 & 0x80u ? 0u : static_cast<uint32_t>(vtab[0][c1]) << 16);
      if (TERMS == 2) lo[p] = (c0 & 0x80u ? 0u : vtab[1][c0]) | (c1 & 0x80u ? 0u : static_cast<uint32_t>(vtab[1][c1]) << 16);
    }
    unsigned char* dst = img + P::kKBytes + umma::sw128_offset(i, k0, D);
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    if (TERMS == 2) *reinterpret_cast<uint4*>(dst + kOp) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  if (tid < 32) {
    const float v0 = nrm_s[1][tid], v1 = nrm_s[1][tid + 32];
    float* nb = a.norms + tile_idx * (kNormBytes / 4);
    float down = 1.f;
    if (TERMS == 1) {
      // weights times norms become single fp16 numbers: the norms leave scaled by a power of two that brings the tile's
      // largest to [2^14, 2^15), so that the product stays inside fp16 and is a normal number down to 2^-28 of it.  A row
      // that sees only tokens 0 .. e of the tile scales up further, by 2^(byte e).  (TERMS = 2: every row for itself.)
      float p0 = fabsf(v0), p1 = fabsf(v1);                             // largest norm of tokens 0 .. tid, 32 .. tid + 32
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float q0 = __shfl_up_sync(QKV_FULL_MASK, p0, o), q1 = __shfl_up_sync(QKV_FULL_MASK, p1, o);
        if (tid >= o) { p0 = fmaxf(p0, q0); p1 = fmaxf(p1, q1); }
      }
      p1 = fmaxf(p1, __shfl_sync(QKV_FULL_MASK, p0, 31));
      down = scale_to<14>(__shfl_sync(QKV_FULL_MASK, p1, 31));
      uint8_t* up = reinterpret_cast<uint8_t*>(nb + 2 * kTok + 4);
      up[tid] = static_cast<uint8_t>((__float_as_uint(scale_to<14>(p0 * down)) >> 23) - 127u);
      up[tid + 32] = static_cast<uint8_t>((__float_as_uint(scale_to<14>(p1 * down)) >> 23) - 127u);
    }
    nb[tid] = nrm_s[0][tid];
    nb[tid + 32] = nrm_s[0][tid + 32];
    nb[kTok + tid] = v0 * down;
    nb[kTok + 32 + tid] = v1 * down;
    if (tid == 0) nb[2 * kTok] = inverse_pow2(down);
  }
}

// ---- attention ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(umma::smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   umma::smem_u32(dst)), "l"(src), "r"(bytes), "r"(umma::smem_u32(bar)) : "memory");
}

// 32 neighbouring elements (the index a multiple of 32): 16-byte loads where the base allows them.
__device__ __forceinline__ void load32(const void* q, int dtype, int64_t idx, bool live, float (&v)[32]) {
  if (!live) {
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = 0.f;
  } else if (reinterpret_cast<uintptr_t>(q) & 15u) {
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = load_float(q, dtype, idx + e);
  } else if (dtype == QKV_F32) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(q) + idx);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float4 x = __ldg(p + e);
      v[4 * e] = x.x; v[4 * e + 1] = x.y; v[4 * e + 2] = x.z; v[4 * e + 3] = x.w;
    }
  } else {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(q) + idx);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint4 x = __ldg(p + e);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (dtype == QKV_BF16) {
          v[8 * e + 2 * i] = __uint_as_float(w[i] << 16);
          v[8 * e + 2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        } else {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
          v[8 * e + 2 * i] = f.x; v[8 * e + 2 * i + 1] = f.y;
        }
      }
    }
  }
}

// v *= s, two at a time.
__device__ __forceinline__ void scale32(float (&v)[32], float s) {
#pragma unroll
  for (int e = 0; e < 32; e += 2)
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\t"
        "mul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}\n"
        : "+f"(v[e]), "+f"(v[e + 1]) : "f"(s));
}

// Sixteen tensor-memory columns of hi and of lo from 32 values.
__device__ __forceinline__ void store_split32(uint32_t t_hi, uint32_t t_lo, const float (&v)[32], bool with_lo) {
  uint32_t hi[16], lo[16];
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const __half2 h = __floats2half2_rn(v[2 * p], v[2 * p + 1]);
    hi[p] = *reinterpret_cast<const uint32_t*>(&h);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(v[2 * p] - f.x, v[2 * p + 1] - f.y);
    lo[p] = *reinterpret_cast<const uint32_t*>(&l);
  }
  umma::tmem_st16(t_hi, hi);
  if (with_lo) umma::tmem_st16(t_lo, lo);
}

// Query rows first .. first + 31 of a segment, one after another, in fp32 on the CUDA cores straight from the cache: the
// way out of a CTA in which a wait ran out.  A warp per row, a lane its coordinates lane, lane + 32, ...; far slower than
// the tensor core, and written only to be right.
template <int D>
__device__ __forceinline__ void attend_rows_fp32(const PrefillArgs& a, int seg, int b, int hkv, int64_t kv_len, int first,
                                                 int nq, int lane) {
  constexpr int PL = D / 32;
  const uint32_t km = (1u << a.wk) - 1u, vm = (1u << a.wv) - 1u;
  auto times = [&](const float (&x)[PL], bool transposed, float (&y)[PL]) {      // y = Pi x, or its transpose
#pragma unroll
    for (int t = 0; t < PL; ++t) y[t] = 0.f;
#pragma unroll
    for (int u = 0; u < PL; ++u) {
#pragma unroll 1
      for (int j = 0; j < 32; ++j) {
        const float xj = __shfl_sync(QKV_FULL_MASK, x[u], j);
        const int from = 32 * u + j;
#pragma unroll
        for (int t = 0; t < PL; ++t) {
          const int to = lane + 32 * t;
          y[t] = fmaf(xj, __ldg(a.Pi + (transposed ? from * D + to : to * D + from)), y[t]);
        }
      }
    }
  };
#pragma unroll 1
  for (int r = first; r < first + 32 && r < nq; ++r) {
    const int64_t qrow = (static_cast<int64_t>(b) * a.Hq + hkv * a.G) * a.q_len + r;
    const int64_t lim = a.causal ? kv_len - a.q_len + r % a.q_len : kv_len - 1;
    float x[PL], y[PL], w[PL], o[PL], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int t = 0; t < PL; ++t) x[t] = load_float(a.q, a.q_dtype, qrow * D + lane + 32 * t);
    times(x, false, y);
#pragma unroll
    for (int t = 0; t < PL; ++t) {
      w[t] = (a.qjl_scale * a.scale) * (fabsf(y[t]) * __ldg(a.S + lane + 32 * t));
      y[t] *= a.scale;
      o[t] = 0.f;
    }
#pragma unroll 1
    for (int64_t tok = 0; tok <= lim; ++tok) {
      float s = 0.f, vc[PL], kn = 0.f, vn = 0.f;
#pragma unroll
      for (int t = 0; t < PL; ++t) {
        uint64_t kbits = 0, vbits = 0;
        uint32_t sbits = 0;
        const int j = lane + 32 * t, c = j & 15;
        load_group16<D>(a, seg, b, hkv, tok, j >> 4, kbits, vbits, sbits, kn, vn);
        s = fmaf(y[t], __ldg(a.kcent + (static_cast<uint32_t>(kbits >> (c * a.wk)) & km)), s) + ((sbits >> c) & 1u ? w[t] : -w[t]);
        vc[t] = __ldg(a.vcent + (static_cast<uint32_t>(vbits >> (c * a.wv)) & vm));
      }
#pragma unroll
      for (int e = 16; e > 0; e >>= 1) s += __shfl_xor_sync(QKV_FULL_MASK, s, e);
      s *= kn;
      if (s > m) {
        const float alpha = m == -INFINITY ? 0.f : expf(m - s);
        m = s;
        l *= alpha;
#pragma unroll
        for (int t = 0; t < PL; ++t) o[t] *= alpha;
      }
      const float p = s == -INFINITY ? 0.f : expf(s - m), pv = p * vn;
      l += p;
#pragma unroll
      for (int t = 0; t < PL; ++t) o[t] = fmaf(pv, vc[t], o[t]);
    }
    const float inv = 1.f / fmaxf(l, 1e-30f);
#pragma unroll
    for (int t = 0; t < PL; ++t) o[t] *= inv;
    times(o, true, y);
#pragma unroll
    for (int t = 0; t < PL; ++t) a.out[qrow * D + lane + 32 * t] = y[t] + a.tab[2];
  }
}

// Query rows of a CTA: rows first .. of a segment (batch entry b, KV head hkv), late positions (more tokens) first.
struct CtaRows { int seg, b, hkv, first; int64_t kv_len; };
template <int D, int TERMS>
__device__ __forceinline__ CtaRows cta_rows(const PrefillArgs& a, uint32_t bx, uint32_t by) {
  constexpr int kRows = Pf<D, TERMS>::NT * kRowsT;
  CtaRows r;
  r.seg = static_cast<int>(bx);
  r.b = r.seg / a.Hkv;
  r.hkv = r.seg % a.Hkv;
  int rt = static_cast<int>(gridDim.y - 1 - by);
  if (a.causal && a.q_len % kRows == 0) {                               // ... over all heads of the segment
    const int per_head = a.q_len / kRows;
    rt = (static_cast<int>(by) % a.G) * per_head + per_head - 1 - static_cast<int>(by) / a.G;
  }
  r.first = rt * kRows;
  r.kv_len = a.kv_len;
  if (a.block_table) r.kv_len = min(static_cast<int64_t>(max(a.seq_lens[r.b], 0)), a.kv_len);
  return r;
}

// Warps 0..3 own row tile 0, warps 4..7 row tile 1 (NT = 2): a thread per query row.  Of the four warps behind them one
// thread issues every MMA and one every copy.  
template <int D, int TERMS>
__global__ void __launch_bounds__(Pf<D, TERMS>::kThreads, 1) prefill_kernel(PrefillArgs a) {
  using P = Pf<D, TERMS>;
  constexpr int NT = P::NT, ST = P::ST;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* q_s = smem;                                            // [NT] query operands; first and last Pi's
  unsigned char* ring = smem + NT * P::kQBytes;
  unsigned char* norm_s = ring + ST * P::kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(norm_s + kNormSlots * kNormBytes);
  uint64_t* pi_full = bars;                 // phase 0: operand of the rotation, 1: of the un-rotation
  uint64_t* k_full = bars + 1;              // [ST]
  uint64_t* v_full = bars + 3;              // [ST]
  uint64_t* k_free = bars + 5;              // [ST]
  uint64_t* v_free = bars + 7;              // [ST]
  uint64_t* out_full = bars + 9;            // [NT] the output rows
  uint64_t* p_ready = bars + 11;            // [NT] operand of the rotation, query operand, then weights, then the sums
  uint64_t* o_full = bars + 13;             // [NT] value sums of a tile
  uint64_t* drain = bars + 15;              // after a wait that ran out
  uint64_t* rot_done = bars + 16;           // every row tile's queries are rotated
  uint64_t* n_full = bars + 17;             // [kNormSlots]
  uint64_t* s_full = bars + 17 + kNormSlots;      // [NT][2] scores of a tile, per buffer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 4);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  const CtaRows rows = cta_rows<D, TERMS>(a, blockIdx.x, blockIdx.y);
  const int nq = a.G * a.q_len, seg = rows.seg, b = rows.b, hkv = rows.hkv, r0 = rows.first;
  const int64_t kv_len = rows.kv_len;
  int64_t seen = kv_len;
  if (a.causal) {
    const int n_rows = nq - r0 < NT * kRowsT ? nq - r0 : NT * kRowsT, p_first = r0 % a.q_len;
    const int last = p_first + n_rows - 1 >= a.q_len ? a.q_len - 1 : p_first + n_rows - 1;
    const int64_t visible = kv_len - a.q_len + last + 1;
    if (seen > visible) seen = visible;
  }
  const int n = seen > 0 ? static_cast<int>((seen + kTok - 1) / kTok) : 0;    // token tiles

  // ---- set-up ----
  if (tid == 0) {
    for (int i = 0; i < 17 + kNormSlots + 4; ++i) umma::mbar_init(bars + i, (i == 11 || i == 12) ? kRowsT : 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    *dead = 0;
  }
  if (warp == 0) umma::tmem_alloc(tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint64_t* bar, uint32_t parity) {                     // bounded; false once anything ran out
    if (*dead) return false;
    if (umma::mbar_wait(bar, parity)) return true;
    *dead = 1;
    atomicAdd(&g_prefill_timeouts, 1u);
    return false;
  };

  if (warp >= NT * 4) {
    // 384 threads start with 168 registers; a thread with a query row holds its D sums: 256 x 224 + 128 x 56 = 384 x 168
    if (NT == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;\n");
    if (warp == NT * 4 + 1 && lane == 0) {
      // ---- copies ----
      const unsigned char* tiles = a.img + 2 * P::kPiBytes + static_cast<int64_t>(seg) * a.tiles * P::kTileBytes;
      const float* norms = a.norms + static_cast<int64_t>(seg) * a.tiles * (kNormBytes / 4);
      expect_tx(pi_full, P::kPiBytes);
      bulk_copy(q_s, a.img, P::kPiBytes, pi_full);
      bool ok = true;
      int issued = 0, pi_phases = 1;
      for (int j = 0; j < n && ok; ++j) {
        const int st = j % ST;
        const uint32_t par = ((j / ST) & 1) ^ 1;
        unsigned char* dst = ring + st * P::kTileBytes;
        // the norm slot is free by then: the scores of tile j - ST were issued after the weights of tile j - ST - SB
        if (j >= ST && !(ok = wait(k_free + st, par))) break;
        expect_tx(k_full + st, P::kKBytes);
        expect_tx(n_full + j % kNormSlots, kNormBytes);
        bulk_copy(dst, tiles + static_cast<int64_t>(j) * P::kTileBytes, P::kKBytes, k_full + st);
        bulk_copy(norm_s + (j % kNormSlots) * kNormBytes, norms + static_cast<int64_t>(j) * (kNormBytes / 4), kNormBytes, n_full + j % kNormSlots);
        issued = j + 1;
        if (j >= ST && !(ok = wait(v_free + st, par))) {                // the key copy in flight is waited for below
          umma::mbar_wait(k_full + st, (j / ST) & 1);
          umma::mbar_wait(n_full + j % kNormSlots, (j / kNormSlots) & 1);
          issued = j;
          break;
        }
        expect_tx(v_full + st, P::kVBytes);
        bulk_copy(dst + P::kKBytes, tiles + static_cast<int64_t>(j) * P::kTileBytes + P::kKBytes, P::kVBytes, v_full + st);
      }
      // the queries' operands have been read once the scores of the last tile are there
      if (ok && (n > 0 ? wait(k_free + (n - 1) % ST, ((n - 1) / ST) & 1) : wait(rot_done, 0))) {
        expect_tx(pi_full, P::kPiBytes);
        bulk_copy(q_s, a.img + P::kPiBytes, P::kPiBytes, pi_full);
        pi_phases = 2;
      }
      for (int j = issued > ST ? issued - ST : 0; j < issued; ++j) {    // nothing may still be on its way at the end
        umma::mbar_wait(k_full + j % ST, (j / ST) & 1);
        umma::mbar_wait(v_full + j % ST, (j / ST) & 1);
        umma::mbar_wait(n_full + j % kNormSlots, (j / kNormSlots) & 1);
      }
      umma::mbar_wait(pi_full, (pi_phases - 1) & 1);
    } else if (warp == NT * 4 && lane == 0) {
      // ---- MMAs ----
      constexpr uint32_t id_s = umma::instr_desc(umma::kFmtF16, 128, kTok), id_d = umma::instr_desc(umma::kFmtF16, 128, D);
      const uint32_t pi_addr = umma::smem_u32(q_s);
      auto rotate = [&](int t) {            // (hi + lo at 128) x (hi + lo of the staged matrix)
        const uint32_t d = tmem + P::kCols * t, ah = d + 128, al = ah + D / 2;
        auto step = [&](uint32_t dst, uint32_t av, uint32_t bv, int ks, bool acc) {
          umma::mma_f16_ts(dst, av + 8 * ks, umma::smem_desc_sw128(bv + (ks >> 2) * (D * 128) + (ks & 3) * 32), id_d, acc);
        };
        constexpr int kS = P::kS, kA = P::kA, kB = P::kB;
#pragma unroll
        for (int ks = 0; ks < kS; ++ks) step(d, al, pi_addr, ks, ks != 0);
#pragma unroll
        for (int ks = 0; ks < kS; ++ks) step(d, ah, pi_addr + D * D * 2, ks, true);
#pragma unroll
        for (int ks = 0; ks < kS; ++ks)
          step(d + (ks < kA ? 0 : (ks < kB ? P::kR1 : P::kR2)), ah, pi_addr, ks, ks != kA && ks != kB);
      };
      auto scores = [&](int t, int j) {
        const uint32_t qa = umma::smem_u32(q_s + t * P::kQBytes), ka = umma::smem_u32(ring + (j % ST) * P::kTileBytes);
        constexpr uint32_t kQOp = kRowsT * D * 2, kKOp = kTok * D * 2;
        const uint32_t d = tmem + P::kCols * t + 64 * (j % P::SB);
        auto product = [&](uint32_t dst, uint32_t qo, uint32_t ko, int k0, int k1, bool acc) {
#pragma unroll
          for (int ks = k0; ks < k1; ++ks) {
            umma::mma_f16(dst, umma::smem_desc_sw128(qa + qo * kQOp + (ks >> 2) * (kRowsT * 128) + (ks & 3) * 32),
                          umma::smem_desc_sw128(ka + ko * kKOp + (ks >> 2) * (kTok * 128) + (ks & 3) * 32), id_s, acc);
            acc = true;
          }
        };
        if (P::kSplit) {
          constexpr int kH = P::kScorePart;
          const uint32_t sign = D == 64 ? d + 64 : d + 256;
          product(d, 2, 0, 0, D / 16, false);                                  // ql ch
          product(d, 0, 2, 0, D / 16, true);                                   // qh cl
          product(sign, 3, 1, 0, D / 16, false);                               // wl sign
          product(d, 0, 0, 0, kH, true);                                       // qh ch
          product(sign, 1, 1, 0, kH, true);                                    // wh sign
          if (D == 128) {
            product(d + 64, 0, 0, kH, D / 16, false);
            product(sign + 64, 1, 1, kH, D / 16, false);
          }
        } else {
          product(d, 1, 1, 0, D / 16, false);
          product(d, 0, 0, 0, D / 16, true);
        }
        umma::commit(s_full + 2 * t + j % P::SB);
      };
      auto values = [&](int t, int j) {
        const uint32_t base = tmem + P::kCols * t, d = base + 128, ph = base + 64 * (j % P::SB), pl = ph + 32;
        const uint32_t va = umma::smem_u32(ring + (j % ST) * P::kTileBytes + P::kKBytes);
        bool acc = false;
#pragma unroll
        for (int pr = P::kSplit ? 0 : 2; pr < 3; ++pr) {                       // pl vh, ph vl, ph vh
          const uint32_t av = pr == 0 ? pl : ph, bv = va + (pr == 1 ? kTok * D * 2 : 0);
#pragma unroll
          for (int ks = 0; ks < kTok / 16; ++ks) {
            const bool second = P::kSplit && pr == 2 && ks >= P::kValuePart;
            umma::mma_f16_ts(second ? base + P::kO2 : d, av + 8 * ks, umma::smem_desc_sw128(bv + ks * 32), id_d,
                             second ? ks != P::kValuePart : acc);
            acc = true;
          }
        }
        umma::commit(o_full + t);
      };
      bool ok = wait(pi_full, 0);
      for (int t = 0; t < NT && ok; ++t) {
        if (!(ok = wait(p_ready + t, 0))) break;
        umma::fence_after_sync();
        rotate(t);
        if (t == NT - 1) umma::commit(rot_done);
      }
      // the scores of a tile are issued SB tiles ahead of its weights
      for (int t = 0; t < NT && ok; ++t) {
        if (!(ok = wait(p_ready + t, 1)) || n == 0) continue;
        if (t == 0 && !(ok = wait(k_full, 0))) break;
        umma::fence_after_sync();
        scores(t, 0);
        if (t == NT - 1) umma::commit(k_free);
      }
      for (int t = 0; t < NT && ok && n > 1 && P::SB == 2; ++t) {
        if (t == 0 && !(ok = wait(k_full + 1 % ST, (1 / ST) & 1))) break;
        scores(t, 1);
        if (t == NT - 1) umma::commit(k_free + 1 % ST);
      }
      for (int j = 0; j < n && ok; ++j) {
        for (int t = 0; t < NT && ok; ++t) {
          if (!(ok = wait(p_ready + t, j & 1))) break;
          if (t == 0 && !(ok = wait(v_full + j % ST, (j / ST) & 1))) break;
          if (a.test_drop_mma && (blockIdx.x | blockIdx.y) == 0 && t == 0 && j == 1) continue;   // test hook
          umma::fence_after_sync();
          values(t, j);
          if (t == NT - 1) umma::commit(v_free + j % ST);
          const int js = j + P::SB;
          if (js < n) {
            if (t == 0 && !(ok = wait(k_full + js % ST, (js / ST) & 1))) break;
            scores(t, js);
            if (t == NT - 1) umma::commit(k_free + js % ST);
          }
        }
      }
      if (ok) ok = wait(pi_full, 1);
      for (int t = 0; t < NT && ok; ++t) {
        if (!(ok = wait(p_ready + t, n & 1))) break;
        umma::fence_after_sync();
        rotate(t);
        umma::commit(out_full + t);
      }
      if (!ok) {                            // whatever was issued has ended before tensor memory is given back
        umma::commit(drain);
        umma::mbar_wait(drain, 0);
      }
    }
  } else {
    // ---- a query row per thread ----
    if (NT == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;\n");
    const int t = warp >> 2, row = 32 * (warp & 3) + lane, r = r0 + t * kRowsT + row;
    const uint32_t my = tmem + P::kCols * t + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    const bool live = r < nq;
    const int64_t qrow = (static_cast<int64_t>(b) * a.Hq + hkv * a.G) * a.q_len + (live ? r : 0);
    int64_t lim64 = -1;                     // last token this row sees
    if (live) lim64 = a.causal ? kv_len - a.q_len + r % a.q_len : kv_len - 1;
    const int lim = lim64 < -1 ? -1 : static_cast<int>(lim64);
    constexpr float kLog2e = static_cast<float>(1.4426950408889634 * P::kScoresUp);

    auto rotated32 = [&](int c, uint32_t (&v)[32]) {        // 32 columns of a rotation's result
      umma::tmem_ld32(my + c, v);
      if (P::kSplit) {
        uint32_t w[32];
        umma::tmem_ld32(my + P::kR2 + c, w);
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(w[e]));
        umma::tmem_ld32(my + P::kR1 + c, w);
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(w[e]));
      }
    };
    auto scores32 = [&](int j, int c, uint32_t (&v)[32]) {
      umma::tmem_ld32(my + 64 * (j % P::SB) + c, v);
      if (P::kSplit) {
        constexpr int kPart[3] = {64, 256, 320};
#pragma unroll
        for (int k = 0; k < (D == 64 ? 1 : 3); ++k) {
          uint32_t w[32];
          umma::tmem_ld32(my + kPart[k] + c, w);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(w[e]));
        }
      }
    };
    float R;
    {
      float mx = 0.f;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        float v[32];
        load32(a.q, a.q_dtype, qrow * D + c, live, v);
#pragma unroll
        for (int e = 0; e < 32; ++e) mx = fmaxf(mx, fabsf(v[e]));
      }
      R = scale_to<13>(mx);
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        float v[32];
        load32(a.q, a.q_dtype, qrow * D + c, live, v);
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] *= R;
        store_split32(my + 128 + c / 2, my + 128 + D / 2 + c / 2, v, true);
      }
      umma::tmem_st_wait();
      umma::fence_before_sync();
      arrive(p_ready + t);
    }
    float rs = 0.f;                         // score units (log2) per unit of the accumulator
    auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(QKV_FULL_MASK, wait(bar, parity)) != 0; };
    bool ok = wait_all(rot_done, 0);                                    // of every row tile: Pi's place is free
    if (ok) {
      umma::fence_after_sync();
      const float un = inverse_pow2(R) * (1.f / kPiScale), ks = a.tab[0];
      float mx = 0.f;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        rotated32(c, v);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float x = __uint_as_float(v[e]) * un;
          const float w = (a.qjl_scale * a.scale) * (fabsf(x) * __ldg(a.S + c + e)) * ks;
          mx = fmaxf(mx, fmaxf(fabsf(x * a.scale), fabsf(w)));
        }
      }
      const float R2 = scale_to<13>(mx);
      rs = kLog2e * inverse_pow2(R2) / ks;
      unsigned char* qo = q_s + t * P::kQBytes;
      constexpr int kQOp = kRowsT * D * 2;
#pragma unroll 1
      for (int c = 0; c < (n > 0 ? D : 0); c += 32) {      // (nothing to see: the place goes to the second Pi at once)
        uint32_t v[32];
        rotated32(c, v);
#pragma unroll
        for (int e8 = 0; e8 < 4; ++e8) {
          uint32_t qh[4], ql[4], wh[4], wl[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            float qv[2], wv[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int i = 8 * e8 + 2 * p + e;
              const float x = __uint_as_float(v[i]) * un;
              qv[e] = x * a.scale * R2;
              wv[e] = (a.qjl_scale * a.scale) * (fabsf(x) * __ldg(a.S + c + i)) * ks * R2;
            }
            const __half2 h = __floats2half2_rn(qv[0], qv[1]), g = __floats2half2_rn(wv[0], wv[1]);
            qh[p] = *reinterpret_cast<const uint32_t*>(&h);
            wh[p] = *reinterpret_cast<const uint32_t*>(&g);
            if (TERMS == 2) {
              const float2 hf = __half22float2(h), gf = __half22float2(g);
              ql[p] = pack_half2(qv[0] - hf.x, qv[1] - hf.y);
              wl[p] = pack_half2(wv[0] - gf.x, wv[1] - gf.y);
            }
          }
          unsigned char* dst = qo + umma::sw128_offset(row, c + 8 * e8, kRowsT);
          *reinterpret_cast<uint4*>(dst) = make_uint4(qh[0], qh[1], qh[2], qh[3]);
          *reinterpret_cast<uint4*>(dst + kQOp) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
          if (TERMS == 2) {
            *reinterpret_cast<uint4*>(dst + 2 * kQOp) = make_uint4(ql[0], ql[1], ql[2], ql[3]);
            *reinterpret_cast<uint4*>(dst + 3 * kQOp) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
          }
        }
      }
      umma::fence_smem_to_async();
      umma::fence_before_sync();
      arrive(p_ready + t);
    }

    float O[D];
#pragma unroll
    for (int i = 0; i < D; ++i) O[i] = 0.f;
    float m = -1e30f, l = 0.f, alpha_prev = 1.f, up_prev = 0.f;
    // O = O * alpha + (value sums of the tile before)
    auto gather = [&](float alpha, float up) {
      const bool keep = __all_sync(QKV_FULL_MASK, alpha == 1.f);        // nearly always after the first tiles
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        umma::tmem_ld32(my + 128 + c, v);
        if (P::kSplit) {
          uint32_t w[32];
          umma::tmem_ld32(my + P::kO2 + c, w);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(w[e]));
        }
        if (keep) {
#pragma unroll
          for (int e = 0; e < 32; ++e) O[c + e] = fmaf(__uint_as_float(v[e]), up, O[c + e]);
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) O[c + e] = fmaf(__uint_as_float(v[e]), up, O[c + e] * alpha);
        }
      }
    };
    for (int j = 0; j < n && ok; ++j) {
      if (!(ok = wait_all(n_full + j % kNormSlots, (j / kNormSlots) & 1) && wait_all(s_full + 2 * t + j % P::SB, (j / P::SB) & 1))) break;
      umma::fence_after_sync();
      const float* nb = reinterpret_cast<const float*>(norm_s + (j % kNormSlots) * kNormBytes);
      const int left = lim - j * kTok;                                  // tokens 0 .. left of the tile are visible
      const bool masked = __any_sync(QKV_FULL_MASK, left < kTok - 1);   // warp-uniform
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < kTok; c += 32) {
        uint32_t v[32];
        scores32(j, c, v);
        if (masked) {
#pragma unroll
          for (int e = 0; e < 32; ++e) mx[e & 1] = fmaxf(mx[e & 1], c + e > left ? -INFINITY : __uint_as_float(v[e]) * nb[c + e]);
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) mx[e & 1] = fmaxf(mx[e & 1], __uint_as_float(v[e]) * nb[c + e]);
        }
      }
      const float m_new = fmaxf(m, ceilf(fmaxf(mx[0], mx[1]) * rs));
      const float alpha = ex2(m - m_new);
      m = m_new;
      if (j > 0) {
        if (!(ok = wait_all(o_full + t, (j - 1) & 1))) break;
        umma::fence_after_sync();
        gather(alpha_prev, up_prev);
      }
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
      auto weigh = [&](int c, const uint32_t (&v)[32], float (&pv)[32]) {
#pragma unroll
        for (int e = 0; e < 32; ++e) pv[e] = ex2(fmaf(__uint_as_float(v[e]) * nb[c + e], rs, -m));
        if (masked) {
#pragma unroll
          for (int e = 0; e < 32; ++e) pv[e] = c + e > left ? 0.f : pv[e];
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          ls[e & 3] += pv[e];
          pv[e] *= nb[kTok + c + e];
        }
      };
      const uint32_t pt = my + 64 * (j % P::SB);
      float up;
      if (P::kSplit) {                    // hi to columns 0 .. 31 of the scores' place, lo to 32 .. 63: read all of it first
        // the row's products are scaled by a power of two that brings their largest to [2^14, 2^15): what another token
        // weighs, or a token that this row cannot see, takes no bits from them
        uint32_t v[2][32];
        float pv[2][32], mp[2] = {0.f, 0.f};
        scores32(j, 0, v[0]);
        scores32(j, 32, v[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          weigh(32 * h, v[h], pv[h]);
#pragma unroll
          for (int e = 0; e < 32; ++e) mp[e & 1] = fmaxf(mp[e & 1], fabsf(pv[h][e]));
        }
        const float down = scale_to<14>(fmaxf(mp[0], mp[1]));
        up = inverse_pow2(down);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          scale32(pv[h], down);
          store_split32(pt + 16 * h, pt + 32 + 16 * h, pv[h], true);
        }
      } else {                            // hi alone stays inside the half that has been read
        // the tile's scale is that of its largest norm; a row that sees only a part of the tile takes the part's
        float more = 1.f;
        if (masked && left >= 0) {
          const uint32_t k = reinterpret_cast<const uint8_t*>(nb + 2 * kTok + 4)[left < kTok ? left : kTok - 1];
          more = __uint_as_float((127u + k) << 23);
        }
        up = nb[2 * kTok] * inverse_pow2(more);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[32];
          float pv[32];
          scores32(j, 32 * h, v);
          weigh(32 * h, v, pv);
          if (masked) {
#pragma unroll
            for (int e = 0; e < 32; ++e) pv[e] *= more;
          }
          store_split32(pt + 16 * h, pt, pv, false);
        }
      }
      l = l * alpha + ((ls[0] + ls[1]) + (ls[2] + ls[3]));
      alpha_prev = alpha;
      up_prev = up;
      umma::tmem_st_wait();
      umma::fence_before_sync();
      arrive(p_ready + t);
    }
    if (ok && n > 0) {
      ok = wait_all(o_full + t, (n - 1) & 1);
      umma::fence_after_sync();
      if (ok) gather(alpha_prev, up_prev);
    }
    if (ok) {
      const float inv = 1.f / (fmaxf(l, 1e-30f) * a.tab[1]);
      float mo = 0.f;
#pragma unroll
      for (int i = 0; i < D; ++i) { O[i] *= inv; mo = fmaxf(mo, fabsf(O[i])); }
      const float R3 = scale_to<13>(mo);
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        float v[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = O[c + e] * R3;
        store_split32(my + 128 + c / 2, my + 128 + D / 2 + c / 2, v, true);
      }
      umma::tmem_st_wait();
      umma::fence_before_sync();
      arrive(p_ready + t);
      ok = wait_all(out_full + t, 0);
      umma::fence_after_sync();
      if (ok) {
        const float un = inverse_pow2(R3) * static_cast<float>(P::kOutputUp / kPiScale) + a.tab[2];
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t v[32];
          rotated32(c, v);
          if (live) {
            float4* dst = reinterpret_cast<float4*>(a.out + qrow * D + c);
#pragma unroll
            for (int e = 0; e < 8; ++e)
              dst[e] = make_float4(__uint_as_float(v[4 * e]) * un, __uint_as_float(v[4 * e + 1]) * un,
                                   __uint_as_float(v[4 * e + 2]) * un, __uint_as_float(v[4 * e + 3]) * un);
          }
        }
      }
    }
    if (!ok) {                              // warp-uniform
      uint32_t bx, by, th;                  // (read again: nothing of this is held in registers through the loop)
      asm volatile("mov.u32 %0, %%ctaid.x;\n\tmov.u32 %1, %%ctaid.y;\n\tmov.u32 %2, %%tid.x;\n" : "=r"(bx), "=r"(by), "=r"(th));
      const CtaRows c = cta_rows<D, TERMS>(a, bx, by);
      attend_rows_fp32<D>(a, c.seg, c.b, c.hkv, c.kv_len, c.first + static_cast<int>(th & ~31u), a.G * a.q_len,
                          static_cast<int>(th & 31u));
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

constexpr size_t kMaxImageBytes = size_t(1) << 30;

int64_t token_tiles(int64_t kv_len) { return (kv_len + kTok - 1) / kTok; }

size_t image_bytes(int B, int Hkv, int64_t kv_len, int d, int terms) {
  const size_t op = static_cast<size_t>(kTok) * d * 2, n = static_cast<size_t>(B) * Hkv * token_tiles(kv_len);
  return 256 + 2 * static_cast<size_t>(2 * d * d * 2) + n * ((2 * terms + 1) * op + kNormBytes);
}

template <int D, int TERMS>
int launch_t(PrefillArgs& a, cudaStream_t st) {
  using P = Pf<D, TERMS>;
  a.tab = reinterpret_cast<float*>(a.img);
  a.img += 256;
  a.tiles = static_cast<int>(token_tiles(a.kv_len));
  a.norms = reinterpret_cast<float*>(a.img + 2 * P::kPiBytes + static_cast<size_t>(a.B) * a.Hkv * a.tiles * P::kTileBytes);
  if (cudaFuncSetAttribute(prefill_kernel<D, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(P::kSmem)) != cudaSuccess)
    return QKV_ELAUNCH;
  prefill_setup_kernel<D, TERMS><<<1 + D / 4, 256, 0, st>>>(a);
  prefill_operands_kernel<D, TERMS><<<dim3(a.tiles, a.B * a.Hkv), 256, 0, st>>>(a);
  const int rows = P::NT * kRowsT, row_tiles = (a.G * a.q_len + rows - 1) / rows;
  prefill_kernel<D, TERMS><<<dim3(a.B * a.Hkv, row_tiles), P::kThreads, P::kSmem, st>>>(a);
  return check_launch();
}

}  // namespace

unsigned int prefill_timeouts() {
  unsigned int v = 0;
  cudaMemcpyFromSymbol(&v, g_prefill_timeouts, sizeof(v));
  return v;
}

// Times in us, fitted to 310 measured pairs (1 to 64 segments, 64 to 8192 rows, 256 to 16384 tokens): this path has a
// constant and a time per token tile and round of CTAs, of which a round behind the first sees what is visible on average;
// the decode kernels a constant and a rate of pairs of query row and token, hidden ones included.  At none of
// them the way taken is more than 15 % behind the other (before, with one time per tile for all widths and half of the
// decode kernels' time: 300 instead of 180 us for 2 segments x 256 rows x 4096 tokens at d = 128, 4 bits, and 104
// instead of 56 us for 64 segments x 256 rows x 256 tokens over records).
bool prefill_pays(int64_t segs, int64_t nq, int q_len, int64_t kv_len, int d, int terms, bool causal) {
  const bool records = terms == 1, wide = d == 128 && !records;
  const double rounds = ceil(segs * ceil(nq / (wide ? 1.0 * kRowsT : 2.0 * kRowsT)) / kNumSMs);
  const double seen = causal && rounds > 1 ? 1.0 - 0.5 * (q_len - 1) / kv_len : 1.0;
  const double mine = (records ? 42.0 : 34.0) + (records ? 3.0 : (wide ? 4.6 : 3.5)) * rounds * seen * ((kv_len + kTok - 1) / kTok);
  const double theirs = (records ? 48.3 : (wide ? 44.0 : 36.0)) + 1.0 * segs * nq * kv_len / (records ? 200e3 : (wide ? 17.5e3 : 39e3));
  return mine < theirs;
}

// Whether the call's form is covered, and (unless forced) whether it is the faster way.
bool prefill_rows_ok(int B, int Hkv, int64_t group, int q_len, int64_t kv_len, int d, int terms, bool causal) {
  const int64_t nq = group * q_len;
  const char* e = getenv("QUASHKV_B200_PREFILL_TCGEN05");      // 0 / 1: never / wherever it can, for A/B checks
  if (e && e[0] == '0') return false;
  if (!((d == 64 || d == 128) && nq <= 128 * 65535 && B * static_cast<int64_t>(Hkv) < 65535)) return false;
  if (e && e[0] == '1') return nq >= 16;
  return nq >= kPrefillRows && prefill_pays(B * static_cast<int64_t>(Hkv), nq, q_len, kv_len, d, terms, causal);
}

size_t prefill_workspace_bytes(int B, int Hq, int Hkv, int q_len, int64_t kv_len, int d) {
  // (asked without the mask: a causal call is taken wherever one without is)
  const int64_t group = Hq / (Hkv > 0 ? Hkv : 1);
  if (!prefill_rows_ok(B, Hkv, group, q_len, kv_len, d, 2, true) && !prefill_rows_ok(B, Hkv, group, q_len, kv_len, d, 1, true))
    return 0;
  const size_t two = image_bytes(B, Hkv, kv_len, d, 2), one = image_bytes(B, Hkv, kv_len, d, 1);
  return two <= kMaxImageBytes ? two : (d == 128 && one <= kMaxImageBytes ? one : 0);
}

bool prefill_ok(const AttnArgs& s, size_t workspace_bytes) {
  if (!prefill_rows_ok(s.B, s.Hkv, s.G, s.q_len, s.kv_len, s.d, s.records ? 1 : 2, s.causal != 0)) return false;
  const size_t need = image_bytes(s.B, s.Hkv, s.kv_len, s.d, s.records ? 1 : 2);
  return need <= kMaxImageBytes && need <= workspace_bytes && (reinterpret_cast<uintptr_t>(s.out) & 15u) == 0;
}

int launch_prefill(const AttnArgs& s, const void* q, int q_dtype, int key_bits, int val_bits, const float* S, float qjl_scale,
                   float scale, void* workspace, cudaStream_t st) {
  PrefillArgs a{};
  a.q = q; a.q_dtype = q_dtype; a.cache = s.cache; a.records = s.records;
  a.block_table = s.block_table; a.seq_lens = s.seq_lens; a.max_blocks = s.max_blocks; a.block_size = s.block_size;
  a.B = s.B; a.Hq = s.Hq; a.Hkv = s.Hkv; a.G = s.G; a.q_len = s.q_len; a.causal = s.causal;
  a.wk = key_bits - 1; a.wv = val_bits; a.kv_len = s.kv_len;
  a.Pi = s.Pi; a.S = S; a.kcent = s.kcent; a.vcent = s.vcent; a.qjl_scale = qjl_scale; a.scale = scale;
  a.out = s.out;
  const char* hook = getenv("QUASHKV_B200_TEST_DROP_MMA");      // 1: tests only
  a.test_drop_mma = hook && hook[0] == '1';
  a.img = static_cast<unsigned char*>(workspace);
  if (s.d == 64) return launch_t<64, 2>(a, st);
  return s.records ? launch_t<128, 1>(a, st) : launch_t<128, 2>(a, st);
}

}  // namespace qkv
