// Compress (normalise -> rotate -> bucketise -> sign bit -> pack) and decompress (unpack -> centroid gather ->
// un-rotate -> rescale) with the rotation as fp32 FMA chains on the CUDA cores: every dimension up to 128, every
// width and layout, and the kernels of small calls at d = 128 as well.
//
// The order of the chain (fp32 FMA, ascending input coordinate) is what the codes are defined by; two kernels keep it:
//
// small (compress_small_kernel, decompress_small_kernel): a thread owns ONE output coordinate, keeps its row (column) of
//   Pi in registers, 128 of them, and has four vectors in flight.  A tile is four vectors (times the groups of d threads
//   that a CTA holds), so that a few hundred vectors are already spread over a hundred CTAs, and the set-up of a CTA is
//   one round trip to L2: Pi (64 KB) goes through shared memory in coalesced 16-byte copies at a pitch of d + 4 words,
//   so that a thread's read of its own row is free of bank conflicts.  Every FMA takes its vector element from shared
//   memory, a broadcast that still costs a return slot of 128 bytes a cycle, so this form runs at a quarter of the FMA
//   rate: right for latency, wrong for bulk.
// bulk (compress_bulk_kernel, decompress_bulk_kernel): a thread owns 8 coordinates x 8 vectors; both operands come from
//   shared memory as float4, 64 FMAs per four loads, where FMA rate and load return balance.  Up to four CTAs share an
//   SM, so that one loads while another multiplies: 400,000 vectors of 64 at 2 bits, compress fp32 300 (two CTAs) -> 211
//   us, bf16 360 -> 198, decompress to fp32 285 -> 165.
//
// The keys and values of an append run as ONE launch (two jobs), and both kernels write their codes straight to where the
// cache keeps them: row-major planes, contiguous or through a block table; the small one also the tile records of the
// d = 128, 3/3-bit cache.
#include "mma_decode.cuh"
#include "rotate_common.cuh"
#include "tile_format.cuh"

namespace qkv {

namespace {

__device__ unsigned long long g_rows_dropped = 0;        // rows without a slot, small paged appends

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kCtasPerSm = 3;                  // 168 registers a thread; 68 KB of shared memory

template <int DR> struct Shape {
  static constexpr int kGroups = kThreads / DR;              // groups of DR threads, each with its own vectors
  static constexpr int kMinTile = 4 * kGroups;               // vectors per tile: four in flight per thread ...
  static constexpr int kMaxTile = 16 * kGroups;              // ... up to sixteen, where the set-up is amortised
  static constexpr int kPerLane = DR / 32;
  static constexpr bool kPrefetch = DR < 128;                // the next tile's vectors in registers during the chains
  static constexpr int kPitch = DR + 4;
  static constexpr size_t kPiBytes = static_cast<size_t>(DR) * kPitch * 4;
  static constexpr size_t kTileBytes = static_cast<size_t>(kMaxTile) * DR * (4 + 1);      // values, codes
  static constexpr size_t kSmem = kPiBytes > kTileBytes ? kPiBytes : kTileBytes;          // (Pi's place is reused)
};

// Rows of Pi into registers: m[j] = Pi[i][j] of this thread's output coordinate i (0 beyond d).
template <int DR>
__device__ __forceinline__ void load_pi_row(const float* __restrict__ Pi, int d, float* stage, int i, float (&m)[DR]) {
  constexpr int P = Shape<DR>::kPitch;
  if (d == DR && (reinterpret_cast<uintptr_t>(Pi) & 15u) == 0) {
    for (int c = threadIdx.x; c < DR * DR / 4; c += kThreads) {
      const int r = c / (DR / 4), q = c % (DR / 4);
      cp_async16(stage + r * P + 4 * q, Pi + r * DR + 4 * q, 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {
    for (int c = threadIdx.x; c < DR * DR; c += kThreads) {
      const int r = c / DR, q = c % DR;
      stage[r * P + q] = (r < d && q < d) ? Pi[r * d + q] : 0.f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < DR / 4; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(stage + i * P + 4 * q);
    m[4 * q] = v.x; m[4 * q + 1] = v.y; m[4 * q + 2] = v.z; m[4 * q + 3] = v.w;
  }
  __syncthreads();                             // the staging area is reused for the tiles
}

// z[k] = sum_j x[k][j] m[j], fp32 FMA in ascending j, for four vectors in rows of DR floats.
template <int DR>
__device__ __forceinline__ void chain4(const float* __restrict__ x, const float (&m)[DR], float (&z)[4]) {
  z[0] = z[1] = z[2] = z[3] = 0.f;
#pragma unroll
  for (int q = 0; q < DR / 4; ++q) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 v = *reinterpret_cast<const float4*>(x + k * DR + 4 * q);
      z[k] = fmaf(v.x, m[4 * q], z[k]);
      z[k] = fmaf(v.y, m[4 * q + 1], z[k]);
      z[k] = fmaf(v.z, m[4 * q + 2], z[k]);
      z[k] = fmaf(v.w, m[4 * q + 3], z[k]);
    }
  }
}

// Stream position of every channel of a mixed row: the outlier channels first (in channel order), then the others.
// slot[i] = position; returns the number of outlier channels.  A CTA-wide call.
__device__ __forceinline__ int build_slots(const uint8_t* is_outlier, int d, uint32_t* words, uint8_t* slot) {
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const bool o = i < d && is_outlier[i] != 0;
  const uint32_t m = __ballot_sync(QKV_FULL_MASK, o);
  if (lane == 0) words[warp] = m;
  __syncthreads();
  int n_out = 0, before = 0;
  for (int w = 0; w < kWarps; ++w) {
    const int c = __popc(words[w]);
    n_out += c;
    if (w < warp) before += c;
  }
  before += __popc(m & ((1u << lane) - 1u));
  if (i < d) slot[i] = static_cast<uint8_t>(o ? before : n_out + (i - before));
  __syncthreads();
  return n_out;
}

// Codes c0 .. of a row (one byte each, `count` of them, at most 32) as `w`-bit fields to dst[0 .. bytes).
__device__ __forceinline__ void pack_store(const uint8_t* codes, int count, int w, uint8_t* dst, int bytes) {
  uint64_t acc = 0;
  int have = 0, done = 0;
  const bool words = (reinterpret_cast<uintptr_t>(dst) & 3u) == 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    uint32_t v = *reinterpret_cast<const uint32_t*>(codes + 4 * q);
    const int left = count - 4 * q;
    if (left < 4) v = left <= 0 ? 0u : v & ((1u << (8 * left)) - 1u);
    const uint32_t f = (v & 15u) | (((v >> 8) & 15u) << w) | (((v >> 16) & 15u) << (2 * w)) | ((v >> 24) << (3 * w));
    acc |= static_cast<uint64_t>(f) << have;
    have += 4 * w;
    if (have >= 32) {
      if (words && done + 4 <= bytes) {
        *reinterpret_cast<uint32_t*>(dst + done) = static_cast<uint32_t>(acc);
      } else {
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (done + b < bytes) dst[done + b] = static_cast<uint8_t>(acc >> (8 * b));
      }
      done += 4;
      acc >>= 32;
      have -= 32;
    }
  }
}

// Block `blk` of a packed row: the first `blocks0` are 32-code blocks of the (outlier) stream, then the regular stream's,
// then 32-bit pieces of the sign plane.  `cs` holds one byte per code in stream order, `ss` per sign in channel order.
__device__ __forceinline__ void store_block(const uint8_t* cs, const uint8_t* ss, int blk, int blocks0, int blocks1,
                                            int n_out, int d, const CompressArgs& a, uint8_t* crow, int seg0_bytes,
                                            int row_bytes, uint8_t* srow, int sign_bytes) {
  if (blk < blocks0) {
    const int off = 4 * blk * a.bits0;
    pack_store(cs + 32 * blk, n_out - 32 * blk, a.bits0, crow + off, seg0_bytes - off);
  } else if (blk < blocks0 + blocks1) {          // the regular stream starts at any byte of `cs` and of the row
    blk -= blocks0;
    const int first = n_out + 32 * blk, count = d - first, off = seg0_bytes + 4 * blk * a.bits1;
    __align__(4) uint8_t tmp[32];
    for (int p = 0; p < 32; ++p) tmp[p] = p < count ? cs[first + p] : 0;
    pack_store(tmp, count, a.bits1, crow + off, row_bytes - off);
  } else {
    blk -= blocks0 + blocks1;
    pack_store(ss + 32 * blk, d - 32 * blk, 1, srow + 4 * blk, sign_bytes - 4 * blk);
  }
}

// Where a lane's channels lane, lane + 32, ... sit in a packed row, and their decoded values.
template <int PER_LANE> struct ChannelFields {
  float sgn[PER_LANE];
  int bitpos[PER_LANE], width[PER_LANE], cls[PER_LANE];
  int row_bytes, sign_bytes;
  __device__ __forceinline__ ChannelFields(const DecompressArgs& a, bool mixed, int n_out, const uint8_t* slot, int lane) {
    const int d = a.d;
    const int seg0_bytes = packed_row_bytes(mixed ? n_out : d, a.bits0);
    row_bytes = mixed ? seg0_bytes + packed_row_bytes(d - n_out, a.bits1) : seg0_bytes;
    sign_bytes = (d + 7) >> 3;
#pragma unroll
    for (int t = 0; t < PER_LANE; ++t) {
      const int j = lane + 32 * t;
      cls[t] = (mixed && j < d && a.is_outlier[j] == 0) ? 1 : 0;
      width[t] = cls[t] ? a.bits1 : a.bits0;
      const int k = (mixed && j < d) ? slot[j] : j;
      bitpos[t] = cls[t] ? 8 * seg0_bytes + (k - n_out) * a.bits1 : k * a.bits0;
      sgn[t] = (a.signs && j < d) ? a.S[j] : 0.f;
    }
  }
  __device__ __forceinline__ uint32_t code(const DecompressArgs& a, int64_t row, int t, int lane) const {
    return a.packed ? read_field(a.codes + row * row_bytes, bitpos[t], width[t], row_bytes) : a.codes[row * a.d + lane + 32 * t];
  }
  __device__ __forceinline__ uint32_t sign(const DecompressArgs& a, int64_t row, int t, int lane) const {
    const int j = lane + 32 * t;
    return a.packed ? ((a.signs[row * sign_bytes + (j >> 3)] >> (j & 7)) & 1u) : a.signs[row * a.d + j];
  }
  __device__ __forceinline__ float sign_term(const DecompressArgs& a, uint32_t sb, int t) const {
    return a.qjl_scale * (sgn[t] * (sb ? 1.f : -1.f));
  }
  __device__ __forceinline__ float value(const DecompressArgs& a, const float (*tab)[16], int64_t row, int t, int lane) const {
    const float y = tab[cls[t]][code(a, row, t, lane) & 15u];
    return a.signs ? y + sign_term(a, sign(a, row, t, lane), t) : y;
  }
};

// 32 codes of one token (coordinates 32 blk ..) into its tile record (tile_format.cuh): 2-bit key codes are whole
// bytes; the values' bits share words with the other token of the pair and are exchanged with atomic AND / OR.
__device__ __forceinline__ void file_key_codes(const uint8_t* codes, uint8_t* rec, int k, int blk) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    w[h] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t v = *reinterpret_cast<const uint32_t*>(codes + 16 * h + 4 * q);
      w[h] |= ((v & 3u) | ((v >> 6) & 0xCu) | ((v >> 12) & 0x30u) | ((v >> 18) & 0xC0u)) << (8 * q);
    }
  }
  *reinterpret_cast<uint2*>(rec + tile::key_code_offset(k, 2 * blk)) = make_uint2(w[0], w[1]);
}
__device__ __forceinline__ void file_value_codes(const uint8_t* codes, uint8_t* rec, int k, int blk) {
  const int hs = tile::val_half_shift(k), grp = tile::val_group(k);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t f[3] = {0u, 0u, 0u};                // the sixteen fields of three bits at a pitch of six
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const uint32_t v = tile::code_to_stored(codes[16 * h + p]);
      f[(6 * p) >> 5] |= v << ((6 * p) & 31);
      if (((6 * p) & 31) > 29) f[((6 * p) >> 5) + 1] |= v >> (32 - ((6 * p) & 31));
    }
    constexpr uint32_t kMask[3] = {0xC71C71C7u, 0x71C71C71u, 0x1C71C71Cu};     // bits 6 p .. 6 p + 2
    const uint32_t bits[3] = {f[0] << hs, __funnelshift_l(f[0], f[1], hs), __funnelshift_l(f[1], f[2], hs)};
    const uint32_t mask[3] = {kMask[0] << hs, __funnelshift_l(kMask[0], kMask[1], hs),
                              __funnelshift_l(kMask[1], kMask[2], hs)};
    const int lane = tile::val_lane(k, 2 * blk + h);
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      uint32_t* word = reinterpret_cast<uint32_t*>(rec + tile::val_word_offset(lane, 3 * grp + w));
      atomicAnd(word, ~mask[w]);
      atomicOr(word, bits[w]);
    }
  }
}

template <int DR>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) compress_small_kernel(ChainArgs args) {
  using Sh = Shape<DR>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float tab_s[2][16], cent_s[2][16];
  __shared__ uint32_t mask_words[kWarps];
  __shared__ uint8_t slot_s[kMaxD];
  __shared__ int64_t row_s[Sh::kMaxTile];
  const bool second = blockIdx.x >= static_cast<unsigned>(args.ctas0);
  const CompressArgs& a = args.job[second ? 1 : 0];
  const int cta = static_cast<int>(blockIdx.x) - (second ? args.ctas0 : 0);
  const int n_cta = second ? static_cast<int>(gridDim.x) - args.ctas0 : args.ctas0;
  const int d = args.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = tid % DR, grp = tid / DR;                     // output coordinate, group of vectors
  const bool active = grp < Sh::kGroups && i < d;             // (DR = 96 leaves a warp without a group)
  const int vt = args.tile_vecs;                              // vectors per tile
  const int per_warp = vt / kWarps;

  // one tile's vectors: warp w takes vectors w, w + 4, ...; a lane its coordinates lane, lane + 32, ...
  float xv[4 * Sh::kGroups][Sh::kPerLane];
  auto load_tile = [&](int64_t v0) {
#pragma unroll
    for (int u = 0; u < 4 * Sh::kGroups; ++u) {
      if (u >= per_warp) break;
      const int64_t n = v0 + warp + kWarps * u;
#pragma unroll
      for (int t = 0; t < Sh::kPerLane; ++t) {
        const int j = lane + 32 * t;
        xv[u][t] = (n < a.n_vec && j < d) ? load_float(a.x, a.x_dtype, n * a.x_pitch + j) : 0.f;
      }
    }
  };
  const int64_t n_tiles = (a.n_vec + vt - 1) / vt;
  int64_t tile = cta;
  if (tile < n_tiles) load_tile(tile * vt);                   // travels with Pi

  const bool mixed = a.mode == MODE_MIXED;
  const bool with_signs = a.mode == MODE_IP || (mixed && a.signs != nullptr);
  const int nb0 = (1 << a.bits0) - 1, nb1 = mixed ? (1 << a.bits1) - 1 : 0;
  if (tid < 16) {
    tab_s[0][tid] = tid < nb0 ? a.bounds0[tid] : INFINITY;
    tab_s[1][tid] = tid < nb1 ? a.bounds1[tid] : INFINITY;
    cent_s[0][tid] = (with_signs && tid <= nb0) ? a.centroids[tid] : 0.f;
    cent_s[1][tid] = (with_signs && mixed && tid <= nb1) ? a.centroids1[tid] : 0.f;
  }
  int n_out = d;
  if (mixed) n_out = build_slots(a.is_outlier, d, mask_words, slot_s);
  if (a.skip_block_aligned && (n_out & 31) == 0) return;      // uniform over the grid: the tcgen05 kernel did it
  const int cls = (mixed && active && a.is_outlier[i] == 0) ? 1 : 0;      // this coordinate's table
  const float sgn = (with_signs && active) ? a.S[i] : 0.f;
  float m[DR];
  load_pi_row<DR>(args.Pi, d, reinterpret_cast<float*>(smem_raw), active ? i : 0, m);

  float* xs = reinterpret_cast<float*>(smem_raw);                                   // [tile][DR]
  uint8_t* cs = smem_raw + static_cast<size_t>(Sh::kMaxTile) * DR * 4;              // [tile][DR] codes in stream order
  const int seg0_bytes = packed_row_bytes(n_out, a.bits0);
  const int row_bytes = mixed ? seg0_bytes + packed_row_bytes(d - n_out, a.bits1) : seg0_bytes;
  const int sign_bytes = (d + 7) >> 3;
  const int cpos = mixed && active ? slot_s[i] : i;           // where this coordinate's code goes in the row

  for (; tile < n_tiles; tile += n_cta) {
    const int64_t v0 = tile * vt;
    // ---- norm (sum of squares in fp64, rounded once), scale, stage ---------------------------------------------
#pragma unroll
    for (int u = 0; u < 4 * Sh::kGroups; ++u) {
      if (u >= per_warp) break;
      const int v = warp + kWarps * u;
      double ss = 0.0;
#pragma unroll
      for (int t = 0; t < Sh::kPerLane; ++t) ss += static_cast<double>(xv[u][t]) * static_cast<double>(xv[u][t]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(QKV_FULL_MASK, ss, o);
      const float norm = fmaxf(static_cast<float>(sqrt(ss)), 1e-8f);
#pragma unroll
      for (int t = 0; t < Sh::kPerLane; ++t) xs[v * DR + lane + 32 * t] = xv[u][t] / norm;
      if (lane == 0) {
        const int64_t n = v0 + v;
        const int64_t row = n < a.n_vec ? chain_row(args, a, n) : -1;
        row_s[v] = row;
        if (row < 0 && n < a.n_vec && !second) atomicAdd(&g_rows_dropped, 1ull);
        if (row >= 0) {
          if (args.records) {
            float* nd = reinterpret_cast<float*>(args.records + (row >> 4) * tile::kBytes +
                                                 (second ? tile::val_norm_offset(row & 15) : tile::key_norm_offset(row & 15)));
            *nd = norm;
          } else {
            a.norms[row] = norm;
          }
        }
      }
    }
    __syncthreads();
    if (Sh::kPrefetch && tile + n_cta < n_tiles) load_tile((tile + n_cta) * vt);    // travels during the chains
    // ---- rotate, bucketise, sign bit ---------------------------------------------------------------------------
    for (int vb = 4 * grp; vb < vt && grp < Sh::kGroups; vb += Sh::kMinTile) {
      float z[4];
      chain4<DR>(xs + vb * DR, m, z);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int v = vb + k;
        const float y = z[k];
        const float* tab = tab_s[cls];
        uint32_t c = 0;                          // boundaries below y: bisection over the (ascending) 15-entry table
        c += y > tab[c + 7] ? 8u : 0u;
        c += y > tab[c + 3] ? 4u : 0u;
        c += y > tab[c + 1] ? 2u : 0u;
        c += y > tab[c] ? 1u : 0u;
        const uint32_t sb = (y - cent_s[cls][c]) * sgn >= 0.f ? 1u : 0u;
        const int64_t row = row_s[v];
        if (a.packed) {
          if (active) cs[v * DR + cpos] = static_cast<uint8_t>(c);
          if (with_signs) {                      // a warp holds 32 neighbouring coordinates of one vector
            const uint32_t w = __ballot_sync(QKV_FULL_MASK, active && sb);
            if (lane == 0 && row >= 0 && (i & ~31) < d) {
              if (args.records) {
                *reinterpret_cast<uint32_t*>(args.records + (row >> 4) * tile::kBytes +
                                             tile::key_sign_offset(row & 15, i >> 5)) = w;
              } else {
                uint8_t* dst = a.signs + row * sign_bytes + (i >> 3);
                if (i + 32 <= d && (reinterpret_cast<uintptr_t>(dst) & 3u) == 0) *reinterpret_cast<uint32_t*>(dst) = w;
                else
                  for (int b = 0; b < 4 && (i >> 3) + b < sign_bytes; ++b) dst[b] = static_cast<uint8_t>(w >> (8 * b));
              }
            }
          }
        } else if (active && row >= 0) {         // one byte per coordinate: 32 bytes of a row per warp and store
          a.codes[row * d + i] = static_cast<uint8_t>(c);
          if (with_signs) a.signs[row * d + i] = static_cast<uint8_t>(sb);
        }
      }
    }
    __syncthreads();
    // ---- pack 32 codes per thread and store them ---------------------------------------------------------------
    if (a.packed) {
      const int blocks0 = (n_out + 31) >> 5, blocks1 = mixed ? (d - n_out + 31) >> 5 : 0;
      const int per_row = blocks0 + blocks1;
      for (int it = tid; it < vt * per_row; it += kThreads) {
        const int v = it / per_row;
        const int blk = it - v * per_row;
        const int64_t row = row_s[v];
        if (row < 0) continue;
        const uint8_t* crow = cs + v * DR;
        if (args.records) {
          uint8_t* rec = args.records + (row >> 4) * tile::kBytes;
          if (second) file_value_codes(crow + 32 * blk, rec, static_cast<int>(row & 15), blk);
          else file_key_codes(crow + 32 * blk, rec, static_cast<int>(row & 15), blk);
        } else {
          store_block(crow, nullptr, blk, blocks0, blocks1, n_out, d, a, a.codes + row * row_bytes, seg0_bytes, row_bytes,
                      nullptr, 0);
        }
      }
    }
    if (!Sh::kPrefetch && tile + n_cta < n_tiles) load_tile((tile + n_cta) * vt);
    __syncthreads();
  }
}

template <int DR>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) decompress_small_kernel(DecompressArgs a, int vt) {
  using Sh = Shape<DR>;
  __shared__ __align__(16) float ys[Sh::kMaxTile * DR];
  __shared__ float tab_s[2][16], nrm_s[Sh::kMaxTile];
  __shared__ uint32_t mask_words[kWarps];
  __shared__ uint8_t slot_s[kMaxD];
  const int d = a.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = tid % DR, grp = tid / DR;
  const bool active = grp < Sh::kGroups && i < d;
  const bool mixed = a.mode == MODE_MIXED;
  int n_out = 0;
  if (mixed) n_out = build_slots(a.is_outlier, d, mask_words, slot_s);
  if (a.skip_block_aligned && (n_out & 31) == 0) return;      // uniform over the grid: the tcgen05 kernel did it
  // column i of Pi: neighbouring threads read neighbouring words, all loads in flight
  float m[DR];
#pragma unroll
  for (int j = 0; j < DR; ++j) m[j] = (active && j < d) ? __ldg(a.Pi + j * d + i) : 0.f;
  if (tid < 16) {
    tab_s[0][tid] = tid < (1 << a.bits0) ? a.cents0[tid] : 0.f;
    tab_s[1][tid] = (mixed && tid < (1 << a.bits1)) ? a.cents1[tid] : 0.f;
  }
  const ChannelFields<Sh::kPerLane> ch(a, mixed, n_out, slot_s, lane);
  __syncthreads();
  const int64_t n_tiles = (a.n_vec + vt - 1) / vt;
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t v0 = tile * vt;
#pragma unroll (DR < 96 ? 4 : 2)
    for (int v = warp; v < vt; v += kWarps) {
      const int64_t n = v0 + v;
      const bool live = n < a.n_vec;
      const int64_t row = live ? map_row(a.rows, n) : 0;
#pragma unroll
      for (int t = 0; t < Sh::kPerLane; ++t) {
        const int j = lane + 32 * t;
        ys[v * DR + j] = (live && j < d) ? ch.value(a, tab_s, row, t, lane) : 0.f;
      }
      if (lane == 0) nrm_s[v] = live ? a.norms[row] : 0.f;
    }
    __syncthreads();
    for (int vb = 4 * grp; vb < vt && grp < Sh::kGroups; vb += Sh::kMinTile) {
      float z[4];
      chain4<DR>(ys + vb * DR, m, z);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t n = v0 + vb + k;
        if (active && n < a.n_vec) store_float(a.out, a.out_dtype, n * a.out_pitch + i, z[k] * nrm_s[vb + k]);
      }
    }
    __syncthreads();
  }
}

// ---- bulk: 8 coordinates x 8 vectors per thread ---------------------------------------------------------------------

template <int DR> struct Bulk {
  static constexpr int kCols = DR / 8;                       // threads along the coordinates
  static constexpr int kRowsT = kThreads / kCols;            // threads along the vectors (DR = 96: ten, 120 threads work)
  static constexpr int kTile = 8 * kRowsT;                   // vectors per tile
  static constexpr int kPitch = kTile + 4;
  static constexpr size_t kMatBytes = static_cast<size_t>(DR) * DR * 4;
  static constexpr size_t kXBytes = static_cast<size_t>(DR) * kPitch * 4;
  static constexpr size_t kCodeBytes = 2 * static_cast<size_t>(kTile) * DR;      // codes, sign bits: in x's place
  static constexpr size_t kSmem = kMatBytes + (kXBytes > kCodeBytes ? kXBytes : kCodeBytes);
  static constexpr int kPerLane = DR / 32;
  // Resident CTAs per SM, as shared memory (50 KB at 64 coordinates, 98 KB at 128) and 128 to 255 registers allow.
  static constexpr int kCtas = DR == 128 ? 2 : (DR == 96 ? 3 : 4);
};

// Word (j, i) of the matrix: groups of four coordinates exchanged with the row so that the transposing writes of a warp
// (eight coordinates x four rows) meet no bank twice; rows stay whole float4s.
template <int DR> __device__ __forceinline__ int mat_at(int j, int i) { return j * DR + (i ^ (8 * ((j >> 2) & 3))); }

// acc[v][c] = sum_j x[j][8 vy + v] mat[j][coordinate c], ascending j.
template <int DR>
__device__ __forceinline__ void bulk_chains(const float* __restrict__ mat, const float* __restrict__ xs, int cx, int vy,
                                            float (&acc)[8][8]) {
#pragma unroll
  for (int v = 0; v < 8; ++v)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[v][c] = 0.f;
#pragma unroll 4
  for (int j = 0; j < DR; ++j) {
    const float4 p0 = *reinterpret_cast<const float4*>(mat + mat_at<DR>(j, 4 * cx));
    const float4 p1 = *reinterpret_cast<const float4*>(mat + mat_at<DR>(j, DR / 2 + 4 * cx));
    const float4 x0 = *reinterpret_cast<const float4*>(xs + j * Bulk<DR>::kPitch + 8 * vy);
    const float4 x1 = *reinterpret_cast<const float4*>(xs + j * Bulk<DR>::kPitch + 8 * vy + 4);
    const float m[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
    const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
    for (int v = 0; v < 8; ++v)
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[v][c] = fmaf(x[v], m[c], acc[v][c]);
  }
}

// Four vectors n0 .. of a warp, a lane its coordinates lane, lane + 32, ...: all loads in flight before the first use.
template <int PL, typename T>
__device__ __forceinline__ void load_four(const T* __restrict__ x, int64_t pitch, int64_t n0, int64_t n_vec, int d, int lane,
                                          float (&xv)[4][PL]) {
  T v[4][PL];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int t = 0; t < PL; ++t) {
      const int j = lane + 32 * t;
      v[u][t] = (n0 + u < n_vec && j < d) ? x[(n0 + u) * pitch + j] : T(0.f);
    }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int t = 0; t < PL; ++t) xv[u][t] = static_cast<float>(v[u][t]);
}

// PAIR: both jobs of an append, by blockIdx.y.  (One job by itself reads its arguments at fixed addresses: 2 us of 37 at
// 20000 vectors of 64 coordinates.)
template <int DR, bool PAIR>
__global__ void __launch_bounds__(kThreads, Bulk<DR>::kCtas) compress_bulk_kernel(ChainArgs args) {
  using B = Bulk<DR>;
  const CompressArgs& a = args.job[PAIR ? blockIdx.y : 0];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float tab_s[2][16], cent_s[2][16], sgn_s[kMaxD];
  __shared__ uint32_t mask_words[kWarps];
  __shared__ uint8_t slot_s[kMaxD], cls_s[kMaxD];
  __shared__ int64_t row_s[B::kTile];
  float* mat = reinterpret_cast<float*>(smem_raw);
  float* xs = reinterpret_cast<float*>(smem_raw + B::kMatBytes);
  uint8_t* cs = smem_raw + B::kMatBytes;                      // [tile][DR] codes in stream order (x is done with by then)
  uint8_t* ss = cs + B::kTile * DR;                           // [tile][DR] sign bits in channel order
  const int d = a.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cx = tid % B::kCols, vy = tid / B::kCols;
  const bool mixed = a.mode == MODE_MIXED;
  const bool with_signs = a.mode == MODE_IP || (mixed && a.signs != nullptr);
  const int nb0 = (1 << a.bits0) - 1, nb1 = mixed ? (1 << a.bits1) - 1 : 0;
  if (tid < 16) {
    tab_s[0][tid] = tid < nb0 ? a.bounds0[tid] : INFINITY;
    tab_s[1][tid] = tid < nb1 ? a.bounds1[tid] : INFINITY;
    cent_s[0][tid] = (with_signs && tid <= nb0) ? a.centroids[tid] : 0.f;
    cent_s[1][tid] = (with_signs && mixed && tid <= nb1) ? a.centroids1[tid] : 0.f;
  }
  slot_s[tid] = static_cast<uint8_t>(tid);
  cls_s[tid] = (mixed && tid < d && a.is_outlier[tid] == 0) ? 1 : 0;
  sgn_s[tid] = (with_signs && tid < d) ? a.S[tid] : 0.f;
  int n_out = d;
  if (mixed) n_out = build_slots(a.is_outlier, d, mask_words, slot_s);
  if (a.skip_block_aligned && (n_out & 31) == 0) return;      // uniform over the grid: the tcgen05 kernel did it
  for (int c = tid; c < DR * DR; c += kThreads) {             // lanes: four neighbouring j of eight coordinates
    const int j = 4 * ((c >> 5) % (DR / 4)) + (c & 3), i = 8 * (c / (8 * DR)) + ((c >> 2) & 7);
    mat[mat_at<DR>(j, i)] = (i < d && j < d) ? __ldg(a.Pi + i * d + j) : 0.f;
  }
  __syncthreads();
  const int seg0_bytes = packed_row_bytes(n_out, a.bits0);
  const int row_bytes = mixed ? seg0_bytes + packed_row_bytes(d - n_out, a.bits1) : seg0_bytes;
  const int sign_bytes = (d + 7) >> 3;
  const int64_t n_tiles = (a.n_vec + B::kTile - 1) / B::kTile;
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t v0 = tile * B::kTile;
    // norm (sum of squares in fp64, rounded once), scale, stage transposed; a warp's vectors four at a time
    for (int u0 = 4 * warp; u0 < B::kTile; u0 += 4 * kWarps) {
      float xv[4][B::kPerLane];
      if (a.x_dtype == QKV_F32) load_four(static_cast<const float*>(a.x), a.x_pitch, v0 + u0, a.n_vec, d, lane, xv);
      else if (a.x_dtype == QKV_BF16) load_four(static_cast<const __nv_bfloat16*>(a.x), a.x_pitch, v0 + u0, a.n_vec, d, lane, xv);
      else load_four(static_cast<const __half*>(a.x), a.x_pitch, v0 + u0, a.n_vec, d, lane, xv);
      float norm[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double ss2 = 0.0;
#pragma unroll
        for (int t = 0; t < B::kPerLane; ++t) ss2 += static_cast<double>(xv[u][t]) * static_cast<double>(xv[u][t]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss2 += __shfl_xor_sync(QKV_FULL_MASK, ss2, o);
        norm[u] = fmaxf(static_cast<float>(sqrt(ss2)), 1e-8f);
      }
#pragma unroll
      for (int t = 0; t < B::kPerLane; ++t)
        *reinterpret_cast<float4*>(xs + (lane + 32 * t) * B::kPitch + u0) =
            make_float4(xv[0][t] / norm[0], xv[1][t] / norm[1], xv[2][t] / norm[2], xv[3][t] / norm[3]);
      if (lane < 4) {
        const int64_t n = v0 + u0 + lane;
        const int64_t row = n < a.n_vec ? (PAIR ? chain_row(args, a, n) : map_row(a.rows, n)) : -1;
        if (PAIR && row < 0 && n < a.n_vec && blockIdx.y == 0) atomicAdd(&g_rows_dropped, 1ull);
        row_s[u0 + lane] = row;
        if (row >= 0) a.norms[row] = lane == 0 ? norm[0] : (lane == 1 ? norm[1] : (lane == 2 ? norm[2] : norm[3]));
      }
    }
    __syncthreads();
    float acc[8][8];
    if (vy < B::kRowsT) bulk_chains<DR>(mat, xs, cx, vy, acc);
    __syncthreads();                                          // x has been read: codes take its place
    if (vy < B::kRowsT) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int i = (c < 4 ? 4 * cx : DR / 2 + 4 * cx - 4) + c;
        const int cls = cls_s[i], pos = a.packed ? slot_s[i] : i;
        const float* tab = tab_s[cls];
        const float sgn = sgn_s[i];
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const float y = acc[v][c];
          uint32_t k = 0;                        // boundaries below y: bisection over the (ascending) 15-entry table
          k += y > tab[k + 7] ? 8u : 0u;
          k += y > tab[k + 3] ? 4u : 0u;
          k += y > tab[k + 1] ? 2u : 0u;
          k += y > tab[k] ? 1u : 0u;
          cs[(8 * vy + v) * DR + pos] = static_cast<uint8_t>(k);
          if (with_signs) ss[(8 * vy + v) * DR + i] = (y - cent_s[cls][k]) * sgn >= 0.f ? 1 : 0;
        }
      }
    }
    __syncthreads();
    const bool whole16 = (d & 15) == 0 &&
        ((reinterpret_cast<uintptr_t>(a.codes) | reinterpret_cast<uintptr_t>(a.signs)) & 15u) == 0;
    if (!a.packed && whole16) {
      const int per_row = d >> 4;
      for (int it = tid; it < B::kTile * per_row; it += kThreads) {
        const int v = it / per_row, c16 = 16 * (it - v * per_row);
        const int64_t row = row_s[v];
        if (row < 0) continue;
        *reinterpret_cast<uint4*>(a.codes + row * d + c16) = *reinterpret_cast<const uint4*>(cs + v * DR + c16);
        if (with_signs) *reinterpret_cast<uint4*>(a.signs + row * d + c16) = *reinterpret_cast<const uint4*>(ss + v * DR + c16);
      }
    } else if (!a.packed) {                      // one byte per coordinate, channel order
      for (int it = tid; it < B::kTile * d; it += kThreads) {
        const int v = it / d, i = it - v * d;
        const int64_t row = row_s[v];
        if (row < 0) continue;
        a.codes[row * d + i] = cs[v * DR + i];
        if (with_signs) a.signs[row * d + i] = ss[v * DR + i];
      }
    } else {
      const int blocks0 = (n_out + 31) >> 5, blocks1 = mixed ? (d - n_out + 31) >> 5 : 0;
      const int blocks_s = with_signs ? (d + 31) >> 5 : 0;
      const int per_row = blocks0 + blocks1 + blocks_s;
      for (int it = tid; it < B::kTile * per_row; it += kThreads) {
        const int v = it / per_row;
        const int64_t row = row_s[v];
        if (row >= 0) store_block(cs + v * DR, ss + v * DR, it - v * per_row, blocks0, blocks1, n_out, d, a,
                                  a.codes + row * row_bytes, seg0_bytes, row_bytes,
                                  with_signs ? a.signs + row * sign_bytes : nullptr, sign_bytes);
      }
    }
    __syncthreads();
  }
}

template <int DR>
__global__ void __launch_bounds__(kThreads, Bulk<DR>::kCtas) decompress_bulk_kernel(DecompressArgs a) {
  using B = Bulk<DR>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float tab_s[2][16], nrm_s[B::kTile];
  __shared__ uint32_t mask_words[kWarps];
  __shared__ uint8_t slot_s[kMaxD];
  float* mat = reinterpret_cast<float*>(smem_raw);
  float* ys = reinterpret_cast<float*>(smem_raw + B::kMatBytes);
  const int d = a.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cx = tid % B::kCols, vy = tid / B::kCols;
  const bool mixed = a.mode == MODE_MIXED;
  int n_out = 0;
  if (mixed) n_out = build_slots(a.is_outlier, d, mask_words, slot_s);
  if (a.skip_block_aligned && (n_out & 31) == 0) return;      // uniform over the grid: the tcgen05 kernel did it
  if (tid < 16) {
    tab_s[0][tid] = tid < (1 << a.bits0) ? a.cents0[tid] : 0.f;
    tab_s[1][tid] = (mixed && tid < (1 << a.bits1)) ? a.cents1[tid] : 0.f;
  }
  for (int c = tid; c < DR * DR; c += kThreads) {
    const int j = c / DR, i = c % DR;
    mat[mat_at<DR>(j, i)] = (i < d && j < d) ? __ldg(a.Pi + j * d + i) : 0.f;
  }
  ChannelFields<B::kPerLane> ch(a, mixed, n_out, slot_s, lane);
  __syncthreads();
  const int64_t n_tiles = (a.n_vec + B::kTile - 1) / B::kTile;
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t v0 = tile * B::kTile;
    for (int u0 = 4 * warp; u0 < B::kTile; u0 += 4 * kWarps) {
      float y[4][B::kPerLane];
      int64_t row[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t n = v0 + u0 + u;
        row[u] = n < a.n_vec ? (n < a.rows.seg_len ? a.rows.seg_off + n : map_row(a.rows, n)) : -1;     // (one segment: no division)
        if (lane == u) nrm_s[u0 + u] = row[u] >= 0 ? a.norms[row[u]] : 0.f;
      }
      uint32_t c[4][B::kPerLane];                // codes of all four vectors before their look-ups
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int t = 0; t < B::kPerLane; ++t) c[u][t] = (row[u] >= 0 && lane + 32 * t < d) ? ch.code(a, row[u], t, lane) : 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int t = 0; t < B::kPerLane; ++t)
          y[u][t] = (row[u] >= 0 && lane + 32 * t < d) ? tab_s[ch.cls[t]][c[u][t] & 15u] : 0.f;
      if (a.signs) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int t = 0; t < B::kPerLane; ++t)
            if (row[u] >= 0 && lane + 32 * t < d) y[u][t] += ch.sign_term(a, ch.sign(a, row[u], t, lane), t);
      }
#pragma unroll
      for (int t = 0; t < B::kPerLane; ++t)
        *reinterpret_cast<float4*>(ys + (lane + 32 * t) * B::kPitch + u0) =
            make_float4(y[0][t], y[1][t], y[2][t], y[3][t]);
    }
    __syncthreads();
    if (vy < B::kRowsT) {
      float acc[8][8];
      bulk_chains<DR>(mat, ys, cx, vy, acc);
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const int64_t n = v0 + 8 * vy + v;
        if (n >= a.n_vec) break;
        const float nrm = nrm_s[8 * vy + v];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i0 = (h ? DR / 2 : 0) + 4 * cx;
          const int64_t at = n * a.out_pitch + i0;
          const float* z = &acc[v][4 * h];
          if (a.out_dtype == QKV_F32 && i0 + 4 <= d && ((at | (reinterpret_cast<uintptr_t>(a.out) >> 2)) & 3) == 0) {
            reinterpret_cast<float4*>(a.out)[at >> 2] = make_float4(z[0] * nrm, z[1] * nrm, z[2] * nrm, z[3] * nrm);
          } else if (a.out_dtype == QKV_BF16 && i0 + 4 <= d && ((at | (reinterpret_cast<uintptr_t>(a.out) >> 1)) & 3) == 0) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(z[0] * nrm, z[1] * nrm), hi = __floats2bfloat162_rn(z[2] * nrm, z[3] * nrm);
            reinterpret_cast<uint2*>(a.out)[at >> 2] =
                make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (i0 + c < d) store_float(a.out, a.out_dtype, at + c, z[c] * nrm);
          }
        }
      }
    }
    __syncthreads();
  }
}

// Vectors per tile and CTAs for n vectors: the smallest tile that still fits the grid into one round of resident CTAs.
template <int DR>
void plan(int64_t n, int ctas_max, int& vt, int& ctas) {
  using Sh = Shape<DR>;
  int64_t want = (n + ctas_max - 1) / ctas_max;
  want = (want + Sh::kMinTile - 1) / Sh::kMinTile * Sh::kMinTile;
  vt = static_cast<int>(want > Sh::kMaxTile ? Sh::kMaxTile : (want < Sh::kMinTile ? Sh::kMinTile : want));
  const int64_t tiles = (n + vt - 1) / vt;
  ctas = static_cast<int>(tiles < ctas_max ? tiles : ctas_max);
}

// From how many vectors (of both jobs) on the bulk kernels are the faster ones: they need a CTA's worth of 64 vectors or
// more on most SMs before their FMA rate counts.  Append of 2 x 16384 vectors of 32 / 64 coordinates: 40 / 61 us in the
// small kernel, 35 / 38 in bulk; of 2 x 4096 of 64, below the line: 19 against 25.
template <int DR> constexpr int64_t bulk_from() { return static_cast<int64_t>(Bulk<DR>::kTile) * kNumSMs / 2; }

template <typename K>
int set_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess
             ? QKV_OK : QKV_ELAUNCH;
}

template <int DR>
int bulk_grid(int64_t n) {
  const int64_t tiles = (n + Bulk<DR>::kTile - 1) / Bulk<DR>::kTile;
  return static_cast<int>(tiles < Bulk<DR>::kCtas * kNumSMs ? tiles : Bulk<DR>::kCtas * kNumSMs);
}

template <int DR>
int launch_compress_t(ChainArgs& args, cudaStream_t st) {
  const int jobs = args.job[1].n_vec > 0 ? 2 : 1;
  if (jobs * args.job[0].n_vec >= bulk_from<DR>() && !args.records) {      // (records: the small kernel alone writes them)
    const auto kernel = jobs == 2 ? compress_bulk_kernel<DR, true> : compress_bulk_kernel<DR, false>;
    if (set_smem(kernel, Bulk<DR>::kSmem)) return QKV_ELAUNCH;
    kernel<<<dim3(bulk_grid<DR>(args.job[0].n_vec), jobs), kThreads, Bulk<DR>::kSmem, st>>>(args);
    return check_launch();
  }
  int ctas = 0;
  plan<DR>(args.job[0].n_vec, kNumSMs * kCtasPerSm / jobs, args.tile_vecs, ctas);
  args.ctas0 = ctas;
  if (set_smem(compress_small_kernel<DR>, Shape<DR>::kSmem)) return QKV_ELAUNCH;
  compress_small_kernel<DR><<<jobs * ctas, kThreads, Shape<DR>::kSmem, st>>>(args);
  return check_launch();
}

template <int DR>
int launch_decompress_t(const DecompressArgs& a, cudaStream_t st) {
  if (a.n_vec >= bulk_from<DR>()) {
    if (set_smem(decompress_bulk_kernel<DR>, Bulk<DR>::kSmem)) return QKV_ELAUNCH;
    decompress_bulk_kernel<DR><<<bulk_grid<DR>(a.n_vec), kThreads, Bulk<DR>::kSmem, st>>>(a);
    return check_launch();
  }
  int vt = 0, ctas = 0;
  plan<DR>(a.n_vec, kNumSMs * kCtasPerSm, vt, ctas);
  decompress_small_kernel<DR><<<ctas, kThreads, 0, st>>>(a, vt);
  return check_launch();
}

}  // namespace

unsigned long long chain_rows_dropped() {
  unsigned long long v = 0;
  cudaMemcpyFromSymbol(&v, g_rows_dropped, sizeof(v));
  return v;
}

int launch_compress_chain(ChainArgs& args, cudaStream_t st) {
  switch ((args.d + 31) / 32) {
    case 1: return launch_compress_t<32>(args, st);
    case 2: return launch_compress_t<64>(args, st);
    case 3: return launch_compress_t<96>(args, st);
    default: return launch_compress_t<128>(args, st);
  }
}

int launch_decompress_chain(const DecompressArgs& a, cudaStream_t st) {
  switch ((a.d + 31) / 32) {
    case 1: return launch_decompress_t<32>(a, st);
    case 2: return launch_decompress_t<64>(a, st);
    case 3: return launch_decompress_t<96>(a, st);
    default: return launch_decompress_t<128>(a, st);
  }
}

}  // namespace qkv
