// Argument blocks shared by the CUDA-core and the tensor-core rotation kernels.
#pragma once

#include "common.cuh"

namespace qkv {

// d = 128: from how many vectors on the tcgen05 kernels are the faster ones.  Their set-up (three bf16 planes of Pi,
// bucket table) takes as long as the fp32 chain needs for the first tens of thousands.
constexpr int64_t kTensorCoreVectors = 6144;
constexpr int64_t kAppendTensorCore = 6144;      // ... of keys (and as many values) of one append

enum { MODE_MSE = 0, MODE_IP = 1, MODE_MIXED = 2 };

struct CompressArgs {
  const void* x; int x_dtype; int64_t x_pitch; int64_t n_vec; int d;
  const float* Pi;
  int mode;
  const float* bounds0; int bits0;     // uniform / outlier table
  const float* bounds1; int bits1;     // regular table (mixed)
  const float* centroids;              // sign stage: centroids of table 0
  const float* centroids1;             // sign stage of the mixed mode: centroids of table 1
  const float* S;                      // sign stage (IP mode, or mixed mode with signs != nullptr)
  const uint8_t* is_outlier;           // mixed
  uint8_t* codes; uint8_t* signs; int packed; float* norms;
  qkv_rows_t rows;
  int skip_block_aligned;              // mixed, CUDA-core kernel: return if the outlier count is a multiple of 32
                                       // (the tcgen05 kernel launched before it took that case)
  int test_drop_mma;                   // test hook of the tcgen05 kernel: CTA 0 issues nothing for its second
                                       // tile, so the bounded wait on that accumulator runs out (nothing is left
                                       // in flight) and the CTA finishes with the fp32 chain
};

// One launch of the fp32-chain kernel (rotate_chain.cu): one job, or the keys (job 0, MODE_IP) and the values (job 1,
// MODE_MSE) of an append, which then share the destination below.
struct ChainArgs {
  CompressArgs job[2];                 // job[1].n_vec == 0: one job
  int d; const float* Pi;
  int ctas0, tile_vecs;                // CTAs of job 0, vectors per tile (set by the launcher)
  uint8_t* records;                    // tile records instead of the jobs' planes (keys and values of a d = 128, 3/3-bit cache)
  // Paged destination (block_table != nullptr): vector n is token n % tokens of head (n / tokens) % heads of sequence
  // n / (heads * tokens), at position start_lens[sequence] + token of its pages; else the jobs' row maps hold.
  const int32_t* block_table; const int32_t* start_lens;
  int max_blocks, block_size, heads, tokens;
};

// Row (token slot) of vector n; -1 for a position outside its sequence's block table.
__device__ __forceinline__ int64_t paged_row(const int32_t* block_table, const int32_t* start_lens, int max_blocks,
                                             int block_size, int heads, int tokens, int64_t n) {
  const unsigned sh = static_cast<unsigned>(n / tokens), t = static_cast<unsigned>(n % tokens);
  const unsigned seq = sh / static_cast<unsigned>(heads), head = sh % static_cast<unsigned>(heads);
  const int64_t pos = static_cast<int64_t>(start_lens[seq]) + t;
  const int64_t entry = pos / block_size;
  if (pos < 0 || entry >= max_blocks) return -1;
  const int64_t blk = block_table[static_cast<int64_t>(seq) * max_blocks + entry];
  return (blk * heads + head) * block_size + pos % block_size;
}
__device__ __forceinline__ int64_t chain_row(const ChainArgs& c, const CompressArgs& a, int64_t n) {
  if (c.block_table)
    return paged_row(c.block_table, c.start_lens, c.max_blocks, c.block_size, c.heads, c.tokens, n);
  return map_row(a.rows, n);
}

struct DecompressArgs {
  const uint8_t* codes; const uint8_t* signs; int packed; const float* norms;
  qkv_rows_t rows; int64_t n_vec; int d;
  const float* Pi;
  int mode;                            // MODE_MSE (signs may be set) or MODE_MIXED
  const float* cents0; int bits0;
  const float* cents1; int bits1;
  const uint8_t* is_outlier;
  const float* S; float qjl_scale;
  void* out; int out_dtype; int64_t out_pitch;
  int skip_block_aligned;              // mixed, CUDA-core kernel: return if the outlier count is a multiple of 32
  int test_drop_mma;                   // test hook of the tcgen05 kernel: CTA 0 issues nothing for its second tile, so
                                       // the bounded wait on that accumulator runs out (nothing is left in flight)
                                       // and the CTA finishes with the fp32 chain
};


// fp32 FMA chains on the CUDA cores (rotate_chain.cu): any dimension up to 128, any width and layout.
int launch_compress_chain(ChainArgs& args, cudaStream_t st);
int launch_decompress_chain(const DecompressArgs& a, cudaStream_t st);
unsigned long long chain_rows_dropped();              // rows of paged appends that had no slot (device-wide counter)
bool compress_prefers_chain(const CompressArgs& a);   // rotate_quant.cu: the dispatch rule
// tcgen05 rotation (rotate_umma.cu, decompress_umma.cu): d == 128, packed rows.
bool compress_umma_ok(const CompressArgs& a);
int launch_compress_umma(const CompressArgs& a, cudaStream_t st);
bool decompress_umma_ok(const DecompressArgs& a);
int launch_decompress_umma(const DecompressArgs& a, cudaStream_t st);
unsigned int umma_timeouts();             // bounded waits on the tensor core that ran out (device-wide counter)

}  // namespace qkv
