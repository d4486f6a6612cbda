// The launches of one pre-norm block of the serving precision in one call: RMSNorm, q/k/v product with rotation and cache
// write, attention, output product, RMSNorm, SwiGLU feed-forward (src/model.cpp:281-305), by the entry points of this library
// and of the attention library of the block's head size, chosen exactly as the parts choose them one by one.
//
// For steps that are not replayed as a graph (prompt portions beside single tokens): eight to ten calls from Python a layer,
// each with its checks and conversions, took the host about 100 us, more than the layer's kernels at the SmolLM2-360M shape.
#include "bw_common.cuh"

BW_API int bw_bf16_rmsnorm(const float* x, const float* weight, __nv_bfloat16* y, const int* rows, int n, int width, float eps,
                           cudaStream_t stream);
BW_API int bw_bf16_rope_cache(__nv_bfloat16* qkv, int row_stride, const int* pos, const int* row_seq, const float* cos_t,
                              const float* sin_t, const int* block_table, int max_blocks, __nv_bfloat16* kcache,
                              __nv_bfloat16* vcache, int n, int heads, int kv_heads, int hd, int page, int write_kv,
                              cudaStream_t stream);
BW_API int bw_bf16_swiglu(const __nv_bfloat16* gate_up, __nv_bfloat16* out, int n, int inter, cudaStream_t stream);
BW_API int bw_bf16_linear(const __nv_bfloat16* x, const __nv_bfloat16* w, void* y, int y_is_f32, const float* residual, int m, int n,
                          int k, float* partials, int* counters, int use_legacy, cudaStream_t stream);
BW_API int bw_bf16_linear_tc_swiglu(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* h, int m, int n, int k,
                                    float* partials, int act, cudaStream_t stream);
BW_API int bw_bf16_linear_tc_kernels(int m, int n, int k, int swiglu, int has_scratch);
BW_API int bw_bf16_linear_split_rows();
BW_API int bw_bf16_linear_rows_rope_usable(const void* x, const void* w, int m, int n, int k, int heads, int kv_heads, int hd);
BW_API int bw_bf16_linear_rows_rope(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* qkv, int m, int n, int k,
                                    const int* pos, const int* row_seq, const float* cos_t, const float* sin_t,
                                    const int* block_table, int max_blocks, __nv_bfloat16* kcache, __nv_bfloat16* vcache, int heads,
                                    int kv_heads, int hd, int page, int write_kv, float* partials, cudaStream_t stream);
BW_API int bw_bf16_linear_rows_norm_usable(const void* w, int m, int n, int width);
BW_API int bw_bf16_linear_rows_norm_rope(const float* x, const float* norm, float eps, const __nv_bfloat16* w, __nv_bfloat16* qkv, int m, int n,
                                         int k, const int* pos, const int* row_seq, const float* cos_t, const float* sin_t,
                                         const int* block_table, int max_blocks, __nv_bfloat16* kcache, __nv_bfloat16* vcache, int heads,
                                         int kv_heads, int hd, int page, int write_kv, cudaStream_t stream);
BW_API int bw_bf16_linear_rows_norm_swiglu(const float* x, const float* norm, float eps, const __nv_bfloat16* w, __nv_bfloat16* h, int m, int n,
                                           int k, int act, cudaStream_t stream);

namespace {

// Every member is eight bytes: the caller fills an array of 64-bit integers in this order.
struct BlockCall {
  // the stream of rows, and buffers of the step
  float* x;
  __nv_bfloat16 *normed, *qkv, *attn, *h, *gate_up;
  float* partials;
  int* counters;
  float* attn_scratch;
  // the block
  const float *norm1, *norm2;
  const __nv_bfloat16 *w_qkv, *w_o, *w_gate_up, *w_down;
  long long fused_glu, width, heads, kv_heads, hd, inter, window;
  const float *cos_t, *sin_t;
  // its cache
  __nv_bfloat16 *k, *v;
  long long num_pages, page, writable;
  const int* block_table;
  long long max_blocks;
  // the step
  long long n, max_keys;
  const int *pos, *row_seq, *seq_pos0, *seq_row0;
  const int *tile_seq, *tile_row0, *tile_rows;  // query tiles of the mma.sync kernels
  long long tiles, tc_rows;                     // and, where the step has them, of the tcgen05 kernel: rows per tile
  const int *tc_seq, *tc_row0, *tc_tile_rows;
  long long tc_tiles;
  // the attention library
  int (*attention)(const __nv_bfloat16*, int, const __nv_bfloat16*, const __nv_bfloat16*, const int*, int, const int*, const int*,
                   const int*, int, const int*, const int*, const int*, const int*, __nv_bfloat16*, int, int, int, int, int, int,
                   int, float, int, float*, cudaStream_t);
  int (*attention_tc)(const __nv_bfloat16*, int, const __nv_bfloat16*, const __nv_bfloat16*, int, const int*, int, const int*,
                      const int*, const int*, int, const int*, const int*, __nv_bfloat16*, int, int, int, int, int, int, int, float,
                      cudaStream_t);
  int (*attention_tc_rows)(int, int, int, int, int);
  int (*attention_stream)(const __nv_bfloat16*, int, const __nv_bfloat16*, const __nv_bfloat16*, int, const int*, int, const int*,
                          const int*, __nv_bfloat16*, int, int, int, int, int, int, int, float, int, float*, cudaStream_t);
  int (*attention_stream_usable)(int, int, int, int, int, int);
  // out: kernels launched, and whether an error came from the attention library
  long long launches, attention_failed;
};
static_assert(sizeof(BlockCall) == 8 * 53, "the caller fills 53 members of eight bytes");

}  // namespace

BW_API int bw_bf16_block_members() { return static_cast<int>(sizeof(BlockCall) / 8); }

BW_API int bw_bf16_block(void* call, float eps1, float eps2, float scale, cudaStream_t stream) {
  BlockCall& c = *static_cast<BlockCall*>(call);
  const int n = static_cast<int>(c.n), width = static_cast<int>(c.width), heads = static_cast<int>(c.heads);
  const int kv_heads = static_cast<int>(c.kv_heads), hd = static_cast<int>(c.hd), inter = static_cast<int>(c.inter);
  const int page = static_cast<int>(c.page), max_blocks = static_cast<int>(c.max_blocks), max_keys = static_cast<int>(c.max_keys);
  const int window = static_cast<int>(c.window), pages = static_cast<int>(c.num_pages), writable = static_cast<int>(c.writable);
  const int q_dim = heads * hd, qkv_dim = (heads + 2 * kv_heads) * hd;
  const bool scratch = n <= bw_bf16_linear_split_rows();
  float* partials = c.partials;  // the caller gives each range of rows the scratch it takes
  int* counters = scratch ? c.counters : nullptr;
  c.launches = 0, c.attention_failed = 0;
  int rc;
#define BW_DO(KERNELS_, CALL_)        \
  if ((rc = (CALL_)) != 0) return rc; \
  c.launches += (KERNELS_)
  auto kernels = [&](int m, int out, int in, int swiglu) { return bw_bf16_linear_tc_kernels(m, out, in, swiglu, scratch && partials != nullptr); };

  const bool rotates = bw_bf16_linear_rows_rope_usable(nullptr, nullptr, n, qkv_dim, width, heads, kv_heads, hd) != 0;
  const bool norm1_rides = rotates && bw_bf16_linear_rows_norm_usable(c.w_qkv, n, qkv_dim, width);
  if (!norm1_rides) {
    BW_DO(1, bw_bf16_rmsnorm(c.x, c.norm1, c.normed, nullptr, n, width, eps1, stream));
  }
  if (norm1_rides) {
    BW_DO(1, bw_bf16_linear_rows_norm_rope(c.x, c.norm1, eps1, c.w_qkv, c.qkv, n, qkv_dim, width, c.pos, c.row_seq, c.cos_t, c.sin_t,
                                           c.block_table, max_blocks, c.k, c.v, heads, kv_heads, hd, page, writable, stream));
  } else if (rotates) {
    BW_DO(1, bw_bf16_linear_rows_rope(c.normed, c.w_qkv, c.qkv, n, qkv_dim, width, c.pos, c.row_seq, c.cos_t, c.sin_t, c.block_table,
                                      max_blocks, c.k, c.v, heads, kv_heads, hd, page, writable, partials, stream));
  } else {
    BW_DO(kernels(n, qkv_dim, width, 0),
          bw_bf16_linear(c.normed, c.w_qkv, c.qkv, 0, nullptr, n, qkv_dim, width, partials, counters, 0, stream));
    BW_DO(1, bw_bf16_rope_cache(c.qkv, qkv_dim, c.pos, c.row_seq, c.cos_t, c.sin_t, c.block_table, max_blocks, c.k, c.v, n, heads,
                                kv_heads, hd, page, writable, stream));
  }

  c.attention_failed = 1;
  const int tiles = static_cast<int>(c.tiles);
  const bool split = tiles == n && max_keys > 128;  // a decode step
  const int tc_rows = split ? 0 : c.attention_tc_rows(heads, kv_heads, hd, page, qkv_dim);
  if (!split && tc_rows > 0 && tc_rows == c.tc_rows && n > tiles) {
    BW_DO(1, c.attention_tc(c.qkv, qkv_dim, c.k, c.v, pages, c.block_table, max_blocks, c.tc_seq, c.tc_row0, c.tc_tile_rows,
                            static_cast<int>(c.tc_tiles), c.seq_pos0, c.seq_row0, c.attn, q_dim, n, heads, kv_heads, hd, page, window,
                            scale, stream));
  } else if (split && c.attention_stream_usable(n, heads, kv_heads, hd, page, qkv_dim)) {
    BW_DO(2, c.attention_stream(c.qkv, qkv_dim, c.k, c.v, pages, c.block_table, max_blocks, c.row_seq, c.pos, c.attn, q_dim, n, heads,
                                kv_heads, hd, page, window, scale, max_keys, c.attn_scratch, stream));
  } else {
    BW_DO(split ? 2 : 1, c.attention(c.qkv, qkv_dim, c.k, c.v, c.block_table, max_blocks, c.tile_seq, c.tile_row0, c.tile_rows, tiles,
                                     c.seq_pos0, c.seq_row0, c.row_seq, c.pos, c.attn, q_dim, n, heads, kv_heads, hd, page, window,
                                     scale, max_keys, split ? c.attn_scratch : nullptr, stream));
  }
  c.attention_failed = 0;

  BW_DO(kernels(n, width, q_dim, 0), bw_bf16_linear(c.attn, c.w_o, c.x, 1, c.x, n, width, q_dim, partials, counters, 0, stream));
  const bool norm2_rides = c.fused_glu && bw_bf16_linear_rows_norm_usable(c.w_gate_up, n, 2 * inter, width);
  if (!norm2_rides) {
    BW_DO(1, bw_bf16_rmsnorm(c.x, c.norm2, c.normed, nullptr, n, width, eps2, stream));
  }
  if (norm2_rides) {
    BW_DO(1, bw_bf16_linear_rows_norm_swiglu(c.x, c.norm2, eps2, c.w_gate_up, c.h, n, 2 * inter, width, bw::kGluSilu, stream));
  } else if (c.fused_glu) {
    BW_DO(kernels(n, 2 * inter, width, 1),
          bw_bf16_linear_tc_swiglu(c.normed, c.w_gate_up, c.h, n, 2 * inter, width, partials, bw::kGluSilu, stream));
  } else {
    BW_DO(kernels(n, 2 * inter, width, 0),
          bw_bf16_linear(c.normed, c.w_gate_up, c.gate_up, 0, nullptr, n, 2 * inter, width, partials, counters, 0, stream));
    BW_DO(1, bw_bf16_swiglu(c.gate_up, c.h, n, inter, stream));
  }
  BW_DO(kernels(n, width, inter, 0), bw_bf16_linear(c.h, c.w_down, c.x, 1, c.x, n, width, inter, partials, counters, 0, stream));
#undef BW_DO
  return 0;
}
