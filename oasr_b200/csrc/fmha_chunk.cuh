// Host interface of the streaming-chunk attention (fmha_chunk.cu), for at most 16 query frames.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ob {
namespace fmha_chunk {

bool applies(int64_t Tq, int64_t block_size, int64_t blocks_per_seq);        // 16-bit pages
bool applies_fp8(int64_t Tq, int64_t block_size, int64_t blocks_per_seq);
// few enough streams, and pools, for one kernel in the place of paged_kv_write(_fp8) and fmha_paged_relpos(_fp8)
bool applies_append(int64_t B, int64_t H, int64_t Tq, int64_t block_size, int64_t blocks_per_seq, const void* k_pool, const void* v_pool);

// k_scale / v_scale null: 16-bit pools; otherwise the pools hold fp8 e4m3 codes with per-head scales.  append_at null: the
// chunk's keys and values are in their pages already; otherwise (applies_append) they are written from position append_at[b] on.
int run(void* out, const void* qkv4, void* k_pool, void* v_pool, const float* k_scale, const float* v_scale, const void* pos,
        int64_t pos_rows, int64_t pos_stride, const int32_t* pos_start, const int32_t* block_table, const int32_t* seqlens,
        int64_t B, int64_t Tq, int64_t H, int64_t blocks_per_seq, int64_t block_size, int64_t num_blocks, double scale,
        int dtype, cudaStream_t stream, const int32_t* append_at);

}  // namespace fmha_chunk
}  // namespace ob
