// Attention inside a chunked-limited window with the Transformer-XL relative-position term (FastConformer / Nemotron):
//
//   out[i, h, :] = softmax_j( ((q_i+u).k_j + (q_i+v).r_{i-j}) * scale ) . v_j ,
//   j in the chunks [chunk(i) - left_chunks, chunk(i)] of the segment,  r_d = relative_k_proj(sinusoid(d))
//
// (oasr/models/nemotron/encoder.py:82-149, 300-410).  A frame sees at most left + chunk keys (60 of the default
// configuration) whatever the segment's length, at most 64 different distances, and neighbouring frames see almost the
// same keys: so the position scores are a 16 x 64 product per 16 frames instead of a (frames x 2T-1) matrix, nothing of
// size T^2 exists, and the work is linear in the frames.  What remains is reading q+u, q+v, k, v and writing the output
// once: HBM-bound (10 D bytes per frame and head).
//
// A warp owns 16 frames of one head.  Their keys are 80 consecutive ones, the first `off` = left + chunk - 1 before the
// first frame.  Products run on warp-level m16n8k16 MMAs: a 128-row tcgen05 tile would need 192 keys for 128 frames (two
// thirds of it masked) and pass scores through tensor memory twice, for a kernel that is bound by its bytes.  K order inside
// a 32-element block is permuted (the same way in both operands) so that a lane's fragments of two MMA steps are 16
// consecutive bytes.  Position scores go to a per-warp buffer and come back shifted: key column x of frame row r needs
// distance column x - r.  All 80 scores of a row are in registers, so the softmax is one pass.
//
// Two forms share the arithmetic: packed segments (64 frames per block; K, V and the 64 table rows shared through shared
// memory by its 4 warps; two blocks per SM), and paged streams (a block per (stream, head, 16 frames); the chunk's own keys
// from the projection, and the block that reads them also writes them to their pages, so that no separate page-write launch
// is needed).  A streaming step has few items and a chain of launches behind it, so what counts there is one item's latency:
// four warps fetch its keys, values and table rows into shared memory, share the position scores and P.V, and repeat the
// content scores (24 streams x 8 heads: 10.1 us; 36.4 us as a warp per item with keys straight from memory into fragments).
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace ob {
namespace fmha_window {

constexpr int kRows = 16;              // query frames of a warp
constexpr int kKeys = 80;              // keys of a warp: 16 + window - 1 <= 80
constexpr int kDist = 64;              // distances of a warp's window
constexpr int kPitch = 74;             // floats per row of the position-score buffer
constexpr int kWarps = 4;
constexpr int kBlockRows = kWarps * kRows, kBlockKeys = 128;

struct Params {
  const void* qkv4;                    // rows of [q+u | q+v | k | v], each H * D wide
  const void* rel_k;                   // (table_rows, H * D): row `center` - d has distance d
  void* out;                           // (rows, H * D)
  int64_t table_rows;
  int H, center, chunk, left_chunks;
  float scale_log2;
  const int32_t* cu;                   // packed: segment boundaries
  // paged
  void *k_pool, *v_pool;               // (num_blocks, block_size, H, D)
  const int32_t *block_table, *cached, *pos_start;
  int B, Tq, blocks_per_seq, block_size, num_blocks;
};

template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
// 16 bytes global -> shared; zeros where `live` is false (the source address must be valid all the same).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A 16-row x D operand as fragments: row g and row g + 8, 8 consecutive elements per 32-element block.
template <int D>
struct QFrag { uint4 lo[D / 32], hi[D / 32]; };

// 16 frames by kSplit warps (this one is number `part`): `key16(n, blk)` / `rel16(n, blk)` give this lane's 16 bytes of key
// (distance) row 8 n + g, block blk; `v_tile` = the 80 value rows in shared memory (D * 2 bytes each, 16-byte chunk c of row r
// at c ^ (r & 7)); `escore` = the item's buffer, >= 16 * kPitch floats and >= 16 rows of output; `v_ready()` waits for the value
// tile, and with several warps for all of them, as `sync()` does.
template <typename T, int D, int kSplit, typename KeyFn, typename RelFn, typename VReady, typename Sync>
__device__ __forceinline__ void warp_attention(const QFrag<D>& qu, const QFrag<D>& qv, KeyFn key16, RelFn rel16, VReady v_ready,
                                               const uint8_t* v_tile, float* escore, T* out, int64_t out_ld, int rows_live,
                                               int j0, const int (&klo)[2], const int (&khi)[2], float scale_log2, int part,
                                               Sync sync) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int kBlk = D / 32;
  // position scores of the 16 frames against the 64 distances
#pragma unroll 4
  for (int nn = 0; nn < kDist / 8 / kSplit; ++nn) {
    const int n = part * (kDist / 8 / kSplit) + nn;
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int b = 0; b < kBlk; ++b) {
      const uint4 w = rel16(n, b);
      mma16816<T>(c, qv.lo[b].x, qv.hi[b].x, qv.lo[b].y, qv.hi[b].y, w.x, w.y);
      mma16816<T>(c, qv.lo[b].z, qv.hi[b].z, qv.lo[b].w, qv.hi[b].w, w.z, w.w);
    }
    *reinterpret_cast<float2*>(escore + g * kPitch + n * 8 + 2 * t) = make_float2(c[0], c[1]);
    *reinterpret_cast<float2*>(escore + (g + 8) * kPitch + n * 8 + 2 * t) = make_float2(c[2], c[3]);
  }
  sync();
  // content scores, shifted position scores, mask
  float s[kKeys / 8][4];
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int n = 0; n < kKeys / 8; ++n) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
#pragma unroll
    for (int b = 0; b < kBlk; ++b) {
      const uint4 w = key16(n, b);
      mma16816<T>(s[n], qu.lo[b].x, qu.hi[b].x, qu.lo[b].y, qu.hi[b].y, w.x, w.y);
      mma16816<T>(s[n], qu.lo[b].z, qu.hi[b].z, qu.lo[b].w, qu.hi[b].w, w.z, w.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int half = i >> 1, x = n * 8 + 2 * t + (i & 1), r = g + 8 * half, j = j0 + x;
      const float v = (s[n][i] + escore[r * kPitch + x - r]) * scale_log2;
      s[n][i] = j >= klo[half] && j < khi[half] ? v : -INFINITY;
      mx[half] = fmaxf(mx[half], s[n][i]);
    }
  }
  float sum[2] = {0.f, 0.f};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
    mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
    if (mx[h] == -INFINITY) mx[h] = 0.f;             // a row past the segment: every weight is zero
  }
#pragma unroll
  for (int n = 0; n < kKeys / 8; ++n) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[n][i] = exp2f(s[n][i] - mx[i >> 1]);
      sum[i >> 1] += s[n][i];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
    sum[h] = sum[h] > 0.f ? 1.f / sum[h] : 0.f;
  }
  uint32_t p[kKeys / 16][4];
#pragma unroll
  for (int k = 0; k < kKeys / 16; ++k) {
    p[k][0] = pack2<T>(s[2 * k][0], s[2 * k][1]);
    p[k][1] = pack2<T>(s[2 * k][2], s[2 * k][3]);
    p[k][2] = pack2<T>(s[2 * k + 1][0], s[2 * k + 1][1]);
    p[k][3] = pack2<T>(s[2 * k + 1][2], s[2 * k + 1][3]);
  }
  v_ready();
  // P . V, then the rows through the score buffer so that the stores are 16 bytes wide and contiguous
  const uint32_t v_addr = ptx::smem_u32(v_tile);
  uint8_t* obuf = reinterpret_cast<uint8_t*>(escore);
  const int vr = (lane & 7) + ((lane >> 3) & 1) * 8, vc = lane >> 4;   // ldmatrix row of this lane, second 8 columns
#pragma unroll 2
  for (int dd = 0; dd < D / 16 / kSplit; ++dd) {
    const int d = part * (D / 16 / kSplit) + dd;
    float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < kKeys / 16; ++k) {
      const int r = k * 16 + vr;
      uint32_t w[4];
      ldmatrix_x4_trans(w, v_addr + r * (D * 2) + (((2 * d + vc) ^ (r & 7)) << 4));
      mma16816<T>(o[0], p[k][0], p[k][1], p[k][2], p[k][3], w[0], w[1]);
      mma16816<T>(o[1], p[k][0], p[k][1], p[k][2], p[k][3], w[2], w[3]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = 2 * d + e;                       // 16-byte chunk of the row: columns 8 c + 2 t, + 1
      *reinterpret_cast<uint32_t*>(obuf + g * (D * 2) + ((c ^ (g & 7)) << 4) + 4 * t) = pack2<T>(o[e][0] * sum[0], o[e][1] * sum[0]);
      *reinterpret_cast<uint32_t*>(obuf + (g + 8) * (D * 2) + ((c ^ (g & 7)) << 4) + 4 * t) = pack2<T>(o[e][2] * sum[1], o[e][3] * sum[1]);
    }
  }
  sync();
  constexpr int kC = D / 8;
#pragma unroll
  for (int i = part * 32 + lane; i < kRows * kC; i += 32 * kSplit) {
    const int r = i / kC, c = i - r * kC;
    if (r < rows_live) *reinterpret_cast<uint4*>(out + r * out_ld + c * 8) = *reinterpret_cast<const uint4*>(obuf + r * (D * 2) + ((c ^ (r & 7)) << 4));
  }
}

template <typename T, int D>
__device__ __forceinline__ void load_q(QFrag<D>& q, const T* base, int64_t ld, int rows_live) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int b = 0; b < D / 32; ++b) {
    q.lo[b] = g < rows_live ? *reinterpret_cast<const uint4*>(base + g * ld + b * 32 + t * 8) : make_uint4(0, 0, 0, 0);
    q.hi[b] = g + 8 < rows_live ? *reinterpret_cast<const uint4*>(base + (g + 8) * ld + b * 32 + t * 8) : make_uint4(0, 0, 0, 0);
  }
}

template <int D>
struct SmemPacked {
  static constexpr int kRow = D * 2, kK = 0, kV = kK + kBlockKeys * kRow, kR = kV + kBlockKeys * kRow, kE = kR + kDist * kRow,
                       kBytes = kE + kWarps * kRows * kPitch * 4;
};

// Packed segments: grid (query blocks of the longest segment, heads, segments).
template <typename T, int D>
__global__ void __launch_bounds__(kWarps * 32, 2) window_packed_kernel(const Params p) {
  using S = SmemPacked<D>;
  ptx::grid_dep_launch();   // no-ops unless launched with programmatic stream serialisation
  ptx::grid_dep_wait();
  const int h = blockIdx.y, row0 = p.cu[blockIdx.z], len = p.cu[blockIdx.z + 1] - row0, q0 = blockIdx.x * kBlockRows;
  if (q0 >= len) return;
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t C = static_cast<int64_t>(p.H) * D, ld = 4 * C;
  const T* q = static_cast<const T*>(p.qkv4) + row0 * ld + h * D;
  const int off = p.left_chunks * p.chunk + p.chunk - 1;
  constexpr int kC = D / 8;             // 16-byte chunks of a row
  // table rows of distances off .. off - 63, keys q0 - off .. + 127 (chunk bit 2 flipped in odd rows: a fragment load of
  // two rows then covers all banks), values of the same keys
  for (int i = threadIdx.x; i < kDist * kC; i += kWarps * 32) {
    const int r = i / kC, c = i - r * kC;
    int64_t at = static_cast<int64_t>(p.center) - off + r;
    at = at < 0 ? 0 : (at >= p.table_rows ? p.table_rows - 1 : at);
    cp_async16(smem + S::kR + r * S::kRow + ((c ^ ((r & 1) << 2)) << 4), static_cast<const T*>(p.rel_k) + at * C + h * D + c * 8, true);
  }
  for (int i = threadIdx.x; i < kBlockKeys * kC; i += kWarps * 32) {
    const int r = i / kC, c = i - r * kC, j = q0 - off + r;
    const bool live = j >= 0 && j < len;
    cp_async16(smem + S::kK + r * S::kRow + ((c ^ ((r & 1) << 2)) << 4), q + (live ? j : 0) * ld + 2 * C + c * 8, live);
  }
  cp_async_commit();
  for (int i = threadIdx.x; i < kBlockKeys * kC; i += kWarps * 32) {
    const int r = i / kC, c = i - r * kC, j = q0 - off + r;
    const bool live = j >= 0 && j < len;
    cp_async16(smem + S::kV + r * S::kRow + ((c ^ (r & 7)) << 4), q + (live ? j : 0) * ld + 3 * C + c * 8, live);
  }
  cp_async_commit();
  const int i0 = q0 + warp * kRows, rows_live = len - i0;
  QFrag<D> qu, qv;
  load_q<T, D>(qu, q + i0 * ld, ld, rows_live);
  load_q<T, D>(qv, q + i0 * ld + C, ld, rows_live);
  cp_async_wait<1>();
  __syncthreads();
  int klo[2], khi[2];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int i = i0 + g + 8 * hh, qc = i / p.chunk;
    klo[hh] = max(0, (qc - p.left_chunks) * p.chunk);
    khi[hh] = i < len ? min((qc + 1) * p.chunk, len) : 0;
  }
  const uint8_t* sK = smem + S::kK + warp * kRows * S::kRow;
  const uint8_t* sR = smem + S::kR;
  auto key16 = [&](int n, int b) { return *reinterpret_cast<const uint4*>(sK + (n * 8 + g) * S::kRow + (((b * 4 + t) ^ ((g & 1) << 2)) << 4)); };
  auto rel16 = [&](int n, int b) { return *reinterpret_cast<const uint4*>(sR + (n * 8 + g) * S::kRow + (((b * 4 + t) ^ ((g & 1) << 2)) << 4)); };
  auto v_ready = [&]() {
    cp_async_wait<0>();
    __syncthreads();
  };
  warp_attention<T, D, 1>(qu, qv, key16, rel16, v_ready, smem + S::kV + warp * kRows * S::kRow,
                          reinterpret_cast<float*>(smem + S::kE) + warp * kRows * kPitch,
                          static_cast<T*>(p.out) + (row0 + i0) * C + h * D, C, rows_live, i0 - off, klo, khi, p.scale_log2, 0,
                          [] { __syncwarp(); });
}

template <int D>
struct SmemPaged {
  static constexpr int kRow = D * 2, kK = 0, kV = kK + kKeys * kRow, kR = kV + kKeys * kRow, kE = kR + kDist * kRow,
                       kBytes = kE + kRows * kPitch * 4;
};

// Paged streams: a block per (stream, block of 16 new frames, head), heads of a stream side by side.
template <typename T, int D>
__global__ void __launch_bounds__(kWarps * 32, 3) window_paged_kernel(const Params p) {
  using S = SmemPaged<D>;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int qblocks = (p.Tq + kRows - 1) / kRows;
  const int item = blockIdx.x, h = item % p.H, rest = item / p.H, qb = rest % qblocks, b = rest / qblocks;
  const int64_t C = static_cast<int64_t>(p.H) * D, ld = 4 * C;
  const T* rows = static_cast<const T*>(p.qkv4) + static_cast<int64_t>(b) * p.Tq * ld + h * D;   // new frame t: row t
  T* kp = static_cast<T*>(p.k_pool);
  T* vp = static_cast<T*>(p.v_pool);
  const int cached = p.cached[b], total = cached + p.Tq, f0 = p.pos_start[b];   // key j of the stream is frame f0 + j
  const int off = p.left_chunks * p.chunk + p.chunk - 1;
  const int i0 = qb * kRows, rows_live = p.Tq - i0, j0 = cached + i0 - off;     // first key of the block (may be negative)
  const int32_t* table = p.block_table + static_cast<int64_t>(b) * p.blocks_per_seq;
  // element offset of key j in the pools, or -1
  auto page_at = [&](int j) -> int64_t {
    const int col = j / p.block_size;
    if (j < 0 || col >= p.blocks_per_seq) return -1;
    const int page = table[col];
    if (page < 0 || page >= p.num_blocks) return -1;
    return ((static_cast<int64_t>(page) * p.block_size + (j - col * p.block_size)) * p.H + h) * D;
  };
  constexpr int kC = D / 8, kStep = kWarps * 32 / kC;      // 16-byte chunks of a row, rows of one pass of the block
  const int lr = threadIdx.x / kC, lc = threadIdx.x - lr * kC;
  // keys, then values: the cached ones from their pages, the chunk's own from the projection
  auto source = [&](int r, const T* pool, int64_t part, bool& live) -> const T* {
    const int j = j0 + r;
    live = false;
    if (j >= cached && j < total) {
      live = true;
      return rows + (j - cached) * ld + part * C + lc * 8;
    }
    if (j >= 0 && j < cached) {
      const int64_t at = page_at(j);
      if (at >= 0) {
        live = true;
        return pool + at + lc * 8;
      }
    }
    return rows;
  };
  for (int r = lr; r < kKeys; r += kStep) {
    bool live;
    const T* src = source(r, kp, 2, live);
    cp_async16(smem + S::kK + r * S::kRow + ((lc ^ ((r & 1) << 2)) << 4), src, live);
  }
  for (int r = lr; r < kDist; r += kStep) {
    int64_t at = static_cast<int64_t>(p.center) - off + r;
    at = at < 0 ? 0 : (at >= p.table_rows ? p.table_rows - 1 : at);
    cp_async16(smem + S::kR + r * S::kRow + ((lc ^ ((r & 1) << 2)) << 4), static_cast<const T*>(p.rel_k) + at * C + h * D + lc * 8, true);
  }
  cp_async_commit();
  for (int r = lr; r < kKeys; r += kStep) {
    bool live;
    const T* src = source(r, vp, 3, live);
    cp_async16(smem + S::kV + r * S::kRow + ((lc ^ (r & 7)) << 4), src, live);
  }
  cp_async_commit();
  QFrag<D> qu, qv;
  load_q<T, D>(qu, rows + i0 * ld, ld, rows_live);
  load_q<T, D>(qv, rows + i0 * ld + C, ld, rows_live);
  // the new keys and values to their pages (the index rule of paged_kv_write: positions outside the table are dropped)
  for (int r = lr; r < kRows && r < rows_live; r += kStep) {
    const int64_t at = page_at(cached + i0 + r);
    if (at >= 0) {
      const T* src = rows + (i0 + r) * ld + 2 * C + lc * 8;
      *reinterpret_cast<uint4*>(kp + at + lc * 8) = *reinterpret_cast<const uint4*>(src);
      *reinterpret_cast<uint4*>(vp + at + lc * 8) = *reinterpret_cast<const uint4*>(src + C);
    }
  }
  int klo[2], khi[2];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int r = i0 + g + 8 * hh, qc = (f0 + cached + r) / p.chunk;            // chunks count absolute frames
    klo[hh] = max(0, (qc - p.left_chunks) * p.chunk - f0);
    khi[hh] = r < p.Tq ? min((qc + 1) * p.chunk - f0, total) : 0;
  }
  cp_async_wait<1>();
  __syncthreads();
  auto key16 = [&](int n, int blk) { return *reinterpret_cast<const uint4*>(smem + S::kK + (n * 8 + g) * S::kRow + (((blk * 4 + t) ^ ((g & 1) << 2)) << 4)); };
  auto rel16 = [&](int n, int blk) { return *reinterpret_cast<const uint4*>(smem + S::kR + (n * 8 + g) * S::kRow + (((blk * 4 + t) ^ ((g & 1) << 2)) << 4)); };
  auto v_ready = [&]() {
    cp_async_wait<0>();
    __syncthreads();
  };
  warp_attention<T, D, kWarps>(qu, qv, key16, rel16, v_ready, smem + S::kV, reinterpret_cast<float*>(smem + S::kE),
                               static_cast<T*>(p.out) + (static_cast<int64_t>(b) * p.Tq + i0) * C + h * D, C, rows_live, j0, klo, khi,
                               p.scale_log2, warp, [] { __syncthreads(); });
}

template <typename K>
int launch(K kern, int bytes, dim3 grid, const Params& p, cudaStream_t s, const char* what) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return set_error(OASR_ERR_CUDA, "%s: cannot reserve %d bytes of shared memory: %s", what, bytes, cudaGetErrorString(e));
  launch_pdl(kern, grid, dim3(kWarps * 32), bytes, s, p);
  return check_launch(what);
}

}  // namespace fmha_window
}  // namespace ob

extern "C" {

int oasr_b200_fmha_window_supported(int64_t head_dim, int64_t chunk, int64_t left_chunks) {
  // the distances i - j of a window, left + chunk - 1 down to -(chunk - 1), fit the kernel's 64 columns
  return (head_dim == 64 || head_dim == 128) && chunk >= 1 && left_chunks >= 0 && chunk <= 64 && left_chunks <= 64 &&
                 left_chunks * chunk + 2 * chunk - 1 <= ob::fmha_window::kDist
             ? 1 : 0;
}

int oasr_b200_fmha_window_packed(void* out, const void* qkv4, const void* rel_k, int64_t table_rows, int64_t center,
                                 const int32_t* cu_seqlens, int64_t num_segs, int64_t max_seg, int64_t total, int64_t heads,
                                 int64_t head_dim, int64_t chunk, int64_t left_chunks, double scale, int dtype, void* stream) {
  using namespace ob;
  using namespace ob::fmha_window;
  OB_REQUIRE(oasr_b200_fmha_window_supported(head_dim, chunk, left_chunks) != 0, OASR_ERR_UNSUPPORTED,
             "fmha_window_packed: head_dim 64 or 128 and a window of at most %d distances (got %lld, %lld chunks of %lld)", kDist,
             (long long)head_dim, (long long)left_chunks, (long long)chunk);
  OB_REQUIRE(num_segs >= 0 && num_segs < 65536 && max_seg >= 0 && total >= 0 && total < (int64_t(1) << 31) && heads > 0 && heads < 65536 &&
                 table_rows > 0 && center >= 0 && center < table_rows,
             OASR_ERR_INVALID, "fmha_window_packed: bad shape");
  if (num_segs == 0 || total == 0 || max_seg == 0) return OASR_OK;
  OB_REQUIRE(out && qkv4 && rel_k && cu_seqlens, OASR_ERR_INVALID, "fmha_window_packed: null pointer argument");
  OB_REQUIRE(is_aligned(out, 16) && is_aligned(qkv4, 16) && is_aligned(rel_k, 16), OASR_ERR_ALIGN, "fmha_window_packed: pointers must be 16-byte aligned");
  Params p{};
  p.qkv4 = qkv4; p.rel_k = rel_k; p.out = out; p.table_rows = table_rows; p.H = (int)heads; p.center = (int)center;
  p.chunk = (int)chunk; p.left_chunks = (int)left_chunks; p.scale_log2 = static_cast<float>(scale * 1.4426950408889634); p.cu = cu_seqlens;
  const dim3 grid(static_cast<unsigned>((max_seg + kBlockRows - 1) / kBlockRows), static_cast<unsigned>(heads), static_cast<unsigned>(num_segs));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return OB_DISPATCH_HALF(dtype, T, [&]() -> int {
    if (head_dim == 128) return launch(window_packed_kernel<T, 128>, SmemPacked<128>::kBytes, grid, p, s, "fmha_window_packed launch");
    return launch(window_packed_kernel<T, 64>, SmemPacked<64>::kBytes, grid, p, s, "fmha_window_packed launch");
  });
}

int oasr_b200_fmha_window_paged(void* out, const void* qkv4, void* k_pool, void* v_pool, const void* rel_k, int64_t table_rows,
                                int64_t center, const int32_t* block_table, const int32_t* cached, const int32_t* pos_start, int64_t B,
                                int64_t Tq, int64_t heads, int64_t head_dim, int64_t blocks_per_seq, int64_t block_size,
                                int64_t num_blocks, int64_t chunk, int64_t left_chunks, double scale, int dtype, void* stream) {
  using namespace ob;
  using namespace ob::fmha_window;
  OB_REQUIRE(oasr_b200_fmha_window_supported(head_dim, chunk, left_chunks) != 0, OASR_ERR_UNSUPPORTED,
             "fmha_window_paged: head_dim 64 or 128 and a window of at most %d distances (got %lld, %lld chunks of %lld)", kDist,
             (long long)head_dim, (long long)left_chunks, (long long)chunk);
  OB_REQUIRE(B >= 0 && Tq > 0 && heads > 0 && blocks_per_seq > 0 && block_size > 0 && num_blocks > 0 && table_rows > 0 && center >= 0 &&
                 center < table_rows && B * Tq * heads < (int64_t(1) << 31),
             OASR_ERR_INVALID, "fmha_window_paged: bad shape");
  if (B == 0) return OASR_OK;
  OB_REQUIRE(out && qkv4 && k_pool && v_pool && rel_k && block_table && cached && pos_start, OASR_ERR_INVALID, "fmha_window_paged: null pointer argument");
  OB_REQUIRE(is_aligned(out, 16) && is_aligned(qkv4, 16) && is_aligned(rel_k, 16) && is_aligned(k_pool, 16) && is_aligned(v_pool, 16),
             OASR_ERR_ALIGN, "fmha_window_paged: pointers must be 16-byte aligned");
  Params p{};
  p.qkv4 = qkv4; p.rel_k = rel_k; p.out = out; p.table_rows = table_rows; p.H = (int)heads; p.center = (int)center;
  p.chunk = (int)chunk; p.left_chunks = (int)left_chunks; p.scale_log2 = static_cast<float>(scale * 1.4426950408889634);
  p.k_pool = k_pool; p.v_pool = v_pool; p.block_table = block_table; p.cached = cached; p.pos_start = pos_start;
  p.B = (int)B; p.Tq = (int)Tq; p.blocks_per_seq = (int)blocks_per_seq; p.block_size = (int)block_size; p.num_blocks = (int)num_blocks;
  const dim3 grid(static_cast<unsigned>(B * ((Tq + kRows - 1) / kRows) * heads));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return OB_DISPATCH_HALF(dtype, T, [&]() -> int {
    if (head_dim == 128) return launch(window_paged_kernel<T, 128>, SmemPaged<128>::kBytes, grid, p, s, "fmha_window_paged launch");
    return launch(window_paged_kernel<T, 64>, SmemPaged<64>::kBytes, grid, p, s, "fmha_window_paged launch");
  });
}

}  // extern "C"
