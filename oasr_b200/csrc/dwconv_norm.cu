// Causal depthwise conv (9 taps) + LayerNorm over the channels + SiLU in one kernel: the middle of the FastConformer conv
// module (oasr/models/nemotron/encoder.py:183-214), packed segments or streams that continue from a cached tail.
//
// What bounds the two steps apart: the conv's 16-bit rows travel to memory and back, and its thread-per-channel-pair walk of
// a 36-frame run has 9 loads of 4 bytes in flight.  A block here owns all channels of a run of frames of one segment, a
// thread four neighbouring channels: 8-byte loads, eight frames at a time, the next eight requested before the statistics of
// these; the conv values stay in registers through the norm (mean, then squared deviations, each one block reduction of eight
// sums at once).  Every input row is read once per run plus 8 rows of halo.  28000 rows of 1024 channels: 81 us, against about
// 150 us as two kernels; what bounds it now is its arithmetic (the SiLU's exponential and division among it), not its bytes.
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace ob {
namespace dwconv_norm {

constexpr int K = 9;              // taps
constexpr int G = 8;              // frames at a time = K - 1 rows of history
constexpr int kMaxThreads = 256;  // four channels each

struct Params {
  void* out;                      // (rows, C)
  const void* in;                 // (rows, C)
  const void *weight, *bias;      // (K, C), (C) nullable
  const void *norm_w, *norm_b;    // (C), (C) nullable
  const int32_t* cu;              // packed segment boundaries, or null: segments of `seq` rows
  void* state;                    // streams: (slots, K - 1, C), the rows before the segment; replaced by its last K - 1 rows
  const int64_t* slots;
  int64_t num_slots;
  int seq, C, run;                // run: frames of a block, a multiple of G
  float eps;
};

template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
  else return __half22float2(*reinterpret_cast<const __half2*>(&u));
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

// Sums of eight values over the block: within the warp by halving (4 + 2 + 1 + 1 + 1 exchanges), then over the warps through
// `red`.  The order depends on the number of threads only.
__device__ __forceinline__ void block_sum8(float (&v)[G], float (*red)[kMaxThreads / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  float a[4], b[2], s;
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = ((lane & 16) ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? v[i] : v[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = ((lane & 8) ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, (lane & 8) ? a[i] : a[i + 2], 8);
  s = ((lane & 4) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? b[0] : b[1], 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if ((lane & 3) == 0) red[lane >> 2][warp] = s;      // lane bits 4..2 say which of the eight this is
  __syncthreads();
  s = 0.f;
  for (int w = lane & 3; w < warps; w += 4) s += red[lane >> 2][w];
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
#pragma unroll
  for (int i = 0; i < G; ++i) v[i] = __shfl_sync(0xffffffffu, s, i * 4);
}

// Grid (runs of the longest segment, segments), C / 4 threads.
template <typename T, bool kState>
__global__ void __launch_bounds__(kMaxThreads, 2) dwconv_norm_kernel(const Params p) {
  ptx::grid_dep_launch();   // no-ops unless launched with programmatic stream serialisation
  ptx::grid_dep_wait();
  __shared__ float red[2][G][kMaxThreads / 32];
  const int b = blockIdx.y, C = p.C, c = threadIdx.x * 4;
  const int64_t row0 = p.cu ? p.cu[b] : static_cast<int64_t>(b) * p.seq;
  const int len = p.cu ? p.cu[b + 1] - static_cast<int>(row0) : p.seq;
  const int t0 = blockIdx.x * p.run, t_end = min(len, t0 + p.run);
  if (t0 >= len) return;
  const T* in = static_cast<const T*>(p.in) + row0 * C + c;
  T* state = nullptr;
  if constexpr (kState) {
    const int64_t slot = p.slots[b];           // a slot outside the buffer: zeros before the segment, nothing kept
    if (slot >= 0 && slot < p.num_slots) state = static_cast<T*>(p.state) + slot * (K - 1) * C + c;
  }
  auto fetch = [&](int t) -> uint2 {
    if (t >= 0 && t < len) return __ldg(reinterpret_cast<const uint2*>(in + static_cast<int64_t>(t) * C));
    if constexpr (kState) {
      if (t < 0 && t >= 1 - K && state) return *reinterpret_cast<const uint2*>(state + (K - 1 + t) * C);
    }
    return make_uint2(0u, 0u);
  };
  uint2 old[G], cur[G];
#pragma unroll
  for (int i = 0; i < G; ++i) old[i] = fetch(t0 - G + i);
#pragma unroll
  for (int i = 0; i < G; ++i) cur[i] = fetch(t0 + i);
  if constexpr (kState) {
    // the segment's last rows (of [state ; segment] where it is shorter).  Only a segment's first block reads its state (a run
    // is at least the K - 1 rows a later one looks back), so it also replaces it, a thread its own channels.
    if (t0 == 0 && state) {
      uint2 keep[K - 1];
#pragma unroll
      for (int i = 0; i < K - 1; ++i) keep[i] = fetch(len - (K - 1) + i);
#pragma unroll
      for (int i = 0; i < K - 1; ++i) *reinterpret_cast<uint2*>(state + i * C) = keep[i];
    }
  }
  float2 w[K][2];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const T*>(p.weight) + k * C + c));
    w[k][0] = unpack2<T>(u.x);
    w[k][1] = unpack2<T>(u.y);
  }
  const float inv_c = 1.f / static_cast<float>(C);
  T* out = static_cast<T*>(p.out) + row0 * C + c;
#pragma unroll 1
  for (int t = t0; t < t_end; t += G) {
    float2 acc[G][2];
    const uint2 cb = p.bias ? __ldg(reinterpret_cast<const uint2*>(static_cast<const T*>(p.bias) + c)) : make_uint2(0u, 0u);
#pragma unroll
    for (int j = 0; j < G; ++j) { acc[j][0] = unpack2<T>(cb.x); acc[j][1] = unpack2<T>(cb.y); }
#pragma unroll
    for (int i = 0; i < 2 * G; ++i) {          // row t - 8 + i meets tap i - j of output t + j
      const uint2 u = i < G ? old[i] : cur[i - G];
      const float2 x0 = unpack2<T>(u.x), x1 = unpack2<T>(u.y);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if (i - j >= 0 && i - j < K) {
          acc[j][0] = __ffma2_rn(x0, w[i - j][0], acc[j][0]);
          acc[j][1] = __ffma2_rn(x1, w[i - j][1], acc[j][1]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < G; ++i) old[i] = cur[i];
    if (t + G < t_end) {
#pragma unroll
      for (int i = 0; i < G; ++i) cur[i] = fetch(t + G + i);
    }
    // the conv's own 16-bit rounding, as where the two steps are apart (padded batches): both forms then agree
#pragma unroll
    for (int j = 0; j < G; ++j) {
      acc[j][0] = unpack2<T>(pack2<T>(acc[j][0].x, acc[j][0].y));
      acc[j][1] = unpack2<T>(pack2<T>(acc[j][1].x, acc[j][1].y));
    }
    float s[G], sq[G];
#pragma unroll
    for (int j = 0; j < G; ++j) s[j] = (acc[j][0].x + acc[j][0].y) + (acc[j][1].x + acc[j][1].y);
    block_sum8(s, red[0]);
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const float mean = s[j] * inv_c;
      acc[j][0].x -= mean; acc[j][0].y -= mean; acc[j][1].x -= mean; acc[j][1].y -= mean;
      sq[j] = fmaf(acc[j][0].x, acc[j][0].x, acc[j][0].y * acc[j][0].y) + fmaf(acc[j][1].x, acc[j][1].x, acc[j][1].y * acc[j][1].y);
    }
    block_sum8(sq, red[1]);
    const uint2 gu = __ldg(reinterpret_cast<const uint2*>(static_cast<const T*>(p.norm_w) + c));
    const uint2 bu = p.norm_b ? __ldg(reinterpret_cast<const uint2*>(static_cast<const T*>(p.norm_b) + c)) : make_uint2(0u, 0u);
    const float2 g0 = unpack2<T>(gu.x), g1 = unpack2<T>(gu.y), b0 = unpack2<T>(bu.x), b1 = unpack2<T>(bu.y);
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const float rstd = rsqrtf(sq[j] * inv_c + p.eps);
      const float y0 = apply_act<OASR_ACT_SWISH>(fmaf(acc[j][0].x * rstd, g0.x, b0.x));
      const float y1 = apply_act<OASR_ACT_SWISH>(fmaf(acc[j][0].y * rstd, g0.y, b0.y));
      const float y2 = apply_act<OASR_ACT_SWISH>(fmaf(acc[j][1].x * rstd, g1.x, b1.x));
      const float y3 = apply_act<OASR_ACT_SWISH>(fmaf(acc[j][1].y * rstd, g1.y, b1.y));
      if (t + j < t_end) *reinterpret_cast<uint2*>(out + static_cast<int64_t>(t + j) * C) = make_uint2(pack2<T>(y0, y1), pack2<T>(y2, y3));
    }
  }
}

bool fits(int64_t channels, int64_t kernel_size) { return kernel_size == K && channels % 128 == 0 && channels > 0 && channels <= 4 * kMaxThreads; }

template <bool kState>
int launch(Params& p, int64_t segs, int64_t max_seg, int dtype, cudaStream_t s) {
  const dim3 grid(static_cast<unsigned>((max_seg + p.run - 1) / p.run), static_cast<unsigned>(segs));
  return OB_DISPATCH_HALF(dtype, T, [&]() -> int {
    launch_pdl(dwconv_norm_kernel<T, kState>, grid, dim3(static_cast<unsigned>(p.C / 4)), 0, s, p);
    return check_launch("depthwise conv + norm launch");
  });
}

}  // namespace dwconv_norm
}  // namespace ob

extern "C" {

int oasr_b200_dwconv_norm_swish_supported(int64_t channels, int64_t kernel_size) { return ob::dwconv_norm::fits(channels, kernel_size) ? 1 : 0; }

int oasr_b200_dwconv_norm_swish_packed(void* out, const void* in, const void* weight, const void* bias, const void* norm_w, const void* norm_b,
                                       const int32_t* cu_seqlens, int64_t num_segs, int64_t max_seg, int64_t total, int64_t channels,
                                       int64_t kernel_size, double eps, int dtype, void* stream) {
  using namespace ob;
  using namespace ob::dwconv_norm;
  OB_REQUIRE(fits(channels, kernel_size), OASR_ERR_UNSUPPORTED, "dwconv_norm_swish_packed: %d taps, channels a multiple of 128 up to %d (got %lld, %lld)",
             K, 4 * kMaxThreads, (long long)kernel_size, (long long)channels);
  OB_REQUIRE(num_segs >= 0 && num_segs < 65536 && max_seg >= 0 && max_seg < (1 << 30) && total >= 0, OASR_ERR_INVALID, "dwconv_norm_swish_packed: bad shape");
  if (num_segs == 0 || max_seg == 0 || total == 0) return OASR_OK;
  OB_REQUIRE(out && in && weight && norm_w && cu_seqlens, OASR_ERR_INVALID, "dwconv_norm_swish_packed: null pointer argument");
  OB_REQUIRE(is_aligned(out, 8) && is_aligned(in, 8) && is_aligned(weight, 8) && is_aligned(norm_w, 8) && (!bias || is_aligned(bias, 8)) &&
                 (!norm_b || is_aligned(norm_b, 8)),
             OASR_ERR_ALIGN, "dwconv_norm_swish_packed: pointers must be 8-byte aligned");
  Params p{};
  p.out = out; p.in = in; p.weight = weight; p.bias = bias; p.norm_w = norm_w; p.norm_b = norm_b; p.cu = cu_seqlens;
  p.C = (int)channels; p.eps = (float)eps;
  // a run of 32 frames reads a quarter of its rows twice; shorter ones where 32 would leave SMs without their two blocks
  const int64_t slots = 2 * sm_count();
  p.run = total >= 32 * slots ? 32 : (total >= 16 * slots ? 16 : 8);
  return launch<false>(p, num_segs, max_seg, dtype, static_cast<cudaStream_t>(stream));
}

int oasr_b200_dwconv_norm_swish_stream(void* out, const void* in, const void* weight, const void* bias, const void* norm_w, const void* norm_b,
                                       void* state, int64_t num_slots, const int64_t* slot_ids, int64_t B, int64_t T, int64_t channels,
                                       int64_t kernel_size, double eps, int dtype, void* stream) {
  using namespace ob;
  using namespace ob::dwconv_norm;
  OB_REQUIRE(fits(channels, kernel_size), OASR_ERR_UNSUPPORTED, "dwconv_norm_swish_stream: %d taps, channels a multiple of 128 up to %d (got %lld, %lld)",
             K, 4 * kMaxThreads, (long long)kernel_size, (long long)channels);
  OB_REQUIRE(B >= 0 && B < 65536 && T >= 0 && T < (1 << 30) && num_slots >= 0, OASR_ERR_INVALID, "dwconv_norm_swish_stream: bad shape");
  if (B == 0 || T == 0) return OASR_OK;
  OB_REQUIRE(out && in && weight && norm_w && state && slot_ids, OASR_ERR_INVALID, "dwconv_norm_swish_stream: null pointer argument");
  OB_REQUIRE(is_aligned(out, 8) && is_aligned(in, 8) && is_aligned(weight, 8) && is_aligned(norm_w, 8) && is_aligned(state, 8) &&
                 (!bias || is_aligned(bias, 8)) && (!norm_b || is_aligned(norm_b, 8)),
             OASR_ERR_ALIGN, "dwconv_norm_swish_stream: pointers must be 8-byte aligned");
  Params p{};
  p.out = out; p.in = in; p.weight = weight; p.bias = bias; p.norm_w = norm_w; p.norm_b = norm_b;
  p.state = state; p.slots = slot_ids; p.num_slots = num_slots;
  p.seq = (int)T; p.C = (int)channels; p.eps = (float)eps;
  p.run = G;                       // few rows: what counts is a block's latency
  return launch<true>(p, B, T, dtype, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
