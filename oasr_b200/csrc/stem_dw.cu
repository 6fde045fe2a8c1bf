// The stem of the FastConformer 8x subsampling and the depthwise conv behind it in one kernel
// (oasr/models/nemotron/subsampling.py:39-53, 204-224): features -> 3x3 / stride-2 conv to C channels + bias + ReLU, rounded
// to 16 bits -> 3x3 / stride-2 depthwise conv + bias; zero padding (2, 1) on time and frequency at both.
//
// Apart, the two are bound by the stem's output, by far the largest tensor of the model (32 KB per feature-frame pair at 128
// bins and 256 channels), which is written once and read once; here it never leaves registers.  What is left is arithmetic:
// a depthwise output needs nine stem values of nine taps each, of which a thread that walks the frequency axis recomputes
// six.  A thread owns four channels of one output frame; the features of a block's frames sit in shared memory (every lane
// of a warp reads the same word), the stem's taps and the depthwise taps in registers, multiply-adds are packed pairs.
// Tap order and roundings are those of the two kernels, so the bits are too.  128 utterances of 5-30 s, 128 bins, 256
// channels: 1.97 ms, against 1.18 + 2.1 ms and a padded copy of the features.
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace ob {
namespace stem_dw {

constexpr int kThreads = 256;

struct Params {
  void* out;                 // (B, To, Fo, C)
  const float* in;           // (B, T, F), unpadded
  const float *w1, *b1;      // (C, 3, 3), (C)
  const void *w2, *b2;       // (C, 3, 3), (C) nullable, 16-bit
  const int32_t *mid_len;    // nullable: stem frames at or past it count as zeros
  const int32_t *out_len;    // nullable: output frames at or past it are zeros
  int T, F, C, T1, F1, To, Fo, pitch, fstep;
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

// Grid (blocks of kThreads / (C / 4) output frames, batch, frequency pieces of fstep outputs).
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) stem_dw_kernel(const Params p) {
  extern __shared__ __align__(16) float xs[];     // feature rows of the block's frames, column f at f + 2, zeros around
  const int groups = p.C / 4, rows = kThreads / groups, r = threadIdx.x / groups, c = (threadIdx.x - r * groups) * 4;
  const int b = blockIdx.y, to0 = blockIdx.x * rows, to = to0 + r;
  const int fo0 = blockIdx.z * p.fstep, fo1 = min(p.Fo, fo0 + p.fstep);
  const int live_end = p.out_len ? min(p.To, p.out_len[b]) : p.To;
  const int mid_end = p.mid_len ? min(p.T1, p.mid_len[b]) : p.T1;
  T* out = static_cast<T*>(p.out) + ((static_cast<int64_t>(b) * p.To + to) * p.Fo) * p.C + c;
  if (to0 >= live_end) {                          // nothing but zeros
    if (to < p.To)
      for (int fo = fo0; fo < fo1; ++fo) *reinterpret_cast<uint2*>(out + static_cast<int64_t>(fo) * p.C) = make_uint2(0u, 0u);
    return;
  }
  const int first = 4 * to0 - 6, n_rows = 4 * rows + 3;
  const float* in = p.in + static_cast<int64_t>(b) * p.T * p.F;
  for (int i = threadIdx.x; i < n_rows * p.pitch; i += kThreads) {
    const int row = i / p.pitch, f = i - row * p.pitch - 2, t = first + row;
    xs[i] = t >= 0 && t < p.T && f >= 0 && f < p.F ? __ldg(in + static_cast<int64_t>(t) * p.F + f) : 0.f;
  }
  float2 w[9][2];
  uint32_t wd[9][2];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const float* w1 = p.w1 + c * 9 + k;
    w[k][0] = make_float2(__ldg(w1), __ldg(w1 + 9));
    w[k][1] = make_float2(__ldg(w1 + 18), __ldg(w1 + 27));
    const uint16_t* w2 = static_cast<const uint16_t*>(p.w2) + c * 9 + k;
    wd[k][0] = __ldg(w2) | static_cast<uint32_t>(__ldg(w2 + 9)) << 16;
    wd[k][1] = __ldg(w2 + 18) | static_cast<uint32_t>(__ldg(w2 + 27)) << 16;
  }
  const float2 bias0 = make_float2(__ldg(p.b1 + c), __ldg(p.b1 + c + 1)), bias1 = make_float2(__ldg(p.b1 + c + 2), __ldg(p.b1 + c + 3));
  uint32_t bd[2] = {0u, 0u};
  if (p.b2) {
    const uint16_t* b2 = static_cast<const uint16_t*>(p.b2) + c;
    bd[0] = __ldg(b2) | static_cast<uint32_t>(__ldg(b2 + 1)) << 16;
    bd[1] = __ldg(b2 + 2) | static_cast<uint32_t>(__ldg(b2 + 3)) << 16;
  }
  __syncthreads();
  if (to >= p.To) return;
  if (to >= live_end) {
    for (int fo = fo0; fo < fo1; ++fo) *reinterpret_cast<uint2*>(out + static_cast<int64_t>(fo) * p.C) = make_uint2(0u, 0u);
    return;
  }
  bool mid[3];                                    // stem frames 2 to - 2 + d that exist
#pragma unroll
  for (int d = 0; d < 3; ++d) mid[d] = 2 * to - 2 + d >= 0 && 2 * to - 2 + d < mid_end;
  const float* x = xs + 4 * r * p.pitch;          // feature row under tap 0 of stem frame 2 to - 2
  // stem column f1 of the three frames, 16-bit; `cur` holds feature columns 2 f1 and 2 f1 + 1 (of seven rows), and becomes
  // those of the next column, whose first is this one's third
  float2 cur[7];
  auto column = [&](int f1, uint32_t (&v)[3][2]) {
    float2 nxt[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) nxt[i] = *reinterpret_cast<const float2*>(x + i * p.pitch + 2 * f1 + 2);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      float2 a0 = bias0, a1 = bias1;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float tap[3] = {cur[2 * d + i].x, cur[2 * d + i].y, nxt[2 * d + i].x};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float2 xx = make_float2(tap[j], tap[j]);
          a0 = __ffma2_rn(xx, w[i * 3 + j][0], a0);
          a1 = __ffma2_rn(xx, w[i * 3 + j][1], a1);
        }
      }
      const bool ok = mid[d];
      v[d][0] = ok ? pack2<T>(fmaxf(a0.x, 0.f), fmaxf(a0.y, 0.f)) : 0u;
      v[d][1] = ok ? pack2<T>(fmaxf(a1.x, 0.f), fmaxf(a1.y, 0.f)) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 7; ++i) cur[i] = nxt[i];
  };
  auto zero = [](uint32_t (&v)[3][2]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d][0] = v[d][1] = 0u;
  };
  auto load_cur = [&](int f1) {
#pragma unroll
    for (int i = 0; i < 7; ++i) cur[i] = *reinterpret_cast<const float2*>(x + i * p.pitch + 2 * f1);
  };
  uint32_t left[3][2], middle[3][2], right[3][2];
  if (fo0 == 0) {
    zero(left);
    load_cur(0);
  } else {
    load_cur(2 * fo0 - 2);
    column(2 * fo0 - 2, left);
  }
#pragma unroll 1
  for (int fo = fo0; fo < fo1; ++fo) {
    if (fo > 0 && 2 * fo - 1 < p.F1) column(2 * fo - 1, middle); else zero(middle);
    if (2 * fo < p.F1) column(2 * fo, right); else zero(right);
    float2 a0 = unpack2<T>(bd[0]), a1 = unpack2<T>(bd[1]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a0 = __ffma2_rn(unpack2<T>(left[d][0]), unpack2<T>(wd[3 * d][0]), a0);
      a1 = __ffma2_rn(unpack2<T>(left[d][1]), unpack2<T>(wd[3 * d][1]), a1);
      a0 = __ffma2_rn(unpack2<T>(middle[d][0]), unpack2<T>(wd[3 * d + 1][0]), a0);
      a1 = __ffma2_rn(unpack2<T>(middle[d][1]), unpack2<T>(wd[3 * d + 1][1]), a1);
      a0 = __ffma2_rn(unpack2<T>(right[d][0]), unpack2<T>(wd[3 * d + 2][0]), a0);
      a1 = __ffma2_rn(unpack2<T>(right[d][1]), unpack2<T>(wd[3 * d + 2][1]), a1);
    }
    *reinterpret_cast<uint2*>(out + static_cast<int64_t>(fo) * p.C) = make_uint2(pack2<T>(a0.x, a0.y), pack2<T>(a1.x, a1.y));
#pragma unroll
    for (int d = 0; d < 3; ++d) { left[d][0] = right[d][0]; left[d][1] = right[d][1]; }
  }
}

// Columns -2 .. 2 F1 + 1 are read (the last ones as part of a pair whose second word nothing uses).
int pitch_of(int64_t F) { return static_cast<int>((2 * (F / 2 + 1) + 4 + 1) / 2 * 2); }
int64_t smem_bytes(int64_t F, int64_t C) { return (4 * (kThreads / (C / 4)) + 3) * static_cast<int64_t>(pitch_of(F)) * 4; }
bool fits(int64_t F, int64_t C) {
  return C >= 4 && C % 4 == 0 && C / 4 <= kThreads && kThreads % (C / 4) == 0 && F >= 1 && F < 4096 && smem_bytes(F, C) <= 48 * 1024;
}

}  // namespace stem_dw
}  // namespace ob

extern "C" {

int oasr_b200_subsample_stem_dw_supported(int64_t F, int64_t C) { return ob::stem_dw::fits(F, C) ? 1 : 0; }

int oasr_b200_subsample_stem_dw(void* out, const float* in, const float* stem_w, const float* stem_b, const void* dw_w, const void* dw_b,
                                const int32_t* mid_len, const int32_t* out_len, int64_t B, int64_t T, int64_t F, int64_t C, int dtype,
                                void* stream) {
  using namespace ob;
  using namespace ob::stem_dw;
  OB_REQUIRE(B >= 0 && B < 65536 && T >= 1 && T < (1 << 30) && F >= 1 && C >= 1, OASR_ERR_INVALID, "subsample_stem_dw: bad shape");
  OB_REQUIRE(fits(F, C), OASR_ERR_UNSUPPORTED, "subsample_stem_dw: channels / 4 must divide %d and the frames fit shared memory (got F %lld, C %lld)",
             kThreads, (long long)F, (long long)C);
  if (B == 0) return OASR_OK;
  OB_REQUIRE(out && in && stem_w && stem_b && dw_w, OASR_ERR_INVALID, "subsample_stem_dw: null pointer argument");
  OB_REQUIRE(is_aligned(out, 8), OASR_ERR_ALIGN, "subsample_stem_dw: out must be 8-byte aligned");
  Params p{};
  p.out = out; p.in = in; p.w1 = stem_w; p.b1 = stem_b; p.w2 = dw_w; p.b2 = dw_b; p.mid_len = mid_len; p.out_len = out_len;
  p.T = (int)T; p.F = (int)F; p.C = (int)C; p.T1 = (int)(T / 2 + 1); p.F1 = (int)(F / 2 + 1);
  p.To = p.T1 / 2 + 1; p.Fo = p.F1 / 2 + 1; p.pitch = pitch_of(F);
  const int rows = kThreads / (int)(C / 4);
  const int64_t blocks = (p.To + rows - 1) / rows * B;
  // a thread walks the whole frequency axis, or a quarter of it where that leaves SMs without their two blocks
  const int pieces = blocks >= 2 * sm_count() ? 1 : (p.Fo < 4 ? p.Fo : 4);
  p.fstep = (p.Fo + pieces - 1) / pieces;
  const dim3 grid(static_cast<unsigned>((p.To + rows - 1) / rows), static_cast<unsigned>(B), static_cast<unsigned>((p.Fo + p.fstep - 1) / p.fstep));
  return OB_DISPATCH_HALF(dtype, T_, [&]() -> int {
    stem_dw_kernel<T_><<<grid, kThreads, static_cast<size_t>(smem_bytes(F, C)), static_cast<cudaStream_t>(stream)>>>(p);
    return check_launch("subsample_stem_dw launch");
  });
}

}  // extern "C"
