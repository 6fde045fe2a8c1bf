// Kaldi-compatible log-mel filterbank features (FBANK) with optional global CMVN, one fused kernel:
//   frame (snip_edges) -> subtract the frame's mean -> pre-emphasis (first sample replicated) -> analysis window ->
//   zero-pad to n_fft -> power spectrum -> mel filterbank -> log(max(., floor)) -> (x - mean) * istd
// It replaces the reference's kernel chain stft_frame -> rfft_power -> mel_log (launchers csrc/features.cu:39-205,
// composed by oasr/features/batched.py:171-206; arithmetic of the torch route batched.py:209-268) and GlobalCMVN
// (oasr/layers/norm.py:571-584): frames, spectra and mel energies never reach HBM.
//
// Two kernels.  n_fft = 512 (25 ms at 16 kHz), fbank512_kernel: a warp takes two consecutive frames at a time.  The same
// radix-2 butterflies with the same roundings as the general kernel, but in registers: a lane holds 8 of a frame's 256
// complex values and runs three (three, two) stages between two exchanges through shared memory whose layouts have no bank
// conflicts; its twiddles stay in registers over all frames, the two frames share them, their overlapping samples, the
// mel weights and every arithmetic instruction (packed fp32 pairs), and the samples of the next pair are in flight under the
// current one.  64 utterances of 2-20 s: 404 -> 118 us (1.8k warp instructions per pair of frames at 0.5 per clock and
// scheduler).  Bound by issue and shared-memory latency at 16 warps per SM (128 registers; 96 spill); its 87 MB would take
// 13 us at the copy rate.  The roundings matter: a weak band under a strong tone keeps few digits, and a radix-8 form with
// both frames as one complex signal (137 us) differed there by as much as the general kernel differs from the exact value.
//
// Other sizes, fbank_kernel: one warp per frame.  The real FFT of n_fft points is a complex FFT of n_fft/2 points on z[n] = x[2n] + i x[2n+1]
// (radix-2, decimation in time, in shared memory, one __syncwarp per stage) followed by the usual split; all
// twiddles come from one table W[k] = exp(-2 pi i k / n_fft), k < n_fft/2, built per block.  The mel filterbank is
// applied from the dense (num_mel, n_fft/2+1) matrix the reference builds, but only over each filter's non-zero
// bin range.  HBM-bound in principle (4 B in per hop sample, 4 B out per mel bin); in practice a few dozen
// microseconds for a batch of a thousand audio-seconds, so the instruction count of the FFT is what it costs.
#include "common.cuh"

namespace ob {
namespace features {

constexpr int kWarps = 4;
constexpr int kMaxFft = 2048;

struct Args {
  const float* wave;       // (B, T)
  const int32_t* lengths;  // (B) samples, nullable = every row is T samples long
  const float* window;     // (frame_length)
  const float* mel;        // (num_mel, n_fft/2 + 1)
  const int32_t* mel_lo;   // (num_mel) first non-zero bin
  const int32_t* mel_hi;   // (num_mel) one past the last non-zero bin
  const float* cmvn_mean;  // (num_mel), nullable
  const float* cmvn_istd;  // (num_mel), nullable
  float* out;              // (B, num_frames, num_mel)
  int64_t B, T;
  int num_frames, frame_length, frame_shift, n_fft, log2_half, num_mel;
  float preemph, log_floor;
};

__global__ void __launch_bounds__(kWarps * 32) fbank_kernel(Args a) {
  extern __shared__ float fb_smem[];
  const int N = a.n_fft, Nh = N >> 1;
  float2* tw = reinterpret_cast<float2*>(fb_smem);                       // Nh entries
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* bufA = fb_smem + 2 * Nh + warp * (2 * N + 2);                   // N + 2 floats: samples, later the power spectrum
  float2* z = reinterpret_cast<float2*>(bufA + N + 2);                   // Nh complex values
  for (int k = threadIdx.x; k < Nh; k += blockDim.x) {
    float s, c;
    sincospif(2.0f * static_cast<float>(k) / static_cast<float>(N), &s, &c);
    tw[k] = make_float2(c, -s);
  }
  __syncthreads();
  const int64_t total = a.B * a.num_frames;
  const int L = a.frame_length;
  for (int64_t f = static_cast<int64_t>(blockIdx.x) * kWarps + warp; f < total; f += static_cast<int64_t>(gridDim.x) * kWarps) {
    const int64_t b = f / a.num_frames;
    const int t = static_cast<int>(f - b * a.num_frames);
    float* out = a.out + f * a.num_mel;
    const int64_t len = a.lengths ? a.lengths[b] : a.T;
    const int64_t start = static_cast<int64_t>(t) * a.frame_shift;
    if (start + L > len) {                       // not a whole frame of this utterance: outside its feature length
      for (int m = lane; m < a.num_mel; m += 32) out[m] = 0.f;
      continue;
    }
    const float* x = a.wave + b * a.T + start;
    // samples and their mean
    float sum = 0.f;
    for (int n = lane; n < L; n += 32) {
      const float v = x[n];
      bufA[n] = v;
      sum += v;
    }
    const float mean = warp_sum(sum) / static_cast<float>(L);
    __syncwarp();
    // DC removal, pre-emphasis, window, zero padding; packed as z[m] = y[2m] + i y[2m+1] at the bit-reversed index
    const int shift = 32 - a.log2_half;
    for (int m = lane; m < Nh; m += 32) {
      float y[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = 2 * m + e;
        float v = 0.f;
        if (n < L) {
          const float cur = bufA[n] - mean;
          const float prev = bufA[n > 0 ? n - 1 : 0] - mean;
          v = (cur - a.preemph * prev) * a.window[n];
        }
        y[e] = v;
      }
      z[__brev(static_cast<unsigned>(m)) >> shift] = make_float2(y[0], y[1]);
    }
    __syncwarp();
    // complex FFT of Nh points, radix 2: stage s joins blocks of half = 2^s
    for (int half = 1; half < Nh; half <<= 1) {
      const int tw_step = N / (2 * half) ;       // W_{2*half}^j = W_N^{j * N / (2*half)}
      for (int i = lane; i < (Nh >> 1); i += 32) {
        const int j = i & (half - 1);
        const int lo = ((i - j) << 1) + j;
        const float2 w = tw[j * tw_step];
        const float2 u = z[lo], v = z[lo + half];
        const float2 wv = make_float2(w.x * v.x - w.y * v.y, w.x * v.y + w.y * v.x);
        z[lo] = make_float2(u.x + wv.x, u.y + wv.y);
        z[lo + half] = make_float2(u.x - wv.x, u.y - wv.y);
      }
      __syncwarp();
    }
    // split into the spectrum of the real signal: X[k] = (Z[k] + conj Z[Nh-k]) / 2 - i W_N^k (Z[k] - conj Z[Nh-k]) / 2
    float* power = bufA;
    for (int k = lane; k <= Nh; k += 32) {
      const float2 zk = z[k == Nh ? 0 : k];
      const float2 zc = z[(Nh - k) == Nh ? 0 : (Nh - k)];
      const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);      // even part
      const float orr = 0.5f * (zk.x - zc.x), oi = 0.5f * (zk.y + zc.y);     // (Z[k] - conj Z[Nh-k]) / 2
      float2 w = k == Nh ? make_float2(-1.f, 0.f) : tw[k];
      // -i * w * (orr + i oi) = -i * ((w.x*orr - w.y*oi) + i (w.x*oi + w.y*orr)) = (w.x*oi + w.y*orr) - i (w.x*orr - w.y*oi)
      const float xr = er + (w.x * oi + w.y * orr);
      const float xi = ei - (w.x * orr - w.y * oi);
      power[k] = xr * xr + xi * xi;
    }
    __syncwarp();
    const int nfreq = Nh + 1;
    for (int m = lane; m < a.num_mel; m += 32) {
      const float* row = a.mel + static_cast<int64_t>(m) * nfreq;
      float acc = 0.f;
      for (int k = a.mel_lo[m]; k < a.mel_hi[m]; ++k) acc = fmaf(power[k], __ldg(row + k), acc);
      float v = logf(fmaxf(acc, a.log_floor));
      if (a.cmvn_mean) v = (v - a.cmvn_mean[m]) * a.cmvn_istd[m];
      out[m] = v;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// n_fft = 512
// ---------------------------------------------------------------------------
constexpr int kWarps512 = 4;
constexpr int kExch = 288;            // 256 complex values of both frames, value P at P + P / 8
constexpr int kSpan = 768;            // samples of two frames: frame_length + frame_shift at most
constexpr int kMelCap = 1024;         // weights of the filters' non-zero ranges kept in shared memory
constexpr int kMelMax = 128;

// A number of each of the two frames in one 64-bit register pair, and the packed fp32 arithmetic on it (each half rounds as
// the scalar instruction does).
typedef unsigned long long Two;
__device__ __forceinline__ Two two(float a, float b) {
  Two r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 halves(Two v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ Two add2(Two a, Two b) { Two r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ Two sub2(Two a, Two b) { Two r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ Two mul2(Two a, Two b) { Two r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) { Two r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
struct C2 { Two x, y; };              // a complex number of each frame

// Radix-2 butterflies of the general kernel: (u, v) -> (u + w v, u - w v), both frames at once.
__device__ __forceinline__ void butterfly(C2& u, C2& v, float2 w) {
  const Two wx = two(w.x, w.x), wy = two(w.y, w.y), ny = two(-w.y, -w.y);
  const C2 s = u, wv{fma2(wx, v.x, mul2(ny, v.y)), fma2(wx, v.y, mul2(wy, v.x))};
  u.x = add2(s.x, wv.x); u.y = add2(s.y, wv.y);
  v.x = sub2(s.x, wv.x); v.y = sub2(s.y, wv.y);
}
__device__ __forceinline__ void butterfly_1(C2& u, C2& v) {    // w = 1
  const C2 s = u, t = v;
  u.x = add2(s.x, t.x); u.y = add2(s.y, t.y);
  v.x = sub2(s.x, t.x); v.y = sub2(s.y, t.y);
}
__device__ __forceinline__ void butterfly_mi(C2& u, C2& v) {   // w = -i
  const C2 s = u, t = v;
  u.x = add2(s.x, t.y); u.y = sub2(s.y, t.x);
  v.x = sub2(s.x, t.y); v.y = add2(s.y, t.x);
}

// kL, kHop: frame length and shift known at compile time (25 / 10 ms at 16 kHz); 0: taken from the arguments.
template <int kL, int kHop>
__global__ void __launch_bounds__(kWarps512 * 32, 4) fbank512_kernel(Args a) {
  __shared__ float2 tw[256];                       // exp(-2 pi i k / 512)
  __shared__ __align__(16) C2 exch_all[kWarps512][kExch];
  __shared__ __align__(16) float span_all[kWarps512][kSpan];
  __shared__ Two mel_w[kMelCap];                   // each weight twice, one per frame
  __shared__ int mel_at[kMelMax + 1], mel_lo[kMelMax];   // start of a filter's weights in mel_w, its first bin
  __shared__ float2 cmvn[kMelMax];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = threadIdx.x; k < 256; k += blockDim.x) {
    float s, c;
    sincospif(2.0f * static_cast<float>(k) / 512.0f, &s, &c);
    tw[k] = make_float2(c, -s);
  }
  for (int m = threadIdx.x; m < a.num_mel; m += blockDim.x) {
    mel_lo[m] = a.mel_lo[m];
    mel_at[m + 1] = max(0, a.mel_hi[m] - a.mel_lo[m]);
    cmvn[m] = a.cmvn_mean ? make_float2(a.cmvn_mean[m], a.cmvn_istd[m]) : make_float2(0.f, 1.f);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mel_at[0] = 0;
    for (int m = 0; m < a.num_mel; ++m) mel_at[m + 1] += mel_at[m];
  }
  __syncthreads();
  const bool compact = mel_at[a.num_mel] <= kMelCap;
  if (compact) {
    for (int m = warp; m < a.num_mel; m += kWarps512)
      for (int k = lane; k < mel_at[m + 1] - mel_at[m]; k += 32) {
        const float w = a.mel[static_cast<int64_t>(m) * 257 + mel_lo[m] + k];
        mel_w[mel_at[m] + k] = two(w, w);
      }
  }
  __syncthreads();
  float* span = span_all[warp];
  C2* z = exch_all[warp];
  const int L = kL ? kL : a.frame_length, hop = kHop ? kHop : a.frame_shift, n_span = L + hop;
  // Positions P of the bit-reversed array: phase 1 (stages of distance 1, 2, 4) holds P = 8 lane + r, whose value is the
  // sample pair brev8(P); phase 2 (8, 16, 32) P = (lane & 7) + 8 r + 64 (lane >> 3); phase 3 (64, 128) P = lane + 32 q.
  const int pair0 = __brev(lane) >> 27;            // + 32 * brev3(r)
  constexpr int kRev3[8] = {0, 4, 2, 6, 1, 5, 3, 7};
  float2 win[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int n = 2 * (pair0 + 32 * kRev3[r]);
    win[r] = make_float2(n < L ? a.window[n] : 0.f, n + 1 < L ? a.window[n + 1] : 0.f);
  }
  const float2 w8_1 = tw[64], w8_3 = tw[192];
  const int j2 = lane & 7;
  const float2 w3 = tw[32 * j2], w4[2] = {tw[16 * j2], tw[16 * (j2 + 8)]}, w5[4] = {tw[8 * j2], tw[8 * (j2 + 8)], tw[8 * (j2 + 16)], tw[8 * (j2 + 24)]};
  const float2 w6[2] = {tw[4 * lane], tw[4 * (lane + 32)]}, w7[4] = {tw[2 * lane], tw[2 * (lane + 32)], tw[2 * (lane + 64)], tw[2 * (lane + 96)]};
  const int at1 = 9 * lane, at2 = (lane & 7) + 72 * (lane >> 3), at3 = lane + (lane >> 3);   // padded: + r, + 9 r, + 36 q
  constexpr int kAhead = kL ? (kL + kHop + 31) / 32 : 18;   // samples of the next pair a lane holds (the rest is loaded when needed)
  float next[kAhead];
  // pair f of the batch = frames t, t + 1 of utterance b; both advance without divisions
  const int pairs = (a.num_frames + 1) / 2;
  const int step = static_cast<int>(gridDim.x) * kWarps512, step_b = step / pairs, step_t = step - step_b * pairs;
  const int first = static_cast<int>(blockIdx.x) * kWarps512 + warp;
  int b = first / pairs, pt = first - b * pairs;
  auto whole_frames = [&](int bb, int p) -> int {  // of the pair: 0, 1, 2
    const int64_t len = a.lengths ? a.lengths[bb] : a.T, end = static_cast<int64_t>(2 * p) * hop + L;
    return end > len ? 0 : (2 * p + 1 < a.num_frames && end + hop <= len ? 2 : 1);
  };
  auto fetch = [&](int bb, int p, int live) {
    const int n_in = live == 2 ? n_span : (live == 1 ? L : 0);
    const float* x = a.wave + (live ? bb * a.T + static_cast<int64_t>(2 * p) * hop : 0) + lane;
#pragma unroll
    for (int i = 0; i < kAhead; ++i) next[i] = 32 * i + lane < n_in ? x[32 * i] : 0.f;
  };
  int live = b < a.B ? whole_frames(b, pt) : 0;
  fetch(b, pt, live);
  while (b < a.B) {
    int nb = b + step_b, npt = pt + step_t;
    if (npt >= pairs) { npt -= pairs; ++nb; }
    const int next_live = nb < a.B ? whole_frames(nb, npt) : 0;
    const bool both = 2 * pt + 1 < a.num_frames;
    float* out = a.out + (static_cast<int64_t>(b) * a.num_frames + 2 * pt) * a.num_mel;
    if (live == 0) {                               // no whole frame of this utterance: outside its feature length
      for (int m = lane; m < (both ? 2 : 1) * a.num_mel; m += 32) out[m] = 0.f;
      fetch(nb, npt, next_live);
    } else {
      // Sums of the frames' samples, lane by lane in steps of 32 from each frame's start
      float sum0 = 0.f, sum1 = 0.f;
      if constexpr (kL > 0 && kHop % 32 == 0) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          if (32 * i < kL) sum0 += 32 * i + 31 < kL || 32 * i + lane < kL ? next[i] : 0.f;
          if (32 * i >= kHop) sum1 += next[i];
        }
      }
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
        if (32 * i + lane < n_span) span[32 * i + lane] = next[i];
      for (int n = 32 * kAhead + lane; n < n_span; n += 32)
        span[n] = live == 2 || n < L ? a.wave[b * a.T + static_cast<int64_t>(2 * pt) * hop + n] : 0.f;
      __syncwarp();
      if constexpr (!(kL > 0 && kHop % 32 == 0)) {
        for (int n = lane; n < L; n += 32) {
          sum0 += span[n];
          sum1 += span[n + hop];
        }
      }
      fetch(nb, npt, next_live);
      const float mean0 = warp_sum(sum0) / static_cast<float>(L), mean1 = warp_sum(sum1) / static_cast<float>(L);
      const Two mean = two(mean0, mean1), npre = two(-a.preemph, -a.preemph);
      // DC removal, pre-emphasis (the first sample is its own predecessor), window, zero padding
      C2 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        v[r] = C2{0ull, 0ull};
        if (kL && 64 * kRev3[r] >= kL) continue;
        const int n = 2 * (pair0 + 32 * kRev3[r]);
        if ((kL && 64 * kRev3[r] + 63 < kL) || n < L) {
          const float* x0 = span + n;
          const float* x1 = x0 + hop;
          const int back = n > 0 ? -1 : 0;
          const bool odd = (kL && kL % 2 == 0) || n + 1 < L;
          const Two c0 = sub2(two(x0[0], x1[0]), mean), p0 = sub2(two(x0[back], x1[back]), mean);
          const Two c1 = sub2(two(odd ? x0[1] : mean0, odd ? x1[1] : mean1), mean);
          v[r].x = mul2(fma2(npre, p0, c0), two(win[r].x, win[r].x));
          v[r].y = mul2(fma2(npre, c0, c1), two(win[r].y, win[r].y));
        }
      }
      butterfly_1(v[0], v[1]); butterfly_1(v[2], v[3]); butterfly_1(v[4], v[5]); butterfly_1(v[6], v[7]);
      butterfly_1(v[0], v[2]); butterfly_mi(v[1], v[3]); butterfly_1(v[4], v[6]); butterfly_mi(v[5], v[7]);
      butterfly_1(v[0], v[4]); butterfly(v[1], v[5], w8_1); butterfly_mi(v[2], v[6]); butterfly(v[3], v[7], w8_3);
#pragma unroll
      for (int r = 0; r < 8; ++r) z[at1 + r] = v[r];
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = z[at2 + 9 * r];
#pragma unroll
      for (int r = 0; r < 8; r += 2) butterfly(v[r], v[r + 1], w3);
#pragma unroll
      for (int r = 0; r < 8; r += 4) {
        butterfly(v[r], v[r + 2], w4[0]);
        butterfly(v[r + 1], v[r + 3], w4[1]);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) butterfly(v[r], v[r + 4], w5[r]);
#pragma unroll
      for (int r = 0; r < 8; ++r) z[at2 + 9 * r] = v[r];
      __syncwarp();
      // P = lane + 32 q: distance 64 = q + 2, distance 128 = q + 4
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = z[at3 + 36 * q];
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        butterfly(v[q], v[q + 2], w6[0]);
        butterfly(v[q + 1], v[q + 3], w6[1]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) butterfly(v[q], v[q + 4], w7[q]);
      __syncwarp();
      // Spectrum of the real signal, X[k] = (Z[k] + conj Z[256-k]) / 2 - i W^k (Z[k] - conj Z[256-k]) / 2; Z[256-k] is value
      // 7 - q of lane 32 - lane (lane 0: its own 8 - q)
      Two* power = reinterpret_cast<Two*>(z);      // (frame, next frame) per bin
      const Two half = two(0.5f, 0.5f);
      auto bin_power = [&](const C2& zk, const C2& zc, float2 w) -> Two {
        const Two er = mul2(half, add2(zk.x, zc.x)), ei = mul2(half, sub2(zk.y, zc.y));      // even part
        const Two orr = mul2(half, sub2(zk.x, zc.x)), oi = mul2(half, add2(zk.y, zc.y));     // (Z[k] - conj Z[256-k]) / 2
        const Two wx = two(w.x, w.x), wy = two(w.y, w.y), ny = two(-w.y, -w.y);
        const Two xr = add2(er, fma2(wx, oi, mul2(wy, orr)));
        const Two xi = sub2(ei, fma2(wx, orr, mul2(ny, oi)));
        return fma2(xr, xr, mul2(xi, xi));
      };
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        C2 zc;
        zc.x = __shfl_sync(0xffffffffu, v[7 - q].x, (32 - lane) & 31);
        zc.y = __shfl_sync(0xffffffffu, v[7 - q].y, (32 - lane) & 31);
        if (lane == 0) zc = v[(8 - q) & 7];
        power[lane + 32 * q] = bin_power(v[q], zc, tw[lane + 32 * q]);
      }
      if (lane == 0) power[256] = bin_power(v[0], v[0], make_float2(-1.f, 0.f));
      __syncwarp();
      for (int m = lane; m < a.num_mel; m += 32) {
        const int lo = mel_lo[m], at = mel_at[m], n = mel_at[m + 1] - at;
        const Two* pw = power + lo;
        Two e = 0ull;
        if (compact) {
#pragma unroll 4
          for (int i = 0; i < n; ++i) e = fma2(pw[i], mel_w[at + i], e);
        } else {
          const float* w = a.mel + static_cast<int64_t>(m) * 257 + lo;
          for (int i = 0; i < n; ++i) e = fma2(pw[i], two(w[i], w[i]), e);
        }
        const float2 ee = halves(e);
        float l0 = logf(fmaxf(ee.x, a.log_floor)), l1 = logf(fmaxf(ee.y, a.log_floor));
        if (a.cmvn_mean) {
          l0 = (l0 - cmvn[m].x) * cmvn[m].y;
          l1 = (l1 - cmvn[m].x) * cmvn[m].y;
        }
        out[m] = l0;
        if (both) out[a.num_mel + m] = live == 2 ? l1 : 0.f;
      }
      __syncwarp();
    }
    b = nb;
    pt = npt;
    live = next_live;
  }
}

}  // namespace features
}  // namespace ob

extern "C" {

int oasr_b200_fbank(float* out, const float* waveforms, const int32_t* lengths, const float* window, const float* mel_mat,
                    const int32_t* mel_lo, const int32_t* mel_hi, const float* cmvn_mean, const float* cmvn_istd,
                    int64_t B, int64_t T, int64_t num_frames, int64_t frame_length, int64_t frame_shift, int64_t n_fft,
                    int64_t num_mel, double preemph, double log_floor, void* stream) {
  using namespace ob;
  using namespace ob::features;
  OB_REQUIRE(B >= 0 && T >= 0 && num_frames >= 0 && num_mel > 0, OASR_ERR_INVALID, "fbank: bad shape");
  if (B == 0 || num_frames == 0) return OASR_OK;
  OB_REQUIRE(out && waveforms && window && mel_mat && mel_lo && mel_hi, OASR_ERR_INVALID, "fbank: null pointer argument");
  OB_REQUIRE((cmvn_mean == nullptr) == (cmvn_istd == nullptr), OASR_ERR_INVALID, "fbank: CMVN needs both mean and istd");
  OB_REQUIRE(n_fft >= 64 && n_fft <= kMaxFft && (n_fft & (n_fft - 1)) == 0, OASR_ERR_UNSUPPORTED,
             "fbank: n_fft must be a power of two in [64, %d] (got %lld)", kMaxFft, (long long)n_fft);
  OB_REQUIRE(frame_length >= 2 && frame_length <= n_fft && frame_shift > 0, OASR_ERR_INVALID,
             "fbank: frame length %lld / shift %lld do not fit n_fft %lld", (long long)frame_length, (long long)frame_shift,
             (long long)n_fft);
  OB_REQUIRE((num_frames - 1) * frame_shift + frame_length <= T, OASR_ERR_INVALID,
             "fbank: %lld frames do not fit %lld samples", (long long)num_frames, (long long)T);
  Args a{};
  a.wave = waveforms; a.lengths = lengths; a.window = window; a.mel = mel_mat; a.mel_lo = mel_lo; a.mel_hi = mel_hi;
  a.cmvn_mean = cmvn_mean; a.cmvn_istd = cmvn_istd; a.out = out;
  a.B = B; a.T = T;
  a.num_frames = static_cast<int>(num_frames); a.frame_length = static_cast<int>(frame_length);
  a.frame_shift = static_cast<int>(frame_shift); a.n_fft = static_cast<int>(n_fft); a.num_mel = static_cast<int>(num_mel);
  int lg = 0;
  while ((int64_t(1) << lg) < n_fft / 2) ++lg;
  a.log2_half = lg;
  a.preemph = static_cast<float>(preemph); a.log_floor = static_cast<float>(log_floor);
  const int64_t total = B * num_frames;
  if (n_fft == 512 && num_mel <= kMelMax && frame_length + frame_shift <= kSpan && B * ((num_frames + 1) / 2) < (int64_t(1) << 30)) {
    const int64_t pairs = B * ((num_frames + 1) / 2);
    int64_t g = (pairs + kWarps512 - 1) / kWarps512;
    if (g > static_cast<int64_t>(sm_count()) * 4) g = static_cast<int64_t>(sm_count()) * 4;   // resident at once: tables are built per block
    const bool standard = frame_length == 400 && frame_shift == 160;
    (standard ? fbank512_kernel<400, 160> : fbank512_kernel<0, 0>)<<<static_cast<unsigned>(g), kWarps512 * 32, 0, static_cast<cudaStream_t>(stream)>>>(a);
    return check_launch("fbank launch");
  }
  int64_t grid = (total + kWarps - 1) / kWarps;
  const int64_t cap = static_cast<int64_t>(sm_count()) * 16;
  if (grid > cap) grid = cap;
  // twiddle table (n_fft/2 complex) + per warp n_fft + 2 floats of samples / power and n_fft/2 complex values
  const size_t smem = sizeof(float) * (static_cast<size_t>(n_fft) + kWarps * (2 * static_cast<size_t>(n_fft) + 2));
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(fbank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return set_error(OASR_ERR_CUDA, "fbank: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  }
  fbank_kernel<<<static_cast<unsigned>(grid), kWarps * 32, smem, static_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("fbank launch");
}

}  // extern "C"
