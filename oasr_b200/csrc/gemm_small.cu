// GEMM for few rows (M up to a few thousand): D[M,N] = epilogue(A[M,K] . B[N,K]^T + bias[N]), A/B fp16 or bf16, fp32
// accumulate.
//
// What bounds these problems is not the tensor pipe but the chain a single tile runs through: launch, descriptor and
// operand latency, a serial K loop on few CTAs, the epilogue, the next launch.  So, against the persistent kernel of
// gemm.cu:
//   * K is split over the CTAs of a cluster (S = 1, 2, 4, 8; about 512 elements of K per CTA).  Each CTA accumulates its
//     slice of K for the whole 128 x BN tile in tensor memory, sends column slices of the partial sums to the CTA that
//     owns them (distributed shared memory, no atomics, no scratch in HBM), and the owner adds the S partials in rank
//     order.  A 2048-deep product of 78 rows went from 25 us on 8 CTAs to about 5 us on 64.
//   * one tile per CTA, about 100 KB of shared memory, so two CTAs share an SM: with programmatic dependent launch the
//     next GEMM of the stream is resident, has its barriers and tensor memory, and has its first WEIGHT tiles in flight
//     (b_static) before this one has finished; only the A tiles wait for the previous kernel.
//   * narrow tiles (BN 32 / 64 / 128) chosen so that as many SMs as possible pull operand bytes: an SM takes about 50 B
//     per clock from L2, and operand bytes per SM are what is left of the time.
//   * few barriers: a stage is several K blocks, fetched by one TMA instruction per operand (the K blocks are a tensor
//     dimension of their own; only rows that exist are fetched), and where the grid leaves SMs free the whole K slice is
//     resident, so that nothing is ever refilled.  A successful mbarrier wait costs its thread about 0.2k clocks and a
//     refill a round trip through MMA, commit, producer and L2: 8 single-block stages took 2.3 us for 16 rows.
//   * the exchange is pushed (st.async credited to the owner's mbarrier), so that an owner waits for its data and not for
//     a cluster-wide barrier.
// The number of splits depends on N and K only, and a tile's K order never depends on M; unsplit products give the bits of
// gemm.cu.  So a row's result does not depend on the rows that share its batch for all unsplit products, and up to kMaxRows
// for all outputs of up to 512 columns.  A split product of a wider output changes its order of sums where takes() hands it
// to gemm.cu.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer and tensor-memory owner, the other 4 (128-wide tiles: 8) epilogue, a
// thread per row (and column half); output goes through padded shared memory so that global accesses are coalesced.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "device_status.cuh"
#include "gemm_small.cuh"
#include "sm100_ptx.cuh"
#include "smem_limit.cuh"
#include "tma_host.cuh"

namespace ob {
namespace gsm {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kMaxStages = 8;

struct Params {
  int M, N;               // rows, output columns of the product (GLU: output columns, the weight has 2N rows)
  int kb_total, kb_per;   // K blocks of 64, and how many of them one CTA of a cluster takes
  int k_whole;            // K is a multiple of 64: the K blocks are a tensor dimension
  int kg, stages;         // K blocks per stage, stages of the ring
  int a_blk;              // bytes of one K block of A: the rows that exist (rounded to 8) x 128
  int ldd;                // output row stride in elements
  int dup_cols;           // kDup: the first dup_cols columns of the product are stored twice
  int act;
  int b_static;           // B does not depend on earlier kernels of the stream: prefetch it before the dependency wait
  int late_launch;        // let the next kernel start only after everything before this one is complete and visible
  float alpha;
  const float* R_in;      // kResid, nullable
  const void* bias;       // nullable
  void* D;
  uint32_t* status;
};

// Shared memory: [bias][barriers] [exchange buffer] [stages, each A blocks then B blocks] [16 KB that MMAs of fewer than
// 128 fetched rows may read past the last A block].
template <int BN, int S>
struct Geo {
  static constexpr int kBBlk = BN * BK * 2;                       // one K block of B
  static constexpr int kW = BN / S;                               // columns of the tile this CTA owns after the exchange
  static constexpr int kHead = 2048;                              // 2 * BN floats of bias, 2 * kMaxStages + 2 barriers, flags
  static constexpr int kRecv = (S - 1) * kW * BM * 4;            // [other rank][4-column group][row] float4
  static constexpr int kEpiWarps = BN == 128 ? 8 : 4;
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr int kHalves = kEpiWarps / 4;                   // epilogue warps that share a row
  static constexpr int kWH = kW / kHalves;                        // columns of one epilogue thread
  static constexpr int kStaging = kEpiWarps * 32 * (kWH + 4) * 4; // the output staging reuses the operand ring
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 16 bytes into another CTA's shared memory, credited to an mbarrier of that CTA.
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
               : "memory");
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

template <int kCols>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t* r) {
  static_assert(kCols == 8 || kCols == 16 || kCols == 32, "columns of one tensor-memory load");
  if constexpr (kCols == 32) ptx::tmem_ld_32x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(r));
  else if constexpr (kCols == 16) ptx::tmem_ld_32x16(taddr, *reinterpret_cast<uint32_t(*)[16]>(r));
  else ptx::tmem_ld_32x8(taddr, *reinterpret_cast<uint32_t(*)[8]>(r));
}

// S = CTAs of a cluster that share one tile's K range.
template <typename T, int BN, int S, int kEpi>
__global__ void __launch_bounds__(Geo<BN, S>::kThreads, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const Params p) {
  using G = Geo<BN, S>;
  constexpr int W = G::kW;
  constexpr uint32_t kIdesc = ptx::umma_idesc_f16(std::is_same<T, __nv_bfloat16>::value, BM, BN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* sbias = reinterpret_cast<float*>(smem);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + 2 * BN * 4);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* tfull_bar = empty_bar + kMaxStages;
  uint64_t* recv_bar = tfull_bar + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv_bar + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float4* recv = reinterpret_cast<float4*>(smem + G::kHead);
  uint8_t* ring = smem + G::kHead + G::kRecv;
  const int kSt = p.stages, KG = p.kg;
  const int stage_bytes = KG * (p.a_blk + G::kBBlk);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp-uniform for the compiler
  const int rank = S == 1 ? 0 : static_cast<int>(ptx::cluster_ctarank());
  const int nt = blockIdx.x / S;
  const int m0 = blockIdx.y * BM;
  const int n0 = nt * BN;                       // first accumulator column (GLU: 2x the first output column)
  const int kb0 = rank * p.kb_per;
  const int nkb = min(p.kb_per, p.kb_total - kb0);
  const int nst = (nkb + KG - 1) / KG;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSt; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    ptx::mbar_init(tfull_bar, 1);
    ptx::mbar_init(recv_bar, 1);
    *abort_flag = 0;
    ptx::fence_barrier_init();
    if constexpr (S > 1) ptx::mbar_expect_tx(recv_bar, (S - 1) * W * BM * 4);
    ptx::prefetch_tensormap(&tmap_b);
    ptx::prefetch_tensormap(&tmap_a);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, BN);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (p.late_launch) ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  if constexpr (S > 1) cluster_arrive();        // waited for before the exchange: every CTA of the cluster has its barriers

  // stage `st` of this CTA's K range: coordinates (0, row, half, K block), or (K, row, half, 0) with one block per stage
  auto load_b = [&](int st, int slot) {
    const int kb = kb0 + st * KG;
    ptx::tma_load_4d(ring + slot * stage_bytes + KG * p.a_blk, &tmap_b, p.k_whole ? 0 : kb * BK, kEpi == kGlu ? n0 / 2 : n0, 0, p.k_whole ? kb : 0,
                     &full_bar[slot]);
  };
  if (warp == 0) {
    // whole warp, one elected lane issues (see the MMA warp)
    const bool issuer = ptx::elect_one();
    const int ahead = p.b_static ? min(kSt, nst) : 0;
    if (issuer) {
      for (int st = 0; st < ahead; ++st) {
        ptx::mbar_expect_tx(&full_bar[st], stage_bytes);
        load_b(st, st);
      }
    }
    ptx::grid_dep_wait();
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int st = 0; st < nst; ++st) {
      if (st >= kSt && !ptx::mbar_wait(&empty_bar[slot], phase ^ 1u, abort_flag)) { ok = false; break; }
      const int kb = kb0 + st * KG;
      if (issuer) {
        if (st >= ahead) ptx::mbar_expect_tx(&full_bar[slot], stage_bytes);
        ptx::tma_load_3d(ring + slot * stage_bytes, &tmap_a, p.k_whole ? 0 : kb * BK, m0, p.k_whole ? kb : 0, &full_bar[slot]);
        if (st >= ahead) load_b(st, slot);
      }
      if (++slot == kSt) { slot = 0; phase ^= 1u; }
    }
    if (!ok && issuer && p.status) atomicOr(p.status, kStatusGemmProducer);
    __syncwarp();
    if constexpr (S > 1) cluster_wait();
  } else if (warp == 1) {
    // The whole warp runs the loop and one elected lane issues: the descriptors then stay in uniform registers, where the
    // instruction wants them.  Under `lane == 0` each MMA took 0.14k clocks to issue, whatever its width.
    const bool issuer = ptx::elect_one();
    int slot = 0;
    uint32_t phase = 0, accumulate = 0;
    bool ok = true;
    for (int st = 0; st < nst; ++st) {
      if (!ptx::mbar_wait(&full_bar[slot], phase, abort_flag)) { ok = false; break; }
      ptx::tc_fence_after_sync();
      const uint32_t a_addr = ptx::smem_u32(ring) + slot * stage_bytes;
      uint64_t ad = ptx::smem_desc_kmajor_sw128(a_addr), bd = ptx::smem_desc_kmajor_sw128(a_addr + KG * p.a_blk);
      const int blocks = min(KG, nkb - st * KG);
      for (int g = 0; g < blocks; ++g) {
        if (issuer) {
          ptx::umma_f16(tmem_base, ad, bd, kIdesc, accumulate);
          ptx::umma_f16(tmem_base, ad + 2, bd + 2, kIdesc, 1u);      // 16 elements of K = 32 bytes = 2 descriptor units
          ptx::umma_f16(tmem_base, ad + 4, bd + 4, kIdesc, 1u);
          ptx::umma_f16(tmem_base, ad + 6, bd + 6, kIdesc, 1u);
        }
        accumulate = 1u;
        ad += p.a_blk >> 4;
        bd += G::kBBlk >> 4;
      }
      if (issuer) ptx::umma_commit(&empty_bar[slot]);
      if (++slot == kSt) { slot = 0; phase ^= 1u; }
    }
    if (issuer) {
      if (ok) ptx::umma_commit(tfull_bar);
      else if (p.status) atomicOr(p.status, kStatusGemmMma);
    }
    __syncwarp();
    if constexpr (S > 1) cluster_wait();
  } else {
    // ------------------------------ epilogue ----------------------------------
    constexpr int WH = G::kWH;
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;             // 128-wide tiles: which half of the columns
    const int row = q * 32 + lane;                // row of the tile = tensor-memory lane
    // columns of the tile this CTA finishes: [own0, own0 + W), GLU: W/2 value columns and the W/2 gate columns behind them;
    // this thread: kOutW output columns from `hc` on
    constexpr int kOutAll = kEpi == kGlu ? W / 2 : W;
    constexpr int kOutW = kOutAll / G::kHalves;
    const int hc = half * kOutW;
    const int col0 = (kEpi == kGlu ? n0 / 2 : n0) + rank * kOutAll;     // first output column of this CTA
    // bias of the own columns (GLU: value | gate; duplicated block: first copy | second copy) as floats; older than every
    // kernel in flight on the stream only when b_static says so
    if (!p.b_static) ptx::grid_dep_wait();
    {
      const T* bias = static_cast<const T*>(p.bias);
      for (int i = threadIdx.x - 64; i < 2 * kOutAll; i += 32 * G::kEpiWarps) {
        const int part = i / kOutAll, c = col0 + (i - part * kOutAll);
        float v = 0.f;
        if (bias && c < p.N) {
          if constexpr (kEpi == kGlu) v = Elem<T>::to_f(bias[part * p.N + c]);
          else if constexpr (kEpi == kDup) v = (part == 0 || c < p.dup_cols) ? Elem<T>::to_f(bias[c + ((part == 1 || c >= p.dup_cols) ? p.dup_cols : 0)]) : 0.f;
          else if (part == 0) v = Elem<T>::to_f(bias[c]);
        }
        sbias[i] = v;
      }
    }
    if (p.b_static) ptx::grid_dep_wait();
    // residual values of the places this lane will store, fetched under the main loop
    constexpr int kC = kEpi == kResid ? WH / 4 : (kOutW >= 8 ? kOutW / 8 : 1);   // 16-byte pieces of a row
    float4 res[kEpi == kResid ? kC : 1];
    if constexpr (kEpi == kResid) {
#pragma unroll
      for (int i = 0; i < kC; ++i) {
        const int at = i * 32 + lane, r = at / kC, c = (at - r * kC) * 4;
        const int m = m0 + q * 32 + r, col = col0 + hc + c;
        res[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.R_in && m < p.M && col < p.N) res[i] = *reinterpret_cast<const float4*>(p.R_in + static_cast<int64_t>(m) * p.ldd + col);
      }
    }
    ptx::named_barrier_sync(1, 32 * G::kEpiWarps);
    bool ok = ptx::mbar_wait(tfull_bar, 0, abort_flag);
    ptx::tc_fence_after_sync();
    const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    // this warp's rows of the output staging (operand ring: all of this CTA's MMAs, hence its loads, are done)
    uint8_t* stg = ring + (half * 4 + q) * 32 * (WH + 4) * 4;

    // accumulators of output columns c .. c+7 of this thread (relative to hc) -> staging, bias and activation applied
    auto finish8 = [&](float (&v)[8], int c, int pass) {
      if constexpr (kEpi == kResid) {
        float* r = reinterpret_cast<float*>(stg) + lane * (WH + 4) + c;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += sbias[hc + c + i];
        *reinterpret_cast<float4*>(r) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(r + 4) = make_float4(v[4], v[5], v[6], v[7]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += sbias[pass * kOutAll + hc + c + i];
        if (p.act == OASR_ACT_SWISH) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = swish_fast(v[i]);
        } else if (p.act != OASR_ACT_NONE) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = apply_act_fast(v[i], p.act);
        }
        *reinterpret_cast<uint4*>(stg + lane * (kOutW * 2 + 16) + c * 2) =
            make_uint4(pack2<T>(v[0], v[1]), pack2<T>(v[2], v[3]), pack2<T>(v[4], v[5]), pack2<T>(v[6], v[7]));
      }
    };
    // this warp's 32 staged rows -> global memory, 16 bytes per lane, neighbouring lanes on neighbouring addresses
    auto flush = [&](int col) {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kC; ++i) {
        const int at = i * 32 + lane, r = at / kC, m = m0 + q * 32 + r;
        if constexpr (kEpi == kResid) {
          const int c = (at - r * kC) * 4;
          if (m < p.M && col + c < p.N) {
            const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(stg) + r * (WH + 4) + c);
            float4 x = res[i];
            x.x = fmaf(p.alpha, v.x, x.x); x.y = fmaf(p.alpha, v.y, x.y);
            x.z = fmaf(p.alpha, v.z, x.z); x.w = fmaf(p.alpha, v.w, x.w);
            *reinterpret_cast<float4*>(static_cast<float*>(p.D) + static_cast<int64_t>(m) * p.ldd + col + c) = x;
          }
        } else {
          const int c = (at - r * kC) * 8;
          if (m < p.M && col + c < p.ldd)
            *reinterpret_cast<uint4*>(static_cast<T*>(p.D) + static_cast<int64_t>(m) * p.ldd + col + c) =
                *reinterpret_cast<const uint4*>(stg + r * (kOutW * 2 + 16) + c * 2);
        }
      }
      __syncwarp();
    };
    auto finish_glu8 = [&](float (&v)[8], const float (&g)[8], int c) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = (v[i] + sbias[hc + c + i]) * sigmoid_fast(g[i] + sbias[kOutAll + hc + c + i]);
      *reinterpret_cast<uint4*>(stg + lane * (kOutW * 2 + 16) + c * 2) =
          make_uint4(pack2<T>(v[0], v[1]), pack2<T>(v[2], v[3]), pack2<T>(v[4], v[5]), pack2<T>(v[6], v[7]));
    };
    const bool twice = kEpi == kDup && col0 < p.dup_cols;
    const int shift = kEpi == kDup && !twice ? p.dup_cols : 0;

    if constexpr (S > 1) {
      // A thread exchanges the columns it will finish: of every CTA's W columns the WH from `half` on (GLU: half of the value
      // and the gate columns behind them).  i-th of them, owner j, relative to the tile:
      auto owned = [&](int j, int i) -> int {
        if constexpr (kEpi == kGlu) return (i < kOutW ? 0 : BN / 2 - kOutW) + j * kOutAll + hc + i;
        else return j * W + hc + i;
      };
      constexpr int kLd = kEpi == kGlu ? kOutW : WH;      // contiguous columns per tensor-memory load
      float4* mine = recv + (half * (WH / 4)) * BM + row;
      auto slot_of = [](int from, int to) { return from < to ? from : from - 1; };   // of `from`'s partial sums in `to`'s buffer
      uint32_t all[S * WH];
#pragma unroll
      for (int j = 0; j < S; ++j) {
#pragma unroll
        for (int c = 0; c < WH; c += kLd) tmem_ld_cols<kLd>(t_acc + owned(j, c), all + j * WH + c);
      }
      ptx::tmem_ld_wait();
      cluster_wait();
      float own[WH];
#pragma unroll
      for (int j = 0; j < S; ++j) {
        const uint32_t* acc = all + j * WH;
        if (j == rank) {
#pragma unroll
          for (int i = 0; i < WH; ++i) own[i] = __uint_as_float(acc[i]);
        } else {
          const uint32_t dst = ptx::map_to_cta(mine + slot_of(rank, j) * (W / 4) * BM, j), bar = ptx::map_to_cta(recv_bar, j);
#pragma unroll
          for (int i = 0; i < WH; i += 4) st_async_v4(dst + (i / 4) * BM * 16, bar, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        }
      }
      ok = ptx::mbar_wait(recv_bar, 0, abort_flag) && ok;
      // sum in rank order, so that the result does not depend on which CTA adds
      float sum[WH];
#pragma unroll
      for (int j = 0; j < S; ++j) {
#pragma unroll
        for (int i = 0; i < WH; i += 4) {
          float4 v = make_float4(own[i], own[i + 1], own[i + 2], own[i + 3]);
          if (j != rank) v = mine[(slot_of(j, rank) * (W / 4) + i / 4) * BM];
          if (j == 0) { sum[i] = v.x; sum[i + 1] = v.y; sum[i + 2] = v.z; sum[i + 3] = v.w; }
          else { sum[i] += v.x; sum[i + 1] += v.y; sum[i + 2] += v.z; sum[i + 3] += v.w; }
        }
      }
      if constexpr (kEpi == kGlu) {
#pragma unroll
        for (int c = 0; c < kOutW; c += 8) {
          float v[8], g[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) { v[i] = sum[c + i]; g[i] = sum[kOutW + c + i]; }
          finish_glu8(v, g, c);
        }
        flush(col0 + hc);
      } else {
#pragma unroll 1
        for (int pass = 0; pass < (twice ? 2 : 1); ++pass) {
#pragma unroll
          for (int c = 0; c < WH; c += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = sum[c + i];
            finish8(v, c, pass);
          }
          flush(col0 + hc + shift + pass * p.dup_cols);
        }
      }
    } else if constexpr (kEpi == kGlu) {
#pragma unroll 1
      for (int c0 = 0; c0 < kOutW; c0 += 16) {
        uint32_t rv[16], rg[16];
        ptx::tmem_ld_32x16(t_acc + hc + c0, rv);
        ptx::tmem_ld_32x16(t_acc + BN / 2 + hc + c0, rg);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 16; c += 8) {
          float v[8], g[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) { v[i] = __uint_as_float(rv[c + i]); g[i] = __uint_as_float(rg[c + i]); }
          finish_glu8(v, g, c0 + c);
        }
      }
      flush(col0 + hc);
    } else {
#pragma unroll 1
      for (int pass = 0; pass < (twice ? 2 : 1); ++pass) {
#pragma unroll 1
        for (int c0 = 0; c0 < WH; c0 += 32) {
          uint32_t acc[32];
          ptx::tmem_ld_32x32(t_acc + hc + c0, acc);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(acc[c + i]);
            finish8(v, c0 + c, pass);
          }
        }
        flush(col0 + hc + shift + pass * p.dup_cols);
      }
    }
    if (!ok && lane == 0 && p.status) atomicOr(p.status, kStatusGemmEpilogue);
    ptx::tc_fence_before_sync();
  }
  __syncthreads();
  if (*abort_flag) {     // copies that may still be in flight get time to land before shared memory and TMEM are released
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, BN);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// CTAs per cluster: about 512 elements of K each while N / 64 tiles times the splits stay within 64 CTAs per 128 rows; a
// wide product has enough tiles of its own, and an unsplit one gives the bits of gemm.cu.  A function of N and K only: see
// the header comment.
int splits_for(int64_t n_acc, int64_t K) {
  int s = K < 1024 ? 1 : (K < 2048 ? 2 : (K < 4096 ? 4 : 8));
  while (s > 1 && (n_acc + 63) / 64 * s > 64) s >>= 1;
  return s;
}

// Tile width: the one that leaves the fewest operand bytes on the busiest SM (a column tile costs its own rows of B and the
// rows of A that exist, and about 24 rows' worth of fixed time); ties go to the wider tile, which moves fewer bytes in all.
int pick_bn(int epi, int64_t M, int64_t n_acc, int S, int64_t dup_cols, int64_t* ctas_out) {
  const int64_t m_tiles = (M + BM - 1) / BM;
  const int rows = static_cast<int>(M < BM ? M : BM);
  int bn = 64;
  double best = 1e30;
  for (int cand = ((S == 1 && epi == kResid) || S == 8 ? 64 : 128); cand >= 32; cand >>= 1) {
    if (cand == 32 && (epi == kGlu || S == 8)) continue;   // at least 8 output columns per CTA
    if (epi == kDup && dup_cols % cand) continue;
    const int64_t ctas = m_tiles * ((n_acc + cand - 1) / cand) * S;
    const int64_t per_sm = (ctas + sm_count() - 1) / sm_count();
    const double cost = static_cast<double>(per_sm) * (rows + cand + 24);
    if (cost < best * 0.999) {
      best = cost;
      bn = cand;
      if (ctas_out) *ctas_out = ctas;
    }
  }
  return bn;
}

// Where the kernel is ahead of the persistent one (B200, weights from HBM, us here / there):
//   N 512, K 2048:  592 rows 5.4 / 17.1, 2048 rows 16.6 / 17.8, 4096 rows 32.7 / 23.8
//   N 2048, K 512:  512 rows 4.5 / 6.3, 2560 rows 11.6 / 18.2, 4096 rows 13.8 / 12.7
//   N 4096, K 1024: 512 rows 7.7 / 9.8, 1536 rows 17.9 / 21.0, 2048 rows 19.9 / 18.3
//   N 1024, K 4096: 512 rows 11.0 / 27.2, 1024 rows 25.0 / 27.5, 1536 rows 35.5 / 33.3
// Each CTA runs its phases (operands, exchange, output) once and in series, so what counts is the number of CTAs: an SM
// hides them with two or three.  Narrow outputs (N up to 512) keep the kernel over its whole range: their K split changes
// the bits, and a row's result is not to depend on its batch.
bool takes(int epi, int64_t M, int64_t N, int64_t K, int64_t dup_cols) {
  if (M <= 0 || M > kMaxRows || N < 32 || K < 64) return false;
  const int64_t n_acc = epi == kGlu ? 2 * N : N;
  const int S = splits_for(n_acc, K);
  if (epi == kGlu && (N % 32 || S > 4)) return false;
  if (S > 1 && n_acc <= 512) return true;
  if (S == 1 && epi == kResid) return true;        // gemm.cu stores fp32 rows a thread each
  int64_t ctas = 0;
  pick_bn(epi, M, n_acc, S, dup_cols, &ctas);
  return S > 1 ? ctas * 5 <= 9 * sm_count() : ctas * 5 <= 13 * sm_count();
}

template <typename T, int BN, int S, int kEpi>
int launch(const Args& a, Params& p, int m_tiles, int dtype, cudaStream_t s) {
  using G = Geo<BN, S>;
  constexpr bool kGluE = kEpi == kGlu;
  const int64_t n_acc = kGluE ? 2 * a.N : a.N;
  const int n_tiles = static_cast<int>((n_acc + BN - 1) / BN);
  // Ring: the whole K slice where one CTA per SM leaves room for it, else what lets two CTAs share an SM.
  const int rows = static_cast<int>(a.M < BM ? (a.M + 7) / 8 * 8 : BM);
  p.a_blk = rows * BK * 2;
  const int fixed = 1024 + G::kHead + G::kRecv + (rows < BM ? 16384 - p.a_blk : 0), blk = p.a_blk + G::kBBlk;
  int fit = (113 * 1024 - fixed) / blk;
  if (fit < 3 || static_cast<int64_t>(m_tiles) * n_tiles * S <= sm_count()) fit = (227 * 1024 - fixed) / blk;
  const int whole = fit < p.kb_per ? fit : p.kb_per;              // K blocks held at a time
  p.kg = !p.k_whole || whole < 4 ? 1 : (whole > 2 * kMaxStages ? 4 : 2);
  p.stages = whole / p.kg < kMaxStages ? whole / p.kg : kMaxStages;
  if (whole == p.kb_per && p.kg * p.stages < whole && p.stages < kMaxStages && (whole + p.kg - 1) / p.kg * p.kg <= fit) ++p.stages;
  if (p.stages < 2) p.stages = 2;
  int ring = p.stages * p.kg * blk;
  if (ring < G::kStaging) ring = G::kStaging;
  const int bytes = fixed + ring;
  CUtensorMap ta, tb;
  const uint64_t k_in = p.k_whole ? BK : a.K, k_out = p.k_whole ? p.kb_total : 1;
  const uint64_t adims[3] = {k_in, (uint64_t)a.M, k_out}, astr[3] = {0, (uint64_t)a.K * 2, BK * 2};
  const uint32_t abox[3] = {BK, (uint32_t)rows, (uint32_t)p.kg};
  if (int rc = make_tensor_map(&ta, tma_dtype(dtype), 3, a.A, adims, astr, abox)) return rc;
  const uint64_t bdims[4] = {k_in, (uint64_t)a.N, kGluE ? 2u : 1u, k_out};
  const uint64_t bstr[4] = {0, (uint64_t)a.K * 2, (uint64_t)a.K * 2 * (uint64_t)a.N, BK * 2};
  const uint32_t bbox[4] = {BK, (uint32_t)(kGluE ? BN / 2 : BN), kGluE ? 2u : 1u, (uint32_t)p.kg};
  if (int rc = make_tensor_map(&tb, tma_dtype(dtype), 4, a.B, bdims, bstr, bbox)) return rc;
  auto kern = gemm_small_kernel<T, BN, S, kEpi>;
  static SmemLimit smem_limit;
  const cudaError_t e = smem_limit.raise(kern, 227 * 1024);
  if (e != cudaSuccess) return set_error(OASR_ERR_CUDA, "gemm_small: cannot reserve shared memory: %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(n_tiles * S), static_cast<unsigned>(m_tiles));
  cfg.blockDim = dim3(G::kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(bytes);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (g_pdl) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (S > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = S;
    at[n].val.clusterDim.y = 1;
    at[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kern, ta, tb, p);
  return check_launch("gemm_small launch");
}

template <typename T, int kEpi>
int run_typed(const Args& a, Params& p, int dtype, cudaStream_t s) {
  constexpr bool kGluE = kEpi == kGlu;
  const int64_t n_acc = kGluE ? 2 * a.N : a.N;
  const int S = splits_for(n_acc, a.K);
  const int m_tiles = static_cast<int>((a.M + BM - 1) / BM);
  const int bn = pick_bn(kEpi, a.M, n_acc, S, a.dup_cols, nullptr);
  p.kb_total = static_cast<int>((a.K + BK - 1) / BK);
  p.kb_per = (p.kb_total + S - 1) / S;
  p.k_whole = a.K % BK == 0;
#define GSM_CASE(BN_, S_) return launch<T, BN_, S_, kEpi>(a, p, m_tiles, dtype, s)
  if (S == 1) {
    if constexpr (kEpi != kResid) {
      if (bn == 128) GSM_CASE(128, 1);
    }
    if constexpr (!kGluE) {
      if (bn == 32) GSM_CASE(32, 1);
    }
    GSM_CASE(64, 1);
  }
  if (S == 2) {
    if (bn == 128) GSM_CASE(128, 2);
    if constexpr (!kGluE) {
      if (bn == 32) GSM_CASE(32, 2);
    }
    GSM_CASE(64, 2);
  }
  if (S == 4) {
    if (bn == 128) GSM_CASE(128, 4);
    if constexpr (!kGluE) {
      if (bn == 32) GSM_CASE(32, 4);
    }
    GSM_CASE(64, 4);
  }
  if constexpr (!kGluE) GSM_CASE(64, 8);
  return set_error(OASR_ERR_UNSUPPORTED, "gemm_small: no kernel for this shape");
#undef GSM_CASE
}

int run(int epi, const Args& a, int dtype, cudaStream_t s) {
  Params p{};
  p.M = static_cast<int>(a.M); p.N = static_cast<int>(a.N);
  p.ldd = static_cast<int>(a.N + (epi == kDup ? a.dup_cols : 0));
  p.dup_cols = static_cast<int>(a.dup_cols);
  p.act = a.act; p.alpha = a.alpha; p.R_in = a.R_in; p.bias = a.bias; p.D = a.D; p.b_static = a.b_static; p.late_launch = a.late_launch;
  p.status = device_status_ptr();
  return OB_DISPATCH_HALF(dtype, T, [&]() -> int {
    switch (epi) {
      case kStore: return run_typed<T, kStore>(a, p, dtype, s);
      case kResid: return run_typed<T, kResid>(a, p, dtype, s);
      case kGlu: return run_typed<T, kGlu>(a, p, dtype, s);
      default: return run_typed<T, kDup>(a, p, dtype, s);
    }
  });
}

}  // namespace gsm
}  // namespace ob
