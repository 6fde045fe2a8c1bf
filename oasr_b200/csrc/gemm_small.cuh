// Host interface of the few-rows GEMM (gemm_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ob {
namespace gsm {

enum Epi { kStore = 0, kResid = 1, kGlu = 2, kDup = 3 };

struct Args {
  void* D = nullptr;            // kResid: fp32
  const void* A = nullptr;      // (M, K), packed rows
  const void* B = nullptr;      // (N, K); kGlu: (2N, K)
  const void* bias = nullptr;   // nullable; kGlu: 2N; kDup: N + dup_cols, per OUTPUT column
  const float* R_in = nullptr;  // kResid: D = R_in + alpha * (A.B^T + bias); null = 0
  int64_t M = 0, N = 0, K = 0, dup_cols = 0;
  int act = -1;
  float alpha = 1.f;
  // How an executor's chain of launches uses programmatic dependent launch.  late_launch: the chain's first GEMM lets its
  // successor start only once everything before the chain is complete and visible; b_static: a later GEMM of the chain,
  // whose weights (B, bias) are therefore settled, fetches them before it waits for its predecessor.  Only behind a first
  // GEMM that starts_late(): the other kernels let their successor start before their own wait.
  int b_static = 0;
  int late_launch = 0;
};

// Rows up to which the kernel is used (takes() says where).
constexpr int64_t kMaxRows = 2560;

bool takes(int epi, int64_t M, int64_t N, int64_t K, int64_t dup_cols = 0);
int run(int epi, const Args& a, int dtype, cudaStream_t s);

}  // namespace gsm

// The C-ABI operators of the same names with the launch-chain flags above (gemm.cu).
struct Chain {
  int b_static = 0, late_launch = 0;
};
// Does the operator with this epilogue run a kernel that honours late_launch?  The chain behind it may then be inner_chain().
bool starts_late(int epi, int64_t M, int64_t N, int64_t K);
inline Chain inner_chain(bool first_starts_late) { return Chain{first_starts_late ? 1 : 0, 0}; }
int gemm_op(void* D, const void* A, const void* B, const void* bias, int64_t M, int64_t N, int64_t K, int activation, int dtype,
            void* stream, Chain chain);
int gemm_glu_op(void* D, const void* A, const void* B, const void* bias, int64_t M, int64_t N, int64_t K, int dtype, void* stream,
                Chain chain);
int gemm_dup_first_op(void* D, const void* A, const void* B, const void* bias, int64_t M, int64_t N, int64_t K, int64_t dup_cols,
                      int dtype, void* stream, Chain chain);
int gemm_residual_f32_op(float* R_out, const float* R_in, const void* A, const void* B, const void* bias, int64_t M, int64_t N,
                         int64_t K, double alpha, int dtype, void* stream, Chain chain);
int gemm_log_softmax_op(void* out, const void* A, const void* B, const void* bias, int64_t M, int64_t N, int64_t K, int dtype,
                        int out_dtype, int32_t* argmax, void* stream, Chain chain);
}  // namespace ob
