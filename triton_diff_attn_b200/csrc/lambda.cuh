// lambda = exp(<q1, k1>) - exp(<q2, k2>) + lambda_init and its gradients: one launch each way.
//
// A few hundred numbers: what counts is that it is ONE launch.  As separate tensor operations (multiply, sum, exponential, ...) the
// forward is eight launches and the backward about fourteen, each 2 us of the device and more of the host, in front of and behind
// the attention kernels of every layer: `DiffAttnCore` forward and backward at B4 H16 N2048 D64 causal 606 -> 553 us.
#pragma once
#include <cuda_runtime.h>

namespace da {

constexpr int LAMBDA_THREADS = 128;

struct LambdaArgs {
  const float* q1; const float* k1; const float* q2; const float* k2;     // [n]
  int n;
  float lambda_init;
  float* out;               // [3]: lambda, exp(<q1, k1>), exp(<q2, k2>)
  const float* dlambda;     // backward: [1]
  float* dq1; float* dk1; float* dq2; float* dk2;
};

__global__ void __launch_bounds__(LAMBDA_THREADS) diffattn_lambda_fwd_kernel(const LambdaArgs a) {
  float s1 = 0.f, s2 = 0.f;
  for (int i = threadIdx.x; i < a.n; i += LAMBDA_THREADS) {
    s1 += a.q1[i] * a.k1[i];
    s2 += a.q2[i] * a.k2[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  __shared__ float red[2][LAMBDA_THREADS / 32];
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = s1; red[1][threadIdx.x >> 5] = s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    s1 = s2 = 0.f;
    for (int w = 0; w < LAMBDA_THREADS / 32; ++w) { s1 += red[0][w]; s2 += red[1][w]; }
    const float e1 = expf(s1), e2 = expf(s2);
    a.out[0] = e1 - e2 + a.lambda_init;
    a.out[1] = e1;
    a.out[2] = e2;
  }
}

__global__ void __launch_bounds__(LAMBDA_THREADS) diffattn_lambda_bwd_kernel(const LambdaArgs a) {
  const float g1 = a.dlambda[0] * a.out[1], g2 = -a.dlambda[0] * a.out[2];
  for (int i = threadIdx.x; i < a.n; i += LAMBDA_THREADS) {
    a.dq1[i] = g1 * a.k1[i];
    a.dk1[i] = g1 * a.q1[i];
    a.dq2[i] = g2 * a.k2[i];
    a.dk2[i] = g2 * a.q2[i];
  }
}

}  // namespace da
