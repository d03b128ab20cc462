// Prefill quantized GEMM on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a.
//
// Replaces mx.quantized_matmul(transpose=True) at prefill-sized M (MLX/mlx/ops.cpp:3984-4021; Metal qmm_t,
// MLX/mlx/backend/metal/kernels/quantized.h:954-1078):  y[m, n] = bf16( sum_k x[m, k] * w_hat[n, k] ),
// w_hat = bf16(scale * q + bias): the weight is dequantised ONCE to the activation type into shared memory
// (QuantizedBlockLoader, quantized.h:411-417, 502-512) and the contraction accumulates in fp32 -- the same rounding
// structure here, with the fp32 accumulator in tensor memory.  The kernel is the GEMM core of pie_gemm.cuh with
// dequantising warps; this file holds the store and the choice of tile.
#include "pie_gemm.cuh"
#include "pie_internal.h"

namespace pie {

// one rounding to bf16; 32 columns of a row, 16 bytes at a time where rows are 16-byte aligned
struct QmmStore {
  uint16_t* y;
  int M, N;
  __device__ __forceinline__ void operator()(int, int row, int col, const uint32_t (&v)[32]) const {
    if (row >= M || col >= N) return;
    uint16_t* dst = y + (size_t)row * N + col;
    if (col + 32 <= N && (N & 7) == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 o;
        o.x = pack_bf16(__uint_as_float(v[8 * q]), __uint_as_float(v[8 * q + 1]));
        o.y = pack_bf16(__uint_as_float(v[8 * q + 2]), __uint_as_float(v[8 * q + 3]));
        o.z = pack_bf16(__uint_as_float(v[8 * q + 4]), __uint_as_float(v[8 * q + 5]));
        o.w = pack_bf16(__uint_as_float(v[8 * q + 6]), __uint_as_float(v[8 * q + 7]));
        reinterpret_cast<uint4*>(dst)[q] = o;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (col + q < N) dst[q] = f2bf(__uint_as_float(v[q]));
    }
  }
};

cudaError_t launch_qmm_tc(uint16_t* y, const uint16_t* x, const uint32_t* wq, const uint16_t* s, const uint16_t* b,
                          int M, int N, int K, int bits, cudaStream_t st) {
  GemmArgs a = {};
  a.M = M; a.N = N; a.K = K; a.nb = 1;
  a.scales = s; a.biases = b;
  a.scale_vec = K % 512 == 0 && ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
  const QmmStore epi = {y, M, N};
  count_launch();
  return bits == 4 ? gemm_run<4>(a, epi, x, (long long)K * 2, 0, wq, 0, num_sms(), st)
                   : gemm_run<8>(a, epi, x, (long long)K * 2, 0, wq, 0, num_sms(), st);
}

unsigned int qmm_pipeline_error() {
  unsigned int v = 0;
  cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(v));
  return v;
}

}  // namespace pie
