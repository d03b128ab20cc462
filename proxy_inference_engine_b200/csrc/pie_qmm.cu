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

// One rounding to bf16.  Rows that are 16-byte aligned go through the warp's shared memory, so that a store instruction writes
// 64-byte runs of 8 rows and not 16 bytes of 32.
struct QmmStore {
  uint16_t* y;
  int M, N;
  __device__ __forceinline__ void operator()(int, int row0, int col, const uint32_t (&v)[32], uint32_t buf, int lane) const {
    if (row0 >= M || col >= N) return;
    uint16_t* const base = y + (size_t)row0 * N + col;
    if ((N & 7) == 0) {
      auto at = [&](int r, int c) { return buf + r * 64 + ((c ^ ((r >> 1) & 3)) << 4); };
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = pack_bf16(__uint_as_float(v[8 * c + 2 * e]), __uint_as_float(v[8 * c + 2 * e + 1]));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at(lane, c)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2), c = lane & 3;
        const uint4 o = lds128(at(r, c));
        if (row0 + r < M && col + 8 * c < N) *reinterpret_cast<uint4*>(base + (size_t)r * N + 8 * c) = o;
      }
      __syncwarp();
    } else if (row0 + lane < M) {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (col + q < N) base[(size_t)lane * N + q] = f2bf(__uint_as_float(v[q]));
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
