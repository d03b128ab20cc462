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
#include "pie_qmt.cuh"

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

// The products of up to three matrices side by side in rows of y, and a residual added to them: (bf16 of the product) + residual, as pie_add
// rounds it.  q, k and v of a 1B layer (2048, 512 and 512 rows of K 2048) as three launches leave half the SMs without a tile, and a sum of its own
// reads and writes what the product has in registers.  A layer of 1531 tokens behind 517: 275.5 -> 253.9 us; 8B, 8192 tokens: 3508 -> 3450 (two sums
// of 28 us; its q, k and v are eleven waves of tiles either way).
struct QmmRows {
  static constexpr bool SEGMENTS = true;
  CUtensorMap map_more[2];
  int tile0[3], N[3], off[3];
  const uint16_t *s[3], *b[3];
  uint16_t* y;
  const uint16_t* residual;
  int M, ld;
  __device__ __forceinline__ int segment(int n) const { return (n >= tile0[1]) + (n >= tile0[2]); }
  __device__ __forceinline__ void operator()(int g, int row0, int col, const uint32_t (&v)[32], uint32_t buf, int lane) const {
    const int n = N[g];
    if (row0 >= M || col >= n) return;
    const size_t first = (size_t)row0 * ld + off[g] + col;
    if (((ld | n | off[g]) & 7) == 0) {   // as QmmStore
      auto at = [&](int r, int c) { return buf + r * 64 + ((c ^ ((r >> 1) & 3)) << 4); };
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = pack_bf16(__uint_as_float(v[8 * c + 2 * e]), __uint_as_float(v[8 * c + 2 * e + 1]));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at(lane, c)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
      }
      const int c = lane & 3;
      uint4 res[4];
      if (residual) {   // (may lie where y goes: a thread reads what it writes)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = 8 * i + (lane >> 2);
          res[i] = make_uint4(0, 0, 0, 0);
          if (row0 + r < M && col + 8 * c < n) res[i] = *reinterpret_cast<const uint4*>(residual + first + (size_t)r * ld + 8 * c);
        }
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        uint4 o = lds128(at(r, c));
        if (residual) { o.x = sum(o.x, res[i].x); o.y = sum(o.y, res[i].y); o.z = sum(o.z, res[i].z); o.w = sum(o.w, res[i].w); }
        if (row0 + r < M && col + 8 * c < n) *reinterpret_cast<uint4*>(y + first + (size_t)r * ld + 8 * c) = o;
      }
      __syncwarp();
    } else if (row0 + lane < M) {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (col + q < n) {
          const size_t p = first + (size_t)lane * ld + q;
          const uint16_t o = f2bf(__uint_as_float(v[q]));
          y[p] = residual ? f2bf(bf16lo(o) + bf16lo(residual[p])) : o;
        }
    }
  }
  static __device__ __forceinline__ uint32_t sum(uint32_t a, uint32_t b) { return pack_bf16(bf16lo(a) + bf16lo(b), bf16hi(a) + bf16hi(b)); }
};

// silu(x . w) * (x . w_up), rounded where the separate operators round: both products, the sigmoid, silu, the result.  It saves the two
// products' way to memory and back and a launch: 8192 x 14336 x 4096 (4 bits)
// 2 x 676 + 130 -> 1275 us, 1531 x 8192 x 2048 87 + 12 -> 83.
struct QmmSwiglu {
  static constexpr bool PAIRED = true;
  CUtensorMap map_up;
  const uint16_t *s_up, *b_up;
  uint16_t* y;
  int M, N;
  __device__ __forceinline__ void gate(const uint32_t (&v)[32], uint32_t (&t)[16]) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) t[e] = silu_bf16x2(pack_bf16(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])));
  }
  __device__ __forceinline__ void operator()(int row0, int col, const uint32_t (&t)[16], const uint32_t (&v)[32], uint32_t buf, int lane) const {
    if (row0 >= M || col >= N) return;
    uint32_t o[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e] = mul_bf16x2_rn(t[e], pack_bf16(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])));
    uint16_t* const base = y + (size_t)row0 * N + col;
    if ((N & 7) == 0) {   // as QmmStore
      auto at = [&](int r, int c) { return buf + r * 64 + ((c ^ ((r >> 1) & 3)) << 4); };
#pragma unroll
      for (int c = 0; c < 4; ++c)
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at(lane, c)), "r"(o[4 * c]), "r"(o[4 * c + 1]), "r"(o[4 * c + 2]),
                     "r"(o[4 * c + 3]) : "memory");
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2), c = lane & 3;
        const uint4 w = lds128(at(r, c));
        if (row0 + r < M && col + 8 * c < N) *reinterpret_cast<uint4*>(base + (size_t)r * N + 8 * c) = w;
      }
      __syncwarp();
    } else if (row0 + lane < M) {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (col + q < N) base[(size_t)lane * N + q] = (uint16_t)(o[q >> 1] >> (16 * (q & 1)));
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

cudaError_t launch_qmm_rows(uint16_t* y, int ld, const uint16_t* x, const pie_qmv_seg* segs, int n, const uint16_t* residual, int M, int K, int bits,
                            cudaStream_t st) {
  GemmArgs a = {};
  QmmRows epi = {};
  const uint32_t* w[3] = {};
  uintptr_t at = 0;
  for (int i = 0, off = 0; i < n; off += segs[i++].N) {
    w[i] = segs[i].wq;
    epi.s[i] = (const uint16_t*)segs[i].scales; epi.b[i] = (const uint16_t*)segs[i].biases;
    epi.N[i] = segs[i].N; epi.off[i] = off;
    at |= reinterpret_cast<uintptr_t>(segs[i].scales) | reinterpret_cast<uintptr_t>(segs[i].biases);
  }
  a.M = M; a.N = segs[0].N; a.K = K; a.nb = 1;
  a.scales = epi.s[0]; a.biases = epi.b[0];
  a.scale_vec = K % 512 == 0 && (at & 15) == 0;
  epi.y = y; epi.residual = residual; epi.M = M; epi.ld = ld;
  count_launch();
  return bits == 4 ? gemm_run_segments<4>(a, epi, n, x, w, num_sms(), st) : gemm_run_segments<8>(a, epi, n, x, w, num_sms(), st);
}

// bn = 0 where two products and the elementwise operator are estimated to be done sooner (its 6 bytes an element at 6 TB/s and two
// launches in cycles of 1.9 GHz beside the products' own estimate), as they are where one wave of single CTAs holds a product: 77 rows of
// 14336 x 4096 take 27 + 27 + 3 us, in pairs' tiles two waves.
static GemmChoice qmm_swiglu_choice(int M, int N, int K, int sms) {
  const double apart = 2 * gemm_choose(M, N, K, 1, sms, true).cycles + (double)M * N * 6 / 3158 + 4000;
  return gemm_choose_paired(M, N, K, sms, apart);
}
bool qmm_swiglu_pays(int M, int N, int K) { return qmm_swiglu_choice(M, N, K, num_sms()).bn != 0; }
cudaError_t launch_qmm_swiglu(uint16_t* y, const uint16_t* x, const uint32_t* const* wq, const uint16_t* const* s, const uint16_t* const* b,
                              int M, int N, int K, int bits, cudaStream_t st) {
  const int sms = num_sms();
  const GemmChoice c = qmm_swiglu_choice(M, N, K, sms);
  if (!c.bn) return cudaErrorNotSupported;
  GemmArgs a = {};
  a.M = M; a.N = N; a.K = K; a.nb = 1;
  a.scales = s[0]; a.biases = b[0];
  uintptr_t at = 0;
  for (int i = 0; i < 2; ++i) at |= reinterpret_cast<uintptr_t>(s[i]) | reinterpret_cast<uintptr_t>(b[i]);
  a.scale_vec = K % 512 == 0 && (at & 15) == 0;
  QmmSwiglu epi = {};
  epi.s_up = s[1]; epi.b_up = b[1]; epi.y = y; epi.M = M; epi.N = N;
  count_launch();
  return bits == 4 ? gemm_run_paired<4>(a, epi, c, x, wq[0], wq[1], sms, st) : gemm_run_paired<8>(a, epi, c, x, wq[0], wq[1], sms, st);
}

// what a product takes (dual: two of them and the elementwise operator, or both in one launch); 4 us besides the main loop's cycles
double qmm_estimate_us(int M, int N, int K, int dual) {
  const int sms = num_sms();
  const double one = gemm_choose(M, N, K, 1, sms, true).cycles / 1900 + 4;
  if (!dual) return one;
  const GemmChoice c = qmm_swiglu_choice(M, N, K, sms);
  const double apart = 2 * one + 2 + (double)M * N * 6 / 6e6;
  return c.bn && c.cycles / 1900 + 4 < apart ? c.cycles / 1900 + 4 : apart;
}

unsigned int qmm_pipeline_error() { return gemm_error_now(); }
cudaError_t qmm_pipeline_post(unsigned int* host, cudaStream_t st) { return gemm_error_post(host, st); }
cudaError_t qmm_pipeline_clear() { return gemm_error_clear(); }

}  // namespace pie
