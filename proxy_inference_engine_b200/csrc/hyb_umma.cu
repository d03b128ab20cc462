// Dense bf16 GEMM on the 5th-generation tensor cores (tcgen05 + TMEM) for prefill-sized steps:
//   y[m, n] = sum_k x[m, k] w[n, k]   (x [M, K] bf16, w [N, K] bf16, fp32 accumulation in tensor memory)
// Two kernels with pieh_linear's epilogues (bias, activations, gated pairs, soft cap, bf16 or fp32 store, the in-place
// residual-stream update), applied to 32 columns of a row at a time as they come out of tensor memory:
//   * dense and batched products: the GEMM core of pie_gemm.cuh (operands by TMA, CTA pairs, persistent).
//   * grouped products (mixture of experts; rows gathered through an index, which a tiled copy cannot do): a CTA owns a
//     128 x 256 tile.  Per 64-element K step and pipeline stage, 256 producer threads bring one 128-byte row piece of x and of
//     w each into the 128B-swizzled K-major layout with cp.async (thread t <-> tile row t), make it visible to the async proxy
//     and arrive on the stage's mbarrier; one elected lane of a ninth warp issues the tcgen05.mma's (M128 N256 K16).
// Every mbarrier wait is bounded: on expiry the CTA raises an error word the host can read, drains its copies, frees its
// tensor memory and returns.
#include "hyb_common.cuh"
#include "pie_gemm.cuh"

namespace pieh {

using pie::smem_u32;

constexpr int kBN = 256, kBK = 64, kProducers = 256, kThreads = kProducers + 32;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr uint32_t IDESC = pie::umma_idesc_bf16_m128(kBN);

__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  uint32_t spins = 0;
  while (!pie::mbar_try_wait(bar, parity)) {
    if (++spins > kWaitLimit || *abort_flag) {
      *abort_flag = 1;
      atomicExch(&pie::g_gemm_error, 1u);
      return false;
    }
  }
  return true;
}

// any number of streams up to 8, any alignment, the edge of the matrix: a column at a time
__device__ __noinline__ void streams_any(const LinArgs& a, int m, int n0, const float* y) {
  float* xs = reinterpret_cast<float*>(a.out) + (size_t)m * a.S * a.N;
  for (int q = 0; q < 32 && n0 + q < a.N; ++q) {
    const int n = n0 + q;
    float old[8];
    for (int s = 0; s < a.S; ++s) old[s] = xs[(size_t)s * a.N + n];
    for (int u = 0; u < a.S; ++u) {
      float acc = a.outw[u] * y[q];
      for (int s = 0; s < a.S; ++s) acc = fmaf(a.mix[s * a.S + u], old[s], acc);
      xs[(size_t)u * a.N + n] = acc;
    }
  }
}
// x_u <- sum_s mix[s, u] x_s + outw[u] y over S residual streams: this lane's four columns of every fourth row of the warp's tile,
// read from the staged y.  Rows are taken in batches: the loads of a batch are in flight together.
template <int S>
__device__ __forceinline__ void streams_tile(const LinArgs& a, int row0, int m_end, int n, uint32_t buf, int lane) {
  constexpr int NB = S <= 2 ? 4 : 2;
  float* xs = reinterpret_cast<float*>(a.out) + n;
#pragma unroll
  for (int i0 = 0; i0 < 8; i0 += NB) {
    float4 old[NB][S];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int m = row0 + 4 * (i0 + j) + (lane >> 3);
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (m < m_end) old[j][s] = *reinterpret_cast<const float4*>(xs + ((size_t)m * S + s) * a.N);
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int r = 4 * (i0 + j) + (lane >> 3), m = row0 + r;
      const uint4 yq = pie::lds128(buf + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
      if (m < m_end)
#pragma unroll
        for (int u = 0; u < S; ++u) {
          const float ow = a.outw[u];
          float4 acc = make_float4(ow * __uint_as_float(yq.x), ow * __uint_as_float(yq.y), ow * __uint_as_float(yq.z), ow * __uint_as_float(yq.w));
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const float mx = a.mix[s * S + u];
            acc.x = fmaf(mx, old[j][s].x, acc.x); acc.y = fmaf(mx, old[j][s].y, acc.y);
            acc.z = fmaf(mx, old[j][s].z, acc.z); acc.w = fmaf(mx, old[j][s].w, acc.w);
          }
          *reinterpret_cast<float4*>(xs + ((size_t)m * S + u) * a.N) = acc;
        }
    }
  }
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Activations whose instructions are many: of 32 values at a time, unrolled, they are more than the instruction caches hold, and the last
// tile of every launch waits for them.  They are applied on the way from shared memory to out, in a loop over four values of a lane, which are
// enough for its warp to go on while one waits.  us behind other kernels, 32 unrolled / one value after the other / four, SOFTCAP, TANH, XIELU, GELU:
//   150 x 32000 x 2048             87.0 / 56.1 / 50.1   45.7 / 45.3 / 40.7   68.4 / 62.3 / 56.6   87.4 / 54.2 / 51.0
//   600 x 8192 x 2048 and a bias   38.5 / 41.9 / 36.8   31.9 / 33.6 / 30.6   44.7 / 46.9 / 41.8   39.9 / 40.5 / 37.4
//   4000 x 8192 x 2048 and a bias  137 / 159 / 132      100 / 126 / 95       165 / 178 / 162      142 / 154 / 137
__device__ __forceinline__ bool act_in_loop(int epi) {
  return epi == PIEH_EPI_SOFTCAP || epi == PIEH_EPI_TANH || epi == PIEH_EPI_XIELU || epi == PIEH_EPI_GELU;
}
__device__ __forceinline__ void act_of(const LinArgs& a, float (&y)[4]) {
  switch (a.epi) {
    case PIEH_EPI_SOFTCAP:
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = a.epi_a * tanhf(y[e] / a.epi_a);
      break;
    case PIEH_EPI_TANH:
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = tanhf(y[e]);
      break;
    case PIEH_EPI_XIELU:
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = xielu_f(y[e], a.epi_a, a.epi_b);
      break;
    default:
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = gelu_f(y[e]);
      break;
  }
}
template <typename OT>
__device__ __forceinline__ void tile_act_out(const LinArgs& a, OT* out, long long ld, int row0, int m_end, int n0, int n_end, const float (&y)[32],
                                             uint32_t buf, int lane) {
  auto at = [&](int r, int c) { return buf + r * 128 + ((c ^ (r & 7)) << 4); };
#pragma unroll
  for (int c = 0; c < 8; ++c)
    sts128(at(lane, c), __float_as_uint(y[4 * c]), __float_as_uint(y[4 * c + 1]), __float_as_uint(y[4 * c + 2]), __float_as_uint(y[4 * c + 3]));
  __syncwarp();
  OT* const base = out + (size_t)row0 * ld + n0;
  const bool whole = (reinterpret_cast<uintptr_t>(base) & (4 * sizeof(OT) - 1)) == 0 && (ld & 3) == 0;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {          // eight lanes a row
    const int r = 4 * i + (lane >> 3), c = lane & 7, n = n0 + 4 * c;
    const uint4 u = pie::lds128(at(r, c));
    float v[4] = {__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w)};
    if (row0 + r >= m_end || n >= n_end) continue;
    act_of(a, v);
    OT* const dst = base + (size_t)r * ld + 4 * c;
    if (whole && n + 4 <= n_end) {
      store4(dst, make_float4(v[0], v[1], v[2], v[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < n_end) elem<OT>::store(dst + e, v[e]);
    }
  }
  __syncwarp();
}
// The warp's 32 x C tile (a lane's row in y[0 .. C - 1]) to out, rows row0 .. that are below m_end, columns n0 .. that are below
// n_end.  Through the warp's 4 KB of shared memory, so that a store instruction writes whole 64- or 128-byte runs of a few rows
// and not 16 bytes of 32 rows; element by element where rows are not 16-byte aligned.
template <typename OT, int C>
__device__ __forceinline__ void tile_out(OT* out, long long ld, int row0, int m_end, int n0, int n_end, const float (&y)[C], uint32_t buf,
                                         int lane) {
  constexpr int PER = 16 / sizeof(OT), CH = C / PER;   // elements of a 16-byte piece, pieces of a row (2, 4 or 8)
  OT* const base = out + (size_t)row0 * ld + n0;
  if ((reinterpret_cast<uintptr_t>(base) & 15) == 0 && (ld * sizeof(OT)) % 16 == 0) {
    constexpr int G = 8 / CH;                          // rows of a 128-byte line of the buffer
    auto at = [&](int r, int c) { return buf + r * (16 * CH) + ((c ^ ((r / G) & (CH - 1))) << 4); };
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (sizeof(OT) == 4) {
        sts128(at(lane, c), __float_as_uint(y[4 * c]), __float_as_uint(y[4 * c + 1]), __float_as_uint(y[4 * c + 2]), __float_as_uint(y[4 * c + 3]));
      } else {
        constexpr int P = C >= 8 ? 8 : C;
        const float* q = y + P * c;
        sts128(at(lane, c), pie::pack_bf16(q[0], q[1]), pie::pack_bf16(q[2], q[3]), pie::pack_bf16(q[4], q[5]), pie::pack_bf16(q[6], q[7]));
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int r = i * (32 / CH) + lane / CH, c = lane % CH, n = n0 + PER * c;
      const uint4 v = pie::lds128(at(r, c));
      if (row0 + r < m_end && n < n_end) {
        OT* dst = base + (size_t)r * ld + PER * c;
        if (n + PER <= n_end) {
          *reinterpret_cast<uint4*>(dst) = v;
        } else {
          const OT* e = reinterpret_cast<const OT*>(&v);
#pragma unroll
          for (int k = 0; k < PER; ++k)
            if (n + k < n_end) dst[k] = e[k];
        }
      }
    }
    __syncwarp();
    return;
  }
  if (row0 + lane < m_end)
#pragma unroll
    for (int q = 0; q < C; ++q)
      if (n0 + q < n_end) elem<OT>::store(base + (size_t)lane * ld + q, y[q]);
}

// 32 columns (n0 ..) of the warp's 32 rows (row0 ..; lane l holds row l's in v) through pieh_linear's epilogue; the whole warp
// calls it.  buf: the warp's 4 KB of shared memory.
template <typename OT>
__device__ __forceinline__ void umma_store(const LinArgs& a, int z, int row0, int m_end, int n0, const uint32_t (&v)[32], uint32_t buf,
                                           int lane) {
  if (a.epi == PIEH_EPI_GLU) {   // columns (2 j, 2 j + 1) are a (gate, linear) pair -> output column j
    float y[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) y[q] = glu_pair(a, __uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1]));
    tile_out<OT, 16>(reinterpret_cast<OT*>(a.out), a.out_ld, row0, m_end, n0 >> 1, a.N >> 1, y, buf, lane);
    return;
  }
  float y[32];
#pragma unroll
  for (int q = 0; q < 32; ++q) y[q] = __uint_as_float(v[q]);
  if (a.bias) {
    if (n0 + 32 <= a.N) {
#pragma unroll
      for (int q = 0; q < 32; ++q) y[q] += __ldg(a.bias + n0 + q);
    } else {
      const float mine = n0 + lane < a.N ? a.bias[n0 + lane] : 0.f;
#pragma unroll
      for (int q = 0; q < 32; ++q) y[q] += __shfl_sync(0xffffffffu, mine, q);
    }
  }
  if (act_in_loop(a.epi)) {
    tile_act_out<OT>(a, reinterpret_cast<OT*>(a.out) + (size_t)z * a.out_bs, a.out_ld, row0, m_end, n0, a.N, y, buf, lane);
    return;
  }
  switch (a.epi) {   // (outside the loops over columns)
    case PIEH_EPI_STREAMS: {
      if (n0 + 32 <= a.N && (a.N & 3) == 0 && (a.S == 1 || a.S == 2 || a.S == 4)) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          sts128(buf + lane * 128 + ((c ^ (lane & 7)) << 4), __float_as_uint(y[4 * c]), __float_as_uint(y[4 * c + 1]),
                 __float_as_uint(y[4 * c + 2]), __float_as_uint(y[4 * c + 3]));
        __syncwarp();
        const int n = n0 + 4 * (lane & 7);
        if (a.S == 1) streams_tile<1>(a, row0, m_end, n, buf, lane);
        else if (a.S == 2) streams_tile<2>(a, row0, m_end, n, buf, lane);
        else streams_tile<4>(a, row0, m_end, n, buf, lane);
        __syncwarp();
      } else if (row0 + lane < m_end) {
        float w[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) w[q] = y[q];
        streams_any(a, row0 + lane, n0, w);
      }
      return;
    }
    case PIEH_EPI_RELU2:
#pragma unroll
      for (int q = 0; q < 32; ++q) { y[q] = fmaxf(y[q], 0.f); y[q] = y[q] * y[q]; }
      break;
    case PIEH_EPI_SIGMUL:
      if (row0 + lane < m_end) {
        const float* gate = a.gate + (size_t)z * a.gate_bs + (size_t)(row0 + lane) * a.gate_ld + n0;
        if (n0 + 32 <= a.N && (reinterpret_cast<uintptr_t>(gate) & 15) == 0) {   // the gate logits of a whole run, 16 bytes at a time
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4) {
            const float4 g = *reinterpret_cast<const float4*>(gate + 4 * q4);
            y[4 * q4] /= 1.f + __expf(-g.x); y[4 * q4 + 1] /= 1.f + __expf(-g.y);
            y[4 * q4 + 2] /= 1.f + __expf(-g.z); y[4 * q4 + 3] /= 1.f + __expf(-g.w);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (n0 + q < a.N) y[q] *= 1.f / (1.f + __expf(-gate[q]));
        }
      }
      break;
    default: break;
  }
  tile_out<OT, 32>(reinterpret_cast<OT*>(a.out) + (size_t)z * a.out_bs, a.out_ld, row0, m_end, n0, a.N, y, buf, lane);
}

// One CTA per SM, four stages.  (Two CTAs per SM with 2 stages each, so that one's epilogue runs under the other's main loop,
// measured 20-30 % slower.)
template <typename OT>
__global__ void __launch_bounds__(kThreads, 1) linear_grouped_kernel(const __grid_constant__ LinArgs a) {
  constexpr int BM = 128, S = 4;
  constexpr int LAG = 2;                // k-steps of loads in flight behind the one the tensor core reads
  constexpr int A_STAGE = BM * kBK * 2, B_STAGE = kBN * kBK * 2;
  constexpr int TMEM_COLS = kBN;

  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S], accum_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  pie::pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smA = base, smB = base + S * A_STAGE;
  const int n0 = blockIdx.x * kBN;
  // this CTA's rows are one expert's run of slots (the whole CTA leaves before anything is set up)
  if ((int)blockIdx.y >= a.g_tiles[0]) return;
  const int32_t* tl = a.g_tiles + 1 + 3 * blockIdx.y;
  const __nv_bfloat16* wmat = reinterpret_cast<const __nv_bfloat16*>(a.w) + (size_t)tl[0] * a.g_wstride;
  const int m0 = tl[1], m_end = tl[1] + tl[2];
  const int nk = a.K / kBK;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) { pie::mbar_init(&full_bar[s], kProducers); pie::mbar_init(&empty_bar[s], 1); }
    pie::mbar_init(&accum_bar, 1);
    abort_flag = 0;
    pie::fence_mbar_init();
  }
  if (warp == kProducers / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  pie::pdl_launch_dependents();   // behind the allocation of tensor memory: a dependent that holds all of an SM's while it waits would keep this CTA from its own

  if (warp < kProducers / 32) {
    const int t = tid;
    const uint32_t swz = (uint32_t)(t & 7);
    const __nv_bfloat16* wsrc = wmat + (size_t)min(n0 + t, a.N - 1) * a.K;
    const int xslot = min(m0 + min(t, BM - 1), m_end - 1);
    const __nv_bfloat16* xsrc = reinterpret_cast<const __nv_bfloat16*>(a.x) +
                                (size_t)(a.g_rows ? a.g_rows[xslot] : xslot) * a.x_ld;
    bool alive = true;
    for (int kb = 0; kb < nk + LAG && alive; ++kb) {
      if (kb < nk) {
        const int s = kb % S, it = kb / S;
        if (it > 0) alive = wait_bounded(&empty_bar[s], (uint32_t)(it - 1) & 1, &abort_flag);
        if (alive) {
          if (t < BM) {
            const uint32_t dA = smA + s * A_STAGE + t * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) pie::cp_async16(dA + ((c ^ swz) << 4), xsrc + kb * kBK + c * 8);
          }
          const uint32_t dB = smB + s * B_STAGE + t * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) pie::cp_async16(dB + ((c ^ swz) << 4), wsrc + kb * kBK + c * 8);
        }
      }
      pie::cp_async_commit();
      if (kb >= LAG && alive) {
        pie::cp_async_wait<LAG>();
        pie::fence_proxy_async();
        pie::mbar_arrive(&full_bar[(kb - LAG) % S]);
      }
    }
    pie::cp_async_wait<0>();
    // ---- epilogue: this warp's TMEM lane quadrant
    if (alive) alive = wait_bounded(&accum_bar, 0, &abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (alive) {
      const int quad = warp & 3;
      const int c_lo = (warp >> 2) * (kBN / 64), c_hi = c_lo + kBN / 64;
      // every MMA has read its operands: the stages' memory is free
      const uint32_t buf = base + warp * 4096;
#pragma unroll 1
      for (int c = c_lo; c < c_hi; ++c) {
        uint32_t v[32];
        pie::tmem_ld32(tmem + (uint32_t)(c * 32) + ((uint32_t)(quad * 32) << 16), v);
        if (n0 + c * 32 < a.N) umma_store<OT>(a, 0, m0 + quad * 32, m_end, n0 + c * 32, v, buf, lane);
      }
    }
  } else {
    bool alive = true;
    for (int kb = 0; kb < nk && alive; ++kb) {
      const int s = kb % S;
      alive = wait_bounded(&full_bar[s], (uint32_t)(kb / S) & 1, &abort_flag);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (lane == 0 && alive) {
        const uint64_t da0 = pie::umma_desc_sw128(smA + s * A_STAGE), db0 = pie::umma_desc_sw128(smB + s * B_STAGE);
#pragma unroll
        for (int k4 = 0; k4 < kBK / 16; ++k4)
          pie::umma_bf16(tmem, da0 + 2 * k4, db0 + 2 * k4, IDESC, (kb > 0 || k4 > 0) ? 1u : 0u);
        pie::umma_commit(&empty_bar[s]);
        if (kb == nk - 1) pie::umma_commit(&accum_bar);
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kProducers / 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
}

// the epilogues as the GEMM core calls them
template <typename OT>
struct DenseEpi {
  LinArgs a;
  __device__ __forceinline__ void operator()(int z, int row0, int col, const uint32_t (&v)[32], uint32_t buf, int lane) const {
    if (row0 < a.M && col < a.N) umma_store<OT>(a, z, row0, a.M, col, v, buf, lane);
  }
};

bool linear_umma_ok(const LinArgs& a, int x_dtype, int w_dtype) {
  static const bool off = [] { const char* e = getenv("PIE_HYBRID_NO_UMMA"); return e && e[0] == '1'; }();
  if (off) return false;
  if (!a.g_tiles && a.N <= 32 && a.K % 8 == 0 && (reinterpret_cast<uintptr_t>(a.w) & 31) == 0 &&
      (reinterpret_cast<uintptr_t>(a.x) & 31) == 0 && a.epi != PIEH_EPI_GLU)
    return false;   // a handful of output columns: linear_skinny_kernel reads x once instead of filling 256-column tiles
  if (a.x_bs % 8 || a.w_bs % 8 || a.x_bs < 0 || a.w_bs < 0) return false;   // every product's operands start on a 16-byte boundary
  // what a tiled copy can describe: rows that go forward, strides below 2^40 bytes (rows that repeat or go backward: linear_tile_kernel)
  if (!a.g_tiles && (a.x_ld <= 0 || ((a.x_ld | a.x_bs | a.w_bs) >> 39) != 0)) return false;
  return x_dtype == PIE_DTYPE_BF16 && w_dtype == PIE_DTYPE_BF16 && a.M > 32 && a.K % kBK == 0 && a.x_ld % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0;
}

template <typename OT>
static cudaError_t launch_grouped(const LinArgs& a, cudaStream_t st) {
  constexpr size_t smem = (size_t)4 * (128 * kBK * 2 + kBN * kBK * 2) + 1024;
  static std::atomic<unsigned long long> served{0};
  const cudaError_t set = pie::once_per_device(served, [] {
    return cudaFuncSetAttribute(linear_grouped_kernel<OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  if (set != cudaSuccess) return set;
  // blockIdx.y walks the list of <= 128-slot tiles, whose length is only known on the device (S = experts)
  const dim3 grid((a.N + kBN - 1) / kBN, a.M / 128 + a.S, 1);
  count_launch();
  linear_grouped_kernel<OT><<<grid, kThreads, smem, st>>>(a);
  return cudaGetLastError();
}

template <typename OT>
static cudaError_t launch_dense(const LinArgs& a, cudaStream_t st) {
  pie::GemmArgs g = {};
  g.M = a.M; g.N = a.N; g.K = a.K; g.nb = a.nb;
  g.zx = a.x_bs != 0; g.zw = a.w_bs != 0;   // a stride of zero: one operand for all products
  const DenseEpi<OT> epi = {a};
  count_launch();
  return pie::gemm_run<0>(g, epi, a.x, a.x_ld * 2, a.x_bs * 2, a.w, a.w_bs * 2, num_sms(), st);
}

cudaError_t launch_linear_umma(const LinArgs& a, int out_dtype, cudaStream_t st) {
  if (out_dtype == PIE_DTYPE_BF16) return a.g_tiles ? launch_grouped<__nv_bfloat16>(a, st) : launch_dense<__nv_bfloat16>(a, st);
  return a.g_tiles ? launch_grouped<float>(a, st) : launch_dense<float>(a, st);
}

}  // namespace pieh

extern "C" unsigned int pieh_pipeline_error(void) { return pie::gemm_error_now(); }
extern "C" int pieh_pipeline_error_clear(void) { return pieh::status_of(pie::gemm_error_clear()); }
extern "C" int pieh_pipeline_words(unsigned int* words, void* stream) {
  return words ? pieh::status_of(pie::gemm_error_post(words, (cudaStream_t)stream)) : PIE_ENULL;
}
