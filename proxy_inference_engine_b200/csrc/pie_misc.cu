// Small operators of the decode path: quantize / dequantize, RMSNorm, SwiGLU glue, residual add, arg-max.
// Each cites the reference operator it stands in for (MLX = src/pie_core/external/mlx, PIE = src/proxy_inference_engine).
#include <cstdlib>

#include "pie_internal.h"
#include "pie_ptx.cuh"

namespace pie {

__device__ __forceinline__ float ld_as_f32(const void* p, long long i, int dtype) {
  return dtype == 0 ? bf16lo((uint32_t) reinterpret_cast<const uint16_t*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ void st_from_f32(void* p, long long i, int dtype, float v) {
  if (dtype == 0) reinterpret_cast<uint16_t*>(p)[i] = f2bf(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

// ---- a1 mx.quantize (MLX/mlx/backend/cpu/quantized.cpp:603-661): one thread per group, same op order ----
__global__ void quantize_kernel(const void* w, int dtype, uint32_t* wq, void* scales, void* biases,
                                long long n_groups, int gs, int bits) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_groups) return;
  const float n_bins = (float)((1 << bits) - 1);
  const int per = 32 / bits, ipg = gs / per;
  const long long w0 = i * gs;
  float w_min = INFINITY, w_max = -INFINITY;
  for (int j = 0; j < gs; ++j) {
    const float v = ld_as_f32(w, w0 + j, dtype);
    w_max = (w_max < v) ? v : w_max;
    w_min = (v < w_min) ? v : w_min;
  }
  const bool mask = fabsf(w_min) > fabsf(w_max);
  float scale = __fdiv_rn(w_max - w_min, n_bins);
  scale = (scale < 1e-7f) ? 1e-7f : scale;
  scale = mask ? scale : -scale;
  const float edge = mask ? w_min : w_max;
  const float q0 = rintf(__fdiv_rn(edge, scale));
  float bias = 0.f;
  if (q0 != 0.f) { scale = __fdiv_rn(edge, q0); bias = edge; }
  for (int j = 0; j < ipg; ++j) {
    uint32_t word = 0;
    for (int k = 0; k < per; ++k) {
      float e = ld_as_f32(w, w0 + (long long)j * per + k, dtype);
      e = rintf(__fdiv_rn(__fsub_rn(e, bias), scale));
      e = fminf(fmaxf(e, 0.f), n_bins);
      word |= ((uint32_t)e) << (k * bits);
    }
    wq[i * ipg + j] = word;
  }
  st_from_f32(scales, i, dtype, scale);
  st_from_f32(biases, i, dtype, bias);
}

cudaError_t launch_quantize(const void* w, int dtype, uint32_t* wq, void* s, void* b, long long rows, int K,
                            int gs, int bits, cudaStream_t st) {
  const long long ng = rows * (K / gs);
  if (ng == 0) return cudaSuccess;
  count_launch();
  quantize_kernel<<<(unsigned)((ng + 127) / 128), 128, 0, st>>>(w, dtype, wq, s, b, ng, gs, bits);
  return cudaGetLastError();
}

// ---- a4 mx.dequantize + row gather (MLX/mlx/fast.cpp:972-1017; quantized.py:100-107) ---------------------
// w_hat = bf16(bf16(q * scale) + bias); one thread per packed word.
__global__ void dequantize_kernel(uint16_t* out, const uint32_t* wq, const uint16_t* s, const uint16_t* b,
                                  const int32_t* ids, long long n_rows, long long table_rows, int K, int gs,
                                  int bits) {
  const int per = 32 / bits, wpr = K / per;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_rows * wpr) return;
  const long long i = idx / wpr;
  const int wi = (int)(idx % wpr);
  long long r = ids ? (long long)ids[i] : i;
  r = r < 0 ? 0 : (r >= table_rows ? table_rows - 1 : r);
  const uint32_t w = wq[r * wpr + wi];
  const int grp = wi * per / gs;
  const float sc = bf16lo((uint32_t)s[r * (K / gs) + grp]), bi = bf16lo((uint32_t)b[r * (K / gs) + grp]);
  const uint32_t mask = (1u << bits) - 1u;
  uint16_t* o = out + i * K + (long long)wi * per;
  for (int e = 0; e < per; ++e) o[e] = f2bf(bfround((float)((w >> (e * bits)) & mask) * sc) + bi);
}

cudaError_t launch_dequantize(uint16_t* out, const uint32_t* wq, const uint16_t* s, const uint16_t* b,
                              const int32_t* ids, long long n_rows, long long table_rows, int K, int gs,
                              int bits, int*, cudaStream_t st) {
  const long long n = n_rows * (K / (32 / bits));
  if (n == 0) return cudaSuccess;
  count_launch();
  dequantize_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, wq, s, b, ids, n_rows, table_rows, K, gs, bits);
  return cudaGetLastError();
}

// ---- a6 mx.fast.rms_norm (MLX/mlx/fast.cpp:93-111; kernels/rms_norm.metal:13-81) --------------------------
// fp32 sum of squares; out = bf16( bf16(x * inv) * w ): the cast to T comes BEFORE the weight multiply.  HBM-bound over many
// rows, one L2 round trip and a barrier over few: a CTA per row, the row held in registers between the two passes in 16-byte
// pieces, NV per thread (rms_norm_rows_kernel); rows that do not fit or are not aligned are read twice, element by element.
// 8192 rows of 4096: 39.0 -> 25.4 us (5.3 TB/s); 1531 of 2048: 8.7 -> 4.3.
__device__ __forceinline__ float rms_row_scale(float ss, int dims, float eps) {
  __shared__ float red[8];
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  return 1.0f / sqrtf(tot / (float)dims + eps);
}
template <int NV>
__global__ void __launch_bounds__(256) rms_norm_rows_kernel(uint16_t* out, const uint16_t* x, const uint16_t* w, int nvec, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  const uint4* xr = reinterpret_cast<const uint4*>(x) + (size_t)blockIdx.x * nvec;
  uint4* o = reinterpret_cast<uint4*>(out) + (size_t)blockIdx.x * nvec;
  uint4 v[NV], wv[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = threadIdx.x + 256 * j;
    v[j] = i < nvec ? xr[i] : make_uint4(0, 0, 0, 0);
    wv[j] = w && i < nvec ? __ldg(reinterpret_cast<const uint4*>(w) + i) : make_uint4(0, 0, 0, 0);
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const uint32_t q[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { ss = fmaf(bf16lo(q[e]), bf16lo(q[e]), ss); ss = fmaf(bf16hi(q[e]), bf16hi(q[e]), ss); }
  }
  const float inv = rms_row_scale(ss, nvec * 8, eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = threadIdx.x + 256 * j;
    if (i >= nvec) break;
    const uint32_t q[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, g[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w};
    uint32_t r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t n = pack_bf16(bf16lo(q[e]) * inv, bf16hi(q[e]) * inv);
      r[e] = w ? pack_bf16(bf16lo(n) * bf16lo(g[e]), bf16hi(n) * bf16hi(g[e])) : n;
    }
    o[i] = make_uint4(r[0], r[1], r[2], r[3]);
  }
}
__global__ void __launch_bounds__(256) rms_norm_kernel(uint16_t* out, const uint16_t* x, const uint16_t* w,
                                                       int dims, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  const uint16_t* xr = x + (size_t)blockIdx.x * dims;
  uint16_t* o = out + (size_t)blockIdx.x * dims;
  float ss = 0.f;
  for (int i = threadIdx.x; i < dims; i += 256) { const float v = bf16lo((uint32_t)xr[i]); ss += v * v; }
  const float inv = rms_row_scale(ss, dims, eps);
  for (int i = threadIdx.x; i < dims; i += 256) {
    float v = bfround(bf16lo((uint32_t)xr[i]) * inv);
    if (w) v = v * bf16lo((uint32_t)w[i]);
    o[i] = f2bf(v);
  }
}

static bool all_aligned16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

cudaError_t launch_rms_norm(uint16_t* out, const uint16_t* x, const uint16_t* w, long long rows, int dims,
                            float eps, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  count_launch();
  const unsigned n = (unsigned)rows;
  if (dims % 8 == 0 && dims <= 8192 && all_aligned16(out, x, w)) {
    auto rows_kernel = dims <= 2048 ? rms_norm_rows_kernel<1> : dims <= 4096 ? rms_norm_rows_kernel<2> : rms_norm_rows_kernel<4>;
    return launch_pdl(rows_kernel, dim3(n), dim3(256), 0, st, out, x, w, dims / 8, eps);
  }
  return launch_pdl(rms_norm_kernel, dim3(n), dim3(256), 0, st, out, x, w, dims, eps);
}

// ---- a11 glue (PIE/models/llama/language.py:126-127,150-154; nn.silu activations.py:125-132) ----------------
// Both read two arrays and write one: HBM-bound.  A thread takes 16 bytes of each per round where the arrays are 16-byte aligned
// (the last n % 8 elements, and arrays that are not, one element at a time).  8192 x 14336, us: SwiGLU 408 -> 130 (5.4 TB/s; it was
// bound by two-byte accesses and a full-range division), 8192 x 4096 sum 73 -> 28.
struct SiluMul {   // bf16 after every operator: sigmoid, gate * sigmoid, * up
  static __device__ __forceinline__ uint32_t pair(uint32_t g, uint32_t u) { return mul_bf16x2_rn(silu_bf16x2(g), u); }
};
struct Add {
  static __device__ __forceinline__ uint32_t pair(uint32_t a, uint32_t b) {
    return pack_bf16(bf16lo(a) + bf16lo(b), bf16hi(a) + bf16hi(b));
  }
};
template <class Op>
__global__ void __launch_bounds__(256) pairwise_kernel(uint16_t* out, const uint16_t* a, const uint16_t* b, long long nvec, long long n) {
  pdl_launch_dependents();
  pdl_wait();
  const long long step = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll 4
  for (long long i = first; i < nvec; i += step) {
    const uint4 x = reinterpret_cast<const uint4*>(a)[i], y = reinterpret_cast<const uint4*>(b)[i];
    reinterpret_cast<uint4*>(out)[i] = make_uint4(Op::pair(x.x, y.x), Op::pair(x.y, y.y), Op::pair(x.z, y.z), Op::pair(x.w, y.w));
  }
  for (long long i = 8 * nvec + first; i < n; i += step) out[i] = (uint16_t)Op::pair(a[i], b[i]);
}
template <class Op>
static cudaError_t launch_pairwise(uint16_t* out, const uint16_t* a, const uint16_t* b, long long n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  count_launch();
  const long long nvec = all_aligned16(out, a, b) ? n / 8 : 0, items = nvec ? nvec : n, grid = (items + 255) / 256;
  return launch_pdl(pairwise_kernel<Op>, dim3((unsigned)(grid < num_sms() * 8 ? grid : num_sms() * 8)), dim3(256), 0, st, out, a, b, nvec, n);
}
cudaError_t launch_silu_mul(uint16_t* out, const uint16_t* g, const uint16_t* u, long long n, cudaStream_t st) {
  return launch_pairwise<SiluMul>(out, g, u, n, st);
}
cudaError_t launch_add(uint16_t* out, const uint16_t* a, const uint16_t* b, long long n, cudaStream_t st) {
  return launch_pairwise<Add>(out, a, b, n, st);
}

// ---- greedy sampler: first index of the row maximum (mx.argmax; PIE/samplers/__init__.py, temp == 0) --------
__global__ void __launch_bounds__(1024) argmax_kernel(int32_t* out, const uint16_t* logits, int vocab,
                                                      int32_t* pos_adv, int32_t* seq_out, int seq_ld) {
  __shared__ float sv[32];
  __shared__ int si[32];
  const uint16_t* row = logits + (size_t)blockIdx.x * vocab;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < vocab; i += 1024) {
    const float v = bf16lo((uint32_t)row[i]);
    if (v > best || (v == best && i < bi)) { best = v; bi = i; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = sv[threadIdx.x]; bi = si[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (threadIdx.x == 0) {
      out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
      if (pos_adv) {  // the token just sampled occupies the next cache slot
        const int np = pos_adv[blockIdx.x] + 1;
        pos_adv[blockIdx.x] = np;
        if (seq_out && np < seq_ld) seq_out[(size_t)blockIdx.x * seq_ld + np] = bi == 0x7fffffff ? 0 : bi;
      }
    }
  }
}
// The same over a thread-block cluster of 8 CTAs per row (one 1024-thread CTA reading 256 KB of logits is a 16 us chain
// of L2 round trips at the end of every decode step): each CTA scans an eighth of the row with 16-byte loads, CTAs 1..7
// push their candidate into CTA 0's shared memory (st.async counted by CTA 0's mbarrier), CTA 0 merges in index order
// -- first maximum, as above -- and does the bookkeeping.  No global scratch, so concurrent calls cannot interfere.
constexpr int kAmCluster = 8;
__global__ void __launch_bounds__(1024) argmax_cluster_kernel(int32_t* out, const uint16_t* logits, int vocab,
                                                              int32_t* pos_adv, int32_t* seq_out, int seq_ld) {
  __shared__ float sv[32];
  __shared__ int si[32];
  __shared__ __align__(8) uint32_t cand[kAmCluster][2];   // CTA 0: (value bits, index) of every part
  __shared__ uint64_t bar;
  const int part = blockIdx.x % kAmCluster, r = blockIdx.x / kAmCluster, tid = threadIdx.x;
  if (part == 0 && tid == 0) {
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, (kAmCluster - 1) * 8);
    fence_mbar_init();
  }
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint16_t* row = logits + (size_t)r * vocab;
  const int per = ((vocab + kAmCluster - 1) / kAmCluster + 7) & ~7;   // multiple of 8 elements: 16-byte pieces
  const int i0 = part * per, i1 = min(vocab, i0 + per);
  float best = -INFINITY;
  int bi = 0x7fffffff;
  auto take = [&](float v, int i) { if (v > best || (v == best && i < bi)) { best = v; bi = i; } };
  if ((reinterpret_cast<uintptr_t>(row + i0) & 15) == 0) {
    const int nv = i1 > i0 ? (i1 - i0) / 8 : 0;
    for (int j = tid; j < nv; j += 1024) {
      const uint4 q = ldcg128(row + i0 + 8 * j);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) { take(bf16lo(w[e]), i0 + 8 * j + 2 * e); take(bf16hi(w[e]), i0 + 8 * j + 2 * e + 1); }
    }
    for (int i = i0 + 8 * nv + tid; i < i1; i += 1024) take(bf16lo((uint32_t)row[i]), i);
  } else {
    for (int i = i0 + tid; i < i1; i += 1024) take(bf16lo((uint32_t)row[i]), i);
  }
  auto merge = [&](float ov, int oi) { if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; } };
  for (int o = 16; o > 0; o >>= 1) merge(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if ((tid & 31) == 0) { sv[tid >> 5] = best; si[tid >> 5] = bi; }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // CTA 0's mbarrier is set up
  if (tid < 32) {
    best = sv[tid]; bi = si[tid];
    for (int o = 16; o > 0; o >>= 1) merge(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
    if (tid == 0) {
      if (part != 0) {
        uint32_t ra, rb;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(&cand[part][0])), "r"(0));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(smem_u32(&bar)), "r"(0));
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(ra),
                     "r"(__float_as_uint(best)), "r"((uint32_t)bi), "r"(rb) : "memory");
      } else {
        mbar_wait(&bar, 0);
        for (int p2 = 1; p2 < kAmCluster; ++p2) merge(__uint_as_float(cand[p2][0]), (int)cand[p2][1]);
        const int tok = bi == 0x7fffffff ? 0 : bi;
        out[r] = tok;
        if (pos_adv) {  // the token just sampled occupies the next cache slot
          const int np = pos_adv[r] + 1;
          pos_adv[r] = np;
          if (seq_out && np < seq_ld) seq_out[(size_t)r * seq_ld + np] = tok;
        }
      }
    }
  }
}

cudaError_t launch_argmax(int32_t* out, const uint16_t* logits, int rows, int vocab, int32_t* pos_adv,
                          int32_t* seq_out, int seq_ld, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  count_launch();
  static const bool no_cluster = getenv("PIE_ARGMAX_CLUSTER") && atoi(getenv("PIE_ARGMAX_CLUSTER")) == 0;
  if (!no_cluster && vocab >= 8192 && rows <= 64) {   // few long rows: the end of a decode step
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(rows * kAmCluster), 1, 1);
    cfg.blockDim = dim3(1024, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kAmCluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, argmax_cluster_kernel, out, logits, vocab, pos_adv, seq_out, seq_ld);
  }
  argmax_kernel<<<rows, 1024, 0, st>>>(out, logits, vocab, pos_adv, seq_out, seq_ld);
  return cudaGetLastError();
}

}  // namespace pie
