// RoPE (mx.fast.rope, MLX/mlx/fast.cpp:353-511; kernels/rope.metal:6-47) and the KV-cache writes of
// ReusableKVCache.update_and_fetch (PIE/cache/kv_cache/reusable.py:96-142).
// theta = (pos + offset) * scale * (1 / freqs[i]) in fp32, range-reduced sine / cosine (rope_sincos, pie_ptx.cuh), one bf16 rounding at the store.
#include "pie_internal.h"
#include "pie_ptx.cuh"

namespace pie {

__device__ __forceinline__ size_t kv_addr(const KvLayout& kv, int b, int h, int t) {
  if (kv.page_table) {
    const int page = kv.page_table[(size_t)b * kv.pt_stride + t / kv.page_size];
    return ((size_t)page * kv.page_size + t % kv.page_size) * kv.tok_stride + (size_t)h * kv.head_stride;
  }
  return (size_t)b * kv.batch_stride + (size_t)h * kv.head_stride + (size_t)t * kv.tok_stride;
}

__device__ __forceinline__ float rope_inv_freq(const float* freqs, float base, int i, int half) {
  if (freqs) return 1.0f / freqs[i];
  return expf((float)(-i) * (logf(base) / (float)half));
}

// general form: x, out [n_batch, L, D]; rotates the first `dims` features
__global__ void rope_kernel(uint16_t* out, const uint16_t* x, long long rows, int L, int D, int dims,
                            int traditional, float base, float scale, int offset, const float* freqs) {
  const int half = dims / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per_row = D - half;  // `half` rotating pairs + (D - dims) pass-through features
  if (idx >= rows * per_row) return;
  const long long row = idx / per_row;
  const int i = (int)(idx % per_row);
  const uint16_t* xr = x + row * D;
  uint16_t* o = out + row * D;
  if (i >= half) { o[dims + (i - half)] = xr[dims + (i - half)]; return; }
  const int p = (int)(row % L);
  const float theta = ((float)p + (float)offset) * scale * rope_inv_freq(freqs, base, i, half);
  float s, c;
  rope_sincos(theta, &s, &c);
  const int i1 = traditional ? 2 * i : i, i2 = traditional ? 2 * i + 1 : i + half;
  const float x1 = bf16lo((uint32_t)xr[i1]), x2 = bf16lo((uint32_t)xr[i2]);
  o[i1] = f2bf(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
  o[i2] = f2bf(__fadd_rn(__fmul_rn(x1, s), __fmul_rn(x2, c)));
}

cudaError_t launch_rope(uint16_t* out, const uint16_t* x, long long n_batch, int L, int D, int dims,
                        int traditional, float base, float scale, int offset, const float* freqs,
                        cudaStream_t st) {
  const long long n = n_batch * L * (D - dims / 2);
  if (n == 0) return cudaSuccess;
  count_launch();
  rope_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, x, n_batch * L, L, D, dims, traditional, base,
                                                            scale, offset, freqs);
  return cudaGetLastError();
}

// The Llama form over whole heads: x [B, H, L, D] with any strides that are multiples of 8 elements (the projection's own rows
// [B, L, H D] seen as heads need no copy first), out [B, H, L, D] contiguous, every feature rotated with its half partner.
// HBM-bound: a thread takes 8 pairs (two 16-byte loads and stores) of one token for every HL-th head, so a sine serves H / HL
// heads; HL is large where there are few tokens (latency) and small where there are many.  A layer's q and k at
// 8192 tokens (32 + 8 heads of 128): copies 84 + rope_kernel 113 -> 33 us.  Same arithmetic as rope_kernel, bit for bit.
__global__ void __launch_bounds__(128) rope_heads_kernel(uint16_t* out, const uint16_t* x, int H, int L, int D, long long sb,
                                                         long long sh, long long sl, int offset, const float* freqs, int HL) {
  const int half = D / 2, PB = half / 8, pb = threadIdx.x % PB, rest = threadIdx.x / PB, hl = rest % HL;
  const int l = blockIdx.x * (128 / PB / HL) + rest / HL, b = blockIdx.y;
  if (l >= L) return;
  float sn[8], cs[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) rope_sincos(((float)l + (float)offset) * (1.0f / freqs[pb * 8 + e]), &sn[e], &cs[e]);
#pragma unroll 4
  for (int h = hl; h < H; h += HL) {
    const uint16_t* xr = x + b * sb + h * sh + l * sl + pb * 8;
    uint16_t* o = out + (((size_t)b * H + h) * L + l) * D + pb * 8;
    const uint4 v1 = *reinterpret_cast<const uint4*>(xr), v2 = *reinterpret_cast<const uint4*>(xr + half);
    const uint32_t a[4] = {v1.x, v1.y, v1.z, v1.w}, c[4] = {v2.x, v2.y, v2.z, v2.w};
    uint32_t r1[4], r2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x1 = bf16lo(a[e]), y1 = bf16hi(a[e]), x2 = bf16lo(c[e]), y2 = bf16hi(c[e]);
      r1[e] = pack_bf16(__fsub_rn(__fmul_rn(x1, cs[2 * e]), __fmul_rn(x2, sn[2 * e])),
                        __fsub_rn(__fmul_rn(y1, cs[2 * e + 1]), __fmul_rn(y2, sn[2 * e + 1])));
      r2[e] = pack_bf16(__fadd_rn(__fmul_rn(x1, sn[2 * e]), __fmul_rn(x2, cs[2 * e])),
                        __fadd_rn(__fmul_rn(y1, sn[2 * e + 1]), __fmul_rn(y2, cs[2 * e + 1])));
    }
    *reinterpret_cast<uint4*>(o) = make_uint4(r1[0], r1[1], r1[2], r1[3]);
    *reinterpret_cast<uint4*>(o + half) = make_uint4(r2[0], r2[1], r2[2], r2[3]);
  }
}

cudaError_t launch_rope_heads(uint16_t* out, const uint16_t* x, int B, int H, int L, int D, long long sb, long long sh,
                              long long sl, int offset, const float* freqs, cudaStream_t st) {
  const int lanes = 128 / (D / 16);   // (token, head) lanes of a block
  const int HL = (long long)B * L >= 1024 ? 4 : lanes, per = lanes / HL;
  count_launch();
  rope_heads_kernel<<<dim3((unsigned)((L + per - 1) / per), (unsigned)B), 128, 0, st>>>(out, x, H, L, D, sb, sh, sl, offset, freqs, HL);
  return cudaGetLastError();
}

// decode (L == 1): one CTA per (head, batch row) of the fused q/k/v projection output
// (Attention.__call__, PIE/models/llama/language.py:84-98): q heads are rotated into q_out, k heads are
// rotated into the cache at positions[b], v heads are copied into the cache.
__global__ void rope_kv_append_kernel(uint16_t* q_out, const uint16_t* qkv, uint16_t* kc, uint16_t* vc,
                                      const KvLayout kv, const int32_t* pos, const float* freqs, int Hq,
                                      int Hkv, int D) {
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.x, b = blockIdx.y, i = threadIdx.x, half = D / 2;
  const int p = pos[b];
  const uint16_t* src = qkv + ((size_t)b * (Hq + 2 * Hkv) + h) * D;
  if (h >= Hq + Hkv) {  // v: plain copy
    uint16_t* dst = vc + kv_addr(kv, b, h - Hq - Hkv, p);
    dst[i] = src[i];
    dst[i + half] = src[i + half];
    return;
  }
  const float theta = (float)p * (1.0f / freqs[i]);
  float s, c;
  rope_sincos(theta, &s, &c);
  const float x1 = bf16lo((uint32_t)src[i]), x2 = bf16lo((uint32_t)src[i + half]);
  const uint16_t o1 = f2bf(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
  const uint16_t o2 = f2bf(__fadd_rn(__fmul_rn(x1, s), __fmul_rn(x2, c)));
  uint16_t* dst = h < Hq ? q_out + ((size_t)b * Hq + h) * D : kc + kv_addr(kv, b, h - Hq, p);
  dst[i] = o1;
  dst[i + half] = o2;
}

cudaError_t launch_rope_kv_append(uint16_t* q_out, const uint16_t* qkv, uint16_t* kc, uint16_t* vc,
                                  const KvLayout& kv, const int32_t* pos, const float* freqs, int B, int Hq,
                                  int Hkv, int D, cudaStream_t st) {
  if (B == 0) return cudaSuccess;
  count_launch();
  return launch_pdl(rope_kv_append_kernel, dim3(Hq + 2 * Hkv, B), dim3(D / 2), 0, st, q_out, qkv, kc, vc, kv, pos, freqs, Hq,
                    Hkv, D);
}

// A layer's whole way from projected rows to attention in one launch: q [B, Hq, L, D] rotated into q_out (contiguous), k rotated and v copied
// into cache rows offset .. offset + L - 1, from wherever the rows lie; pos_out[b] = offset + L - 1 where a decode step asks for it.  Bit for
// bit what rope of q, rope of k and kv_write give, of which this replaces the three launches (and the fill of the positions): the rotated k is
// not written and read once more, and a layer of few rows is bound by its launches.  From the projection's end to this one's, three launches / one:
// 8192 tokens of 32 + 8 heads of 128 53 -> 40 us, 1531 of 64 16 -> 12.
// Few rows: a block per (token, head), a thread per pair -- one sine each, nothing but latency.
__global__ void rope_kv_pairs_kernel(uint16_t* q_out, int32_t* pos_out, const RopeRows r, uint16_t* kc, uint16_t* vc, const KvLayout kv,
                                     const float* freqs, int Hq, int Hkv, int D, int offset) {
  pdl_launch_dependents();
  pdl_wait();
  const int l = blockIdx.x, L = gridDim.x, h = blockIdx.y, b = blockIdx.z, i = threadIdx.x, half = D / 2;
  if (pos_out && h == 0 && i == 0 && l == L - 1) pos_out[b] = offset + l;
  if (h >= Hq + Hkv) {
    const uint16_t* src = r.v + b * r.vs.sb + (h - Hq - Hkv) * r.vs.sh + l * r.vs.sl;
    uint16_t* dst = vc + kv_addr(kv, b, h - Hq - Hkv, offset + l);
    dst[i] = src[i];
    dst[i + half] = src[i + half];
    return;
  }
  const uint16_t* src = h < Hq ? r.q + b * r.qs.sb + h * r.qs.sh + l * r.qs.sl : r.k + b * r.ks.sb + (h - Hq) * r.ks.sh + l * r.ks.sl;
  float s, c;
  rope_sincos(((float)l + (float)offset) * (1.0f / freqs[i]), &s, &c);
  const float x1 = bf16lo((uint32_t)src[i]), x2 = bf16lo((uint32_t)src[i + half]);
  uint16_t* dst = h < Hq ? q_out + (((size_t)b * Hq + h) * L + l) * D : kc + kv_addr(kv, b, h - Hq, offset + l);
  dst[i] = f2bf(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
  dst[i + half] = f2bf(__fadd_rn(__fmul_rn(x1, s), __fmul_rn(x2, c)));
}
// More: rope_heads_kernel's way over all Hq + 2 Hkv heads, 16 bytes an access, a token's sines for all heads of a lane.
__global__ void __launch_bounds__(128) rope_kv_heads_kernel(uint16_t* q_out, int32_t* pos_out, const RopeRows r, uint16_t* kc, uint16_t* vc,
                                                            const KvLayout kv, const float* freqs, int Hq, int Hkv, int L, int D,
                                                            int offset, int HL) {
  pdl_launch_dependents();
  pdl_wait();
  const int half = D / 2, PB = half / 8, pb = threadIdx.x % PB, rest = threadIdx.x / PB, hl = rest % HL;
  const int l = blockIdx.x * (128 / PB / HL) + rest / HL, b = blockIdx.y;
  if (l >= L) return;
  if (pos_out && l == L - 1 && hl == 0 && pb == 0) pos_out[b] = offset + l;
  float sn[8], cs[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) rope_sincos(((float)l + (float)offset) * (1.0f / freqs[pb * 8 + e]), &sn[e], &cs[e]);
  const size_t slot = kv_addr(kv, b, 0, offset + l) + pb * 8;
  // heads hl, hl + HL ...: the loads of four of them in flight before the first store
  auto heads = [&](const uint16_t* src, long long sh, uint16_t* dst, long long dh, int H, bool turn) {
    for (int h0 = hl; h0 < H; h0 += 4 * HL) {
      uint4 v1[4], v2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (h0 + i * HL < H) {
          const uint16_t* xr = src + (h0 + i * HL) * sh;
          v1[i] = *reinterpret_cast<const uint4*>(xr);
          v2[i] = *reinterpret_cast<const uint4*>(xr + half);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (h0 + i * HL >= H) break;
        if (turn) {
          const uint32_t a[4] = {v1[i].x, v1[i].y, v1[i].z, v1[i].w}, c[4] = {v2[i].x, v2[i].y, v2[i].z, v2[i].w};
          uint32_t r1[4], r2[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float x1 = bf16lo(a[e]), y1 = bf16hi(a[e]), x2 = bf16lo(c[e]), y2 = bf16hi(c[e]);
            r1[e] = pack_bf16(__fsub_rn(__fmul_rn(x1, cs[2 * e]), __fmul_rn(x2, sn[2 * e])),
                              __fsub_rn(__fmul_rn(y1, cs[2 * e + 1]), __fmul_rn(y2, sn[2 * e + 1])));
            r2[e] = pack_bf16(__fadd_rn(__fmul_rn(x1, sn[2 * e]), __fmul_rn(x2, cs[2 * e])),
                              __fadd_rn(__fmul_rn(y1, sn[2 * e + 1]), __fmul_rn(y2, cs[2 * e + 1])));
          }
          v1[i] = make_uint4(r1[0], r1[1], r1[2], r1[3]);
          v2[i] = make_uint4(r2[0], r2[1], r2[2], r2[3]);
        }
        uint16_t* o = dst + (h0 + i * HL) * dh;
        *reinterpret_cast<uint4*>(o) = v1[i];
        *reinterpret_cast<uint4*>(o + half) = v2[i];
      }
    }
  };
  heads(r.q + b * r.qs.sb + l * r.qs.sl + pb * 8, r.qs.sh, q_out + ((size_t)b * Hq * L + l) * D + pb * 8, (long long)L * D, Hq, true);
  heads(r.k + b * r.ks.sb + l * r.ks.sl + pb * 8, r.ks.sh, kc + slot, kv.head_stride, Hkv, true);
  heads(r.v + b * r.vs.sb + l * r.vs.sl + pb * 8, r.vs.sh, vc + slot, kv.head_stride, Hkv, false);
}

cudaError_t launch_rope_kv_rows(uint16_t* q_out, int32_t* pos_out, const RopeRows& r, uint16_t* kc, uint16_t* vc, const KvLayout& kv,
                                const float* freqs, int B, int Hq, int Hkv, int L, int D, int offset, cudaStream_t st) {
  if (B == 0 || L == 0) return cudaSuccess;
  count_launch();
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) |
                         reinterpret_cast<uintptr_t>(r.q) | reinterpret_cast<uintptr_t>(r.k) | reinterpret_cast<uintptr_t>(r.v);
  const long long strides = r.qs.sb | r.qs.sh | r.qs.sl | r.ks.sb | r.ks.sh | r.ks.sl | r.vs.sb | r.vs.sh | r.vs.sl | kv.batch_stride |
                            kv.head_stride | kv.tok_stride;
  // 32 + 8 heads, rows: pairs / heads, us, 32 2.1 / 2.9, 48 2.9 / 2.9, 64 3.6 / 2.9, 256 13.2 / 3.6 (D 64; 128 the same)
  if ((long long)B * L > 48 && (ptrs & 15) == 0 && strides % 8 == 0) {
    const int lanes = 128 / (D / 16), HL = (long long)B * L >= 1024 ? 4 : lanes, per = lanes / HL;
    return launch_pdl(rope_kv_heads_kernel, dim3((unsigned)((L + per - 1) / per), (unsigned)B), dim3(128), 0, st, q_out, pos_out, r, kc, vc, kv,
                      freqs, Hq, Hkv, L, D, offset, HL);
  }
  return launch_pdl(rope_kv_pairs_kernel, dim3((unsigned)L, (unsigned)(Hq + 2 * Hkv), (unsigned)B), dim3((unsigned)(D / 2)), 0, st, q_out,
                    pos_out, r, kc, vc, kv, freqs, Hq, Hkv, D, offset);
}

// prefill: k, v [B, Hkv, L, D], any strides with contiguous features -> cache rows offset .. offset + L - 1.  A copy: a thread per
// 16 bytes where everything is 16-byte aligned, else a block per row, element by element.  8192 tokens of
// 8 heads of 128: copy of v 42 + 36 -> 10 us.  Few rows are all latency, and a block that knows its row has no divisions in front of its
// loads: 32 rows of 64 1.7 us by rows, 2.1 by pieces, 256 rows 1.8 / 2.1, 1024 rows the same.
__global__ void __launch_bounds__(256) kv_write_vec_kernel(uint16_t* kc, uint16_t* vc, const KvLayout kv, const uint16_t* k,
                                                           const uint16_t* v, const KvSrc ks, const KvSrc vs, int Hkv, int L, int cpr,
                                                           int offset, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long row = i / cpr;                       // rows are walked (b, l, h): the order the projection wrote them in
  const int c = (int)(i - row * cpr) * 8, h = (int)(row % Hkv);
  const long long bl = row / Hkv;
  const int l = (int)(bl % L), b = (int)(bl / L);
  const size_t dst = kv_addr(kv, b, h, offset + l) + c;
  const uint4 kq = *reinterpret_cast<const uint4*>(k + b * ks.sb + h * ks.sh + l * ks.sl + c);
  const uint4 vq = *reinterpret_cast<const uint4*>(v + b * vs.sb + h * vs.sh + l * vs.sl + c);
  *reinterpret_cast<uint4*>(kc + dst) = kq;
  *reinterpret_cast<uint4*>(vc + dst) = vq;
}
__global__ void kv_write_kernel(uint16_t* kc, uint16_t* vc, const KvLayout kv, const uint16_t* k, const uint16_t* v,
                                const KvSrc ks, const KvSrc vs, int D, int offset) {
  const int l = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const uint16_t* kr = k + b * ks.sb + h * ks.sh + l * ks.sl;
  const uint16_t* vr = v + b * vs.sb + h * vs.sh + l * vs.sl;
  const size_t dst = kv_addr(kv, b, h, offset + l);
  for (int i = threadIdx.x; i < D; i += blockDim.x) { kc[dst + i] = kr[i]; vc[dst + i] = vr[i]; }
}

cudaError_t launch_kv_write(uint16_t* kc, uint16_t* vc, const KvLayout& kv, const uint16_t* k, const uint16_t* v, const KvSrc& ks,
                            const KvSrc& vs, int B, int Hkv, int L, int D, int offset, cudaStream_t st) {
  if (B == 0 || L == 0) return cudaSuccess;
  count_launch();
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) | reinterpret_cast<uintptr_t>(k) |
                         reinterpret_cast<uintptr_t>(v);
  const long long strides = ks.sb | ks.sh | ks.sl | vs.sb | vs.sh | vs.sl | kv.batch_stride | kv.head_stride | kv.tok_stride;
  if ((long long)B * L * Hkv > 512 && D % 8 == 0 && (ptrs & 15) == 0 && strides % 8 == 0) {
    const long long n = (long long)B * L * Hkv * (D / 8);
    kv_write_vec_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(kc, vc, kv, k, v, ks, vs, Hkv, L, D / 8, offset, n);
  } else {
    kv_write_kernel<<<dim3(L, Hkv, B), 64, 0, st>>>(kc, vc, kv, k, v, ks, vs, D, offset);
  }
  return cudaGetLastError();
}

}  // namespace pie
