// Gated delta rule over ragged steps: a matrix state S [dk, dv] per (sequence, head) in fp32, carried in a slot.
//   per token:  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
// delta_prepare_kernel  short causal convolution (history of taps - 1 inputs per sequence slot) + silu on q, k, v; q and k
//                       to unit length (q also times dk^-1/2); beta = sigmoid(.), g = exp(-exp(A_log) softplus(. + dt_bias))
// conv_advance_kernel   moves every sequence's convolution history past this step's rows
// delta_scan_kernel     the recurrence: a column of S lives in the registers of R adjacent lanes (RPT rows each), so a
//                       token costs 4 RPT multiply-adds and one log2(R)-step shuffle round per thread and no barrier; the
//                       step's q / k / v rows are staged through shared memory a chunk of tokens at a time.  One warp per
//                       scheduler walks a serial chain, so what counts is the chain's length: rows of a column are dealt four
//                       at a time (a lane reads k and q 16 bytes at a time), a token's k is read while the token before it is
//                       worked on, and the decay is applied to S beside the shuffles, not in front of the prediction
//                       (S^T k with the old S, times g).  1200 rows, 16 heads of 128 x 128: 477 -> 244 us.
// delta_gate_kernel     per-head RMS norm of o, times the norm weight, times silu(gate)
// Everything that enters the recurrence is fp32; only delta_gate's output takes the act dtype.
#include "hyb_common.cuh"

namespace pieh {

constexpr int kMaxTaps = 8;

// grid (T, 2 G + H): one CTA per token and head-sized unit -- the G heads of q, the G heads of k, the H heads of v
__global__ void __launch_bounds__(128) delta_prepare_kernel(float* q, float* k, float* v, float* beta, float* decay,
                                                            const float* proj, long long ld, const pieh_delta d,
                                                            const pieh_batch b) {
  __shared__ float red[33];
  pdl_sync();
  const int t = blockIdx.x, u = blockIdx.y;
  const int i = b.tok_seq[t], start = b.seq_start[i], ctx = b.seq_ctx[i], slot = b.seq_slot[i];
  const int j = t - start;
  const int nq = d.G * d.dk, C = 2 * nq + d.H * d.dv, taps = d.taps;
  const float* hist = d.conv_state + (size_t)slot * (taps - 1) * C;
  const bool is_v = u >= 2 * d.G;
  const int n = is_v ? d.dv : d.dk;
  const int base = is_v ? 2 * nq + (u - 2 * d.G) * d.dv : u * d.dk;
  float y[4], ss = 0.f;   // n <= 512
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int c = base + threadIdx.x + 128 * e;
    y[e] = 0.f;
    if (threadIdx.x + 128 * e < n) {
      float acc = 0.f;
      for (int r = 0; r < taps; ++r) {
        float x;
        if (r <= j) x = proj[(size_t)(t - r) * ld + c];
        else {
          const int back = r - j;   // 1 .. taps - 1 tokens before this step
          x = ctx - back >= 0 ? hist[(size_t)(taps - 1 - back) * C + c] : 0.f;
        }
        acc = fmaf(d.conv_w[(size_t)c * taps + (taps - 1 - r)], x, acc);
      }
      y[e] = silu_f(acc);
      ss = fmaf(y[e], y[e], ss);
    }
  }
  float inv = 1.f;
  float* dst;
  if (is_v) dst = v + (size_t)t * d.H * d.dv + (base - 2 * nq);
  else {
    ss = block_sum(ss, red);
    inv = 1.f / sqrtf(ss + 1e-6f);
    if (u < d.G) { inv *= 1.f / sqrtf((float)d.dk); dst = q + (size_t)t * nq + base; }
    else dst = k + (size_t)t * nq + (base - nq);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (threadIdx.x + 128 * e < n) dst[threadIdx.x + 128 * e] = y[e] * inv;
  if (u == 0) {
    const float* row = proj + (size_t)t * ld + C + d.H * d.dv;   // behind the gate columns: b, then a
    for (int h = threadIdx.x; h < d.H; h += 128) {
      beta[(size_t)t * d.H + h] = 1.f / (1.f + expf(-row[h]));
      decay[(size_t)t * d.H + h] = expf(-expf(d.A_log[h]) * softplus_f(row[d.H + h] + d.dt_bias[h]));
    }
  }
}

// The same with a WARP per token and unit, four channels a lane (16-byte loads; units of n = dk or dv channels, multiples of 4):
// no barrier, a quarter of the loads and of the index arithmetic.  1200 rows of 48 units of 128: 84.9 -> 39.0 us, and 30.5 with a channel's
// weights in one load (a load a weight is 16 lines of 128 bytes each time, more than the rows').  TAPS: the convolution's length, its weights in registers.
template <int TAPS>
__global__ void __launch_bounds__(256) delta_prepare_warp_kernel(float* q, float* k, float* v, float* beta, float* decay,
                                                                 const float* proj, long long ld, const pieh_delta d,
                                                                 const pieh_batch b) {
  pdl_sync();
  constexpr int TOKENS = 4;                        // consecutive rows of a warp: the weights are read once for them
  const int lane = threadIdx.x & 31, u = blockIdx.y * 8 + (threadIdx.x >> 5), units = 2 * d.G + d.H;
  if (u >= units) return;
  const int nq = d.G * d.dk, C = 2 * nq + d.H * d.dv;
  const bool is_v = u >= 2 * d.G;
  const int n = is_v ? d.dv : d.dk, base = is_v ? 2 * nq + (u - 2 * d.G) * d.dv : u * d.dk;
  for (int c0 = 4 * lane; c0 < ((n + 127) & ~127); c0 += 128) {   // n <= 128 here unless the unit is a value (see below)
    const bool in = c0 < n;
    const int c = base + (in ? c0 : 0);
    static_assert(TAPS == 4, "a channel's weights are one load");
    float w[4][TAPS];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 f = __ldg(reinterpret_cast<const float4*>(d.conv_w) + c + e);
      w[e][0] = f.x; w[e][1] = f.y; w[e][2] = f.z; w[e][3] = f.w;
    }
#pragma unroll
    for (int x = 0; x < TOKENS; ++x) {
      const int t = blockIdx.x * TOKENS + x;
      if (t >= b.T) break;
      const int i = b.tok_seq[t], j = t - b.seq_start[i], ctx = b.seq_ctx[i];
      const float* hist = d.conv_state + (size_t)b.seq_slot[i] * (TAPS - 1) * C;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int r = 0; r < TAPS; ++r) {
        const int back = r - j;                    // > 0: that many tokens before this step
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        if (back <= 0) p = *reinterpret_cast<const float4*>(proj + (size_t)(t - r) * ld + c);
        else if (ctx - back >= 0) p = *reinterpret_cast<const float4*>(hist + (size_t)(TAPS - 1 - back) * C + c);
        acc.x = fmaf(w[0][TAPS - 1 - r], p.x, acc.x); acc.y = fmaf(w[1][TAPS - 1 - r], p.y, acc.y);
        acc.z = fmaf(w[2][TAPS - 1 - r], p.z, acc.z); acc.w = fmaf(w[3][TAPS - 1 - r], p.w, acc.w);
      }
      float4 y = make_float4(silu_f(acc.x), silu_f(acc.y), silu_f(acc.z), silu_f(acc.w));
      float* dst;
      if (is_v) {
        dst = v + (size_t)t * d.H * d.dv + (base - 2 * nq);
      } else {
        float ss = in ? fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, y.w * y.w))) : 0.f;
        float inv = 1.f / sqrtf(warp_sum(ss) + 1e-6f);
        if (u < d.G) { inv *= 1.f / sqrtf((float)d.dk); dst = q + (size_t)t * nq + base; }
        else dst = k + (size_t)t * nq + (base - nq);
        y.x *= inv; y.y *= inv; y.z *= inv; y.w *= inv;
      }
      if (in) *reinterpret_cast<float4*>(dst + c0) = y;
      if (u == 0) {
        const float* row = proj + (size_t)t * ld + C + d.H * d.dv;   // behind the gate columns: b, then a
        for (int h = lane; h < d.H; h += 32) {
          beta[(size_t)t * d.H + h] = 1.f / (1.f + expf(-row[h]));
          decay[(size_t)t * d.H + h] = expf(-expf(d.A_log[h]) * softplus_f(row[d.H + h] + d.dt_bias[h]));
        }
      }
    }
  }
}
// rows, channels and units that warps of four-channel lanes can take; a head's keys in one warp's pass (the norm is over them).  Few
// (row, unit) pairs are one or two waves of the other kernel's CTAs, and a warp's four rows in a row are a longer chain than that (16
// heads of 128, us, by CTAs / by warps: 4 rows 6.2 / 12.7, 57 rows 8.5 / 11.3, 300 rows 23.3 / 15.0; 8 heads of 16: 57 rows 6.0 / 10.3, 300
// rows 11.8 / 10.7).  Four taps are what the configurations have; another length takes the other kernel.
static bool delta_prepare_by_warps(const float* q, const float* k, const float* v, const float* proj, long long ld,
                                   const pieh_delta& d, int T) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                      reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(d.conv_state) | reinterpret_cast<uintptr_t>(d.conv_w);
  return (long long)T * (2 * d.G + d.H) >= 6144 && d.taps == 4 && d.dk <= 128 && d.dk % 4 == 0 && d.dv % 4 == 0 && ld % 4 == 0 && (p & 15) == 0;
}

__global__ void conv_advance_kernel(const float* proj, long long ld, const pieh_delta d, const pieh_batch b) {
  pdl_sync();
  const int i = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int C = 2 * d.G * d.dk + d.H * d.dv, taps = d.taps;
  if (c >= C) return;
  const int start = b.seq_start[i], n = b.seq_len[i], ctx = b.seq_ctx[i];
  float* hist = d.conv_state + (size_t)b.seq_slot[i] * (taps - 1) * C;
  float nv[kMaxTaps];
  for (int jj = 0; jj < taps - 1; ++jj) {
    const int p = ctx + n - (taps - 1) + jj;   // position this entry has to hold afterwards
    float x = 0.f;
    if (p >= ctx) x = proj[(size_t)(start + p - ctx) * ld + c];
    else if (p >= 0) x = hist[(size_t)(p - ctx + taps - 1) * C + c];
    nv[jj] = x;
  }
  for (int jj = 0; jj < taps - 1; ++jj) hist[(size_t)jj * C + c] = nv[jj];
}

constexpr int kScanThreads = 128, kScanChunk = 16;

__device__ __forceinline__ void cp_async_f(float* smem_dst, const float* gsrc, int bytes) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_dst);
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gsrc) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(gsrc) : "memory");
}

template <int RPT, int R, int CTAS>   // rows of a state column in a lane, lanes of a column, CTAs of an SM
__global__ void __launch_bounds__(kScanThreads, CTAS) delta_scan_kernel(float* o, const float* q, const float* k, const float* v,
                                                                     const float* beta, const float* decay,
                                                                     const pieh_delta d, const pieh_batch b) {
  extern __shared__ __align__(16) float sm[];
  pdl_sync();
  constexpr int cols = kScanThreads / R;
  const int h = blockIdx.y, i = blockIdx.z;
  const int hk = h / (d.H / d.G);
  const int start = b.seq_start[i], n = b.seq_len[i], ctx = b.seq_ctx[i];
  const int rl = threadIdx.x % R, cl = threadIdx.x / R;
  const int j = blockIdx.x * cols + cl;           // column of S (feature of v)
  const bool col_ok = j < d.dv;
  const int dk = d.dk, dv = d.dv;
  // two chunk buffers: while the recurrence walks one chunk of tokens, cp.async fills the other
  constexpr int dkp = RPT * R;                    // rows as the lanes hold them: dk and zeros behind
  constexpr int buf_floats = kScanChunk * (2 * dkp + cols + 2);
  float* S_g = d.state + (((size_t)b.seq_slot[i] * d.H + h) * dk) * dv;
  float S[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int row = (r >> 2) * 4 * R + 4 * rl + (r & 3);
    S[r] = (ctx > 0 && col_ok && row < dk) ? S_g[(size_t)row * dv + j] : 0.f;
  }
  const bool vec = (dk & 3) == 0;
  if (dkp != dk) {   // the zeros behind dk, once: no copy touches them
    for (int e = threadIdx.x; e < 2 * kScanChunk * 2 * (dkp - dk); e += kScanThreads) {
      const int line = e / (dkp - dk), c = dk + e - line * (dkp - dk);   // line: [buffer][k rows, q rows]
      sm[(line / (2 * kScanChunk)) * buf_floats + (line % (2 * kScanChunk)) * dkp + c] = 0.f;
    }
  }
  auto fill = [&](int which, int c0) {
    float* ks = sm + which * buf_floats;
    float* qs = ks + kScanChunk * dkp;
    float* vs = qs + kScanChunk * dkp;
    float* gb = vs + kScanChunk * cols;
    const int nc = min(kScanChunk, n - c0);
    if (vec) {
      const int per = dk >> 2;
      for (int e = threadIdx.x; e < nc * per; e += kScanThreads) {
        const int tt = e / per, r = (e - tt * per) << 2;
        const size_t src = ((size_t)(start + c0 + tt) * d.G + hk) * dk + r;
        cp_async_f(ks + tt * dkp + r, k + src, 16);
        cp_async_f(qs + tt * dkp + r, q + src, 16);
      }
    } else {
      for (int e = threadIdx.x; e < nc * dk; e += kScanThreads) {
        const int tt = e / dk, r = e - tt * dk;
        const size_t src = ((size_t)(start + c0 + tt) * d.G + hk) * dk + r;
        cp_async_f(ks + tt * dkp + r, k + src, 4);
        cp_async_f(qs + tt * dkp + r, q + src, 4);
      }
    }
    for (int e = threadIdx.x; e < nc * cols; e += kScanThreads) {
      const int tt = e / cols, c = e - tt * cols;
      const int jj = min(blockIdx.x * cols + c, dv - 1);
      cp_async_f(vs + e, v + ((size_t)(start + c0 + tt) * d.H + h) * dv + jj, 4);
    }
    for (int e = threadIdx.x; e < nc; e += kScanThreads) {
      cp_async_f(gb + 2 * e, decay + (size_t)(start + c0 + e) * d.H + h, 4);
      cp_async_f(gb + 2 * e + 1, beta + (size_t)(start + c0 + e) * d.H + h, 4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float out_prev = 0.f;   // this lane's share of the last token's read-out, not yet summed over the R lanes
  int row_prev = -1;
  fill(0, 0);
  for (int c0 = 0, which = 0; c0 < n; c0 += kScanChunk, which ^= 1) {
    const int nc = min(kScanChunk, n - c0);
    if (c0 + kScanChunk < n) {
      fill(which ^ 1, c0 + kScanChunk);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* ks = sm + which * buf_floats;
    const float* qs = ks + kScanChunk * dkp;
    const float* vs = qs + kScanChunk * dkp;
    const float* gb = vs + kScanChunk * cols;
    float kk[RPT], vv = vs[cl], g = gb[0], be = gb[1];
    auto load_rows = [&](float* dst, const float* row) {
#pragma unroll
      for (int r = 0; r < RPT; r += 4) {
        const float4 f = *reinterpret_cast<const float4*>(row + r * R + 4 * rl);
        dst[r] = f.x; dst[r + 1] = f.y; dst[r + 2] = f.z; dst[r + 3] = f.w;
      }
    };
    load_rows(kk, ks);
#pragma unroll 2
    for (int tt = 0; tt < nc; ++tt) {
      float pp[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < RPT; ++r) pp[r & 3] = fmaf(S[r], kk[r], pp[r & 3]);
      float pred = (pp[0] + pp[1]) + (pp[2] + pp[3]);
      float qq[RPT], kn[RPT];
      load_rows(qq, qs + tt * dkp);
      const int nx = min(tt + 1, nc - 1);
      load_rows(kn, ks + nx * dkp);
      const float vn = vs[nx * cols + cl], gn = gb[2 * nx], bn = gb[2 * nx + 1];
#pragma unroll
      for (int r = 0; r < RPT; ++r) S[r] *= g;
      // the read-out of the PREVIOUS token is reduced over the R lanes together with this token's prediction: two
      // independent shuffle chains instead of two in a row on the recurrence's critical path
#pragma unroll
      for (int off = 1; off < R; off <<= 1) {
        pred += __shfl_xor_sync(0xffffffffu, pred, off);
        out_prev += __shfl_xor_sync(0xffffffffu, out_prev, off);
      }
      if (row_prev >= 0 && rl == 0 && col_ok) o[((size_t)row_prev * d.H + h) * dv + j] = out_prev;
      const float u = be * (vv - g * pred);
      float oo[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        S[r] = fmaf(kk[r], u, S[r]);
        oo[r & 3] = fmaf(S[r], qq[r], oo[r & 3]);
        kk[r] = kn[r];
      }
      out_prev = (oo[0] + oo[1]) + (oo[2] + oo[3]);
      row_prev = start + c0 + tt;
      vv = vn; g = gn; be = bn;
    }
    __syncthreads();   // everyone is done with this buffer before the next fill overwrites it
  }
#pragma unroll
  for (int off = 1; off < R; off <<= 1) out_prev += __shfl_xor_sync(0xffffffffu, out_prev, off);
  if (row_prev >= 0 && rl == 0 && col_ok) o[((size_t)row_prev * d.H + h) * dv + j] = out_prev;
  if (col_ok) {
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int row = (r >> 2) * 4 * R + 4 * rl + (r & 3);
      if (row < dk) S_g[(size_t)row * dv + j] = S[r];
    }
  }
}

template <typename OT>
__global__ void delta_gate_kernel(OT* out, const float* o, const float* proj, long long ld, long long gate_off,
                                  const pieh_delta d, int T) {
  pdl_sync();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= T * d.H) return;
  const int t = w / d.H, h = w - t * d.H;
  const float* src = o + (size_t)w * d.dv;
  float ss = 0.f;
  for (int c = lane; c < d.dv; c += 32) ss = fmaf(src[c], src[c], ss);
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)d.dv + d.eps);
  const float* gate = proj + (size_t)t * ld + gate_off + (size_t)h * d.dv;
  for (int c = lane; c < d.dv; c += 32)
    elem<OT>::store(out + (size_t)w * d.dv + c, src[c] * inv * d.out_norm[c] * silu_f(gate[c]));
}

template <int RPT, int R>
static cudaError_t launch_scan(float* o, const float* q, const float* k, const float* v, const float* beta, const float* decay,
                               const pieh_delta& d, const pieh_batch& b, cudaStream_t st) {
  constexpr int cols = kScanThreads / R;
  constexpr size_t smem = (size_t)2 * kScanChunk * (2 * RPT * R + cols + 2) * 4;
  // One token a sequence (decode) is reading and writing the state: registers are worth most as CTAs in flight.  16 heads of 128 x 128,
  // 4 / 32 sequences, us: 162 registers 6.2 / 28.3, 124 registers 4.8 / 23.6.
  auto* kern = b.T == b.n_seq ? delta_scan_kernel<RPT, R, 4> : delta_scan_kernel<RPT, R, 1>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_k(kern, dim3((d.dv + cols - 1) / cols, d.H, b.n_seq), dim3(kScanThreads), smem, st, o, q, k, v,
                  beta, decay, d, b);
}

static bool delta_ok(const pieh_delta* d) {
  return d && d->H > 0 && d->G > 0 && d->H % d->G == 0 && d->dk > 0 && d->dv > 0 && d->taps >= 1 && d->taps <= kMaxTaps &&
         d->dk <= 512 && d->dv <= 512;
}

}  // namespace pieh

using namespace pieh;

extern "C" int pieh_delta_prepare(float* q, float* k, float* v, float* beta, float* decay, const float* proj, long long ld,
                                  const pieh_delta* d, const pieh_batch* b, void* stream) {
  if (!q || !k || !v || !beta || !decay || !proj || !d || !b) return PIE_ENULL;
  if (!delta_ok(d)) return PIE_EINVAL_SHAPE;
  if (b->T == 0) return PIE_OK;
  cudaStream_t st = (cudaStream_t)stream;
  count_launch(2);
  if (delta_prepare_by_warps(q, k, v, proj, ld, *d, b->T))
    launch_k(delta_prepare_warp_kernel<4>, dim3((b->T + 3) / 4, (2 * d->G + d->H + 7) / 8), dim3(256), 0, st, q, k, v, beta, decay, proj,
             ld, *d, *b);
  else
    launch_k(delta_prepare_kernel, dim3(b->T, 2 * d->G + d->H), dim3(128), 0, st, q, k, v, beta, decay, proj, ld, *d, *b);
  if (d->taps > 1) {
    const int C = 2 * d->G * d->dk + d->H * d->dv;
    launch_k(conv_advance_kernel, dim3((C + 127) / 128, b->n_seq), dim3(128), 0, st, proj, ld, *d, *b);
  }
  return status_of(cudaGetLastError());
}

extern "C" int pieh_delta_scan(float* o, const float* q, const float* k, const float* v, const float* beta,
                               const float* decay, const pieh_delta* d, const pieh_batch* b, void* stream) {
  if (!o || !q || !k || !v || !beta || !decay || !d || !b) return PIE_ENULL;
  if (!delta_ok(d)) return PIE_EINVAL_SHAPE;
  if (b->T == 0) return PIE_OK;
  // 16 rows of a state column per lane.  Measured on a 4096-row portion (dk = dv = 128, 16 heads, one sequence):
  // 8 rows per lane (16 lanes, 4 shuffle steps) 2.10 ms, 16 rows 1.74 ms, 32 rows (4 lanes, 2 steps, 64 CTAs) 2.62 ms
  constexpr int RPT = 16;
  cudaStream_t st = (cudaStream_t)stream;
  count_launch();
  if (d->dk <= RPT) return status_of(launch_scan<RPT, 1>(o, q, k, v, beta, decay, *d, *b, st));
  if (d->dk <= 2 * RPT) return status_of(launch_scan<RPT, 2>(o, q, k, v, beta, decay, *d, *b, st));
  if (d->dk <= 4 * RPT) return status_of(launch_scan<RPT, 4>(o, q, k, v, beta, decay, *d, *b, st));
  if (d->dk <= 8 * RPT) return status_of(launch_scan<RPT, 8>(o, q, k, v, beta, decay, *d, *b, st));
  if (d->dk <= 16 * RPT) return status_of(launch_scan<RPT, 16>(o, q, k, v, beta, decay, *d, *b, st));
  return status_of(launch_scan<RPT, 32>(o, q, k, v, beta, decay, *d, *b, st));
}

extern "C" int pieh_delta_gate(void* out, int out_dtype, const float* o, const float* proj, long long ld,
                               long long gate_off, const pieh_delta* d, int T, void* stream) {
  if (!out || !o || !proj || !d) return PIE_ENULL;
  if (!delta_ok(d)) return PIE_EINVAL_SHAPE;
  if (T == 0) return PIE_OK;
  const long long warps = (long long)T * d->H;
  count_launch();
  PIEH_DISPATCH_DTYPE(out_dtype, OT, launch_k(delta_gate_kernel<OT>, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, (OT*)out, o, proj, ld, gate_off, *d, T));
  return status_of(cudaGetLastError());
}
