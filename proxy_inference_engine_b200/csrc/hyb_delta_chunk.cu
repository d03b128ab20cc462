// The gated delta rule over prompts, 32 tokens at a time (fp32 throughout; one token at a time: delta_scan_kernel in hyb_delta.cu).
//   per token:  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
// With S the state in front of a chunk, G_t the product of its decays up to t and D[t, i] = g_{i+1} .. g_t, the chunk's u solve
//   u_t = beta_t v_t - beta_t G_t S^T k_t - sum_{i < t} A[t, i] u_i,   A[t, i] = beta_t D[t, i] (k_t . k_i),
// so U = U0 - W S, where U0 and W solve the same triangle for beta v and beta G k and know nothing of S; and with M[t, i] = D[t, i] (q_t . k_i), i <= t,
//   o = M U0 + (G q - M W) S,       S <- G S + sum_i D[end, i] k_i u_i^T.
// delta_chunk_kernel   a CTA per chunk and head, all at once: A, M, the triangle solved for the dk + dv columns of [W | U0], a thread a column, and the products of M
//                      with them.  (Half the threads with two columns each: 75 us for 56.)
// delta_walk_kernel    a CTA per head and 16 columns of S walks the chunks: [W; G q - M W] S, and the update of S.
// Ratios of decays are products of decays, never quotients: every one is at most 1 and none is 0 / 0 where a decay is tiny.  They and the products k . k and
// q . k, which most of the error comes from, are computed in double (on its matrix instructions) and rounded once.  Off from float64 by, o / state, a token
// at a time and so (1200 rows, 16 heads of 128 x 128, relative): keys as the model makes them 9.2e-8 / 8.0e-8 and 7.2e-8 / 7.5e-8, random 1.1e-7 / 8.0e-8 and
// 7.8e-8 / 7.6e-8, keys that all but coincide 5.9e-8 / 7.4e-8 and 8.8e-8 / 9.7e-8.
// The walk is a chain not of a token's few operations but of a chunk's two products through shared memory, which bound it: a token at a
// time is 200 ns.  1200 rows, 16 heads of 128 x 128, one sequence: 245 us -> 167 (chunks 56, walk 109).
// A sum of the chunk form holds terms that come later than the token (with a zero in front), and is in parts that may be infinite where the whole is
// not: where some u of a chunk, or some o, is no number, or infinite, the CTA takes that chunk a token at a time, so that it spoils what comes after it and
// nothing else.
#include "hyb_common.cuh"

namespace pieh {

constexpr int kC = 32;                       // tokens of a chunk
constexpr int kChunkThreads = 256, kWalkCols = 16, kWalkThreads = 256;

// scratch: W and G q - M W [T, H, dk], U0 [T, H, dv], (G_t, D[end, t]) [T, H, 2]
struct ChunkScratch { float *w, *q, *u, *a; };
__host__ __device__ inline size_t chunk_floats(int dk, int dv) { return 2 * (size_t)dk + dv + 2; }   // of a row and head
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

// C += A B of 8 x 8 x 4 in double: lane l has A[l / 4][l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}]
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

constexpr int kChunkCols = kChunkThreads;   // columns of [W | U0] in hand at once, one a thread
template <int DK>
struct ChunkSmem {
  static constexpr int LD = DK + 4;
  static constexpr int XS = kC * kChunkCols;    // the columns' values; before that, the warps' parts of A and M (60 tiles of 64 doubles: 7680 floats)
  static constexpr int FLOATS = 2 * kC * LD + 2 * kC * kC + XS;
};

template <int DK>
__global__ void __launch_bounds__(kChunkThreads, 3) delta_chunk_kernel(float* o, const ChunkScratch s, const float* q, const float* k, const float* v,
                                                                       const float* beta, const float* decay, const pieh_delta d, const pieh_batch b) {
  using L = ChunkSmem<DK>;
  constexpr int LD = L::LD;
  extern __shared__ __align__(16) float sm[];
  __shared__ double Ds[kC][kC + 1];
  __shared__ float bs[kC], gs[kC], Gs[kC];
  float *const ks = sm, *const qs = ks + kC * LD, *const As = qs + kC * LD, *const Ms = As + kC * kC, *const xs = Ms + kC * kC;
  pdl_sync();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x >> 1, h = blockIdx.y, hk = h / (d.H / d.G), dk = d.dk, dv = d.dv;
  const int i = b.tile_seq[tile], row0 = b.tile_row[tile] + (blockIdx.x & 1) * kC;
  const int n = min(kC, min(b.tile_row[tile] + 2 * kC, b.seq_start[i] + b.seq_len[i]) - row0);
  if (n <= 0) return;
#pragma unroll 4
  for (int e = tid; e < kC * (DK / 4); e += kChunkThreads) {
    const int t = e / (DK / 4), c = (e % (DK / 4)) * 4;
    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), qv = kv;
    if (t < n && c < dk) {
      const size_t at = ((size_t)(row0 + t) * d.G + hk) * dk + c;
      kv = *reinterpret_cast<const float4*>(k + at);
      qv = *reinterpret_cast<const float4*>(q + at);
    }
    *reinterpret_cast<float4*>(ks + t * LD + c) = kv;
    *reinterpret_cast<float4*>(qs + t * LD + c) = qv;
  }
  for (int e = tid; e < 2 * kC * kC; e += kChunkThreads) As[e] = 0.f;   // (and Ms behind it)
  if (tid < kC) {
    bs[tid] = tid < n ? beta[(size_t)(row0 + tid) * d.H + h] : 0.f;
    gs[tid] = tid < n ? decay[(size_t)(row0 + tid) * d.H + h] : 1.f;
  }
  __syncthreads();
  if (tid < kC) {                // D[., tid] and G
    double p = 1., g = 1.;
    for (int t = 0; t < kC; ++t) {
      const double gt = gs[t];
      if (t > tid) p *= gt;
      if (t <= tid) g *= gt;
      Ds[t][tid] = p;
    }
    Gs[tid] = (float)g;
    if (tid < n) *reinterpret_cast<float2*>(s.a + ((size_t)(row0 + tid) * d.H + h) * 2) = make_float2((float)g, tid == n - 1 ? 1.f : (float)Ds[n - 1][tid]);
  }
  // k . k (warps 0 to 3) and q . k (4 to 7) in tiles of 8 x 8 on and below the diagonal, every fourth run of four k a warp; a tile's parts meet in one warp
  const int part = warp & 3;
  const bool with_q = warp >= 4;
  double acc[10][2];             // [row of tiles r, column e <= r: r (r + 1) / 2 + e]
#pragma unroll
  for (int j = 0; j < 10; ++j) acc[j][0] = acc[j][1] = 0.;
#pragma unroll 1
  for (int c = 4 * part; c < DK; c += 16) {
    double kf[4], xf[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int at = (8 * r + (lane >> 2)) * LD + c + (lane & 3);
      kf[r] = ks[at];
      xf[r] = with_q ? qs[at] : ks[at];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e <= r; ++e) mma_f64(acc[r * (r + 1) / 2 + e], xf[r], kf[e]);
  }
  double2* const parts = reinterpret_cast<double2*>(xs) + (with_q ? 10 * 3 * 32 : 0);
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    const int from = ((part - j) & 3) - 1;   // -1: the tile's own warp
    if (from >= 0) parts[(j * 3 + from) * 32 + lane] = make_double2(acc[j][0], acc[j][1]);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int e = 0; e <= r; ++e) {
      const int j = r * (r + 1) / 2 + e;
      if ((j & 3) == part) {
        double y[2] = {acc[j][0], acc[j][1]};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
          const double2 p = parts[(j * 3 + f) * 32 + lane];
          y[0] += p.x; y[1] += p.y;
        }
        const int t = 8 * r + (lane >> 2);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int m = 8 * e + 2 * (lane & 3) + u;
          if (with_q) { if (m <= t) Ms[t * kC + m] = (float)(m < t ? Ds[t][m] * y[u] : y[u]); }
          else if (m < t) As[t * kC + m] = (float)((double)bs[t] * Ds[t][m] * y[u]);
        }
      }
    }
  __syncthreads();
  // A column of [W | U0] a thread: eight rows at a time, what the rows before them take from them in a loop (unrolled, the triangle is more
  // instructions than the caches hold), and the products of M with them on the way
  for (int c0 = tid; c0 < dk + dv; c0 += kChunkCols) {
    const bool is_v = c0 >= dk;
    const size_t step = (size_t)d.H * (is_v ? dv : dk), at = is_v ? ((size_t)row0 * d.H + h) * dv + (c0 - dk) : ((size_t)row0 * d.H + h) * dk + c0;
    float* const column = xs + tid;
#pragma unroll 8
    for (int t = 0; t < kC; ++t) column[t * kChunkCols] = bs[t] * (is_v ? (t < n ? v[at + t * step] : 0.f) : Gs[t] * ks[t * LD + c0]);
#pragma unroll 1
    for (int t0 = 0; t0 < kC; t0 += 8) {
      float y[8], m[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) y[r] = m[r] = 0.f;
#pragma unroll 1
      for (int j = 0; j < t0; j += 4) {
        const float* const p = column + j * kChunkCols;
        const float4 x = make_float4(p[0], p[kChunkCols], p[2 * kChunkCols], p[3 * kChunkCols]);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          y[r] += dot4(*reinterpret_cast<const float4*>(As + (t0 + r) * kC + j), x);
          m[r] += dot4(*reinterpret_cast<const float4*>(Ms + (t0 + r) * kC + j), x);
        }
      }
      float x[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float* const ar = As + (t0 + r) * kC + t0;
        const float* const mr = Ms + (t0 + r) * kC + t0;
        const float4 a0 = *reinterpret_cast<const float4*>(ar), a1 = *reinterpret_cast<const float4*>(ar + 4);
        const float4 m0 = *reinterpret_cast<const float4*>(mr), m1 = *reinterpret_cast<const float4*>(mr + 4);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, mm[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
        float p = 0.f, f = 0.f;
#pragma unroll
        for (int e = 0; e < r; ++e) { p = fmaf(a[e], x[e], p); f = fmaf(mm[e], x[e], f); }
        float* const place = column + (t0 + r) * kChunkCols;
        x[r] = *place - (y[r] + p);
        *place = x[r];
        m[r] += fmaf(mm[r], x[r], f);
        const int t = t0 + r;
        if (t < n) {
          (is_v ? s.u : s.w)[at + t * step] = x[r];
          if (is_v) o[at + t * step] = m[r];
          else s.q[at + t * step] = fmaf(Gs[t], qs[t * LD + c0], -m[r]);
        }
      }
    }
  }
}

__device__ __forceinline__ void walk_copy(float* dst, const float* src, int bytes) {
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(src) : "memory");
}

// two fp32 multiply-adds an instruction
typedef unsigned long long pair32;
__device__ __forceinline__ pair32 fma2(pair32 a, pair32 b, pair32 c) {
  pair32 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float2 halves(pair32 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

template <int DK>
struct WalkSmem {
  static constexpr int LD = DK + 4, RLD = 2 * kWalkCols + 4;
  static constexpr int BUF = 3 * kC * LD + kC * kWalkCols + kC * 2;       // W, G q - M W, K, U0, (G, R) of a chunk
  static constexpr int FLOATS = 2 * kWalkCols * LD + kC * RLD + 2 * BUF;  // S and half of an update (by column), R U, two chunks
};

// o holds M U0 on the way in: the thread that adds to an element reads it.
template <int DK>
__global__ void __launch_bounds__(kWalkThreads, 1) delta_walk_kernel(float* o, const ChunkScratch s, const float* q, const float* k, const float* v,
                                                                     const float* beta, const float* decay, const pieh_delta d, const pieh_batch b) {
  using L = WalkSmem<DK>;
  constexpr int LD = L::LD, RLD = L::RLD, J = DK / 32, PER = DK / 4;   // J: 32-wide pieces of K, four of each a lane of eight
  constexpr float top = 3.402823466e38f;
  extern __shared__ __align__(16) float sm[];
  float* const S = sm;                            // [column][k]
  float* const P = S + kWalkCols * LD;            // the second half of a chunk's tokens' update of S
  float* const Rs = P + kWalkCols * LD;           // [t][column]: R_t u_t, twice
  float* const bufs = Rs + kC * RLD;
  pdl_sync();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, i = blockIdx.z, hk = h / (d.H / d.G), j0 = blockIdx.x * kWalkCols, dk = d.dk, dv = d.dv;
  const int start = b.seq_start[i], len = b.seq_len[i], ctx = b.seq_ctx[i];
  if (len <= 0) return;
  float* const S_g = d.state + ((size_t)b.seq_slot[i] * d.H + h) * dk * dv;
  for (int e = tid; e < L::FLOATS; e += kWalkThreads) sm[e] = 0.f;      // (what no copy touches stays zero: k behind dk, columns behind dv)
  __syncthreads();
  if (ctx > 0)
    for (int e = tid; e < dk * kWalkCols; e += kWalkThreads) {
      const int r = e / kWalkCols, c = e % kWalkCols;
      if (j0 + c < dv) S[c * LD + r] = S_g[(size_t)r * dv + j0 + c];
    }
  auto fill = [&](int which, int c0) {
    float* const W = bufs + which * L::BUF;
    float *const Q = W + kC * LD, *const K = Q + kC * LD, *const U = K + kC * LD, *const A = U + kC * kWalkCols;
    const int n = min(kC, len - c0), c = tid % PER * 4;
#pragma unroll
    for (int t = tid / PER; t < kC; t += kWalkThreads / PER) {
      if (c >= dk) break;
      if (t < n) {
        const size_t row = start + c0 + t, wq = (row * d.H + h) * dk + c;
        walk_copy(W + t * LD + c, s.w + wq, 16);
        walk_copy(Q + t * LD + c, s.q + wq, 16);
        walk_copy(K + t * LD + c, k + (row * d.G + hk) * dk + c, 16);
      } else {                                    // the last chunk's missing rows
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(W + t * LD + c) = z;
        *reinterpret_cast<float4*>(Q + t * LD + c) = z;
        *reinterpret_cast<float4*>(K + t * LD + c) = z;
      }
    }
    if (tid < kC * (kWalkCols / 4)) {
      const int t = tid >> 2, e = (tid & 3) * 4;
      if (t < n && j0 + e < dv) walk_copy(U + t * kWalkCols + e, s.u + ((size_t)(start + c0 + t) * d.H + h) * dv + j0 + e, 16);
      else *reinterpret_cast<float4*>(U + t * kWalkCols + e) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < kC) {
      if (tid < n) walk_copy(A + 2 * tid, s.a + ((size_t)(start + c0 + tid) * d.H + h) * 2, 8);
      else A[2 * tid] = A[2 * tid + 1] = 0.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fill(0, 0);
  // Of [W; G q - M W] S a warp takes eight rows, a lane four columns (cg) and every eighth run of four k (kq); the eight lanes' parts meet so that lane
  // kq has row kq: the warps 0 to 3 u, the others o of the chunk's token t
  const int cg = lane >> 3, kq = lane & 7, t = 8 * (warp & 3) + kq;
  for (int c0 = 0, which = 0; c0 < len; c0 += kC, which ^= 1) {
    const int n = min(kC, len - c0);
    float* const mine = o + ((size_t)(start + c0 + t) * d.H + h) * dv + j0 + 4 * cg;
    const bool live = t < n && j0 + 4 * cg < dv;
    float4 first = make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp >= 4 && live) first = *reinterpret_cast<const float4*>(mine);
    if (c0 + kC < len) {
      fill(which ^ 1, c0 + kC);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* const W = bufs + which * L::BUF;      // W and behind it G q - M W: 64 rows
    const float *const K = W + 2 * kC * LD, *const U = K + kC * LD, *const A = U + kC * kWalkCols;
    pair32 two[8][4];          // sums over even and over odd k
#pragma unroll
    for (int r = 0; r < 8; ++r) two[r][0] = two[r][1] = two[r][2] = two[r][3] = 0;
#pragma unroll
    for (int jj = 0; jj < J; ++jj) {
      ulonglong2 sv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) sv[c] = *reinterpret_cast<const ulonglong2*>(S + (4 * cg + c) * LD + 32 * jj + 4 * kq);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(W + (8 * warp + r) * LD + 32 * jj + 4 * kq);
#pragma unroll
        for (int c = 0; c < 4; ++c) two[r][c] = fma2(w.y, sv[c].y, fma2(w.x, sv[c].x, two[r][c]));
      }
    }
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = halves(two[r][c]);
        acc[r][c] = f.x + f.y;
      }
    float y[4];
    {
      float a4[4][4], a2[2][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float keep = kq & 4 ? acc[r + 4][c] : acc[r][c], other = kq & 4 ? acc[r][c] : acc[r + 4][c];
          a4[r][c] = keep + __shfl_xor_sync(0xffffffffu, other, 4);
        }
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float keep = kq & 2 ? a4[r + 2][c] : a4[r][c], other = kq & 2 ? a4[r][c] : a4[r + 2][c];
          a2[r][c] = keep + __shfl_xor_sync(0xffffffffu, other, 2);
        }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float keep = kq & 1 ? a2[1][c] : a2[0][c], other = kq & 1 ? a2[0][c] : a2[1][c];
        y[c] = keep + __shfl_xor_sync(0xffffffffu, other, 1);
      }
    }
    if (warp < 4) {
      const float4 u0 = *reinterpret_cast<const float4*>(U + t * kWalkCols + 4 * cg);
      const float R = A[2 * t + 1];
      y[0] = u0.x - y[0]; y[1] = u0.y - y[1]; y[2] = u0.z - y[2]; y[3] = u0.w - y[3];
      const float r4[4] = {R * y[0], R * y[1], R * y[2], R * y[3]};
      *reinterpret_cast<float4*>(Rs + t * RLD + 8 * cg) = make_float4(r4[0], r4[0], r4[1], r4[1]);
      *reinterpret_cast<float4*>(Rs + t * RLD + 8 * cg + 4) = make_float4(r4[2], r4[2], r4[3], r4[3]);
    } else {
      y[0] += first.x; y[1] += first.y; y[2] += first.z; y[3] += first.w;
    }
    if (__syncthreads_or(!(fabsf(y[0]) <= top && fabsf(y[1]) <= top && fabsf(y[2]) <= top && fabsf(y[3]) <= top))) {
      // a token at a time, from S as it is: column tid / 16, rows 4 (tid % 16) + 64 x
      const int c = tid >> 4, r = tid & 15, j = min(j0 + c, dv - 1);
      for (int x = 0; x < n; ++x) {
        const size_t row = start + c0 + x;
        const float g = decay[row * d.H + h], be = beta[row * d.H + h];
        float pred = 0.f;
        for (int e = 4 * r; e < DK; e += 64)
          for (int y4 = 0; y4 < 4; ++y4) pred = fmaf(S[c * LD + e + y4], K[x * LD + e + y4], pred);
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) pred += __shfl_xor_sync(0xffffffffu, pred, off);
        const float u = be * (v[(row * d.H + h) * dv + j] - g * pred);
        float out = 0.f;
        for (int e = 4 * r; e < dk; e += 64)         // (only what exists: 0 * u is no zero here)
          for (int y4 = 0; y4 < 4; ++y4) {
            const float sn = fmaf(K[x * LD + e + y4], u, g * S[c * LD + e + y4]);
            S[c * LD + e + y4] = sn;
            out = fmaf(sn, q[(row * d.G + hk) * dk + e + y4], out);
          }
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) out += __shfl_xor_sync(0xffffffffu, out, off);
        if (r == 0 && j0 + c < dv) o[(row * d.H + h) * dv + j] = out;
      }
    } else {
      if (warp >= 4 && live) *reinterpret_cast<float4*>(mine) = make_float4(y[0], y[1], y[2], y[3]);
      // S <- G S + K^T (R U): four columns a pair of warps, a lane's run of four k; warp + 4 takes the second half of the tokens
      const int w4 = 4 * (warp & 3), r = 4 * lane;
      const bool has = r < DK;                       // (64 k: half of the lanes; the barrier below is for whole warps)
      float4 w[4];
      pair32 lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
      if (has) {
#pragma unroll 8
        for (int e = kC / 2 * (warp >> 2); e < kC / 2 * (warp >> 2) + kC / 2; ++e) {
          const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(K + e * LD + r);
          const ulonglong2 u01 = *reinterpret_cast<const ulonglong2*>(Rs + e * RLD + 2 * w4), u23 = *reinterpret_cast<const ulonglong2*>(Rs + e * RLD + 2 * w4 + 4);
          lo[0] = fma2(kv.x, u01.x, lo[0]); hi[0] = fma2(kv.y, u01.x, hi[0]);
          lo[1] = fma2(kv.x, u01.y, lo[1]); hi[1] = fma2(kv.y, u01.y, hi[1]);
          lo[2] = fma2(kv.x, u23.x, lo[2]); hi[2] = fma2(kv.y, u23.x, hi[2]);
          lo[3] = fma2(kv.x, u23.y, lo[3]); hi[3] = fma2(kv.y, u23.y, hi[3]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 a = halves(lo[c]), e = halves(hi[c]);
          w[c] = make_float4(a.x, a.y, e.x, e.y);
        }
        if (warp >= 4) {
#pragma unroll
          for (int c = 0; c < 4; ++c) *reinterpret_cast<float4*>(P + (w4 + c) * LD + r) = w[c];
        }
      }
      __syncwarp();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
      if (warp < 4 && has) {
        const float G = A[2 * (n - 1)];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float4* const at = reinterpret_cast<float4*>(S + (w4 + c) * LD + r);
          const float4 p = *reinterpret_cast<const float4*>(P + (w4 + c) * LD + r), old = *at;
          *at = make_float4(fmaf(G, old.x, w[c].x + p.x), fmaf(G, old.y, w[c].y + p.y), fmaf(G, old.z, w[c].z + p.z), fmaf(G, old.w, w[c].w + p.w));
        }
      }
    }
    __syncthreads();   // S is the next chunk's, and this buffer may be filled again
  }
  for (int e = tid; e < dk * kWalkCols; e += kWalkThreads) {
    const int r = e / kWalkCols, c = e % kWalkCols;
    if (j0 + c < dv) S_g[(size_t)r * dv + j0 + c] = S[c * LD + r];
  }
}

template <int DK>
static cudaError_t launch_chunks(float* o, const float* q, const float* k, const float* v, const float* beta, const float* decay, const pieh_delta& d,
                                 const pieh_batch& b, const ChunkScratch& s, cudaStream_t st) {
  constexpr size_t chunk_smem = ChunkSmem<DK>::FLOATS * 4, walk_smem = WalkSmem<DK>::FLOATS * 4;
  static std::atomic<unsigned long long> served{0};
  const cudaError_t set = pie::once_per_device(served, [] {
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chunk_smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(delta_walk_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem);
  });
  if (set != cudaSuccess) return set;
  const cudaError_t e = launch_k(delta_chunk_kernel<DK>, dim3(2 * b.n_tiles, d.H), dim3(kChunkThreads), chunk_smem, st, o, s, q, k, v, beta, decay, d, b);
  if (e != cudaSuccess) return e;
  return launch_k(delta_walk_kernel<DK>, dim3((d.dv + kWalkCols - 1) / kWalkCols, d.H, b.n_seq), dim3(kWalkThreads), walk_smem, st, o, s, q, k, v,
                  beta, decay, d, b);
}

// Where chunks are sooner done than a token at a time: as long as every column of S has an SM of its own (beyond that the other kernel, of which six CTAs
// share an SM, loses nothing), from sequences of 224 tokens on (from some 150 the two are within 5 us, and this is one launch more).  us, a token at a time /
// chunks, 16 heads of 128 x 128: 128 tokens 30 / 36, 256 56 / 46, 400 85 / 63, 4096 825 / 560; four sequences of 300 166 / 179; 32 heads, 1200 tokens 325 / 349; 16
// heads of 64 x 64: 128 tokens 27 / 29, 256 50 / 39, 1200 214 / 124.  (Scratch is 1.5 KB a row and head: up to half a GB, some 20000 rows.)
static bool chunks_pay(const pieh_delta& d, const pieh_batch& b) {
  return d.dk % 4 == 0 && d.dk > 32 && d.dk <= 128 && d.dv % 4 == 0 && b.n_tiles > 0 && b.T >= 224LL * b.n_seq &&
         (size_t)b.T * d.H * chunk_floats(d.dk, d.dv) * 4 <= (size_t)512 << 20 &&
         (long long)b.n_seq * d.H * ((d.dv + kWalkCols - 1) / kWalkCols) <= num_sms();
}

}  // namespace pieh

using namespace pieh;

extern "C" size_t pieh_delta_scan_scratch(const pieh_delta* d, const pieh_batch* b) {
  if (!d || !b || b->T <= 0 || d->H <= 0 || !chunks_pay(*d, *b)) return 0;
  return (size_t)b->T * d->H * chunk_floats(d->dk, d->dv) * 4;
}

extern "C" int pieh_delta_scan_chunks(float* o, const float* q, const float* k, const float* v, const float* beta, const float* decay,
                                      const pieh_delta* d, const pieh_batch* b, void* scratch, size_t scratch_bytes, void* stream) {
  if (!o || !q || !k || !v || !beta || !decay || !d || !b || !scratch) return PIE_ENULL;
  if (d->H <= 0 || d->G <= 0 || d->H % d->G || d->dk <= 0 || d->dv <= 0) return PIE_EINVAL_SHAPE;
  if (b->T == 0) return PIE_OK;
  if (d->dk % 4 || d->dk > 128 || d->dv % 4 || b->n_tiles <= 0 || b->n_seq > 65535 || d->H > 65535) return PIE_EUNSUPPORTED;
  const uintptr_t at = reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(scratch);
  if (at & 15) return PIE_EALIGN;
  const size_t rows = (size_t)b->T * d->H;
  if (scratch_bytes < rows * chunk_floats(d->dk, d->dv) * 4) return PIE_EWORKSPACE;
  ChunkScratch s;
  s.w = (float*)scratch;
  s.q = s.w + rows * d->dk;
  s.u = s.q + rows * d->dk;
  s.a = s.u + rows * d->dv;
  count_launch(2);
  return status_of(d->dk <= 64 ? launch_chunks<64>(o, q, k, v, beta, decay, *d, *b, s, (cudaStream_t)stream)
                               : launch_chunks<128>(o, q, k, v, beta, decay, *d, *b, s, (cudaStream_t)stream));
}
