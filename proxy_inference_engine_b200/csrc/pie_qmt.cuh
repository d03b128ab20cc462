// Quantized matmul for some dozens of activation rows, weights through tensor memory (tcgen05 + TMA, sm_100a); part of pie_qmm.cu.
//
//   y[m, n] = sum_k x[m, k] (s[n, g] q[n, k] + b[n, g]),   4- and 8-bit codes, groups of 64, 1 .. kQtMaxRows activation rows.
//
// The weights are the MMA's A operand (128 rows of the matrix a tile) and the activations its N side.  What bounds such a call is
// the stream of packed weights and, close behind it, the instructions that turn a code into an operand, so that is kept short:
//   * s (q - 8) of a 4-bit code has at most 11 significant bits (8 of a bf16 scale, 3 of q - 8): it IS an fp16 number.  A thread lifts
//     two codes with one mask-or and an exact multiply-add or two: 11 instructions for eight codes, and the products of many
//     groups can run on in one fp32 accumulator of tensor memory -- no sums per group to be scaled and added afterwards.
//   * an 8-bit code is two of them, q = 16 h + l: h against 16 x and l against x.  One kernel serves both; a matrix of 8-bit codes
//     is a matrix of twice as many 4-bit ones, in the order the bytes have.
//   * what is missing, (8 s + b) times the group's sum of x (136 s + b), is 16 more columns of K behind every 128 codes, the sum in three
//     fp16 pieces (33 bits).
//   * the operand goes from registers straight to tensor memory (a thread per row of the tile, tcgen05.st), where the MMA reads it:
//     through shared memory it would cost 2 bytes written and 2 read for each half byte that arrives, and that was the limit of
//     the earlier kernels.
// x as fp16: the preparing kernel (RMS norm of the rows where asked for) scales each row by the power of two that brings its
// largest value into [256, 512) (8 bits: [16, 32)), the most that a group's sum leaves room for, which is exact down to 2^-25 (2^-21) of it, and
// 2^-33 (2^-29) of it is the largest error below; the GEMV, whose operands are 128 + q, loses 2^-17 of a group's largest value.  It writes the rows in the order
// the codes are lifted in.  Scales from 6e-8 to 7 (or 0) and |b| < 512 fit; a row of the matrix with others is marked (its operand
// becomes NaN) and summed in fp32 by the warp that finds the NaN: slow, and right.  A row of x with infinities is found the same way, and its results are
// what they make of the weights' signs.
// Roles of a CTA (one an SM): warp 0 packed rows, scales and biases by TMA; warp 1 the prepared x by bulk copies; warp 2 MMAs; warps 4-7
// the results; warps 8-19 in three sets dequantise, 128 codes of 128 rows in turn.  The work, tiles x 256 codes, is dealt out evenly: a
// CTA's share may begin and end inside a tile, and the CTA that comes last adds a tile's parts, in the order of K.
// Measured, 4 bits, us a call with the preparing kernel (the kernels before it: mma.sync GEMV in passes of 32 rows, or the tile kernel from 64
// rows on -> this one): 4096 x 14336 16 rows 27.6 -> 17.5, 32 37.1 -> 20.9, 48 62.0 -> 25.2; 2 x 14336 x 4096 with SwiGLU 16 rows 42.5 -> 27.0,
// 32 60.5 -> 32.5, 77 54.6 -> 47.5; 128256 x 4096 16 rows 147 -> 74.5 (4.0 TB/s of packed weights), 32 198 -> 82.  A call of next to no work takes
// 10: 3 of preparation, 2 until the first words are there, 1.3 for the first turn, 3.5 from the last sum to the stored result.  What
// bounds the rest is issue and the chain of a turn: 3800 warp instructions for 256 codes of 128 rows, set-up and hand-over among them (4096 x 14336, 16
// rows: issue slots 45 % busy, half of that launch being set-up and hand-over), 0.6 us a turn where the words alone would take 0.37.
// Tried and left: operands of a whole turn unrolled, or the next quarter's words and scales ahead (no faster: 73 -> 76 for the head), more
// accumulators (no change), scales in a ring of their own (73 -> 79), MMAs handed over by 128 codes (84: the issuing warp's turn-round).
#pragma once
#include "pie_gemm.cuh"
#include "pie_internal.h"

namespace pie {

constexpr int kQtMaxRows = kQmtRows, kQtMaxK = 32768;
constexpr int kQtPacked = 128 * 128;            // packed bytes of a stage: 128 rows, 256 codes
constexpr int kQtStage = kQtPacked + 2 * 128 * 16;   // ... and scales and biases of 128 rows, the 8 groups its own are among
constexpr int kQtCols = 72;                     // tensor-memory columns of 128 codes (64) and the 16 columns behind them (8)
constexpr int kQtMaxStages = 9;               // what 16 rows leave room for
constexpr int kQtThreads = 640;
constexpr int kQtSmem = 226 * 1024;             // dynamic; the barriers are static

struct QtSeg { const uint32_t* wq; const uint16_t *s, *b; int N, tile0, out_off; };
struct QtArgs {
  int nseg, dual, M, K, np;       // np: M rounded up to 16
  int ntiles, ks;                 // tiles of 128 rows (dual: 64 and 64), stages of a tile
  int nw;                         // stages of packed rows
  int split;                      // > 0: a tile is this many CTAs', and a CTA has no part of a second one
  int run;                        // turns that one accumulator takes; more are added in fp32
  int totals_smem;                // where: tensor memory has no room for 32 columns more of turns of 256 codes
  int epi, out_ld;
  uint32_t mask0, mask1, magic0, magic1;   // of qt_word: as arguments, so that a mask-or is one instruction
  QtSeg seg[kMaxSeg];
  uint16_t* out;
  const uint16_t* residual;
  const uint8_t* img;             // prepared x: per 128 codes [18][np][8] fp16
  const float* rscale;            // [np] what a row's sums are multiplied by
  float* part;                    // [2 grid][np][128]
  unsigned int* cnt;              // [ntiles], zeroed by the preparing kernel
  CUtensorMap wmap[kMaxSeg], smap[kMaxSeg], bmap[kMaxSeg];
};

// ---- activations -> fp16 rows in lifting order, row scales, group sums --------------------------------------------------------------
__device__ __forceinline__ uint32_t qt_pack_f16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ float qt_f16lo(uint32_t v) {
  float f;
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tcvt.f32.f16 %0, l;\n\t}" : "=f"(f) : "r"(v));
  return f;
}
__device__ __forceinline__ float qt_f16hi(uint32_t v) { return qt_f16lo(v >> 16); }
__device__ __forceinline__ uint32_t qt_fma(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t qt_mul(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t qt_add(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// v in three fp16 pieces: the pieces' bits as (p0, p1, p2)
__device__ __forceinline__ void qt_pieces(float v, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = qt_pack_f16(v, 0.f) & 0xffffu;
  const float r = v - qt_f16lo(p0);
  p1 = qt_pack_f16(r, 0.f) & 0xffffu;
  p2 = qt_pack_f16(r - qt_f16lo(p1), 0.f) & 0xffffu;
}

// Where entry i of a row's list of infinities lies in its image: k, and bit 15 for a negative one.
__device__ __forceinline__ size_t qt_list_at(unsigned int i, int np, int m) {
  return (size_t)(i >> 7) * np * 288 + (size_t)((i >> 3 & 15) * np + m) * 16 + (i & 7) * 2;
}

// One CTA per row.  U: 8 * 1024 * U >= K.
template <int BITS, int U>
__global__ void __launch_bounds__(1024) qmt_prep_kernel(uint8_t* img, float* rscale, unsigned int* cnt, int ntiles, const uint16_t* x,
                                                        int x_ld, const uint16_t* norm_w, float eps, int np, int K) {
  __shared__ float red[64];
  __shared__ unsigned int infinities;
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, chunks = K / 8;
  // the matmul may set itself up and ask for weights, which nothing queued before it writes any more, but reads nothing of this kernel
  pdl_wait();
  pdl_launch_dependents();
  if (m == 0)
    for (int i = tid; i < ntiles; i += 1024) cnt[i] = 0;
  uint4 v[U];
  float ss = 0.f;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = u * 1024 + tid;
    v[u] = make_uint4(0, 0, 0, 0);
    if (c < chunks) v[u] = ldcg128(x + (size_t)m * x_ld + (size_t)c * 8);
  }
  if (norm_w) {
    uint4 w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = u * 1024 + tid;
      w[u] = make_uint4(0, 0, 0, 0);
      if (c < chunks) w[u] = __ldg(reinterpret_cast<const uint4*>(norm_w) + c);
      const uint32_t x4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float lo = bf16lo(x4[j]), hi = bf16hi(x4[j]); ss = fmaf(lo, lo, ss); ss = fmaf(hi, hi, ss); }
    }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    const float inv = 1.0f / sqrtf(warp_sum(red[lane]) / (float)K + eps);
#pragma unroll
    for (int u = 0; u < U; ++u) {   // mx.fast.rms_norm: bf16(bf16(x * inv) * w)   (MLX/mlx/fast.cpp:93-111)
      uint32_t* const x4 = reinterpret_cast<uint32_t*>(&v[u]);
      const uint32_t w4[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        x4[j] = pack_bf16(bfround(bf16lo(x4[j]) * inv) * bf16lo(w4[j]), bfround(bf16hi(x4[j]) * inv) * bf16hi(w4[j]));
    }
  }
  uint32_t top = 0;   // largest magnitude, as bits
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t x4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) top = max(top, max(x4[j] & 0x7fffu, (x4[j] >> 16) & 0x7fffu));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) reinterpret_cast<uint32_t*>(red)[32 + warp] = top;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, reinterpret_cast<uint32_t*>(red)[32 + lane]);
  // x 2^sh has its largest value in [256, 512), or in [16, 32) where 16 x is to be a number as well; infinities and NaN stay what they are
  const int e = max((int)(top >> 7), 1) - 127;
  const int sh = top == 0 || e == 128 ? 0 : (BITS == 4 ? 8 : 4) - e;     // -123 .. 134
  const float f1 = __int_as_float((127 + sh / 2) << 23), f2 = __int_as_float((127 + sh - sh / 2) << 23);
  // 2^-141 at the least: a subnormal, and exact.  A row with a NaN has NaN for results, and nobody looks for a marked row there; one
  // with infinities and none has their number here, negative, and a list of them for an image.
  if (tid == 0 && top != 0x7f80u) rscale[m] = e == 128 ? __int_as_float(0x7fffffff) : ldexpf(1.f, -sh - 7);
  const size_t slot_bytes = (size_t)np * 288;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = u * 1024 + tid;
    if (U > 1 && __all_sync(0xffffffffu, c >= chunks)) break;
    const uint32_t x4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
    uint32_t h[4];   // fp16 (x0, x1) (x2, x3) (x4, x5) (x6, x7)
    float sum = 0.f, sum16 = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[j] = qt_pack_f16(bf16lo(x4[j]) * f1 * f2, bf16hi(x4[j]) * f1 * f2);
      sum += qt_f16lo(h[j]) + qt_f16hi(h[j]);
    }
    if (BITS == 4) {
      // codes 0 .. 7 of a word are lifted in pairs (0, 4) (1, 5) (2, 6) (3, 7)
      const uint4 o = make_uint4(__byte_perm(h[0], h[2], 0x5410), __byte_perm(h[0], h[2], 0x7632), __byte_perm(h[1], h[3], 0x5410),
                                 __byte_perm(h[1], h[3], 0x7632));
      if (c < chunks) *reinterpret_cast<uint4*>(img + (size_t)(c >> 4) * slot_bytes + (size_t)((c & 15) * np + m) * 16) = o;
    } else {
      // 4-bit codes 2 k (low, x) and 2 k + 1 (high, 16 x): word pairs (x0, x2) (16 x0, 16 x2) (x1, x3) (16 x1, 16 x3)
      uint32_t t[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        t[j] = qt_pack_f16(bf16lo(x4[j]) * f1 * f2 * 16.f, bf16hi(x4[j]) * f1 * f2 * 16.f);
        sum16 += qt_f16lo(t[j]) + qt_f16hi(t[j]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 o = make_uint4(__byte_perm(h[2 * i], h[2 * i + 1], 0x5410), __byte_perm(t[2 * i], t[2 * i + 1], 0x5410),
                                   __byte_perm(h[2 * i], h[2 * i + 1], 0x7632), __byte_perm(t[2 * i], t[2 * i + 1], 0x7632));
        const int w = 2 * c + i;
        if (c < chunks) *reinterpret_cast<uint4*>(img + (size_t)(w >> 4) * slot_bytes + (size_t)((w & 15) * np + m) * 16) = o;
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (BITS == 8) sum16 += __shfl_xor_sync(0xffffffffu, sum16, o);
    }
    if ((c & 7) == 0 && c < chunks) {   // the group's sums, against (E, E, E, B, B, B) / (E x 3, E x 3, B x 3)
      const int g = c >> 3;
      uint32_t p0, p1, p2;
      qt_pieces(sum, p0, p1, p2);
      if (BITS == 4) {
        uint8_t* const at = img + (size_t)(g >> 1) * slot_bytes + (size_t)((16 + (g & 1)) * np + m) * 16;
        *reinterpret_cast<uint4*>(at) = make_uint4(p0 | p1 << 16, p2 | p0 << 16, p1 | p2 << 16, 0);
      } else {
        uint32_t q0, q1, q2, r0, r1, r2;
        qt_pieces(sum16, q0, q1, q2);
        qt_pieces(sum16 * 0.0625f, r0, r1, r2);
        uint8_t* const at = img + (size_t)g * slot_bytes + (size_t)(16 * np + m) * 16;
        *reinterpret_cast<uint4*>(at) = make_uint4(p0 | p1 << 16, p2 | q0 << 16, q1 | q2 << 16, r0 | r1 << 16);
        *reinterpret_cast<uint4*>(at + (size_t)np * 16) = make_uint4(r2, 0, 0, 0);
      }
    }
  }
  if (top == 0x7f80u) {   // (what the MMAs make of a list stays in the row's own column)
    __syncthreads();
    if (tid == 0) infinities = 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t x4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t b = j & 1 ? x4[j / 2] >> 16 : x4[j / 2] & 0xffffu;
        if ((b & 0x7fffu) == 0x7f80u)
          *reinterpret_cast<uint16_t*>(img + qt_list_at(atomicAdd(&infinities, 1u), np, m)) = (uint16_t)(((u * 1024 + tid) * 8 + j) | (b & 0x8000u));
      }
    }
    __syncthreads();
    if (tid == 0) {
      *reinterpret_cast<uint16_t*>(img + (size_t)(16 * np + m) * 16) = 0x7fff;   // a group's sum: NaN for all results, which sends for the list
      rscale[m] = -(float)infinities;
    }
  }
}

// ---- the matmul ---------------------------------------------------------------------------------------------------------------------
// shared-memory descriptor of a K-major operand without swizzle: 16-byte rows of 8 k, 8 rows in a run of 128 bytes, runs one behind
// the other along N, the next 8 k np * 16 bytes on
__device__ __forceinline__ uint64_t qt_desc_x(uint32_t smem_addr, int np) {
  return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)np << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
// (without a cache hint: the lines of scales are come back to)
__device__ __forceinline__ void qt_tma_2d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
               "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void qt_tmem_st4(uint32_t taddr, uint32_t u0, uint32_t u1, uint32_t u2, uint32_t u3) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};" ::"r"(u0), "r"(u1), "r"(u2), "r"(u3), "r"(taddr) : "memory");
}
__device__ __forceinline__ void qt_tmem_st8(uint32_t taddr, const uint32_t (&u)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]),
               "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void qt_tmem_st16(uint32_t taddr, const uint32_t (&u)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(u[0]), "r"(u[1]),
               "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]),
               "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void qt_tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]),
               "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
}
// Issued by the lanes that say `go` (one), without a branch: inside one the operands would leave the uniform registers, and an MMA take
// longer to issue than to run.
__device__ __forceinline__ void qt_mma_if(uint32_t go, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p, g;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 g, %5, 0;\n\t"
      "@g tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc),
      "r"(accum), "r"(go) : "memory");
}
__device__ __forceinline__ void qt_commit_if(uint32_t go, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred g;\n\tsetp.ne.b32 g, %1, 0;\n\t"
      "@g tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(bar), "r"(go) : "memory");
}
// a barrier of the four result warps that also tells whether all of them go on
__device__ __forceinline__ bool qt_results_and(bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(all) : "r"((uint32_t)ok) : "memory");
  return all != 0;
}
__device__ __forceinline__ uint32_t qt_lift(uint32_t w, uint32_t mask, uint32_t magic) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(mask), "r"(magic));
  return d;
}
// What a group's codes become, S q - E, for a word's eight codes in pairs (0, 4) (1, 5) (2, 6) (3, 7).  E is 8 S or next to it, see below.
// 1024 + q and 64 + q (codes four bits up) are fp16 numbers that one mask-or makes of two codes; every step is exact.
struct QtScale { uint32_t s, c, e, me, b; };   // (S, S), (C, C), (E, E), (-E, -E), (B, B)
__device__ __forceinline__ void qt_word(const QtArgs& a, uint32_t w, const QtScale& g, uint32_t* o) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    o[2 * j] = qt_fma(qt_add(qt_lift(w, a.mask0, a.magic0), 0xE400E400u), g.s, g.me);
    o[2 * j + 1] = qt_fma(qt_lift(w, a.mask1, a.magic1), g.s, g.c);
    w >>= 8;
  }
}
// S = 128 s and B = 128 b.  C is -72 S rounded to fp16, E = -64 S - C: with n the 8-bit significand of S, 9 n has at most 12 bits, so that C is
// off by eight of S's last places or by none, E is 8 (n, n - 1 or n + 1) of them and S q - E at most 2048: numbers that fp16 has.
// S is NaN where it is no fp16 number.  (Where 72 S is too large C and E are infinite, and the sums NaN as well.)  A b that is none may be off
// by s 2^-19: sums of products with 128 + q in fp32, which other kernels here take, are off by s 2^-17 times the same sum of |x|.
__device__ __forceinline__ QtScale qt_scale(uint32_t s_bits, uint32_t b_bits) {   // bf16 bits in the upper half
  const float s = __uint_as_float(s_bits) * 128.f, b = __uint_as_float(b_bits) * 128.f;
  const uint32_t p = qt_pack_f16(s, b);
  const bool ok = qt_f16lo(p) == s && fabsf(qt_f16hi(p) - b) <= fabsf(s) * 0x1p-19f;
  QtScale r;
  r.s = ok ? __byte_perm(p, 0, 0x1010) : 0x7fff7fffu;
  r.b = __byte_perm(p, 0, 0x3232);
  r.c = qt_mul(r.s, 0xD480D480u);
  r.me = qt_fma(r.s, 0x54005400u, r.c);
  r.e = r.me ^ 0x80008000u;
  return r;
}

struct QtAt { int si, n0; };
__device__ __forceinline__ QtAt qt_tile(const QtArgs& a, int tile) {
  if (a.dual) return {0, tile * 64};
  int si = 0;
  if (a.nseg > 1 && tile >= a.seg[1].tile0) si = 1;
  if (a.nseg > 2 && tile >= a.seg[2].tile0) si = 2;
  return {si, (tile - a.seg[si].tile0) * 128};
}
// Is row n of a segment one whose scales or biases the operand cannot hold?  A whole warp asks.
__device__ __noinline__ bool qt_row_marked(const QtSeg& g, int K, int n) {
  bool hit = false;
  for (int i = threadIdx.x & 31; i < K / kGroup; i += 32) {
    const size_t at = (size_t)n * (K / kGroup) + i;
    const QtScale q = qt_scale((uint32_t)__ldg(g.s + at) << 16, (uint32_t)__ldg(g.b + at) << 16);
    hit |= q.s == 0x7fff7fffu || (q.c & 0x7fffu) == 0x7c00u;
  }
  return __any_sync(0xffffffffu, hit);
}
// ... whose product with row m (scale f) a warp sums here, a word of codes a lane at a time, from the prepared x.  f < 0: the row has -f infinities,
// and the product is theirs.
template <int BITS>
__device__ __noinline__ float qt_row_dot(const QtSeg& g, const uint8_t* img, int np, int K, int n, int m, float f) {
  constexpr int PER = 32 / BITS;
  float y = 0.f;
  auto scale = [&](const uint16_t* p, int k) { return __uint_as_float((uint32_t)__ldg(p + (size_t)n * (K / kGroup) + k / kGroup) << 16); };
  if (f < 0.f) {
    for (int i = threadIdx.x & 31; i < (int)-f; i += 32) {
      const uint32_t entry = __ldcg(reinterpret_cast<const uint16_t*>(img + qt_list_at(i, np, m)));
      const int k = entry & 0x7fff;
      const uint32_t q = __ldg(g.wq + (size_t)n * (K / PER) + k / PER) >> (BITS * (k % PER)) & ((1u << BITS) - 1);
      y += fmaf(scale(g.s, k), (float)q, scale(g.b, k)) * (entry & 0x8000u ? -INFINITY : INFINITY);
    }
    return warp_sum(y);
  }
  for (int i = threadIdx.x & 31; i < K / PER; i += 32) {
    const float s = scale(g.s, i * PER), b = scale(g.b, i * PER);
    const uint32_t w = __ldg(g.wq + (size_t)n * (K / PER) + i);
    float d = 0.f, sx = 0.f;
    for (int j = 0; j < PER; ++j) {
      const int e = BITS == 4 ? j : 2 * j;   // 4-bit code of the word; its place in the prepared row
      const float xv = qt_f16lo(__ldcg(reinterpret_cast<const uint16_t*>(img + (size_t)(i >> 4) * np * 288 + (size_t)((i & 15) * np + m) * 16 +
                                                                         ((e & 3) * 2 + (e >> 2)) * 2)));
      d = fmaf((float)((w >> (BITS * j)) & ((1u << BITS) - 1)), xv, d);
      sx += xv;
    }
    y += s * d + b * sx;
  }
  return warp_sum(y) * (f * 128.f);
}

// PER: 128 codes a turn of the dequantisers, or twice as many
template <int BITS, int PER>
__global__ void __launch_bounds__(kQtThreads, 1) qmt_kernel(const __grid_constant__ QtArgs a) {
  constexpr int SPB = BITS == 4 ? 2 : 4;   // stages that share 16 bytes a row of scales
  constexpr int TURN_COLS = PER * kQtCols;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t w_full[kQtMaxStages], w_empty[kQtMaxStages], a_full[3], a_empty[3], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, last_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smW = base, smX = smW + a.nw * kQtStage;
  const long long total = (long long)a.ntiles * a.ks;
  long long lo = blockIdx.x * total / gridDim.x, hi = (blockIdx.x + 1) * total / gridDim.x;
  if (a.split) {
    const int t = blockIdx.x / a.split, p = blockIdx.x - t * a.split;
    lo = (long long)t * a.ks + p * a.ks / a.split;
    hi = (long long)t * a.ks + (p + 1) * a.ks / a.split;
  }
  const int stages = (int)(hi - lo);
  const int tile_lo = (int)(lo / a.ks), kk_lo = (int)(lo - (long long)tile_lo * a.ks);   // first tile, first stage in it
  const int x_bytes = PER * a.np * 288;   // of a turn
  const int turns = stages * (2 / PER), tile_turns = a.ks * (2 / PER);

  if (warp == 0 && lane < 9) {
    const int i = lane / 3, kind = lane - 3 * i;
    if (i < a.nseg) tma_prefetch_desc(kind == 0 ? &a.wmap[i] : kind == 1 ? &a.smap[i] : &a.bmap[i]);
  }
  if (warp == 1) {
    for (int i = lane; i < a.nw; i += 32) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], PER == 2 ? 4 : 8); }
    if (lane < 3) { mbar_init(&a_full[lane], 5); mbar_init(&a_empty[lane], 1); }
    if (lane < 2) { mbar_init(&acc_full[lane], 1); mbar_init(&acc_empty[lane], 4); }
    if (lane == 0) abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* const abortp = &abort_flag;
  pdl_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------------ packed rows, scales, biases
    if (lane == 0) {
      const uint64_t pol = l2_policy_evict_first();
      int tile = tile_lo, kk = kk_lo, ws = 0;
      uint32_t ph = 1;
      for (int i = 0; i < stages; ++i) {
        const QtAt at = qt_tile(a, tile);
        if (!gemm_wait(smem_u32(&w_empty[ws]), ph, abortp)) break;
        mbar_arrive_expect_tx(&w_full[ws], kQtStage);
        const uint32_t dst = smW + ws * kQtStage;
        const int g8 = kk / SPB * 8;
        if (a.dual) {
#pragma unroll 1
          for (int d = 0; d < 2; ++d) {
            tma_load_2d(dst + d * (kQtPacked / 2), &a.wmap[d], &w_full[ws], kk * 128, at.n0, pol);
            qt_tma_2d(dst + kQtPacked + d * 1024, &a.smap[d], &w_full[ws], g8, at.n0);
            qt_tma_2d(dst + kQtPacked + 2048 + d * 1024, &a.bmap[d], &w_full[ws], g8, at.n0);
          }
        } else {
          tma_load_2d(dst, &a.wmap[at.si], &w_full[ws], kk * 128, at.n0, pol);
          qt_tma_2d(dst + kQtPacked, &a.smap[at.si], &w_full[ws], g8, at.n0);
          qt_tma_2d(dst + kQtPacked + 2048, &a.bmap[at.si], &w_full[ws], g8, at.n0);
        }
        if (++ws == a.nw) { ws = 0; ph ^= 1; }
        if (++kk == a.ks) { kk = 0; ++tile; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------------ prepared x, into the slots of the operand
    if (lane == 0) {
      pdl_wait();
      int kk = kk_lo * (2 / PER), as = 0;
      uint32_t ph = 1;
      for (int t = 0; t < turns; ++t) {
        if (!gemm_wait(smem_u32(&a_empty[as]), ph, abortp)) break;
        mbar_arrive_expect_tx(&a_full[as], x_bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smX + as * x_bytes),
                     "l"(a.img + (size_t)kk * x_bytes), "r"(x_bytes), "r"(smem_u32(&a_full[as])) : "memory");
        if (++as == 3) { as = 0; ph ^= 1; }
        if (++kk == tile_turns) kk = 0;
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------------------------------------ MMAs: a converged warp, one lane issues
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t idesc = (1u << 4) | ((uint32_t)(a.np >> 3) << 17) | ((128u >> 4) << 24);   // fp32 sums of fp16 products
    const uint32_t step_k = (uint32_t)(2 * a.np);   // 16 k of x, in 16-byte units
    const bool lead = elect_one();
    int rest = tile_turns - kk_lo * (2 / PER), left = min(rest, a.run), sg = 0;   // turns to the end of the tile behind this accumulator's
    rest -= left;
    uint32_t aph = 0, started = 0;
    bool alive = true;
    for (int t0 = 0; t0 < turns; t0 += 3, aph ^= 1) {
#pragma unroll
      for (int as = 0; as < 3; ++as) {
        if (t0 + as >= turns) break;
        const uint32_t acc = tm + (uint32_t)((sg & 1) * a.np), ta = tm + (uint32_t)(2 * a.np + as * TURN_COLS);
        const uint64_t db = qt_desc_x(smX + as * x_bytes, a.np);
        if (!started) {
          alive &= gemm_wait(smem_u32(&acc_empty[sg & 1]), ((sg >> 1) & 1) ^ 1, abortp);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        alive &= gemm_wait(smem_u32(&a_full[as]), aph, abortp);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t go = lead && alive;
#pragma unroll
        for (int k = 0; k < 9 * PER; ++k) qt_mma_if(go, acc, ta + 8 * k, db + (uint64_t)(k * step_k), idesc, k > 0 ? 1u : started);
        qt_commit_if(go, smem_u32(&a_empty[as]));
        started = 1;
        if (--left == 0 || t0 + as + 1 == turns) {
          qt_commit_if(go, smem_u32(&acc_full[sg & 1]));
          started = 0;
          rest = rest ? rest : tile_turns;
          left = min(rest, a.run);
          rest -= left;
          ++sg;
        }
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------------------------------------ dequantisers: a thread per row, sets in turn
    // Turn t is a stage (PER 2) or half of one, and set t % 3 takes it to a place of its own.  A wait tells a barrier's phase only from the
    // one before it: that of the place sees only this set's turns, and that of the stage was last filled before MMAs that this set's turn
    // before has waited for (tests/test_cpu_qmt.py walks it).
    const int set = (warp - 8) >> 2, quad = warp & 3, row = quad * 32 + lane;
    const uint32_t swz = (uint32_t)(row & 7), row_w = smW + row * 128, row_s = smW + kQtPacked + row * 16;
    const uint32_t t0 = tmem + (uint32_t)(2 * a.np + set * TURN_COLS) + ((uint32_t)(quad * 32) << 16);
    int ws = set * PER / 2;
    uint32_t wph = 0, aph = 1;
    bool alive = true, dry = true;   // (the first time round as the results': what it leaves in tensor memory is written over)
    for (int t = set; t < turns && alive;) {
      if (!dry && !(alive = gemm_wait_warp(smem_u32(&w_full[ws]), wph, abortp))) break;
      const int run = (kk_lo + t * PER / 2) % SPB, c_lo = PER == 2 ? 0 : 2 * (t & 1);
      const uint32_t src = row_w + ws * kQtStage, sc = row_s + ws * kQtStage + (uint32_t)(run * (BITS == 4 ? 8 : 4));
      uint2 sv, bv;   // the stage's scales and biases, this quarter's in the lowest bits
      if (BITS == 4) { sv = lds64(sc); bv = lds64(sc + 2048); }
      else {           // two groups, each of them two quarters'
        const uint32_t s2 = lds32(sc), b2 = lds32(sc + 2048);
        sv = make_uint2(__byte_perm(s2, 0, 0x1010), __byte_perm(s2, 0, 0x3232));
        bv = make_uint2(__byte_perm(b2, 0, 0x1010), __byte_perm(b2, 0, 0x3232));
      }
      if (c_lo) { sv.x = sv.y; bv.x = bv.y; }
      uint32_t ta = t0;
#pragma unroll 1
      for (int c = c_lo; c < c_lo + (dry ? 1 : 2 * PER); ++c) {   // 64 codes, 32 columns; behind every second one the columns of the sums
        const uint4 w0 = lds128(src + (((uint32_t)(2 * c) ^ swz) << 4)), w1 = lds128(src + (((uint32_t)(2 * c + 1) ^ swz) << 4));
        const QtScale g = qt_scale(sv.x << 16, bv.x << 16);
        sv = make_uint2(__funnelshift_r(sv.x, sv.y, 16), sv.y >> 16);
        bv = make_uint2(__funnelshift_r(bv.x, bv.y, 16), bv.y >> 16);
        uint32_t o[32];
        qt_word(a, w0.x, g, o); qt_word(a, w0.y, g, o + 4); qt_word(a, w0.z, g, o + 8); qt_word(a, w0.w, g, o + 12);
        qt_word(a, w1.x, g, o + 16); qt_word(a, w1.y, g, o + 20); qt_word(a, w1.z, g, o + 24); qt_word(a, w1.w, g, o + 28);
        if (c == c_lo && !dry) {
          alive &= gemm_wait_warp(smem_u32(&a_empty[set]), aph, abortp);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        tmem_st32(ta, o);
        const uint32_t tail = ta + ((c & 1) ? 36 : 64);
        if (BITS == 4) qt_tmem_st4(tail, g.e, __byte_perm(g.e, g.b, 0x5410), g.b, 0);
        else if (c & 1) qt_tmem_st4(tail, g.b & 0xffffu, 0, 0, 0);
        else qt_tmem_st4(tail, g.e, g.e, g.e, g.b);
        ta += (c & 1) ? kQtCols - 32 : 32;
      }
      tmem_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (dry) { dry = false; continue; }
      if (lane == 0) {
        mbar_arrive(&a_full[set]);
        mbar_arrive(&w_empty[ws]);
      }
      aph ^= 1;
      ws += PER == 2 ? 3 : 1 + (t & 1);
      if (ws >= a.nw) { ws -= a.nw; wph ^= 1; }
      t += 3;
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------------------------------------ results: thread = row of the tile
    const int quad = warp & 3, row = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const uint32_t xch = smX + 3 * x_bytes;   // dual: [16][64] fp32, the up rows' values on their way to the gate rows'
    const uint32_t smR = xch + 4096;          // the rows' scales
    pdl_wait();
    sts32(smR + (uint32_t)(tid - 128) * 4, tid - 128 < a.M ? __float_as_uint(__ldcg(a.rscale + tid - 128)) : 0u);
    int tile = tile_lo, kk = kk_lo, left = stages, sg = 0;
    // The first time round nothing is there yet and nothing is stored but this CTA's own parts: it is for the instructions, which otherwise
    // come from L2, line by line, when the whole launch waits for these warps.
    bool dry = true;
    while (left > 0) {
      const int take = min(left, a.ks - kk), rows = dry ? 0 : a.M;
      const bool whole = take == a.ks && !dry;
      // accumulators before the last: all are added up, in tensor memory behind the operands or in shared memory, and the sum takes the last one's
      // place.  (Not in registers: with 32 more of them live some are spilled, and every call took 1 to 2 us longer.)
      const int before = dry ? 0 : (take * (2 / PER) - 1) / a.run;
      bool ok = true;
      for (int j = 0;; ++j, ++sg) {
        const uint32_t acc = tmem + (uint32_t)((sg & 1) * a.np) + lanes;
        ok = dry || gemm_wait_warp(smem_u32(&acc_full[sg & 1]), (sg >> 1) & 1, abortp);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (before == 0) break;
        const uint32_t kept = tmem + (uint32_t)(2 * a.np + 3 * TURN_COLS) + lanes, kept_s = smR + kQtMaxRows * 4 + (uint32_t)row * 4;
        if constexpr (PER == 2) {
#pragma unroll 1
          for (int c = 0; c < a.np; c += 8) {
            uint32_t v[8], t[8];   // (t, j = 0: not yet written, and not added)
            qt_tmem_ld8(acc + c, v);
            if (a.totals_smem) {
#pragma unroll
              for (int q = 0; q < 8; ++q) t[q] = lds32(kept_s + (uint32_t)(c + q) * 512);
            } else {
              qt_tmem_ld8(kept + c, t);
            }
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (j > 0) v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(t[q]));
            if (a.totals_smem && j < before) {
#pragma unroll
              for (int q = 0; q < 8; ++q) sts32(kept_s + (uint32_t)(c + q) * 512, v[q]);
            } else {
              qt_tmem_st8((j == before ? acc : kept) + c, v);
            }
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < a.np; c += 16) {
            uint32_t v[16], t[16];
            tmem_ld16(acc + c, v);
            tmem_ld16(kept + c, t);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 16; ++q)
              if (j > 0) v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(t[q]));
            qt_tmem_st16((j == before ? acc : kept) + c, v);
          }
        }
        tmem_st_wait();
        if (j == before) break;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[sg & 1]);
      }
      if (!qt_results_and(ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int b = sg & 1;
      const QtAt at = qt_tile(a, tile);
      const QtSeg& seg = a.seg[a.dual ? quad >> 1 : at.si];
      const int n = at.n0 + (a.dual ? row & 63 : row);
      const bool live = n < seg.N;
      const uint32_t acc = tmem + (uint32_t)(b * a.np) + lanes;
      bool finish = true;
      int c0 = 0, nparts = 1, second = 0;   // the CTAs that share the tile
      if (!whole) {
        // this CTA's part -> workspace
        const long long t0 = (long long)tile * a.ks;
        float4* const mine = reinterpret_cast<float4*>(a.part) + (size_t)(2 * blockIdx.x + (lo < t0 ? 1 : 0)) * a.np * 32 + row;
#pragma unroll 1
        for (int c = 0; c < a.np; c += 16) {
          uint32_t v[16];
          tmem_ld16(acc + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q)
            __stcg(mine + (size_t)(c / 4 + q) * 128, make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                                                                 __uint_as_float(v[4 * q + 3])));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0 && !dry) mbar_arrive(&acc_empty[b]);
        if (a.split) {
          c0 = tile * a.split;
          nparts = a.split;
        } else {
          c0 = (int)(((t0 + 1) * gridDim.x - 1) / total);
          nparts = (int)(((t0 + a.ks) * gridDim.x - 1) / total) - c0 + 1;
          second = c0 * total / gridDim.x < t0;
        }
        qt_results_and(true);
        if (tid == 128 && !dry) {
          __threadfence();   // (behind the barrier: for all four warps' parts)
          last_flag = atomicAdd(a.cnt + tile, 1u) == (unsigned)nparts - 1;
          __threadfence();
        }
        qt_results_and(true);
        finish = dry || last_flag != 0;
        if (dry) nparts = 1;
      }
      if (finish) {
#pragma unroll 1
        for (int c = 0; c < (dry ? 16 : a.np); c += 16) {
          float y[16];
          if (whole) {
            tmem_ld16(acc + c, reinterpret_cast<uint32_t(&)[16]>(y));
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int q = 0; q < 16; ++q) y[q] = 0.f;
            // (only the first CTA's part can be its second: the others' shares begin inside the tile)
            const float4* part = reinterpret_cast<const float4*>(a.part) + (size_t)(2 * c0 + second) * a.np * 32 + (size_t)(c / 4) * 128 + row;
            const float4* const rest = part + (size_t)(2 - second) * a.np * 32;
#pragma unroll 1
            for (int p = 0; p < nparts; p += 2) {   // two parts' loads in flight
              float4 v[2][4];
#pragma unroll
              for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int q = 0; q < 4; ++q) v[u][q] = p + u < nparts ? __ldcg(part + q * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
                part = p + u == 0 ? rest : part + (size_t)a.np * 64;
              }
#pragma unroll
              for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int q = 0; q < 4; ++q) { y[4 * q] += v[u][q].x; y[4 * q + 1] += v[u][q].y; y[4 * q + 2] += v[u][q].z; y[4 * q + 3] += v[u][q].w; }
            }
          }
          bool odd = false;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 rs = lds128(smR + (uint32_t)(c + 4 * q) * 4);
            const uint32_t r4[4] = {rs.x, rs.y, rs.z, rs.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float f = __uint_as_float(r4[e]);
              if (c + 4 * q + e < rows) odd |= y[4 * q + e] != y[4 * q + e] && f == f;
              y[4 * q + e] *= f;
            }
          }
          for (unsigned left_odd = __ballot_sync(0xffffffffu, odd && live); left_odd; left_odd &= left_odd - 1) {
            const int who = __ffs(left_odd) - 1, row_n = __shfl_sync(0xffffffffu, n, who);
            const bool marked = qt_row_marked(seg, a.K, row_n);   // (if not, and no list: the NaN is the caller's)
#pragma unroll
            for (int q = 0; q < 16; ++q)
              if (c + q < rows) {
                const float f = __uint_as_float(lds32(smR + (uint32_t)(c + q) * 4));
                if (!marked && !(f < 0.f)) continue;
                const float d = qt_row_dot<BITS>(seg, a.img, a.np, a.K, row_n, c + q, f);
                if (lane == who) y[q] = d;
              }
          }
          if (a.dual) {
            if (quad >= 2) {
#pragma unroll
              for (int q = 0; q < 16; ++q) sts32(xch + (uint32_t)(q * 64 + (row & 63)) * 4, __float_as_uint(bfround(y[q])));
            }
            qt_results_and(true);
            if (quad < 2 && live) {
              uint16_t* const to = a.out + (size_t)c * a.out_ld + n;
#pragma unroll
              for (int q = 0; q < 16; ++q) {
                const float up = __uint_as_float(lds32(xch + (uint32_t)(q * 64 + row) * 4)), gt = bfround(y[q]);
                const float sg = bfround(1.f / (1.f + expf(-gt)));   // nn.silu = x * sigmoid(x), each op rounded
                if (c + q < rows) to[(size_t)q * a.out_ld] = f2bf(bfround(gt * sg) * up);
              }
            }
            qt_results_and(true);
          } else if (live) {
            const size_t first = (size_t)c * a.out_ld + seg.out_off + n;
            uint16_t res[16];
            if (a.epi == EPI_RESADD) {   // all of them before the first store: they may lie where it goes
#pragma unroll
              for (int q = 0; q < 16; ++q) res[q] = c + q < rows ? a.residual[first + (size_t)q * a.out_ld] : 0;
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              float r = bfround(y[q]);
              if (a.epi == EPI_RESADD) r = bf16lo((uint32_t)res[q]) + r;
              if (c + q < rows) a.out[first + (size_t)q * a.out_ld] = f2bf(r);
            }
          }
        }
        if (whole) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[b]);
        }
      }
      if (dry) { dry = false; continue; }
      left -= take;
      kk = 0;
      ++tile;
      ++sg;
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abortp) gemm_drain();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
}

// ---- host side ------------------------------------------------------------------------------------------------------------------------
static bool qt_map(CUtensorMap* m, const void* p, bool packed, long long inner, long long rows, long long pitch, int box_inner, int box_rows) {
  const GemmEncodeFn fn = gemm_encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows}, one[2] = {1, 1};
  return fn(m, packed ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(p), dims, strides, box, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, packed ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
            packed ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool qmt_shape_ok(int M, int K, int group_size, int bits) {
  return M >= 1 && M <= kQtMaxRows && K > 0 && K % 512 == 0 && K <= kQtMaxK && group_size == kGroup && (bits == 4 || bits == 8);
}
// [counters | row scales | prepared x | parts]
static size_t qt_cnt_bytes(long long ntiles) { return ((size_t)ntiles * 4 + 255) & ~(size_t)255; }
static size_t qt_img_bytes(int np, int K, int bits) { return (size_t)(K * bits / 4 / 128) * np * 288; }
size_t qmt_ws_bytes(int M, long long ntiles, int K, int bits) {
  const int np = (M + 15) & ~15;
  return qt_cnt_bytes(ntiles) + kQtMaxRows * 4 + qt_img_bytes(np, K, bits) + (size_t)2 * num_sms() * np * 512;
}

template <int BITS, int PER>
static cudaError_t qmt_launch(const QtArgs& a, int grid, size_t smem, float* rscale, const uint16_t* x, int x_ld, const uint16_t* norm_w,
                              float eps, cudaStream_t st) {
  static std::atomic<unsigned long long> served{0};
  cudaError_t e = once_per_device(served, [] { return cudaFuncSetAttribute(qmt_kernel<BITS, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, kQtSmem); });
  if (e != cudaSuccess) return e;
  count_launch(2);
  auto prep = a.K <= 8192 ? qmt_prep_kernel<BITS, 1> : a.K <= 16384 ? qmt_prep_kernel<BITS, 2> : qmt_prep_kernel<BITS, 4>;
  e = launch_pdl(prep, dim3((unsigned)a.M), dim3(1024), 0, st, const_cast<uint8_t*>(a.img), rscale, a.cnt, a.ntiles, x, x_ld, norm_w, eps, a.np, a.K);
  if (e != cudaSuccess) return e;
  return launch_pdl(qmt_kernel<BITS, PER>, dim3((unsigned)grid), dim3(kQtThreads), smem, st, a);
}

cudaError_t launch_qmt(void* out, int out_ld, const void* x, int x_ld, int M, int K, const pie_qmv_seg* segs, int nseg, int bits,
                       const void* norm_w, float eps, int epi, const void* residual, void* ws, cudaStream_t st) {
  QtArgs a = {};
  a.nseg = nseg; a.dual = epi == EPI_SILUMUL; a.M = M; a.K = K; a.np = (M + 15) & ~15;
  const long long row_bytes = (long long)K * bits / 8;
  const int box = a.dual ? 64 : 128;
  int tile = 0, off = 0;
  for (int i = 0; i < nseg; ++i) {
    a.seg[i] = {segs[i].wq, (const uint16_t*)segs[i].scales, (const uint16_t*)segs[i].biases, segs[i].N, tile, off};
    if (!qt_map(&a.wmap[i], segs[i].wq, true, row_bytes, segs[i].N, row_bytes, 128, box) ||
        !qt_map(&a.smap[i], segs[i].scales, false, K / kGroup, segs[i].N, K / kGroup * 2, 8, box) ||
        !qt_map(&a.bmap[i], segs[i].biases, false, K / kGroup, segs[i].N, K / kGroup * 2, 8, box))
      return cudaErrorNotSupported;
    if (!a.dual || i == 0) tile += (segs[i].N + box - 1) / box;
    off += segs[i].N;
  }
  a.ntiles = tile;
  a.ks = (int)(row_bytes / 128);
  a.epi = epi; a.out_ld = out_ld; a.out = (uint16_t*)out; a.residual = (const uint16_t*)residual;
  a.mask0 = 0x000f000fu; a.mask1 = 0x00f000f0u; a.magic0 = 0x64006400u; a.magic1 = 0x54005400u;
  const int per = 2 * a.np + 6 * kQtCols <= 512 ? 2 : 1;   // tensor memory has the room for turns of 256 codes
  // The tensor core cuts the sums it returns, towards zero.  What that makes before the rounding to bf16, measured on products that are next to zero (rms,
  // of a usual product's size): one accumulator for all of K 1.8e-6 at K 4096 and 8.0e-6 at 14336, a new one every 2048 codes 8.8e-7 and 1.0e-6, every 1024
  // 3.8e-7 and 5.0e-7; the mma.sync GEMV, which has chains of four, 1.4e-6 and 1.1e-6.  So 1024 codes, and the sums added in fp32 (us, one accumulator / this:
  // 2 x 14336 x 4096 with SwiGLU 16 rows 26.4 / 27.0, 32 31.2 / 32.4; 128256 x 4096, 16 rows 72.6 / 74.4).  65 rows and more, which the tile kernel would
  // serve with one accumulator and rounded weights, keep one: at 112 tensor memory has no room for totals.
  a.run = a.np <= 64 ? 8 / per : 1 << 30;
  a.totals_smem = a.np <= 64 && 3 * a.np + 3 * per * kQtCols > 512;
  const int fixed = 1024 + 3 * per * a.np * 288 + 4096 + kQtMaxRows * 4 + (a.totals_smem ? a.np * 512 : 0), room = (kQtSmem - fixed) / kQtStage;
  a.nw = room < kQtMaxStages ? room : kQtMaxStages;
  const size_t smem = (size_t)fixed + (size_t)a.nw * kQtStage;
  uint8_t* p = (uint8_t*)ws;
  a.cnt = (unsigned int*)p; p += qt_cnt_bytes(a.ntiles);
  float* const rscale = (float*)p; p += kQtMaxRows * 4;
  a.rscale = rscale;
  a.img = p; p += qt_img_bytes(a.np, K, bits);
  a.part = (float*)p;
  const long long total = (long long)a.ntiles * a.ks;
  // Even shares, or whole parts of one tile each where those are no longer than by a stage: a CTA with parts of two tiles has its
  // results to hand over twice, 2 to 3 us.
  const int sms = num_sms(), even = (int)((total + sms - 1) / sms);
  int grid = (int)(total < sms ? total : sms);
  if (a.ntiles <= sms) {
    const int split = min(sms / a.ntiles, a.ks);
    if ((a.ks + split - 1) / split <= even + 1) { a.split = split; grid = a.ntiles * split; }
  }
  auto go = [&](auto f) { return f(a, grid, smem, rscale, (const uint16_t*)x, x_ld, (const uint16_t*)norm_w, eps, st); };
  if (per == 2) return bits == 4 ? go(qmt_launch<4, 2>) : go(qmt_launch<8, 2>);
  return bits == 4 ? go(qmt_launch<4, 1>) : go(qmt_launch<8, 1>);
}

}  // namespace pie
