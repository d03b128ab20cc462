// Prefill attention (L > 1, causal) on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a.
//
// Replaces mx.fast.scaled_dot_product_attention with the additive causal mask of create_attention_mask
// (PIE/models/base.py:18-53, 92-113; Metal steel_attention, MLX/mlx/backend/metal/scaled_dot_product_attention.cpp:
// 16-131): out[b, l, h] = softmax(scale * q[b,h,l] . K[b, h / n_rep, :offset+l+1]) . V.  The mask value -1e9 makes
// masked probabilities exactly 0 in fp32, so masked keys are skipped (tiles beyond the diagonal are never loaded).
//
// A CTA owns 256 query rows of one head as two tiles of 128, and walks the keys in tiles of 128.  Per (query tile, key tile)
// the tensor pipe needs 2 x 128 x 128 x D multiply-adds and the softmax 128 x 128 exponentials; at D = 128 the two take the
// same ~1000 cycles of an SM, so the kernel is built to keep both going at once:
//   * warps 0-3 / 4-7: the softmax of query tile 0 / 1, a thread per row.  S comes out of tensor memory (128 columns), is
//     masked on the diagonal, the running maximum moves only when exceeded by 8 (log2 units; the same sums, and O is rescaled
//     rarely), p = exp2(scale s - m), three quarters of them by the approximation unit (16 a cycle of an SM: at D = 64 that alone
//     would take twice the MMAs' time) and the rest by a polynomial on the multiply-add pipe, is rounded to bf16 and put back over
//     S as the A operand of the second product.  Row sums are of the unrounded p, in fp32.
//   * warp 8: TMA.  Q once; K and V tiles of the contiguous or paged cache into two-deep rings (128-byte swizzle).
//   * warp 9: MMAs.  S_g = Q_g K^T (both operands in shared memory), O_g += P_g V (P in tensor memory, V as it lies:
//     its rows are keys, so it is an MN-major operand).  Order: PV of tile 0, QK^T of tile 0's next keys, then the same for
//     tile 1: one tile's softmax runs under the other's MMAs.
// Tensor memory: S/P 2 x 128 columns, O 2 x D.
// A CTA per SM walks its share of the 256-row items, longest first (causal: tile i sees i + 1 key tiles).  An item's first scores are issued behind the
// last product of the one before it, query tile by query tile, while that one's other tile and its results are still worked on; nothing is set up
// twice.  (One CTA an item, 5.2 of them an SM at 2 x 3000 tokens: 156.8 us; this 146.4; 8192 tokens 464 -> 447; D 64, 2 x 3000 127.5 -> 123.9, but
// 1500 tokens 23.3 -> 23.9 and 6001 219.9 -> 222.3.  With three eighths of the exponentials off the approximation unit 150, with half 160.  An eighth at D 128 is
// 144.7, but the unit is off by 2.4e-7 and the polynomial by 2.0e-7.)
// Every wait is bounded (pie_gemm.cuh).
// Measured, 32 query / 8 kv heads, us (TFLOP/s): the mma.sync kernel of pie_fa.cu -> this one with a lane of its own issuing the MMAs
// and all exponentials on the approximation unit -> as it is.  D 128: 8192 tokens 2190 (251) -> 547 (1005) -> 460 (1196); 2 x 3000
// tokens 640 (231) -> 190 (774) -> 164 (901).  D 64: 1531 behind 517 92 -> 51 -> 42; 8192 tokens 485 -> 386 (712).
// (The last figures are those of a CTA an item.)  What is left is one tile's chain, which the other tile covers only in part: of about 3000
// cycles per pair of tiles, 1700 are a softmax and 1300 the two products and their hand-overs.
#include "pie_gemm.cuh"
#include "pie_internal.h"

namespace pie {

struct FapArgs {
  uint16_t* out;
  int Hq, Hkv, L, offset, B;
  int qt;                      // items of 256 query rows a head
  float scale_log2e;
  const int32_t* page_table;   // paged cache, else nullptr
  int pt_stride, page_size;
};

template <int D>
struct FapTile {
  static constexpr int CH = D / 64;                     // 64-feature chunks of a row: 128 bytes each
  static constexpr int TILE = 128 * D * 2;              // bytes of 128 rows
  static constexpr int SMEM = 1024 + 6 * TILE;          // Q0, Q1, K x 2, V x 2
  static constexpr int THREADS = 384;
};

__device__ __forceinline__ void fap_tma_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// shared-memory descriptor of an MN-major operand in the 128-byte swizzle: rows of 64 features, 8 rows (keys) per atom,
// atoms 1024 bytes apart along the keys, 64-feature chunks 128 rows apart
__device__ __forceinline__ uint64_t fap_desc_mn(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)(128 * 128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// 32 columns of this warp's 32 lanes, not waited for
__device__ __forceinline__ void fap_tmem_ld(uint32_t taddr, float* v) {
  uint32_t* u = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]),
        "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]),
        "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ float fap_exp2(float x) {   // results below 2^-126 are 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 operations an instruction
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// 2^x of two values by the multiply-add pipe: x = n + f with f in [-1/2, 1/2] (adding 3 * 2^22 rounds to an integer and leaves it
// in the low bits), 2^f by its least-squares polynomial of degree 5 in the Chebyshev weight (relative error 2.0e-7 in fp32, against
// the approximation unit's 2.4e-7), times 2^n.  Arguments of -127 and below (a masked key's -inf) give 0, NaN gives NaN.
__device__ __forceinline__ void fap_exp2_poly(f32x2 x2, float& ya, float& yb) {
  float xa, xb;
  f2_unpack(x2, xa, xb);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(xa) : "f"(-127.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(xb) : "f"(-127.f));
  const f32x2 x = f2_pack(xa, xb);
  const f32x2 r = f2_add(x, f2_pack(12582912.f, 12582912.f));
  const f32x2 f = f2_fma(f2_add(r, f2_pack(-12582912.f, -12582912.f)), f2_pack(-1.f, -1.f), x);
  f32x2 p = f2_pack(0.00132669706f, 0.00132669706f);
  p = f2_fma(p, f, f2_pack(0.00967545994f, 0.00967545994f));
  p = f2_fma(p, f, f2_pack(0.0555074252f, 0.0555074252f));
  p = f2_fma(p, f, f2_pack(0.240221217f, 0.240221217f));
  p = f2_fma(p, f, f2_pack(0.693146944f, 0.693146944f));
  p = f2_fma(p, f, f2_pack(1.00000012f, 1.00000012f));
  float ra, rb;
  f2_unpack(r, ra, rb);
  f2_unpack(f2_mul(p, f2_pack(__int_as_float((__float_as_int(ra) << 23) + 0x3f800000), __int_as_float((__float_as_int(rb) << 23) + 0x3f800000))), ya, yb);
}
__device__ __forceinline__ void fap_commit(uint64_t* bar) { gemm_commit<1>(smem_u32(bar)); }

// An item of work: 256 query rows of one head.  Items are ordered by length, longest first, and dealt out in turns that change direction, so that
// a CTA's share is the same within a short item.
struct FapItem { int b, h, q0, n0, n1; };
__device__ __forceinline__ bool fap_item(const FapArgs& a, int round, FapItem& it) {
  const int G = (int)gridDim.x, i = round * G + ((round & 1) ? G - 1 - (int)blockIdx.x : (int)blockIdx.x), heads = a.B * a.Hq;
  if (i >= heads * a.qt) return false;
  const int y = i / heads, bh = i - y * heads;
  it.b = bh / a.Hq;
  it.h = bh - it.b * a.Hq;
  it.q0 = (a.qt - 1 - y) * 256;
  // key tiles of a query tile: up to the diagonal of its last live row; none if the tile lies beyond the queries
  it.n0 = (a.offset + min(it.q0 + 128, a.L) - 1) / 128 + 1;
  it.n1 = it.q0 + 128 < a.L ? (a.offset + min(it.q0 + 256, a.L) - 1) / 128 + 1 : 0;
  return true;
}

template <int D>
__global__ void __launch_bounds__(FapTile<D>::THREADS, 1)
fa_prefill_umma_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ FapArgs a) {
  using T = FapTile<D>;
  constexpr uint32_t ID_S = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
  constexpr uint32_t ID_O = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((128u >> 4) << 24);
  constexpr int COL_S = 0, COL_O = 256;   // + g * 128, + g * D
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_full[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smQ = base, smK = base + 2 * T::TILE, smV = base + 4 * T::TILE;
  const int keys = a.offset + a.L;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 8 && lane < 3) tma_prefetch_desc(lane == 0 ? &map_q : lane == 1 ? &map_k : &map_v);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* const abortp = &abort_flag;
  pdl_launch_dependents();
  pdl_wait();   // (the set-up above ran under the end of the launch before this one)

  // All barriers are counted over the CTA's items: a role keeps the number of key tiles (of its query tile, of K and V) before its item.
  // Registers: 384 threads x 168 at launch = 64512; the eight softmax warps hold a row of scores each and take 216, the other
  // four give theirs up to 64: 8 x 32 x 216 + 4 x 32 x 64 = 63488.
  if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------------------------------------ softmax of tile g
    const int g = warp >> 2, quad = warp & 3;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const uint32_t tS = tmem + COL_S + g * 128 + lanes, tO = tmem + COL_O + g * D + lanes;
    const int tail = keys & 127;   // rows of the last key tile that exist
    int c = 0, cv = 0;             // tiles of this query tile, tiles of V, before this item
    bool alive = true;
    FapItem it;
    for (int round = 0; alive && fap_item(a, round, it); ++round) {
      const int ng = g ? it.n1 : it.n0, row = it.q0 + g * 128 + quad * 32 + lane, lim = a.offset + row;   // last key this row sees
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < ng; ++j) {
        if (!(alive = gemm_wait_warp(smem_u32(&s_full[g]), (c + j) & 1, abortp))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float s[128];
#pragma unroll
        for (int q = 0; q < 4; ++q) fap_tmem_ld(tS + 32 * q, s + 32 * q);
        tmem_ld_wait();
        if (j * 128 + 127 > a.offset + it.q0 + g * 128 + quad * 32) {   // a key of this tile lies beyond some row of the warp
          const int last = lim - j * 128;
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i > last) s[i] = -INFINITY;
        }
        float x0 = s[0], x1 = s[1], x2 = s[2], x3 = s[3];
#pragma unroll
        for (int i = 4; i < 128; i += 4) {
          x0 = fmaxf(x0, s[i]); x1 = fmaxf(x1, s[i + 1]); x2 = fmaxf(x2, s[i + 2]); x3 = fmaxf(x3, s[i + 3]);
        }
        const float mx = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)) * a.scale_log2e;   // (the scale is positive)
        const bool move = mx > m + 8.f;
        if (j == 0) {
          m = mx;
        } else if (__any_sync(0xffffffffu, move)) {
          const float f = move ? fap_exp2(m - mx) : 1.f;   // m == -inf: 0, and everything it multiplies is 0
          if (move) m = mx;
          l *= f;
          // O holds the tiles before this one once their product has finished
          if (!(alive = gemm_wait_warp(smem_u32(&o_full[g]), (c + j - 1) & 1, abortp))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 32) {
            float o[32];
            fap_tmem_ld(tO + c0, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= f;
            tmem_st32(tO + c0, reinterpret_cast<uint32_t*>(o));
          }
          tmem_st_wait();
        }
        const float ms = m == -INFINITY ? 0.f : m;
        const f32x2 sc2 = f2_pack(a.scale_log2e, a.scale_log2e), ms2 = f2_pack(-ms, -ms);
        f32x2 l01 = f2_pack(0.f, 0.f), l23 = l01;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t p[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const f32x2 x = f2_fma(f2_pack(s[64 * hf + 2 * i], s[64 * hf + 2 * i + 1]), sc2, ms2);
            float e0, e1;
            if (i % 4 == 3) {        // every fourth pair off the approximation unit, which would otherwise bound the tile
              fap_exp2_poly(x, e0, e1);
            } else {
              float x0, x1;
              f2_unpack(x, x0, x1);
              e0 = fap_exp2(x0);
              e1 = fap_exp2(x1);
            }
            p[i] = pack_bf16(e0, e1);
            if (i & 1) l23 = f2_add(l23, f2_pack(e0, e1));
            else l01 = f2_add(l01, f2_pack(e0, e1));
          }
          tmem_st32(tS + 32 * hf, p);
        }
        {
          float l0, l1;
          f2_unpack(f2_add(l01, l23), l0, l1);
          l += l0 + l1;
        }
        tmem_st_wait();
        if (a.page_table && tail && j == (keys - 1) / 128) {
          // the slots behind the last key of a page may hold anything, and 0 * NaN is not 0: clear them
          const int v = cv + j;
          if (!(alive = gemm_wait_warp(smem_u32(&v_full[v & 1]), (v >> 1) & 1, abortp))) break;
          const int r = quad * 32 + lane;
          if (r >= tail)
#pragma unroll
            for (int q = 0; q < 8 * T::CH; ++q)
              asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(smV + (v & 1) * T::TILE + (q >> 3) * 16384 + r * 128 + (q & 7) * 16),
                           "r"(0) : "memory");
          fence_proxy_async();
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g]);
      }
      c += ng;
      cv += max(it.n0, it.n1);
      // O is read before this warp says that the next item's first P is there, which its first product, overwriting O, waits for
      if (alive && ng > 0 && (alive = gemm_wait_warp(smem_u32(&o_full[g]), (c - 1) & 1, abortp))) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = 1.f / l;
        uint16_t* o_row = a.out + (((size_t)it.b * a.L + row) * a.Hq + it.h) * D;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          float o[32];
          fap_tmem_ld(tO + c0, o);
          tmem_ld_wait();
          if (row < a.L)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              *reinterpret_cast<uint4*>(o_row + c0 + 8 * q) =
                  make_uint4(pack_bf16(o[8 * q] * inv, o[8 * q + 1] * inv), pack_bf16(o[8 * q + 2] * inv, o[8 * q + 3] * inv),
                             pack_bf16(o[8 * q + 4] * inv, o[8 * q + 5] * inv), pack_bf16(o[8 * q + 6] * inv, o[8 * q + 7] * inv));
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // ------------------------------------------------------------------------------------------------ TMA
    if (warp == 8 && lane == 0) {
      bool alive = true;
      int cq[2] = {0, 0}, ck = 0;   // items with a query tile g, key tiles, before this item
      FapItem it;
      for (int round = 0; alive && fap_item(a, round, it); ++round) {
        const int n = max(it.n0, it.n1), kvh = it.h / (a.Hq / a.Hkv);
        auto fetch_q = [&](int g) {
          if ((g ? it.n1 : it.n0) == 0) return true;
          if (!gemm_wait(smem_u32(&q_empty[g]), (cq[g] & 1) ^ 1, abortp)) return false;
          ++cq[g];
          mbar_arrive_expect_tx(&q_full[g], T::TILE);
          for (int c = 0; c < T::CH; ++c)
            gemm_tma_3d<1>(smQ + g * T::TILE + c * 16384, &map_q, smem_u32(&q_full[g]), c * 64, it.q0 + g * 128, it.b * a.Hq + it.h);
          return true;
        };
        auto fetch = [&](int j, const CUtensorMap* map, uint32_t dst, uint64_t* full) {
          mbar_arrive_expect_tx(full, T::TILE);
          for (int r = 0; r < 2; ++r) {   // 64 keys at a time: a page, or half a tile
            int t = j * 128 + r * 64, c1 = t, c2 = kvh, c3 = it.b;
            if (a.page_table) {
              t = min(t, (keys - 1) / 64 * 64);   // behind the last key: any page that exists
              c1 = t % a.page_size;
              c3 = __ldg(a.page_table + (size_t)it.b * a.pt_stride + t / a.page_size);
            }
            for (int c = 0; c < T::CH; ++c) fap_tma_4d(dst + c * 16384 + r * 8192, map, smem_u32(full), c * 64, c1, c2, c3);
          }
        };
        // In the order in which the MMAs ask for them: tile 0's first product of this item may come before tile 1's last of the item before,
        // which Q1 has to wait for.
        if (!(alive = fetch_q(0))) break;
        for (int j = 0; j < n && alive; ++j, ++ck) {
          const int i = ck & 1, ph = (ck >> 1) & 1;
          if (!(alive = gemm_wait(smem_u32(&k_empty[i]), ph ^ 1, abortp))) break;
          fetch(j, &map_k, smK + i * T::TILE, &k_full[i]);
          if (j == 0 && !(alive = fetch_q(1))) break;
          if (!(alive = gemm_wait(smem_u32(&v_empty[i]), ph ^ 1, abortp))) break;
          fetch(j, &map_v, smV + i * T::TILE, &v_full[i]);
        }
      }
    }
    // ------------------------------------------------------------------------------------------------ MMAs
    if (warp == 9) {
      // The whole warp walks the loop, so that addresses and descriptors stay warp-uniform; one elected lane issues, and nothing
      // brings the lanes together but the election (a lane's own branch took 80 cycles an MMA; 4096 tokens, D 128: 155 -> 127 us).
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t dq0 = umma_desc_sw128(smQ), dk0 = umma_desc_sw128(smK), dv0 = fap_desc_mn(smV);
      auto qk = [&](int g, int slot, bool last) {   // last: of the item; Q's place is free behind it
        const uint64_t dq = dq0 + (uint64_t)(g * (T::TILE >> 4)), dk = dk0 + (uint64_t)(slot * (T::TILE >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16(tm + COL_S + g * 128, dq + (k >> 2) * 1024 + 2 * (k & 3), dk + (k >> 2) * 1024 + 2 * (k & 3), ID_S, k > 0 ? 1u : 0u);
        fap_commit(&s_full[g]);
        if (last) fap_commit(&q_empty[g]);
      };
      auto pv = [&](int g, int slot, int j) {
        const uint64_t dv = dv0 + (uint64_t)(slot * (T::TILE >> 4));
#pragma unroll
        for (int k = 0; k < 8; ++k)   // 16 keys: 8 columns of P, two 8-key atoms of V
          umma_f16_ts(tm + COL_O + g * D, tm + COL_S + g * 128 + 8 * k, dv + k * (2048 >> 4), ID_O, (j > 0 || k > 0) ? 1u : 0u);
        fap_commit(&o_full[g]);
      };
      bool alive = true;   // a lane's own: once a wait expires it only keeps the lane from issuing
      int c[2] = {0, 0}, cq[2] = {0, 0}, ck = 0;   // tiles of query tile g, items with one, tiles of K and V, before this item
      bool ahead[2] = {false, false};              // this item's first product of tile g is issued already
      FapItem it, next;
      bool more = fap_item(a, 0, it);
      for (int round = 0; more; ++round) {
        const int n = max(it.n0, it.n1);
        more = fap_item(a, round + 1, next);
        alive &= gemm_wait(smem_u32(&k_full[ck & 1]), (ck >> 1) & 1, abortp);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int ng = g ? it.n1 : it.n0;
          if (ng > 0 && !ahead[g]) {
            alive &= gemm_wait(smem_u32(&q_full[g]), cq[g] & 1, abortp);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one() && alive) qk(g, ck & 1, ng == 1);
          }
          if (ng > 0) ++cq[g];
          ahead[g] = false;
        }
        if (elect_one() && alive) fap_commit(&k_empty[ck & 1]);
        for (int j = 0; j < n; ++j) {
          const int t = ck + j, i = t & 1, i2 = (t + 1) & 1;
          alive &= gemm_wait(smem_u32(&v_full[i]), (t >> 1) & 1, abortp);
          if (j + 1 < n) alive &= gemm_wait(smem_u32(&k_full[i2]), ((t + 1) >> 1) & 1, abortp);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int ng = g ? it.n1 : it.n0;
            if (j < ng) {
              alive &= gemm_wait(smem_u32(&p_full[g]), (c[g] + j) & 1, abortp);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              if (elect_one() && alive) {
                pv(g, i, j);
                if (j + 1 < ng) qk(g, i2, j + 2 == ng);
              }
              const int nn = more ? (g ? next.n1 : next.n0) : 0, tn = ck + n;
              if (j + 1 == ng && nn > 0) {   // the next item's scores, while this item's last tiles and its O are worked on
                alive &= gemm_wait(smem_u32(&q_full[g]), cq[g] & 1, abortp);
                alive &= gemm_wait(smem_u32(&k_full[tn & 1]), (tn >> 1) & 1, abortp);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one() && alive) qk(g, tn & 1, nn == 1);
                ahead[g] = true;
              }
            }
          }
          if (elect_one() && alive) {
            fap_commit(&v_empty[i]);
            if (j + 1 < n) fap_commit(&k_empty[i2]);
          }
        }
        c[0] += it.n0; c[1] += it.n1; ck += n;
        it = next;
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abortp) gemm_drain();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
}

// What a tiled copy of the cache asks for: 16-byte aligned arrays, positive strides where there is more than one head / row,
// pages of whole 64-key boxes, and grid limits.
bool fa_prefill_umma_ok(const uint16_t* out, const uint16_t* q, const uint16_t* kc, const uint16_t* vc, const KvLayout& kv, int B,
                        int Hq, int Hkv, int L, int D, int offset, float scale) {
  if (!(scale > 0.f)) return false;   // the running maximum is taken before the scale
  auto off16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
  if (off16(out) || off16(q) || off16(kc) || off16(vc) || (long long)B * Hq * ((L + 255) / 256) > (1 << 30)) return false;
  if (kv.tok_stride <= 0 || (Hkv > 1 && kv.head_stride <= 0)) return false;
  return kv.page_table ? kv.page_size % 64 == 0 : (B == 1 || kv.batch_stride > 0);
}

template <int D>
static cudaError_t launch_fap(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FapArgs& a, cudaStream_t st) {
  using T = FapTile<D>;
  static std::atomic<unsigned long long> served{0};
  const cudaError_t set = once_per_device(served, [] {
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, fa_prefill_umma_kernel<D>);
    if (e != cudaSuccess) return e;
    // the warps' register shares must fit what the block is launched with, or they would wait for registers for good
    if (at.numRegs * T::THREADS < 8 * 32 * 216 + 4 * 32 * 64) return cudaErrorInvalidConfiguration;
    return cudaFuncSetAttribute(fa_prefill_umma_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
  });
  if (set != cudaSuccess) return set;
  count_launch();
  const long long items = (long long)a.B * a.Hq * a.qt;
  return launch_pdl(fa_prefill_umma_kernel<D>, dim3((unsigned)(items < num_sms() ? items : num_sms())), dim3(T::THREADS), T::SMEM, st, mq, mk, mv, a);
}

cudaError_t launch_fa_prefill_umma(uint16_t* out, const uint16_t* q, const uint16_t* kc, const uint16_t* vc, const KvLayout& kv, int B,
                                   int Hq, int Hkv, int L, int D, int offset, float scale, cudaStream_t st) {
  FapArgs a;
  a.out = out; a.Hq = Hq; a.Hkv = Hkv; a.L = L; a.offset = offset; a.B = B; a.qt = (L + 255) / 256;
  a.scale_log2e = scale * 1.4426950408889634f;
  a.page_table = kv.page_table; a.pt_stride = kv.pt_stride; a.page_size = kv.page_size;
  CUtensorMap mq, maps[2];
  if (!gemm_map(&mq, q, 2, D, L, (long long)D * 2, B * Hq, (long long)L * D * 2, 128)) return cudaErrorNotSupported;
  const GemmEncodeFn fn = gemm_encode_fn();
  const long long tok = kv.tok_stride * 2, head = Hkv > 1 ? kv.head_stride * 2 : tok;
  for (int i = 0; i < 2; ++i) {
    // contiguous: [rows][heads][keys][D] with the keys that exist; paged: [pages][heads][slots][D]
    const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)(kv.page_table ? kv.page_size : offset + L), (cuuint64_t)Hkv,
                                (cuuint64_t)(kv.page_table ? 0x7fffffff : B)};
    const cuuint64_t strides[3] = {(cuuint64_t)tok, (cuuint64_t)head,
                                   (cuuint64_t)(kv.page_table ? kv.page_size * tok : B > 1 ? kv.batch_stride * 2 : tok)};
    const cuuint32_t box[4] = {64, 64, 1, 1}, one[4] = {1, 1, 1, 1};
    if (fn(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<uint16_t*>(i ? vc : kc), dims, strides, box, one,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorNotSupported;
  }
  return D == 128 ? launch_fap<128>(mq, maps[0], maps[1], a, st) : launch_fap<64>(mq, maps[0], maps[1], a, st);
}

unsigned int fa_prefill_pipeline_error() { return gemm_error_now(); }
cudaError_t fa_prefill_pipeline_post(unsigned int* host, cudaStream_t st) { return gemm_error_post(host, st); }
cudaError_t fa_prefill_pipeline_clear() { return gemm_error_clear(); }

}  // namespace pie
