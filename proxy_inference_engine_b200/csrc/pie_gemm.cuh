// Persistent tcgen05 GEMM core, sm_100a:  acc[m, n] = sum_k x[m, k] w[n, k]  (bf16 operands, fp32 in tensor memory), shared
// by the prefill quantized GEMM (pie_qmm.cu: w is dequantised into shared memory on the way) and the dense linear of the
// hybrid families (hyb_umma.cu: w arrives by TMA).  What bounds it is the tensor pipe; the shape of the kernel follows from
// keeping that pipe fed:
//   * CG = 2: a CTA pair (two SMs) owns a 256 x BN tile (BN = 256, or less where fewer columns fill the last wave better).  Each CTA stages 128 rows of x and HALF of the w rows
//     (128), so a 64-element K step moves 32 KB into each SM for 512 tensor-pipe cycles (64 B / cycle of shared-memory reads
//     and 64 of writes, the 128 the SM has); a 128 x 256 tile of one CTA would need 192.
//   * CG = 1: one CTA owns a 128 x BN tile: few rows or few tiles, where the pair would leave SMs idle.  SPLIT cuts K over the
//     ranks of a cluster; partial tiles meet in the owners' shared memory and are added in rank order (no workspace, no
//     atomics, the same sum every time).
//   * operands by TMA into an S-deep ring of 128-byte-swizzled stages; one thread issues the MMAs; two accumulator buffers, so
//     the epilogue of a tile runs under the main loop of the next; a CTA (pair) walks tiles blockIdx, + grid, ... with the row
//     tiles of a group of `group_m` innermost, so that what is in flight at once shares rows of x and of w in L2.
//   * an epilogue warp turns 32 x 32 pieces of its tile through 4 KB of shared memory, so that rows are written in runs of 64 or 128
//     bytes: 16 bytes of 32 rows an instruction took a third of a short-K tile's time.
//   * QB = 4 / 8: a further TMA warp brings the packed rows of w, 128 bytes each, and groups of four warps turn them into
//     the stage's bf16 rows, w_hat = bf16(scale q + bias) rounded once (fused bf16x2 / fp32 multiply-add): a thread takes one
//     row of a K step, the groups take the K steps in turn (one step's chain of wait, load, store and proxy fence is longer
//     than its MMAs).
// No wait is unbounded: one that expires raises g_gemm_error and a CTA-wide flag, every role leaves its loop, copies and MMAs in
// flight are given time to land, tensor memory is freed and the kernel returns.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pie_once.h"
#include "pie_ptx.cuh"
#include "pie_umma.cuh"

namespace pie {

__attribute__((visibility("hidden"))) bool gemm_programmatic();   // each library's own: whether its switch for programmatic launches (PIE_PDL_AUX, pieh_set_pdl) leaves them on

static __device__ unsigned int g_gemm_error = 0;   // 1: a pipeline wait of a kernel of this source file expired
// the word on the host: now (waits for the device), behind what is queued on a stream, and set back
static inline unsigned int gemm_error_now() {
  unsigned int v = 0;
  cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(v));
  return v;
}
// A thread writes the word into page-locked memory: every step asks, and a copy would have the stream wait for the copy engine (a prompt and
// six decode steps of four sequences, 3400 us, took 1.2 % longer with a copy behind each and nothing that could be measured with this).
// Memory the device cannot write to is copied to.
static __global__ void gemm_error_tell(unsigned int* host) { *host = g_gemm_error; }
static inline cudaError_t gemm_error_post(unsigned int* host, cudaStream_t st) {
  void* there = nullptr;
  if (cudaHostGetDevicePointer(&there, host, 0) != cudaSuccess) {
    cudaGetLastError();
    return cudaMemcpyFromSymbolAsync(host, g_gemm_error, sizeof(*host), 0, cudaMemcpyDeviceToHost, st);
  }
  gemm_error_tell<<<1, 1, 0, st>>>((unsigned int*)there);
  return cudaGetLastError();
}
static inline cudaError_t gemm_error_clear() {
  const unsigned int v = 0;
  return cudaMemcpyToSymbol(g_gemm_error, &v, sizeof(v));
}

// ---------------------------------------------------------------------------------------------------- cluster / mbarrier
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {   // every thread of every CTA of the cluster, warps converged
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
  return d;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
constexpr uint32_t kGemmWaitLimit = 1u << 22;
// false: the wait expired here or the CTA is already leaving
__device__ __forceinline__ bool gemm_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  uint32_t ok, spins = 0;
  while (true) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if (++spins > kGemmWaitLimit || *abort_flag) {
      *abort_flag = 1;
      atomicExch(&g_gemm_error, 1u);
      return false;
    }
  }
}

// A wait of some role expired: the roles that issue have left their loops, what they asked for lands within microseconds, and nothing
// of it may outlive the CTA's shared and tensor memory.  (The issuing role need not be the one whose wait expired, and may have come to
// its end: the whole CTA waits, behind its last barrier.)
__device__ __forceinline__ void gemm_drain() {
  for (int w = 0; w < 1000; ++w) __nanosleep(1000);
}
// gemm_wait for a whole warp whose lanes go on together: one lane's expiry takes the warp out
__device__ __forceinline__ bool gemm_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, gemm_wait(bar, parity, abort_flag));
}

// ---------------------------------------------------------------------------------------------------- TMA / MMA, 1 or 2 CTAs
template <int CG>
__device__ __forceinline__ void gemm_tma_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  if (CG == 2)   // the barrier may be the leader CTA's
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void gemm_prefetch_3d(const CUtensorMap* map, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
template <int CG>
__device__ __forceinline__ void gemm_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  if (CG == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accum)
        : "memory");
  else
    umma_bf16(tmem_d, da, db, idesc, accum);
}
// arrives on `bar` (in both CTAs of a pair) once every MMA issued so far has finished
template <int CG>
__device__ __forceinline__ void gemm_commit(uint32_t bar) {
  if (CG == 2)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((uint16_t)3) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---------------------------------------------------------------------------------------------------- arguments
struct GemmArgs {
  int M, N, K;            // one product; K a multiple of 64
  int mt, nt, nb;         // tiles along m and n, independent products
  int zx, zw;             // 0: one x / one w for all products
  int group_m;            // row tiles walked together
  int k_per;              // SPLIT: K steps (of 64) per cluster rank
  const uint16_t* scales; // QB: [N, K / 64] bf16
  const uint16_t* biases;
  int scale_vec;          // QB: rows of scales / biases can be read 16 bytes (8 K steps) at a time
};

template <int CG, int BN, int QB, bool SPLIT>
struct GemmTile {
  static constexpr int BM = 128 * CG, NB = BN / CG;              // tile rows; w rows staged by one CTA
  static constexpr int A_STAGE = 128 * 128, B_STAGE = NB * 128;  // bytes of one 64-element K step
  static constexpr int CHUNK = NB * 128, RING = QB ? 3 : 0;      // packed rows: 128 bytes each, 256 (4-bit) / 128 (8-bit) of K
  static constexpr int S = QB ? 5 : 6;
  static constexpr int EPI_WARPS = QB ? 4 : 8;
  static constexpr int W_TMA = EPI_WARPS, W_MMA = EPI_WARPS + 1, W_PACK = EPI_WARPS + 2, W_DEQ = EPI_WARPS + 4;
  static constexpr int GROUPS = 3;                                // dequantising groups of four warps, a K step each in turn
  static constexpr int THREADS = 32 * (QB ? W_DEQ + 4 * GROUPS : EPI_WARPS + 4);
  static constexpr int SMEM = 1024 + S * (A_STAGE + B_STAGE) + RING * CHUNK + EPI_WARPS * 4096;
  static constexpr int ACC = BN > 128 ? 256 : 128;              // columns between the two accumulators
  static constexpr int TMEM_COLS = 2 * ACC;                      // a power of two
  static_assert(SMEM <= 227 * 1024 && TMEM_COLS <= 512 && BN % (8 * EPI_WARPS) == 0 && NB % 8 == 0, "tile");
  static_assert(!QB || NB <= 128, "a dequantising thread per row, 128 threads a group");
  // A group waits only for the packed chunks it reads, by the parity of their ring slot.  That is sound while no chunk it skipped
  // can still be on its way when it waits for the slot's next one: with these numbers the K step it dequantised last had its
  // stage freed by an MMA that came after a step of the skipped chunk.  (One slot or four groups break it: a stale chunk is read
  // and the slot's arrivals overflow.  tests/test_cpu_gemm_schedule.py walks all tile lengths.)
  static_assert(!QB || (GROUPS == 3 && RING == 3 && S == 5), "see tests/test_cpu_gemm_schedule.py before changing these");
  static_assert(!(SPLIT && CG == 2), "K is split over single CTAs");
};

// eight 4-bit codes of one word -> eight bf16 scale * q + bias in order.  128 + q is a bf16 number (one mask-or for two codes);
// subtracting 128 is exact, and the fused multiply-add rounds once.
__device__ __forceinline__ uint4 gemm_dequant4(uint32_t w, uint32_t s2, uint32_t b2) {
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t p = ((w >> (4 * j)) & 0x000f000fu) | 0x43004300u;
    o[j] = fma_bf16x2(fma_bf16x2(p, 0x3f803f80u, 0xc300c300u), s2, b2);
  }
  return make_uint4(__byte_perm(o[0], o[1], 0x5410), __byte_perm(o[2], o[3], 0x5410), __byte_perm(o[0], o[1], 0x7632),
                    __byte_perm(o[2], o[3], 0x7632));
}
// four 8-bit codes of one word -> four bf16: 2^23 + q is one byte permutation, the rest is fp32 and one rounding
__device__ __forceinline__ uint2 gemm_dequant8(uint32_t w, float s, float b) {
  float q[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) q[j] = fmaf(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + j)) - 8388608.f, s, b);
  return make_uint2(pack_bf16(q[0], q[1]), pack_bf16(q[2], q[3]));
}

struct GemmTileAt { int z, m, n; };
__device__ __forceinline__ GemmTileAt gemm_tile_at(const GemmArgs& a, int t) {
  const int per = a.mt * a.nt, z = t / per, r = t - z * per;
  const int span = a.group_m * a.nt, g = r / span, rr = r - g * span, first = g * a.group_m;
  const int gm = min(a.group_m, a.mt - first);
  return {z, first + rr % gm, rr / gm};
}

// An epilogue with a member PAIRED works on two products of one x: CTA 0 of a pair stages rows of w, CTA 1 the same rows of a second
// matrix (map_up, s_up, b_up), so a tile's accumulator holds BN / 2 columns of the one and behind them the same columns of the other.
// It is called as gate(v, t) on 32 columns of the first product and then, t in hand, on those of the second.
template <class E, class = void> struct gemm_paired { static constexpr bool value = false; };
template <class E> struct gemm_paired<E, decltype((void)E::PAIRED)> { static constexpr bool value = true; };

// An epilogue with a member SEGMENTS has the rows of up to three matrices of one K side by side for w: column tiles [tile0[i], tile0[i + 1]) are
// matrix i's, whose packed rows are map_w's or map_more[i - 1]'s and whose scales are s[i], b[i].  It is told the matrix and the column in it.
template <class E, class = void> struct gemm_segments { static constexpr bool value = false; };
template <class E> struct gemm_segments<E, decltype((void)E::SEGMENTS)> { static constexpr bool value = true; };

// Epi: void operator()(int z, int row0, int col0, const uint32_t (&v)[32], uint32_t buf, int lane), called by whole warps: 32 columns
// of rows row0 .. row0 + 31, lane l holding row l's; any row and column, the callee checks the bounds.  buf: 4 KB of shared memory
// of the warp's own, to turn the tile so that rows are written in whole runs.
template <int CG, int BN, int QB, bool SPLIT, class Epi>
__global__ void __launch_bounds__(GemmTile<CG, BN, QB, SPLIT>::THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ GemmArgs a,
            const __grid_constant__ Epi epi) {
  using T = GemmTile<CG, BN, QB, SPLIT>;
  constexpr bool PAIRED = gemm_paired<Epi>::value, SEGMENTS = gemm_segments<Epi>::value;
  static_assert(!PAIRED || (CG == 2 && QB && T::NB % 32 == 0), "each CTA of a pair stages one matrix, in whole runs");
  static_assert(!SEGMENTS || (QB && !PAIRED), "matrices side by side are dequantised ones");
  constexpr int COLS = PAIRED ? T::NB : BN;   // columns of y in a tile
  constexpr int S = T::S, RING = T::RING > 0 ? T::RING : 1, KPC = QB == 4 ? 4 : 2;   // K steps per packed chunk
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(T::BM >> 4) << 24);
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S], tfull_bar[2], tempty_bar[2], pfull_bar[RING], pempty_bar[RING];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t rank = (CG == 2 || SPLIT) ? cluster_rank() : 0;
  const uint32_t lead = CG == 2 ? 0 : rank;      // the CTA that issues this CTA's MMAs
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smA = base, smB = base + S * T::A_STAGE, smP = smB + S * T::B_STAGE;
  const int nk_all = a.K / 64;
  const int k_lo = SPLIT ? (int)rank * a.k_per : 0, k_hi = SPLIT ? min(nk_all, k_lo + a.k_per) : nk_all;
  constexpr int CL = CG;                         // CTAs per tile step of the grid; SPLIT: the whole cluster shares blockIdx.y
  const int first_tile = SPLIT ? (int)blockIdx.y : (int)blockIdx.x / CL, tile_step = SPLIT ? (int)gridDim.y : (int)gridDim.x / CL;
  const int ntiles = a.mt * a.nt * a.nb;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full_bar[s], 1 + (QB ? 4 * CG : 0));
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], T::EPI_WARPS * CG);
    }
    for (int p = 0; p < RING; ++p) {
      mbar_init(&pfull_bar[p], 1);
      mbar_init(&pempty_bar[p], 4 * KPC);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == T::W_MMA) {
    if (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                   "n"(T::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                   "n"(T::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if (warp == T::W_TMA && lane == 0) { tma_prefetch_desc(&map_x); tma_prefetch_desc(&map_w); }
  // The first operands of w on their way to L2 while the launch before this one drains.  (Nothing is read ahead of the wait: it may have written them.)
  if (warp == (QB ? T::W_PACK : T::W_TMA) && lane == 0) {
    const GemmTileAt at = gemm_tile_at(a, first_tile);
    if (QB) {
      const CUtensorMap* map = &map_w;
      int col = at.n * COLS + (int)(CG == 2 && !PAIRED ? rank : 0) * T::NB;
      if constexpr (PAIRED) map = rank ? &epi.map_up : &map_w;
      if constexpr (SEGMENTS) {
        const int g = epi.segment(at.n);
        map = g == 0 ? &map_w : &epi.map_more[g - 1];
        col -= epi.tile0[g] * BN;
      }
      for (int c = 0; c < RING && k_lo + c * KPC < k_hi; ++c) gemm_prefetch_3d(map, (k_lo / KPC + c) * 128, col, 0);
    } else {
      for (int c = 0; c < S && k_lo + c < k_hi; ++c) gemm_prefetch_3d(&map_w, (k_lo + c) * 64, at.n * BN + (int)(CG == 2 ? rank : 0) * T::NB, at.z * a.zw);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (CG == 2 || SPLIT) cluster_sync_all();      // the peers' barriers are set up
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* const abortp = &abort_flag;
  pdl_launch_dependents();   // (behind the allocation of tensor memory: a dependent may want some as well)
  pdl_wait();                // what this launch reads was written by launches before it

  if (warp < T::EPI_WARPS) {
    // ---------------------------------------------------------------- epilogue: TMEM lane quadrant warp % 4
    const int quad = warp & 3;
    const uint32_t ebuf = smP + T::RING * T::CHUNK + warp * 4096;
    constexpr int PARTS = T::EPI_WARPS / 4, RUNS = BN / 32 / PARTS;   // 32-column runs of this warp
    const int c_lo = (warp >> 2) * RUNS;
    if (!SPLIT) {
      int i = 0;
      for (int t = first_tile; t < ntiles; t += tile_step, ++i) {
        const GemmTileAt at = gemm_tile_at(a, t);
        const int b = i & 1;
        if (!gemm_wait_warp(smem_u32(&tfull_bar[b]), (i >> 1) & 1, abortp)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row0 = at.m * T::BM + (int)(CG == 2 ? rank : 0) * 128 + quad * 32;
#pragma unroll 1
        for (int c = 0; c < (PAIRED ? RUNS / 2 : RUNS); ++c) {
          uint32_t v[32], t[PAIRED ? 16 : 1];
          const uint32_t run = tmem + (uint32_t)(b * T::ACC + (c_lo + c) * 32) + ((uint32_t)(quad * 32) << 16);
          tmem_ld32(run, v);
          if constexpr (PAIRED) {
            epi.gate(v, t);
            tmem_ld32(run + T::NB, v);
          }
          if (c == (PAIRED ? RUNS / 2 : RUNS) - 1) {   // the accumulator may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              if (CG == 2) mbar_arrive_remote(map_to_rank(smem_u32(&tempty_bar[b]), lead));
              else mbar_arrive(&tempty_bar[b]);
            }
          }
          if constexpr (PAIRED) epi(row0, at.n * COLS + c * 32, t, v, ebuf, lane);
          else if constexpr (SEGMENTS) { const int g = epi.segment(at.n); epi(g, row0, (at.n - epi.tile0[g]) * BN + (c_lo + c) * 32, v, ebuf, lane); }
          else epi(at.z, row0, at.n * BN + (c_lo + c) * 32, v, ebuf, lane);
        }
      }
    } else {
      gemm_wait_warp(smem_u32(&tfull_bar[0]), 0, abortp);
    }
  } else if (warp == T::W_TMA) {
    // ---------------------------------------------------------------- operands that arrive as they are
    if (lane == 0) {
      int it = 0;
      bool alive = true;
      for (int t = first_tile; t < ntiles && alive; t += tile_step) {
        const GemmTileAt at = gemm_tile_at(a, t);
        const int row = at.m * T::BM + (int)(CG == 2 ? rank : 0) * 128, col = at.n * BN + (int)(CG == 2 ? rank : 0) * T::NB;
        for (int kb = k_lo; kb < k_hi; ++kb, ++it) {
          const int s = it % S;
          if (!(alive = gemm_wait(smem_u32(&empty_bar[s]), ((it / S) & 1) ^ 1, abortp))) break;
          const uint32_t bar = CG == 2 ? map_to_rank(smem_u32(&full_bar[s]), lead) : smem_u32(&full_bar[s]);
          if (rank == lead) mbar_arrive_expect_tx(&full_bar[s], CG * (T::A_STAGE + (QB ? 0 : T::B_STAGE)));
          gemm_tma_3d<CG>(smA + s * T::A_STAGE, &map_x, bar, kb * 64, row, at.z * a.zx);
          if (!QB) gemm_tma_3d<CG>(smB + s * T::B_STAGE, &map_w, bar, kb * 64, col, at.z * a.zw);
        }
        if (SPLIT) break;
      }
    }
  } else if (warp == T::W_MMA) {
    // ---------------------------------------------------------------- MMA issue
    // The loop's own instructions are on the critical path (a step of four MMAs is 250 to 500 cycles): the whole warp runs it,
    // so that addresses and descriptors stay warp-uniform, one elected lane issues, and nothing in it brings the lanes together
    // but the election.  (A lane's own loop with a vote per wait: 8192 x 4096 x 4096, 4 bits, 223 us; this one 197.)
    if (rank == lead) {
      const uint32_t acc = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t da0 = umma_desc_sw128(smA), db0 = umma_desc_sw128(smB);
      int i = 0, s = 0;
      uint32_t ph = 0;
      bool alive = true;   // a lane's own: a wait that expires (and every one after it) only keeps the elected lane from issuing
      for (int t = first_tile; t < ntiles; t += tile_step, ++i) {
        const int b = i & 1;
        alive &= gemm_wait(smem_u32(&tempty_bar[b]), ((i >> 1) & 1) ^ 1, abortp);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = k_lo; kb < k_hi; ++kb) {
          alive &= gemm_wait(smem_u32(&full_bar[s]), ph, abortp);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = da0 + (uint64_t)(s * (T::A_STAGE >> 4)), db = db0 + (uint64_t)(s * (T::B_STAGE >> 4));
          if (elect_one() && alive) {
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)   // 16 elements of K: 32 bytes inside the swizzle atom
              gemm_mma<CG>(acc + b * T::ACC, da + 2 * k4, db + 2 * k4, IDESC, (kb > k_lo || k4 > 0) ? 1u : 0u);
            gemm_commit<CG>(smem_u32(&empty_bar[s]));
            if (kb == k_hi - 1) gemm_commit<CG>(smem_u32(&tfull_bar[b]));
          }
          if (++s == S) { s = 0; ph ^= 1; }
        }
        if (SPLIT) break;
      }
    }
  } else if (QB && warp == T::W_PACK) {
    // ---------------------------------------------------------------- packed rows of w
    if (lane == 0) {
      int pc = 0;
      bool alive = true;
      for (int t = first_tile; t < ntiles && alive; t += tile_step) {
        const GemmTileAt at = gemm_tile_at(a, t);
        int col = at.n * COLS + (int)(CG == 2 && !PAIRED ? rank : 0) * T::NB;
        if constexpr (SEGMENTS) col -= epi.tile0[epi.segment(at.n)] * BN;
        for (int kb = k_lo; kb < k_hi; kb += KPC, ++pc) {
          const int p = pc % RING;
          if (!(alive = gemm_wait(smem_u32(&pempty_bar[p]), ((pc / RING) & 1) ^ 1, abortp))) break;
          mbar_arrive_expect_tx(&pfull_bar[p], T::CHUNK);
          const CUtensorMap* map = &map_w;
          if constexpr (PAIRED) map = rank ? &epi.map_up : &map_w;
          if constexpr (SEGMENTS) { const int g = epi.segment(at.n); map = g == 0 ? &map_w : &epi.map_more[g - 1]; }
          gemm_tma_3d<1>(smP + p * T::CHUNK, map, smem_u32(&pfull_bar[p]), kb / KPC * 128, col, 0);
        }
        if (SPLIT) break;
      }
    }
  } else if (QB && warp >= T::W_DEQ) {
    // ---------------------------------------------------------------- dequantisers: thread = row, group = every GROUPS-th K step
    const int r = (tid - 32 * T::W_DEQ) & 127, grp = (warp - T::W_DEQ) >> 2;
    const uint32_t swz = (uint32_t)(r & 7);
    const int chunks = (k_hi - k_lo + KPC - 1) / KPC;      // of one tile
    int it0 = 0, pc0 = 0;                                   // K steps and chunks of the tiles before this one
    bool alive = true;
    for (int t = first_tile; t < ntiles && alive; t += tile_step, it0 += k_hi - k_lo, pc0 += chunks) {
      const GemmTileAt at = gemm_tile_at(a, t);
      int row = at.n * COLS + (int)(CG == 2 && !PAIRED ? rank : 0) * T::NB + min(r, T::NB - 1);
      const uint16_t *sp = a.scales, *bp = a.biases;
      if constexpr (SEGMENTS) {
        const int g = epi.segment(at.n);
        row = min(row - epi.tile0[g] * BN, epi.N[g] - 1);
        sp = epi.s[g]; bp = epi.b[g];
      } else {
        row = min(row, a.N - 1);
      }
      if constexpr (PAIRED)
        if (rank) { sp = epi.s_up; bp = epi.b_up; }
      sp += (size_t)row * nk_all;
      bp += (size_t)row * nk_all;
      int kb = k_lo + (grp + T::GROUPS - it0 % T::GROUPS) % T::GROUPS;
      uint4 sv = make_uint4(0, 0, 0, 0), bv = sv, sn = sv, bn = sv;   // scale_vec: eight K steps' values, and the next eight
      uint32_t s_next = 0, b_next = 0;                      // otherwise: the next step's
      int have = -1;
      if (a.scale_vec) {
        sn = __ldg(reinterpret_cast<const uint4*>(sp + k_lo));
        bn = __ldg(reinterpret_cast<const uint4*>(bp + k_lo));
      } else if (kb < k_hi) {
        s_next = __ldg(sp + kb);
        b_next = __ldg(bp + kb);
      }
      for (; kb < k_hi; kb += T::GROUPS) {
        const int it = it0 + kb - k_lo, pc = pc0 + (kb - k_lo) / KPC;
        const int s = it % S, p = pc % RING, j = kb % KPC;
        uint32_t sc, bi;                                    // bf16 bits
        if (a.scale_vec) {
          const int e = kb & 7;
          if ((kb >> 3) != have) {
            have = kb >> 3;
            sv = sn; bv = bn;
            if (8 * have + 8 < k_hi) {
              sn = __ldg(reinterpret_cast<const uint4*>(sp + 8 * have + 8));
              bn = __ldg(reinterpret_cast<const uint4*>(bp + 8 * have + 8));
            }
          }
          const uint32_t sw = e < 4 ? (e < 2 ? sv.x : sv.y) : (e < 6 ? sv.z : sv.w);
          const uint32_t bw = e < 4 ? (e < 2 ? bv.x : bv.y) : (e < 6 ? bv.z : bv.w);
          sc = (e & 1) ? sw >> 16 : sw & 0xffffu;
          bi = (e & 1) ? bw >> 16 : bw & 0xffffu;
        } else {
          sc = s_next; bi = b_next;
          if (kb + T::GROUPS < k_hi) { s_next = __ldg(sp + kb + T::GROUPS); b_next = __ldg(bp + kb + T::GROUPS); }
        }
        if (!(alive = gemm_wait_warp(smem_u32(&pfull_bar[p]), (pc / RING) & 1, abortp))) break;
        const uint32_t src = smP + p * T::CHUNK + min(r, T::NB - 1) * 128, dst = smB + s * T::B_STAGE + r * 128;
        uint4 w[QB == 4 ? 2 : 4];
#pragma unroll
        for (int c = 0; c < QB / 2; ++c) w[c] = lds128(src + (((uint32_t)(QB / 2 * j + c) ^ swz) << 4));
        if (!(alive = gemm_wait_warp(smem_u32(&empty_bar[s]), ((it / S) & 1) ^ 1, abortp))) break;
        if (T::NB < 128 && r >= T::NB) {
          // (no row of this tile: the thread only keeps the warp's count)
        } else if (QB == 4) {
          const uint32_t s2 = sc | (sc << 16), b2 = bi | (bi << 16);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 q = w[c >> 2];
            const uint4 o = gemm_dequant4((c & 3) == 0 ? q.x : (c & 3) == 1 ? q.y : (c & 3) == 2 ? q.z : q.w, s2, b2);
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (((uint32_t)c ^ swz) << 4)), "r"(o.x), "r"(o.y),
                         "r"(o.z), "r"(o.w) : "memory");
          }
        } else {
          const float sf = __uint_as_float(sc << 16), bf = __uint_as_float(bi << 16);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 q = w[c >> 1];
            const uint2 o0 = gemm_dequant8(c & 1 ? q.z : q.x, sf, bf), o1 = gemm_dequant8(c & 1 ? q.w : q.y, sf, bf);
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (((uint32_t)c ^ swz) << 4)), "r"(o0.x), "r"(o0.y),
                         "r"(o1.x), "r"(o1.y) : "memory");
          }
        }
        fence_proxy_async();   // generic-proxy stores -> the tensor core's async proxy
        __syncwarp();
        if (lane == 0) {
          if (CG == 2) mbar_arrive_remote(map_to_rank(smem_u32(&full_bar[s]), lead));
          else mbar_arrive(&full_bar[s]);
          mbar_arrive_n(&pempty_bar[p], kb == k_hi - 1 ? KPC - j : 1);   // the last chunk of a tile may hold fewer steps
        }
      }
      if (SPLIT) break;
    }
  }

  __syncwarp();
  if (SPLIT) {
    // ---- partial tiles meet: the 32-column run g belongs to rank g % ranks, which adds the ranks' parts in rank order.  The
    // parts lie where the operand stages were (every rank is past its main loop), [run][source][4 columns][row] in 16 bytes.
    const uint32_t ranks = gridDim.x;
    cluster_sync_all();
    if (warp < 4 && !*abortp) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int row_in = warp * 32 + lane;
#pragma unroll 1
      for (int g = 0; g < BN / 32; ++g) {
        uint32_t v[32];
        tmem_ld32(tmem + (uint32_t)(g * 32) + ((uint32_t)(warp * 32) << 16), v);
        const uint32_t dst = map_to_rank(base, g % ranks) + ((uint32_t)((g / ranks) * ranks + rank) * 8 * 128 + row_in) * 16;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + q * 128 * 16), "r"(v[4 * q]), "r"(v[4 * q + 1]),
                       "r"(v[4 * q + 2]), "r"(v[4 * q + 3]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < T::EPI_WARPS && !*abortp) {
      const GemmTileAt at = gemm_tile_at(a, first_tile);
      const int row_in = (warp & 3) * 32 + lane;
      for (int gi = warp >> 2; gi * (int)ranks + (int)rank < BN / 32; gi += T::EPI_WARPS / 4) {
        uint32_t v[32];
        float acc[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) acc[q] = 0.f;
        for (int src = 0; src < (int)ranks; ++src) {
          const uint32_t p = base + ((uint32_t)(gi * (int)ranks + src) * 8 * 128 + row_in) * 16;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 u = lds128(p + q * 128 * 16);
            acc[4 * q] += __uint_as_float(u.x); acc[4 * q + 1] += __uint_as_float(u.y);
            acc[4 * q + 2] += __uint_as_float(u.z); acc[4 * q + 3] += __uint_as_float(u.w);
          }
        }
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(acc[q]);
        if constexpr (SEGMENTS) {
          const int g = epi.segment(at.n);
          epi(g, at.m * T::BM + (warp & 3) * 32, (at.n - epi.tile0[g]) * BN + (gi * (int)ranks + (int)rank) * 32, v,
              smP + T::RING * T::CHUNK + warp * 4096, lane);
        } else if constexpr (!PAIRED) {
          epi(at.z, at.m * T::BM + (warp & 3) * 32, at.n * BN + (gi * (int)ranks + (int)rank) * 32, v,
              smP + T::RING * T::CHUNK + warp * 4096, lane);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abortp) gemm_drain();
  if (CG == 2) cluster_sync_all();   // neither CTA of a pair leaves while the other may still use its memory
  if (warp == T::W_MMA) {
    if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(T::TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(T::TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------- host side
typedef CUresult (*GemmEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline GemmEncodeFn gemm_encode_fn() {
  static const GemmEncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess ? (GemmEncodeFn)p : (GemmEncodeFn) nullptr;
  }();
  return fn;
}
// rows of `inner` elements (2 bytes, or 1: packed words) `pitch` bytes apart, `nb` such matrices `bpitch` bytes apart; boxes of
// 128 bytes x box_rows, 128-byte swizzle, zeros beyond the ends.  base and pitches are multiples of 16 bytes.
inline bool gemm_map(CUtensorMap* m, const void* p, int elem_bytes, long long inner, long long rows, long long pitch, int nb,
                     long long bpitch, int box_rows) {
  const GemmEncodeFn fn = gemm_encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)nb};
  const cuuint64_t strides[2] = {(cuuint64_t)pitch, (cuuint64_t)(nb > 1 ? bpitch : pitch)};
  const cuuint32_t box[3] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows, 1}, one[3] = {1, 1, 1};
  return fn(m, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(p), dims,
            strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Measured, B200, 4-bit weights, us (TFLOP/s) with the 256 x 256 tile of one CTA, cp.async producers and no overlap of the
// epilogue that this replaced -> here: 8192 x 14336 x 4096 1590 (605) -> 676 (1424); 1000 rows 290 -> 97; 200 rows 29; 77 rows 400 -> 27;
// 77 x 4096 x 14336 720 -> 29 (a cluster's ranks).  8 bits, 1000 rows: 280 -> 111.  bf16 weights: 8192 x 4096 x 4096 179 (1537).
// The tile for a shape: a pair's 256 x {256, 224, 192, 128}, or a single CTA's 128 x 128 with K over 1..4 ranks of a cluster --
// whichever the estimate (waves x K steps x SM cycles of a step, and the fixed cost of a cluster's reduction) says is done first.
// The steps' cycles are measured (1.9 GHz; waves x 64 steps of N 14336, M 1000): pairs with bf16 weights 720 / 612 / 575 for BN = 256 /
// 192 / 128, dequantised 770 / 765 / 680 / 630 for 256 / 224 / 192 / 128, single CTAs 580 and 650.  Over 190 shapes (M 77 to 3000) the
// choice takes 1.02 times the best tile's time on average.
struct GemmChoice { int pair, bn, ranks, k_per, mt, nt; double cycles; };
inline double gemm_pair_step(int bn, bool quant) { return quant ? 490 + 280 * bn / 256.0 : 430 + 290 * bn / 256.0; }
inline GemmChoice gemm_choose(int M, int N, int K, int nb, int sms, bool quant, int N1 = 0, int N2 = 0) {   // N1, N2: matrices beside it
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  auto cols = [&](int bn) { return up(N, bn) + up(N1, bn) + up(N2, bn); };
  const long long nk = K / 64;
  GemmChoice best = {1, 256, 1, (int)nk, (int)up(M, 256), (int)cols(256), 1e30};
  for (int bn : {256, 224, 192, 128}) {
    if (bn == 224 && !quant) continue;   // (the eight epilogue warps of the dense kernel share 64-column runs)
    const long long tiles = up(M, 256) * cols(bn) * nb;
    const double c = (double)up(tiles, sms / 2) * nk * gemm_pair_step(bn, quant);
    if (c < best.cycles) best = {1, bn, 1, (int)nk, (int)up(M, 256), (int)cols(bn), c};
  }
  const long long tiles = up(M, 128) * cols(128) * nb;
  const double step = quant ? 650 : 580;
  for (int r = 1; r <= 4; ++r) {
    const long long per = up(up(nk, r), 8) * 8;     // ranks start on 16-byte runs of the scales and on whole packed chunks
    if (up(nk, per) != r || tiles > 65535) continue;
    // clusters of three or four do not fill every SM: what is resident at once was 128 CTAs and more for four, not 144 for three
    const long long slots = r == 3 ? sms * 3 / 4 : r == 4 ? sms * 7 / 8 : sms;
    const double c = (double)up(tiles * r, slots) * (per * step + (r > 1 ? 4500 : 0));
    if (c < best.cycles) best = {0, 128, r, (int)per, (int)up(M, 128), (int)cols(128), c};
  }
  return best;
}

template <int CG, int BN, int QB, bool SPLIT, class Epi>
cudaError_t gemm_launch(const CUtensorMap& mx, const CUtensorMap& mw, const GemmArgs& a, const Epi& epi, int ranks, int sms,
                        cudaStream_t st) {
  using T = GemmTile<CG, BN, QB, SPLIT>;
  auto kern = gemm_kernel<CG, BN, QB, SPLIT, Epi>;
  static std::atomic<unsigned long long> served{0};
  const cudaError_t set = once_per_device(served, [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM); });
  if (set != cudaSuccess) return set;
  const int tiles = a.mt * a.nt * a.nb, slots = sms / CG;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = SPLIT ? dim3((unsigned)ranks, (unsigned)tiles, 1) : dim3((unsigned)((tiles < slots ? tiles : slots) * CG), 1, 1);
  cfg.blockDim = dim3(T::THREADS, 1, 1);
  cfg.dynamicSmemBytes = T::SMEM;
  cfg.stream = st;
  // A programmatic dependent of the launch before it: the set-up (barriers, tensor memory, the peers, descriptors) runs under that one's end.  A prompt
  // layer's eight launches, all of them such, 1531 tokens of the 1B sizes: 251.7 -> 246 us; 77 rows of an 8B feed-forward 78.0 -> 75.1.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = SPLIT ? (unsigned)ranks : (unsigned)CG;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  const bool pdl = gemm_programmatic(), cluster = CG == 2 || SPLIT;
  cfg.attrs = pdl ? attr : attr + 1;
  cfg.numAttrs = (pdl ? 1 : 0) + (cluster ? 1 : 0);
  return cudaLaunchKernelEx(&cfg, kern, mx, mw, a, epi);
}

// One product (or nb of them): picks the tile, describes the operands and launches.  w_inner / w_pitch in bytes: a row of w as it
// lies (packed words for QB).
template <int QB, class Epi>
cudaError_t gemm_run(GemmArgs a, const Epi& epi, const void* x, long long x_pitch, long long x_bpitch, const void* w,
                     long long w_bpitch, int sms, cudaStream_t st) {
  GemmChoice c = gemm_choose(a.M, a.N, a.K, a.nb, sms, QB != 0);
  a.mt = c.mt; a.nt = c.nt; a.k_per = c.k_per; a.group_m = 8;
  const long long w_row = QB ? (long long)a.K * QB / 8 : (long long)a.K * 2;
  CUtensorMap mx, mw;
  if (!gemm_map(&mx, x, 2, a.K, a.M, x_pitch, a.zx ? a.nb : 1, x_bpitch, 128) ||
      !gemm_map(&mw, w, QB ? 1 : 2, QB ? w_row : a.K, a.N, w_row, a.zw ? a.nb : 1, w_bpitch, c.pair ? c.bn / 2 : c.bn))
    return cudaErrorNotSupported;
  if (!c.pair)
    return c.ranks == 1 ? gemm_launch<1, 128, QB, false>(mx, mw, a, epi, 1, sms, st) : gemm_launch<1, 128, QB, true>(mx, mw, a, epi, c.ranks, sms, st);
  if (c.bn == 256) return gemm_launch<2, 256, QB, false>(mx, mw, a, epi, 1, sms, st);
  if constexpr (QB != 0)
    if (c.bn == 224) return gemm_launch<2, 224, QB, false>(mx, mw, a, epi, 1, sms, st);
  return c.bn == 192 ? gemm_launch<2, 192, QB, false>(mx, mw, a, epi, 1, sms, st) : gemm_launch<2, 128, QB, false>(mx, mw, a, epi, 1, sms, st);
}

// One x, up to three matrices of N[i] rows side by side (an Epi with SEGMENTS, whose maps and tile0 are filled in here).
template <int QB, class Epi>
cudaError_t gemm_run_segments(GemmArgs a, Epi epi, int n, const void* x, const uint32_t* const* w, int sms, cudaStream_t st) {
  const GemmChoice c = gemm_choose(a.M, epi.N[0], a.K, 1, sms, true, n > 1 ? epi.N[1] : 0, n > 2 ? epi.N[2] : 0);
  a.mt = c.mt; a.nt = c.nt; a.k_per = c.k_per; a.group_m = 8;
  const int bn = c.pair ? c.bn : 128;
  const long long w_row = (long long)a.K * QB / 8;
  CUtensorMap mx, mw;
  if (!gemm_map(&mx, x, 2, a.K, a.M, (long long)a.K * 2, 1, 0, 128)) return cudaErrorNotSupported;
  for (int i = 0, t = 0; i < 3; ++i) {
    epi.tile0[i] = i < n ? t : 0x7fffffff;
    if (i >= n) continue;
    if (!gemm_map(i == 0 ? &mw : &epi.map_more[i - 1], w[i], 1, w_row, epi.N[i], w_row, 1, 0, c.pair ? bn / 2 : bn)) return cudaErrorNotSupported;
    t += (epi.N[i] + bn - 1) / bn;
  }
  if (!c.pair)
    return c.ranks == 1 ? gemm_launch<1, 128, QB, false>(mx, mw, a, epi, 1, sms, st) : gemm_launch<1, 128, QB, true>(mx, mw, a, epi, c.ranks, sms, st);
  if (bn == 256) return gemm_launch<2, 256, QB, false>(mx, mw, a, epi, 1, sms, st);
  if (bn == 224) return gemm_launch<2, 224, QB, false>(mx, mw, a, epi, 1, sms, st);
  return bn == 192 ? gemm_launch<2, 192, QB, false>(mx, mw, a, epi, 1, sms, st) : gemm_launch<2, 128, QB, false>(mx, mw, a, epi, 1, sms, st);
}

// Two products of one x in pairs' tiles (an Epi with PAIRED), of 256, 192 or 128 columns.  bn = 0: not worth it.
inline GemmChoice gemm_choose_paired(int M, int N, int K, int sms, double apart) {
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long nk = K / 64;
  GemmChoice best = {1, 0, 1, (int)nk, 0, 0, apart};
  for (int bn : {256, 192, 128}) {
    const double c = (double)up(up(M, 256) * up(N, bn / 2), sms / 2) * nk * gemm_pair_step(bn, true);
    if (c < best.cycles) best = {1, bn, 1, (int)nk, (int)up(M, 256), (int)up(N, bn / 2), c};
  }
  return best;
}
template <int QB, class Epi>
cudaError_t gemm_run_paired(GemmArgs a, Epi epi, const GemmChoice& c, const void* x, const void* w, const void* w_up, int sms, cudaStream_t st) {
  a.mt = c.mt; a.nt = c.nt; a.k_per = c.k_per; a.group_m = 8;
  const long long w_row = (long long)a.K * QB / 8;
  CUtensorMap mx, mw;
  if (!gemm_map(&mx, x, 2, a.K, a.M, (long long)a.K * 2, 1, 0, 128) || !gemm_map(&mw, w, 1, w_row, a.N, w_row, 1, 0, c.bn / 2) ||
      !gemm_map(&epi.map_up, w_up, 1, w_row, a.N, w_row, 1, 0, c.bn / 2))
    return cudaErrorNotSupported;
  if (c.bn == 256) return gemm_launch<2, 256, QB, false>(mx, mw, a, epi, 1, sms, st);
  return c.bn == 192 ? gemm_launch<2, 192, QB, false>(mx, mw, a, epi, 1, sms, st) : gemm_launch<2, 128, QB, false>(mx, mw, a, epi, 1, sms, st);
}

}  // namespace pie
