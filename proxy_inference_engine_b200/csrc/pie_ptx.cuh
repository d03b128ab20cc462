// sm_100a PTX wrappers used by the decode engine: mbarrier, TMA (cp.async.bulk.tensor), mma.sync,
// cache-hinted global loads.  Every spin has a watchdog that traps instead of hanging the GPU.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace pie {

#ifndef PIE_SPIN_LIMIT
#define PIE_SPIN_LIMIT (1u << 20)  // try_wait itself blocks for a while: ~ seconds in total; a healthy wait is microseconds
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity) {
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (++spins > PIE_SPIN_LIMIT) __trap();
  }
}

// ------------------------------------------------------------------ TMA
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// bytes (a multiple of 16, from a 16-byte boundary) on their way to L2
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const void* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
// 2-D tiled load: coordinates are (c0 = innermost element index, c1 = row index).
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const void* map, uint64_t* bar, int c0,
                                            int c1, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_dst),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}

// ------------------------------------------------------------------ tensor-core MMA (legacy warp path)
// D(16x8,f32) = A(16x16,bf16,row) * B(16x8,bf16,col) + C.  Fragment layout (g = lane>>2, t = lane&3):
//   a0:(g, 2t..2t+1) a1:(g+8, 2t..) a2:(g, 2t+8..) a3:(g+8, 2t+8..)   b0:(k 2t..2t+1, n g) b1:(k 2t+8.., n g)
//   c0,c1:(g, 2t..2t+1)  c2,c3:(g+8, 2t..2t+1)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                               uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------ shared / global access helpers
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
// L2-coherent loads for data another CTA wrote earlier in the same launch (L1 may be stale).
__device__ __forceinline__ uint4 ldcg128(const void* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ldcg64(const void* p) {
  uint2 v;
  asm volatile("ld.global.cg.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ldcg32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ldcg_f32(const void* p) { return __uint_as_float(ldcg32(p)); }
__device__ __forceinline__ uint16_t ldcg16(const void* p) {
  uint16_t v;
  asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ------------------------------------------------------------------ system-scope flags (tensor-parallel exchanges)
__device__ __forceinline__ void st_release_sys(unsigned int* p, unsigned int v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void wait_flag(const unsigned int* p, unsigned int e) {
  unsigned long long spins = 0;
  while ((int)(ld_acquire_sys(p) - e) < 0) {
    if (++spins > 4096) __nanosleep(256);
    if (spins > (1ull << 28)) __trap();  // ~ a minute: a peer died
  }
}
// ------------------------------------------------------------------ cp.async (LDGSTS) per-thread copies
__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// Programmatic dependent launch (PDL): wait for the producer grid / let the dependent grid start.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------------------------ bf16 helpers
__device__ __forceinline__ float bf16lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// fp32 -> bf16, round to nearest even, NaN -> 0x7FFF canonical.  Always through the PACKED conversion
// (F2FP.BF16.F32.PACK_AB, full-rate ALU pipe): the scalar F2F.BF16.F32 issues on the quarter-rate XU pipe and was the top
// stall in the dequantising producers.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ uint16_t f2bf(float f) { return (uint16_t)(pack_bf16(f, 0.f) & 0xffffu); }
__device__ __forceinline__ float bfround(float f) { return __uint_as_float(pack_bf16(0.f, f) & 0xffff0000u); }
// 1 / (1 + e^-a), approximately, in six instructions.  Divisors beyond 2^126, whose reciprocal is subnormal (__fdividef makes it 0),
// are taken a quarter at a time; rcp.approx.f32, which handles them itself, cost the whole kernel 28 % of its time.
__device__ __forceinline__ float sigmoid_approx(float a) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(a * -1.4426950408889634f));   // (e^-a below 2^-126 adds nothing to 1)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaf(e, 0.25f, 0.25f)));
  return r * 0.25f;
}
// silu of two bf16 values, bf16 after every operator: sigmoid, gate * sigmoid.  The approximations are off by a few units of fp32's
// last place and the sigmoid is rounded to bf16 at once: for all 65536 gates the bits are those of 1 / (1 + expf(-g)) with a full
// division, which the layers of up to 32 rows use and which the memory-bound kernel over a prompt's rows has no time for
// (8192 x 14336: 2-byte accesses and full division 408 us, 16-byte accesses and this 130; 123 with __fdividef).
__device__ __forceinline__ uint32_t silu_bf16x2(uint32_t g) {
  const float a = __uint_as_float(g << 16), b = __uint_as_float(g & 0xffff0000u);
  const uint32_t s = pack_bf16(sigmoid_approx(a), sigmoid_approx(b));
  return pack_bf16(a * __uint_as_float(s << 16), b * __uint_as_float(s & 0xffff0000u));
}
__device__ __forceinline__ uint32_t mul_bf16x2_rn(uint32_t t, uint32_t u) {   // products in fp32, one rounding
  return pack_bf16(__uint_as_float(t << 16) * __uint_as_float(u << 16), __uint_as_float(t & 0xffff0000u) * __uint_as_float(u & 0xffff0000u));
}
// bf16x2 fused multiply-add (HFMA2.BF16, FMA pipe): fp32-exact product and sum, ONE rounding per lane
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// sin / cos of a rotary angle theta >= 0 (up to ~1e5 rad): theta is reduced to [-pi, pi] with 2 pi split in two fp32 pieces
// (each FMA rounds once, at magnitude <= pi: ~2.5e-7 absolute), then the SFU approximations (~5e-7 absolute on that range).
// The rotated values are rounded to bf16 (2^-9 relative); the library sincosf costs ~500 cycles per call here because of
// its large-argument path.  Every rotary kernel of this library uses this one function, so they agree bit for bit.
__device__ __forceinline__ void rope_sincos(float theta, float* sn, float* cs) {
  const float k = rintf(theta * 0.15915494309189535f);
  float r = fmaf(-k, 6.2831854820251465f, theta);
  r = fmaf(k, 1.7484555e-7f, r);
  *sn = __sinf(r);
  *cs = __cosf(r);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace pie
