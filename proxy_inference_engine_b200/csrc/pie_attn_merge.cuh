// The partial results of decode attention's splits: who adds them up, and how (pie_attn.cu, pie_fa.cu, pie_kvq.cu).
//   part  [rows][nsplit][D + 2] floats: acc[D], running maximum (base 2), running sum
// A CTA per split; the last one to arrive adds all of them up in split order.  What it costs is trips to the L2: one thread's fence and counter, then
// the maxima and the first eight splits' rows together, then eight splits a trip.  (A fence by every thread, and loops over the splits that the compiler
// cuts in fours and that take a trip a split for what is left over, cost 4 to 8 us: 32 query heads on 8, D 128, us before -> now, 8-bit cache bs1 ctx4000
// 7 splits 18.9 -> 10.8, bs5 ctx7002 7 splits 30.1 -> 21.1; bf16 bs1 ctx1000 16 splits 10.2 -> 7.1, bs5 ctx7002 7 splits 34.3 -> 27.4.)
#pragma once
#include "pie_ptx.cuh"

namespace pie {

// true in every thread of the last of n CTAs; what the others stored before is then theirs to read (ld.cg)
__device__ __forceinline__ bool last_to_arrive(unsigned int* count, int n, int* flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int before;   // (release and acquire reach, through the barriers, what every thread of the CTA stored and will read)
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(count) : "memory");
    *flag = before == (unsigned)n - 1;
    if (*flag) *count = 0;   // for the next launch: nobody else comes
  }
  __syncthreads();
  return *flag;
}

// out [rows][D].  A warp a row, a lane every 32nd feature.
template <int D>
__device__ __forceinline__ void merge_splits(uint16_t* out, const float* part, int rows, int nsplit) {
  constexpr int PW = D + 2, E = D / 32, N = 8;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int r = threadIdx.x >> 5; r < rows; r += warps) {
    const float* const rec = part + (size_t)r * nsplit * PW;
    float mn = lane < nsplit ? ldcg_f32(rec + (size_t)lane * PW + D) : -INFINITY;
    float lt = 0.f, at[E];
#pragma unroll
    for (int e = 0; e < E; ++e) at[e] = 0.f;
    for (int s0 = 0; s0 < nsplit; s0 += N) {
      const int n = min(N, nsplit - s0);
      float v[N][E], ms = -INFINITY, ls = 0.f;
      if (lane < n) {
        ms = ldcg_f32(rec + (size_t)(s0 + lane) * PW + D);
        ls = ldcg_f32(rec + (size_t)(s0 + lane) * PW + D + 1);
      }
#pragma unroll
      for (int s = 0; s < N; ++s)
#pragma unroll
        for (int e = 0; e < E; ++e) v[s][e] = s < n ? ldcg_f32(rec + (size_t)(s0 + s) * PW + 32 * e + lane) : 0.f;
      if (s0 == 0) {
        for (int s = 32 + lane; s < nsplit; s += 32) mn = fmaxf(mn, ldcg_f32(rec + (size_t)s * PW + D));
        mn = warp_max(mn);
      }
      const float w = ms == -INFINITY ? 0.f : exp2f(ms - mn);
#pragma unroll
      for (int s = 0; s < N; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s), l = __shfl_sync(0xffffffffu, ls, s);
        if (s < n) {
          lt += l * ws;
#pragma unroll
          for (int e = 0; e < E; ++e) at[e] += v[s][e] * ws;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) out[(size_t)r * D + 32 * e + lane] = f2bf(at[e] / lt);
  }
}

}  // namespace pie
