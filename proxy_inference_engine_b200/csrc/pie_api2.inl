// Second half of the C ABI (included by pie_api.cu): qmm, norm, rope, KV cache, attention, glue, sampler.
static pie::KvLayout to_kv(const pie_kv_layout* k) {
  pie::KvLayout o;
  o.batch_stride = k->batch_stride; o.head_stride = k->head_stride; o.tok_stride = k->tok_stride;
  o.page_table = k->page_table; o.pt_stride = k->pt_stride; o.page_size = k->page_size;
  return o;
}
static int check_kv(const pie_kv_layout* k, int D) {
  if (!k) return PIE_ENULL;
  if (k->tok_stride < D || k->tok_stride % 8 || k->head_stride % 8 || k->batch_stride % 8) return PIE_EINVAL_SHAPE;
  if (k->page_table && (k->page_size <= 0 || k->pt_stride <= 0)) return PIE_EINVAL_SHAPE;
  return PIE_OK;
}

extern "C" {

// M >= 64: the tcgen05 / TMEM tile kernel (pie_qmm.cu), weights dequantised once to bf16 into shared memory; up to 128 rows the kernel
// of pie_qmt.cuh where it is sooner done and the workspace has room for it (pie_qmv finds that out).
// Smaller M, or shapes off its grid (K % 128, unaligned pointers): pie_qmv.  (33 .. 63 rows do not go to the tile kernel, which multiplies weights
// rounded to bf16, where the others multiply the exact codes.)
int pie_qmm(void* y, const void* x, const uint32_t* wq, const void* scales, const void* biases, int M, int N,
            int K, int group_size, int bits, void* workspace, size_t workspace_bytes, void* stream) {
  if (M == 0 || N == 0) return PIE_OK;
  if (!y || !x || !wq || !scales || !biases) return PIE_ENULL;
  if (M < 0 || N < 0 || K <= 0) return PIE_EINVAL_SHAPE;
  const bool tc = M >= 64 && quant_supported(group_size, bits) && K % 128 == 0 && aligned16(x) && aligned16(wq) &&
                  aligned16(y) && !(reinterpret_cast<uintptr_t>(scales) & 3) &&
                  !(reinterpret_cast<uintptr_t>(biases) & 3) && env_int("PIE_QMM_TC", 1) != 0;
  if (tc && workspace && M <= kQmtRows && qmt_pays(M, N, K, bits, 0)) {
    pie_qmv_seg seg = {wq, scales, biases, N};
    if (qmt_takes(M, K, K, &seg, 1, group_size, bits) && kWsCntBytes + qmt_scratch(M, N, K, group_size, bits, 0) <= workspace_bytes) {
      const cudaError_t e = launch_qmt(y, N, x, K, M, K, &seg, 1, bits, nullptr, 0.f, PIE_EPI_STORE, nullptr, (uint8_t*)workspace + kWsCntBytes,
                                       (cudaStream_t)stream);
      if (e != cudaErrorNotSupported) return cuda_status(e);
    }
  }
  if (tc)
    return cuda_status(launch_qmm_tc((uint16_t*)y, (const uint16_t*)x, wq, (const uint16_t*)scales,
                                     (const uint16_t*)biases, M, N, K, bits, (cudaStream_t)stream));
  return pie_qmv(y, x, wq, scales, biases, M, N, K, group_size, bits, workspace, workspace_bytes, stream);
}

int pie_qmm_swiglu_pays(int M, int N, int K, int group_size, int bits) {
  return M >= 64 && N > 0 && K > 0 && K % 128 == 0 && quant_supported(group_size, bits) && qmm_swiglu_pays(M, N, K);
}
// silu(x w_gate^T) * (x w_up^T) on the same tile kernel.  Another status than PIE_OK: nothing was launched.
int pie_qmm_swiglu(void* y, const void* x, const pie_qmv_seg* gate_up, int M, int K, int group_size, int bits, void* stream) {
  if (!y || !x || !gate_up || !gate_up[0].wq || !gate_up[1].wq || !gate_up[0].scales || !gate_up[1].scales || !gate_up[0].biases ||
      !gate_up[1].biases)
    return PIE_ENULL;
  const int N = gate_up[0].N;
  if (M < 0 || N < 0 || K <= 0 || gate_up[1].N != N) return PIE_EINVAL_SHAPE;
  if (M == 0 || N == 0) return PIE_OK;
  if (M < 64 || !quant_supported(group_size, bits) || K % 128 || !aligned16(x) || !aligned16(y) || env_int("PIE_QMM_TC", 1) == 0)
    return PIE_EUNSUPPORTED;
  const uint32_t* wq[2];
  const uint16_t *s[2], *b[2];
  for (int i = 0; i < 2; ++i) {
    wq[i] = gate_up[i].wq; s[i] = (const uint16_t*)gate_up[i].scales; b[i] = (const uint16_t*)gate_up[i].biases;
    if (!aligned16(wq[i]) || ((reinterpret_cast<uintptr_t>(s[i]) | reinterpret_cast<uintptr_t>(b[i])) & 3)) return PIE_EUNSUPPORTED;
  }
  const cudaError_t e = launch_qmm_swiglu((uint16_t*)y, (const uint16_t*)x, wq, s, b, M, N, K, bits, (cudaStream_t)stream);
  return e == cudaErrorNotSupported ? PIE_EUNSUPPORTED : cuda_status(e);
}

// Another status than PIE_OK: nothing was launched.
int pie_qmm_rows(void* y, int y_ld, const void* x, const pie_qmv_seg* segs, int nseg, const void* residual, int M, int K, int group_size, int bits,
                 void* stream) {
  if (!y || !x || !segs) return PIE_ENULL;
  if (M < 0 || K <= 0 || nseg < 1 || nseg > kMaxSeg) return PIE_EINVAL_SHAPE;
  long long n = 0;
  bool ok = M >= 64 && quant_supported(group_size, bits) && K % 128 == 0 && aligned16(x) && aligned16(y) && aligned16(residual) &&
            env_int("PIE_QMM_TC", 1) != 0;
  for (int i = 0; i < nseg; ++i) {
    if (!segs[i].wq || !segs[i].scales || !segs[i].biases) return PIE_ENULL;
    if (segs[i].N <= 0) return PIE_EINVAL_SHAPE;
    n += segs[i].N;
    ok = ok && aligned16(segs[i].wq) && !((reinterpret_cast<uintptr_t>(segs[i].scales) | reinterpret_cast<uintptr_t>(segs[i].biases)) & 3);
  }
  if (y_ld < n) return PIE_EINVAL_SHAPE;
  if (M == 0) return PIE_OK;
  if (!ok || n > 0x7fffffff) return PIE_EUNSUPPORTED;
  const cudaError_t e = launch_qmm_rows((uint16_t*)y, y_ld, (const uint16_t*)x, segs, nseg, (const uint16_t*)residual, M, K, bits, (cudaStream_t)stream);
  return e == cudaErrorNotSupported ? PIE_EUNSUPPORTED : cuda_status(e);
}

int pie_rms_norm(void* out, const void* x, const void* weight, long long rows, int dims, float eps, void* stream) {
  if (rows == 0) return PIE_OK;
  if (!out || !x) return PIE_ENULL;
  if (rows < 0 || dims <= 0) return PIE_EINVAL_SHAPE;
  return cuda_status(launch_rms_norm((uint16_t*)out, (const uint16_t*)x, (const uint16_t*)weight, rows, dims, eps,
                                     (cudaStream_t)stream));
}

int pie_rope(void* out, const void* x, long long n_batch, int L, int D, int dims, int traditional, float base,
             float scale, int offset, const float* freqs, void* stream) {
  if (n_batch == 0 || L == 0) return PIE_OK;
  if (!out || !x) return PIE_ENULL;
  if (n_batch < 0 || L < 0 || D <= 0 || dims <= 0 || dims > D || dims % 2) return PIE_EINVAL_SHAPE;
  if (!freqs && !(base > 0.f)) return PIE_EINVAL_SHAPE;
  return cuda_status(launch_rope((uint16_t*)out, (const uint16_t*)x, n_batch, L, D, dims, traditional, base, scale,
                                 offset, freqs, (cudaStream_t)stream));
}

int pie_rope_kv_append(void* q_out, const void* qkv, void* kcache, void* vcache, const pie_kv_layout* kv,
                       const int32_t* positions, const float* freqs, int B, int Hq, int Hkv, int D, void* stream) {
  if (B == 0) return PIE_OK;
  if (!q_out || !qkv || !kcache || !vcache || !positions || !freqs) return PIE_ENULL;
  if (B < 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || (D != 64 && D != 128)) return PIE_EINVAL_SHAPE;
  if (int s = check_kv(kv, D)) return s;
  return cuda_status(launch_rope_kv_append((uint16_t*)q_out, (const uint16_t*)qkv, (uint16_t*)kcache,
                                           (uint16_t*)vcache, to_kv(kv), positions, freqs, B, Hq, Hkv, D,
                                           (cudaStream_t)stream));
}

int pie_rope_heads(void* out, const void* x, int B, int H, int L, int D, long long stride_b, long long stride_h,
                   long long stride_l, int offset, const float* freqs, void* stream) {
  if (B == 0 || H == 0 || L == 0) return PIE_OK;
  if (!out || !x || !freqs) return PIE_ENULL;
  if (B < 0 || H < 0 || L < 0 || (D != 64 && D != 128) || B > 65535) return PIE_EINVAL_SHAPE;
  if (!aligned16(out) || !aligned16(x) || (stride_b | stride_h | stride_l) % 8) return PIE_EALIGN;
  return cuda_status(launch_rope_heads((uint16_t*)out, (const uint16_t*)x, B, H, L, D, stride_b, stride_h, stride_l, offset, freqs,
                                       (cudaStream_t)stream));
}

int pie_rope_kv_rows(void* q_out, void* kcache, void* vcache, const pie_kv_layout* kv, const pie_head_rows* q, const pie_head_rows* k,
                     const pie_head_rows* v, int32_t* positions_out, const float* freqs, int B, int Hq, int Hkv, int L, int D, int offset,
                     void* stream) {
  if (B == 0 || L == 0) return PIE_OK;
  if (!q_out || !kcache || !vcache || !q || !k || !v || !q->p || !k->p || !v->p || !freqs) return PIE_ENULL;
  if (B < 0 || Hq <= 0 || Hkv <= 0 || L < 0 || offset < 0 || (D != 64 && D != 128) || B > 65535 || Hq > 65535 - 2LL * Hkv) return PIE_EINVAL_SHAPE;
  if (int s = check_kv(kv, D)) return s;
  const RopeRows r = {(const uint16_t*)q->p, (const uint16_t*)k->p, (const uint16_t*)v->p, {q->stride_b, q->stride_h, q->stride_l},
                      {k->stride_b, k->stride_h, k->stride_l}, {v->stride_b, v->stride_h, v->stride_l}};
  return cuda_status(launch_rope_kv_rows((uint16_t*)q_out, positions_out, r, (uint16_t*)kcache, (uint16_t*)vcache, to_kv(kv), freqs, B, Hq, Hkv,
                                         L, D, offset, (cudaStream_t)stream));
}

int pie_kv_write_strided(void* kcache, void* vcache, const pie_kv_layout* kv, const void* k, long long k_stride_b,
                         long long k_stride_h, long long k_stride_l, const void* v, long long v_stride_b, long long v_stride_h,
                         long long v_stride_l, int B, int Hkv, int L, int D, int offset, void* stream) {
  if (B == 0 || L == 0) return PIE_OK;
  if (!kcache || !vcache || !k || !v) return PIE_ENULL;
  if (B < 0 || Hkv <= 0 || L < 0 || D <= 0 || offset < 0) return PIE_EINVAL_SHAPE;
  if (int s = check_kv(kv, D)) return s;
  const KvSrc ks = {k_stride_b, k_stride_h, k_stride_l}, vs = {v_stride_b, v_stride_h, v_stride_l};
  return cuda_status(launch_kv_write((uint16_t*)kcache, (uint16_t*)vcache, to_kv(kv), (const uint16_t*)k, (const uint16_t*)v, ks, vs,
                                     B, Hkv, L, D, offset, (cudaStream_t)stream));
}

int pie_kv_write(void* kcache, void* vcache, const pie_kv_layout* kv, const void* k, const void* v, int B, int Hkv,
                 int L, int D, int offset, void* stream) {
  const long long sl = D, sh = sl * L, sb = sh * Hkv;
  return pie_kv_write_strided(kcache, vcache, kv, k, sb, sh, sl, v, sb, sh, sl, B, Hkv, L, D, offset, stream);
}

size_t pie_decode_attn_workspace_bytes(int B, int Hq, int D, int nsplit) {
  if (B <= 0 || Hq <= 0 || D <= 0 || nsplit <= 0) return 0;
  const size_t cnt = (((size_t)B * Hq * 4) + 255) & ~(size_t)255;
  return cnt + (size_t)B * Hq * nsplit * (D + 2) * sizeof(float);
}

int pie_decode_attn_pick_splits(int B, int Hq, int Hkv, int max_context) {
  if (B <= 0 || Hq <= 0 || Hkv <= 0) return 1;
  const int n_rep = Hq / Hkv;
  long long ctas = (long long)B * Hkv, want = 2LL * num_sms();   // tensor-core kernel: one CTA per (sequence, kv head, split), 2 resident per SM (96 KB of stages)
  if (n_rep > 16) {
    ctas *= n_rep % 4 == 0 ? n_rep / 4 : (n_rep % 2 == 0 ? n_rep / 2 : n_rep);
    want *= 2;
  }
  // ONE wave of resident CTAs, never a wave and a fraction: measured on B200 (8B shapes, paged, us per layer at
  // 1 / 2 / 3 / 4 splits): bs32 ctx2048 (256 CTAs per split) 45 / 59 / 62 / 66; bs16 ctx4096 (128) 70 / 50 / 65 / 57;
  // bs8 ctx2048 (64), 2 / 4 / 5 / 8 splits: 27 / 23 / 29 / 24
  int ns = (int)(want / ctas);
  const int cap = (max_context + 63) / 64;  // >= 64 tokens (one stage) per split
  if (ns > cap) ns = cap;
  if (ns > 32) ns = 32;  // kFaMaxSplits (pie_fa.cu)
  return ns < 1 ? 1 : ns;
}

int pie_decode_attn_pick_splits_for(int B, int Hq, int Hkv, int D, int max_context) {
  const int ns = pie_decode_attn_pick_splits(B, Hq, Hkv, max_context);
  if (D != 64 || B <= 0 || Hq <= 0 || Hkv <= 0 || Hq / Hkv > 16) return ns;
  // Heads of 64: a CTA's stages are half the bytes and four fit an SM, which a wave of two leaves waiting for memory.  Up to four while a split has 128 tokens;
  // us, two / four: bs32 ctx2048 38.1 / 26.8, ctx6000 103.5 / 67.9, ctx500 13.1 / 11.8, bs16 ctx1000 14.7 / 11.8, bs8 ctx4000 22.9 / 17.5, ctx1066 9.9 / 8.4, bs5
  // ctx7002 23.0 / 18.2.  Not for a few more (bs4 ctx1300 9 / 10 splits 9.2 / 9.7), nor a first sum of splits below 384 (bs32 ctx256 8.3 / 8.9, ctx384 10.7 / 10.7, ctx450
  // 13.2 / 11.9).
  const int more = (int)std::min<long long>({4LL * num_sms() / ((long long)B * Hkv), max_context / 128, 32});   // (kFaMaxSplits)
  return (ns == 1 && max_context < 384) || more < ns + (ns + 3) / 4 ? ns : more;
}

int pie_decode_attn(void* out, const void* q, const void* kcache, const void* vcache, const pie_kv_layout* kv,
                    const int32_t* positions, int B, int Hq, int Hkv, int D, float scale, int nsplit,
                    void* workspace, size_t workspace_bytes, void* stream) {
  if (B == 0) return PIE_OK;
  if (!out || !q || !kcache || !vcache || !positions) return PIE_ENULL;
  if (B < 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return PIE_EINVAL_SHAPE;
  if (D != 64 && D != 128) return PIE_EUNSUPPORTED;
  if (int s = check_kv(kv, D)) return s;
  if (!aligned16(q) || !aligned16(kcache) || !aligned16(vcache)) return PIE_EALIGN;
  if (nsplit <= 0) nsplit = 1;
  if (nsplit > 1 && (!workspace || workspace_bytes < pie_decode_attn_workspace_bytes(B, Hq, D, nsplit)))
    return PIE_EWORKSPACE;
  return cuda_status(launch_decode_attn((uint16_t*)out, (const uint16_t*)q, (const uint16_t*)kcache,
                                        (const uint16_t*)vcache, to_kv(kv), positions, B, Hq, Hkv, D, scale, nsplit,
                                        (float*)workspace, (cudaStream_t)stream));
}

int pie_prefill_attn(void* out, const void* q, const void* kcache, const void* vcache, const pie_kv_layout* kv, int B,
                     int Hq, int Hkv, int L, int D, int offset, float scale, void* stream) {
  if (B == 0 || L == 0) return PIE_OK;
  if (!out || !q || !kcache || !vcache) return PIE_ENULL;
  if (B < 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || L < 0 || offset < 0) return PIE_EINVAL_SHAPE;
  if (D != 64 && D != 128) return PIE_EUNSUPPORTED;
  if (int s = check_kv(kv, D)) return s;
  return cuda_status(launch_prefill_attn((uint16_t*)out, (const uint16_t*)q, (const uint16_t*)kcache,
                                         (const uint16_t*)vcache, to_kv(kv), B, Hq, Hkv, L, D, offset, scale,
                                         (cudaStream_t)stream));
}

// 1: a pipeline wait of the prefill GEMM or of the prefill attention expired (the call's results are void); 0: none did
unsigned int pie_pipeline_error(void) { return qmm_pipeline_error() | fa_prefill_pipeline_error(); }
int pie_pipeline_error_clear(void) {
  if (int s = cuda_status(qmm_pipeline_clear())) return s;
  return cuda_status(fa_prefill_pipeline_clear());
}
int pie_pipeline_words(unsigned int* words, void* stream) {
  if (!words) return PIE_ENULL;
  if (int s = cuda_status(qmm_pipeline_post(words, (cudaStream_t)stream))) return s;
  return cuda_status(fa_prefill_pipeline_post(words + 1, (cudaStream_t)stream));
}

int pie_silu_mul(void* out, const void* gate, const void* up, long long n, void* stream) {
  if (n == 0) return PIE_OK;
  if (!out || !gate || !up) return PIE_ENULL;
  return cuda_status(launch_silu_mul((uint16_t*)out, (const uint16_t*)gate, (const uint16_t*)up, n, (cudaStream_t)stream));
}
int pie_add(void* out, const void* a, const void* b, long long n, void* stream) {
  if (n == 0) return PIE_OK;
  if (!out || !a || !b) return PIE_ENULL;
  return cuda_status(launch_add((uint16_t*)out, (const uint16_t*)a, (const uint16_t*)b, n, (cudaStream_t)stream));
}
int pie_argmax(int32_t* out_idx, const void* logits, int rows, int vocab, int32_t* positions_to_advance,
               int32_t* seq_out, int seq_ld, void* stream) {
  if (rows == 0) return PIE_OK;
  if (!out_idx || !logits) return PIE_ENULL;
  if (rows < 0 || vocab <= 0) return PIE_EINVAL_SHAPE;
  return cuda_status(launch_argmax(out_idx, (const uint16_t*)logits, rows, vocab, positions_to_advance, seq_out, seq_ld,
                                   (cudaStream_t)stream));
}

}  // extern "C"
