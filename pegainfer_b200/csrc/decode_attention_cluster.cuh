// Argument block of the cluster decode-attention kernel (decode_attention_cluster.cu), shared with the entry point
// in decode_attention.cu.
#pragma once
#include "common.cuh"

namespace pk {

// L2 prefetch span: the weight rows a FOLLOWING GEMV launch will stream.  The rows are cut into `slices` row ranges
// exactly as that GEMV's grid cuts them ([s*rows/slices, (s+1)*rows/slices)); the first `pf_rows` rows of every
// slice are requested, so every GEMV CTA finds the same share of its slice in L2.
struct PfSpan {
  const uint8_t* base;
  int rows, row_bytes, slices, pf_rows;
};
constexpr int kMaxPfSpans = 4;

struct ClusterAttnArgs {
  const bf16 *q, *k_new, *v_new;
  bf16* out;
  bf16* kv;
  int64_t k_off, v_off, stride_page;
  const int *page_indices, *page_indptr, *last_page_len, *positions;
  const int* request_indices;  // plain mode (k_new == nullptr): batch slot -> request, may be null (identity)
  const bf16 *qw, *kw, *cosc, *sinc;
  float eps, sm_scale_log2;
  int nq, nkv;
  int npf, pf_y;  // prefetch spans; extra cluster rows (blockIdx.y >= nkv) that only issue L2 prefetches
  PfSpan pf[kMaxPfSpans];
};
cudaError_t launch_decode_attention_cluster(const ClusterAttnArgs& a, int nkv, int bs, cudaStream_t stream);
// the default kernel (decode_attention_tma.cu): TMA page tiles + mma.sync, up to 16-CTA clusters.  Same argument block
// (prefetch spans ignored).  Returns a cudaError, or -2 when it cannot take the call.
int launch_decode_attention_tma(const ClusterAttnArgs& a, int nkv, int bs, cudaStream_t stream);
// decode_attention_flat.cu: many requests, equal runs of pages for every SM.  -2: not a call for it
int launch_decode_attention_flat(const ClusterAttnArgs& a, int nkv, int bs, float* partial, long places, int* counters, cudaStream_t stream);

// ---- a page of one kv head in shared memory, 128-byte swizzle, and what both TMA kernels do with it
constexpr int kDaHalf = 16 * 128;  // bytes of 64 columns of 16 tokens

__device__ __forceinline__ float da_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void da_ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void da_ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// A operand: rows 0-3 are the query heads, rows 8-15 are zero
__device__ __forceinline__ void da_mma(float (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}
// byte offset of 16-byte piece c (0..15) of row r of a K (V) tile: two halves with the 128-byte swizzle (piece ^= row & 7)
__device__ __forceinline__ uint32_t da_at(int r, int c) { return (uint32_t)((c >> 3) * kDaHalf + r * 128 + (((c & 7) ^ (r & 7)) << 4)); }

// norm + rotation of one head of 128, four entries to a lane (the arithmetic of qk_norm_rope.cu): the head's row, the norm's weights, this lane's cosines
// and sines
__device__ __forceinline__ void da_norm_rope(uint2 raw, uint2 wr, uint2 cr, uint2 sr, float eps, bf16* dst, int lane) {
  const float v[4] = {bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y)};
  float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / 128.f + eps);
  const float wv[4] = {bf16_lo(wr.x), bf16_hi(wr.x), bf16_lo(wr.y), bf16_hi(wr.y)};
  const float c[4] = {bf16_lo(cr.x), bf16_hi(cr.x), bf16_lo(cr.y), bf16_hi(cr.y)};
  const float s[4] = {bf16_lo(sr.x), bf16_hi(sr.x), bf16_lo(sr.y), bf16_hi(sr.y)};
  float o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float t = round_bf16(round_bf16(v[j] * inv) * wv[j]);
    const float other = __shfl_xor_sync(0xffffffffu, t, 16);
    o[j] = lane < 16 ? t * c[j] - other * s[j] : other * s[j] + t * c[j];
  }
  reinterpret_cast<uint2*>(dst)[lane] = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
}

}  // namespace pk
