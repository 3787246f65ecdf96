// Append K/V token rows into the page-first KV pool.  Replaces csrc/paged_attention.cu:274-311
// (FlashInfer page.cuh:259-284 AppendPagedKVCache) of the reference.
//
// Pool layout (pegainfer-core/src/kv_pool.rs:66-75): [page][layer][K | V][slot 0..15][kv head][128].
// Token i goes to entry e = page_indptr[batch_indices[i]] * page_size + positions[i]:
// page = page_indices[e / page_size], slot = e % page_size.  Pure 16-byte copies.
#include "common.cuh"

namespace pk {

// A warp per token, up to 128 16-byte pieces of K and of V at a time: the rows are on their way while the token's place is looked up (three loads that wait
// for one another), which is done once for a token.  A thread per piece looked it up for each, behind three divisions of 64 bits, and asked for the row after
// that.  8 heads of 128, B200, us in a train: 3333 tokens 5.6 -> 4.4, 2048 4.5 -> 3.5, 24 2.1 2.1.
constexpr int kScThreads = 128, kScPieces = 4;
__global__ void __launch_bounds__(kScThreads) paged_kv_scatter_kernel(bf16* __restrict__ kv, int64_t k_off, int64_t v_off, const int* __restrict__ page_indices,
                                                                      const int* __restrict__ page_indptr, const bf16* __restrict__ src_k,
                                                                      const bf16* __restrict__ src_v, const int* __restrict__ batch_indices,
                                                                      const int* __restrict__ positions, int nnz, int nkv, int hd, int page_size,
                                                                      int64_t stride_page, int64_t src_stride_n, int64_t src_stride_h) {
  pdl_wait();
  const int lane = threadIdx.x & 31, per_head = hd >> 3, pieces = nkv * per_head;
  for (int i = blockIdx.x * (kScThreads / 32) + (threadIdx.x >> 5); i < nnz; i += gridDim.x * (kScThreads / 32)) {
    const int b = __ldg(batch_indices + i), pos = __ldg(positions + i);
    const int64_t src0 = (int64_t)i * src_stride_n;
    int64_t dst0 = -1;
    for (int p0 = lane; p0 < pieces; p0 += 32 * kScPieces) {
      uint4 k[kScPieces], v[kScPieces];
#pragma unroll
      for (int j = 0; j < kScPieces; ++j) {
        const int p = p0 + 32 * j;
        if (p >= pieces) break;
        const int64_t src = src0 + (int64_t)(p / per_head) * src_stride_h + p % per_head * 8;
        k[j] = *reinterpret_cast<const uint4*>(src_k + src);
        v[j] = *reinterpret_cast<const uint4*>(src_v + src);
      }
      if (dst0 < 0) {
        const int entry = __ldg(page_indptr + b) * page_size + pos;
        dst0 = (int64_t)__ldg(page_indices + entry / page_size) * stride_page + (int64_t)(entry % page_size) * nkv * hd;
      }
#pragma unroll
      for (int j = 0; j < kScPieces; ++j) {
        const int p = p0 + 32 * j;
        if (p >= pieces) break;
        *reinterpret_cast<uint4*>(kv + k_off + dst0 + (int64_t)p * 8) = k[j];
        *reinterpret_cast<uint4*>(kv + v_off + dst0 + (int64_t)p * 8) = v[j];
      }
    }
  }
}

}  // namespace pk

extern "C" int paged_kv_scatter_cuda(const pk_bf16* kv_data, int64_t k_offset_elems,
                                     int64_t v_offset_elems, const int* page_indices,
                                     const int* page_indptr, const int* last_page_len_d,
                                     const pk_bf16* src_k, const pk_bf16* src_v,
                                     const int* batch_indices, const int* positions, int nnz,
                                     int num_kv_heads, int head_dim, int page_size,
                                     int64_t stride_page, int64_t src_stride_n,
                                     int64_t src_stride_h, pk_stream stream) {
  (void)last_page_len_d;
  if (nnz <= 0) return 0;
  if (head_dim % 8 != 0 || src_stride_n % 8 != 0 || src_stride_h % 8 != 0 || stride_page % 8 != 0)
    return (int)cudaErrorInvalidValue;
  const int64_t cap = (int64_t)pk::sm_count() * 16;
  int64_t grid = ((int64_t)nnz * 32 + pk::kScThreads - 1) / pk::kScThreads;
  if (grid > cap) grid = cap;
  pk::launch(pk::paged_kv_scatter_kernel, dim3((unsigned)grid), dim3(pk::kScThreads), 0, stream, true,
             (pk::bf16*)kv_data, k_offset_elems, v_offset_elems, page_indices, page_indptr,
             (const pk::bf16*)src_k, (const pk::bf16*)src_v, batch_indices, positions, nnz,
             num_kv_heads, head_dim, page_size, stride_page, src_stride_n, src_stride_h);
  return (int)cudaGetLastError();
}
