// Per-head QK RMSNorm + NeoX RoPE, in place on Q and K.  Replaces
// csrc/prefill_attention.cu:12-159 of the reference, same rounding points:
//   normed = bf16(x * inv_rms);  t = bf16(f32(normed) * w);
//   lo' = bf16(lo*c - hi*s), hi' = bf16(lo*s + hi*c)  with bf16 cos/sin tables.
// Half a warp per (head, token): lane l of the half owns elements 8l..8l+7 (one 16-byte access); the RoPE partner (i, i+64) lives in lane l^8,
// exchanged with a shuffle -- no shared memory, no block barrier.  A warp takes HEADS heads of one token, so that the token's cos / sin rows and
// the weights are loaded once for all of them, and all its rows are on their way before the first is used.  HBM / L2-bound: 2 x 2 bytes an element.
#include "common.cuh"

namespace pk {

template <int HEADS>
__global__ void __launch_bounds__(128) qk_norm_rope_kernel(bf16* __restrict__ q, bf16* __restrict__ k, const bf16* __restrict__ qw,
                                                           const bf16* __restrict__ kw, const bf16* __restrict__ cosc, const bf16* __restrict__ sinc,
                                                           const int* __restrict__ positions, int start_pos, int nq, int nkv, int tokens, float eps,
                                                           bool vec) {
  constexpr int HD = 128, N = (HEADS + 1) / 2;
  const int lane = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1, heads = nq + nkv, groups = (heads + HEADS - 1) / HEADS;
  const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait();
  if (warp >= groups * tokens) return;
  const int token = warp / groups, head0 = (warp - token * groups) * HEADS;
  const int pos = positions ? __ldg(positions + token) : start_pos + token;
  auto row_of = [&](int head) { return head < nq ? q + ((size_t)token * nq + head) * HD : k + ((size_t)token * nkv + (head - nq)) * HD; };
  auto unpack = [](const uint4& u, float (&v)[8]) {
    v[0] = bf16_lo(u.x); v[1] = bf16_hi(u.x); v[2] = bf16_lo(u.y); v[3] = bf16_hi(u.y);
    v[4] = bf16_lo(u.z); v[5] = bf16_hi(u.z); v[6] = bf16_lo(u.w); v[7] = bf16_hi(u.w);
  };
  auto piece = [&](const bf16* p, int i) {  // 16 bytes; two halves where a pointer is only on an 8-byte boundary
    if (vec) return reinterpret_cast<const uint4*>(p)[i];
    const uint2 a = reinterpret_cast<const uint2*>(p)[2 * i], b = reinterpret_cast<const uint2*>(p)[2 * i + 1];
    return make_uint4(a.x, a.y, b.x, b.y);
  };
  uint4 raw[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 2 * i + half;
    raw[i] = 2 * i + half < HEADS && head < heads ? piece(row_of(head), lane) : make_uint4(0, 0, 0, 0);
  }
  // table layout [pos*128 + i] duplicated for i and i+64 (weight_loader.rs:210-244)
  float c[8], s[8], wq[8] = {}, wk[8] = {};
  unpack(piece(cosc + (size_t)pos * HD, lane & 7), c);
  unpack(piece(sinc + (size_t)pos * HD, lane & 7), s);
  if (nq > 0) unpack(piece(qw, lane), wq);  // a call without query (key) heads may come without their weights
  if (nkv > 0) unpack(piece(kw, lane), wk);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 2 * i + half;
    float v[8];
    unpack(raw[i], v);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = rsqrtf(ss / (float)HD + eps);
    float t[8], o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = round_bf16(round_bf16(v[j] * inv) * (head < nq ? wq[j] : wk[j]));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, t[j], 8);
      // lanes 0..7 hold "lo" (d < 64): lo*c - hi*s ; lanes 8..15 hold "hi": lo*s + hi*c
      o[j] = lane < 8 ? t[j] * c[j] - other * s[j] : other * s[j] + t[j] * c[j];
    }
    if (2 * i + half < HEADS && head < heads) {
      const uint4 r = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
      uint4* dst = reinterpret_cast<uint4*>(row_of(head)) + lane;
      if (vec) {
        *dst = r;
      } else {
        reinterpret_cast<uint2*>(dst)[0] = make_uint2(r.x, r.y);
        reinterpret_cast<uint2*>(dst)[1] = make_uint2(r.z, r.w);
      }
    }
  }
}

static void launch_qk(pk_bf16* q, pk_bf16* k, const pk_bf16* qw, const pk_bf16* kw,
                      const pk_bf16* cosc, const pk_bf16* sinc, const int* positions,
                      int start_pos, int nq, int nkv, int head_dim, int tokens, float eps,
                      pk_stream stream) {
  if (head_dim != 128 || tokens <= 0) return;  // HEAD_DIM is hard-coded 128 in the reference too
  const bool vec = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(qw) | reinterpret_cast<uintptr_t>(kw) |
                     reinterpret_cast<uintptr_t>(cosc) | reinterpret_cast<uintptr_t>(sinc)) & 15) == 0;
  // eight heads per warp once that still gives every SM a few warps; two where tokens are few
  auto go = [&](auto kern, int per) {
    const int warps = (nq + nkv + per - 1) / per * tokens;
    launch(kern, dim3((warps + 3) / 4), dim3(128), 0, stream, true, (bf16*)q, (bf16*)k, (const bf16*)qw, (const bf16*)kw, (const bf16*)cosc,
           (const bf16*)sinc, positions, start_pos, nq, nkv, tokens, eps, vec);
  };
  if ((long)tokens * (nq + nkv) >= 8L * 16 * sm_count()) go(qk_norm_rope_kernel<8>, 8);
  else go(qk_norm_rope_kernel<2>, 2);
}

}  // namespace pk

extern "C" {

void prefill_qk_norm_rope_only_cuda(pk_bf16* q_batch, pk_bf16* k_batch,
                                    const pk_bf16* q_norm_weight, const pk_bf16* k_norm_weight,
                                    const pk_bf16* cos_cache, const pk_bf16* sin_cache,
                                    int num_q_heads, int num_kv_heads, int head_dim, int seq_len,
                                    int start_pos, float rms_eps, pk_stream stream) {
  pk::launch_qk(q_batch, k_batch, q_norm_weight, k_norm_weight, cos_cache, sin_cache, nullptr,
                start_pos, num_q_heads, num_kv_heads, head_dim, seq_len, rms_eps, stream);
}

void qk_norm_rope_batched_decode_cuda(pk_bf16* q, pk_bf16* k, const pk_bf16* q_norm_weight,
                                      const pk_bf16* k_norm_weight, const pk_bf16* cos_cache,
                                      const pk_bf16* sin_cache, const int* positions,
                                      int num_q_heads, int num_kv_heads, int head_dim,
                                      int batch_size, float rms_eps, pk_stream stream) {
  pk::launch_qk(q, k, q_norm_weight, k_norm_weight, cos_cache, sin_cache, positions, 0,
                num_q_heads, num_kv_heads, head_dim, batch_size, rms_eps, stream);
}

}  // extern "C"
