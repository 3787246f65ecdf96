// Per-head QK RMSNorm + NeoX RoPE, in place on Q and K.  Replaces
// csrc/prefill_attention.cu:12-159 of the reference, same rounding points:
//   normed = bf16(x * inv_rms);  t = bf16(f32(normed) * w);
//   lo' = bf16(lo*c - hi*s), hi' = bf16(lo*s + hi*c)  with bf16 cos/sin tables.
// Half a warp per (head, token): lane l of the half owns the partners 4l..4l+3 and 64+4l..64+4l+3 (two 8-byte accesses, whole lines for the half), so that
// the rotation needs no exchange.  A warp takes HEADS heads of one token, so that the token's cos / sin rows and the weights are loaded once for all of them,
// and all its rows are on their way before the first is used.  bf16(normed * w) is one packed bf16 multiply (a product of two bf16 is exact in fp32, so its
// one rounding is the same); the products of the rotation are exact in fp32, too.
// Bound by issue slots, then HBM / L2 (2 x 2 bytes an element).  32 + 8 heads, B200, us, 3333 / 2048 / 1024 tokens (68 / 42 / 21 MB): 19.6 11.8 6.7 with a
// 16-byte piece per lane, the partner fetched by shuffles and all arithmetic in fp32, 15.5 9.5 5.6 like this.
#include "common.cuh"

namespace pk {

template <int HEADS>
__global__ void __launch_bounds__(128) qk_norm_rope_kernel(bf16* __restrict__ q, bf16* __restrict__ k, const bf16* __restrict__ qw,
                                                           const bf16* __restrict__ kw, const bf16* __restrict__ cosc, const bf16* __restrict__ sinc,
                                                           const int* __restrict__ positions, int start_pos, int nq, int nkv, int tokens, float eps) {
  constexpr int HD = 128, N = (HEADS + 1) / 2;
  const int lane = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1, heads = nq + nkv, groups = (heads + HEADS - 1) / HEADS;
  const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait();
  if (warp >= groups * tokens) return;
  const int token = warp / groups, head0 = (warp - token * groups) * HEADS;
  const int pos = positions ? __ldg(positions + token) : start_pos + token;
  auto row_of = [&](int head) {
    return reinterpret_cast<uint2*>(head < nq ? q + ((size_t)token * nq + head) * HD : k + ((size_t)token * nkv + (head - nq)) * HD) + lane;
  };
  auto piece = [&](const bf16* p, int half_row) { return reinterpret_cast<const uint2*>(p)[half_row * 16 + lane]; };
  uint2 raw[N][2];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 2 * i + half;
    const bool on = 2 * i + half < HEADS && head < heads;
    raw[i][0] = on ? row_of(head)[0] : make_uint2(0, 0);
    raw[i][1] = on ? row_of(head)[16] : make_uint2(0, 0);
  }
  // table layout [pos*128 + i] duplicated for i and i+64 (weight_loader.rs:210-244)
  const uint2 c2 = piece(cosc + (size_t)pos * HD, 0), s2 = piece(sinc + (size_t)pos * HD, 0), none = make_uint2(0, 0);
  uint2 wq[2] = {none, none}, wk[2] = {none, none};  // a call without query (key) heads may come without their weights
  if (nq > 0) wq[0] = piece(qw, 0), wq[1] = piece(qw, 1);
  if (nkv > 0) wk[0] = piece(kw, 0), wk[1] = piece(kw, 1);
  const float c[4] = {bf16_lo(c2.x), bf16_hi(c2.x), bf16_lo(c2.y), bf16_hi(c2.y)}, s[4] = {bf16_lo(s2.x), bf16_hi(s2.x), bf16_lo(s2.y), bf16_hi(s2.y)};
  auto mul2 = [](uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmul2(reinterpret_cast<const __nv_bfloat162&>(a), reinterpret_cast<const __nv_bfloat162&>(b));
    return reinterpret_cast<const uint32_t&>(r);
  };
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 2 * i + half;
    float v[2][4], ss = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[h][0] = bf16_lo(raw[i][h].x), v[h][1] = bf16_hi(raw[i][h].x), v[h][2] = bf16_lo(raw[i][h].y), v[h][3] = bf16_hi(raw[i][h].y);
#pragma unroll
      for (int e = 0; e < 4; ++e) ss = fmaf(v[h][e], v[h][e], ss);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = rsqrtf(ss / (float)HD + eps);
    float t[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint2 w = head < nq ? wq[h] : wk[h];
      const uint32_t a = mul2(pack_bf16(v[h][0] * inv, v[h][1] * inv), w.x), b = mul2(pack_bf16(v[h][2] * inv, v[h][3] * inv), w.y);
      t[h][0] = bf16_lo(a), t[h][1] = bf16_hi(a), t[h][2] = bf16_lo(b), t[h][3] = bf16_hi(b);
    }
    if (2 * i + half < HEADS && head < heads) {
      float o[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[0][e] = t[0][e] * c[e] - t[1][e] * s[e];
        o[1][e] = t[0][e] * s[e] + t[1][e] * c[e];
      }
      uint2* dst = row_of(head);
      dst[0] = make_uint2(pack_bf16(o[0][0], o[0][1]), pack_bf16(o[0][2], o[0][3]));
      dst[16] = make_uint2(pack_bf16(o[1][0], o[1][1]), pack_bf16(o[1][2], o[1][3]));
    }
  }
}

static void launch_qk(pk_bf16* q, pk_bf16* k, const pk_bf16* qw, const pk_bf16* kw,
                      const pk_bf16* cosc, const pk_bf16* sinc, const int* positions,
                      int start_pos, int nq, int nkv, int head_dim, int tokens, float eps,
                      pk_stream stream) {
  if (head_dim != 128 || tokens <= 0) return;  // HEAD_DIM is hard-coded 128 in the reference too
  // eight heads per warp once that still gives every SM a few warps; two where tokens are few
  auto go = [&](auto kern, int per) {
    const int warps = (nq + nkv + per - 1) / per * tokens;
    launch(kern, dim3((warps + 3) / 4), dim3(128), 0, stream, true, (bf16*)q, (bf16*)k, (const bf16*)qw, (const bf16*)kw, (const bf16*)cosc,
           (const bf16*)sinc, positions, start_pos, nq, nkv, tokens, eps);
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
