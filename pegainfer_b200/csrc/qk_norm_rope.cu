// Per-head QK RMSNorm + NeoX RoPE, in place on Q and K.  Replaces
// csrc/prefill_attention.cu:12-159 of the reference, same rounding points:
//   normed = bf16(x * inv_rms);  t = bf16(f32(normed) * w);
//   lo' = bf16(lo*c - hi*s), hi' = bf16(lo*s + hi*c)  with bf16 cos/sin tables.
// A quarter warp per (head, token): lane l of the quarter owns the partners 8l..8l+7 and 64+8l..64+8l+7 (two 16-byte accesses, whole lines for the quarter),
// so that the rotation needs no exchange.  A warp takes HEADS heads of one token, so that the token's cos / sin rows and the weights are loaded once for all of
// them, and all its rows are on their way before the first is used.  bf16(normed * w) is one packed bf16 multiply (a product of two bf16 is exact in fp32, so
// its one rounding is the same); the products of the rotation are exact in fp32, too.  The squares are added eight to a chain, then the halves of the head, then
// by distance 4, 2, 1 of the chains: the order of the sixteen lanes that had 16 bytes each before, and their bits.
// Bound by issue slots, then HBM / L2 (2 x 2 bytes an element).  32 + 8 heads, B200, us, 3333 / 2048 / 1024 tokens (68 / 42 / 21 MB): 20.2 11.0 6.4 with 16
// bytes per lane, the partner fetched by shuffles and all arithmetic in fp32, 15.3 7.1 4.6 like this; half a warp with two 8-byte pieces per lane 15.6 8.5 5.3
// (and another order of the squares).
#include "common.cuh"

namespace pk {

template <int HEADS>
__global__ void __launch_bounds__(128, 7) qk_norm_rope_kernel(bf16* __restrict__ q, bf16* __restrict__ k, const bf16* __restrict__ qw,
                                                              const bf16* __restrict__ kw, const bf16* __restrict__ cosc, const bf16* __restrict__ sinc,
                                                              const int* __restrict__ positions, int start_pos, int nq, int nkv, int tokens, float eps,
                                                              bool vec) {
  constexpr int HD = 128, N = HEADS / 4;
  const int lane = threadIdx.x & 7, quarter = (threadIdx.x >> 3) & 3, heads = nq + nkv, groups = (heads + HEADS - 1) / HEADS;
  const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait();
  if (warp >= groups * tokens) return;
  const int token = warp / groups, head0 = (warp - token * groups) * HEADS + quarter;
  const int pos = positions ? __ldg(positions + token) : start_pos + token;
  auto row_of = [&](int head) { return head < nq ? q + ((size_t)token * nq + head) * HD : k + ((size_t)token * nkv + (head - nq)) * HD; };
  auto unpack = [](const uint4& u, float (&v)[8]) {
    v[0] = bf16_lo(u.x); v[1] = bf16_hi(u.x); v[2] = bf16_lo(u.y); v[3] = bf16_hi(u.y);
    v[4] = bf16_lo(u.z); v[5] = bf16_hi(u.z); v[6] = bf16_lo(u.w); v[7] = bf16_hi(u.w);
  };
  auto piece = [&](const bf16* p, int half) {  // 16 bytes; two halves where a pointer is only on an 8-byte boundary
    const uint2* at = reinterpret_cast<const uint2*>(p) + half * 16 + 2 * lane;
    if (vec) return *reinterpret_cast<const uint4*>(at);
    const uint2 a = at[0], b = at[1];
    return make_uint4(a.x, a.y, b.x, b.y);
  };
  const uint4 none = make_uint4(0, 0, 0, 0);
  uint4 raw[N][2];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 4 * i;
#pragma unroll
    for (int h = 0; h < 2; ++h) raw[i][h] = head < heads ? piece(row_of(head), h) : none;
  }
  // table layout [pos*128 + i] duplicated for i and i+64 (weight_loader.rs:210-244)
  float c[8], s[8];
  unpack(piece(cosc + (size_t)pos * HD, 0), c);
  unpack(piece(sinc + (size_t)pos * HD, 0), s);
  uint4 wq[2] = {none, none}, wk[2] = {none, none};  // a call without query (key) heads may come without their weights
  if (nq > 0) wq[0] = piece(qw, 0), wq[1] = piece(qw, 1);
  if (nkv > 0) wk[0] = piece(kw, 0), wk[1] = piece(kw, 1);
  auto mul2 = [](uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmul2(reinterpret_cast<const __nv_bfloat162&>(a), reinterpret_cast<const __nv_bfloat162&>(b));
    return reinterpret_cast<const uint32_t&>(r);
  };
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int head = head0 + 4 * i;
    float t[2][8], ss[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unpack(raw[i][h], t[h]);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss[h] = fmaf(t[h][e], t[h][e], ss[h]);
    }
    float sum = ss[0] + ss[1];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = rsqrtf(sum / (float)HD + eps);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 w = head < nq ? wq[h] : wk[h];
      unpack(make_uint4(mul2(pack_bf16(t[h][0] * inv, t[h][1] * inv), w.x), mul2(pack_bf16(t[h][2] * inv, t[h][3] * inv), w.y),
                        mul2(pack_bf16(t[h][4] * inv, t[h][5] * inv), w.z), mul2(pack_bf16(t[h][6] * inv, t[h][7] * inv), w.w)),
             t[h]);
    }
    if (head < heads) {
      float o[2][8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        o[0][e] = t[0][e] * c[e] - t[1][e] * s[e];
        o[1][e] = t[0][e] * s[e] + t[1][e] * c[e];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 r = make_uint4(pack_bf16(o[h][0], o[h][1]), pack_bf16(o[h][2], o[h][3]), pack_bf16(o[h][4], o[h][5]), pack_bf16(o[h][6], o[h][7]));
        uint2* dst = reinterpret_cast<uint2*>(row_of(head)) + h * 16 + 2 * lane;
        if (vec) {
          *reinterpret_cast<uint4*>(dst) = r;
        } else {
          dst[0] = make_uint2(r.x, r.y);
          dst[1] = make_uint2(r.z, r.w);
        }
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
  // eight heads per warp once that still gives every SM a few warps; four where tokens are few (1 / 128 / 512 tokens: 1.6 2.0 2.8 us with eight, 1.3 1.8 3.0 with four)
  auto go = [&](auto kern, int per) {
    const int warps = (nq + nkv + per - 1) / per * tokens;
    launch(kern, dim3((warps + 3) / 4), dim3(128), 0, stream, true, (bf16*)q, (bf16*)k, (const bf16*)qw, (const bf16*)kw, (const bf16*)cosc,
           (const bf16*)sinc, positions, start_pos, nq, nkv, tokens, eps, vec);
  };
  if ((long)tokens * (nq + nkv) >= 8L * 16 * sm_count()) go(qk_norm_rope_kernel<8>, 8);
  else go(qk_norm_rope_kernel<4>, 4);
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
