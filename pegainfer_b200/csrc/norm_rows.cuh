// RMSNorm over many rows (norm.cu, qwen35_ops.cu): all pointers on 16-byte boundaries, dim a multiple of 8.
#pragma once
#include "common.cuh"

namespace pk {

// W warps of a CTA of eight per row, the row in registers, one barrier; all of a lane's pieces and the weights' are on their way before the first is used
// (with the weights read behind the sum, the compiler asked for them only there).  Four warps per row; eight, which share the latency of one row, where
// rows are few.  B200, us, rows x dim, a warp per row with the weights read behind the sum -> this: 1024 x 2560
// 4.3 -> 3.1, 2048 x 2560 4.8 -> 4.1, 3333 x 2560 8.7 -> 8.2, 325 x 4096 5.4 -> 2.1, 3001 x 4096 12.7 -> 9.8; residual sums (MODE 1) 2048 x 2560 6.5 -> 6.4,
// 3001 x 4096 16.9 -> 14.1.  One row per CTA from shared memory (norm.cu, longer rows) is as fast as this up to some 50 rows.
constexpr int kRowVecs = 16;  // 16-byte pieces per 32 lanes: rows of up to 4096
// MODE 0: rms_norm, 1: fused_add_rms_norm (norm.cu), 2: rms_norm with 1 + w (qwen35_ops.cu).
template <int MODE, int NV, int W>
__global__ void __launch_bounds__(256) rms_norm_rows_kernel(const bf16* __restrict__ x, bf16* __restrict__ hidden, const bf16* __restrict__ residual,
                                                            const bf16* __restrict__ w, bf16* __restrict__ out, int dim, int rows, float eps) {
  __shared__ float red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = dim >> 3, at = warp % W * 32 + lane;
  const int row = blockIdx.x * (8 / W) + warp / W;
  pdl_wait();
  const bool on = row < rows;
  const size_t base = (size_t)(on ? row : 0) * dim;
  const uint4 *in = reinterpret_cast<const uint4*>((MODE == 1 ? hidden : x) + base), none = make_uint4(0, 0, 0, 0);
  uint4 a[NV], b[NV], g[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) a[j] = at + 32 * W * j < nv ? in[at + 32 * W * j] : none;
  if constexpr (MODE == 1) {
#pragma unroll
    for (int j = 0; j < NV; ++j) b[j] = at + 32 * W * j < nv ? reinterpret_cast<const uint4*>(residual + base)[at + 32 * W * j] : none;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) g[j] = at + 32 * W * j < nv ? reinterpret_cast<const uint4*>(w)[at + 32 * W * j] : none;
  float v[NV][8], ss = 0.f;  // (MODE 1: the unrounded sums)
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const uint32_t aw[4] = {a[j].x, a[j].y, a[j].z, a[j].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[j][2 * e] = bf16_lo(aw[e]);
      v[j][2 * e + 1] = bf16_hi(aw[e]);
    }
    if constexpr (MODE == 1) {
      const uint32_t bw[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[j][2 * e] += bf16_lo(bw[e]);
        v[j][2 * e + 1] += bf16_hi(bw[e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(v[j][e], v[j][e], ss);
  }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < W; ++i) ss += red[warp / W * W + i];
  const float r = rsqrtf(ss / (float)dim + eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = at + 32 * W * j;
    if (i >= nv || !on) continue;
    if constexpr (MODE == 1)
      reinterpret_cast<uint4*>(hidden + base)[i] = make_uint4(pack_bf16(v[j][0], v[j][1]), pack_bf16(v[j][2], v[j][3]), pack_bf16(v[j][4], v[j][5]), pack_bf16(v[j][6], v[j][7]));
    constexpr float one = MODE == 2 ? 1.f : 0.f;
    const uint32_t gw[4] = {g[j].x, g[j].y, g[j].z, g[j].w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = pack_bf16(v[j][2 * e] * r * (one + bf16_lo(gw[e])), v[j][2 * e + 1] * r * (one + bf16_hi(gw[e])));
    reinterpret_cast<uint4*>(out + base)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

inline bool rms_rows_fit(int dim) { return dim % 8 == 0 && dim <= 256 * kRowVecs; }

template <int MODE>
void launch_rms_rows(const bf16* x, bf16* hidden, const bf16* residual, const bf16* w, bf16* out, int dim, int rows, float eps, cudaStream_t stream) {
  const int nv = (dim + 255) / 256;
  auto go = [&](auto kern, int warps) {
    const int per = 8 / warps;
    launch(kern, dim3((rows + per - 1) / per), dim3(256), 0, stream, true, x, hidden, residual, w, out, dim, rows, eps);
  };
  if (rows < 2 * sm_count()) {
    if (nv <= 8) go(rms_norm_rows_kernel<MODE, 1, 8>, 8);
    else go(rms_norm_rows_kernel<MODE, 2, 8>, 8);
  } else {
    if (nv <= 4) go(rms_norm_rows_kernel<MODE, 1, 4>, 4);
    else if (nv <= 12) go(rms_norm_rows_kernel<MODE, 3, 4>, 4);
    else go(rms_norm_rows_kernel<MODE, 4, 4>, 4);
  }
}

}  // namespace pk
