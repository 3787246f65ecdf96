// RMSNorm over many rows (norm.cu, qwen35_ops.cu): all pointers on 16-byte boundaries, dim a multiple of 8.
#pragma once
#include "common.cuh"

namespace pk {

// Many rows: a warp per row, the row in registers, no barrier.  A CTA per row spends most of its time on two barriers and on the weights, which it
// asks for only after them; here a lane has all its pieces and the weights' on their way at once. 
constexpr int kRowVecs = 16;  // 16-byte pieces per lane: rows of up to 4096
// MODE 0: rms_norm, 1: fused_add_rms_norm (norm.cu), 2: rms_norm with 1 + w (qwen35_ops.cu).
template <int MODE, int NV>
__global__ void __launch_bounds__(128) rms_norm_rows_kernel(const bf16* __restrict__ x, bf16* __restrict__ hidden, const bf16* __restrict__ residual,
                                                            const bf16* __restrict__ w, bf16* __restrict__ out, int dim, int rows, float eps) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, nv = dim >> 3;
  pdl_wait();
  if (row >= rows) return;
  const size_t base = (size_t)row * dim;
  const uint4* in = reinterpret_cast<const uint4*>((MODE == 1 ? hidden : x) + base);
  uint4 a[NV];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) a[j] = lane + 32 * j < nv ? in[lane + 32 * j] : make_uint4(0, 0, 0, 0);
  if constexpr (MODE == 1) {  // the unrounded sums stay in registers
    float v[NV][8];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint4 r = lane + 32 * j < nv ? reinterpret_cast<const uint4*>(residual + base)[lane + 32 * j] : make_uint4(0, 0, 0, 0);
      v[j][0] = bf16_lo(a[j].x) + bf16_lo(r.x); v[j][1] = bf16_hi(a[j].x) + bf16_hi(r.x);
      v[j][2] = bf16_lo(a[j].y) + bf16_lo(r.y); v[j][3] = bf16_hi(a[j].y) + bf16_hi(r.y);
      v[j][4] = bf16_lo(a[j].z) + bf16_lo(r.z); v[j][5] = bf16_hi(a[j].z) + bf16_hi(r.z);
      v[j][6] = bf16_lo(a[j].w) + bf16_lo(r.w); v[j][7] = bf16_hi(a[j].w) + bf16_hi(r.w);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(v[j][e], v[j][e], ss);
    }
    const float r = rsqrtf(warp_sum(ss) / (float)dim + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i >= nv) continue;
      const uint4 g = reinterpret_cast<const uint4*>(w)[i];
      reinterpret_cast<uint4*>(hidden + base)[i] = make_uint4(pack_bf16(v[j][0], v[j][1]), pack_bf16(v[j][2], v[j][3]), pack_bf16(v[j][4], v[j][5]), pack_bf16(v[j][6], v[j][7]));
      reinterpret_cast<uint4*>(out + base)[i] =
          make_uint4(pack_bf16(v[j][0] * r * bf16_lo(g.x), v[j][1] * r * bf16_hi(g.x)), pack_bf16(v[j][2] * r * bf16_lo(g.y), v[j][3] * r * bf16_hi(g.y)),
                     pack_bf16(v[j][4] * r * bf16_lo(g.z), v[j][5] * r * bf16_hi(g.z)), pack_bf16(v[j][6] * r * bf16_lo(g.w), v[j][7] * r * bf16_hi(g.w)));
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const float v[8] = {bf16_lo(a[j].x), bf16_hi(a[j].x), bf16_lo(a[j].y), bf16_hi(a[j].y), bf16_lo(a[j].z), bf16_hi(a[j].z), bf16_lo(a[j].w), bf16_hi(a[j].w)};
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(v[e], v[e], ss);
    }
    const float r = rsqrtf(warp_sum(ss) / (float)dim + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i >= nv) continue;
      const uint4 g = reinterpret_cast<const uint4*>(w)[i];
      constexpr float one = MODE == 2 ? 1.f : 0.f;
      reinterpret_cast<uint4*>(out + base)[i] =
          make_uint4(pack_bf16(bf16_lo(a[j].x) * r * (one + bf16_lo(g.x)), bf16_hi(a[j].x) * r * (one + bf16_hi(g.x))),
                     pack_bf16(bf16_lo(a[j].y) * r * (one + bf16_lo(g.y)), bf16_hi(a[j].y) * r * (one + bf16_hi(g.y))),
                     pack_bf16(bf16_lo(a[j].z) * r * (one + bf16_lo(g.z)), bf16_hi(a[j].z) * r * (one + bf16_hi(g.z))),
                     pack_bf16(bf16_lo(a[j].w) * r * (one + bf16_lo(g.w)), bf16_hi(a[j].w) * r * (one + bf16_hi(g.w))));
    }
  }
}

// From about two rows per SM on the rows themselves fill the GPU and a warp takes one; fewer rows keep a CTA each, whose threads share the latency
// of one row.
inline bool rms_rows_fit(int dim, int rows) { return dim % 8 == 0 && dim <= 256 * kRowVecs && rows >= 2 * sm_count(); }

template <int MODE>
void launch_rms_rows(const bf16* x, bf16* hidden, const bf16* residual, const bf16* w, bf16* out, int dim, int rows, float eps, cudaStream_t stream) {
  const int nv = (dim + 255) / 256;
  auto go = [&](auto kern) { launch(kern, dim3((rows + 3) / 4), dim3(128), 0, stream, true, x, hidden, residual, w, out, dim, rows, eps); };
  if (nv <= 4) go(rms_norm_rows_kernel<MODE, 4>);
  else if (nv <= 10) go(rms_norm_rows_kernel<MODE, 10>);
  else go(rms_norm_rows_kernel<MODE, kRowVecs>);
}

}  // namespace pk
