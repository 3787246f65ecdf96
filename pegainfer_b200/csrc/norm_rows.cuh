// RMSNorm over many rows (norm.cu, qwen35_ops.cu): all pointers on 16-byte boundaries, dim a multiple of 8.
#pragma once
#include "common.cuh"

namespace pk {

// A row in registers, 16-byte pieces; all of a lane's pieces and the weights' are on their way before the first is used.  The squares are added in the order of
// the kernels that these took the place of, so a row has the same bits as there:
//   few rows    norm.cu's (a piece per thread, warps by exchange, then the warps), a CTA of 256 per row
//   many rows   a warp's per row (lane l: pieces l, l + 32, .. one after the other); W warps share a row and hand the lanes' chains on, which costs a barrier each
// B200, us, rows x dim, each row's pieces asked for at once by one warp and the weights behind the sum (few rows: norm.cu's kernel) -> this, MODE 0 / MODE 1:
//   1 x 2560    1.65 1.73 -> 1.22 1.33        48 x 4096  1.91 2.04 -> 1.38 1.58       295 x 4096  2.50 2.75 -> 1.78 2.16
//   512 x 2560  3.70 4.18 -> 1.86 2.37      1024 x 2560  4.06 5.12 -> 2.36 3.29      2048 x 2560  6.26 10.4 -> 3.86 7.73      3001 x 2560  10.2 15.3 -> 6.47 10.8
//   512 x 4096  5.28 6.09 -> 2.30 3.17      1024 x 4096  5.82 10.2 -> 2.88 5.48      2048 x 4096  14.2 20.2 -> 7.15 11.7      3001 x 4096  16.2 24.7 -> 9.43 16.2
//   512 x 1024  2.14 2.35 -> 1.32 1.60      3001 x 1024  2.81 3.73 -> 2.15 3.16
// Two warps a row of 4096 take 10.1 and 16.4 (3001 rows), four a row of 2560 6.82 and 10.8; blocks of 256 threads 0.1 to 1 more.  Sums added warp by warp, in
// another order, save 0.1 of few rows and 0.1 to 0.3 of 300 to 500.
constexpr int kRowVecs = 16;  // 16-byte pieces per 32 lanes: rows of up to 4096

// asked for where it stands (the compiler moved plain loads of the weights behind the few-row kernel's sums: 0.1 us a call)
__device__ __forceinline__ uint4 ld_in_place(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// pieces at, at + step, .. below nv of a row and of the weights; MODE 1: v = the unrounded sums
template <int MODE, int NV, bool IN_PLACE>
__device__ __forceinline__ void rms_load(const uint4* in, const uint4* residual, const uint4* w, int at, int step, int nv, float (&v)[NV][8], uint4 (&g)[NV]) {
  auto ld = [](const uint4* p) { return IN_PLACE ? ld_in_place(p) : *p; };
  const uint4 none = make_uint4(0, 0, 0, 0);
  uint4 a[NV], b[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) a[j] = at + step * j < nv ? ld(in + at + step * j) : none;
  if constexpr (MODE == 1) {
#pragma unroll
    for (int j = 0; j < NV; ++j) b[j] = at + step * j < nv ? ld(residual + at + step * j) : none;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) g[j] = at + step * j < nv ? ld(w + at + step * j) : none;
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
  }
}
template <int MODE, int NV>
__device__ __forceinline__ void rms_store(uint4* hidden, uint4* out, int at, int step, int nv, const float (&v)[NV][8], const uint4 (&g)[NV], float r) {
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = at + step * j;
    if (i >= nv) continue;
    if constexpr (MODE == 1)
      hidden[i] = make_uint4(pack_bf16(v[j][0], v[j][1]), pack_bf16(v[j][2], v[j][3]), pack_bf16(v[j][4], v[j][5]), pack_bf16(v[j][6], v[j][7]));
    constexpr float one = MODE == 2 ? 1.f : 0.f;
    const uint32_t gw[4] = {g[j].x, g[j].y, g[j].z, g[j].w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = pack_bf16(v[j][2 * e] * r * (one + bf16_lo(gw[e])), v[j][2 * e + 1] * r * (one + bf16_hi(gw[e])));
    out[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// MODE 0: rms_norm, 1: fused_add_rms_norm (norm.cu), 2: rms_norm with 1 + w (qwen35_ops.cu).
template <int MODE, int NV>
__global__ void __launch_bounds__(256) rms_norm_few_kernel(const bf16* __restrict__ x, bf16* __restrict__ hidden, const bf16* __restrict__ residual,
                                                           const bf16* __restrict__ w, bf16* __restrict__ out, int dim, float eps) {
  __shared__ float4 red[2 * NV];  // the sums of the warps' pieces
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = dim >> 3;
  pdl_wait();
  const size_t base = (size_t)blockIdx.x * dim;
  float v[NV][8], ss[NV];
  uint4 g[NV];
  rms_load<MODE, NV, true>(reinterpret_cast<const uint4*>((MODE == 1 ? hidden : x) + base), reinterpret_cast<const uint4*>(residual + base),
                           reinterpret_cast<const uint4*>(w), threadIdx.x, 256, nv, v, g);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    ss[j] = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss[j] = fmaf(v[j][e], v[j][e], ss[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < NV; ++j) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j) reinterpret_cast<float*>(red)[8 * j + warp] = ss[j];
  }
  __syncthreads();
  float4 t0 = red[0], t1 = red[1];  // as block_sum adds them
  if constexpr (NV == 2) {
    t0.x += red[2].x; t0.y += red[2].y; t0.z += red[2].z; t0.w += red[2].w;
    t1.x += red[3].x; t1.y += red[3].y; t1.z += red[3].z; t1.w += red[3].w;
  }
  const float sum = ((t0.x + t1.x) + (t0.z + t1.z)) + ((t0.y + t1.y) + (t0.w + t1.w));
  rms_store<MODE, NV>(reinterpret_cast<uint4*>(hidden + base), reinterpret_cast<uint4*>(out + base), threadIdx.x, 256, nv, v, g, rsqrtf(sum / (float)dim + eps));
}

template <int MODE, int NV, int W>
__global__ void __launch_bounds__(128) rms_norm_rows_kernel(const bf16* __restrict__ x, bf16* __restrict__ hidden, const bf16* __restrict__ residual,
                                                            const bf16* __restrict__ w, bf16* __restrict__ out, int dim, int rows, float eps) {
  __shared__ float chain[4 / W][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = warp % W, at = part * NV * 32 + lane, mine = warp / W;
  const int row = blockIdx.x * (4 / W) + mine;
  pdl_wait();
  const int nv = row < rows ? dim >> 3 : 0;  // (nothing is read or written behind the last row)
  const size_t base = (size_t)row * dim;
  float v[NV][8], ss = 0.f;
  uint4 g[NV];
  rms_load<MODE, NV, false>(reinterpret_cast<const uint4*>((MODE == 1 ? hidden : x) + base), reinterpret_cast<const uint4*>(residual + base),
                            reinterpret_cast<const uint4*>(w), at, 32, nv, v, g);
#pragma unroll
  for (int s = 0; s < W; ++s) {
    if (part == s) {
      if (s > 0) ss = chain[mine][lane];
#pragma unroll
      for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(v[j][e], v[j][e], ss);
      if (W > 1) chain[mine][lane] = ss;
    }
    if (W > 1) __syncthreads();
  }
  if (W > 1) ss = chain[mine][lane];
  ss = warp_sum(ss);
  rms_store<MODE, NV>(reinterpret_cast<uint4*>(hidden + base), reinterpret_cast<uint4*>(out + base), at, 32, nv, v, g, rsqrtf(ss / (float)dim + eps));
}

inline bool rms_rows_fit(int dim) { return dim % 8 == 0 && dim <= 256 * kRowVecs; }

template <int MODE>
void launch_rms_rows(const bf16* x, bf16* hidden, const bf16* residual, const bf16* w, bf16* out, int dim, int rows, float eps, cudaStream_t stream) {
  const int nv = (dim + 255) / 256;
  // (fewer than two rows to an SM: a CTA's threads share the latency of one)
  if (rows < 2 * sm_count()) {
    auto few = [&](auto kern) { launch(kern, dim3(rows), dim3(256), 0, stream, true, x, hidden, residual, w, out, dim, eps); };
    if (nv <= 8) few(rms_norm_few_kernel<MODE, 1>);
    else few(rms_norm_few_kernel<MODE, 2>);
    return;
  }
  auto go = [&](auto kern, int per) { launch(kern, dim3((rows + per - 1) / per), dim3(128), 0, stream, true, x, hidden, residual, w, out, dim, rows, eps); };
  if (nv <= 4) go(rms_norm_rows_kernel<MODE, 4, 1>, 4);
  else if (nv <= 10) go(rms_norm_rows_kernel<MODE, 5, 2>, 2);
  else go(rms_norm_rows_kernel<MODE, 4, 4>, 1);
}

}  // namespace pk
