// GEMM for few output tiles: Y[M, N] = W[M, K] x X[K, N] with N of a decode batch or a short prompt (from 5 tokens on; how far up depends
// on M, see sk_plan).  The pass is a read of W: 2 M K bytes of HBM against few tokens' worth of MMAs, so what counts is that every SM
// streams the same share of W and that the sum over K costs no round trip through global memory.
//
//   A = W : `rows` <= 128 features per tile (UMMA M = 128, TMEM lane = feature), B = X : NT tokens (UMMA N = NT, TMEM column = token), so
//   a weight row enters shared memory once and a tile's accumulator is only NT columns (gemm.cu has the tokens on the M axis and pads
//   8 of them to 128 rows).
//   A tile's K is cut into S parts, one CTA each, and the S CTAs are a cluster: every CTA leaves its fp32 partial in its own shared
//   memory ([token][feature], over the operand ring), and after a cluster barrier CTA r adds up the S partials of its share of the
//   tile in rank order over distributed shared memory and stores bf16.  The order is fixed, so a result does not depend on timing.
//   Any number of rows may make a tile: the MMAs always read 128 rows of A, and what the rows behind the tile's own hold ends in
//   accumulator lanes that nobody reads.  So the tiles can be cut to fill all SMs evenly.
//   warp 0 TMA producer | warp 1 MMA issuer | warps 2-5 partial -> shared memory | all warps: sum -> output.
// Bound: HBM for large W, else the chain launch -> first load -> MMAs -> cluster sum (about 4.3 us a launch in a train, 0.25 us per K block
// of 64, most of it the issue of four narrow MMAs at 52 clocks each).  The figures stand at sk_plan.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int SK_BM = 128, SK_BK = 64, SK_THREADS = 192;
constexpr int SK_MAX_SPLIT = 8, SK_MAX_STAGES = 12;  // 8: the portable cluster size

__device__ __forceinline__ float4 sk_ld_dsmem(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
// two CTAs on an SM: at most half of its shared memory each
constexpr int SK_SMEM_MAX = 112 * 1024;
constexpr size_t sk_smem(int rows, int nt, int stages) {
  return (size_t)stages * (rows + nt) * SK_BK * 2 + (SK_BM - rows) * SK_BK * 2 + 1024 + (2 * SK_MAX_STAGES + 1) * 8 + 16;
}

struct SkArgs {
  bf16 *Y, *Y1, *Y2;
  int e0, e1;         // features [0, e0) -> Y (rows of e0), [e0, e1) -> Y1, the rest -> Y2
  int M, N, K;        // features, tokens, reduction
  int n_tiles;        // token tiles
  int rows;           // features per tile (multiple of 8, <= 128)
  int stages;
  unsigned int* err;  // counts waits that ran out (null: not counted)
};

template <int NT>
__global__ void __launch_bounds__(SK_THREADS)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const SkArgs a) {
  const int stages = a.stages, rows = a.rows;
  const int A_BYTES = rows * SK_BK * 2, STAGE_BYTES = A_BYTES + NT * SK_BK * 2;
  constexpr uint32_t TMEM_COLS = NT <= 32 ? 32 : NT <= 64 ? 64 : 128;
  extern __shared__ uint8_t sk_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sk_smem_raw) + 1023) & ~(uintptr_t)1023);
  // (behind the last stage lies room for the rows of A that the MMAs read beyond the tile's own)
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)stages * STAGE_BYTES + (SK_BM - rows) * SK_BK * 2);
  uint64_t* empty = full + SK_MAX_STAGES;
  uint64_t* done = empty + SK_MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = gridDim.x, sp = (int)cluster_ctarank();  // the cluster spans the whole x axis
  const int m0 = (blockIdx.y / a.n_tiles) * rows, t0 = (blockIdx.y % a.n_tiles) * NT;
  const int k_blocks = (a.K + SK_BK - 1) / SK_BK;
  const int kb0 = (sp * k_blocks) / S, nk = ((sp + 1) * k_blocks) / S - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(done, 1);
    *dead = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // no early trigger: gemv.cu streams its weights before it waits for its predecessor, and they may be this kernel's output
  pdl_wait();

  if (warp == 0) {
    if (tc_elect_one()) {
      int s = 0, i = 0;
      uint32_t ph = 1;
      for (; i < nk; ++i) {
        if (!mbar_wait_bounded(empty + s, ph, dead)) break;
        mbar_expect_tx(full + s, STAGE_BYTES);
        uint8_t* st = smem + (size_t)s * STAGE_BYTES;
        tma_load_2d(st, &map_w, (kb0 + i) * SK_BK, m0, full + s);
        tma_load_2d(st + A_BYTES, &map_x, (kb0 + i) * SK_BK, t0, full + s);
        if (++s == stages) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (i < nk) ring_drain(full, stages, i);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (tc_elect_one()) {
      // instruction descriptor: D = f32 [4,6) = 1, A = bf16 [7,10) = 1, B = bf16 [10,13) = 1, both K-major, N >> 3 at [17,23), M >> 4 at [24,29)
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(SK_BM >> 4) << 24);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < nk; ++i) {
        if (!mbar_wait_bounded(full + s, ph, dead)) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + (size_t)s * STAGE_BYTES);
        const uint64_t adesc = make_sw128_desc(a_addr), bdesc = make_sw128_desc(a_addr + A_BYTES);
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k) umma_bf16(tmem_base, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(empty + s);
        if (++s == stages) {
          s = 0;
          ph ^= 1u;
        }
      }
      umma_commit(done);
    }
    __syncwarp();
  }
  // ---- every MMA has read its operands once `done` completes: the ring now takes the partial [NT tokens][rows features]
  if (!mbar_wait_bounded(done, 0, dead)) mbar_drain(done, 0);
  __syncwarp();
  tc_fence_after();
  float* part = reinterpret_cast<float*>(smem);
  if (warp >= 2 && (warp & 3) * 32 < rows) {
    const int q = warp & 3, f = q * 32 + lane;  // TMEM lane quarter this warp may read; lane = feature
#pragma unroll
    for (int c = 0; c < NT; c += 16) {
      uint32_t v[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
            "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c));
      // the wait names the registers it makes valid, so that no use of them can be moved in front of it
      asm volatile("tcgen05.wait::ld.sync.aligned;"
                   : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                     "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                   :
                   : "memory");
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (f < rows) part[(c + j) * rows + f] = __uint_as_float(v[j]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_barrier();
  // ---- this CTA's share of the tile: (token, 4 features) items, added up in rank order
  const int quads = rows / 4, items = min(NT, a.N - t0) * quads;
  const int i0 = (sp * items) / S, i1 = ((sp + 1) * items) / S;
  const uint32_t part_addr = smem_u32(part);
  for (int it = i0 + threadIdx.x; it < i1; it += SK_THREADS) {
    const int t = it / quads, f = m0 + (it - t * quads) * 4;
    float4 v[SK_MAX_SPLIT];
#pragma unroll
    for (int r = 0; r < SK_MAX_SPLIT; ++r)
      if (r < S) v[r] = S > 1 ? sk_ld_dsmem(part_addr + (uint32_t)it * 16u, (uint32_t)r) : *reinterpret_cast<const float4*>(part + (size_t)it * 4);
    float4 s = v[0];
#pragma unroll
    for (int r = 1; r < SK_MAX_SPLIT; ++r)
      if (r < S) {
        s.x += v[r].x;
        s.y += v[r].y;
        s.z += v[r].z;
        s.w += v[r].w;
      }
    if (f >= a.M) continue;
    const int lo = f < a.e0 ? 0 : (f < a.e1 ? a.e0 : a.e1), hi = f < a.e0 ? a.e0 : (f < a.e1 ? a.e1 : a.M);
    bf16* base = f < a.e0 ? a.Y : (f < a.e1 ? a.Y1 : a.Y2);
    bf16* dst = base + (size_t)(t0 + t) * (hi - lo) + (f - lo);
    if (f + 4 <= hi && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
    } else {  // a quad across the border of two outputs, or rows of an odd length
      const float o[4] = {s.x, s.y, s.z, s.w};
      for (int j = 0; j < 4 && f + j < a.M; ++j) {
        const int g = f + j;
        bf16* d = g < a.e0 ? a.Y + (size_t)(t0 + t) * a.e0 + g
                           : (g < a.e1 ? a.Y1 + (size_t)(t0 + t) * (a.e1 - a.e0) + (g - a.e0) : a.Y2 + (size_t)(t0 + t) * (a.M - a.e1) + (g - a.e1));
        *d = f2bf(o[j]);
      }
    }
  }
  if (threadIdx.x == 0) count_run_out(dead, a.err);  // (every wait lies before the barrier above)
  __syncwarp();
  if (S > 1) cluster_barrier();  // the others may still read this CTA's partial
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int NT>
cudaError_t sk_launch(const CUtensorMap& mx, const CUtensorMap& mw, const SkArgs& a, int tiles, int splits, cudaStream_t stream) {
  auto kern = gemm_skinny_kernel<NT>;
  static std::atomic<uint64_t> smem_set{0};
  if (const cudaError_t e = allow_smem(smem_set, (const void*)kern, SK_SMEM_MAX); e != cudaSuccess) return e;
  ThreadState& ts = tls();
  ts.launches++;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(splits, tiles);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = sk_smem(a.rows, NT, a.stages);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = ts.pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, mx, mw, a);
}

// Clusters of `splits` CTAs that can be resident at once, two CTAs on an SM.  A cluster lives inside one GPC, so large ones leave slots empty:
// on B200 (148 SMs) 8-CTA clusters fit 32 times at most and the 33rd would wait for a whole round (o_proj of Qwen3-4B at 8 tokens: 30 tiles 7.9 us, 36 tiles 12.3 us).
int sk_resident(int splits, int sms) { return splits == 8 ? sms * 32 / 148 : splits == 4 ? sms * 70 / 148 : 2 * sms / splits; }

struct SkPlan {
  int rows, splits, stages;  // rows 0: more tiles than fit on the GPU at once
};

// The most K parts for which all tiles run at once, and the lowest tiles for which they still do, so that every SM has the same share of W.
// Beyond 128 tokens gemm2.cu is the faster one as soon as its CTA pairs (256 tokens x 128 features each) are half in use; here -> gemm2.cu, us:
// 2560 x 9728 25.2 -> 35.1 at 160 tokens and 37.4 -> 35.3 at 400;  4096 x 12288 43.2 -> 49.8 and 58.5 -> 51.3;  6144 x 2560 19.2 -> 15.1 at 160.
// But gemm2.cu adds up over K in one go and this kernel in parts, and what a stack of projections gets in one call and each of them in a call of its own
// is the same, bit for bit, only if both take the same kernel (pk_b200_gemm_segments promises it from 129 tokens on).  The number of features must not
// decide, then, wherever it could differ between the two: only reductions of 8192 or more (they come from a feed-forward's inner width; projections are
// stacked over the hidden width) and fewer than 64 features (gates of a head each, no head's row is so short) come here.  What that gives up at 160
// tokens: 2560 x 4096 13.7 -> 16.4, 1024 x 4096 11.7 -> 15.4.  Parts follow from K (4 from 4096 on, where they fit, else 2), and
// below 64 features, which no stacking has to agree with, they are as many as fit: 32 x 2560 of 300 / 1024 / 2048 tokens 9.0 9.1 9.2 us with two, 6.1 6.3 7.0.
// Measured on B200, us a launch in a train over cold weights (before: the split-K form of gemm.cu; from 129 tokens on gemm2.cu), M x K:
//   tokens            8            48           128          160
//   6144 x 2560   20.1 -> 9.5  19.9 -> 10.4  24.9 -> 12.6     (gemm2)
//   2560 x 4096   15.9 -> 8.2  15.9 -> 9.2   18.7 -> 11.4     (gemm2)
//   2560 x 9728   20.0 -> 13.1 20.6 -> 13.5  23.5 -> 16.3  61.2 -> 20.5
//   19456 x 2560  31.3 -> 20.2 23.5 -> 21.2     (gemm.cu)     (gemm2)
//   24576 x 4096  49.1 -> 37.1 43.2 -> 38.6     (gemm.cu)     (gemm2)
//   4096 x 12288  29.9 -> 20.8 30.4 -> 22.2  33.9 -> 25.8  76.7 -> 30.9
//   32 x 2560     10.3 -> 4.3  10.2 -> 4.5   10.7 -> 5.4
// Where the SMs are full without cutting K (one part), each CTA reads all of X beside its rows of W: from 65 tokens on the 128-token tiles of
// gemm.cu are as fast (24.3 us both at 19456 x 2560), and from 129 on gemm2.cu is faster.
SkPlan sk_plan(int M, int N, int K, int nt, int sms) {
  const int n_tiles = (N + nt - 1) / nt, kb = (K + SK_BK - 1) / SK_BK;
  for (int S = N <= 128 || M < 64 ? SK_MAX_SPLIT : K >= 4096 ? 4 : 2; S >= 1; S /= 2) {
    if (S > 1 && S > kb / 4) continue;  // at least 4 K blocks per part
    const int fit = sk_resident(S, sms) / n_tiles;  // feature tiles
    if ((long)fit * SK_BM < M) continue;
    int rows = ((M + fit - 1) / fit + 7) / 8 * 8;
    if (rows < 32) rows = 32;
    int stages = SK_MAX_STAGES;
    while (stages > 2 && sk_smem(rows, nt, stages) > SK_SMEM_MAX) --stages;
    const int nk = (kb + S - 1) / S, hold = (nt * rows * 4 + (rows + nt) * SK_BK * 2 - 1) / ((rows + nt) * SK_BK * 2);  // stages that the partial covers
    if (stages > nk) stages = nk > hold ? nk : hold;
    return SkPlan{rows, S, stages};
  }
  return SkPlan{0, 1, 0};
}

bool sk_many_tokens(int M, int N, int K, int sms) { return M < 64 || (K >= 8192 && (long)((N + 255) / 256) * ((M + 127) / 128) * 4 <= sms); }

template <int NT>
int sk_run(const bf16* W, const bf16* X, bf16* Y, bf16* Y1, bf16* Y2, int e0, int e1, int M, int N, int K, cudaStream_t stream) {
  const SkPlan p = sk_plan(M, N, K, NT, sm_count());
  if (p.rows == 0 || (p.splits == 1 && (N > 128 || (N > 64 && M > SK_BM * sm_count())))) return -2;
  if (N > 128 && !sk_many_tokens(M, N, K, sm_count())) return -2;
  const int n_tiles = (N + NT - 1) / NT, tiles = ((M + p.rows - 1) / p.rows) * n_tiles;
  CUtensorMap mx, mw;
  if (!make_rows_map(&mx, X, N, K, NT) || !make_rows_map(&mw, W, M, K, p.rows)) return -2;
  const SkArgs a{Y, Y1, Y2, e0, e1, M, N, K, n_tiles, p.rows, p.stages, wait_err_word()};
  return (int)sk_launch<NT>(mx, mw, a, tiles, p.splits, stream);
}

}  // namespace

// 0 = launched, -2 = not for this kernel
int launch_gemm_skinny(const bf16* W, const bf16* X, bf16* Y, bf16* Y1, bf16* Y2, int e0, int e1, int M, int N, int K, cudaStream_t stream) {
  if (K % 8 != 0 || (reinterpret_cast<uintptr_t>(W) & 15) != 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0) return -2;
#define PK_SK_RUN(NT) return sk_run<NT>(W, X, Y, Y1, Y2, e0, e1, M, N, K, stream)
  if (N <= 16) PK_SK_RUN(16);
  if (N <= 32) PK_SK_RUN(32);
  if (N <= 48) PK_SK_RUN(48);
  if (N <= 64) PK_SK_RUN(64);
  if (N <= 96) PK_SK_RUN(96);
  PK_SK_RUN(128);
#undef PK_SK_RUN
}

}  // namespace pk
