// Mixture-of-experts feed-forward for many tokens at once (prompt portions): the (token, choice) pairs are bucketed by
// expert, and each expert's rows run as one tensor-core GEMM over that expert's weights, so a weight tile is read once
// per 256 rows instead of once per token (moe.cu is the per-token form for a few tokens).
//   1. moe_bucket_kernel     one CTA: histogram of the routed ids, offsets per expert, a slot for every pair, and the list of row tiles: an
//                            expert's rows in as few tiles of at most 256 as they need, of equal size.  Which slot a pair gets inside its
//                            expert's run may vary from run to run; every row's result is independent of its slot, so outputs do not.
//   2. moe_gather_kernel     xs[slot] = x[token(slot)]  (TMA then reads an expert's rows as a block)
//      moe_place_kernel      both, for up to 32768 pairs
//   3. moe_grouped_gemm<0>   hid[slot] = relu(W_up[e] xs[slot])^2
//      moe_grouped_gemm<2>   hid[slot] = silu(W_gate[e] x) * (W_up[e] x)            (gated experts, gate / up rows interleaved)
//      moe_grouped_gemm<3>   hid[slot] = g logistic(p1 g) (u + 1), g = min(W_gate[e] x, p0), u = clamp(W_up[e] x, -p0, p0)
//   4. moe_grouped_gemm<1>   part[slot] = weight(pair) * W_down[e] hid[slot]     (fp32)
//   5. moe_combine_kernel    y[t] = sum_k part[slot(t, k)] (+ logistic(g_t) * shared[t]), summed in the order of k
// GEMM: tcgen05, persistent CTA pairs (cta_group::2).  The weights are the M axis (256 features, 128 to a CTA, TMEM lane = feature) and the rows the N axis
// (TMEM column = row, half of them staged by each CTA), so that a tile costs MMAs for its own rows (to the next 16) and not for a full tile of 128; an
// expert of the usual 100-250 rows reads its weights once.
//   warp 0 TMA (6 stages of 64 deep) | warp 1 of the leader MMA | warps 2-9 epilogue from the other of two accumulators.
// Bound: HBM for few rows per expert (all weights are read once), the operand traffic out of L2 for many: single CTAs read an expert's rows once per 128
// features, 12 TB/s in all.  2048 tokens, 64 experts of 2048 x 1408, top 6 (B200, whole call): 1025 us with 64 x 64 tiles of mma.sync, 320 with single CTAs and
// four epilogue warps, 312 in pairs, 281 with eight (the gated epilogue's exponentials and divisions set the pace), 278 with one launch for places and rows
// (one box under one clock; on three others 357 to 360 -> 310 to 315); 32 tokens 187 -> 175, where the weights alone take 163.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

constexpr int kMoeTile = 256;   // rows per tile at most (UMMA N)
constexpr int kMoeSlack = 64;   // the workspace has room for a tile per so many pairs

// meta layout (ints): [0] number of row tiles, [1 .. E+1] offsets (exclusive scan, E + 1 entries), then tile_expert[max_tiles],
// tile_row0[max_tiles] (one entry more than tiles: the end); slot_pair[pairs] and pair_slot[pairs] are separate arrays.
constexpr int kBucketThreads = 1024, kBucketIds = 16;  // ids a thread keeps in registers
__global__ void __launch_bounds__(kBucketThreads) moe_bucket_kernel(const int* __restrict__ ids, int pairs, int experts, int max_tiles,
                                                                    int* __restrict__ meta, int* __restrict__ slot_pair, int* __restrict__ pair_slot) {
  extern __shared__ int sh[];  // [experts] counts, then [experts] cursors, then [2 * 33] sums per warp
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  int* cnt = sh;
  int* cur = sh + experts;
  int* wsum = sh + 2 * experts;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < experts; e += kBucketThreads) cnt[e] = 0;
  int mine[kBucketIds];  // all loads on their way before the first is used
#pragma unroll
  for (int i = 0; i < kBucketIds; ++i) mine[i] = tid + i * kBucketThreads < pairs ? ids[tid + i * kBucketThreads] : -1;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kBucketIds; ++i)
    if (mine[i] >= 0) atomicAdd(&cnt[mine[i]], 1);
  for (int p = tid + kBucketIds * kBucketThreads; p < pairs; p += kBucketThreads) atomicAdd(&cnt[ids[p]], 1);
  __syncthreads();
  // exclusive scans of the row and the tile counts over the experts, kBucketThreads experts at a time
  int* off = meta + 1;
  int* te = meta + 2 + experts;
  int* tr = te + max_tiles;
  int rows0 = 0, tiles0 = 0;
  for (int e0 = 0; e0 < experts; e0 += kBucketThreads) {
    const int e = e0 + tid, c = e < experts ? cnt[e] : 0, nt = (c + kMoeTile - 1) / kMoeTile;
    int rc = c, rt = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, rc, o), b = __shfl_up_sync(0xffffffffu, rt, o);
      if (lane >= o) {
        rc += a;
        rt += b;
      }
    }
    if (lane == 31) {
      wsum[warp] = rc;
      wsum[33 + warp] = rt;
    }
    __syncthreads();
    if (warp == 0) {
      int a = wsum[lane], b = wsum[33 + lane];
      const int a0 = a, b0 = b;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
          a += x;
          b += y;
        }
      }
      wsum[lane] = a - a0;
      wsum[33 + lane] = b - b0;
      if (lane == 31) {
        wsum[32] = a;
        wsum[65] = b;
      }
    }
    __syncthreads();
    if (e < experts) {
      const int row = rows0 + wsum[warp] + rc - c, tile = tiles0 + wsum[33 + warp] + rt - nt;
      off[e] = row;
      cur[e] = row;
      const int size = nt ? ((c + nt - 1) / nt + 15) / 16 * 16 : 0;
      for (int i = 0; i < nt; ++i) {
        te[tile + i] = e;
        tr[tile + i] = row + i * size;
      }
    }
    rows0 += wsum[32];
    tiles0 += wsum[65];
    __syncthreads();
  }
  if (tid == 0) {
    off[experts] = rows0;
    tr[tiles0] = rows0;
    meta[0] = tiles0;
  }
#pragma unroll
  for (int i = 0; i < kBucketIds; ++i) {
    if (mine[i] < 0) continue;
    const int p = tid + i * kBucketThreads, s = atomicAdd(&cur[mine[i]], 1);
    slot_pair[s] = p;
    pair_slot[p] = s;
  }
  for (int p = tid + kBucketIds * kBucketThreads; p < pairs; p += kBucketThreads) {
    const int s = atomicAdd(&cur[ids[p]], 1);
    slot_pair[s] = p;
    pair_slot[p] = s;
  }
}

// xs[slot] = x[slot_pair[slot] / top], 16-byte pieces
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* __restrict__ x, const int* __restrict__ slot_pair, bf16* __restrict__ xs, int width,
                                                         int top) {
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int s = blockIdx.x, nv = width >> 3;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(slot_pair[s] / top) * width);
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)s * width);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) dst[i] = src[i];
}

// Both at once, for up to kPlacePairs pairs and kPlaceThreads experts: each CTA takes an equal share of the pairs, counts all ids by itself (its own
// pairs' predecessors in the upper half of the same word), so that it knows where its pairs go, and copies their rows; the first also writes the lists.  One
// launch instead of two, and no step on a single SM (281 -> 278 us of the call above, 26.9 -> 25.7 of 64 tokens on 16 experts of 1024 x 768).
constexpr int kPlacePairs = 32768, kPlaceThreads = 512, kPlaceHead = 8;
__global__ void __launch_bounds__(kPlaceThreads) moe_place_kernel(const int* __restrict__ ids, int pairs, int experts, int max_tiles, int* __restrict__ meta,
                                                                  int* __restrict__ slot_pair, int* __restrict__ pair_slot, const bf16* __restrict__ x,
                                                                  bf16* __restrict__ xs, int width, int top) {
  __shared__ unsigned cnt[kPlaceThreads];  // all pairs of the expert | those before this CTA's << 16
  __shared__ int cur[kPlaceThreads], wsum[2][kPlaceThreads / 32];
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = (int)((long)blockIdx.x * pairs / gridDim.x), end = (int)((long)(blockIdx.x + 1) * pairs / gridDim.x);
  // the warp's first pair's row, under way while its place is looked for
  const int nv = width >> 3;
  uint4 head[kPlaceHead];
#pragma unroll
  for (int i = 0; i < kPlaceHead; ++i)
    if (first + warp < end && lane + 32 * i < nv) head[i] = reinterpret_cast<const uint4*>(x + (size_t)((first + warp) / top) * width)[lane + 32 * i];
  cnt[tid] = 0;
  __syncthreads();
#pragma unroll 8
  for (int p = tid; p < pairs; p += kPlaceThreads) atomicAdd(&cnt[ids[p]], p < first ? 0x10001u : 1u);
  __syncthreads();
  // exclusive scans of the row and the tile counts over the experts
  const int c = tid < experts ? (int)(cnt[tid] & 0xffffu) : 0, before = tid < experts ? (int)(cnt[tid] >> 16) : 0, nt = (c + kMoeTile - 1) / kMoeTile;
  int rc = c, rt = nt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, rc, o), b = __shfl_up_sync(0xffffffffu, rt, o);
    if (lane >= o) {
      rc += a;
      rt += b;
    }
  }
  if (lane == 31) {
    wsum[0][warp] = rc;
    wsum[1][warp] = rt;
  }
  __syncthreads();
  int row = rc - c, tile = rt - nt;
  for (int w = 0; w < warp; ++w) {
    row += wsum[0][w];
    tile += wsum[1][w];
  }
  cur[tid] = row + before;
  if (blockIdx.x == 0 && tid <= experts) {
    int *off = meta + 1, *te = meta + 2 + experts, *tr = te + max_tiles;
    off[tid] = row;
    if (tid == experts) {
      tr[tile] = row;
      meta[0] = tile;
    } else {
      const int size = nt ? ((c + nt - 1) / nt + 15) / 16 * 16 : 0;
      for (int i = 0; i < nt; ++i) {
        te[tile + i] = tid;
        tr[tile + i] = row + i * size;
      }
    }
  }
  __syncthreads();
  for (int p = first + warp; p < end; p += kPlaceThreads / 32) {
    int s = 0;
    if (lane == 0) {
      s = atomicAdd(&cur[ids[p]], 1);
      slot_pair[s] = p;
      pair_slot[p] = s;
    }
    s = __shfl_sync(0xffffffffu, s, 0);
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(p / top) * width);
    uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)s * width);
    int i = lane;
    if (p == first + warp) {
#pragma unroll
      for (int k = 0; k < kPlaceHead; ++k, i += 32)
        if (i < nv) dst[i] = head[k];
    }
#pragma unroll 8
    for (; i < nv; i += 32) dst[i] = src[i];
  }
}

constexpr int kMgStages = 6, kMgEpi = 8, kMgThreads = 64 + 32 * kMgEpi, kMgChunk = 32;  // chunk: rows of an epilogue step
constexpr int kMgA = 128 * 64 * 2, kMgBox = 64 * 64 * 2, kMgStage = kMgA + kMoeTile / 2 * 64 * 2;  // bytes: a CTA's features, 64 rows, a stage
constexpr size_t kMgSmem = (size_t)kMgStages * kMgStage + 1024 + kMgEpi / 4 * kMgChunk * 128 * 2 + (2 * kMgStages + 5) * 8 + 16;

struct MgArgs {
  void* out;
  const int* meta;
  const int* slot_pair;
  const float* weights;
  int experts, max_tiles, N, K;  // N: weight rows per expert
  float p0, p1;
  unsigned int* err;
};

// EPI 0: out bf16 [slots][N] = relu(acc)^2.   EPI 1: out fp32 [slots][N] = acc * weights[pair of the slot].
// EPI 2: W rows interleaved (2f = gate f, 2f + 1 = up f): out bf16 [slots][N / 2] = silu(acc[2f]) * acc[2f + 1].
// EPI 3: the same rows with clamped pre-activations: g = min(acc[2f], p0), u = clamp(acc[2f + 1], -p0, p0), out = g logistic(p1 g) (u + 1).
// W_FIRST: the weights are the first to leave L2.
template <int EPI, bool W_FIRST>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMgThreads, 1) moe_grouped_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                        const MgArgs a) {
  extern __shared__ uint8_t mg_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mg_smem_raw) + 1023) & ~(uintptr_t)1023);
  bf16* tiles_out = reinterpret_cast<bf16*>(smem + (size_t)kMgStages * kMgStage);  // epilogue, per four warps: [32 rows][64 or 128 outputs]
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles_out + kMgEpi / 4 * kMgChunk * 128);  // the leader's: bytes of both CTAs
  uint64_t* empty = full + kMgStages;
  uint64_t* tfull = empty + kMgStages;
  uint64_t* tempty = tfull + 2;
  uint64_t* done = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMgStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull + s, 1);
      mbar_init(tempty + s, 2 * kMgEpi);  // the leader's: an arrival per epilogue warp of both CTAs
    }
    mbar_init(done, 1);
    *dead = 0;
    mbar_fence_init();
  }
  if (warp == 1) g2_tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_barrier();  // both CTAs' barriers and accumulators are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, rank = cluster_ctarank();
  pdl_wait();
  pdl_launch_dependents();  // after the allocation: a dependent that came first would hold the TMEM while it waits for this grid
  const int* te = a.meta + 2 + a.experts;
  const int* tr = te + a.max_tiles;
  const int n_ft = (a.N + 255) / 256, tiles = a.meta[0] * n_ft, k_blocks = (a.K + 63) / 64;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;  // neighbouring pairs share an expert's rows
  if (warp == 0) {
    if (tc_elect_one()) {
      int s = 0;
      uint32_t ph = 1;
      [[maybe_unused]] const uint64_t first = W_FIRST ? l2_evict_first_policy() : 0;
      for (int t = pair; t < tiles && !*dead; t += pairs) {
        const int rt = t / n_ft, n16 = (tr[rt + 1] - tr[rt] + 15) / 16, boxes = (n16 * 8 + 63) / 64;
        const int r0 = tr[rt] + (int)rank * n16 * 8, w0 = te[rt] * a.N + (t - rt * n_ft) * 256 + (int)rank * 128;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait_bounded(empty + s, ph, dead)) break;
          const uint32_t fb = g2_map(smem_u32(full + s), 0);
          if (rank == 0) mbar_expect_tx(full + s, 2 * (kMgA + boxes * kMgBox));
          uint8_t* st = smem + (size_t)s * kMgStage;
          if constexpr (W_FIRST) g2_tma_2d(st, &map_w, kb * 64, w0, fb, first);
          else g2_tma_2d(st, &map_w, kb * 64, w0, fb);
          for (int b = 0; b < boxes; ++b) g2_tma_2d(st + kMgA + b * kMgBox, &map_x, kb * 64, r0 + b * 64, fb);
          if (++s == kMgStages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // Behind a run-out no barrier of this CTA says when its copies under way have landed: two milliseconds, where a copy takes a thousandth of that
      if (*dead)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
  } else if (warp == 1) {
    if (rank == 0 && tc_elect_one()) {
      int s = 0, lt = 0;
      uint32_t ph = 0;
      for (int t = pair; t < tiles && !*dead; t += pairs, ++lt) {
        const int rt = t / n_ft, n16 = (tr[rt + 1] - tr[rt] + 15) / 16, as = lt & 1;
        // instruction descriptor: D = f32 [4,6) = 1, A = bf16 [7,10) = 1, B = bf16 [10,13) = 1, both K-major, N >> 3 at [17,23), M >> 4 at [24,29)
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n16 * 2) << 17) | ((uint32_t)(256 >> 4) << 24);
        if (!mbar_wait_bounded(tempty + as, (uint32_t)(((lt >> 1) & 1) ^ 1), dead)) break;
        tc_fence_after();
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait_bounded(full + s, ph, dead)) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + (size_t)s * kMgStage);
          const uint64_t ad = make_sw128_desc(a_addr), bd = make_sw128_desc(a_addr + kMgA);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            g2_umma(tmem_base + (uint32_t)(as * kMoeTile), ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          g2_commit_both(empty + s);
          if (++s == kMgStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        g2_commit_both(tfull + as);
      }
      if (*dead) {
        g2_commit_both(done);
        mbar_drain(done, 0);
      }
    }
  } else {
    // two groups of four warps take turns at the chunks.  TMEM lane quarter this warp may read; group; thread of the group
    const int q = warp & 3, grp = (warp - 2) >> 2, et = (threadIdx.x - 64) & 127;
    bf16* tile = tiles_out + grp * kMgChunk * 128;
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
    const int out_n = EPI >= 2 ? a.N / 2 : a.N;
    const uint32_t tempty0 = g2_map(smem_u32(tempty), 0);
    int lt = 0;
    // (to the last tile even when a wait ran out: a warp that left on its own reading of the flag would leave the others at barrier 1)
    for (int t = pair; t < tiles; t += pairs, ++lt) {
      const int rt = t / n_ft, m0 = tr[rt], rows = tr[rt + 1] - m0, f0 = (t - rt * n_ft) * 256 + (int)rank * 128, as = lt & 1;
      mbar_wait_bounded(tfull + as, (uint32_t)((lt >> 1) & 1), dead);
      __syncwarp();
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * kMoeTile);
      auto weight_of = [&](int r) { return EPI == 1 && r < rows ? a.weights[a.slot_pair[m0 + r]] : 0.f; };  // asked for a chunk ahead
      float next = weight_of(grp * kMgChunk + lane);
      for (int c = grp * kMgChunk; c < rows; c += kMgEpi / 4 * kMgChunk) {
        uint32_t v[32];
        const float wl = next;
        next = weight_of(c + kMgEpi / 4 * kMgChunk + lane);
        tmem_ld32(t_row + (uint32_t)c, v);
        const int n = min(kMgChunk, rows - c);
        if (EPI == 1) {  // fp32: a row's 32 features of a warp are 128 contiguous bytes
          const int f = f0 + q * 32 + lane;
          float* o = static_cast<float*>(a.out) + (size_t)(m0 + c) * a.N + f;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float w = __shfl_sync(0xffffffffu, wl, j);
            if (j < n && f < a.N) o[(size_t)j * a.N] = __uint_as_float(v[j]) * w;
          }
          continue;
        }
        // bf16: through shared memory, [row][output], so that a row leaves in 16-byte pieces
        constexpr int OW = EPI >= 2 ? 64 : 128;
        group_sync();  // the last chunk has left
        if (EPI == 0) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float z = fmaxf(__uint_as_float(v[j]), 0.f);
            tile[j * OW + q * 32 + lane] = f2bf(z * z);
          }
        } else {
          // gate in the even lane, up in the odd one: of two rows the even lane takes the first, the odd lane the second
          // (exponentials, then divisions: side by side, where one loop would run an element's chain after the other's)
          float gt[16], up[16], den[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float give = __uint_as_float(lane & 1 ? v[2 * j] : v[2 * j + 1]), keep = __uint_as_float(lane & 1 ? v[2 * j + 1] : v[2 * j]);
            const float got = __shfl_xor_sync(0xffffffffu, give, 1);
            gt[j] = lane & 1 ? got : keep;
            up[j] = lane & 1 ? keep : got;
            if (EPI == 3) {
              gt[j] = fminf(gt[j], a.p0);
              up[j] = fminf(fmaxf(up[j], -a.p0), a.p0) + 1.f;
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) den[j] = 1.f + expf(EPI == 3 ? -a.p1 * gt[j] : -gt[j]);
#pragma unroll
          for (int j = 0; j < 16; ++j) tile[(2 * j + (lane & 1)) * OW + q * 16 + (lane >> 1)] = f2bf(gt[j] / den[j] * up[j]);
        }
        group_sync();
        const int o0 = EPI >= 2 ? f0 / 2 : f0;
        for (int i = et; i < kMgChunk * OW / 8; i += 128) {
          const int r = i / (OW / 8), p = (i % (OW / 8)) * 8;
          if (r < n && o0 + p < out_n)
            *reinterpret_cast<uint4*>(static_cast<bf16*>(a.out) + (size_t)(m0 + c + r) * out_n + o0 + p) = *reinterpret_cast<const uint4*>(tile + r * OW + p);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) g2_arrive_cluster(tempty0 + (uint32_t)(as * 8));
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) count_run_out(dead, a.err);
  cluster_barrier();  // the peer's MMAs and copies may still have this CTA's memory as their target
  if (warp == 1) {
    tc_fence_after();
    g2_tmem_dealloc(tmem_base, 512);
  }
}

// y[t] = sum over k of part[slot(t, k)], in the order of k; float4 pieces (width is a multiple of 8)
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ part, const int* __restrict__ pair_slot, const bf16* __restrict__ shared,
                                                          const float* __restrict__ sg, float* __restrict__ y, int width, int top) {
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t = blockIdx.x, nv = width >> 2;
  const float g = shared ? (sg ? 1.f / (1.f + expf(-sg[t])) : 1.f) : 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    // two rows under way (four: 0.5 to 1 % of a call more up to 512 tokens, the same beyond), which leave L2 first (2048 tokens 260 -> 256 us)
#pragma unroll 2
    for (int k = 0; k < top; ++k) {
      const float4 p = __ldcs(reinterpret_cast<const float4*>(part + (size_t)pair_slot[(size_t)t * top + k] * width) + i);
      acc.x += p.x;
      acc.y += p.y;
      acc.z += p.z;
      acc.w += p.w;
    }
    if (shared) {
      const bf16* s = shared + (size_t)t * width + i * 4;
      acc.x += g * bf2f(s[0]);
      acc.y += g * bf2f(s[1]);
      acc.z += g * bf2f(s[2]);
      acc.w += g * bf2f(s[3]);
    }
    float* o = y + (size_t)t * width + i * 4;
    if ((reinterpret_cast<uintptr_t>(y) & 15) == 0) {
      *reinterpret_cast<float4*>(o) = acc;
    } else {
      o[0] = acc.x;
      o[1] = acc.y;
      o[2] = acc.z;
      o[3] = acc.w;
    }
  }
}

template <int EPI, bool W_FIRST>
static cudaError_t mg_launch(const void* rows, long n_rows, const void* w, const MgArgs& a, cudaStream_t st) {
  CUtensorMap mx, mw;
  if (!make_rows_map(&mx, rows, n_rows, a.K, 64) || !make_rows_map(&mw, w, (long)a.experts * a.N, a.K, 128)) return cudaErrorInvalidValue;
  auto kern = moe_grouped_gemm_kernel<EPI, W_FIRST>;
  static std::atomic<uint64_t> smem_set{0};
  if (const cudaError_t e = allow_smem(smem_set, (const void*)kern, kMgSmem); e != cudaSuccess) return e;
  // as many pairs as there can be tiles, one CTA per SM at most
  const long tiles = (n_rows / kMoeTile + (n_rows < a.experts ? n_rows : a.experts)) * ((a.N + 255) / 256);
  const long pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  return launch(kern, dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs))), dim3(kMgThreads), kMgSmem, st, true, mx, mw, a);
}

template <int EPI>
static cudaError_t mg_gemm(bool w_first, const void* rows, long n_rows, const void* w, const MgArgs& a, cudaStream_t st) {
  return w_first ? mg_launch<EPI, true>(rows, n_rows, w, a, st) : mg_launch<EPI, false>(rows, n_rows, w, a, st);
}

}  // namespace pk

using namespace pk;

extern "C" long pk_moe_grouped_workspace_bytes(int tokens, int top, int experts, int width, int ff) {
  const long pairs = (long)tokens * top, max_tiles = pairs / kMoeSlack + experts + 1;
  long b = (2 + experts + 2 * max_tiles + 2 * pairs) * 4;  // meta, slot_pair, pair_slot
  b = (b + 255) / 256 * 256;
  b += (pairs * ff * 2 + 255) / 256 * 256;  // hid
  b += pairs * width * 4;                   // part; before that, the gathered rows
  return b + 256;
}

// y [tokens, width] fp32 = routed experts (+ gated shared expert); bf16 operands; width % 8 == 0 and ff % 8 == 0.
extern "C" int pk_moe_grouped_act(const void* xa, const void* w_up, const void* w_down, const int* ids, const float* weights, const void* shared,
                                  const float* shared_gate, float* y, void* workspace, int tokens, int top, int experts, int width, int ff, int act,
                                  pk_stream st) {
  if (act < 0 || act > 1) return -1;
  return pk_moe_grouped_act_p(xa, w_up, w_down, ids, weights, shared, shared_gate, y, workspace, tokens, top, experts, width, ff, act, 0.f, 0.f, st);
}

// act 2: clamped gated experts (limit p0, slope p1); shared_gate may be NULL with a shared expert (added without a gate)
extern "C" int pk_moe_grouped_act_p(const void* xa, const void* w_up, const void* w_down, const int* ids, const float* weights, const void* shared,
                                    const float* shared_gate, float* y, void* workspace, int tokens, int top, int experts, int width, int ff, int act,
                                    float p0, float p1, pk_stream st) {
  if (!xa || !w_up || !w_down || !ids || !weights || !y || !workspace || tokens <= 0 || top <= 0 || experts <= 0 || experts > 4096 || act < 0 || act > 2 ||
      (act == 2 && !(p0 > 0.f)))
    return -1;
  if (width % 8 || ff % 8 || (reinterpret_cast<uintptr_t>(xa) & 15) || (reinterpret_cast<uintptr_t>(w_up) & 15) ||
      (reinterpret_cast<uintptr_t>(w_down) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return -2;
  const long pairs = (long)tokens * top;
  const int max_tiles = (int)(pairs / kMoeSlack) + experts + 1;
  char* ws = static_cast<char*>(workspace);
  int* meta = reinterpret_cast<int*>(ws);
  int* slot_pair = meta + 2 + experts + 2 * max_tiles;
  int* pair_slot = slot_pair + pairs;
  long o = ((2 + experts + 2 * (long)max_tiles + 2 * pairs) * 4 + 255) / 256 * 256;
  bf16* hid = reinterpret_cast<bf16*>(ws + o);
  o += (pairs * ff * 2 + 255) / 256 * 256;
  float* part = reinterpret_cast<float*>(ws + o);
  bf16* xs = reinterpret_cast<bf16*>(part);  // done with when `part` is written
  if (pairs <= kPlacePairs && experts < kPlaceThreads) {
    launch(moe_place_kernel, dim3((unsigned)(pairs < 2L * sm_count() ? pairs : 2L * sm_count())), dim3(kPlaceThreads), 0, st, true, ids, (int)pairs, experts, max_tiles, meta,
           slot_pair, pair_slot, (const bf16*)xa, xs, width, top);
  } else {
    launch(moe_bucket_kernel, dim3(1), dim3(kBucketThreads), (size_t)(2 * experts + 66) * sizeof(int), st, true, ids, (int)pairs, experts, max_tiles, meta,
           slot_pair, pair_slot);
    launch(moe_gather_kernel, dim3((unsigned)pairs), dim3(width >= 2048 ? 256 : 128), 0, st, true, (const bf16*)xa, (const int*)slot_pair, xs, width, top);
  }
  // From 24 rows an expert on the rows, hidden values and partial sums (100 MB in the call of 2048 tokens) are worth their room in L2, and up to a row tile
  // an expert the weights are read once: they leave first, where they are too many to be found in L2 again.  B200, 64 experts of 2048 x 1408, top 6, gated, us:
  // 256 / 512 / 1024 / 2048 tokens 189 199 220 262 -> 181 184 205 257 in a train over other weights each time (a single call with cold caches spreads by as much);
  // without the bounds it would be 64 tokens 187 197, 4096 438 445.
  const bool w_first = pairs >= 24l * experts && pairs <= (kMoeTile - 16l) * experts && (long)experts * width * ff * (act ? 6 : 4) > (256l << 20);
  MgArgs a{hid, meta, slot_pair, weights, experts, max_tiles, act ? 2 * ff : ff, width, p0, p1, wait_err_word()};
  cudaError_t e = act == 2 ? mg_gemm<3>(w_first, xs, pairs, w_up, a, st) : act == 1 ? mg_gemm<2>(w_first, xs, pairs, w_up, a, st) : mg_gemm<0>(w_first, xs, pairs, w_up, a, st);
  if (e != cudaSuccess) return (int)e;
  a.out = part;
  a.N = width;
  a.K = ff;
  if ((e = mg_gemm<1>(w_first, hid, pairs, w_down, a, st)) != cudaSuccess) return (int)e;
  launch(moe_combine_kernel, dim3(tokens), dim3(256), 0, st, true, (const float*)part, (const int*)pair_slot, (const bf16*)shared, shared_gate, y, width,
         top);
  return (int)cudaGetLastError();
}

extern "C" int pk_moe_grouped_relu2(const void* xa, const void* w_up, const void* w_down, const int* ids, const float* weights, const void* shared,
                                    const float* shared_gate, float* y, void* workspace, int tokens, int top, int experts, int width, int ff,
                                    pk_stream st) {
  return pk_moe_grouped_act(xa, w_up, w_down, ids, weights, shared, shared_gate, y, workspace, tokens, top, experts, width, ff, 0, st);
}
