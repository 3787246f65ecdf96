// Absorbed latent attention of prompt portions on tcgen05 (see latent_attention.cu for the math and the cache layout), bf16.
// All heads read the same cache line [c_j | kr_j], so a tile is 128 consecutive (token, head) rows of the flattened [tokens * heads] axis.
//
// CTA = (128 rows, up to 256 of the `rank` output columns): TMEM holds two S tiles of 64 keys (128 columns) and O (256 columns), so a wide latent is
// split over two CTAs that both compute S -- 1.5 times the MMAs of one pass, and no exchange.  Shared memory: Q (128 rows, all chunks of 64 features) and
// ONE block of 64 keys as chunks of 64 features.  A chunk that is no value of this CTA is free again as soon as S has read it, a value chunk when P V
// has; S takes the others first, so the next block's chunks arrive under the softmax and its S is under way before P V.
//   warps 0-3 softmax (thread = row; P goes back to TMEM over S and is the A operand of P V; O is scaled when a row's maximum has grown.  The reference
//             is the maximum itself: the largest weight is then 1, which bf16 holds exactly -- behind a maximum that lags by up to 2^8 its rounding alone
//             made the result's error 1.2 times as large for peaked scores)
//   warp 4    MMA issuer     S = Q K^T (SS),  O += P V (A from TMEM, V = the key chunks read N-major)
//   warp 5    TMA: Q once, then the pages of every key block
// A tile whose rows belong to several requests walks each request's keys in turn with the other rows masked, starts O anew for each and writes that
// request's rows behind it: what another request's cache holds (a NaN times a weight of zero) never reaches them.  Keys outside the run (slots behind
// the context's end, keys before the window) are masked in S, and their value rows are cleared in shared memory before P V: they may hold anything.
// Tensor-bound (operand reads of the narrow MMAs): 2 * rows * keys * (2 rank + rot) flop of result, 1.5 times that executed at rank 512.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int LT_ROWS = 128, LT_KEYS = 64, LT_MAXC = 9, LT_VC = 4;  // rows, keys per block, feature chunks, value chunks per CTA
constexpr int LT_QC = LT_ROWS * 128, LT_KC = LT_KEYS * 128;         // bytes of a chunk of Q / of keys
constexpr int LT_THREADS = 192;

struct LtRun {  // consecutive tokens of one request inside a tile
  int t0, t1;    // first and last token
  int k0, lo, end;  // first key of the first block (on a page border), first visible key of any row, one past the last
  int pages;     // offset of the request's page list
};

struct LtArgs {
  const bf16* sink;
  const int *pos, *req, *page_off, *pages;
  bf16* out;
  int page_size, tokens, heads, rank, nc, halves, window;
  float scale_log2;
  unsigned int* err;
};

__device__ __forceinline__ void lt_tma_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void lt_tma_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ float lt_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct LtSmem {  // behind Q and the key chunks
  uint64_t q_full, k_full[LT_MAXC], k_empty[LT_MAXC], s_full[2], p_ready[2], pv_done, done;
  uint32_t tmem_slot;
  int dead, n_runs;
  int tok_req[LT_ROWS], tok_pos[LT_ROWS];
  LtRun runs[LT_ROWS];
};

__global__ void __launch_bounds__(LT_THREADS, 1) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                          const LtArgs a) {
  extern __shared__ uint8_t lt_smem_raw[];
  uint8_t* Qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lt_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* Ks = Qs + (size_t)a.nc * LT_QC;
  LtSmem& m = *reinterpret_cast<LtSmem*>(Ks + (size_t)a.nc * LT_KC);
  volatile int* dead = &m.dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x % a.halves, tile = gridDim.x / a.halves - 1 - blockIdx.x / a.halves;  // late tokens (long contexts) first
  const int R0 = tile * LT_ROWS, total = a.tokens * a.heads;
  const int t_first = R0 / a.heads, n_tok = (min(total, R0 + LT_ROWS) - 1) / a.heads - t_first + 1;
  const int vc0 = half * LT_VC, nvc = min(LT_VC, a.rank / 64 - vc0);
  if (threadIdx.x == 0) {
    mbar_init(&m.q_full, 1);
    for (int c = 0; c < LT_MAXC; ++c) {
      mbar_init(m.k_full + c, 1);
      mbar_init(m.k_empty + c, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(m.s_full + i, 1);
      mbar_init(m.p_ready + i, LT_ROWS);
    }
    mbar_init(&m.pv_done, 1);
    mbar_init(&m.done, 1);
    m.dead = 0;
    mbar_fence_init();
  }
  if (warp == 4) tmem_alloc(&m.tmem_slot, 512);
  pdl_wait();
  for (int i = threadIdx.x; i < n_tok; i += LT_THREADS) {
    m.tok_req[i] = a.req[t_first + i];
    m.tok_pos[i] = a.pos[t_first + i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int t = 0; t < n_tok;) {
      int e = t;
      while (e + 1 < n_tok && m.tok_req[e + 1] == m.tok_req[t]) ++e;
      LtRun r;
      r.t0 = t;
      r.t1 = e;
      r.lo = a.window > 0 ? max(m.tok_pos[t] - a.window + 1, 0) : 0;
      r.k0 = r.lo / a.page_size * a.page_size;
      r.end = m.tok_pos[e] + 1;
      r.pages = a.page_off[m.tok_req[t]];
      m.runs[n++] = r;
      t = e + 1;
    }
    m.n_runs = n;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();  // after the allocation: a dependent that came first would hold the TMEM while it waits for this grid
  const uint32_t tmem = m.tmem_slot;
  const int n_runs = m.n_runs;
  auto blocks_of = [&](const LtRun& r) { return (r.end - r.k0 + LT_KEYS - 1) / LT_KEYS; };

  if (warp == 5) {
    if (lane == 0) {
      mbar_expect_tx(&m.q_full, (uint32_t)(a.nc * LT_QC));
      for (int c = 0; c < a.nc; ++c) lt_tma_2d(Qs + (size_t)c * LT_QC, &map_q, c * 64, R0, &m.q_full);
    }
    // lane j copies the j-th piece (a page, or 64 slots of one) of every chunk; its page number is looked up once per block, a block ahead
    const int box = min(a.page_size, LT_KEYS), pieces = LT_KEYS / box;
    uint32_t n = 0;
    int fills = 0;  // of the key chunks, in the order in which they are loaded
    bool on = true;
    for (int i = 0; i < n_runs && on; ++i) {
      const LtRun r = m.runs[i];
      const int* pg = a.pages + r.pages;
      const int nb = blocks_of(r), last = (r.end - 1) / a.page_size;
      auto page_of = [&](int b) { return pg[min((r.k0 + b * LT_KEYS + lane * box) / a.page_size, last)]; };  // behind the end: the last page again (masked)
      int next = lane < pieces ? page_of(0) : 0;
      for (int b = 0; b < nb && on; ++b, ++n) {
        const int page = next, slot = (r.k0 + b * LT_KEYS + lane * box) % a.page_size;
        if (lane < pieces && b + 1 < nb) next = page_of(b + 1);
        for (int x = 0; x < a.nc; ++x, ++fills) {
          const int c = (x + vc0 + nvc) % a.nc;  // the value chunks last
          on = __all_sync(0xffffffffu, mbar_wait_bounded(m.k_empty + c, (n & 1) ^ 1, dead));
          if (!on) break;
          if (lane == 0) mbar_expect_tx(m.k_full + c, LT_KC);
          __syncwarp();
          if (lane < pieces) lt_tma_3d(Ks + (size_t)c * LT_KC + lane * box * 128, &map_k, c * 64, slot, page, m.k_full + c);
        }
      }
    }
    if (!on) {
      mbar_drain(&m.q_full, 0);
      for (int j = max(0, fills - a.nc); j < fills; ++j) mbar_drain(m.k_full + (j % a.nc + vc0 + nvc) % a.nc, (uint32_t)((j / a.nc) & 1));
    }
    __syncwarp();
  } else if (warp == 4) {
    if (tc_elect_one()) {
      // instruction descriptors: D = f32, A = B = bf16, A K-major; S: N = 64, B K-major; P V: N = 64 nvc, B (= V) N-major
      constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_ROWS >> 4) << 24);
      constexpr uint32_t idesc_s = base | ((uint32_t)(LT_KEYS >> 3) << 17);
      const uint32_t idesc_pv = base | (1u << 16) | ((uint32_t)(nvc * 8) << 17);
      uint32_t total_blocks = 0;
      for (int i = 0; i < n_runs; ++i) total_blocks += blocks_of(m.runs[i]);
      const int n_other = a.nc - nvc;
      // chunks [x0, x1) of block n in the order of the loads
      auto issue_s = [&](uint32_t n, int x0, int x1) {
        for (int x = x0; x < x1; ++x) {
          const int c = (x + vc0 + nvc) % a.nc;
          mbar_wait_bounded(m.k_full + c, n & 1, dead);
          tc_fence_after();
          const uint64_t qd = make_sw128_desc(smem_u32(Qs + (size_t)c * LT_QC)), kd = make_sw128_desc(smem_u32(Ks + (size_t)c * LT_KC));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16(tmem + (n & 1) * LT_KEYS, qd + (uint64_t)(k * 2), kd + (uint64_t)(k * 2), idesc_s, (x > 0 || k > 0) ? 1u : 0u);
          if (x < n_other) umma_commit(m.k_empty + c);
        }
        if (x1 == a.nc) umma_commit(m.s_full + (n & 1));
      };
      mbar_wait_bounded(&m.q_full, 0, dead);
      if (total_blocks > 0) issue_s(0, 0, a.nc);
      uint32_t run_end = 0;  // block at which the next run starts
      int run = 0;
      const uint64_t vd = make_sw128_mn_desc(smem_u32(Ks + (size_t)vc0 * LT_KC), LT_KC, 1024);
      for (uint32_t n = 0; n < total_blocks; ++n) {
        if (n + 1 < total_blocks) issue_s(n + 1, 0, n_other);
        mbar_wait_bounded(m.p_ready + (n & 1), (n >> 1) & 1, dead);
        tc_fence_after();
        const bool anew = n == run_end;
        while (n == run_end) run_end += blocks_of(m.runs[run++]);
#pragma unroll
        for (int k = 0; k < LT_KEYS / 16; ++k)
          umma_bf16_tmem_a(tmem + 256, tmem + (n & 1) * LT_KEYS + (uint32_t)(k * 8), vd + (uint64_t)(k * (2048 >> 4)), idesc_pv, (!anew || k > 0) ? 1u : 0u);
        for (int c = vc0; c < vc0 + nvc; ++c) umma_commit(m.k_empty + c);
        umma_commit(&m.pv_done);
        if (n + 1 < total_blocks) issue_s(n + 1, n_other, a.nc);
      }
      if (*dead) {
        umma_commit(&m.done);
        mbar_drain(&m.done, 0);
      }
    }
    __syncwarp();
  } else {
    const int row = threadIdx.x, R = R0 + row;  // 0 .. 127
    const int tok = R < total ? R / a.heads - t_first : -1, my_pos = tok >= 0 ? m.tok_pos[tok] : -1;
    const int my_lo = a.window > 0 ? my_pos - a.window + 1 : 0;
    const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16), t_o = t_lane + 256;
    uint32_t n = 0;
    for (int i = 0; i < n_runs; ++i) {
      const LtRun r = m.runs[i];
      const bool act = tok >= r.t0 && tok <= r.t1;
      const int nb = blocks_of(r);
      float mx = -INFINITY, l = 0.f;  // running maximum (scaled, log2 units) and sum
      for (int b = 0; b < nb; ++b, ++n) {
        const int j0 = r.k0 + b * LT_KEYS;
        mbar_wait_bounded(m.s_full + (n & 1), (n >> 1) & 1, dead);
        __syncwarp();
        tc_fence_after();
        const uint32_t t_s = t_lane + (n & 1) * LT_KEYS;
        uint32_t v[64];
        tmem_ld32_nowait(t_s, v);
        tmem_ld32_nowait(t_s + 32, v + 32);
        tmem_ld_wait64(v);
        // visible keys of this row in the block: [c0, c1)
        const int c0 = act ? max(my_lo - j0, 0) : LT_KEYS, c1 = act ? my_pos + 1 - j0 : 0;
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (__all_sync(0xffffffffu, c0 == 0 && c1 >= LT_KEYS)) {
#pragma unroll
          for (int x = 0; x < 64; ++x) m4[x & 3] = fmaxf(m4[x & 3], __uint_as_float(v[x]));
        } else {
#pragma unroll
          for (int x = 0; x < 64; ++x) {
            if (x < c0 || x >= c1) v[x] = 0xff800000u;  // -inf
            m4[x & 3] = fmaxf(m4[x & 3], __uint_as_float(v[x]));
          }
        }
        const float blk = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2;
        const bool grow = blk > mx;
        if (__any_sync(0xffffffffu, grow)) {
          const float to = grow ? blk : mx, corr = grow ? lt_exp2(mx - to) : 1.f;
          mx = to;
          l *= corr;
          if (b > 0) {  // O holds the blocks before this one
            mbar_wait_bounded(&m.pv_done, (n - 1) & 1, dead);
            __syncwarp();
            tc_fence_after();
            for (int c = 0; c < nvc * 64; c += 64) {
              uint32_t t[64];
              tmem_ld32_nowait(t_o + c, t);
              tmem_ld32_nowait(t_o + c + 32, t + 32);
              tmem_ld_wait64(t);
#pragma unroll
              for (int x = 0; x < 64; ++x) t[x] = __float_as_uint(__uint_as_float(t[x]) * corr);
              tmem_put32(t_o + c, t);
              tmem_put32(t_o + c + 32, t + 32);
            }
            tmem_put_wait();
          }
        }
        const float ref = mx == -INFINITY ? 0.f : mx;  // a row without a key so far: every p is 2^-inf = 0
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t p[32];
#pragma unroll
        for (int x = 0; x < 64; x += 2) {
          const float p0 = lt_exp2(fmaf(__uint_as_float(v[x]), a.scale_log2, -ref)), p1 = lt_exp2(fmaf(__uint_as_float(v[x + 1]), a.scale_log2, -ref));
          s4[x & 2] += p0;
          s4[(x & 2) + 1] += p1;
          p[x / 2] = pack_bf16(p0, p1);
        }
        l += (s4[0] + s4[1]) + (s4[2] + s4[3]);
        tmem_put32(t_s, p);
        tmem_put_wait();
        if (j0 < r.lo || j0 + LT_KEYS > r.end) {  // clear the value rows of keys that are not the run's
          const int rr = row & 63, key = j0 + rr;
          if (key < r.lo || key >= r.end)
            for (int c = vc0 + (row >> 6); c < vc0 + nvc; c += 2) {
              uint4* z = reinterpret_cast<uint4*>(Ks + (size_t)c * LT_KC + rr * 128);
#pragma unroll
              for (int y = 0; y < 8; ++y) z[y] = make_uint4(0, 0, 0, 0);
            }
          fence_proxy_async_smem();
        }
        tc_fence_before();
        mbar_arrive(m.p_ready + (n & 1));
      }
      // ---- O / l -> bf16, the rows of this run (the next one's first P V waits for all 128 threads' next p_ready)
      if (nb > 0) mbar_wait_bounded(&m.pv_done, (n - 1) & 1, dead);
      __syncwarp();
      tc_fence_after();
      const float sk = a.sink && act ? bf2f(a.sink[R % a.heads]) * 1.4426950408889634f : -INFINITY;
      const float M = fmaxf(mx, sk), w = lt_exp2(mx - M);
      const float inv = w / (l * w + (a.sink ? lt_exp2(sk - M) : 0.f));
      uint4* dst = reinterpret_cast<uint4*>(a.out + (size_t)(act ? R : 0) * a.rank + vc0 * 64);
      for (int c = 0; c < nvc * 64; c += 64) {
        uint32_t t[64] = {};
        if (nb > 0) {  // no visible key at all (a position before the first): O is zero, as the sum is
          tmem_ld32_nowait(t_o + c, t);
          tmem_ld32_nowait(t_o + c + 32, t + 32);
          tmem_ld_wait64(t);
        }
        if (act) {
#pragma unroll
          for (int x = 0; x < 64; x += 8)
            dst[(c + x) >> 3] = make_uint4(pack_bf16(__uint_as_float(t[x]) * inv, __uint_as_float(t[x + 1]) * inv),
                                           pack_bf16(__uint_as_float(t[x + 2]) * inv, __uint_as_float(t[x + 3]) * inv),
                                           pack_bf16(__uint_as_float(t[x + 4]) * inv, __uint_as_float(t[x + 5]) * inv),
                                           pack_bf16(__uint_as_float(t[x + 6]) * inv, __uint_as_float(t[x + 7]) * inv));
        }
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) count_run_out(dead, a.err);
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace

// 0 = launched; -2 = shape / alignment outside this kernel (the caller runs the mma.sync kernel)
int launch_latent_attention_tc(const bf16* qa, const bf16* cache, const bf16* sink, const int* pos, const int* req, const int* page_off, const int* pages,
                               bf16* out, long page_stride, int page_size, int tokens, int heads, int rank, int rot, float scale, int window,
                               cudaStream_t st) {
  const int D = rank + rot, nc = (D + 63) / 64, halves = (rank / 64 + LT_VC - 1) / LT_VC;
  // (rot % 16, rank <= 512: what the mma.sync kernel takes too.  The shapes beyond go to the generic kernel, whose weights stay fp32.)
  if (rank % 64 || rot % 16 || rank > 512 || nc > LT_MAXC || page_size < 8 || (page_size & (page_size - 1)) || page_stride % 8 || !(scale > 0.f) ||
      ((reinterpret_cast<uintptr_t>(qa) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -2;
  const long rows = (long)tokens * heads, tiles = (rows + LT_ROWS - 1) / LT_ROWS;
  if (tiles * halves < sm_count() / 2 || tiles * halves > 0x7fffffff || rows > 0x7fffffff) return -2;  // few rows: the key axis has to be split
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -2;
  CUtensorMap mq, mk;
  {
    cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)D * 2};
    cuuint32_t box[2] = {64, LT_ROWS}, estr[2] = {1, 1};
    if (fn(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(qa), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -2;
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)page_size, (cuuint64_t)1 << 30}, strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)page_stride * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)(page_size < LT_KEYS ? page_size : LT_KEYS), 1}, estr[3] = {1, 1, 1};
    if (fn(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(cache), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -2;
  }
  const size_t smem = (size_t)nc * (LT_QC + LT_KC) + sizeof(LtSmem) + 1024;
  static std::atomic<uint64_t> smem_set{0};
  if (allow_smem(smem_set, (const void*)latent_attention_tc_kernel, LT_MAXC * (LT_QC + LT_KC) + sizeof(LtSmem) + 1024) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  const LtArgs a{sink, pos, req, page_off, pages, out, page_size, tokens, heads, rank, nc, halves, window, scale * 1.4426950408889634f, wait_err_word()};
  return (int)launch(latent_attention_tc_kernel, dim3((unsigned)(tiles * halves)), dim3(LT_THREADS), smem, st, true, mq, mk, a);
}

}  // namespace pk
