// Absorbed latent attention of prompt portions on tcgen05 (see latent_attention.cu for the math and the cache layout), bf16.
// All heads read the same cache line [c_j | kr_j], so a tile is 128 consecutive (token, head) rows of the flattened [tokens * heads] axis.
//
// CTA = (128 rows, up to 256 of the `rank` output columns): TMEM holds two S tiles of 64 keys (128 columns) and O (256 columns), so a wide latent is
// split over two CTAs that both compute S -- 1.5 times the MMAs of one pass, and no exchange.  Shared memory: Q (128 rows, all chunks of 64 features) and
// ONE block of 64 keys as chunks of 64 features.  A chunk that is no value of this CTA is free again as soon as S has read it, a value chunk when P V
// has; S takes the others first, so the next block's chunks arrive under the softmax and its S is under way before P V.
//   warps 0-3 softmax (thread = row; P goes back to TMEM over S and is the A operand of P V; O is scaled when a row's maximum has grown.  The reference
//             is the maximum itself: the largest weight is then 1, which bf16 holds exactly -- behind a maximum that lags by up to 2^8 its rounding alone
//             made the result's error 1.2 times as large for peaked scores; it saved 8 of 272 us)
//   warp 4    MMA issuer     S = Q K^T (SS),  O += P V (A from TMEM, V = the key chunks read N-major)
//   warp 5    TMA: the item's Q, then the pages of every key block
// Work item = (tile, run): the rows of a tile that belong to one request, with the tile's other rows masked, from an empty O.  What another request's
// cache holds (a NaN times a weight of zero) never reaches a row, and requests that share a tile -- decoded tokens beside a prompt portion, each with a
// context of its own -- do not wait for one another.  A tile's CTAs take its first run; the others, which start at a token whose first row is inside a
// tile, go to the helper CTAs, every helpers-th token to the same ones, so that the decoded tokens of a step spread over the GPU.  A helper that finds
// none ends at once.  B200, us, 16 heads, latent 512 + 64 (a tile's runs one after the other; latent_attention_mma.cu for all): 2048-token portion beside
// 8 tokens at contexts of 4096 307 (2345; 1169), 1000 beside 24 at 2000 154 (1146; 444), 320 tokens at 1000 376 (592; 334), 2048 alone 272 (271; 662).
// Keys outside the run (slots behind the context's end, keys before the window) are masked in S, and their value rows are cleared in shared memory
// before P V: they may hold anything.
// Tensor-bound (operand reads of the narrow MMAs): 2 * rows * keys * (2 rank + rot) flop of result, 1.5 times that executed at rank 512.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int LT_ROWS = 128, LT_KEYS = 64, LT_MAXC = 9, LT_VC = 4;  // rows, keys per block, feature chunks, value chunks per CTA
constexpr int LT_QC = LT_ROWS * 128, LT_KC = LT_KEYS * 128;         // bytes of a chunk of Q / of keys
constexpr int LT_THREADS = 192, LT_ITEMS = 128;  // items of a CTA at most

struct LtItem {  // consecutive tokens of one request inside a tile
  int R0, t0, t1;   // the tile's first row, first and last token
  int k0, lo, end;  // first key of the first block (on a page border), first visible key of any row, one past the last
  int pages;        // offset of the request's page list
};

struct LtArgs {
  const bf16* sink;
  const int *pos, *req, *page_off, *pages;
  bf16* out;
  int page_size, tokens, heads, rank, nc, halves, window;
  int helpers, helpers_first;  // helper CTAs per half; whether they come before the tiles' in the grid
  float scale_log2;
  unsigned int* err;
};

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
  uint64_t q_full, q_empty, k_full[LT_MAXC], k_empty[LT_MAXC], s_full[2], p_ready[2], pv_done, done;
  uint32_t tmem_slot;
  int dead, n_items, first_end;
  LtItem items[LT_ITEMS];
};

__global__ void __launch_bounds__(LT_THREADS, 1) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                          const LtArgs a) {
  extern __shared__ uint8_t lt_smem_raw[];
  uint8_t* Qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lt_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* Ks = Qs + (size_t)a.nc * LT_QC;
  LtSmem& m = *reinterpret_cast<LtSmem*>(Ks + (size_t)a.nc * LT_KC);
  volatile int* dead = &m.dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x % a.halves, total = a.tokens * a.heads, tiles = (total + LT_ROWS - 1) / LT_ROWS;
  const int group = blockIdx.x / a.halves, helper = a.helpers_first ? group : group - tiles;  // 0 .. helpers - 1: a helper
  const bool help = helper >= 0 && helper < a.helpers;
  auto item_of = [&](int R0, int t0, int t1) {
    const int rq = a.req[t0], lo = a.window > 0 ? max(a.pos[t0] - a.window + 1, 0) : 0;
    return LtItem{R0, t0, t1, lo / a.page_size * a.page_size, lo, a.pos[t1] + 1, a.page_off[rq]};
  };
  auto last_token = [&](int R0) { return (min(total, R0 + LT_ROWS) - 1) / a.heads; };
  bool starts = false;  // this thread's token starts a run inside a tile
  const int my_token = helper + (int)threadIdx.x * a.helpers;
  if (help) {
    pdl_wait();
    if (threadIdx.x < LT_ITEMS && my_token > 0 && my_token < a.tokens && (long)my_token * a.heads % LT_ROWS != 0) starts = a.req[my_token] != a.req[my_token - 1];
    if (__syncthreads_count(starts) == 0) return;
  }
  const int vc0 = half * LT_VC, nvc = min(LT_VC, a.rank / 64 - vc0);
  if (threadIdx.x == 0) {
    mbar_init(&m.q_full, 1);
    mbar_init(&m.q_empty, 1);
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
    m.n_items = 0;
    m.first_end = 0x7fffffff;
    mbar_fence_init();
  }
  if (warp == 4) tmem_alloc(&m.tmem_slot, 512);
  if (!help) pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (help) {
    if (starts) {
      const int R0 = my_token * a.heads / LT_ROWS * LT_ROWS, last = last_token(R0), rq = a.req[my_token];
      int e = my_token;
      while (e < last && a.req[e + 1] == rq) ++e;
      m.items[atomicAdd(&m.n_items, 1)] = item_of(R0, my_token, e);
    }
  } else {
    const int tile = tiles - 1 - (a.helpers_first ? group - a.helpers : group);  // late tokens (long contexts) first
    const int R0 = tile * LT_ROWS, t0 = R0 / a.heads, last = last_token(R0), t = t0 + 1 + (int)threadIdx.x;  // at most 128 tokens
    if (t <= last && a.req[t] != a.req[t - 1]) atomicMin(&m.first_end, t - 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      m.items[0] = item_of(R0, t0, min(last, m.first_end));
      m.n_items = 1;
    }
  }
  __syncthreads();
  pdl_launch_dependents();  // after the allocation: a dependent that came first would hold the TMEM while it waits for this grid
  const uint32_t tmem = m.tmem_slot;
  const int n_items = m.n_items;
  auto blocks_of = [&](const LtItem& r) { return (r.end - r.k0 + LT_KEYS - 1) / LT_KEYS; };  // 0: no visible key

  if (warp == 5) {
    // lane j copies the j-th piece (a page, or 64 slots of one) of every chunk; its page number is looked up once per block, a block ahead
    const int box = min(a.page_size, LT_KEYS), pieces = LT_KEYS / box;
    uint32_t n = 0, q = 0;  // blocks and queries so far
    for (int i = 0; i < n_items; ++i) {
      const LtItem r = m.items[i];
      const int* pg = a.pages + r.pages;
      const int nb = blocks_of(r), last = (r.end - 1) / a.page_size;
      if (nb <= 0) continue;
      if (q > 0) mbar_wait_bounded(&m.q_empty, (q - 1) & 1, dead);
      if (lane == 0) {
        mbar_expect_tx(&m.q_full, (uint32_t)(a.nc * LT_QC));
        for (int c = 0; c < a.nc; ++c) tma_load_2d(Qs + (size_t)c * LT_QC, &map_q, c * 64, r.R0, &m.q_full);
      }
      ++q;
      auto page_of = [&](int b) { return pg[min((r.k0 + b * LT_KEYS + lane * box) / a.page_size, last)]; };  // behind the end: the last page again (masked)
      int next = lane < pieces ? page_of(0) : 0;
      for (int b = 0; b < nb; ++b, ++n) {
        const int page = next, slot = (r.k0 + b * LT_KEYS + lane * box) % a.page_size;
        if (lane < pieces && b + 1 < nb) next = page_of(b + 1);
        for (int x = 0; x < a.nc; ++x) {
          const int c = (x + vc0 + nvc) % a.nc;  // the value chunks last
          mbar_wait_bounded(m.k_empty + c, (n & 1) ^ 1, dead);
          if (lane == 0) mbar_expect_tx(m.k_full + c, LT_KC);
          __syncwarp();
          if (lane < pieces) lt_tma_3d(Ks + (size_t)c * LT_KC + lane * box * 128, &map_k, c * 64, slot, page, m.k_full + c);
        }
      }
    }
    // Behind a run-out the copies go on, in bounds but without waiting for their places, and no barrier says when the last has landed: two milliseconds,
    // where a copy takes a thousandth of that
    if (*dead)
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncwarp();
  } else if (warp == 4) {
    if (tc_elect_one()) {
      // instruction descriptors: D = f32, A = B = bf16, A K-major; S: N = 64, B K-major; P V: N = 64 nvc, B (= V) N-major
      constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_ROWS >> 4) << 24);
      constexpr uint32_t idesc_s = base | ((uint32_t)(LT_KEYS >> 3) << 17);
      const uint32_t idesc_pv = base | (1u << 16) | ((uint32_t)(nvc * 8) << 17);
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
      const uint64_t vd = make_sw128_mn_desc(smem_u32(Ks + (size_t)vc0 * LT_KC), LT_KC, 1024);
      uint32_t n = 0, q = 0;  // blocks and queries so far
      for (int i = 0; i < n_items; ++i) {
        const uint32_t end = n + (uint32_t)max(blocks_of(m.items[i]), 0), first = n;
        if (n == end) continue;
        mbar_wait_bounded(&m.q_full, q++ & 1, dead);
        issue_s(n, 0, a.nc);
        if (n + 1 == end) umma_commit(&m.q_empty);
        for (; n < end; ++n) {
          if (n + 1 < end) issue_s(n + 1, 0, n_other);
          mbar_wait_bounded(m.p_ready + (n & 1), (n >> 1) & 1, dead);
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < LT_KEYS / 16; ++k)
            umma_bf16_tmem_a(tmem + 256, tmem + (n & 1) * LT_KEYS + (uint32_t)(k * 8), vd + (uint64_t)(k * (2048 >> 4)), idesc_pv, (n > first || k > 0) ? 1u : 0u);
          for (int c = vc0; c < vc0 + nvc; ++c) umma_commit(m.k_empty + c);
          umma_commit(&m.pv_done);
          if (n + 1 < end) issue_s(n + 1, n_other, a.nc);
          if (n + 2 == end) umma_commit(&m.q_empty);  // the item's last scores: then the next one's queries may come
        }
      }
      if (*dead) {
        umma_commit(&m.done);
        mbar_drain(&m.done, 0);
      }
    }
    __syncwarp();
  } else {
    const int row = threadIdx.x;  // 0 .. 127
    const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16), t_o = t_lane + 256;
    uint32_t n = 0;
    for (int i = 0; i < n_items; ++i) {
      const LtItem r = m.items[i];
      const int R = r.R0 + row, tok = R < total ? R / a.heads : -1, nb = blocks_of(r);
      const bool act = tok >= r.t0 && tok <= r.t1;
      const int my_pos = act ? a.pos[tok] : -1, my_lo = a.window > 0 ? my_pos - a.window + 1 : 0;
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
          if (b > 0) {  // O holds the blocks before this one (their P V were issued before this block's last scores, so they are complete)
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
      // ---- O / l -> bf16, the rows of this item (the next one's first P V waits for all 128 threads' next p_ready)
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
  if (tiles * halves < sm_count() / 2 || tiles * halves > 0x3fffffff || rows > 0x7fffffff) return -2;  // few rows: the key axis has to be split
  EncodeTiledFn fn = encode_fn();
  if (!fn) return -2;
  CUtensorMap mq, mk;
  if (!make_rows_map(&mq, qa, rows, D, LT_ROWS)) return -2;
  {
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)page_size, (cuuint64_t)1 << 30}, strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)page_stride * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)(page_size < LT_KEYS ? page_size : LT_KEYS), 1}, estr[3] = {1, 1, 1};
    if (fn(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(cache), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -2;
  }
  // Runs that start inside a tile are for the helpers, one CTA per half and SM (more where a helper would have over LT_ITEMS tokens to look at); none
  // where each token fills whole tiles.  They come first, since their contexts may be the longest, unless all CTAs fit at once.
  int helpers = heads % LT_ROWS == 0 ? 0 : (sm_count() + halves - 1) / halves;
  if (helpers > 0 && helpers < (tokens + LT_ITEMS - 1) / LT_ITEMS) helpers = (tokens + LT_ITEMS - 1) / LT_ITEMS;
  const size_t smem = (size_t)nc * (LT_QC + LT_KC) + sizeof(LtSmem) + 1024;
  static std::atomic<uint64_t> smem_set{0};
  if (allow_smem(smem_set, (const void*)latent_attention_tc_kernel, LT_MAXC * (LT_QC + LT_KC) + sizeof(LtSmem) + 1024) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  const LtArgs a{sink, pos, req, page_off, pages, out, page_size, tokens, heads, rank, nc, halves, window, helpers, tiles * halves > sm_count(), scale * 1.4426950408889634f, wait_err_word()};
  return (int)launch(latent_attention_tc_kernel, dim3((unsigned)((tiles + helpers) * halves)), dim3(LT_THREADS), smem, st, true, mq, mk, a);
}

}  // namespace pk
