// Absorbed latent attention of prompt portions on tcgen05 (see latent_attention.cu for the math and the cache layout), bf16.
// All heads read the same cache line [c_j | kr_j], so a tile is 128 consecutive (token, head) rows of the flattened [tokens * heads] axis.
//
// CTA = (128 rows, up to 256 of the `rank` output columns): a wide latent is split over two CTAs that both compute S -- 1.5 times the MMAs of one pass, and
// no exchange.  TMEM holds two S tiles of 64 keys (128 columns), the part of Q that belongs to this CTA's value chunks (128 columns: an A operand in TMEM
// saves the 32 clocks in which one in shared memory is read, 46 instead of 78 for 64 keys) and O (256 columns).  Shared memory: the rest of Q, two blocks'
// value chunks, and a ring of other chunks, so that the next block's scores are computed under this block's softmax.
//   warps 0-7   softmax: two threads per row, each half of the keys and of the output columns; the halves' maxima meet in shared memory.  P goes back to
//               TMEM over S and is the A operand of P V; O is scaled when a row's maximum has grown, behind the exponentials, once the last P V is through.
//               The reference is the maximum itself: the largest weight is then 1, which bf16 holds exactly -- behind a maximum that lags by up to 2^8 its
//               rounding alone made the result's error 1.2 times as large for peaked scores
//   warp 8      MMA issuer     S = Q K^T,  O += P V (A from TMEM, V = the key chunks read N-major)
//   warps 9-14  TMA: Q and the pages of every key block
//   warp 15     items, in a queue to all roles: those of this CTA, then those of the grid's next CTA, taken away from the launch when the loads of the
//               last item near their end (earlier, and a long tile could be held here that another SM would begin sooner).  A CTA's start and end are 12 us:
//               the launch, page numbers, Q, the first scores, O; here the next item's Q and scores come under the last products and results of this one
// Rows of Q and of the result are 1 KB and more apart: a thread that moves its own row touches a line per 16 bytes (the Q of an item took 3500 clocks, its
// result 4000).  Four lanes move 64 bytes of a row at a time and exchange pieces by shuffles.
// B200, us, 16 heads: 2048-token prompt, latent 512 + 64 132 -> 106 (a tile after the other by the launch 132, taken 117, and by 64 bytes 106); 3 prompts
// of 2048 tokens in all 82 -> 58; latent 256 + 32 58 -> 52; 592 tokens, one tile per SM, 27 -> 24.  Bound by the tensor cores and, for
// the operands outside TMEM, their shared-memory reads: a block of 64 keys takes 3000 clocks, 20 score MMAs of 78, 16 of 46 and 4 value MMAs of 142 2860.
// Work item = (tile, run): the rows of a tile that belong to one request, with the tile's other rows masked, from an empty O.  What another request's
// cache holds (a NaN times a weight of zero) never reaches a row, and requests that share a tile -- decoded tokens beside a prompt portion, each with a
// context of its own -- do not wait for one another.  A tile's CTAs take its first run; the others, which start at a token whose first row is inside a
// tile, go to the helper CTAs, every helpers-th token to the same ones, so that the decoded tokens of a step spread over the GPU.  A helper that finds
// none goes on with a tile.  B200, us, 16 heads, latent 512 + 64 (latent_attention_mma.cu in brackets): 2048-token portion beside 8
// tokens at contexts of 4096 123 (1169), 1000 beside 24 at 2000 64 (444), 320 tokens at 1000 150 (334).
// Keys outside the run (slots behind the context's end, keys before the window) are masked in S, and their value rows are cleared in shared memory
// before P V: they may hold anything.
// 2 * rows * keys * (2 rank + rot) flop of result, 1.5 times that executed at rank 512.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int LT_ROWS = 128, LT_KEYS = 64, LT_MAXC = 9, LT_VC = 4;  // rows, keys per block, feature chunks, value chunks per CTA
constexpr int LT_SOFT = 256, LT_LOAD_O = 2, LT_LOADS = LT_LOAD_O + LT_VC;  // softmax threads (two per row); loading warps
constexpr int LT_THREADS = LT_SOFT + 32 + 32 * LT_LOADS + 32, LT_SCAN = 128;  // tokens that a helper looks at, at most
constexpr int LT_QUEUE = 4, LT_READERS = LT_SOFT / 32 + 1 + LT_LOADS;  // items on their way to the roles; softmax warps, MMA issuer, loaders
constexpr int LT_QC = LT_ROWS * 128, LT_KC = LT_KEYS * 128;         // bytes of a chunk of Q / of keys
// places for other chunks: two blocks' or what Q and two blocks' value chunks leave of 216 KB, and never less than one block's (S waits for all of them)
constexpr int LT_RING = 9;
__host__ __device__ constexpr int lt_ring(int n_other, int nvc) {
  const int left = 27 - 2 * n_other - 2 * nvc, two = 2 * n_other < LT_RING ? 2 * n_other : LT_RING;
  return two < left ? two : left;
}
constexpr size_t lt_bytes(int n_other, int nvc) { return (size_t)n_other * LT_QC + (size_t)(2 * nvc + lt_ring(n_other, nvc)) * LT_KC; }
constexpr bool lt_fits() {
  for (int nvc = 0; nvc <= LT_VC; ++nvc)
    for (int o = 0; o <= LT_MAXC - nvc; ++o)
      if (lt_ring(o, nvc) < o || lt_bytes(o, nvc) > 216 * 1024) return false;
  return true;
}
static_assert(lt_fits(), "places for chunks");

struct LtItem {  // consecutive tokens of one request inside a tile
  int R0, t0, t1;   // the tile's first row, first and last token
  int k0, lo, end;  // first key of the first block (on a page border), first visible key of any row, one past the last
  int pages;        // offset of the request's page list
  int vc0;          // first value chunk of the half
};

struct LtArgs {
  const bf16 *qa, *sink;
  const int *pos, *req, *page_off, *pages;
  bf16* out;
  int page_size, tokens, heads, rank, D, nc, halves, window;
  int helpers, helpers_first;  // helper CTAs per half; whether they come before the tiles' in the grid
  int take;                    // whether a CTA goes on with the grid's next one
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

// The grid's next CTA that has not begun, taken away from the launch: the answer (16 bytes) comes with the barrier's phase
__device__ __forceinline__ void lt_take_next(void* answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ int lt_taken(const void* answer) {  // its blockIdx.x; -1: there is none
  int x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "ld.shared.b128 h, [%1];\n\t"
      "mov.b32 %0, -1;\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, h;\n\t}"
      : "=r"(x)
      : "r"(smem_u32(answer))
      : "memory");
  return x;
}

struct LtSmem {  // behind Q and the key chunks
  alignas(16) uint4 answer;
  uint64_t item_full[LT_QUEUE], item_empty[LT_QUEUE], taken, q_full, q_empty, q_tmem, k_full[2], k_empty[LT_RING], v_full[2], v_empty[2], s_full[2], p_ready[2], pv_done, done;
  uint32_t tmem_slot;
  int dead, near_end;  // near_end: items whose last blocks are being loaded, or that are done
  float top[2][LT_SOFT], sum[LT_SOFT];  // of the half rows: maxima (by the block's parity), sums
  LtItem items[LT_QUEUE];
};

__global__ void __launch_bounds__(LT_THREADS, 1) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                          const LtArgs a) {
  extern __shared__ uint8_t lt_smem_raw[];
  uint8_t* Qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lt_smem_raw) + 1023) & ~(uintptr_t)1023);
  // (where CTAs go on with others, the halves are alike)
  const int nvc = min(LT_VC, a.rank / 64 - (int)(blockIdx.x % a.halves) * LT_VC), n_other = a.nc - nvc;
  const int ring = lt_ring(n_other, nvc);
  uint8_t* Vs = Qs + (size_t)n_other * LT_QC;          // two of nvc chunks
  uint8_t* Ks = Vs + (size_t)2 * nvc * LT_KC;          // the ring of other chunks
  LtSmem& m = *reinterpret_cast<LtSmem*>(Ks + (size_t)ring * LT_KC);
  volatile int* dead = &m.dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = a.tokens * a.heads, tiles = (total + LT_ROWS - 1) / LT_ROWS;
  // which helper the grid's CTA `id` is, or -1
  auto helper_of = [&](int id) {
    const int group = id / a.halves, h = a.helpers_first ? group : group - tiles;
    return h >= 0 && h < a.helpers ? h : -1;
  };
  auto starts = [&](int t) { return t > 0 && t < a.tokens && (long)t * a.heads % LT_ROWS != 0 && a.req[t] != a.req[t - 1]; };  // a run begins inside a tile
  const int help = helper_of(blockIdx.x);
  if (help >= 0 && !a.take) {
    pdl_wait();
    if (__syncthreads_count(threadIdx.x < LT_SCAN && starts(help + (int)threadIdx.x * a.helpers)) == 0) return;
  }
  if (threadIdx.x == 0) {
    mbar_init(&m.q_full, 1);
    mbar_init(&m.q_empty, 1);
    mbar_init(&m.q_tmem, LT_SOFT);
    for (int c = 0; c < LT_RING; ++c) mbar_init(m.k_empty + c, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(m.k_full + i, 1);
      mbar_init(m.v_full + i, 1);
      mbar_init(m.v_empty + i, 1);
      mbar_init(m.s_full + i, 1);
      mbar_init(m.p_ready + i, LT_SOFT);
    }
    mbar_init(&m.pv_done, 1);
    mbar_init(&m.done, 1);
    mbar_init(&m.taken, 1);
    for (int i = 0; i < LT_QUEUE; ++i) {
      mbar_init(m.item_full + i, 1);
      mbar_init(m.item_empty + i, LT_READERS);
    }
    m.dead = 0;
    m.near_end = 0;
    mbar_fence_init();
  }
  if (warp == LT_SOFT / 32) tmem_alloc(&m.tmem_slot, 512);
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();  // after the allocation: a dependent that came first would hold the TMEM while it waits for this grid
  const uint32_t tmem = m.tmem_slot;
  // the CTA's k-th item, in the order of all roles; false: no more
  auto item = [&](uint32_t k, LtItem& r) {
    if (!mbar_wait_bounded(m.item_full + k % LT_QUEUE, (k / LT_QUEUE) & 1, dead)) return false;
    r = m.items[k % LT_QUEUE];
    return r.R0 >= 0;
  };
  auto blocks_of = [&](const LtItem& r) { return (r.end - r.k0 + LT_KEYS - 1) / LT_KEYS; };  // 0: no visible key

  if (warp == LT_THREADS / 32 - 1) {
    // Items: those of this CTA, then, while the last one's end is being computed, those of the grid's next CTA
    uint32_t n = 0, asked = 0;
    auto give = [&](const LtItem& r) {  // by one lane
      if (mbar_wait_bounded(m.item_empty + n % LT_QUEUE, ((n / LT_QUEUE) & 1) ^ 1, dead)) {
        m.items[n % LT_QUEUE] = r;
        mbar_arrive(m.item_full + n % LT_QUEUE);
      }
    };
    auto item_of = [&](int R0, int t0, int t1, int half) {
      const int rq = a.req[t0], lo = a.window > 0 ? max(a.pos[t0] - a.window + 1, 0) : 0;
      return LtItem{R0, t0, t1, lo / a.page_size * a.page_size, lo, a.pos[t1] + 1, a.page_off[rq], half * LT_VC};
    };
    auto last_token = [&](int R0) { return (min(total, R0 + LT_ROWS) - 1) / a.heads; };
    int id = blockIdx.x;
    while (id >= 0) {
      const int half = id % a.halves, h = helper_of(id);
      if (h >= 0) {
        bool st[LT_SCAN / 32];
#pragma unroll
        for (int j = 0; j < LT_SCAN / 32; ++j) st[j] = starts(h + (lane + 32 * j) * a.helpers);
#pragma unroll
        for (int j = 0; j < LT_SCAN / 32; ++j) {
          uint32_t which = __ballot_sync(0xffffffffu, st[j]);
          if (which == 0) continue;
          LtItem r{};
          if (st[j]) {
            const int t = h + (lane + 32 * j) * a.helpers, R0 = t * a.heads / LT_ROWS * LT_ROWS, last = last_token(R0), rq = a.req[t];
            int e = t;
            while (e < last && a.req[e + 1] == rq) ++e;
            r = item_of(R0, t, e, half);
          }
          for (; which; which &= which - 1, ++n) {
            if (lane == __ffs(which) - 1) give(r);
            __syncwarp();
          }
        }
      } else {
        const int group = id / a.halves, tile = tiles - 1 - (a.helpers_first ? group - a.helpers : group);  // late tokens (long contexts) first
        const int R0 = tile * LT_ROWS, t0 = R0 / a.heads, last = last_token(R0);
        int end = last;
        for (int t = t0 + 1; t <= last; t += 32) {  // (at most 128 tokens)
          const uint32_t other = __ballot_sync(0xffffffffu, t + lane <= last && a.req[min(t + lane, last)] != a.req[t0]);
          if (other) {
            end = t + __ffs(other) - 2;
            break;
          }
        }
        if (lane == 0) give(item_of(R0, t0, end, half));
        __syncwarp();
        ++n;
      }
      id = -1;
      if (!a.take) break;
      if (lane == 0) {
        // not before: what is taken early may be a long tile that another CTA could begin sooner
        for (uint32_t spins = 0; *reinterpret_cast<volatile int*>(&m.near_end) < (int)n && !*dead; ++spins) {
          __nanosleep(64);
          if (spins > kWaitSpins) *dead = 1;
        }
        if (!*dead) {
          fence_proxy_async_smem();  // the last answer has been read
          mbar_expect_tx(&m.taken, 16);
          lt_take_next(&m.answer, &m.taken);
          if (mbar_wait_bounded(&m.taken, asked & 1, dead)) id = lt_taken(&m.answer);
          else mbar_drain(&m.taken, asked & 1);
        }
      }
      ++asked;
      id = __shfl_sync(0xffffffffu, id, 0);
    }
    if (lane == 0) {
      LtItem none{};
      none.R0 = -1;
      give(none);
    }
    __syncwarp();
  } else if (warp > LT_SOFT / 32) {
    // Loads: two warps take the other chunks in turn (one of them their Q), one warp each the value chunks.  One thread of a warp issues (the operands of a
    // copy are uniform registers: with a lane per page the compiler walked through the lanes, about 200 clocks each), which takes 400 clocks for the four
    // pages of a chunk; page numbers are looked up a block ahead.
    if (tc_elect_one()) {
      const int me = warp - LT_SOFT / 32 - 1, v = me - LT_LOAD_O;
      const bool values = v >= 0;
      const int box = min(a.page_size, LT_KEYS), pieces = LT_KEYS / box;
      uint32_t n = 0, q = 0, place = 0, par = 1;  // blocks and queries so far; the ring's next place and its parity
      bool go = true;  // false behind a run-out: a barrier must not be armed twice in one phase
      LtItem r;
      for (uint32_t k = 0; go && item(k, r); ++k) {
        mbar_arrive(m.item_empty + k % LT_QUEUE);
        const int vc0 = r.vc0;
        const int* pg = a.pages + r.pages;
        const int nb = blocks_of(r), last = (r.end - 1) / a.page_size;
        if (nb <= 0) {
          if (v == 0) *reinterpret_cast<volatile int*>(&m.near_end) = (int)k + 1;
          continue;
        }
        if (me == 0) {
          if (q > 0 && !mbar_wait_bounded(&m.q_empty, (q - 1) & 1, dead)) break;
          mbar_expect_tx(&m.q_full, (uint32_t)(n_other * LT_QC));
          for (int x = 0; x < n_other; ++x) tma_load_2d(Qs + (size_t)x * LT_QC, &map_q, (x < vc0 ? x : x + nvc) * 64, r.R0, &m.q_full);
        }
        ++q;
        int next[8];
        auto look_up = [&](int b) {
          const int p0 = (r.k0 + b * LT_KEYS) / a.page_size;
#pragma unroll
          for (int j = 0; j < 8; ++j) next[j] = j < pieces ? pg[min(p0 + j, last)] : 0;  // behind the end: the last page again (masked)
        };
        look_up(0);
        for (int b = 0; b < nb && go; ++b, ++n) {
          const int slot = (r.k0 + b * LT_KEYS) & (a.page_size - 1);
          int page[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) page[j] = next[j];
          if (b + 1 < nb) look_up(b + 1);
          auto copy = [&](uint8_t* dst, int c, uint64_t* bar) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (j < pieces) lt_tma_3d(dst + j * box * 128, &map_k, c * 64, slot, page[j], bar);
          };
          if (values) {
            if (v >= nvc) continue;
            go = mbar_wait_bounded(m.v_empty + (n & 1), ((n >> 1) & 1) ^ 1, dead);
            if (!go) break;
            if (v == 0 && b == max(nb - 2, 0)) *reinterpret_cast<volatile int*>(&m.near_end) = (int)k + 1;
            if (v == 0) mbar_expect_tx(m.v_full + (n & 1), (uint32_t)(nvc * LT_KC));  // (the other warps' bytes may be counted before)
            copy(Vs + (size_t)((n & 1) * nvc + v) * LT_KC, vc0 + v, m.v_full + (n & 1));
          } else {
            for (int x = 0; x < n_other && go; ++x) {
              if ((x & 1) == me) {
                go = mbar_wait_bounded(m.k_empty + place, par, dead);
                if (!go) break;
                if (x == 0) mbar_expect_tx(m.k_full + (n & 1), (uint32_t)(n_other * LT_KC));
                copy(Ks + (size_t)place * LT_KC, x < vc0 ? x : x + nvc, m.k_full + (n & 1));
              }
              if (++place == (uint32_t)ring) {
                place = 0;
                par ^= 1u;
              }
            }
          }
        }
      }
    }
    __syncwarp();
    // Behind a run-out no barrier says when the copies under way have landed: two milliseconds, where a copy takes a thousandth of that
    if (*dead)
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncwarp();
  } else if (warp == LT_SOFT / 32) {
    if (tc_elect_one()) {
      // instruction descriptors: D = f32, A = B = bf16, A K-major; S: N = 64, B K-major; P V: N = 64 nvc, B (= V) N-major
      constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_ROWS >> 4) << 24);
      constexpr uint32_t idesc_s = base | ((uint32_t)(LT_KEYS >> 3) << 17);
      const uint32_t idesc_pv = base | (1u << 16) | ((uint32_t)(nvc * 8) << 17);
      uint32_t place = 0;
      auto issue_s = [&](uint32_t n) {  // (a wait costs 200 clocks even where there is nothing to wait for: one for all other chunks of a block)
        const uint32_t d = tmem + (n & 1) * LT_KEYS;
        if (n_other > 0) mbar_wait_bounded(m.k_full + (n & 1), (n >> 1) & 1, dead);
        tc_fence_after();
        for (int x = 0; x < n_other; ++x) {
          const uint64_t qd = make_sw128_desc(smem_u32(Qs + (size_t)x * LT_QC)), kd = make_sw128_desc(smem_u32(Ks + (size_t)place * LT_KC));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(d, qd + (uint64_t)(k * 2), kd + (uint64_t)(k * 2), idesc_s, (x > 0 || k > 0) ? 1u : 0u);
          umma_commit(m.k_empty + place);
          if (++place == (uint32_t)ring) place = 0;
        }
        mbar_wait_bounded(m.v_full + (n & 1), (n >> 1) & 1, dead);
        tc_fence_after();
        for (int v = 0; v < nvc; ++v) {
          const uint64_t kd = make_sw128_desc(smem_u32(Vs + (size_t)((n & 1) * nvc + v) * LT_KC));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_tmem_a(d, tmem + 128 + (uint32_t)(v * 32 + k * 8), kd + (uint64_t)(k * 2), idesc_s, (n_other > 0 || v > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(m.s_full + (n & 1));
      };
      uint32_t n = 0, q = 0;  // blocks and queries so far
      LtItem r;
      for (uint32_t k = 0; item(k, r); ++k) {
        mbar_arrive(m.item_empty + k % LT_QUEUE);
        const uint32_t end = n + (uint32_t)max(blocks_of(r), 0), first = n;
        if (n == end) continue;
        mbar_wait_bounded(&m.q_full, q & 1, dead);
        mbar_wait_bounded(&m.q_tmem, q++ & 1, dead);
        issue_s(n);
        if (n + 1 == end) umma_commit(&m.q_empty);
        for (; n < end; ++n) {
          if (n + 1 < end) {
            issue_s(n + 1);
            if (n + 2 == end) umma_commit(&m.q_empty);  // the item's last scores: then the next one's queries may come
          }
          mbar_wait_bounded(m.p_ready + (n & 1), (n >> 1) & 1, dead);
          tc_fence_after();
          const uint64_t vd = make_sw128_mn_desc(smem_u32(Vs + (size_t)((n & 1) * nvc) * LT_KC), LT_KC, 1024);
#pragma unroll
          for (int k = 0; k < LT_KEYS / 16; ++k)
            umma_bf16_tmem_a(tmem + 256, tmem + (n & 1) * LT_KEYS + (uint32_t)(k * 8), vd + (uint64_t)(k * (2048 >> 4)), idesc_pv, (n > first || k > 0) ? 1u : 0u);
          umma_commit(m.v_empty + (n & 1));
          umma_commit(&m.pv_done);
        }
      }
      if (*dead) {
        umma_commit(&m.done);
        mbar_drain(&m.done, 0);
      }
    }
    __syncwarp();
  } else {
    // a thread has half a row: 32 of the block's keys, and half of the CTA's output columns
    const int row = threadIdx.x & (LT_ROWS - 1), side = threadIdx.x >> 7, ow = nvc * 32;
    const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16), t_o = t_lane + 256 + side * ow;
    auto both_halves = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory"); };  // the two warps of 32 rows
    auto both_have = [&](bool x) {  // (behind a run-out the two could part, and wait for each other)
      uint32_t y;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, %2, 64, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(y)
                   : "r"((uint32_t)x), "r"(1 + (warp & 3))
                   : "memory");
      return y != 0;
    };
    // the value chunks' Q of an item, once the last one's scores are complete
    auto put_q = [&](const LtItem& r) {
      const int R = r.R0 + (warp & 3) * 32 + (lane & ~3);  // four lanes read 64 bytes of a row at a time: a lane by itself would touch a line per 16 bytes
      for (int c = side; c < nvc; c += 2) {
        uint32_t t[32];
        const bf16* src = a.qa + (size_t)R * a.D + (r.vc0 + c) * 64 + (lane & 3) * 8;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const uint4 u = R + (x & 3) < total ? *reinterpret_cast<const uint4*>(src + (size_t)(x & 3) * a.D + (x >> 2) * 32) : make_uint4(0, 0, 0, 0);
          t[4 * x] = u.x;
          t[4 * x + 1] = u.y;
          t[4 * x + 2] = u.z;
          t[4 * x + 3] = u.w;
        }
        transpose4(t, lane);
        transpose4(t + 16, lane);
        tmem_put32(t_lane + 128 + c * 32, t);
      }
      tmem_put_wait();
      tc_fence_before();
      mbar_arrive(&m.q_tmem);
    };
    uint32_t n = 0, k = 0;
    auto next_item = [&](LtItem& r) {
      const bool more = item(k, r);
      __syncwarp();
      if (!both_have(more)) return false;
      if (lane == 0) mbar_arrive(m.item_empty + k % LT_QUEUE);
      ++k;
      if (blocks_of(r) > 0) put_q(r);
      return true;
    };
    LtItem r, ahead;
    for (bool more = next_item(r); more; r = ahead) {
      const int R = r.R0 + row, tok = R < total ? R / a.heads : -1, nb = blocks_of(r);
      const bool act = tok >= r.t0 && tok <= r.t1;
      const int my_pos = act ? a.pos[tok] : -1, my_lo = a.window > 0 ? my_pos - a.window + 1 : 0;
      float mx = -INFINITY, l = 0.f;  // running maximum of the row (scaled, log2 units) and sum of the half
      for (int b = 0; b < nb; ++b, ++n) {
        const int j0 = r.k0 + b * LT_KEYS, h0 = j0 + side * 32;
        mbar_wait_bounded(m.s_full + (n & 1), (n >> 1) & 1, dead);
        __syncwarp();
        tc_fence_after();
        const uint32_t t_s = t_lane + (n & 1) * LT_KEYS;
        uint32_t v[32];
        tmem_ld32(t_s + side * 32, v);
        // visible keys of this row in the half block: [c0, c1)
        const int c0 = act ? max(my_lo - h0, 0) : 32, c1 = act ? my_pos + 1 - h0 : 0;
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (!__all_sync(0xffffffffu, c0 == 0 && c1 >= 32)) {
#pragma unroll
          for (int x = 0; x < 32; ++x)
            if (x < c0 || x >= c1) v[x] = 0xff800000u;  // -inf
        }
#pragma unroll
        for (int x = 0; x < 32; ++x) m4[x & 3] = fmaxf(m4[x & 3], __uint_as_float(v[x]));
        const float own = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale_log2;
        m.top[n & 1][threadIdx.x] = own;
        tc_fence_before();  // both have read their scores: P may take their place
        both_halves();
        tc_fence_after();
        const float blk = fmaxf(own, m.top[n & 1][threadIdx.x ^ LT_ROWS]);
        const bool grow = blk > mx, any = __any_sync(0xffffffffu, grow);
        const float to = grow ? blk : mx, corr = grow ? lt_exp2(mx - to) : 1.f;
        mx = to;
        const float ref = mx == -INFINITY ? 0.f : mx;  // a row without a key so far: every p is 2^-inf = 0
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t p[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          const float p0 = lt_exp2(fmaf(__uint_as_float(v[x]), a.scale_log2, -ref)), p1 = lt_exp2(fmaf(__uint_as_float(v[x + 1]), a.scale_log2, -ref));
          s4[x & 2] += p0;
          s4[(x & 2) + 1] += p1;
          p[x / 2] = pack_bf16(p0, p1);
        }
        l = l * corr + ((s4[0] + s4[1]) + (s4[2] + s4[3]));
        tmem_put16(t_s + side * 16, p);
        if (any && b > 0) {  // O holds the blocks before this one, once their last P V is through
          // (blocks whose pv_done this thread did not wait for have left the barrier no phase behind: the P V of block n - 2 was complete when these scores were)
          mbar_wait_bounded(&m.pv_done, (n - 1) & 1, dead);
          __syncwarp();
          tc_fence_after();
          for (int c = 0; c < ow; c += 32) {
            uint32_t t[32];
            tmem_ld32(t_o + c, t);
#pragma unroll
            for (int x = 0; x < 32; ++x) t[x] = __float_as_uint(__uint_as_float(t[x]) * corr);
            tmem_put32(t_o + c, t);
          }
        }
        tmem_put_wait();
        if (j0 < r.lo || j0 + LT_KEYS > r.end) {  // clear the value rows of keys that are not the run's
          const int rr = threadIdx.x & 63, key = j0 + rr;
          if (key < r.lo || key >= r.end)
            for (int c = threadIdx.x >> 6; c < nvc; c += LT_SOFT / 64) {
              uint4* z = reinterpret_cast<uint4*>(Vs + (size_t)((n & 1) * nvc + c) * LT_KC + rr * 128);
#pragma unroll
              for (int y = 0; y < 8; ++y) z[y] = make_uint4(0, 0, 0, 0);
            }
          fence_proxy_async_smem();
        }
        tc_fence_before();
        mbar_arrive(m.p_ready + (n & 1));
      }
      more = next_item(ahead);  // its first scores are computed under what follows
      // ---- O / l -> bf16, the rows of this item (the next one's first P V waits for all threads' next p_ready)
      if (nb > 0) mbar_wait_bounded(&m.pv_done, (n - 1) & 1, dead);
      __syncwarp();
      tc_fence_after();
      m.sum[threadIdx.x] = l;
      both_halves();
      l += m.sum[threadIdx.x ^ LT_ROWS];
      both_halves();  // (before the next item's)
      const float sk = a.sink && act ? bf2f(a.sink[R % a.heads]) * 1.4426950408889634f : -INFINITY;
      const float M = fmaxf(mx, sk), w = lt_exp2(mx - M);
      const float inv = w / (l * w + (a.sink ? lt_exp2(sk - M) : 0.f));
      const uint32_t rows = __ballot_sync(0xffffffffu, act);
      bf16* dst = a.out + (size_t)(r.R0 + (warp & 3) * 32 + (lane & ~3)) * a.rank + r.vc0 * 64 + side * ow + (lane & 3) * 8;
      for (int c = 0; c < ow; c += 32) {
        uint32_t t[32] = {}, u[16];
        if (nb > 0) tmem_ld32(t_o + c, t);  // no visible key at all (a position before the first): O is zero, as the sum is
#pragma unroll
        for (int x = 0; x < 16; ++x) u[x] = pack_bf16(__uint_as_float(t[2 * x]) * inv, __uint_as_float(t[2 * x + 1]) * inv);
        transpose4(u, lane);
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (rows >> ((lane & ~3) + x) & 1)
            *reinterpret_cast<uint4*>(dst + (size_t)x * a.rank + c) = make_uint4(u[4 * x], u[4 * x + 1], u[4 * x + 2], u[4 * x + 3]);
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) count_run_out(dead, a.err);
  if (warp == LT_SOFT / 32) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace

// 0 = launched; -2 = shape / alignment outside this kernel (the caller runs the mma.sync kernel)
int launch_latent_attention_tc(const bf16* qa, const bf16* cache, const bf16* sink, const int* pos, const int* req, const int* page_off, const int* pages,
                               bf16* out, long page_stride, int page_size, int tokens, int heads, int rank, int rot, float scale, int window,
                               int max_kv_len, cudaStream_t st) {
  const int D = rank + rot, nc = (D + 63) / 64, halves = (rank / 64 + LT_VC - 1) / LT_VC;
  // (rot % 16, rank <= 512: what the mma.sync kernel takes too.  The shapes beyond go to the generic kernel, whose weights stay fp32.)
  if (rank % 64 || rot % 16 || rank > 512 || nc > LT_MAXC || page_size < 8 || (page_size & (page_size - 1)) || page_stride % 8 || !(scale > 0.f) ||
      ((reinterpret_cast<uintptr_t>(qa) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -2;
  const long rows = (long)tokens * heads, tiles = (rows + LT_ROWS - 1) / LT_ROWS;
  if (tiles * halves > 0x3fffffff || rows > 0x7fffffff) return -2;
  const int v0 = rank / 64 < LT_VC ? rank / 64 : LT_VC, v1 = halves == 1 ? v0 : rank / 64 - LT_VC;  // value chunks of the halves
  // Few CTAs: the key axis has to be cut, which the mma.sync kernel does, unless contexts are short.  This kernel takes 11 us and 1.3 to 1.5 for every 64
  // keys of the longest context; that one 11 and, for every 16 rows of 64 keys, 0.05 (latent 512), 0.02 (256) or 0.007 (128), so that short contexts cancel
  // out and the number of rows decides.  Up to 512 keys a request that is longer than all others costs little here (140 decoding, one of them
  // at 510, latent 512 + 64, 8 heads, 33.3 31.2), and one CTA in twelve SMs is enough; latents below 128 and unequal halves, which gain less, take one
  // in six.  One or two blocks of keys are one pass in that kernel while its CTAs, one to an SM above latents of 256, fit at once.  Us, 16 heads, 512 + 64, that kernel and this one: 200 tokens 51.7 16.8, 150 37.4 14.9,
  // 100 behind 400 keys 57.9 23.1, 80 decoding at 480 55.8 39.3; 8 heads, 500 tokens 92.7 23.0; latent 256 + 32, 16 heads, 200 tokens 27.0 14.8.
  const int keys = window > 0 && window + (long)tokens < max_kv_len ? window + tokens : max_kv_len;
  const bool few_keys = keys <= 8 * LT_KEYS && (keys > 2 * LT_KEYS || (keys > LT_KEYS && rank > 256 && rows > 16l * sm_count()));
  if (tiles * halves < sm_count() / (!few_keys ? 2 : rank < 128 || v0 != v1 ? 6 : 12)) return -2;
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
  // Runs that start inside a tile are for the helpers, one CTA per half and SM (more where a helper would have over LT_SCAN tokens to look at); none
  // where each token fills whole tiles.  They come first, since their contexts may be the longest, unless all CTAs fit at once.
  int helpers = heads % LT_ROWS == 0 ? 0 : (sm_count() + halves - 1) / halves;
  if (helpers > 0 && helpers < (tokens + LT_SCAN - 1) / LT_SCAN) helpers = (tokens + LT_SCAN - 1) / LT_SCAN;
  const size_t b0 = lt_bytes(nc - v0, v0), b1 = lt_bytes(nc - v1, v1), smem = (b0 > b1 ? b0 : b1) + sizeof(LtSmem) + 1024, most = 216 * 1024 + sizeof(LtSmem) + 1024;
  static_assert(most <= 227 * 1024, "shared memory");
  static std::atomic<uint64_t> smem_set{0};
  if (allow_smem(smem_set, (const void*)latent_attention_tc_kernel, most) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  const LtArgs a{qa, sink, pos, req, page_off, pages, out, page_size, tokens, heads, rank, D, nc, halves, window, helpers, tiles * halves > sm_count(), v0 == v1, scale * 1.4426950408889634f, wait_err_word()};
  return (int)launch(latent_attention_tc_kernel, dim3((unsigned)((tiles + helpers) * halves)), dim3(LT_THREADS), smem, st, true, mq, mk, a);
}

}  // namespace pk
