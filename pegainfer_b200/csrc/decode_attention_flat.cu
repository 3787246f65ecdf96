// Fused decode attention of a batch with many cached tokens: every SM gets the same number of pages.
//
// A cluster of CTAs per (request, kv head) (decode_attention_tma.cu) leaves SMs idle when there are more such pairs than SMs: contexts differ, and the
// pairs that do not fit wait for a second round.  Here the pages of all requests, one after the other as `page_indices` lists them, are cut into
// gridDim.x equal runs, one per CTA, and a CTA's eight warps are the eight kv heads: together they read whole pages (64 KB in one place), a warp walks its
// head's tiles by itself -- a ring of three 8 KB tiles, no barrier between warps -- and keeps the online softmax of the group's four query heads.  Where a
// run begins or ends inside a request, the warp leaves its state in `partial` (at most two places per CTA, the request's first piece of a run in the
// first); the warp that counts the request's last piece adds them up.  Tiles, products, rounding points and the step's own row as in
// decode_attention_tma.cu.
// Bound by the pages' bytes: the walk itself runs at the copy rate (24 requests of 650 to 2600 cached tokens, 173 MB: 26 us), beside 8 us from the launch to
// the first tile and 3 for the last states.  B200, us, cold, with a launch gap of 12, clusters -> here: 24 requests of 650 to 2600 tokens 62 -> 53, 64 of 750
// to 3000 115 -> 109, 48 of 150 to 600 42 -> 34, 64 of up to 100 36 -> 24; the attention block of a 4B layer around the first 70.6 -> 63.4.
#include "decode_attention_cluster.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int F_HD = 128, F_GROUP = 4, F_PAGE = 16, F_WARPS = 8, F_THREADS = F_WARPS * 32;
constexpr int F_TILE = 4 * kDaHalf;    // K lo | K hi | V lo | V hi (V first where it lies first in the pool)
constexpr int F_SLOTS = 3;
constexpr int F_MIN_PAGES = 2;        // pages of a CTA at least

struct FlatArgs {
  const bf16 *q, *k_new, *v_new;
  bf16 *out, *kv;
  int64_t k_off, v_off, stride_page;
  const int *page_indices, *page_indptr, *last_page_len, *positions;
  const bf16 *qw, *kw, *cosc, *sinc;
  float eps, sm_scale_log2;
  int bs, k_at;  // k_at: K in a tile (bytes)
  float* partial;  // [2 gridDim.x][32 heads][128] outputs, then as many (maximum, sum)
  int* counters;   // [bs][8]
  unsigned int* err;
};

__device__ __forceinline__ void f_tma_page(uint32_t dst, const CUtensorMap* map, int head, int page, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3, %2, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(0), "r"(2 * head), "r"(page), "r"(smem_u32(bar))
      : "memory");
}

__global__ void __launch_bounds__(F_THREADS, 1) decode_attention_flat_kernel(const __grid_constant__ CUtensorMap map, const FlatArgs a) {
  extern __shared__ uint8_t f_smem_raw[];
  constexpr int NQ = F_WARPS * F_GROUP;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(f_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int head = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  uint8_t* tiles = smem + (size_t)head * F_SLOTS * F_TILE;
  bf16* q_s = reinterpret_cast<bf16*>(smem + (size_t)F_WARPS * F_SLOTS * F_TILE) + head * (F_GROUP + 2) * F_HD;  // [4][128], then the step's k and v
  bf16 *k_s = q_s + F_GROUP * F_HD, *v_s = k_s + F_HD;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)F_WARPS * F_SLOTS * F_TILE + F_WARPS * (F_GROUP + 2) * F_HD * 2) + head * F_SLOTS;
  __shared__ int dead_flag;
  volatile int* dead = &dead_flag;
  if (threadIdx.x == 0) *dead = 0;
  if (lane == 0) {
    for (int s = 0; s < F_SLOTS; ++s) mbar_init(full + s, 1);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  // this CTA's run of pages.  The lanes hold the requests w0 .. w0 + 31 of the batch: all that the pieces need is loaded at once
  int w0 = 0, w_ptr = 0, w_len = 0, w_pos = 0;
  auto window = [&](int from) {
    w0 = from;
    const int r = min(from + lane, a.bs - 1);
    w_ptr = a.page_indptr[r + 1];
    w_len = a.last_page_len[r];
    w_pos = a.positions[r];
  };
  window(0);
  const int base = a.page_indptr[0], total = a.page_indptr[a.bs] - base;
  const int n = max(1, min((int)gridDim.x, total / F_MIN_PAGES)), me = blockIdx.x;
  auto run_start = [&](int i) { return (int)((int64_t)i * total / n); };
  auto owner = [&](int page) { return (int)(((int64_t)(page + 1) * n + total - 1) / total) - 1; };
  const int start = me < n ? run_start(me) : 0, count = me < n ? run_start(me + 1) - start : 0;
  const int* pages = a.page_indices + base + start;
  auto issue = [&](int i, int page) {  // one lane
    const int s = i % F_SLOTS;
    mbar_expect_tx(full + s, F_TILE);
    f_tma_page(smem_u32(tiles + (size_t)s * F_TILE), &map, head, page, full + s);
  };
  if (lane == 0) {  // cached rows do not depend on the previous kernel
    int pg[F_SLOTS];
#pragma unroll
    for (int i = 0; i < F_SLOTS; ++i) pg[i] = i < count ? __ldg(pages + i) : 0;
#pragma unroll
    for (int i = 0; i < F_SLOTS; ++i)
      if (i < count) issue(i, pg[i]);
  }
  // the request that holds page `at`, from request b on (requests without a page lie between)
  auto find = [&](int b, int at) {
    for (;;) {
      if (b < w0 || b >= w0 + 32) window(b);
      const unsigned behind = __ballot_sync(0xffffffffu, w0 + lane >= b && w0 + lane < a.bs && w_ptr - base > at);
      if (behind) return w0 + __ffs(behind) - 1;
      b = w0 + 32;
    }
  };
  const uint2 qw = reinterpret_cast<const uint2*>(a.qw)[lane], kw = reinterpret_cast<const uint2*>(a.kw)[lane];
  int b = count > 0 ? find(0, start) : 0, b_first = 0, pos = 0, len16 = 0;
  uint2 cr, sr;
  auto enter = [&] {  // what is known of request b without the previous kernel
    const int j = b - w0;
    b_first = j > 0 ? __shfl_sync(0xffffffffu, w_ptr, j - 1) : a.page_indptr[b];
    pos = __shfl_sync(0xffffffffu, w_pos, j);
    len16 = __shfl_sync(0xffffffffu, w_len, j);
    cr = *reinterpret_cast<const uint2*>(a.cosc + (size_t)pos * F_HD + (lane & 15) * 4);
    sr = *reinterpret_cast<const uint2*>(a.sinc + (size_t)pos * F_HD + (lane & 15) * 4);
  };
  if (count > 0) enter();
  pdl_wait();  // q, k_new, v_new come from the projection

  for (int z = me; z < a.bs; z += gridDim.x)  // requests without a page
    if (a.page_indptr[z + 1] == a.page_indptr[z])
      for (int h = 0; h < F_GROUP; ++h) reinterpret_cast<uint2*>(a.out + ((size_t)z * NQ + head * F_GROUP + h) * F_HD)[lane] = make_uint2(0, 0);

  // ldmatrix addressing (matrix lane / 8, row lane % 8)
  const int lm_i = lane >> 3, lm_r = lane & 7;
  const int k_tok = ((lm_i >> 1) << 3) + lm_r, k_c = lm_i & 1, v_tok = ((lm_i & 1) << 3) + lm_r, v_c = lm_i >> 1;
  int i = 0;  // page of the run
  uint32_t par = 0;
  int slot = 0;
  while (i < count) {
    // ---- a piece: the run's pages of request b
    if (i > 0) {
      b = find(b + 1, start + i);
      enter();
    }
    const int first = b_first - base, last = __shfl_sync(0xffffffffu, w_ptr, b - w0) - base;  // the request's pages
    const int piece = start + i, end = min(last, start + count);
    const int len = (last - first - 1) * F_PAGE + len16, own = pos >> 4 < (len + F_PAGE - 1) / F_PAGE ? first + (pos >> 4) : -1;  // own: the page of the step's row
    {
      const uint2* q = reinterpret_cast<const uint2*>(a.q + ((size_t)b * NQ + head * F_GROUP) * F_HD);
      uint2 raw[F_GROUP];
#pragma unroll
      for (int h = 0; h < F_GROUP; ++h) raw[h] = q[h * 32 + lane];
#pragma unroll
      for (int h = 0; h < F_GROUP; ++h) da_norm_rope(raw[h], qw, cr, sr, a.eps, q_s + h * F_HD, lane);
      if (own >= piece && own < end) {
        const size_t row = ((size_t)b * F_WARPS + head) * F_HD;
        const uint2 kr = reinterpret_cast<const uint2*>(a.k_new + row)[lane], vr = reinterpret_cast<const uint2*>(a.v_new + row)[lane];
        da_norm_rope(kr, kw, cr, sr, a.eps, k_s, lane);
        reinterpret_cast<uint2*>(v_s)[lane] = vr;
        __syncwarp();
        const int64_t dst = (int64_t)pages[own - start] * a.stride_page + ((int64_t)(pos & 15) * F_WARPS + head) * F_HD;
        reinterpret_cast<uint2*>(a.kv + a.k_off + dst)[lane] = reinterpret_cast<uint2*>(k_s)[lane];
        reinterpret_cast<uint2*>(a.kv + a.v_off + dst)[lane] = vr;
      }
    }
    __syncwarp();
    uint32_t qa[8][2];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      qa[kk][0] = g < F_GROUP ? *reinterpret_cast<const uint32_t*>(q_s + g * F_HD + kk * 16 + 2 * tq) : 0u;
      qa[kk][1] = g < F_GROUP ? *reinterpret_cast<const uint32_t*>(q_s + g * F_HD + kk * 16 + 8 + 2 * tq) : 0u;
    }
    float o[16][4];
#pragma unroll
    for (int d = 0; d < 16; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    float m_run = -INFINITY, l_run = 0.f;
    for (; start + i < end; ++i) {
      const int at = start + i;  // page
      const int refill = i + F_SLOTS < count ? __ldg(pages + i + F_SLOTS) : 0;  // looked up while this page is worked on
      mbar_wait_bounded(full + slot, par, dead);
      __syncwarp();
      uint8_t* k_tile = tiles + (size_t)slot * F_TILE + a.k_at;
      uint8_t* v_tile = tiles + (size_t)slot * F_TILE + (2 * kDaHalf - a.k_at);
      if (at == own) {  // the step's own row: the copy may have come before it was written
        const int r = pos & 15;
        if (lane < 16) *reinterpret_cast<uint4*>(k_tile + da_at(r, lane)) = reinterpret_cast<const uint4*>(k_s)[lane];
        else *reinterpret_cast<uint4*>(v_tile + da_at(r, lane - 16)) = reinterpret_cast<const uint4*>(v_s)[lane - 16];
      }
      if (at == last - 1 && len16 < F_PAGE)  // rows past the context (a page may be there before its first token): V zero, so that 0 times what lies there stays 0
        for (int x = lane; x < (F_PAGE - len16) * 16; x += 32) *reinterpret_cast<uint4*>(v_tile + da_at(len16 + (x >> 4), x & 15)) = make_uint4(0, 0, 0, 0);
      __syncwarp();
      const uint32_t kt = smem_u32(k_tile), vt = smem_u32(v_tile);
      float s[2][4] = {}, s1[2][4] = {};  // even and odd k steps apart: half as long a chain
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t r[4];
        da_ldsm4(kt + da_at(k_tok, kk * 2 + k_c), r);
        da_mma(kk & 1 ? s1[0] : s[0], qa[kk][0], qa[kk][1], r[0], r[1]);
        da_mma(kk & 1 ? s1[1] : s[1], qa[kk][0], qa[kk][1], r[2], r[3]);
      }
      const int tb = (at - first) * F_PAGE + 2 * tq;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[j][0] = tb + j * 8 < len ? (s[j][0] + s1[j][0]) * a.sm_scale_log2 : -INFINITY;
        s[j][1] = tb + j * 8 + 1 < len ? (s[j][1] + s1[j][1]) * a.sm_scale_log2 : -INFINITY;
        mx = fmaxf(mx, fmaxf(s[j][0], s[j][1]));
      }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run, mx), m_safe = m_new == -INFINITY ? 0.f : m_new, alpha = da_ex2(m_run - m_safe);
      m_run = m_new;
      uint32_t ph[2], pl[2];  // P = hi + lo, bf16 each: 16 bits of p
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float p0 = da_ex2(s[j][0] - m_safe), p1 = da_ex2(s[j][1] - m_safe);
        sum += p0 + p1;
        ph[j] = pack_bf16(p0, p1);
        pl[j] = pack_bf16(p0 - bf16_lo(ph[j]), p1 - bf16_hi(ph[j]));
      }
      l_run = l_run * alpha + sum;
#pragma unroll
      for (int d = 0; d < 16; ++d) {
        o[d][0] *= alpha;
        o[d][1] *= alpha;
      }
#pragma unroll
      for (int dp = 0; dp < 8; ++dp) {
        uint32_t r[4];
        da_ldsm4_t(vt + da_at(v_tok, dp * 2 + v_c), r);
        da_mma(o[2 * dp], ph[0], ph[1], r[0], r[1]);
        da_mma(o[2 * dp + 1], ph[0], ph[1], r[2], r[3]);
        da_mma(o[2 * dp], pl[0], pl[1], r[0], r[1]);
        da_mma(o[2 * dp + 1], pl[0], pl[1], r[2], r[3]);
      }
      __syncwarp();
      if (i + F_SLOTS < count && lane == 0 && !*dead) {
        fence_proxy_async_smem();
        issue(i + F_SLOTS, refill);
      }
      if (++slot == F_SLOTS) {
        slot = 0;
        par ^= 1u;
      }
    }
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    const size_t row0 = (size_t)b * NQ + head * F_GROUP;
    if (piece == first && end == last) {  // the whole request
      if (g < F_GROUP)
#pragma unroll
        for (int d = 0; d < 16; ++d)
          *reinterpret_cast<uint32_t*>(a.out + (row0 + g) * F_HD + d * 8 + 2 * tq) = l_run > 0.f ? pack_bf16(__fdividef(o[d][0], l_run), __fdividef(o[d][1], l_run)) : 0u;
      continue;
    }
    const int place = 2 * me + (piece == start ? 0 : 1);
    float* po = a.partial + ((size_t)place * NQ + head * F_GROUP) * F_HD;
    float* pm = a.partial + (size_t)2 * gridDim.x * NQ * F_HD;  // [place][head][2]
    if (g < F_GROUP) {
#pragma unroll
      for (int d = 0; d < 16; ++d) *reinterpret_cast<float2*>(po + g * F_HD + d * 8 + 2 * tq) = make_float2(o[d][0], o[d][1]);
      if (tq == 0) *reinterpret_cast<float2*>(pm + ((size_t)place * NQ + head * F_GROUP + g) * 2) = make_float2(m_run, l_run);
    }
    __threadfence();
    __syncwarp();
    const int c0 = owner(first), pieces = owner(last - 1) - c0 + 1;
    int before = 0;
    if (lane == 0) before = atomicAdd(a.counters + b * F_WARPS + head, 1);
    if (__shfl_sync(0xffffffffu, before, 0) != pieces - 1) continue;
    __threadfence();
    if (lane == 0) a.counters[b * F_WARPS + head] = 0;
    const int skip = run_start(c0) == first ? 0 : 1;  // the first piece's place in its CTA
    auto place_of = [&](int p) { return 2 * (c0 + p) + (p == 0 ? skip : 0); };
    float4 acc[F_GROUP] = {};
    float M[F_GROUP], L[F_GROUP] = {};
#pragma unroll
    for (int h = 0; h < F_GROUP; ++h) M[h] = -INFINITY;
    for (int p = lane; p < pieces; p += 32)
#pragma unroll
      for (int h = 0; h < F_GROUP; ++h) M[h] = fmaxf(M[h], __ldcg(pm + ((size_t)place_of(p) * NQ + head * F_GROUP + h) * 2));
#pragma unroll
    for (int h = 0; h < F_GROUP; ++h) M[h] = warp_max(M[h]);
#pragma unroll 2
    for (int p = 0; p < pieces; ++p) {
      const size_t at = (size_t)place_of(p) * NQ + head * F_GROUP;
#pragma unroll
      for (int h = 0; h < F_GROUP; ++h) {
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(pm + (at + h) * 2));
        const float4 x = __ldcg(reinterpret_cast<const float4*>(a.partial + (at + h) * F_HD) + lane);
        const float w = ml.x == -INFINITY ? 0.f : da_ex2(ml.x - M[h]);
        L[h] = fmaf(ml.y, w, L[h]);
        acc[h] = make_float4(fmaf(x.x, w, acc[h].x), fmaf(x.y, w, acc[h].y), fmaf(x.z, w, acc[h].z), fmaf(x.w, w, acc[h].w));
      }
    }
#pragma unroll
    for (int h = 0; h < F_GROUP; ++h)
      reinterpret_cast<uint2*>(a.out + (row0 + h) * F_HD)[lane] =
          L[h] > 0.f ? make_uint2(pack_bf16(__fdividef(acc[h].x, L[h]), __fdividef(acc[h].y, L[h])), pack_bf16(__fdividef(acc[h].z, L[h]), __fdividef(acc[h].w, L[h])))
                     : make_uint2(0, 0);
  }
  if (*dead)  // copies under way: their barriers were armed in order
    for (int s = 0; s < F_SLOTS; ++s) {
      mbar_drain(full + s, 0);
      mbar_drain(full + s, 1);
    }
  __syncthreads();
  if (threadIdx.x == 0) count_run_out(dead, a.err);
}

// {64 columns, slot, half of a kv head, K or V (whichever lies first), page}; box = K and V of one page of one head as four half tiles, 128-byte swizzle
bool make_flat_map(CUtensorMap* map, const bf16* kv, int64_t k_off, int64_t v_off, int64_t stride_page) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const int64_t first = k_off < v_off ? k_off : v_off, apart = k_off < v_off ? v_off - k_off : k_off - v_off;
  cuuint64_t dims[5] = {64, (cuuint64_t)F_PAGE, (cuuint64_t)F_WARPS * 2, 2, (cuuint64_t)1 << 20};  // page ids come from the page table
  cuuint64_t strides[4] = {(cuuint64_t)F_WARPS * F_HD * 2, 128, (cuuint64_t)apart * 2, (cuuint64_t)stride_page * 2};
  cuuint32_t box[5] = {64, (cuuint32_t)F_PAGE, 2, 2, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(kv + first), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Taken when there are more (request, kv head) pairs than SMs: up to there the pairs' clusters run at once, and their merge is the cheaper one.
// B200, us, clusters / here: 16 requests of 650 to 2600 tokens 43.0 / 44.8, 8 28.7 / 36.9; 20 58.8 / 47.6, 20 of 75 to 300 23.3 / 24.4, 24 19.5 / 19.4 (16 tokens).
// 0 = launched, a cudaError, or -2: not a call for this kernel.  `partial` holds `places` states of 32 heads x 130 floats.
int launch_decode_attention_flat(const ClusterAttnArgs& c, int nkv, int bs, float* partial, long places, int* counters, cudaStream_t stream) {
  if (nkv != F_WARPS || c.nq != F_WARPS * F_GROUP || !c.k_new || !partial || !counters) return -2;
  const int sms = sm_count();
  if ((long)nkv * bs <= sms || places < 2L * sms) return -2;
  if ((c.stride_page * 2) % 16 != 0 || (c.k_off * 2) % 16 != 0 || (c.v_off * 2) % 16 != 0 || c.k_off == c.v_off ||
      ((reinterpret_cast<uintptr_t>(c.kv) | reinterpret_cast<uintptr_t>(partial)) & 15) != 0 ||
      ((reinterpret_cast<uintptr_t>(c.q) | reinterpret_cast<uintptr_t>(c.k_new) | reinterpret_cast<uintptr_t>(c.v_new) | reinterpret_cast<uintptr_t>(c.out) |
        reinterpret_cast<uintptr_t>(c.qw) | reinterpret_cast<uintptr_t>(c.kw) | reinterpret_cast<uintptr_t>(c.cosc) | reinterpret_cast<uintptr_t>(c.sinc)) & 7) != 0)
    return -2;
  CUtensorMap map;
  if (!make_flat_map(&map, c.kv, c.k_off, c.v_off, c.stride_page)) return -2;
  constexpr size_t smem = 1024 + (size_t)F_WARPS * (F_SLOTS * F_TILE + (F_GROUP + 2) * F_HD * 2 + F_SLOTS * 8);
  static std::atomic<uint64_t> smem_set{0};
  if (allow_smem(smem_set, (const void*)decode_attention_flat_kernel, smem) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  const FlatArgs a{c.q, c.k_new, c.v_new, c.out, c.kv, c.k_off, c.v_off, c.stride_page, c.page_indices, c.page_indptr, c.last_page_len, c.positions,
                   c.qw, c.kw, c.cosc, c.sinc, c.eps, c.sm_scale_log2, bs, c.k_off < c.v_off ? 0 : 2 * kDaHalf, partial, counters, wait_err_word()};
  return (int)launch(decode_attention_flat_kernel, dim3(sms), dim3(F_THREADS), smem, stream, true, map, a);
}

}  // namespace pk
