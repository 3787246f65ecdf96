// Grouped-query softmax attention over a paged K/V cache for ragged batches, with the options that newer decoder
// designs combine: projection biases, a rotary embedding over the first `dims` entries of each head from a frequency
// table (pairs interleaved (2i, 2i+1) or split in halves (i, i + dims/2); plain, YaRN or any other schedule is the
// host's table), a chunk-local causal mask (query at position p sees keys floor(p / chunk) * chunk .. p; chunk 0 = plain
// causal) and a learned per-head sink that adds exp(sink) to the softmax denominator without a value.
// Further options (pk_attn_extra): a sliding window (keys p - window + 1 .. p), a soft cap on the scaled score
// (cap * tanh(score / cap)), a linear distance bias (head h subtracts 2^(-slope_log2 (h + 1) / heads) * (p - j)), a
// logistic gate on the output, element by element or one per head, and -- in the append -- an unweighted RMS norm of every cached value head.
// A window may keep the first `keep_first` positions of the sequence visible for good (they keep their true positions).
// gqa_norm_append_kernel is the append for designs that norm q and k (per head with one weight for all heads or none, or over the whole
// projection at once) beside rotating them (a layer that reads another layer's cache brings queries only), stretch the query by a factor that grows with the logarithm of the position, or
// cache the keys as projected in the place of values.
//
// Cache: token at position p of a request lives in page pages[page_off[req] + p / page_size], slot p % page_size, at
//   cache + page * page_stride + slot * (G * dim + G * vdim):  [K of G heads | V of G heads].
// Element type E (bf16 or float) for activations / cache / weights; scores, softmax and accumulation are fp32.
//   gqa_rope_append_kernel      bias + rotation of q and k, q to its buffer, k / v into the cache.  HBM-bound.
//   gqa_attention_kernel        one CTA per (query row, query head): warps stride over the visible keys with an online
//                               softmax each (lanes split the features), merged with the sink at the end.  Any sizes.
//   gqa_attention_mma_kernel    bf16 prompt portions on the tensor cores (64 query rows of one head per CTA).
//   gqa_attention_cluster_kernel  the same where these CTAs leave SMs idle: a cluster shares the keys.
//   gqa_decode_kernel           bf16, fewer than 64 rows: request by request on the tensor cores, a group's query heads as the rows of a tile.
#include "common.cuh"
#include "mma.cuh"
#include "typed.cuh"

namespace pk {

// qkv [tokens, ld] = [q (H*dim) | k (G*dim) | v (G*vdim)] rows of the stacked projection; bias (same layout) may be null.
template <typename E>
__global__ void gqa_rope_append_kernel(const E* __restrict__ qkv, int ld, const E* __restrict__ bias, const int* __restrict__ pos,
                                       const int* __restrict__ req, const int* __restrict__ page_off, const int* __restrict__ pages,
                                       E* __restrict__ q_out, E* __restrict__ cache, long page_stride, int page_size, int H, int G, int dim, int vdim,
                                       int dims, int interleaved, const float* __restrict__ freq, float mag, float v_eps) {
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t = blockIdx.x, p = pos[t];
  const E* row = qkv + (size_t)t * ld;
  const int nq = H * dim, nk = G * dim, nv = G * vdim, half = dims >> 1;
  E* slot = cache + (size_t)pages[page_off[req[t]] + p / page_size] * page_stride + (size_t)(p % page_size) * (nk + nv);
  if (v_eps > 0.f) {  // cached values are unit-RMS per head: one warp per value head
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int g = blockIdx.y * nw + (threadIdx.x >> 5); g < G; g += gridDim.y * nw) {
      const int e0 = nq + nk + g * vdim;
      float ss = 0.f;
      for (int d = lane; d < vdim; d += 32) {
        const float v = to_f(row[e0 + d]) + (bias ? to_f(bias[e0 + d]) : 0.f);
        ss = fmaf(v, v, ss);
      }
      const float inv = 1.f / sqrtf(warp_sum(ss) / (float)vdim + v_eps);
      for (int d = lane; d < vdim; d += 32) slot[e0 - nq + d] = from_f<E>((to_f(row[e0 + d]) + (bias ? to_f(bias[e0 + d]) : 0.f)) * inv);
    }
  }
  const int n_el = v_eps > 0.f ? nq + nk : nq + nk + nv;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < n_el; e += gridDim.y * blockDim.x) {
    float v = to_f(row[e]) + (bias ? to_f(bias[e]) : 0.f);
    if (e < nq + nk) {
      const int d = (e < nq ? e : e - nq) % dim;
      if (d < dims) {
        int i, pe;
        bool first;
        if (interleaved) {
          i = d >> 1;
          first = (d & 1) == 0;
          pe = first ? e + 1 : e - 1;
        } else {
          first = d < half;
          i = first ? d : d - half;
          pe = first ? e + half : e - half;
        }
        const float o = to_f(row[pe]) + (bias ? to_f(bias[pe]) : 0.f);
        const float a = (float)p * freq[i];
        const float c = cosf(a) * mag, s = sinf(a) * mag;
        v = first ? v * c - o * s : v * c + o * s;
      }
    }
    if (e < nq) q_out[(size_t)t * nq + e] = from_f<E>(v);
    else slot[e - nq] = from_f<E>(v);
  }
}

// Append for designs that norm q and k before they rotate.  qkv [tokens, ld] = [q (H*dim) | k (G*dim) | v (G*vdim)]; with `v_from_k` there
// is no v part and the cached values are the keys as projected (vdim == dim); with `q_only` the row is q alone and nothing is cached.  norm_kind 1: every head of q (of k) is divided by its own
// root mean square and multiplied by qw (kw) [dim], one weight for all heads (null: no weight; a rotation keeps
// the root mean square, so dividing by it before or after the rotation is the same); 2: the whole q row (k row) is divided by ONE root mean
// square and multiplied by qw [H*dim] (kw [G*dim]); 0: no norm.  Then the first `dims` entries of every head rotate, and q is
// multiplied by 1 + temp_coef * ln(floor((p + 1) / temp_every) + 1) (temp_every 0: not).  One CTA per token; the row lives in shared
// memory as fp32; sums of squares are added per head by one warp and then in head order, so a row's result does not depend on timing.
template <typename E>
__global__ void gqa_norm_append_kernel(const E* __restrict__ qkv, int ld, const int* __restrict__ pos, const int* __restrict__ req,
                                       const int* __restrict__ page_off, const int* __restrict__ pages, E* __restrict__ q_out, E* __restrict__ cache,
                                       long page_stride, int page_size, int H, int G, int dim, int vdim, int dims, int interleaved,
                                       const float* __restrict__ freq, float mag, const E* __restrict__ qw, const E* __restrict__ kw, int norm_kind,
                                       float eps, float temp_coef, int temp_every, int v_from_k, int q_only) {
  extern __shared__ float na_sm[];
  if (q_only) G = 0;
  float* row = na_sm;             // [nq + nk]
  float* inv = row + (H + G) * dim;  // [H + G] sum of squares per head
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t = blockIdx.x, p = pos[t], lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const E* src = qkv + (size_t)t * ld;
  const int nq = H * dim, nk = G * dim, nv = G * vdim, half = dims >> 1;
  // the page lookup (three dependent loads) and the weights of the last phase travel while the row is loaded and summed
  const int page = q_only ? 0 : pages[page_off[req[t]] + p / page_size];
  if (norm_kind && qw)
    for (int e = threadIdx.x * 64; e < (norm_kind == 1 ? dim : nq + nk); e += blockDim.x * 64)
      prefetch_l2(norm_kind == 1 ? (e < dim ? qw + e : kw + e - dim) : (e < nq ? qw + e : kw + e - nq));  // a line of 64 entries each
  if (norm_kind == 1 && kw && threadIdx.x * 64 < dim) prefetch_l2(kw + threadIdx.x * 64);
  // 16-byte accesses where every piece of the row and of the slot starts on such a boundary (bf16, sizes multiples of 8)
  const bool vec = sizeof(E) == 2 && ((nq | nk | nv | ld | (int)(page_stride & 7)) & 7) == 0 &&
                   ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(cache)) & 15) == 0;
  if (vec) {
    for (int e = threadIdx.x * 8; e < nq + nk; e += blockDim.x * 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(src + e);
      *reinterpret_cast<float4*>(row + e) = make_float4(bf16_lo(u.x), bf16_hi(u.x), bf16_lo(u.y), bf16_hi(u.y));
      *reinterpret_cast<float4*>(row + e + 4) = make_float4(bf16_lo(u.z), bf16_hi(u.z), bf16_lo(u.w), bf16_hi(u.w));
    }
  } else {
    for (int e = threadIdx.x; e < nq + nk; e += blockDim.x) row[e] = to_f(src[e]);
  }
  __syncthreads();
  if (norm_kind) {
    for (int hd = warp; hd < H + G; hd += nw) {
      float ss = 0.f;
      for (int d = lane; d < dim; d += 32) ss = fmaf(row[hd * dim + d], row[hd * dim + d], ss);
      ss = warp_sum(ss);
      if (lane == 0) inv[hd] = ss;
    }
    __syncthreads();
  }
  // reciprocal root mean square of the whole q row / k row (norm_kind 2): the heads' sums added in head order by every thread
  float iq = 1.f, ik = 1.f;
  if (norm_kind == 2) {
    float sq = 0.f, sk = 0.f;
    for (int hd = 0; hd < H; ++hd) sq += inv[hd];
    for (int hd = 0; hd < G; ++hd) sk += inv[H + hd];
    iq = 1.f / sqrtf(sq / (float)nq + eps);
    ik = 1.f / sqrtf(sk / (float)nk + eps);
  }
  const float stretch = temp_every > 0 ? 1.f + temp_coef * logf((float)((p + 1) / temp_every) + 1.f) : 1.f;
  E* slot = q_only ? nullptr : cache + (size_t)page * page_stride + (size_t)(p % page_size) * (nk + nv);
  // norm, rotation and the query's factor head by head (a warp per head, lanes over its entries: no index arithmetic per entry)
  for (int hd = warp; hd < H + G; hd += nw) {
    const bool is_q = hd < H;
    const float f = norm_kind == 1 ? 1.f / sqrtf(inv[hd] / (float)dim + eps) : norm_kind == 2 ? (is_q ? iq : ik) : 1.f;
    const E* w = norm_kind == 1 ? (is_q ? qw : kw) : norm_kind == 2 ? (is_q ? qw + hd * dim : kw + (hd - H) * dim) : nullptr;
    const float* hrow = row + hd * dim;
    E* dst = is_q ? q_out + (size_t)t * nq + hd * dim : slot + (hd - H) * dim;
    const float out_f = is_q ? stretch : 1.f;
    for (int d = lane; d < dim; d += 32) {
      float v = hrow[d] * f * (w ? to_f(w[d]) : 1.f);
      if (d < dims) {
        int i, pd;
        bool first;
        if (interleaved) {
          i = d >> 1;
          first = (d & 1) == 0;
          pd = first ? d + 1 : d - 1;
        } else {
          first = d < half;
          i = first ? d : d - half;
          pd = first ? d + half : d - half;
        }
        const float o = hrow[pd] * f * (w ? to_f(w[pd]) : 1.f);
        const float a = (float)p * freq[i];
        const float c = cosf(a) * mag, sn = sinf(a) * mag;
        v = first ? v * c - o * sn : v * c + o * sn;
      }
      dst[d] = from_f<E>(v * out_f);
    }
  }
  const E* vsrc = src + (v_from_k ? nq : nq + nk);  // the values: the keys as projected, or the value projection
  const int n_val = v_from_k ? nk : nv;
  if (vec) {
    for (int e = threadIdx.x * 8; e < n_val; e += blockDim.x * 8) *reinterpret_cast<uint4*>(slot + nk + e) = *reinterpret_cast<const uint4*>(vsrc + e);
  } else {
    for (int e = threadIdx.x; e < n_val; e += blockDim.x) slot[nk + e] = vsrc[e];
  }
}

// the options of pk_attn_extra as the kernels take them (all off when zero / null)
struct AttnExtra {
  int window;
  float softcap, slope_log2;
  const void* gate;
  long gate_ld;
  int max_kv_len;
  int keep_first;
  int gate_per_head;
  long out_ld;  // elements from one row of the output to the next
};
// logistic gate of entry (t, h, d); x.gate is not null
template <typename E>
__device__ __forceinline__ float out_gate(const AttnExtra& x, int t, int h, int d, int vdim) {
  const int at = x.gate_per_head ? h : h * vdim + d;
  return 1.f / (1.f + expf(-to_f(static_cast<const E*>(x.gate)[(size_t)t * x.gate_ld + at])));
}
__device__ __forceinline__ int first_visible(int p, int chunk, int window) {
  int lo = chunk > 0 ? (p / chunk) * chunk : 0;
  if (window > 0) lo = max(lo, p - window + 1);
  return lo;
}
__device__ __forceinline__ float head_slope(float slope_log2, int h, int H) { return slope_log2 > 0.f ? exp2f(-slope_log2 * (float)(h + 1) / (float)H) : 0.f; }
// scaled score -> soft cap -> minus the distance bias
__device__ __forceinline__ float shape_score(float s, float softcap, float slope, int distance) {
  if (softcap > 0.f) s = softcap * tanhf(s / softcap);
  return s - slope * (float)distance;
}
// 2^x on the special-function unit (relative error about 2^-22; 2^-inf = 0)
__device__ __forceinline__ float fast_ex2(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

constexpr int kGqaWarps = 8;
constexpr int kGqaMaxPerLane = 8;  // features per lane: dim, vdim <= 256

template <typename E>
__global__ void __launch_bounds__(kGqaWarps * 32) gqa_attention_kernel(const E* __restrict__ q, const E* __restrict__ cache, const E* __restrict__ sink,
                                                                      const int* __restrict__ pos, const int* __restrict__ req,
                                                                      const int* __restrict__ page_off, const int* __restrict__ pages,
                                                                      E* __restrict__ out, long page_stride, int page_size, int H, int G, int dim,
                                                                      int vdim, float scale, int chunk, AttnExtra x) {
  __shared__ float sm_m[kGqaWarps], sm_l[kGqaWarps];
  extern __shared__ float sm_acc[];  // [warps][vdim]
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t = blockIdx.x, h = blockIdx.y, g = h / (H / G), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = pos[t], lo = first_visible(p, chunk, x.window);
  const float slope = head_slope(x.slope_log2, h, H);
  const int* pg = pages + page_off[req[t]];
  const int tok = G * (dim + vdim);
  float qr[kGqaMaxPerLane], acc[kGqaMaxPerLane];
#pragma unroll
  for (int i = 0; i < kGqaMaxPerLane; ++i) {
    const int d = lane + 32 * i;
    qr[i] = d < dim ? to_f(q[((size_t)t * H + h) * dim + d]) * scale : 0.f;
    acc[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  // visible keys: the first `nf` positions (kept for good, when the window has left them behind), then lo .. p
  const int nf = min(x.keep_first, lo), n_vis = nf + p - lo + 1;
  // two keys per trip (i and i + warps): their loads, dot products and exponentials overlap, which halves the dependent chain per key
  for (int i = warp; i < n_vis; i += 2 * kGqaWarps) {
    const int i2 = i + kGqaWarps;
    const bool two = i2 < n_vis;
    const int j = i < nf ? i : lo + (i - nf), j2 = i2 < nf ? i2 : lo + (i2 - nf);
    const E* kv_a = cache + (size_t)pg[j / page_size] * page_stride + (size_t)(j % page_size) * tok;
    const E* kv_b = two ? cache + (size_t)pg[j2 / page_size] * page_stride + (size_t)(j2 % page_size) * tok : kv_a;
    float ka[kGqaMaxPerLane], kb[kGqaMaxPerLane], va[kGqaMaxPerLane], vb[kGqaMaxPerLane];
#pragma unroll
    for (int i = 0; i < kGqaMaxPerLane; ++i) {
      const int d = lane + 32 * i;
      ka[i] = d < dim ? to_f(kv_a[g * dim + d]) : 0.f;
      kb[i] = d < dim ? to_f(kv_b[g * dim + d]) : 0.f;
      va[i] = d < vdim ? to_f(kv_a[G * dim + g * vdim + d]) : 0.f;
      vb[i] = d < vdim ? to_f(kv_b[G * dim + g * vdim + d]) : 0.f;
    }
    float sa = 0.f, sb = 0.f;
#pragma unroll
    for (int i = 0; i < kGqaMaxPerLane; ++i) {
      sa = fmaf(qr[i], ka[i], sa);
      sb = fmaf(qr[i], kb[i], sb);
    }
    sa = shape_score(warp_sum(sa), x.softcap, slope, p - j);
    sb = two ? shape_score(warp_sum(sb), x.softcap, slope, p - j2) : -INFINITY;
    const float mn = fmaxf(m, fmaxf(sa, sb)), c = expf(m - mn), ea = expf(sa - mn), eb = two ? expf(sb - mn) : 0.f;
    l = l * c + (ea + eb);
#pragma unroll
    for (int i = 0; i < kGqaMaxPerLane; ++i) acc[i] = acc[i] * c + (ea * va[i] + eb * vb[i]);
    m = mn;
  }
  if (lane == 0) {
    sm_m[warp] = m;
    sm_l[warp] = l;
  }
#pragma unroll
  for (int i = 0; i < kGqaMaxPerLane; ++i) {
    const int d = lane + 32 * i;
    if (d < vdim) sm_acc[warp * vdim + d] = acc[i];
  }
  __syncthreads();
  const float sk = sink ? to_f(sink[h]) : -INFINITY;
  float mt = sk;
#pragma unroll
  for (int w = 0; w < kGqaWarps; ++w) mt = fmaxf(mt, sm_m[w]);
  float den = sink ? expf(sk - mt) : 0.f;
  float cw[kGqaWarps];
#pragma unroll
  for (int w = 0; w < kGqaWarps; ++w) {
    cw[w] = sm_m[w] == -INFINITY ? 0.f : expf(sm_m[w] - mt);
    den += sm_l[w] * cw[w];
  }
  for (int d = threadIdx.x; d < vdim; d += blockDim.x) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < kGqaWarps; ++w) o += sm_acc[w * vdim + d] * cw[w];
    o /= den;
    if (x.gate) o *= out_gate<E>(x, t, h, d, vdim);
    out[(size_t)t * x.out_ld + h * vdim + d] = from_f<E>(o);
  }
}

// ---- tensor cores (bf16): one CTA = 64 consecutive rows of the step (4 warps x 16 rows) for one query head.  Rows of a
// tile may belong to several requests: the tile walks each request's visible key range in 64-key blocks with the other
// rows masked.  dim, vdim multiples of 16 up to 128.  K and V blocks go through a two-stage cp.async ring in shared memory (the
// next block's copy overlaps this block's products); S = Q K^T and O += P V with mma.sync m16n8k16, P rounded to bf16 for the
// second product, statistics in fp32.
constexpr int kAmRows = 64, kAmKeys = 64;
// two floats at this address of CTA `rank` of the cluster
__device__ __forceinline__ void gqa_ld_state(uint32_t addr, uint32_t rank, float& a, float& b) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(at) : "memory");
}
constexpr int kGdTileFrom = 8;  // tokens of a request, at least, that run in tiles in a step of few rows

template <int DQ, int DV>
__global__ void __launch_bounds__(128, 3) gqa_attention_mma_kernel(const bf16* __restrict__ q, const bf16* __restrict__ cache, const bf16* __restrict__ sink,
                                                               const int* __restrict__ pos, const int* __restrict__ req,
                                                               const int* __restrict__ page_off, const int* __restrict__ pages,
                                                               bf16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml,
                                                               long page_stride, int page_size, int T, int H, int G, float scale, int chunk,
                                                               AttnExtra x) {
  extern __shared__ __align__(16) unsigned char am_smem[];
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  // grid (head, tile, split): the heads of a tile start together (a group's heads read the same keys), and the tiles run from the
  // end of the step backwards, so that the CTAs that start last are the ones with the fewest visible keys
  const int t0 = (gridDim.y - 1 - blockIdx.y) * kAmRows, h = blockIdx.x, g = h / (H / G);
#define GQA_T_END T
#define GQA_SPLIT blockIdx.z
#define GQA_SPLITS gridDim.z
#define GQA_PART_LD nsplit
#include "gqa_tile.cuh"
}

// The same for steps whose (tile, head) pairs leave SMs idle: the keys are dealt out to the CTAs of a cluster (the grid's z axis), which combine their states
// over distributed shared memory.  B200, us (heads / groups x size): 229 tokens of 6 requests behind 480 (8 / 2 x 128) 74.6 -> 33.8, 100 behind 500 (8 / 4 x 64)
// 21.3 -> 13.0, 64 behind 2000 (8 / 2 x 128) 93.6 -> 26.9.
template <int DQ, int DV>
__global__ void __launch_bounds__(128, 3) gqa_attention_cluster_kernel(const bf16* __restrict__ q, const bf16* __restrict__ cache, const bf16* __restrict__ sink,
                                                               const int* __restrict__ pos, const int* __restrict__ req,
                                                               const int* __restrict__ page_off, const int* __restrict__ pages,
                                                               bf16* __restrict__ out,
                                                               long page_stride, int page_size, int T, int H, int G, float scale, int chunk,
                                                               AttnExtra x) {
  extern __shared__ __align__(16) unsigned char am_smem[];
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t0 = (gridDim.y - 1 - blockIdx.y) * kAmRows, h = blockIdx.x, g = h / (H / G);
#define GQA_T_END T
#define GQA_CLUSTER 1
#define GQA_SPLIT blockIdx.z
#define GQA_SPLITS gridDim.z
#define GQA_PART_LD nsplit
#include "gqa_tile.cuh"
}

// Steps of fewer than 64 rows (below): how a request with several tokens in the step runs.  Launched are cs CTAs for each of its tokens and kv heads; request by
// request most of them leave, and what stays walks long contexts in tiles of 16 keys, a chain of about 1.2 us each (0.9 for heads of 64).  In tiles of 64 rows all
// of them take a share of the keys, which needs a merge.
struct GdRun {
  int start, len;  // its tokens of the step
  int shares;      // 0: request by request (gqa_decode_kernel); else in tiles of 64 rows per query head, the keys dealt out to so many CTAs each
};
// All lanes of a warp call; T < 64.  `slots`: CTAs that the GPU holds at once (0: never in tiles); a request counts on its part of them.
__device__ __forceinline__ GdRun gd_run(const int* req, const int* pos, int T, int t, int H, int G, int cs, int keep_first, int window, int chunk, int slots, int from) {
  const int lane = threadIdx.x & 31, rq = req[t], r0 = lane < T ? req[lane] : -1, r1 = lane + 32 < T ? req[lane + 32] : -1;
  const int p0 = slots > 0 && lane < T ? pos[lane] : 0, p1 = slots > 0 && lane + 32 < T ? pos[lane + 32] : 0;
  const unsigned long long other = (unsigned long long)__ballot_sync(0xffffffffu, lane >= T || r0 != rq) |
                                   (unsigned long long)__ballot_sync(0xffffffffu, lane + 32 >= T || r1 != rq) << 32;
  const unsigned long long below = other & ((1ull << t) - 1), above = other >> t;  // (T < 64: there is one above)
  GdRun r;
  r.start = below ? 64 - __clzll((long long)below) : 0;
  r.len = t + __ffsll((long long)above) - 1 - r.start;
  r.shares = 0;
  if (slots > 0 && r.len >= kGdTileFrom) {
    auto pos_of = [&](int u) { return __shfl_sync(0xffffffffu, u < 32 ? p0 : p1, u & 31); };
    const int lo = first_visible(pos_of(r.start), chunk, window), seen = min(keep_first, lo) + pos_of(r.start + r.len - 1) - lo + 1;
    const int n = min(slots * r.len / (T * H), r.len * G * cs / H);
    // a CTA of a tile walks 1 / n of the keys, a warp of a cluster 1 / (4 cs), which take it twice as long
    if (seen > from && n >= 2 * cs) r.shares = min(min(n, 64), (seen + kAmKeys - 1) / kAmKeys + 1);
  }
  return r;
}

// Steps of fewer than 64 rows (below): one request in tiles, share `split` of `nsplit` (most: places for them)
template <int DQ, int DV>
__device__ __forceinline__ void gqa_tile_of_run(unsigned char* am_smem, const bf16* __restrict__ q, const bf16* __restrict__ cache, const bf16* __restrict__ sink,
                                                const int* __restrict__ pos, const int* __restrict__ req, const int* __restrict__ page_off,
                                                const int* __restrict__ pages, bf16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml,
                                                long page_stride, int page_size, int T, int H, int G, float scale, int chunk, const AttnExtra& x,
                                                const GdRun run, int h, int share, int most) {
  const int t0 = run.start, g = h / (H / G);
#define GQA_T_END run.start + run.len
#define GQA_SPLIT share
#define GQA_SPLITS run.shares
#define GQA_PART_LD most
#include "gqa_tile.cuh"
}

// one CTA per (row, head): combine the splits' (m, l, O), join the sink, apply the output gate
__global__ void gqa_attention_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const bf16* __restrict__ sink,
                                           bf16* __restrict__ out, int nsplit, int T, int H, int vdim, AttnExtra x) {
  __shared__ float wgt[64];  // per split: exp(m_s - M) / denominator
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  const int t = blockIdx.x, h = blockIdx.y;
  if (threadIdx.x < 32) {
    const float sk = sink ? bf2f(sink[h]) : -INFINITY;
    float m[2], l[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int sp = threadIdx.x + 32 * i;
      const size_t slot = (size_t)(h * nsplit + sp) * T + t;
      m[i] = sp < nsplit ? part_ml[slot * 2] : -INFINITY;
      l[i] = sp < nsplit ? part_ml[slot * 2 + 1] : 0.f;
    }
    const float M = fmaxf(warp_max(fmaxf(m[0], m[1])), sk);  // finite: a query always sees its own position
    const float e0 = m[0] == -INFINITY ? 0.f : expf(m[0] - M), e1 = m[1] == -INFINITY ? 0.f : expf(m[1] - M);
    const float inv = 1.f / (warp_sum(l[0] * e0 + l[1] * e1) + (sink ? expf(sk - M) : 0.f));
    wgt[threadIdx.x] = e0 * inv;
    wgt[threadIdx.x + 32] = e1 * inv;
  }
  __syncthreads();
  for (int d = threadIdx.x; d < vdim; d += blockDim.x) {
    float a4[4] = {0.f, 0.f, 0.f, 0.f};
    int sp = 0;
    for (; sp + 4 <= nsplit; sp += 4) {  // the splits' loads are independent: four in flight
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = part_o[((size_t)(h * nsplit + sp + u) * T + t) * vdim + d];
#pragma unroll
      for (int u = 0; u < 4; ++u) a4[u] = fmaf(v[u], wgt[sp + u], a4[u]);
    }
    for (; sp < nsplit; ++sp) a4[0] = fmaf(part_o[((size_t)(h * nsplit + sp) * T + t) * vdim + d], wgt[sp], a4[0]);
    float o = (a4[0] + a4[1]) + (a4[2] + a4[3]);
    if (x.gate) o *= out_gate<bf16>(x, t, h, d, vdim);
    out[(size_t)t * x.out_ld + h * vdim + d] = f2bf(o);
  }
}

// The same for a step whose requests may run in tiles (gd_run): a warp per (row, head), and rows of requests that do not stay as they are.  What the choice
// follows from is older than the kernel before this one, so it is looked at ahead of the wait for it.
template <int D>
__global__ void __launch_bounds__(256) gqa_run_merge_kernel(const float* __restrict__ part, const bf16* __restrict__ sink, const int* __restrict__ pos,
                                                           const int* __restrict__ req, bf16* __restrict__ out, int most, int T, int H, int G, int cs, int chunk,
                                                           AttnExtra x, int slots, int from) {
  const int t = blockIdx.x, lane = threadIdx.x & 31, h = blockIdx.y * 8 + (threadIdx.x >> 5);
  const GdRun run = gd_run(req, pos, T, t, H, G, cs, x.keep_first, x.window, chunk, slots, from);
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  if (run.shares < 2 || h >= H) return;
  const float* ml = part + (size_t)H * most * T * D;
  const size_t row0 = (size_t)h * most * T + t;  // row of share s: row0 + s T
  float m[2], l[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int s = lane + 32 * i;
    m[i] = s < run.shares ? ml[(row0 + (size_t)s * T) * 2] : -INFINITY;
    l[i] = s < run.shares ? ml[(row0 + (size_t)s * T) * 2 + 1] : 0.f;
  }
  const float sk = sink ? bf2f(sink[h]) : -INFINITY, M = fmaxf(warp_max(fmaxf(m[0], m[1])), sk);  // finite: a query always sees its own position
#pragma unroll
  for (int i = 0; i < 2; ++i) m[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - M);
  const float inv = 1.f / (warp_sum(l[0] * m[0] + l[1] * m[1]) + (sink ? expf(sk - M) : 0.f));
  constexpr int PAIRS = D / 2, NP = (PAIRS + 31) / 32;
  float2 o[NP] = {};
  constexpr int AT_ONCE = 12 / NP;  // loads under way
  for (int s0 = 0; s0 < run.shares; s0 += AT_ONCE) {
    float2 v[AT_ONCE][NP];
#pragma unroll
    for (int u = 0; u < AT_ONCE; ++u)
#pragma unroll
      for (int i = 0; i < NP; ++i)
        v[u][i] = s0 + u < run.shares && lane + 32 * i < PAIRS ? *reinterpret_cast<const float2*>(part + (row0 + (size_t)(s0 + u) * T) * D + 2 * (lane + 32 * i))
                                                              : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < AT_ONCE; ++u) {
      const int s = s0 + u;
      const float w = s < run.shares ? __shfl_sync(0xffffffffu, s < 32 ? m[0] : m[1], s & 31) * inv : 0.f;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        o[i].x = fmaf(v[u][i].x, w, o[i].x);
        o[i].y = fmaf(v[u][i].y, w, o[i].y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NP; ++i)
    if (lane + 32 * i < PAIRS) {
      const int d = 2 * (lane + 32 * i);
      const float g0 = x.gate ? out_gate<bf16>(x, t, h, d, D) : 1.f, g1 = x.gate ? out_gate<bf16>(x, t, h, d + 1, D) : 1.f;
      *reinterpret_cast<uint32_t*>(out + (size_t)t * x.out_ld + h * D + d) = pack_bf16(o[i].x * g0, o[i].y * g1);
    }
}

// ---- fewer than 64 rows (decode steps, small portions), bf16: a cluster of CTAs per (tokens of one request, kv head).  The 16 rows of a tile are the group's
// query heads, for as many tokens of the request as fit (a cluster is launched for every token, and the first of each tile's stays), so that a key is fetched
// once for all of them and requests do not wait for one another.  A warp takes every (4 cs)-th tile of 16 visible keys through a cp.async ring of its own;
// the warps' states meet in shared memory, the CTAs' in the cluster's.
// Bound by latency: lookups, keys, exchange.  Figures at launch_gqa_mma.
constexpr int kGdWarps = 4, kGdRing = 3;
__device__ __forceinline__ float2 gd_remote(const float2* p, uint32_t rank) {  // the same place in another CTA of the cluster
  uint32_t at;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
  return v;
}

// TILES: requests with several tokens of the step may run in tiles (gd_run), `most` shares at most, whose states go to `part`
struct GdExtra : AttnExtra {
  float* part;
  int most, slots, from;
};
template <int D, bool TILES>
__global__ void __launch_bounds__(kGdWarps * 32, TILES && D <= 64 ? 3 : 2) gqa_decode_kernel(const bf16* __restrict__ q, const bf16* __restrict__ cache, const bf16* __restrict__ sink,
                                                                    const int* __restrict__ pos, const int* __restrict__ req, const int* __restrict__ page_off,
                                                                    const int* __restrict__ pages, bf16* __restrict__ out, long page_stride, int page_size, int T,
                                                                    int H, int G, float scale, int chunk, std::conditional_t<TILES, GdExtra, AttnExtra> x) {
  constexpr int LD = D + 8, TILE = 16 * LD;
  extern __shared__ __align__(16) unsigned char gd_smem[];  // [warps][ring][K, V][16][LD]; later the states, [warps][16][D] floats at the warps' rings
  __shared__ long long s_off[kGdWarps][kGdRing][16];
  __shared__ float2 s_ml[kGdWarps][16];  // (maximum, sum) of the warps' rows; later of the CTA's
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, tq = lane & 3;
  const int rank = (int)cluster_ctarank(), cs = gridDim.x, g = blockIdx.y, t = blockIdx.z, R = H / G, per = 16 / R;
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  // the tokens of this one's request around it
  GdRun run;
  if constexpr (TILES) {
    run = gd_run(req, pos, T, t, H, G, cs, x.keep_first, x.window, chunk, x.slots, x.from);
    if (run.shares > 0) {
      const int nth = ((t - run.start) * G + g) * cs + rank;
      if (nth < H * run.shares)
        gqa_tile_of_run<D, D>(gd_smem, q, cache, sink, pos, req, page_off, pages, out, x.part, x.part + (size_t)H * x.most * T * D, page_stride, page_size, T, H, G,
                              scale, chunk, x, run, nth % H, nth / H, x.most);
      return;  // (the whole cluster)
    }
  } else {
    run = gd_run(req, pos, T, t, H, G, cs, x.keep_first, x.window, chunk, 0, 0);
  }
  const int start = run.start, left = run.start + run.len - t;
  if ((t - start) % per != 0) return;  // (the whole cluster)
  const int n_tok = min(per, left);
  const int p_max = pos[t + n_tok - 1], lo = first_visible(pos[t], chunk, x.window), nf = min(x.keep_first, lo), n_vis = nf + p_max - lo + 1;
  const int* pg = pages + page_off[req[t]];
  const int tok = 2 * G * D, n_tiles = (n_vis + 15) / 16, step = cs * kGdWarps;
  bf16* ring = reinterpret_cast<bf16*>(gd_smem) + warp * kGdRing * 2 * TILE;
  auto key_of = [&](int i) { return i < nf ? i : lo + i - nf; };  // position of visible key i
  auto load = [&](int tile, int st) {
    if (tile < n_tiles) {
      if (lane < 16) {
        const int i = tile * 16 + lane, j = key_of(i);
        s_off[warp][st][lane] = i < n_vis ? (long long)pg[j / page_size] * page_stride + (long long)(j % page_size) * tok + g * D : -1;
      }
      __syncwarp();
      bf16* dst = ring + st * 2 * TILE;
#pragma unroll
      for (int c = lane; c < 16 * (D / 8); c += 32) {
        const int r = c / (D / 8), cc = (c % (D / 8)) * 8;
        const long long at = s_off[warp][st][r];
        const bf16* src = cache + (at < 0 ? 0 : at) + cc;
        const uint32_t bytes = at < 0 ? 0 : 16;  // zeros behind the last key
        cp_async16(dst + r * LD + cc, src, bytes);
        cp_async16(dst + TILE + r * LD + cc, at < 0 ? src : src + G * D, bytes);
      }
    }
    cp_async_commit();
  };
  int tile = rank * kGdWarps + warp;
#pragma unroll
  for (int s = 0; s < kGdRing; ++s) load(tile + s * step, s);
  // rows gq and gq + 8: (token, head) of the group
  const int ta = gq / R, tb = (gq + 8) / R, ha = g * R + gq % R, hb = g * R + (gq + 8) % R;
  const bool on_a = ta < n_tok, on_b = tb < n_tok;  // (n_tok <= per: rows behind R * per are off)
  const int pos_a = on_a ? pos[t + ta] : -1, pos_b = on_b ? pos[t + tb] : -1;
  uint32_t qa[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const bf16* qra = q + ((size_t)(t + (on_a ? ta : 0)) * H + ha) * D + kk * 16 + 2 * tq;
    const bf16* qrb = q + ((size_t)(t + (on_b ? tb : 0)) * H + hb) * D + kk * 16 + 2 * tq;
    qa[kk][0] = on_a ? *reinterpret_cast<const uint32_t*>(qra) : 0u;
    qa[kk][1] = on_b ? *reinterpret_cast<const uint32_t*>(qrb) : 0u;
    qa[kk][2] = on_a ? *reinterpret_cast<const uint32_t*>(qra + 8) : 0u;
    qa[kk][3] = on_b ? *reinterpret_cast<const uint32_t*>(qrb + 8) : 0u;
  }
  // scores in units of log2, shaped as in the kernel above
  const bool capped = x.softcap > 0.f;
  const float cap2 = x.softcap * kLog2e, c1 = capped ? 2.f * scale / x.softcap * kLog2e : scale * kLog2e;
  const float slope_a = head_slope(x.slope_log2, ha, H) * kLog2e, slope_b = head_slope(x.slope_log2, hb, H) * kLog2e;
  const int lo_a = on_a ? first_visible(pos_a, chunk, x.window) : 0, lo_b = on_b ? first_visible(pos_b, chunk, x.window) : 0;
  float oa[D / 8][4] = {};
  float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
  for (int st = 0; tile < n_tiles; tile += step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGdRing - 1) : "memory");
    __syncwarp();
    const bf16 *Ks = ring + st * 2 * TILE, *Vs = Ks + TILE;
    float s[2][4] = {}, s1[2][4] = {};  // even and odd k steps apart
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t b[4];
      ldsm_x4(b, &Ks[((lane & 7) + ((lane >> 4) & 1) * 8) * LD + kk * 16 + ((lane >> 3) & 1) * 8]);
      mma_bf16_16816(kk & 1 ? s1[0] : s[0], qa[kk], b[0], b[1]);
      mma_bf16_16816(kk & 1 ? s1[1] : s[1], qa[kk], b[2], b[3]);
    }
    float mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = tile * 16 + ni * 8 + 2 * tq + (e & 1), j = key_of(i);
        const bool top = e < 2;
        const int dist = (top ? pos_a : pos_b) - j;
        const bool ok = i < n_vis && dist >= 0 && (j >= (top ? lo_a : lo_b) || j < x.keep_first);
        float v = (s[ni][e] + s1[ni][e]) * c1;
        if (capped) v = fmaf(-2.f * cap2, __fdividef(1.f, fast_ex2(fminf(v, 80.f)) + 1.f), cap2);
        v = fmaf(-(top ? slope_a : slope_b), (float)dist, v);
        v = ok ? v : -INFINITY;
        s[ni][e] = v;
        if (top) mx_a = fmaxf(mx_a, v);
        else mx_b = fmaxf(mx_b, v);
      }
    mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
    mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
    mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
    mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
    const float mn_a = fmaxf(m_a, mx_a), mn_b = fmaxf(m_b, mx_b);
    const float sub_a = mn_a == -INFINITY ? 0.f : mn_a, sub_b = mn_b == -INFINITY ? 0.f : mn_b;
    const float f_a = fast_ex2(m_a - sub_a), f_b = fast_ex2(m_b - sub_b);
    uint32_t pa[4];  // P rounded to bf16 once, for the second product; the sums add the rounded values
#pragma unroll
    for (int ni = 0; ni < 2; ++ni) {
      pa[ni * 2] = pack_bf16(fast_ex2(s[ni][0] - sub_a), fast_ex2(s[ni][1] - sub_a));
      pa[ni * 2 + 1] = pack_bf16(fast_ex2(s[ni][2] - sub_b), fast_ex2(s[ni][3] - sub_b));
    }
    l_a = l_a * f_a + ((bf16_lo(pa[0]) + bf16_hi(pa[0])) + (bf16_lo(pa[2]) + bf16_hi(pa[2])));
    l_b = l_b * f_b + ((bf16_lo(pa[1]) + bf16_hi(pa[1])) + (bf16_lo(pa[3]) + bf16_hi(pa[3])));
    m_a = mn_a;
    m_b = mn_b;
#pragma unroll
    for (int ni = 0; ni < D / 8; ++ni) {
      oa[ni][0] *= f_a;
      oa[ni][1] *= f_a;
      oa[ni][2] *= f_b;
      oa[ni][3] *= f_b;
    }
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      uint32_t b[4];
      ldsm_x4_trans(b, &Vs[((lane & 7) + ((lane >> 3) & 1) * 8) * LD + np * 16 + ((lane >> 4) & 1) * 8]);
      mma_bf16_16816(oa[np * 2], pa, b[0], b[1]);
      mma_bf16_16816(oa[np * 2 + 1], pa, b[2], b[3]);
    }
    __syncwarp();
    load(tile + kGdRing * step, st);
    if (++st == kGdRing) st = 0;
  }
  cp_async_wait_all();
  __syncwarp();
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
  l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
  l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
  // ---- the warps' states -> this CTA's
  float* st_o = reinterpret_cast<float*>(gd_smem);
  constexpr int WARP_F = kGdRing * TILE;  // floats of a warp's ring
#pragma unroll
  for (int ni = 0; ni < D / 8; ++ni) {
    float* p = st_o + warp * WARP_F + gq * D + ni * 8 + 2 * tq;
    *reinterpret_cast<float2*>(p) = make_float2(oa[ni][0], oa[ni][1]);
    *reinterpret_cast<float2*>(p + 8 * D) = make_float2(oa[ni][2], oa[ni][3]);
  }
  if (tq == 0) {
    s_ml[warp][gq] = make_float2(m_a, l_a);
    s_ml[warp][gq + 8] = make_float2(m_b, l_b);
  }
  __syncthreads();
  // rows by turns to the warps, two columns to a lane.  Row r: token t + r / R, head g R + r % R (a lane each: divisions once)
  constexpr int PAIRS = D / 2, NP = (PAIRS + 31) / 32;
  const int rows = R * n_tok, l_tok = lane / R, l_head = g * R + lane % R;
  auto finish = [&](int r, float M, float den, float2 (&o)[NP]) {  // M: of the states; the sink and the gate join here
    const int tt = t + __shfl_sync(0xffffffffu, l_tok, r), h = __shfl_sync(0xffffffffu, l_head, r);
    float f = 1.f;
    if (sink) {
      const float sk = bf2f(sink[h]) * kLog2e, top = fmaxf(M, sk);
      f = fast_ex2(M - top);
      den = den * f + fast_ex2(sk - top);
    }
    f /= den;
    if (x.gate && x.gate_per_head) f *= out_gate<bf16>(x, tt, h, 0, D);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = 2 * (lane + 32 * i);
      if (d >= D) break;
      float g0 = f, g1 = f;
      if (x.gate && !x.gate_per_head) {
        g0 *= out_gate<bf16>(x, tt, h, d, D);
        g1 *= out_gate<bf16>(x, tt, h, d + 1, D);
      }
      *reinterpret_cast<uint32_t*>(out + (size_t)tt * x.out_ld + h * D + d) = pack_bf16(o[i].x * g0, o[i].y * g1);
    }
  };
  for (int r = warp; r < rows; r += kGdWarps) {  // the four warps' states of a row -> this CTA's, in the first warp's place
    float2 ml[kGdWarps], o[NP] = {};
    float M = -INFINITY, den = 0.f;
#pragma unroll
    for (int w = 0; w < kGdWarps; ++w) {
      ml[w] = s_ml[w][r];
      M = fmaxf(M, ml[w].x);
    }
#pragma unroll
    for (int w = 0; w < kGdWarps; ++w) {
      const float f = ml[w].x == -INFINITY ? 0.f : fast_ex2(ml[w].x - M);
      den = fmaf(ml[w].y, f, den);
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (lane + 32 * i < PAIRS) {
          const float2 v = *reinterpret_cast<const float2*>(st_o + w * WARP_F + r * D + 2 * (lane + 32 * i));
          o[i].x = fmaf(v.x, f, o[i].x);
          o[i].y = fmaf(v.y, f, o[i].y);
        }
    }
    if (cs == 1) {
      finish(r, M, den, o);
    } else {
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (lane + 32 * i < PAIRS) *reinterpret_cast<float2*>(st_o + r * D + 2 * (lane + 32 * i)) = o[i];
      __syncwarp();
      if (lane == 0) s_ml[0][r] = make_float2(M, den);
    }
  }
  if (cs == 1) return;
  cluster_barrier();
  for (int r = rank * kGdWarps + warp; r < rows; r += cs * kGdWarps) {  // the CTAs' states: every warp of the cluster finishes rows
    float2 ml = make_float2(-INFINITY, 0.f), o[NP] = {};
    if (lane < cs) ml = gd_remote(&s_ml[0][r], lane);
    const float M = warp_max(ml.x), f = ml.x == -INFINITY ? 0.f : fast_ex2(ml.x - M), den = warp_sum(ml.y * f);
    float2 v[8][NP];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (c < cs && lane + 32 * i < PAIRS) v[c][i] = gd_remote(reinterpret_cast<const float2*>(st_o + r * D) + lane + 32 * i, c);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float fc = __shfl_sync(0xffffffffu, f, c);
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (c < cs && lane + 32 * i < PAIRS) {
          o[i].x = fmaf(v[c][i].x, fc, o[i].x);
          o[i].y = fmaf(v[c][i].y, fc, o[i].y);
        }
    }
    finish(r, M, den, o);
  }
  cluster_barrier();  // nobody leaves while its states are read
}

template <int D>
static cudaError_t launch_gqa_decode(const bf16* q, const bf16* cache, const bf16* sink, const int* pos, const int* req, const int* page_off, const int* pages,
                                   bf16* out, long page_stride, int page_size, int T, int H, int G, float scale, int chunk, AttnExtra x, int span,
                                   cudaStream_t st) {
  constexpr size_t smem = (size_t)kGdWarps * kGdRing * 2 * 16 * (D + 8) * sizeof(bf16);
  static_assert(smem >= (size_t)2 * kAmKeys * 2 * (D + 8) * sizeof(bf16), "gqa_tile's stages");
  // No more CTAs than the keys occupy, and as many as the GPU holds twice (four times from 41 tokens on: portions more often, of whose clusters most leave at
  // once), but not where each token, or every second one, has a tile of its own.  B200, us, in a graph, by cluster size 1 / 2 / 4 / 8.  16 heads of 128 in 4 groups,
  // 1 / 16 / 32 / 48 / 63 decoding requests at 2000: 40.0 24.6 15.0 10.1 | 40.6 25.3 18.8 24.3 | 43.3 35.0 39.3 51.1 | 53.0 62.3 57.4 75.4 | 55.1 65.5 74.4 98.6;
  // portions of 8 / 16 / 32 / 60 tokens behind 400: 12.4 11.0 8.5 8.6 | 12.4 11.1 9.9 9.2 | 12.5 12.8 10.3 12.4 | 16.0 13.7 12.8 20.5 (a step's requests are not
  // known here: the rule lies between the two).  In one group, 40 behind 400: 12.5 11.2 10.4 16.4.  64 heads of 64 in 8 groups, 60 behind 400: 14.4 19.9 23.2 36.4.
  const int per = 16 / (H / G);
  const long hold = (per == 1 ? 2L : per > 2 && T > 40 ? 8L : 4L) * sm_count();
  int cs = 8;
  while (cs > 1 && ((long)cs * G * T > hold || (cs / 2) * kGdWarps * 16 >= span)) cs /= 2;
  ThreadState& ts = tls();
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(cs, G, T);
  lc.blockDim = dim3(kGdWarps * 32);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = ts.pdl ? 1 : 0;
  lc.attrs = at;
  lc.numAttrs = 2;
  // A request with several tokens may run in tiles (gd_run) where its keys are many: below, the merge and the tiles' longer start cost more than they save.
  // slots: at 128 entries a head two CTAs fit on an SM, but clusters of 8 not on every pair of them (304 of 296 or 288: a second round, 48 instead of 31 us).
  // B200, us, in a graph, request by request -> in tiles (tiles of 64 rows for all requests, as before there was a choice): 16 heads of 128 in 4 groups, 24
  // tokens behind 2000 18.7 -> 16.2 (15.7), 40 behind 2000 31.6 -> 16.1 (19.4), 60 behind 8000 59.3 -> 39.9 (42.4); in 8 groups, 24 behind 400 12.7 -> 9.9 (9.3);
  // 16 heads of 64 in 16 groups, 24 behind 2000 / 8000 32.6 -> 14.5 (12.5), 118.7 -> 24.3 (23.4); 64 heads of 64 in 8 groups, 60 behind 8000 160 -> 84 (75).
  const int from = max((D <= 64 ? 600 : cs == 8 ? 300 : 150) * cs, 400);
  if (T >= kGdTileFrom && span > from) {
    const int slots = (D <= 64 ? 20 : 14) * sm_count() / 8, most = min(max(slots / H, 1), 64);
    if ((size_t)H * most * T * (D + 2) * sizeof(float) <= ts.work_bytes()) {
      static std::atomic<uint64_t> smem_set{0};
      if (const cudaError_t e = allow_smem(smem_set, (const void*)gqa_decode_kernel<D, true>, smem); e != cudaSuccess) return e;
      float* part = ts.work();
      ts.launches++;
      if (const cudaError_t e = cudaLaunchKernelEx(&lc, gqa_decode_kernel<D, true>, q, cache, sink, pos, req, page_off, pages, out, page_stride, page_size, T, H, G, scale,
                                                   chunk, GdExtra{x, part, most, slots, from});
          e != cudaSuccess)
        return e;
      return launch(gqa_run_merge_kernel<D>, dim3(T, (H + 7) / 8), dim3(256), 0, st, true, (const float*)part, sink, pos, req, out, most, T, H, G, cs, chunk, x, slots,
                    from);
    }
  }
  static std::atomic<uint64_t> smem_set{0};
  if (const cudaError_t e = allow_smem(smem_set, (const void*)gqa_decode_kernel<D, false>, smem); e != cudaSuccess) return e;
  ts.launches++;
  return cudaLaunchKernelEx(&lc, gqa_decode_kernel<D, false>, q, cache, sink, pos, req, page_off, pages, out, page_stride, page_size, T, H, G, scale, chunk, x);
}

template <int D>
static void launch_gqa_mma(const bf16* q, const bf16* cache, const bf16* sink, const int* pos, const int* req, const int* page_off, const int* pages,
                           bf16* out, long page_stride, int page_size, int T, int H, int G, float scale, int chunk, AttnExtra x, cudaStream_t st) {
  const size_t smem = (size_t)2 * kAmKeys * 2 * (D + 8) * sizeof(bf16);
  static bool attr_set = false;  // per template instance
  if (!attr_set) {
    cudaFuncSetAttribute(gqa_attention_mma_kernel<D, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr_set = true;
  }
  // The span a row can see is bounded by the window / chunk, else by the longest context of the step (when the caller knows it).
  // Fewer than 64 rows run request by request (requests with many tokens and keys in tiles, in the same launch); more, and groups of over 16 heads, in tiles of
  // 64, the few-row ones with the key axis dealt out to several CTAs per (tile, head) so that the step fills the GPU.  B200, us, in a graph, 16 heads of 128 in 4
  // groups, tiles of 64 -> the other form: 4 / 16 / 32 / 63 decoding requests at 2000 (the first with a window of 1024) 18.8 107 221 429 -> 8.5 23.7 39.0 73.7.
  // One token of up to 16 heads of up to 64 entries behind more than 5000 stays in tiles: 8000 keys, 8 heads in 4 groups 15.1 there, 18.8 in a cluster (16 heads in
  // 16 groups 19.4, 21.6; behind 2000 9.8, 8.1).
  const int tiles = (T + kAmRows - 1) / kAmRows;
  int span = x.max_kv_len;
  if (x.window > 0) span = span > 0 ? min(span, x.window + x.keep_first + T) : x.window + x.keep_first + T;
  if (chunk > 0) span = span > 0 ? min(span, chunk) : chunk;
  if (T < kAmRows && H / G <= 16 && !(T == 1 && D <= 64 && H <= 16 && span > 5000)) {
    launch_gqa_decode<D>(q, cache, sink, pos, req, page_off, pages, out, page_stride, page_size, T, H, G, scale, chunk, x, span > 0 ? span : 1 << 30, st);
    return;
  }
  int splits = 1;
  ThreadState& ts = tls();
  if (T < kAmRows && span > 2 * kAmKeys && ts.work()) {
    const int blocks = (span + kAmKeys - 1) / kAmKeys + 1;
    splits = min(min(blocks, (2 * sm_count() + tiles * H - 1) / (tiles * H)), 64);
    while (splits > 1 && (size_t)H * splits * T * (D + 2) * sizeof(float) > ts.work_bytes()) --splits;
  }
  float* po = ts.work();
  float* pml = po ? po + (size_t)H * splits * T * D : nullptr;
  // From 64 rows on: as many CTAs of a cluster to a (tile, head) as the GPU holds at once, where there are keys enough.  A share's start and the exchange cost
  // 9 us with two CTAs (each finishes 32 rows), 7 with four or eight, a block of 64 keys 2.7, so eight pay from 4 blocks on, four from 5 and two from 16; counted
  // are the longest context's, half of them where it is no longer than the step (a prompt from its start), none where the length is unknown.  B200, us, 1 / 2 /
  // 4 / 8 CTAs, 16 heads of 128 in 4 groups: 64 rows behind 100 13.9 20.8 16.0 15.6, behind 200 19.2 23.8 19.0 16.1, behind 700 37.9 32.7 22.0 19.8; 200
  // behind 300 27.3 27.1 23.7 31.4; 400 behind 700 51.5 51.0 54.3 65.5; prompts of 512 / 1024 27.4 33.2 37.9 53.4 / 59.3 52.3 73.3 116; 3 of 333 32.4 44.4 58.6 103.
  // (Of 390 steps of six shapes none is more than 2 % slower than without clusters, the mean 0.727 of it, the best choice each time 0.703.)
  const int blocks = (span > T ? span : span / 2) / kAmKeys;
  auto holds = [&](int n) { return (long)H * tiles * n <= 3 * sm_count(); };
  const int cs = T < kAmRows ? 1 : blocks >= 4 && holds(8) ? 8 : blocks >= 5 && holds(4) ? 4 : blocks >= 16 && holds(2) ? 2 : 1;
  if (cs > 1) {
    static std::atomic<uint64_t> smem_set{0};  // per template instance
    if (allow_smem(smem_set, (const void*)gqa_attention_cluster_kernel<D, D>, smem) == cudaSuccess) {
      cudaLaunchConfig_t lc{};
      lc.gridDim = dim3(H, tiles, cs);
      lc.blockDim = dim3(128);
      lc.dynamicSmemBytes = smem;
      lc.stream = st;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = ts.pdl ? 1 : 0;
      attr[1].id = cudaLaunchAttributeClusterDimension;
      attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
      attr[1].val.clusterDim.z = cs;
      lc.attrs = attr;
      lc.numAttrs = 2;
      ts.launches++;
      cudaLaunchKernelEx(&lc, gqa_attention_cluster_kernel<D, D>, q, cache, sink, pos, req, page_off, pages, out, page_stride, page_size, T, H, G, scale, chunk, x);
      return;
    }
    cudaGetLastError();
  }
  launch(gqa_attention_mma_kernel<D, D>, dim3(H, tiles, splits), dim3(128), smem, st, true, q, cache, sink, pos, req, page_off, pages, out, po, pml,
         page_stride, page_size, T, H, G, scale, chunk, x);
  if (splits > 1)
    launch(gqa_attention_merge_kernel, dim3(T, H), dim3(D >= 128 ? 128 : 64), 0, st, true, (const float*)po, (const float*)pml, sink, out, splits, T, H, D, x);
}

}  // namespace pk

using namespace pk;

extern "C" int pk_gqa_rope_append(const void* qkv, int ld, const void* bias, const int* positions, const int* req, const int* page_off,
                                  const int* pages, void* q_out, void* cache, long page_stride, int page_size, int heads, int kv_heads, int dim,
                                  int vdim, int dims, int interleaved, const float* freq, float mag, int tokens, int f32, pk_stream st) {
  return pk_gqa_rope_append_ex(qkv, ld, bias, positions, req, page_off, pages, q_out, cache, page_stride, page_size, heads, kv_heads, dim, vdim, dims,
                               interleaved, freq, mag, 0.f, tokens, f32, st);
}

extern "C" int pk_gqa_rope_append_ex(const void* qkv, int ld, const void* bias, const int* positions, const int* req, const int* page_off,
                                     const int* pages, void* q_out, void* cache, long page_stride, int page_size, int heads, int kv_heads, int dim,
                                     int vdim, int dims, int interleaved, const float* freq, float mag, float value_norm_eps, int tokens, int f32,
                                     pk_stream st) {
  if (!qkv || !positions || !req || !page_off || !pages || !q_out || !cache || tokens <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads ||
      dim <= 0 || vdim <= 0 || dims < 0 || dims > dim || (dims & 1) || (dims > 0 && !freq) || page_size <= 0)
    return -1;
  // few tokens (decoding): a token's features are spread over several CTAs
  const int n_all = heads * dim + kv_heads * (dim + vdim);
  const dim3 grid(tokens, tokens >= 128 ? 1 : std::min((n_all + 255) / 256, 16));
  if (f32)
    launch(gqa_rope_append_kernel<float>, grid, dim3(256), 0, st, true, (const float*)qkv, ld, (const float*)bias, positions, req, page_off, pages,
           (float*)q_out, (float*)cache, page_stride, page_size, heads, kv_heads, dim, vdim, dims, interleaved, freq, mag, value_norm_eps);
  else
    launch(gqa_rope_append_kernel<bf16>, grid, dim3(256), 0, st, true, (const bf16*)qkv, ld, (const bf16*)bias, positions, req, page_off, pages,
           (bf16*)q_out, (bf16*)cache, page_stride, page_size, heads, kv_heads, dim, vdim, dims, interleaved, freq, mag, value_norm_eps);
  return (int)cudaGetLastError();
}

extern "C" int pk_gqa_norm_append(const void* qkv, int ld, const int* positions, const int* req, const int* page_off, const int* pages, void* q_out,
                                  void* cache, long page_stride, int page_size, int heads, int kv_heads, int dim, int vdim, int dims, int interleaved,
                                  const float* freq, float mag, const pk_qk_prep* prep, int tokens, int f32, pk_stream st) {
  if (!qkv || !positions || !q_out || !prep || (!prep->q_only && (!req || !page_off || !pages || !cache)) || tokens <= 0 || heads <= 0 || kv_heads <= 0 ||
      heads % kv_heads || dim <= 0 || vdim <= 0 || dims < 0 || dims > dim || (dims & 1) || (dims > 0 && !freq) || page_size <= 0 ||
      prep->norm_kind < 0 || prep->norm_kind > 2 || (prep->norm_kind == 2 && (!prep->q_weight || !prep->k_weight)) ||
      (prep->norm_kind == 1 && (!prep->q_weight != !prep->k_weight)) || prep->temp_every < 0 ||
      (prep->values_are_keys && vdim != dim))
    return -1;
  const size_t smem = ((size_t)(heads + kv_heads) * dim + heads + kv_heads) * sizeof(float);
  if (smem > 200 * 1024) return -2;
  const int threads = tokens > 64 ? 256 : std::min(1024, std::max(128, ((heads + kv_heads) * dim / 2 + 31) / 32 * 32));
#define PK_NA(E)                                                                                                                                   \
  do {                                                                                                                                             \
    if (smem > 48 * 1024) cudaFuncSetAttribute(gqa_norm_append_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);                \
    launch(gqa_norm_append_kernel<E>, dim3(tokens), dim3(threads), smem, st, true, (const E*)qkv, ld, positions, req, page_off, pages, (E*)q_out,  \
           (E*)cache, page_stride, page_size, heads, kv_heads, dim, vdim, dims, interleaved, freq, mag, (const E*)prep->q_weight,                  \
           (const E*)prep->k_weight, prep->norm_kind, prep->eps, prep->temp_coef, prep->temp_every, prep->values_are_keys,                      \
           prep->q_only);                        \
  } while (0)
  if (f32) PK_NA(float);
  else PK_NA(bf16);
#undef PK_NA
  return (int)cudaGetLastError();
}

extern "C" int pk_gqa_attention(const void* q, const void* cache, const void* sink, const int* positions, const int* req, const int* page_off,
                                const int* pages, void* out, long page_stride, int page_size, int tokens, int heads, int kv_heads, int dim,
                                int vdim, float scale, int chunk, int f32, pk_stream st) {
  return pk_gqa_attention_ex(q, cache, sink, positions, req, page_off, pages, out, page_stride, page_size, tokens, heads, kv_heads, dim, vdim, scale,
                             chunk, nullptr, f32, st);
}

extern "C" int pk_gqa_attention_ex(const void* q, const void* cache, const void* sink, const int* positions, const int* req, const int* page_off,
                                   const int* pages, void* out, long page_stride, int page_size, int tokens, int heads, int kv_heads, int dim,
                                   int vdim, float scale, int chunk, const pk_attn_extra* extra, int f32, pk_stream st) {
  if (!q || !cache || !positions || !req || !page_off || !pages || !out || tokens <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads ||
      dim <= 0 || vdim <= 0 || chunk < 0 || page_size <= 0)
    return -1;
  AttnExtra x{0, 0.f, 0.f, nullptr, 0, 0, 0, 0, (long)heads * vdim};
  if (extra) {
    if (extra->window < 0 || extra->softcap < 0.f || extra->slope_log2 < 0.f || extra->max_kv_len < 0 || extra->keep_first < 0 ||
        (extra->out_ld && extra->out_ld < (long)heads * vdim))
      return -1;
    x = AttnExtra{extra->window,     extra->softcap,    extra->slope_log2, extra->gate, extra->gate_ld,
                  extra->max_kv_len, extra->window > 0 ? extra->keep_first : 0, extra->gate_per_head, extra->out_ld ? extra->out_ld : (long)heads * vdim};
  }
  if (dim > 32 * kGqaMaxPerLane || vdim > 32 * kGqaMaxPerLane) return -2;
  const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                       page_stride % 8 == 0 && x.out_ld % 2 == 0;
  // bf16 prompt portions always; single decoded tokens too when the caller asked through the _ex entry (the key axis is then split)
  if (!f32 && (tokens >= 32 || extra) && aligned && dim == vdim && (dim == 64 || dim == 128 || dim == 32 || dim == 96) && (dim * kv_heads) % 8 == 0) {
#define PK_GQA_MMA(D) \
  launch_gqa_mma<D>((const bf16*)q, (const bf16*)cache, (const bf16*)sink, positions, req, page_off, pages, (bf16*)out, page_stride, page_size, tokens, heads, kv_heads, scale, chunk, x, st)
    if (dim == 32) PK_GQA_MMA(32);
    else if (dim == 64) PK_GQA_MMA(64);
    else if (dim == 96) PK_GQA_MMA(96);
    else PK_GQA_MMA(128);
#undef PK_GQA_MMA
    return (int)cudaGetLastError();
  }
  const size_t smem = (size_t)kGqaWarps * vdim * sizeof(float);
  if (f32)
    launch(gqa_attention_kernel<float>, dim3(tokens, heads), dim3(kGqaWarps * 32), smem, st, true, (const float*)q, (const float*)cache, (const float*)sink,
           positions, req, page_off, pages, (float*)out, page_stride, page_size, heads, kv_heads, dim, vdim, scale, chunk, x);
  else
    launch(gqa_attention_kernel<bf16>, dim3(tokens, heads), dim3(kGqaWarps * 32), smem, st, true, (const bf16*)q, (const bf16*)cache, (const bf16*)sink,
           positions, req, page_off, pages, (bf16*)out, page_stride, page_size, heads, kv_heads, dim, vdim, scale, chunk, x);
  return (int)cudaGetLastError();
}
