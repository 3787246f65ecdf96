// The two products of moe.cu for a few tokens, bf16: a chosen expert's weight rows are read once for up to 16 tokens that chose it, and on the tensor cores.
//   up    hid[t, k, f] = act(W_up[ids[t, k]] x_t)             down  y[t] = sum_k wts[t, k] W_down[ids[t, k]] hid[t, k] (+ shared expert)
// The (token, choice) pairs are listed by expert, in entries of at most 16 pairs (every CTA lists them for itself: some hundred ids).  A CTA streams units
// of up to 16 weight rows of an entry's expert by bulk copies through rings in shared memory, one ring to a group of four warps that share the elements of a
// row and multiply with mma.sync: m = the entry's pairs, n = weight rows.  (16 rows and at most 16 pairs: a tcgen05
// tile would be 1/8 full, and the products are a twentieth of the time that the weights take.)
//   up    the units of all entries, one behind the other, in equal runs for the CTAs
//   down  each CTA has the same <= 16 rows of every entry: it holds all of a token's choices, and adds them in the order of k
// Bound by HBM: the bytes of the distinct experts, once per 16 pairs of one (entries are numbered by their first pair: a crowded expert's rows may
// have left L2 when its next entry asks for them).  A pair's sums do not depend on the other pairs.
// Both products, us, 64 experts of 2048 x 1408, top 6, relu^2, 1 / 3 / 8 / 16 / 31 tokens (B200; floor 11 29 61 89 107): 44 79 126 228 413 with the warp-per-row
// kernels of moe.cu, which read an expert's rows once per pair, 24 46 85 117 145 here; gated 54 89 179 314 581 -> 30 63 115 168 200; 16 experts of
// 1024 x 768, top 2, 1 / 8 / 31 tokens 14 23 46 -> 14 20 28.  8 / 16 / 24 / 31 tokens of which every second chooses the same six experts 126 224 323 408 -> 68 121
// 151 186, of which all do 119 220 320 403 -> 28 43 59 64.  On the way there: the copies of a stage by one warp 41 (1 token) and 296 (16), by eight 29 and 181
// (a warp's copies are issued one after the other), the pairs' rows out of L2 instead of through the ring 24 and 117 (half the copies, chunks twice as long).
#include "common.cuh"
#include "mma.cuh"

namespace pk {

constexpr int kMfGroups = 3, kMfWarps = 4 * kMfGroups, kMfLoads = 4, kMfThreads = 32 * (kMfWarps + kMfLoads), kMfRows = 16, kMfSlots = 16, kMfKc = 1024, kMfStages = 6, kMfOwn = kMfStages / kMfGroups;  // stages: a ring of its own for each group
constexpr int kMfStage = kMfRows * kMfKc * 2;             // a chunk of up to kMfKc elements of a unit's rows
constexpr int kMfPairs = 192;                             // pairs of a call at most: 31 tokens of 6 choices (a thread each, and 64 bytes of sums; 256 would fit)

static_assert(kMfPairs <= kMfThreads, "a thread per pair");

struct MfArgs {
  const bf16 *act, *w;     // rows of x (up) or hid (down); weights [experts][R][K]
  const int* ids;
  int pairs, top, R, K, kc, rows;  // kc: elements of a chunk; rows: per unit (<= 16)
  bf16* hid;               // up
  float p0, p1;
  const float *wts, *sg;   // down
  const bf16* shared;
  float* y;
  unsigned int* err;
};

struct MfSmem {
  uint64_t full[kMfStages], empty[kMfStages];
  alignas(16) int ids[kMfPairs];  // padded with -1
  short list[kMfPairs];    // pairs by entry
  int expert[kMfPairs];    // of an entry
  short start[kMfPairs + 1];
  int wsum[kMfWarps + kMfLoads], dead;
  alignas(16) float part[kMfWarps][kMfSlots][kMfRows];  // the warps' sums of a unit
};

// GATED as in moe.cu; DOWN: the second product
template <int GATED, bool DOWN>
__global__ void __launch_bounds__(kMfThreads, 1) moe_few_kernel(const MfArgs a) {
  extern __shared__ __align__(128) uint8_t mf_smem[];
  uint8_t* ring = mf_smem;
  MfSmem& m = *reinterpret_cast<MfSmem*>(mf_smem + (size_t)kMfStages * kMfStage);
  float* dots = reinterpret_cast<float*>(&m + 1);  // DOWN: [pairs][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, P = a.pairs;
  if (tid == 0) {
    for (int s = 0; s < kMfStages; ++s) {
      mbar_init(m.full + s, kMfLoads);
      mbar_init(m.empty + s, 4);
    }
    m.dead = 0;
    mbar_fence_init();
  }
  volatile int* dead = &m.dead;
  pdl_wait();
  pdl_launch_dependents();  // the next kernel may start its launch; it waits for this grid to finish before it reads
  // ---- entries
  const int P4 = (P + 3) & ~3;
  for (int p = tid; p < P4; p += kMfThreads) m.ids[p] = p < P ? a.ids[p] : -1;
  __syncthreads();
  // a thread per pair: earlier pairs of its expert, all of them, and whether an entry begins with it
  int at = 0, all = 0;
  if (tid < P) {
    const int e = m.ids[tid];
    for (int i = 0; i < P4; i += 4) {
      const int4 v = *reinterpret_cast<const int4*>(m.ids + i);
      const int o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        all += o[k] == e;
        at += o[k] == e && i + k < tid;
      }
    }
  }
  const bool head = tid < P && at % kMfSlots == 0;
  const unsigned heads = __ballot_sync(0xffffffffu, head);  // exclusive sum over the threads = the entry's number
  if (lane == 0) m.wsum[warp] = __popc(heads);
  __syncthreads();
  int before = __popc(heads & ((1u << lane) - 1)), entries = 0;
  for (int w = 0; w < kMfWarps + kMfLoads; ++w) {
    if (w < warp) before += m.wsum[w];
    entries += m.wsum[w];
  }
  if (head) {
    m.expert[before] = m.ids[tid];
    m.list[tid] = (short)before;  // (for now: the entry that this pair begins)
    m.start[before + 1] = (short)min(kMfSlots, all - at);
  }
  if (tid == 0) m.start[0] = 0;
  __syncthreads();
  int entry = -1;
  if (tid < P) {  // the entry's first pair: the expert's (at - at % 16)-th
    int h = tid;
    for (int back = at % kMfSlots; back > 0;) back -= m.ids[--h] == m.ids[tid];
    entry = m.list[h];
  }
  __syncthreads();
  if (warp == 0) {  // starts: inclusive sums of the sizes
    int carry = 0;
    for (int i = 0; i < entries; i += 32) {
      int v = i + lane < entries ? m.start[i + lane + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (i + lane < entries) m.start[i + lane + 1] = (short)(carry + v);
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  if (entry >= 0) m.list[m.start[entry] + at % kMfSlots] = (short)tid;
  __syncthreads();

  // ---- units: a piece of work (up: this CTA's run of the units of all entries; down: all entries for a block of rows) after the other, in rounds of
  // kMfGroups units, one to a group of four warps.  Stages: the round's units in turn, chunk by chunk.
  const int K = a.K, kc = a.kc, chunks = (K + kc - 1) / kc, groups = (a.R + a.rows - 1) / a.rows;
  const long units = (long)entries * groups;
  const int u0 = DOWN ? 0 : (int)(units * blockIdx.x / gridDim.x), n_units = DOWN ? entries : (int)(units * (blockIdx.x + 1) / gridDim.x) - u0;
  struct Unit {
    int e, r0, nr, n;  // entry, first row, rows, pairs
  };
  auto unit = [&](int blk, int u) {
    Unit x;
    x.e = DOWN ? u : (u0 + u) / groups;
    x.r0 = DOWN ? blk * a.rows : (u0 + u) % groups * a.rows;
    x.nr = min(a.rows, a.R - x.r0);
    x.n = m.start[x.e + 1] - m.start[x.e];
    return x;
  };
  const int blk0 = DOWN ? (int)blockIdx.x : 0, blk_end = DOWN ? groups : 1;
  if (warp >= kMfWarps) {
    // Loads: the rows of a stage in turn, four to a warp.  A warp issues its lanes' copies one after the other, about 160 clocks each, so that one warp
    // alone set the pace
    const int mine = lane * kMfLoads + warp - kMfWarps;  // row of the stage
    const uint64_t pol = l2_evict_first_policy();
    int fills[kMfGroups] = {};
    bool go = true;
    for (int blk = blk0; blk < blk_end && go; blk += gridDim.x)
      for (int first = 0; first < n_units && go; first += kMfGroups) {
        const int live = min(kMfGroups, n_units - first);
        const bf16* src[kMfGroups];
        uint32_t rows[kMfGroups];
#pragma unroll
        for (int g = 0; g < kMfGroups; ++g) {
          src[g] = nullptr;
          if (g < live) {
            const Unit x = unit(blk, first + g);
            if (mine < x.nr) src[g] = a.w + ((size_t)m.expert[x.e] * a.R + x.r0 + mine) * K;
          }
          rows[g] = (uint32_t)__popc(__ballot_sync(0xffffffffu, src[g] != nullptr));
        }
        for (int c = 0; c < chunks && go; ++c) {
          const uint32_t bytes = (uint32_t)min(kc, K - c * kc) * 2;
#pragma unroll
          for (int g = 0; g < kMfGroups; ++g) {
            if (g >= live) break;
            const int s = g * kMfOwn + fills[g] % kMfOwn;
            if (lane == 0) {
              go = mbar_wait_bounded(m.empty + s, ((uint32_t)(fills[g] / kMfOwn) & 1u) ^ 1u, dead);
              if (go) mbar_expect_tx(m.full + s, bytes * rows[g]);
            }
            go = __shfl_sync(0xffffffffu, go, 0);
            if (!go) break;
            if (src[g]) bulk_g2s(ring + (size_t)s * kMfStage + (size_t)mine * kc * 2, src[g] + c * kc, bytes, m.full + s, pol);
            ++fills[g];
          }
        }
      }
    // Behind a run-out no barrier says when the copies under way have landed: two milliseconds, where a copy takes a thousandth of that
    if (!go)
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  const int group = warp >> 2, wg = warp & 3, g = lane >> 2, tq = lane & 3;
  auto bar = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
  auto bar_all = [] { asm volatile("bar.sync 14, %0;" ::"n"(32 * kMfWarps) : "memory"); };
  int used = 0;  // stages of this group
  for (int blk = warp < kMfWarps ? blk0 : blk_end; blk < blk_end; blk += gridDim.x) {
    for (int first = 0; first < n_units; first += kMfGroups) {
      const int live = min(kMfGroups, n_units - first);
      if (group < live) {
        const Unit x = unit(blk, first + group);
        float acc[2][2][2][4] = {};  // [8 pairs][8 weight rows][chain]
        const bf16* xr[2];           // rows of the pairs in slots g and 8 + g
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int p = i * 8 + g < x.n ? m.list[m.start[x.e] + i * 8 + g] : -1;
          xr[i] = p < 0 ? nullptr : a.act + (size_t)(DOWN ? p : p / a.top) * K + tq * 8;
        }
        for (int c = 0; c < chunks; ++c, ++used) {
          const int nvec = min(kc, K - c * kc) >> 3, s = group * kMfOwn + used % kMfOwn;
          const uint8_t* st = ring + (size_t)s * kMfStage + g * kc * 2;
          // which elements an instruction calls k is free as long as both operands agree: a lane takes 16-byte pieces of its rows.  The rows lie in the
          // same banks, so odd weight rows take the halves of a block of 64 elements the other way round; m rows 8 .. 15 hold the pairs in that order, and
          // of the products the even columns of the upper half and the odd ones of the lower are used.  The pairs' rows come out of L2 (L1 for the entry's
          // next units): asked for before the wait.
          constexpr int NB = kMfKc / 256;  // blocks of a warp at most
          auto ld_x = [&](int i, int piece) { return xr[i] && piece < nvec ? *reinterpret_cast<const uint4*>(xr[i] + c * kc + (piece & ~3) * 8) : make_uint4(0u, 0u, 0u, 0u); };
          uint4 xv[NB][2];
#pragma unroll
          for (int k = 0; k < NB; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) xv[k][h] = ld_x(0, (wg + 4 * k) * 8 + h * 4 + tq);
          mbar_wait_bounded(m.full + s, (uint32_t)(used / kMfOwn) & 1u, dead);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < NB; ++k) {
            const int b = (wg + 4 * k) * 8;
            if (b >= nvec) break;
            uint4 w[2][2];  // behind the row's end: nothing (shared memory may hold anything there)
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int piece = b + tq + ((g & 1) ^ h) * 4;
                w[t][h] = piece < nvec ? *reinterpret_cast<const uint4*>(st + t * 8 * kc * 2 + piece * 16) : make_uint4(0u, 0u, 0u, 0u);
              }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (i * 8 >= x.n) break;
              const uint4 xa = i ? ld_x(1, b + tq) : xv[k][0], xb = i ? ld_x(1, b + 4 + tq) : xv[k][1];
              const uint32_t a0[4] = {xa.x, xb.x, xa.y, xb.y}, a1[4] = {xa.z, xb.z, xa.w, xb.w};
              const uint32_t a2[4] = {xb.x, xa.x, xb.y, xa.y}, a3[4] = {xb.z, xa.z, xb.w, xa.w};
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                if (t * 8 >= x.nr) break;
                mma_bf16_16816(acc[i][t][0], a0, w[t][0].x, w[t][0].y);
                mma_bf16_16816(acc[i][t][1], a1, w[t][0].z, w[t][0].w);
                mma_bf16_16816(acc[i][t][0], a2, w[t][1].x, w[t][1].y);
                mma_bf16_16816(acc[i][t][1], a3, w[t][1].z, w[t][1].w);
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(m.empty + s);
        }
        // sum over the group's warps
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i * 8 >= x.n) break;
#pragma unroll
          for (int t = 0; t < 2; ++t)
            *reinterpret_cast<float2*>(&m.part[warp][i * 8 + g][t * 8 + 2 * tq]) = make_float2(acc[i][t][0][0] + acc[i][t][1][0], acc[i][t][0][3] + acc[i][t][1][3]);
        }
        bar();
        const int row = tid & 15;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i * 8 + wg * 2 >= x.n) break;  // (the warp's two slots)
          const int slot = i * 8 + ((tid & 127) >> 4);
          const float(*pt)[kMfSlots][kMfRows] = m.part + group * 4;
          const float d = (pt[0][slot][row] + pt[1][slot][row]) + (pt[2][slot][row] + pt[3][slot][row]);
          const int p = slot < x.n ? m.list[m.start[x.e] + slot] : 0;
          if (DOWN) {
            if (slot < x.n) dots[p * kMfRows + row] = d;
          } else if (GATED) {
            float up = __shfl_down_sync(0xffffffffu, d, 1), gt = d, r;
            if (GATED == 2) {
              gt = fminf(gt, a.p0);
              up = fminf(fmaxf(up, -a.p0), a.p0);
              r = gt / (1.f + expf(-a.p1 * gt)) * (up + 1.f);
            } else {
              r = gt / (1.f + expf(-gt)) * up;
            }
            if (slot < x.n && (row & 1) == 0 && row < x.nr) a.hid[(size_t)p * (a.R / 2) + (x.r0 + row) / 2] = f2bf(r);
          } else {
            const float r = fmaxf(d, 0.f);
            if (slot < x.n && row < x.nr) a.hid[(size_t)p * a.R + x.r0 + row] = f2bf(r * r);
          }
        }
        bar();  // (before the next unit's sums)
      }
    }
    if (DOWN) {  // all entries of these rows
      bar_all();
      const int r0 = blk * a.rows, nr = min(a.rows, a.R - r0);
      for (int i = tid; i < P / a.top * kMfRows; i += 32 * kMfWarps) {
        const int t = i / kMfRows, r = i % kMfRows;
        if (r >= nr) continue;
        float tot = 0.f;
        for (int k = 0; k < a.top; ++k) tot = fmaf(a.wts[t * a.top + k], dots[(t * a.top + k) * kMfRows + r], tot);
        const size_t o = (size_t)t * a.R + r0 + r;
        if (a.shared) tot += (a.sg ? 1.f / (1.f + expf(-a.sg[t])) : 1.f) * bf2f(a.shared[o]);
        a.y[o] = tot;
      }
      bar_all();  // (before the next rows' first)
    }
  }
  __syncthreads();  // every role is through with its waits
  if (tid == 0) count_run_out(dead, a.err);
}

static bool mf_takes(const void* act, const void* w, long pairs, int R, int K) {
  return pairs <= kMfPairs && K % 8 == 0 && R <= 1 << 20 && ((reinterpret_cast<uintptr_t>(act) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}
template <int GATED, bool DOWN>
static int mf_launch(MfArgs a, cudaStream_t st) {
  constexpr size_t fixed = (size_t)kMfStages * kMfStage + sizeof(MfSmem), most = fixed + (DOWN ? (size_t)kMfPairs * kMfRows * 4 : 0);
  static_assert(most <= 227 * 1024, "shared memory");
  static std::atomic<uint64_t> smem_set{0};
  if (allow_smem(smem_set, (const void*)moe_few_kernel<GATED, DOWN>, most) != cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  a.err = wait_err_word();
  const int chunks = (a.K + kMfKc - 1) / kMfKc;  // of equal length, whole blocks of 64 elements
  a.kc = ((a.K + chunks - 1) / chunks + 63) / 64 * 64;
  const long groups = (a.R + a.rows - 1) / a.rows, units = DOWN ? groups : groups * a.pairs;
  const int grid = (int)(units < sm_count() ? units : sm_count());
  return (int)launch(moe_few_kernel<GATED, DOWN>, dim3(grid), dim3(kMfThreads), fixed + (DOWN ? (size_t)a.pairs * kMfRows * 4 : 0), st, true, a);
}

// 0 = launched; -2 = not for these kernels (moe.cu has one for every shape)
int launch_moe_up_few(const bf16* x, const bf16* w, const int* ids, bf16* hid, int tokens, int top, int width, int ff, int act, float p0, float p1,
                      cudaStream_t st) {
  if (!mf_takes(x, w, (long)tokens * top, act ? 2 * ff : ff, width)) return -2;
  MfArgs a{};
  a.act = x;
  a.w = w;
  a.ids = ids;
  a.pairs = tokens * top;
  a.top = top;
  a.R = act ? 2 * ff : ff;
  a.K = width;
  a.rows = kMfRows;
  a.hid = hid;
  a.p0 = p0;
  a.p1 = p1;
  return act == 2 ? mf_launch<2, false>(a, st) : act == 1 ? mf_launch<1, false>(a, st) : mf_launch<0, false>(a, st);
}
int launch_moe_down_few(const bf16* hid, const bf16* w, const int* ids, const float* wts, const bf16* shared, const float* sg, float* y, int tokens, int top,
                        int width, int ff, cudaStream_t st) {
  if (!mf_takes(hid, w, (long)tokens * top, width, ff)) return -2;
  MfArgs a{};
  a.act = hid;
  a.w = w;
  a.ids = ids;
  a.pairs = tokens * top;
  a.top = top;
  a.R = width;
  a.K = ff;
  const int sms = sm_count(), rounds = (width + kMfRows * sms - 1) / (kMfRows * sms);  // blocks of rows for a CTA
  a.rows = (width + sms * rounds - 1) / (sms * rounds);
  a.wts = wts;
  a.sg = sg;
  a.shared = shared;
  a.y = y;
  return mf_launch<0, true>(a, st);
}

}  // namespace pk
