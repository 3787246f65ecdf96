// Prefill GEMM on CTA PAIRS: Y[M, N] = W[M, K] x X[K, N] with tcgen05.mma.cta_group::2.
//
// Why: the single-CTA kernel (gemm.cu, cta_group::1, M128 x N256 x K16 per instruction) reads 12 KB of operands from
// shared memory per 128-cycle instruction and TMA writes another 12 KB: ~190 B/clk against a 128 B/clk shared-memory
// port.  ncu shows the tensor pipe 61-64 % active and cuBLAS' sm_100 kernels
// 1.27-1.53 PFLOP/s against our 0.77-1.20 on the same shapes.  A CTA pair (two SMs of one TPC) computes a
// 256-token x BN-feature tile: each CTA stages its OWN 128 tokens of A and only HALF of B (BN/2 features), the
// pair's tensor cores share the B halves, so per SM the operand traffic is 8 KB read + 8 KB written per instruction.
//
//   cluster (2,1,1): rank 0 = leader.   A = X [tokens, K] (UMMA M = 256 tokens, 128 per CTA), B = W [features, K]
//   (UMMA N = BN features, BN/2 per CTA), D in TMEM: each CTA holds its 128 token rows x BN columns (fp32), double buffered.
//   warp 0  TMA producer (both CTAs): A tile + B half per stage, complete_tx on the LEADER's full barrier
//           (cp.async.bulk.tensor ... .cta_group::2); the leader arms it with the bytes of both CTAs
//   warp 1  MMA issuer (leader only): tcgen05.mma.cta_group::2 M256 x BN x K16, tcgen05.commit ... multicast::cluster
//           frees the stage in BOTH CTAs / publishes the accumulator to BOTH epilogues
//   warps 2-9 epilogue (both CTAs): tcgen05.ld 32x32b.x32 -> bf16 -> 64-byte row stores; tmem-empty arrives on the
//           leader's barrier (remote mbarrier arrive for the peer)
// SwiGLU mode (gate_up projection): the pair's B halves are the SAME 128 features of the gate block (leader CTA) and
// of the up block (peer CTA) of the stacked [gate; up] weight, so columns [0,128) / [128,256) of every accumulator row
// are gate / up of one feature: the epilogue writes bf16(silu(bf16(g)) * bf16(u)) (csrc/fused_proj.cu:44-63 rounding)
// and the separate SiLU-mul pass over 2*I*T elements disappears.
// The MMA issuer and the producer are threads chosen by elect.sync: with threads picked by `lane == 0` a K block took 0.42 us whatever the tile's width.
// B200, us a launch over cold weights, before -> after (2048 tokens):
// 6144 x 2560 59.5 -> 48.4, 2560 x 4096 45.6 -> 37.5, 2560 x 9728 88.8 -> 74.3, 4096 x 12288 160.6 -> 144.1.
// The gated epilogue evaluates its 32 columns side by side, on two warps per lane quarter; one after the other (a branch on the activation per
// element) a tile's epilogue took 26 us and set the pace: 9728 x 2560 gated 253 -> 154, 12288 x 4096 gated (3001 tokens) 557 -> 433.
// Every barrier wait is bounded (mbar_wait_bounded, common.cuh).
#include <cuda.h>

#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "tcgen05.cuh"

namespace pk {

namespace {

constexpr int G2_BM = 128;       // tokens per CTA (UMMA M = 256 per pair)
constexpr int G2_BK = 64;        // K elements per stage (one 128-byte swizzle span)
constexpr int G2_EPI = 8;        // epilogue warps: two for each quarter of the TMEM lanes, taking turns at blocks of 32 columns
constexpr int G2_THREADS = 64 + 32 * G2_EPI;  // warp 0 TMA, warp 1 MMA, then the epilogue

struct G2Args {
  bf16 *Y, *Y1, *Y2;
  int e0, e1;     // output segments (the fused q|k|v projection): features [0,e0) -> Y, [e0,e1) -> Y1, rest -> Y2
  int M, N, K;    // features, tokens, reduction
  int swiglu;     // 1: W = [gate (M rows); up (M rows)], Y[tok][M] = silu(gate) * up; 2: relu(gate) * up; 3: gelu (tanh form) of gate * up
  int ldy;        // gated output: elements from one token's row to the next
  unsigned int* err;  // wait_err_word()
};

// A pair tile is 256 tokens x (NSUB * BN) features: NSUB accumulators of BN columns side by side in TMEM, one
// tcgen05.mma per accumulator per K step (NSUB = 2, BN = 160: the 320-wide tile that turns the 2560-feature
// projections of Qwen3-4B into ONE wave of 64 tiles on 74 pairs instead of two waves of 256-wide tiles).
template <int BN, int NSUB, int STAGES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2_THREADS, 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const G2Args a) {
  constexpr int HB = BN / 2;          // B rows (features) staged per CTA per accumulator
  constexpr int TN = NSUB * BN;       // features per tile
  constexpr int A_BYTES = G2_BM * G2_BK * 2, B_SUB = HB * G2_BK * 2, B_BYTES = NSUB * B_SUB, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int NBUF = (2 * TN <= 512) ? 2 : 1;  // TMEM accumulator buffers
  constexpr uint32_t TMEM_COLS = (NBUF * TN <= 256) ? 256 : 512;
  static_assert(B_SUB % 1024 == 0, "each B sub-tile must start on a swizzle-atom boundary");
  static_assert(NSUB == 1 || TN <= 512, "accumulators exceed TMEM");
  extern __shared__ uint8_t g2_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(g2_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);  // used in the leader
  uint64_t* empty = full + STAGES;   // one per CTA (multicast commit)
  uint64_t* tfull = empty + STAGES;  // [2] one per CTA
  uint64_t* tempty = tfull + 2;      // [2] used in the leader (an arrival per epilogue warp of both CTAs)
  uint64_t* done = tempty + 2;       // behind a run-out: the MMAs under way
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * STAGES + 5) * 8 + 8 <= 256, "room behind the stages");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int M = a.M, N = a.N, K = a.K;
  const int m_tiles = (N + 2 * G2_BM - 1) / (2 * G2_BM);  // pair tiles along tokens
  const int n_tiles = a.swiglu ? (M + HB - 1) / HB : (M + TN - 1) / TN;
  const int num_tiles = m_tiles * n_tiles;
  const int k_blocks = (K + G2_BK - 1) / G2_BK;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull + s, 1);
      mbar_init(tempty + s, 2 * G2_EPI);
    }
    mbar_init(done, 1);
    *dead = 0;
    mbar_fence_init();
  }
  if (warp == 1) g2_tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_barrier();  // both CTAs' barriers are initialised and both TMEM allocations are done
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (tc_elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
      int it = 0;
      bool go = true;
      for (int tile = pair; tile < num_tiles && go; tile += num_pairs) {
        const int mb = tile % m_tiles, nb = tile / m_tiles;
        const int tok0 = mb * 2 * G2_BM + (int)rank * G2_BM;
        // this CTA's B rows: its half of the BN features, or (SwiGLU) the gate block (leader) / up block (peer)
        const int wrow0 = a.swiglu ? (int)rank * M + nb * HB : nb * TN + (int)rank * HB;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          go = mbar_wait_bounded(empty + s, (uint32_t)(((it / STAGES) & 1) ^ 1), dead);
          if (!go) break;
          const uint32_t fb = g2_map(smem_u32(full + s), 0);
          if (leader) mbar_expect_tx(full + s, 2 * STAGE_BYTES);
          uint8_t* st = smem + (size_t)s * STAGE_BYTES;
          g2_tma_2d(st, &map_x, kb * G2_BK, tok0, fb);
#pragma unroll
          for (int j = 0; j < NSUB; ++j) g2_tma_2d(st + A_BYTES + j * B_SUB, &map_w, kb * G2_BK, wrow0 + j * BN, fb);
        }
      }
      if (!go) wait_for_copies();  // (some complete on the leader's barriers)
    }
  } else if (warp == 1) {
    // by elect.sync, not by `lane == 0` (see the head of this file)
    if (leader && tc_elect_one()) {
      // instruction descriptor: D=f32 [4,6)=1, A=bf16 [7,10)=1, B=bf16 [10,13)=1, K-major both, N>>3 at [17,23), M>>4 at [24,29)
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      int it = 0, lt = 0;
      bool go = true;
      for (int tile = pair; tile < num_tiles && go; tile += num_pairs, ++lt) {
        const int as = lt % NBUF;
        go = mbar_wait_bounded(tempty + as, (uint32_t)(((lt / NBUF) & 1) ^ 1), dead);
        if (!go) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(as * TN);
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          go = mbar_wait_bounded(full + s, (uint32_t)((it / STAGES) & 1), dead);
          if (!go) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + (size_t)s * STAGE_BYTES);
          const uint64_t adesc = make_sw128_desc(a_addr);
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k)
#pragma unroll
            for (int j = 0; j < NSUB; ++j)
              g2_umma(d_tmem + (uint32_t)(j * BN), adesc + (uint64_t)(k * 2),
                      make_sw128_desc(a_addr + A_BYTES + j * B_SUB) + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          g2_commit_both(empty + s);
        }
        g2_commit_both(tfull + as);
      }
      if (!go) {
        g2_commit_both(done);
        mbar_drain(done, 0);
      }
    }
  } else {
    const int q = warp & 3, c0 = (warp - 2) / 4 * 32;  // TMEM lane quarter this warp may access, its first column
    const bool vec_ok = (a.e0 % 32 == 0) && (a.e1 % 32 == 0) && (M % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.Y) & 15) == 0) &&
                        ((reinterpret_cast<uintptr_t>(a.Y1) & 15) == 0) && ((reinterpret_cast<uintptr_t>(a.Y2) & 15) == 0);
    const uint32_t tempty_leader0 = g2_map(smem_u32(tempty), 0);
    int lt = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs, ++lt) {
      const int mb = tile % m_tiles, nb = tile / m_tiles;
      const int as = lt % NBUF;
      mbar_wait_bounded(tfull + as, (uint32_t)((lt / NBUF) & 1), dead);
      tc_fence_after();
      const int tok = mb * 2 * G2_BM + (int)rank * G2_BM + q * 32 + lane;
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * TN);
      // 32 columns of the warp's 32 rows, four lanes 64 bytes of a row at a time: a lane that stored its own row would touch a line per 16 bytes, and a tile of
      // 256 columns would take 4100 clocks to leave -- the last one of a launch, or the only one, with nothing beside it (2560 x 4096, 2048 tokens: 33.8 -> 31.6 us,
      // 12288 x 2560, 200 tokens 23.3 -> 18.6)
      auto store_rows = [&](bf16* base, int ld, const float* r) {
        uint32_t u[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) u[j] = pack_bf16(r[2 * j], r[2 * j + 1]);
        transpose4(u, lane);
        const int tok4 = tok & ~3;
        bf16* dst = base + (size_t)tok4 * ld + (lane & 3) * 8;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (tok4 + j < N) *reinterpret_cast<uint4*>(dst + (size_t)j * ld) = make_uint4(u[4 * j], u[4 * j + 1], u[4 * j + 2], u[4 * j + 3]);
      };
      if (a.swiglu) {
        // columns [0, HB) = gate, [HB, BN) = up of features nb*HB + c
#pragma unroll 1
        for (int c = c0; c < HB; c += 8 * G2_EPI) {
          uint32_t gv[32], uv[32];
          tmem_ld32_nowait(t_row + (uint32_t)c, gv);
          tmem_ld32(t_row + (uint32_t)(HB + c), uv);
          const int f0 = nb * HB + c;
          if (tok - lane < N && f0 < M) {  // (a warp at a time: the lanes store for one another)
            // one loop per activation and step: a branch per element would leave the elements' long chains one behind the other
            float g[32], u[32], r[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              // gate_up_out is bf16 in the reference.  1 behind the last token: a division of zero leaves its fast path (9728 x 2560, 200 tokens: 42 us for 30)
              g[j] = tok < N ? round_bf16(__uint_as_float(gv[j])) : 1.f;
              u[j] = round_bf16(__uint_as_float(uv[j]));
            }
            if (a.swiglu == 2) {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = fmaxf(g[j], 0.f) * u[j];
            } else if (a.swiglu == 3) {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = gelu_tanh_gate(g[j]) * u[j];
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = 1.0f + expf(-g[j]);
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = g[j] / r[j] * u[j];
            }
            if (M % 8 == 0 && a.ldy % 8 == 0 && f0 + 32 <= M && (reinterpret_cast<uintptr_t>(a.Y) & 15) == 0) {
              store_rows(a.Y + f0, a.ldy, r);
            } else if (tok < N) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (f0 + j < M) a.Y[(size_t)tok * a.ldy + f0 + j] = f2bf(r[j]);
            }
          }
        }
      } else {
#pragma unroll 1
        for (int c = c0; c < TN; c += 8 * G2_EPI) {
          uint32_t v[32];
          tmem_ld32(t_row + (uint32_t)c, v);
          const int f0 = nb * TN + c;
          if (tok - lane < N && f0 < M) {  // (a warp at a time: the lanes store for one another)
            if (vec_ok && f0 + 32 <= M) {
              if (f0 < a.e0) store_rows(a.Y + f0, a.e0, reinterpret_cast<const float*>(v));
              else if (f0 < a.e1) store_rows(a.Y1 + (f0 - a.e0), a.e1 - a.e0, reinterpret_cast<const float*>(v));
              else store_rows(a.Y2 + (f0 - a.e1), M - a.e1, reinterpret_cast<const float*>(v));
            } else if (tok < N) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int f = f0 + j;
                if (f >= M) break;
                bf16* d1 = f < a.e0 ? a.Y + (size_t)tok * a.e0 + f
                                    : (f < a.e1 ? a.Y1 + (size_t)tok * (a.e1 - a.e0) + (f - a.e0) : a.Y2 + (size_t)tok * (M - a.e1) + (f - a.e1));
                *d1 = f2bf(__uint_as_float(v[j]));
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) g2_arrive_cluster(tempty_leader0 + (uint32_t)(as * 8));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_barrier();  // the peer's MMAs / loads may still target this CTA's shared memory and TMEM
  if (warp == 1) {
    tc_fence_after();
    g2_tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0) count_run_out(dead, a.err);
}

template <int BN, int NSUB, int STAGES>
cudaError_t g2_launch(const CUtensorMap& mx, const CUtensorMap& mw, const G2Args& a, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (G2_BM * G2_BK * 2 + NSUB * (BN / 2) * G2_BK * 2) + 1024 + 256;
  auto kern = gemm_tc2_kernel<BN, NSUB, STAGES>;
  static thread_local bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return cudaErrorInvalidValue;
    configured = true;
  }
  const int m_tiles = (a.N + 2 * G2_BM - 1) / (2 * G2_BM);
  const int n_tiles = a.swiglu ? (a.M + BN / 2 - 1) / (BN / 2) : (a.M + NSUB * BN - 1) / (NSUB * BN);
  const int tiles = m_tiles * n_tiles;
  int pairs = sm_count() / 2;
  if (pairs > tiles) pairs = tiles;
  if (pairs < 1) pairs = 1;
  return launch(kern, dim3(2 * pairs), dim3(G2_THREADS), smem, stream, true, mx, mw, a);
}

}  // namespace

// Tile choice by wave count: a wave of tiles takes as long as its width + 32 columns (M = 6144, K = 2560, B200: 9.2 us a wave at 128 columns, 10.5 at
// 160, 12.9 at 192, 14.8 at 224, 16.8 at 256, beside 6 us once), so the width whose last wave is fullest wins:
//   M x K, tokens           256     224     192     160     128     us a launch over cold weights
//   6144 x 2560,  400       23.3    21.2    19.1    25.2    23.1
//   6144 x 2560, 1024       34.0    31.4    28.0    33.4    29.4
//   2560 x 4096, 1024       33.9    29.2    27.0    23.5    32.9
//   2560 x 9728, 1024       55.1    49.8    43.6    39.5    58.9
//   2560 x 9728, 3001      111.2   105.2   129.8   112.4   124.0
//   9728 x 2560,  400       57.9            53.9            53.5    (gated)
//   4096 x 12288, 4096     305.2   378.3   332.9   336.4   331.9
// (A launch has since become 1 to 3 us shorter at every width: how the results leave, see store_rows.)
// Beyond three waves of 256 the last one matters less than what narrower tiles read more often, and 256 columns stand.
// In the units of gemm.cu's model: a pair tile of 256 tokens on sms/2 pairs costs what a 128-token tile of the same width costs on sms single CTAs.
// Returns the index into g2_widths, or -2 when the single-CTA kernel of gemm.cu should take the shape.
// Pure host arithmetic (exported as pk_b200_gemm_plan so the calibration is pinned by a CPU test).
struct G2Width {
  int bn, nsub;  // columns per accumulator, accumulators per tile
  bool gated;    // halves of 32 columns each: a gated tile's epilogue reads gate and up 32 columns at a time
};
constexpr int kG2Widths = 6;
constexpr G2Width g2_widths[kG2Widths] = {{256, 1, true}, {160, 2, false}, {128, 1, true}, {192, 1, true}, {160, 1, false}, {224, 1, false}};

static int g2_plan(int M, int N, int K, int swiglu, int sms) {
  if (K % 8 != 0 || M <= 0 || sms < 2) return -2;
  if (N <= G2_BM) return -2;  // one token tile: nothing for the second CTA of a pair to do
  const int pairs = sms / 2;
  const long m_tiles = (N + 2 * G2_BM - 1) / (2 * G2_BM);
  int best = -1;
  long best_cost = -1;
  for (int ci = 0; ci < kG2Widths; ++ci) {
    if (swiglu && !g2_widths[ci].gated) continue;
    const int bn = g2_widths[ci].bn, nsub = g2_widths[ci].nsub, tn = bn * nsub;
    const long nt = swiglu ? (M + bn / 2 - 1) / (bn / 2) : (M + tn - 1) / tn;
    const long waves = (m_tiles * nt + pairs - 1) / pairs;
    if (ci >= 2 && m_tiles * (swiglu ? (M + 127) / 128 : (M + 255) / 256) > 3 * pairs) continue;
    // a 320-wide tile has ONE accumulator buffer in TMEM: its epilogue is not hidden behind the next tile's MMAs, so it only pays as a single wave
    const long cost = waves * (nsub == 2 ? tn + 64 + (waves > 1 ? tn / 3 : 0) : tn + 32);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = ci;
    }
  }
  if (!swiglu) {  // is the single-CTA kernel (gemm.cu: 128-token tiles of width 256 / 160 / 128 on every SM) strictly better?
    // One cost unit of the single-CTA kernel takes 1.75-2.3 x as long as one of the pair kernel (it is bound by its own
    // shared-memory port, see the header): at 2048 tokens o_proj 80.8 us (2 waves of 160-wide tiles, 384 units) vs 46.5 us
    // for the pair's one wave of 320-wide tiles (458 units), down_proj 173 vs 88 us.  Without
    // the factor the model sent both back to the single-CTA kernel (r2_v3_prefill_decode_launches.csv: 2 x 89 us per layer).
    const long m1 = (N + G2_BM - 1) / G2_BM;
    const int w1[3] = {256, 160, 128};
    for (int i = 0; i < 3; ++i) {
      const long waves = (m1 * ((M + w1[i] - 1) / w1[i]) + sms - 1) / sms;
      if (waves * (w1[i] + 32) * 7 / 4 < best_cost) return -2;
    }
  }
  return best;
}

// Returns 0 when launched, -2 when the shape / alignment is not for this kernel (caller uses the 1-CTA kernel).
int launch_gemm_pair(const bf16* W, const bf16* X, bf16* Y, bf16* Y1, bf16* Y2, int e0, int e1, int M, int N, int K, int swiglu, int ldy,
                     cudaStream_t stream) {
  if (K % 8 != 0 || (reinterpret_cast<uintptr_t>(W) & 15) != 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0) return -2;
  const int best = g2_plan(M, N, K, swiglu, sm_count());
  if (best < 0) return -2;
  G2Args a{Y, Y1, Y2, e0, e1, M, N, K, swiglu, ldy, wait_err_word()};
  CUtensorMap mx, mw;
  if (!make_rows_map(&mx, X, N, K, G2_BM)) return -2;
  const int rows_w = swiglu ? 2 * M : M;
  if (!make_rows_map(&mw, W, rows_w, K, g2_widths[best].bn / 2)) return -2;
  cudaError_t e;
  switch (best) {
    case 0: e = g2_launch<256, 1, 6>(mx, mw, a, stream); break;
    case 1: e = g2_launch<160, 2, 5>(mx, mw, a, stream); break;
    case 2: e = g2_launch<128, 1, 8>(mx, mw, a, stream); break;
    case 3: e = g2_launch<192, 1, 7>(mx, mw, a, stream); break;
    case 4: e = g2_launch<160, 1, 8>(mx, mw, a, stream); break;
    default: e = g2_launch<224, 1, 7>(mx, mw, a, stream); break;
  }
  return e == cudaSuccess ? 0 : (int)e;
}

}  // namespace pk

// Which prefill GEMM kernel a [M features] x [N tokens] x [K] problem gets on a GPU with `sms` SMs: 128 .. 320 = tile
// width of the CTA-pair kernel, -2 = another kernel (gemm_skinny.cu, gemm.cu).  No CUDA call.
extern "C" int pk_b200_gemm_plan(int M, int N, int K, int swiglu, int sms) {
  const int best = pk::g2_plan(M, N, K, swiglu, sms);
  return best < 0 ? -2 : pk::g2_widths[best].bn * pk::g2_widths[best].nsub;
}
