// Gated delta rule over a sequence in chunks of 16 tokens, fp32 throughout, for bf16 q / k / v and one decay per head (recurrent_mixers.cu,
// qwen35_ops.cu).  The recurrence  S <- g_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t  unrolled over a chunk that
// starts with state S0, with r(t, s) = g_(s+1) ... g_t and c_t = g_1 ... g_t:
//   w_t = beta_t (v_t - c_t S0^T k_t)                         u = (I + A)^-1 w,   A[t][s] = beta_t r(t, s) (k_t . k_s),  s < t
//   o_t = c_t S0^T q_t + sum_(s <= t) B[t][s] u_s             B[t][s] = r(t, s) (q_t . k_s)
//   S  <- c_16 S0 + sum_s r(16, s) k_s u_s^T
// so that the long products (S0 with 32 vectors, the update with 16) have no dependency from token to token, and what is left of the chain is a
// 16 x 16 triangle per chunk.  Factors r and c are products of decays, never quotients: nothing can overflow.
//
// CTA = (entry, head, COLS value columns).  Warps 0-3 hold S in fp32 registers, warp w the rows [w DK/4, (w+1) DK/4), as accumulators of
// S^T tiles (m16n8k16: m = column, n = row).  In that layout the state is also the B operand of the products with k and q, so it never moves.  The
// products run on the tensor cores without giving up fp32: k and q are bf16 rows, taken as they are (their unit factors are applied to the results),
// and an fp32 operand (S, u) enters as the sum of three bf16 parts, which hold all of its 24 bits, each part with an accumulator of its own or added
// smallest first; every product is exact and the sums are fp32.  What a chunk adds to S is summed from zero and added with one rounding.
// Warps 4-7 read out, a chunk behind: q . S0 of the four warps, and B u.
// The other warps each prepare every kDcPrep-th chunk by themselves, start to end (rows by cp.async, Gram matrices, decay products, the triangle's
// inverse by forward substitution with a lane per column), so that their latency is spread over kDcPrep chunks; they hand it over in a ring of stages.
// Bound by the chain products -> sum over the warps -> triangle -> update (three barriers of the four warps a chunk); the figures stand where it is launched.
// The roles' loops run side by side and have to share the SM's instruction cache: with the preparation unrolled to the end every role waited for its
// instructions (hit rate 0.69 in one form), so its loops are rolled as far as their latency allows; keys of 64 gain nothing by it.  2048 tokens, 16 heads of 128: 173 -> 149 us,
// 1024 tokens, 32 heads, 32 columns to a CTA: 180 -> 107 us (105 with the stages looked at early), 24 tokens 7.4 -> 6.8 us (B200, the kernel alone; same
// sums in the same order).
// Sums over s <= t leave the later tokens out by selection, not by a factor of zero: a NaN reaches the same tokens as token by token, and so does an
// infinity, as a NaN (its parts are differences of infinities).
#pragma once
#include "common.cuh"
#include "mma.cuh"

namespace pk {

constexpr int kDcT = 16;    // tokens per chunk
constexpr int kDcPrep = 4;  // preparing warps = stages; with 12 warps a thread may hold 168 registers (four of them were enough to keep the state warps busy)
constexpr int kDcThreads = 256 + 32 * kDcPrep;

struct DeltaRows {      // what one (entry, head) of the step works on
  const bf16 *q, *k, *v;  // first token's row of the head's q, k and (from the CTA's first column on) v; rows `ld` elements apart
  int ld, n;            // tokens
  bool vec;             // rows of q and k start on 16-byte boundaries
  float* state;         // [DK][vdim]
  int vdim, col0;       // first column of this CTA
  float unit_eps, q_scale;
  unsigned int* err;    // counts waits that ran out (null: not counted)
};

// shared-memory layout, in floats
template <int DK, int COLS>
struct DcSmem {
  static constexpr int LDR = DK + 8, PLD = COLS + 8, UBLD = 24;  // strides that keep fragment loads and partial stores free of bank conflicts
  // a stage
  static constexpr int RAW = 0;                        // bf16 [32][LDR]: k of 16 tokens, then q
  static constexpr int TM = RAW + 2 * kDcT * LDR / 2;  // [16][16]: (I + A)^-1
  static constexpr int BM = TM + 256;                  // [16][16]
  static constexpr int VB = BM + 256;                  // [16][COLS]: beta v
  static constexpr int CK = VB + kDcT * COLS;          // beta_t c_t kf_t
  static constexpr int CQ = CK + kDcT;                 // c_t qf_t
  static constexpr int CS = CQ + kDcT;                 // r(16, s) kf_s
  static constexpr int GC = CS + kDcT;                 // c_16 (4 floats)
  static constexpr int GM = GC + 4;                    // scratch: [2][16][17] k . k and q . k
  static constexpr int AM = GM + 2 * kDcT * 17;        // scratch: A [16][16]
  static constexpr int FT = AM + 256;                  // scratch: beta_t kf_t, qf_t, decays
  static constexpr int STAGE = FT + 3 * kDcT;
  // the four state warps
  static constexpr int WLD = kDcT + 4;                 // a column's 16 tokens, 16-byte reads without conflicts
  static constexpr int PK = kDcPrep * STAGE;           // [4][16][PLD]: S0^T k over each warp's rows
  static constexpr int PQ = PK + 4 * kDcT * PLD;       // two of [4][16][PLD]: S0^T q
  static constexpr int W = PQ + 2 * 4 * kDcT * PLD;    // [COLS][WLD]
  static constexpr int U = W + COLS * WLD;             // two of [COLS][WLD]
  static constexpr int UB = U + 2 * COLS * WLD;        // bf16 [3][COLS][UBLD]: the parts of u_s r(16, s) kf_s, transposed
  static constexpr int BARS = UB + 3 * COLS * UBLD / 2;
  static constexpr int FLOATS = BARS + 4 * kDcPrep + 4;
  static constexpr size_t BYTES = (size_t)FLOATS * 4;
  static_assert(STAGE % 4 == 0 && AM % 4 == 0 && PK % 4 == 0 && W % 4 == 0 && UB % 4 == 0 && BARS % 2 == 0, "alignment");
};

// x = hi + mid + lo, bf16 each: cut off after 8 and 16 of the 24 bits, so the sum is exact (for finite x that does not underflow)
__device__ __forceinline__ void dc_split(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t ux = __float_as_uint(x), uy = __float_as_uint(y);
    p[i] = __byte_perm(ux, uy, 0x7632);
    x -= __uint_as_float(ux & 0xffff0000u);
    y -= __uint_as_float(uy & 0xffff0000u);
  }
}

// `gates(t, g, beta)`: decay and write strength of token t (t < n).  `store(t, col, value)`: the read-out of token t.  All kDcThreads threads call.
template <int DK, int COLS, typename Gates, typename Store>
__device__ __forceinline__ void delta_chunks(const DeltaRows a, float* sm, Gates gates, Store store) {
  using L = DcSmem<DK, COLS>;
  constexpr int LDR = L::LDR, RW = DK / 4, RB = RW / 8, KS = RB / 2, MT = COLS / 16;  // rows, row blocks, k steps per warp; column tiles
  constexpr int NTK = COLS / 8;                                                      // (token, column) pairs per thread in the triangle
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n, n_chunks = (n + kDcT - 1) / kDcT;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + L::BARS);
  uint64_t* empty = full + kDcPrep;
  volatile int* dead = reinterpret_cast<volatile int*>(empty + kDcPrep);
  if (tid == 0) {
    for (int i = 0; i < kDcPrep; ++i) {
      mbar_init(full + i, 32);
      mbar_init(empty + i, 8);
    }
    *dead = 0;
    mbar_fence_init();
  }
  __syncthreads();
  const int fr = (lane & 7) + ((lane >> 3) & 1) * 8, fc = ((lane >> 4) & 1) * 8;  // this lane's row and column in a 16 x 16 ldmatrix.x4
  if (warp >= 8) {
    // ---- preparation
    constexpr int PR = DK / 8, NVL = kDcT * COLS / 32;  // 16-byte pieces per row; values per lane
    constexpr int ROLL_P = DK > 64 ? 4 : 8, ROLL_T = DK > 64 ? 8 : 16, ROLL_I = DK > 64 ? 1 : 4;  // rows of 64 leave room for more
    const int pw = warp - 8, half = lane >> 4, s = lane & 15;
    float* st = sm + pw * L::STAGE;
    bf16* raw = reinterpret_cast<bf16*>(st + L::RAW);
    uint32_t ph = 1;
    for (int b = pw; b < n_chunks; b += kDcPrep, ph ^= 1u) {
      const int t0 = b * kDcT, nb = min(kDcT, n - t0);  // tokens past the end: zero rows, decay 1, write strength 0
      mbar_wait_bounded(empty + pw, ph, dead);
      __syncwarp();
      if (a.vec) {
        const bf16* src = a.k + (size_t)t0 * a.ld + lane % PR * 8;
        const ptrdiff_t to_q = a.q - a.k;
        bf16* dst = raw + lane / PR * LDR + lane % PR * 8;
#pragma unroll ROLL_P
        for (int t = lane / PR; t < kDcT; t += 32 / PR, dst += 32 / PR * LDR) {
          const bf16* row = src + (ptrdiff_t)min(t, nb - 1) * a.ld;
          const uint32_t bytes = t < nb ? 16 : 0;  // zeros behind the end
          cp_async16(dst, row, bytes);
          cp_async16(dst + kDcT * LDR, row + to_q, bytes);
        }
      } else {
#pragma unroll 8
        for (int i = lane; i < 2 * kDcT * DK; i += 32) {
          const int row = i / DK, t = row & (kDcT - 1);
          raw[row * LDR + i % DK] = t < nb ? (row < kDcT ? a.k : a.q)[(size_t)(t0 + t) * a.ld + i % DK] : f2bf(0.f);
        }
      }
      cp_async_commit();
      {  // this warp's next chunk on its way to L2: a lane per row, two lines each
        const int t = t0 + kDcPrep * kDcT + s;
        if (t < n) {
          const bf16* src = (half ? a.q : a.k) + (size_t)t * a.ld;
          prefetch_l2(src);
          if (DK > 64) prefetch_l2(src + 64);
          if (half) prefetch_l2(a.v + (size_t)t * a.ld);
        }
      }
      float g = 1.f, beta = 0.f;
      if (half == 0 && s < nb) gates(t0 + s, g, beta);
      bf16 vr[NVL];
#pragma unroll
      for (int i = 0; i < NVL; ++i) {
        const int at = lane + 32 * i, t = at / COLS, c = at % COLS;
        vr[i] = t < nb && a.col0 + c < a.vdim ? a.v[(size_t)(t0 + t) * a.ld + c] : f2bf(0.f);
      }
      cp_async_wait_all();
      __syncwarp();
      // unit factors: lane = row
      float d[4] = {};
#pragma unroll ROLL_P
      for (int i = 0; i < PR; ++i) {
        const uint4 u = *reinterpret_cast<const uint4*>(raw + lane * LDR + i * 8);
        d[0] = fmaf(bf16_lo(u.x), bf16_lo(u.x), d[0]);
        d[1] = fmaf(bf16_hi(u.x), bf16_hi(u.x), d[1]);
        d[2] = fmaf(bf16_lo(u.y), bf16_lo(u.y), d[2]);
        d[3] = fmaf(bf16_hi(u.y), bf16_hi(u.y), d[3]);
        d[0] = fmaf(bf16_lo(u.z), bf16_lo(u.z), d[0]);
        d[1] = fmaf(bf16_hi(u.z), bf16_hi(u.z), d[1]);
        d[2] = fmaf(bf16_lo(u.w), bf16_lo(u.w), d[2]);
        d[3] = fmaf(bf16_hi(u.w), bf16_hi(u.w), d[3]);
      }
      const float unit = (half ? a.q_scale : 1.f) / sqrtf((d[0] + d[1]) + (d[2] + d[3]) + a.unit_eps);
      const float kf = __shfl_sync(0xffffffffu, unit, s), ft = half ? unit : beta * unit;
      st[L::FT + lane] = ft;
      if (half == 0) st[L::FT + 2 * kDcT + s] = g;
      // Gram matrices k . k and q . k.  A fragments are rows of k (q); as B operand (its columns are rows of k) the same registers serve: tokens
      // 0-7 in registers 0 and 2, 8-15 in 1 and 3.  Odd and even k steps add up apart.
      float kk[2][2][4] = {}, qk[2][2][4] = {};
#pragma unroll
      for (int k0 = 0; k0 < DK / 16; ++k0) {
        uint32_t fk[4], fq[4];
        ldsm_x4(fk, raw + fr * LDR + k0 * 16 + fc);
        ldsm_x4(fq, raw + (kDcT + fr) * LDR + k0 * 16 + fc);
        mma_bf16_16816(kk[k0 & 1][0], fk, fk[0], fk[2]);
        mma_bf16_16816(kk[k0 & 1][1], fk, fk[1], fk[3]);
        mma_bf16_16816(qk[k0 & 1][0], fq, fk[0], fk[2]);
        mma_bf16_16816(qk[k0 & 1][1], fq, fk[1], fk[3]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int at = ((lane >> 2) + (e >> 1) * 8) * 17 + j * 8 + (lane & 3) * 2 + (e & 1);
          st[L::GM + at] = kk[0][j][e] + kk[1][j][e];
          st[L::GM + kDcT * 17 + at] = qk[0][j][e] + qk[1][j][e];
        }
      __syncwarp();
      // lanes 0-15: column s of A;  16-31: column s of B
      float r = 1.f, c = 1.f, cs = 1.f;
      {
        const float* gm = st + L::GM + half * kDcT * 17 + s;
        float* to = st + (half ? L::BM : L::AM) + s;
#pragma unroll ROLL_T
        for (int t = 0; t < kDcT; ++t) {
          const float gt = st[L::FT + 2 * kDcT + t], f = st[L::FT + half * kDcT + t], m = gm[t * 17];
          r = t > s ? r * gt : r;
          c *= gt;
          cs = t == s ? c : cs;
          to[t * kDcT] = t > s || (half && t == s) ? (f * kf) * r * m : 0.f;
        }
      }
      st[(half ? L::CQ : L::CK) + s] = ft * cs;
      if (half == 0) st[L::CS + s] = r * kf;
      if (lane == 0) st[L::GC] = c;
#pragma unroll
      for (int i = 0; i < NVL; ++i) {
        const int at = lane + 32 * i;
        st[L::VB + at] = __shfl_sync(0xffffffffu, beta, at / COLS) * bf2f(vr[i]);
      }
      __syncwarp();
      // column s of (I + A)^-1, four rows at a time (both halves of the warp alike)
#pragma unroll ROLL_I
      for (int t = 0; t < kDcT; t += 4) {
        const float4* A = reinterpret_cast<const float4*>(st + L::AM + t * kDcT);
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = t + i == s ? 1.f : 0.f;
#pragma unroll ROLL_I
        for (int j = 0; j < t; j += 4) {
          float y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = st[L::TM + (j + i) * kDcT + s];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 w = A[i * 4 + (j >> 2)];
            x[i] = fmaf(-w.w, y[3], fmaf(-w.z, y[2], fmaf(-w.y, y[1], fmaf(-w.x, y[0], x[i]))));
          }
        }
        const float4 w1 = A[4 + (t >> 2)], w2 = A[8 + (t >> 2)], w3 = A[12 + (t >> 2)];
        x[1] = fmaf(-w1.x, x[0], x[1]);
        x[2] = fmaf(-w2.y, x[1], fmaf(-w2.x, x[0], x[2]));
        x[3] = fmaf(-w3.z, x[2], fmaf(-w3.y, x[1], fmaf(-w3.x, x[0], x[3])));
#pragma unroll
        for (int i = 0; i < 4; ++i) st[L::TM + (t + i) * kDcT + s] = x[i];
      }
      mbar_arrive(full + pw);
    }
    asm volatile("bar.arrive 2, %0;" ::"n"(kDcThreads) : "memory");
    return;
  }
  const int pc = (tid & 127) % COLS, pt0 = (tid & 127) / COLS * NTK;  // triangle and read-out: column pc, tokens pt0 .. pt0 + NTK - 1
  // sum over s <= t of m[t][s] x[s] for this thread's tokens, w: their rows of m
  auto rows_of = [&](const float* m, float4 (&w)[NTK][kDcT / 4]) {
#pragma unroll
    for (int i = 0; i < NTK; ++i)
#pragma unroll
      for (int j = 0; j < kDcT / 4; ++j) w[i][j] = *reinterpret_cast<const float4*>(m + (pt0 + i) * kDcT + 4 * j);
  };
  auto lower = [&](const float4 (&w)[NTK][kDcT / 4], const float* x, float (&acc)[NTK]) {
    float4 v[kDcT / 4];
#pragma unroll
    for (int j = 0; j < kDcT / 4; ++j) v[j] = *reinterpret_cast<const float4*>(x + pc * L::WLD + 4 * j);
#pragma unroll
    for (int i = 0; i < NTK; ++i) {
      const int t = pt0 + i;
      float a1 = 0.f;  // two chains
#pragma unroll
      for (int j = 0; j < kDcT / 4; ++j) {
        acc[i] = fmaf(w[i][j].x, 4 * j <= t ? v[j].x : 0.f, acc[i]);
        a1 = fmaf(w[i][j].y, 4 * j + 1 <= t ? v[j].y : 0.f, a1);
        acc[i] = fmaf(w[i][j].z, 4 * j + 2 <= t ? v[j].z : 0.f, acc[i]);
        a1 = fmaf(w[i][j].w, 4 * j + 3 <= t ? v[j].w : 0.f, a1);
      }
      acc[i] += a1;
    }
  };
  // Named barriers: 1 the state warps, 2 the end, 4 / 5 u and S0^T q of an even / odd chunk are there, 6 / 7 they have been read
  if (warp >= 4) {
    // ---- read-out
    int slot = 0;
    uint32_t ph = 0;
    for (int b = 0; b < n_chunks; ++b) {
      const float* st = sm + slot * L::STAGE;
      mbar_wait_bounded(full + slot, ph, dead);
      __syncwarp();
      if (b & 1) asm volatile("bar.sync 5, 256;" ::: "memory");
      else asm volatile("bar.sync 4, 256;" ::: "memory");
      float o[NTK];
      const float* pq = sm + L::PQ + (b & 1) * 4 * kDcT * L::PLD + pc;
#pragma unroll
      for (int i = 0; i < NTK; ++i) {
        const int t = pt0 + i;
        o[i] = st[L::CQ + t] * ((pq[t * L::PLD] + pq[(kDcT + t) * L::PLD]) + (pq[(2 * kDcT + t) * L::PLD] + pq[(3 * kDcT + t) * L::PLD]));
      }
      float4 w[NTK][kDcT / 4];
      rows_of(st + L::BM, w);
      lower(w, sm + L::U + (b & 1) * COLS * L::WLD, o);
      if (b & 1) asm volatile("bar.arrive 7, 256;" ::: "memory");
      else asm volatile("bar.arrive 6, 256;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + slot);
#pragma unroll
      for (int i = 0; i < NTK; ++i)
        if (b * kDcT + pt0 + i < n && a.col0 + pc < a.vdim) store(b * kDcT + pt0 + i, pc, o[i]);
      if (++slot == kDcPrep) {
        slot = 0;
        ph ^= 1u;
      }
    }
    asm volatile("bar.arrive 2, %0;" ::"n"(kDcThreads) : "memory");
    return;
  }
  // ---- state and products
  const int g = lane >> 2, tq = lane & 3, row0 = warp * RW;
  float S[MT][RB][4];  // [..][e]: column 16 mt + g + 8 (e >> 1), row row0 + 8 j + 2 tq + (e & 1)
  auto each_state = [&](auto body) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < RB; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = a.col0 + mt * 16 + g + (e >> 1) * 8;
          body(S[mt][j][e], a.state + (size_t)(row0 + j * 8 + 2 * tq + (e & 1)) * a.vdim + col, col < a.vdim);
        }
  };
  each_state([](float& x, const float* p, bool on) { x = on ? *p : 0.f; });
  auto bar = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
  bf16* ub = reinterpret_cast<bf16*>(sm + L::UB);
  int slot = 0;
  uint32_t ph = 0;
  bool ready = false;  // the stage has been seen full
  for (int b = 0; b < n_chunks; ++b) {
    const float* st = sm + slot * L::STAGE;
    const bf16* raw = reinterpret_cast<const bf16*>(st + L::RAW);
    // the state's parts as B operand: k step ks, columns 8 nt ..
    uint32_t sp[KS][2 * MT][2][3];
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int nt = 0; nt < 2 * MT; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i) dc_split(S[nt >> 1][2 * ks + i][(nt & 1) * 2], S[nt >> 1][2 * ks + i][(nt & 1) * 2 + 1], sp[ks][nt][i]);
    if (!ready) mbar_wait_bounded(full + slot, ph, dead);
    __syncwarp();
    // S0^T x over this warp's rows, x = k (0) or q (1)
    auto products = [&](int x, float (&p)[2 * MT][3][4]) {
#pragma unroll
      for (int nt = 0; nt < 2 * MT; ++nt)
#pragma unroll
        for (int part = 0; part < 3; ++part) p[nt][part][0] = p[nt][part][1] = p[nt][part][2] = p[nt][part][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t f[4];
        ldsm_x4(f, raw + (x * kDcT + fr) * LDR + row0 + ks * 16 + fc);
#pragma unroll
        for (int part = 0; part < 3; ++part)
#pragma unroll
          for (int nt = 0; nt < 2 * MT; ++nt) mma_bf16_16816(p[nt][part], f, sp[ks][nt][0][part], sp[ks][nt][1][part]);
      }
    };
    auto put = [&](float* to, const float (&p)[2 * MT][3][4]) {
      to += (warp * kDcT + g) * L::PLD + 2 * tq;
#pragma unroll
      for (int nt = 0; nt < 2 * MT; ++nt) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = p[nt][0][e] + (p[nt][1][e] + p[nt][2][e]);
        *reinterpret_cast<float2*>(to + nt * 8) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(to + 8 * L::PLD + nt * 8) = make_float2(v[2], v[3]);
      }
    };
    float p[2 * MT][3][4];
    products(0, p);
    put(sm + L::PK, p);
    float ck[NTK], vb[NTK], cs[NTK];  // on their way before the barrier
#pragma unroll
    for (int i = 0; i < NTK; ++i) {
      ck[i] = st[L::CK + pt0 + i];
      cs[i] = st[L::CS + pt0 + i];
      vb[i] = st[L::VB + (pt0 + i) * COLS + pc];
    }
    const float gc = st[L::GC];
    bar();
    const float* pk = sm + L::PK + pc;
#pragma unroll
    for (int i = 0; i < NTK; ++i) {
      const int t = pt0 + i;
      const float x = (pk[t * L::PLD] + pk[(kDcT + t) * L::PLD]) + (pk[(2 * kDcT + t) * L::PLD] + pk[(3 * kDcT + t) * L::PLD]);
      sm[L::W + pc * L::WLD + t] = fmaf(-ck[i], x, vb[i]);
    }
    products(1, p);  // under the barrier and the triangle
    bar();
    float4 tw[NTK][kDcT / 4];
    rows_of(st + L::TM, tw);  // (asked for before the barrier they cost registers and 4 %)
    float u[NTK];
#pragma unroll
    for (int i = 0; i < NTK; ++i) u[i] = 0.f;
    lower(tw, sm + L::W, u);
    if (b >= 2) {  // the read-out warps are done with this buffer's last contents
      if (b & 1) asm volatile("bar.sync 7, 256;" ::: "memory");
      else asm volatile("bar.sync 6, 256;" ::: "memory");
    }
#pragma unroll
    for (int i = 0; i < NTK; i += 2) {
      *reinterpret_cast<float2*>(sm + L::U + ((b & 1) * COLS + pc) * L::WLD + pt0 + i) = make_float2(u[i], u[i + 1]);
      uint32_t q[3];
      dc_split(u[i] * cs[i], u[i + 1] * cs[i + 1], q);
#pragma unroll
      for (int part = 0; part < 3; ++part) *reinterpret_cast<uint32_t*>(ub + (part * COLS + pc) * L::UBLD + pt0 + i) = q[part];
    }
    ready = mbar_test_wait(full + (slot + 1 == kDcPrep ? 0 : slot + 1), slot + 1 == kDcPrep ? ph ^ 1u : ph);  // the next stage
    bar();
    put(sm + L::PQ + (b & 1) * 4 * kDcT * L::PLD, p);
    if (b & 1) asm volatile("bar.arrive 5, 256;" ::: "memory");
    else asm volatile("bar.arrive 4, 256;" ::: "memory");
    // ---- state update: S^T = c S^T + U^T K
    uint32_t fu[MT][3][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int part = 0; part < 3; ++part) ldsm_x4(fu[mt][part], ub + (part * COLS + mt * 16 + fr) * L::UBLD + fc);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t fk[4];
      ldsm_x4_trans(fk, raw + fr * LDR + row0 + ks * 16 + fc);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float add[4] = {};
#pragma unroll
          for (int part = 2; part >= 0; --part) mma_bf16_16816(add, fu[mt][part], fk[2 * i], fk[2 * i + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[mt][2 * ks + i][e] = fmaf(S[mt][2 * ks + i][e], gc, add[e]);
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + slot);  // this warp has read all of the stage
    if (++slot == kDcPrep) {
      slot = 0;
      ph ^= 1u;
    }
  }
  each_state([](float& x, float* p, bool on) {
    if (on) *p = x;
  });
  asm volatile("bar.sync 2, %0;" ::"n"(kDcThreads) : "memory");  // every role is through with its waits
  if (tid == 0) count_run_out(dead, a.err);
}

}  // namespace pk
