// Body of a CTA that works on 64 rows of one query head (gqa_attention.cu): rows t0 .. t0 + 63 as far as they lie below GQA_T_END, share GQA_SPLIT of GQA_SPLITS of
// the keys of their requests; several shares leave their states at part_o / part_ml [head][GQA_PART_LD][T].  Included where the kernel of whole steps and
// the one of few rows need it: as a function that both call, the first was 3 to 5 % slower (registers).  With GQA_CLUSTER the shares are the CTAs of a cluster,
// and their states meet over distributed shared memory.  am_smem: two stages of [keys][LDK] K and [keys][LDV] V.  The macros end with the file.
#ifndef GQA_CLUSTER
#define GQA_CLUSTER 0
#endif
  constexpr int LDK = DQ + 8, LDV = DV + 8;
  bf16* const Ks0 = reinterpret_cast<bf16*>(am_smem);
  bf16* const Vs0 = Ks0 + 2 * kAmKeys * LDK;
  __shared__ int s_req[kAmRows], s_pos[kAmRows];
  __shared__ long long s_slot[2][kAmKeys];  // per stage: element offset of every key row's cache slot (-1: not to be read)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  if (tid < kAmRows) {
    const int t = t0 + tid;
    s_req[tid] = t < GQA_T_END ? req[t] : -1;
    s_pos[tid] = t < GQA_T_END ? pos[t] : -1;
  }
  __syncthreads();
  const int tok = G * (DQ + DV);
  // this warp's rows: r0 = warp * 16 + gq and r0 + 8
  const int ra = warp * 16 + gq, rb = ra + 8;
  const int req_a = s_req[ra], req_b = s_req[rb], pos_a = s_pos[ra], pos_b = s_pos[rb];
  const int lo_a = pos_a >= 0 ? first_visible(pos_a, chunk, x.window) : 0, lo_b = pos_b >= 0 ? first_visible(pos_b, chunk, x.window) : 0;
  // The tensor-core kernel keeps scores in units of log2 (every exponential is one ex2), and shapes a raw score q.k with
  //   cap * tanh(z) = cap - 2 cap / (e^(2z) + 1),  z = q.k * scale / cap      (fast exponential and reciprocal: absolute error of a few
  //   1e-7 of the cap, far below the bf16 rounding of P)
  const bool capped = x.softcap > 0.f;
  const float slope2 = head_slope(x.slope_log2, h, H) * kLog2e, cap2 = x.softcap * kLog2e;
  const float c1 = capped ? 2.f * scale / x.softcap * kLog2e : scale * kLog2e;  // raw score -> ex2 argument of e^(2z) / -> plain scaled score
  const int split = GQA_SPLIT, nsplit = GQA_SPLITS;  // few rows: every request's 64-key blocks are dealt out to nsplit CTAs
  // Q fragments (A operand, row-major 16 x DQ)
  uint32_t qa[DQ / 16][4];
#pragma unroll
  for (int kk = 0; kk < DQ / 16; ++kk) {
    const int c = kk * 16 + 2 * tq;
    const bf16* qra = q + ((size_t)(t0 + ra) * H + h) * DQ + c;
    const bf16* qrb = q + ((size_t)(t0 + rb) * H + h) * DQ + c;
    qa[kk][0] = req_a >= 0 ? *reinterpret_cast<const uint32_t*>(qra) : 0u;
    qa[kk][1] = req_b >= 0 ? *reinterpret_cast<const uint32_t*>(qrb) : 0u;
    qa[kk][2] = req_a >= 0 ? *reinterpret_cast<const uint32_t*>(qra + 8) : 0u;
    qa[kk][3] = req_b >= 0 ? *reinterpret_cast<const uint32_t*>(qrb + 8) : 0u;
  }
  float oa[DV / 8][4] = {};
  float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
  // requests of the tile are contiguous runs: walk them one after the other
  int r_first = 0;
  while (r_first < kAmRows && s_req[r_first] >= 0) {
    const int rq = s_req[r_first];
    int r_last = r_first;
    while (r_last + 1 < kAmRows && s_req[r_last + 1] == rq) ++r_last;
    const int p_min = s_pos[r_first], p_max = s_pos[r_last];
    const int k_lo = first_visible(p_min, chunk, x.window);
    const int* pg = pages + page_off[rq];
    // stage `buf` <- keys k0 .. k0 + 63 of this request (cp.async; rows outside [k_lo, p_max] and not among the kept first are zero-filled)
    auto load = [&](int k0, int buf) {
      bf16* Kd = Ks0 + buf * kAmKeys * LDK;
      bf16* Vd = Vs0 + buf * kAmKeys * LDV;
      if (tid < kAmKeys) {  // one page-table read per key row, not one per 16-byte piece
        const int j = k0 + tid;
        s_slot[buf][tid] = (j <= p_max && (j >= k_lo || j < x.keep_first)) ? (long long)pg[j / page_size] * page_stride + (long long)(j % page_size) * tok : -1;
      }
      __syncthreads();
#pragma unroll 4
      for (int c = tid; c < kAmKeys * (DQ / 8); c += 128) {
        const int r = c / (DQ / 8), cc = (c % (DQ / 8)) * 8;
        const long long at = s_slot[buf][r];
        if (at >= 0) cp_async16(&Kd[r * LDK + cc], cache + at + g * DQ + cc);
        else *reinterpret_cast<uint4*>(&Kd[r * LDK + cc]) = make_uint4(0, 0, 0, 0);
      }
#pragma unroll 4
      for (int c = tid; c < kAmKeys * (DV / 8); c += 128) {
        const int r = c / (DV / 8), cc = (c % (DV / 8)) * 8;
        const long long at = s_slot[buf][r];
        if (at >= 0) cp_async16(&Vd[r * LDV + cc], cache + at + G * DQ + g * DV + cc);
        else *reinterpret_cast<uint4*>(&Vd[r * LDV + cc]) = make_uint4(0, 0, 0, 0);
      }
      cp_async_commit();
    };
    // blocks to walk: those that hold kept first keys and lie wholly before the window's first block, then the window's blocks
    const int k_start = k_lo - (k_lo % kAmKeys);
    const int n_kept = min((x.keep_first + kAmKeys - 1) / kAmKeys, k_start / kAmKeys);
    const int n_blocks = n_kept + (p_max - k_start) / kAmKeys + 1, per_split = (n_blocks + nsplit - 1) / nsplit;
    const int b_first = split * per_split, b_end = min(n_blocks, b_first + per_split);
    auto block_k0 = [&](int b) { return b < n_kept ? b * kAmKeys : k_start + (b - n_kept) * kAmKeys; };
    __syncthreads();  // the previous request's readers are done with both stages
    if (b_first < b_end) load(block_k0(b_first), 0);
    for (int b = b_first, it = 0; b < b_end; ++b, ++it) {
      const int buf = it & 1, k0 = block_k0(b);
      cp_async_wait_all();
      __syncthreads();  // this block has landed, and nobody reads the other stage any more
      if (b + 1 < b_end) load(block_k0(b + 1), buf ^ 1);  // overlaps the products below
      const bf16* Ks = Ks0 + buf * kAmKeys * LDK;
      const bf16* Vs = Vs0 + buf * kAmKeys * LDV;
      const bool on_a = req_a == rq, on_b = req_b == rq;
      if (!__any_sync(0xffffffffu, on_a || on_b)) continue;  // warp-uniform: the tensor-core instructions below need all 32 lanes
      // S = Q K^T: 16 rows x 64 keys per warp
      float s[kAmKeys / 8][4] = {};
#pragma unroll
      for (int kk = 0; kk < DQ / 16; ++kk)
#pragma unroll
        for (int np = 0; np < kAmKeys / 16; ++np) {
          uint32_t b[4];
          ldsm_x4(b, &Ks[(np * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * LDK + kk * 16 + ((lane >> 3) & 1) * 8]);
          mma_bf16_16816(s[np * 2], qa[kk], b[0], b[1]);
          mma_bf16_16816(s[np * 2 + 1], qa[kk], b[2], b[3]);
        }
      // key j = k0 + 2 tq + c of this thread's column c is seen from a row at position p iff 0 <= p - j <= p - first_visible(p)
      const int da = on_a ? pos_a - k0 - 2 * tq : -(1 << 20), db = on_b ? pos_b - k0 - 2 * tq : -(1 << 20);
      const unsigned span_a = on_a ? pos_a - lo_a : 0, span_b = on_b ? pos_b - lo_b : 0;
      const float fa = (float)da, fb = (float)db;
      const int kept = x.keep_first - k0 - 2 * tq;  // column c holds one of the kept first keys iff c < kept
      float mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
      for (int ni = 0; ni < kAmKeys / 8; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = ni * 8 + (e & 1);
          const bool top = e < 2;
          const int dist = (top ? da : db) - c;
          const bool ok = (unsigned)dist <= (top ? span_a : span_b) || (c < kept && dist >= 0);
          float v = s[ni][e] * c1;
          if (capped) v = fmaf(-2.f * cap2, __fdividef(1.f, fast_ex2(fminf(v, 80.f)) + 1.f), cap2);
          v = fmaf(-slope2, (top ? fa : fb) - (float)c, v);
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
      // a row that has seen nothing yet keeps its maximum at -inf; subtracting 0 instead leaves its (all -inf) scores at 2^-inf = 0
      const float sub_a = mn_a == -INFINITY ? 0.f : mn_a, sub_b = mn_b == -INFINITY ? 0.f : mn_b;
      const float c_a = fast_ex2(m_a - sub_a), c_b = fast_ex2(m_b - sub_b);
      float sum_a = 0.f, sum_b = 0.f;
      uint32_t pa[kAmKeys / 16][4];
#pragma unroll
      for (int ni = 0; ni < kAmKeys / 8; ++ni) {
        // P is rounded to bf16 once, for the second product; the row sum adds the rounded values
        const uint32_t pk_a = pack_bf16(fast_ex2(s[ni][0] - sub_a), fast_ex2(s[ni][1] - sub_a));
        const uint32_t pk_b = pack_bf16(fast_ex2(s[ni][2] - sub_b), fast_ex2(s[ni][3] - sub_b));
        sum_a += bf16_lo(pk_a) + bf16_hi(pk_a);
        sum_b += bf16_lo(pk_b) + bf16_hi(pk_b);
        pa[ni >> 1][(ni & 1) * 2] = pk_a;
        pa[ni >> 1][(ni & 1) * 2 + 1] = pk_b;
      }
      sum_a += __shfl_xor_sync(0xffffffffu, sum_a, 1);
      sum_a += __shfl_xor_sync(0xffffffffu, sum_a, 2);
      sum_b += __shfl_xor_sync(0xffffffffu, sum_b, 1);
      sum_b += __shfl_xor_sync(0xffffffffu, sum_b, 2);
      l_a = l_a * c_a + sum_a;
      l_b = l_b * c_b + sum_b;
      m_a = mn_a;
      m_b = mn_b;
#pragma unroll
      for (int ni = 0; ni < DV / 8; ++ni) {
        oa[ni][0] *= c_a;
        oa[ni][1] *= c_a;
        oa[ni][2] *= c_b;
        oa[ni][3] *= c_b;
      }
      // O += P V: V block is [keys][DV] row-major = the B operand's k-major form through ldmatrix.trans
#pragma unroll
      for (int kk = 0; kk < kAmKeys / 16; ++kk)
#pragma unroll
        for (int np = 0; np < DV / 16; ++np) {
          uint32_t b[4];
          ldsm_x4_trans(b, &Vs[(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDV + np * 16 + ((lane >> 4) & 1) * 8]);
          mma_bf16_16816(oa[np * 2], pa[kk], b[0], b[1]);
          mma_bf16_16816(oa[np * 2 + 1], pa[kk], b[2], b[3]);
        }
    }
    r_first = r_last + 1;
  }
#if GQA_CLUSTER
  {
    // this share's state of its 64 rows over the key blocks, then each CTA finishes every nsplit-th part of the rows, a warp per row
    constexpr int LDO = DV + 2;  // [DV] unnormalised output, maximum, sum
    float* st = reinterpret_cast<float*>(Ks0);
    __syncthreads();  // the last block has been read
#pragma unroll
    for (int ni = 0; ni < DV / 8; ++ni) {
      const int c = ni * 8 + 2 * tq;
      *reinterpret_cast<float2*>(st + ra * LDO + c) = make_float2(oa[ni][0], oa[ni][1]);
      *reinterpret_cast<float2*>(st + rb * LDO + c) = make_float2(oa[ni][2], oa[ni][3]);
    }
    if (tq == 0) {
      *reinterpret_cast<float2*>(st + ra * LDO + DV) = make_float2(m_a, l_a);
      *reinterpret_cast<float2*>(st + rb * LDO + DV) = make_float2(m_b, l_b);
    }
    cluster_barrier();
    const float sk = sink ? bf2f(sink[h]) * kLog2e : -INFINITY;
    const uint32_t base = smem_u32(st);
    const int rows = kAmRows / nsplit;
    for (int r = split * rows + warp; r < (split + 1) * rows; r += 4) {
      if (s_req[r] < 0) continue;
      const int t = t0 + r;
      float m = -INFINITY, l = 0.f;
      if (lane < nsplit) gqa_ld_state(base + (uint32_t)(r * LDO + DV) * 4, lane, m, l);
      const float top = fmaxf(warp_max(m), sk), e = m == -INFINITY ? 0.f : exp2f(m - top);
      const float wgt = e / (warp_sum(l * e) + (sink ? exp2f(sk - top) : 0.f));
      float w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = __shfl_sync(0xffffffffu, wgt, i);  // (lanes of no share: zero)
      for (int d = 2 * lane; d < DV; d += 64) {
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= nsplit) break;
          float x0, x1;
          gqa_ld_state(base + (uint32_t)(r * LDO + d) * 4, i, x0, x1);
          o0 = fmaf(x0, w[i], o0);
          o1 = fmaf(x1, w[i], o1);
        }
        if (x.gate) {
          o0 *= out_gate<bf16>(x, t, h, d, DV);
          o1 *= out_gate<bf16>(x, t, h, d + 1, DV);
        }
        *reinterpret_cast<uint32_t*>(out + (size_t)t * x.out_ld + h * DV + d) = pack_bf16(o0, o1);
      }
    }
    cluster_barrier();  // the other CTAs have read this one's shared memory
  }
#else
  if (nsplit > 1) {  // partial state (running maximum, sum, unnormalised output) of this split; gqa_attention_merge_kernel finishes the rows
    const size_t sa = ((size_t)(h * GQA_PART_LD + split) * T + (t0 + ra)), sb = ((size_t)(h * GQA_PART_LD + split) * T + (t0 + rb));
    if (req_a >= 0 && tq == 0) part_ml[sa * 2] = m_a * kLn2, part_ml[sa * 2 + 1] = l_a;  // maxima leave in natural units
    if (req_b >= 0 && tq == 0) part_ml[sb * 2] = m_b * kLn2, part_ml[sb * 2 + 1] = l_b;
#pragma unroll
    for (int ni = 0; ni < DV / 8; ++ni) {
      const int c = ni * 8 + 2 * tq;
      if (req_a >= 0) *reinterpret_cast<float2*>(part_o + sa * DV + c) = make_float2(oa[ni][0], oa[ni][1]);
      if (req_b >= 0) *reinterpret_cast<float2*>(part_o + sb * DV + c) = make_float2(oa[ni][2], oa[ni][3]);
    }
    return;
  }
  const float sk = sink ? bf2f(sink[h]) * kLog2e : -INFINITY;  // the sink joins in the same log2 units
  const float mt_a = fmaxf(m_a, sk), mt_b = fmaxf(m_b, sk);
  const float f_a = m_a == -INFINITY ? 0.f : exp2f(m_a - mt_a), f_b = m_b == -INFINITY ? 0.f : exp2f(m_b - mt_b);
  const float d_a = l_a * f_a + (sink ? exp2f(sk - mt_a) : 0.f), d_b = l_b * f_b + (sink ? exp2f(sk - mt_b) : 0.f);
  float i_a = f_a / d_a, i_b = f_b / d_b;
  if (x.gate && x.gate_per_head) {
    if (req_a >= 0) i_a *= out_gate<bf16>(x, t0 + ra, h, 0, DV);
    if (req_b >= 0) i_b *= out_gate<bf16>(x, t0 + rb, h, 0, DV);
  }
#pragma unroll
  for (int ni = 0; ni < DV / 8; ++ni) {
    const int c = ni * 8 + 2 * tq;
    float g0 = 1.f, g1 = 1.f, g2 = 1.f, g3 = 1.f;
    if (x.gate && !x.gate_per_head) {
      const bf16* ga = static_cast<const bf16*>(x.gate) + (size_t)(t0 + ra) * x.gate_ld + h * DV + c;
      const bf16* gb = static_cast<const bf16*>(x.gate) + (size_t)(t0 + rb) * x.gate_ld + h * DV + c;
      if (req_a >= 0) g0 = 1.f / (1.f + expf(-bf2f(ga[0]))), g1 = 1.f / (1.f + expf(-bf2f(ga[1])));
      if (req_b >= 0) g2 = 1.f / (1.f + expf(-bf2f(gb[0]))), g3 = 1.f / (1.f + expf(-bf2f(gb[1])));
    }
    if (req_a >= 0) *reinterpret_cast<uint32_t*>(out + (size_t)(t0 + ra) * x.out_ld + h * DV + c) = pack_bf16(oa[ni][0] * i_a * g0, oa[ni][1] * i_a * g1);
    if (req_b >= 0) *reinterpret_cast<uint32_t*>(out + (size_t)(t0 + rb) * x.out_ld + h * DV + c) = pack_bf16(oa[ni][2] * i_b * g2, oa[ni][3] * i_b * g3);
  }
#endif
#undef GQA_T_END
#undef GQA_CLUSTER
#undef GQA_SPLIT
#undef GQA_SPLITS
#undef GQA_PART_LD
