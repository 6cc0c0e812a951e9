// One-launch encoder for calls between the decode-time append and the very long prompt (included by encode.cu): exact
// threshold, nearest codewords and either packed rows or the dense fake-quantised tensor, in ONE kernel.
//
// As separate passes such a call was a dozen launches (samples, selects, histograms, flags, fix-ups), each of a few
// microseconds, and its main pass copied 60-150 KB of tables into shared memory per 128 tokens.  Here a head's tokens are
// split over a few CTAs that stay resident (one per SM, cooperative launch): the tables are fetched by bulk copies while
// the three radix-select levels run -- each CTA histograms its norms, the CTAs of the head meet at a counter in global
// memory (bounded wait), everyone scans the head's histogram -- and the main pass then knows the exact threshold, so flags
// and radius codes are final as they are written; the waits for the others are filled with the first tokens.  Bound: the issue
// slots of the search, then what happens once: 57 k clocks of a 4096-token call of 8 heads (fake-quant, s24) are 27 k of search, 7 k
// until the norms are there, three levels of about 1500 for the histogram, 1800 for its sum, 1400 to see the others' and 1700 to
// scan.  K and V: 75.0 -> 69.8 us, 63.8 with the shorter search.
constexpr int kFusedEarly = 3;                // rounds of tokens encoded between the levels, see below
struct FusedArgs {
  // (what a CTA needs first lies together: a line of the parameters that is not in the constant cache costs some 500 clocks)
  EncGeom g;                  // the call's own geometry: n = 32 chunks per token, or 16 (two tokens per warp)
  const uint16_t* x;
  const uint32_t* gate;       // return unless this word is set (nullptr: run)
  int cph, per;               // CTAs per head, warp tokens per CTA
  uint32_t t2_mul; int t2_sh; // w / T2 = umulhi(w, t2_mul) >> t2_sh for w < 2^31, T2 the warp tokens of a sequence (t2_mul 0: T2 = 1)
  const unsigned char* lut;
  const float* qs;
  const float* joint;
  float C, quantile;          // C <= 0: no outliers
  const float* med_in;        // medians given by the caller
  float* med_out;
  uint32_t* hist;             // [H][3][2][kHistBins], zero
  uint32_t* bars;             // [H] arrivals, zero
  uint32_t* status;
  uint16_t* out;              // (B, H, T, 4 n) contiguous, element type of x (DENSE = true)
  uint32_t* n_flagged;        // DENSE: + the call's flagged chunks (optional)
  hqmq_packed dst;            // packed rows (DENSE = false)
  int t_start;
  int rcp_rn;                 // directions are normalised with the rounded reciprocal (as the generic passes do)
  int early;                  // rounds of tokens that may be written ahead of the threshold: kFusedEarly, 0 where out overlaps x
};
struct FusedPair { FusedArgs t[2]; };            // blockIdx.y: the tensor (K and V of a layer in one launch, or one tensor)
constexpr uint32_t kFusedPolls = 1u << 20;       // about a second

__device__ __forceinline__ void fused_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Shared memory: secondaries, two histograms, row scratch, joint table, look-up table (rows, cells, candidates, products).
__host__ __device__ inline size_t fused_smem_bytes(int S, size_t lut_foot) {
  return (size_t)S * 16 + 2 * kHistBins * 4 + (size_t)kEnc32Warps * kMaxRowWords * 4 + (size_t)24 * S * 16 + lut_foot + 64;
}

// IB, RB: field widths of the layouts in common use, or 0: any other, from the geometry.
template <int DT, int IB, int RB, bool DENSE>
__global__ void __launch_bounds__(kEnc32Threads, 1) encode_fused_kernel(const FusedPair pr, const Maps24 maps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_warp[2][32], s_sel[4], s_flagged, s_gave_up;
  const FusedArgs& a = pr.t[DENSE ? 0 : blockIdx.y];        // (fake-quant calls have one tensor)
  if (a.gate && *a.gate == 0u) return;
  const EncGeom& g = a.g;
  const int ib = IB ? IB : g.ib, CB = IB ? IB + RB : g.ib + g.rbits;
  const float qmaxf = (float)(IB ? (1 << RB) - 1 : g.qmax);
  const int S = g.S, h = blockIdx.x / a.cph, part = blockIdx.x - h * a.cph;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4* qs = reinterpret_cast<float4*>(smem_raw);
  uint32_t* sh = reinterpret_cast<uint32_t*>(qs + S);                      // [2][kHistBins]
  uint32_t* rows = sh + 2 * kHistBins;                                       // [warps][kMaxRowWords]
  float4* sjoint = reinterpret_cast<float4*>(rows + kEnc32Warps * kMaxRowWords);
  unsigned char* slut = reinterpret_cast<unsigned char*>(sjoint + 24 * S);

  // ---- this CTA's tokens: warp token w = (b, i), i a token or (16 chunks) a pair of tokens -----------------------------
  const bool pair = (IB == 0 || IB + RB == 16) && g.n == 16;      // (pairs have fields of 16 bits)
  const int T2 = pair ? (g.T_new + 1) >> 1 : g.T_new, W = g.B * T2;
  const int w0 = part * a.per, w1 = min(W, w0 + a.per);
  const int sub = pair ? lane >> 4 : 0, c = pair ? lane & 15 : lane;
  // A place in this sequence of tokens, advanced by a round of the CTA's warps: index in the sequence, chunk in x, output row (of
  // the token of this lane; pairs: each half-warp its own).  (Located by division for every token, a fifth of the instructions.)
  struct Place { int i; const uint16_t* x; int64_t row; };
  const int rpt = pair ? 2 : 1;
  const int64_t x_step = (int64_t)rpt * kEnc32Warps * g.xs_t, x_wrap = g.xs_b - (int64_t)rpt * T2 * g.xs_t;
  const int64_t r_seq = DENSE ? g.T_new : a.dst.T_cap, r_wrap = (int64_t)g.H * r_seq - (int64_t)rpt * T2;
  auto sequences = [&](int w) { return a.t2_mul ? (int)(__umulhi((uint32_t)w, a.t2_mul) >> a.t2_sh) : w; };      // w / T2
  auto place_of = [&](int w) {
    const int b = sequences(w), i = w - b * T2, t = rpt * i + sub;
    return Place{i, a.x + h * g.xs_h + 4 * c + b * g.xs_b + (int64_t)t * g.xs_t, ((int64_t)b * g.H + h) * r_seq + (DENSE ? 0 : a.t_start) + t};
  };
  auto advance = [&](Place& at) {
    at.i += kEnc32Warps; at.x += x_step; at.row += rpt * kEnc32Warps;
    if (at.i >= T2) {
      const int n_seq = sequences(at.i);
      at.i -= n_seq * T2; at.x += n_seq * x_wrap; at.row += n_seq * r_wrap;
    }
  };
  auto is_live = [&](const Place& at) { return !pair || 2 * at.i + sub < g.T_new; };
  auto fetch = [&](const Place& at) { return is_live(at) ? *reinterpret_cast<const uint2*>(at.x) : make_uint2(0u, 0u); };
  auto norm_of = [&](const uint2& raw) {
    float v[4] = {bits16_to_float(raw.x & 0xffff, DT), bits16_to_float(raw.x >> 16, DT), bits16_to_float(raw.y & 0xffff, DT),
                  bits16_to_float(raw.y >> 16, DT)};
    return chunk_norm(v);
  };

  // The norms of a warp's first tokens stay in registers for all three levels of the threshold's search (each level used to read
  // them again: 4.6 us of load latency and norm arithmetic a level).  Eight tokens a warp are 4096 tokens of 8 heads; what is beyond
  // is read again, which the call's time does not show.  They are on their way before anything else.
  constexpr int kKeep = 8;
  uint32_t keys[kKeep];                        // bits of the norms; 0xffffffff, which no prefix equals: no token
  const bool select = a.C > 0.f && !a.med_in;
  uint2 first[kKeep];
  if (select) {
    Place at = place_of(min(w0 + warp, W - 1));
#pragma unroll
    for (int u = 0; u < kKeep; ++u) {
      const bool mine = w0 + warp + u * kEnc32Warps < w1;
      first[u] = mine ? fetch(at) : make_uint2(0u, 0u);
      keys[u] = mine && is_live(at) ? 0u : 0xffffffffu;
      if (mine) advance(at);
    }
  }

  // ---- tables on their way ------------------------------------------------------------------------------------------
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_bar);
  const uint32_t* gh = reinterpret_cast<const uint32_t*>(a.lut);
  const unsigned char* head = a.lut + kLutOffHeads + (size_t)h * kLutHeadBytes;
  const int n = (int)gh[0], n_cells = (int)gh[1];
  const uint32_t total = reinterpret_cast<const uint32_t*>(head)[0];
  const uint32_t b_rows = (uint32_t)n * n * 4, b_cells = ((uint32_t)n_cells * 2 + 15) & ~15u, b_cands = (total * 2 + 15) & ~15u;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(slut), bj = (uint32_t)(24 * S * 16), bq = (uint32_t)S * 16u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bj + bq + b_rows + b_cells + b_cands + (uint32_t)sizeof(Mul24)) : "memory");
    fused_bulk((uint32_t)__cvta_generic_to_shared(sjoint), a.joint + (int64_t)h * 24 * S * 4, bj, bar);
    fused_bulk((uint32_t)__cvta_generic_to_shared(qs), a.qs + (int64_t)h * S * 4, bq, bar);
    fused_bulk(d, a.lut + kLutOffRows, b_rows, bar);
    fused_bulk(d + b_rows, head + 16, b_cells, bar);
    if (b_cands) fused_bulk(d + b_rows + b_cells, head + 16 + (size_t)kLutCellCap * 2, b_cands, bar);
    // (DENSE decodes with the joint table: its indices, then)
    fused_bulk(d + b_rows + b_cells + b_cands, a.lut + kLutOffHeads + (size_t)g.H * kLutHeadBytes + (DENSE ? sizeof(Mul24) : 0), (uint32_t)sizeof(Mul24), bar);
    s_flagged = s_gave_up = 0u;
  }
  LutView L;
  L.rows = reinterpret_cast<const uint32_t*>(slut); L.cells = reinterpret_cast<const uint16_t*>(slut + b_rows);
  L.cands = reinterpret_cast<const uint16_t*>(slut + b_rows + b_cells);
  L.nm = reinterpret_cast<const uint16_t*>(slut + b_rows + b_cells + b_cands);
  lut_set(L, n, S, DENSE);

  // The tables have arrived (all threads; bounded).  A CTA without tables goes on for the others' sake: it counts and meets them,
  // and gives its tokens up at the end.
  auto tables = [&] {
    __syncthreads();                           // (the barrier that is waited for has been initialised)
    uint32_t ok = 0u, tries = 0u;
    while (!ok && ++tries < (1u << 24))
      asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar) : "memory");
    return !__syncthreads_or(!ok);
  };

  // ---- one token: radius codes, nearest codewords, row or dense values ---------------------------------------------------------
  uint32_t* myrow = rows + warp * kMaxRowWords;
  uint32_t n_fl = 0u;
  float thr = INFINITY;
  auto encode_token = [&](const uint2& raw, bool live, int64_t row) {
    float v[4] = {bits16_to_float(raw.x & 0xffff, DT), bits16_to_float(raw.x >> 16, DT), bits16_to_float(raw.y & 0xffff, DT),
                  bits16_to_float(raw.y >> 16, DT)};
    const float nrm = chunk_norm(v);
    const float radius = fmaxf(nrm, 1e-8f);
    // (radii are positive: their bits order like the values)
    const float rmax = __uint_as_float(pair ? __reduce_max_sync(lane & 16 ? 0xffff0000u : 0xffffu, __float_as_uint(radius))
                                          : __reduce_max_sync(0xffffffffu, __float_as_uint(radius)));
    const float scale = IB ? div_whole<(1 << (IB ? RB : 1)) - 1>(rmax) : __fdiv_rn(rmax, qmaxf);
    // (radius code: see encode_main32_kernel)
    const float quo = radius * rcp_approx(scale);
    float rqf = rintf(quo);
    if (fabsf(quo - rqf) > 0.499f) rqf = rintf(__fdiv_rn(radius, scale));
    rqf = fminf(fmaxf(rqf, 0.f), qmaxf);
    const bool flagged = live && nrm > thr;
    const uint32_t flag_word = __ballot_sync(0xffffffffu, flagged);
    n_fl += __popc(flag_word);
    const float inv_r = a.rcp_rn ? __frcp_rn(radius) : rcp_approx(radius);
    uint32_t ni;                                   // native index (DENSE: index in the joint table)
    const float u0 = v[0] * inv_r, u1 = v[1] * inv_r, u2 = v[2] * inv_r, u3 = v[3] * inv_r;
    if (!search_fold24(sjoint, L, S, u0, u1, u2, u3, ni)) {
      int p = 0, sidx = 0;
      if (fmaxf(fmaxf(fabsf(u0), fabsf(u1)), fmaxf(fabsf(u2), fabsf(u3))) > 0.f) p = search_exhaustive(qs, S, u0, u1, u2, u3, sidx);
      ni = code_of<DENSE>(p, sidx, S, maps);
    }
    if constexpr (DENSE) {
      uint2 o = raw;
      if (!flagged) {
        const float rad = __fmul_rn(rqf, scale);
        const float4 cw = sjoint[ni];
        o.x = float_to_bits16(__fmul_rn(cw.x, rad), DT) | ((uint32_t)float_to_bits16(__fmul_rn(cw.y, rad), DT) << 16);
        o.y = float_to_bits16(__fmul_rn(cw.z, rad), DT) | ((uint32_t)float_to_bits16(__fmul_rn(cw.w, rad), DT) << 16);
      }
      if (live) *reinterpret_cast<uint2*>(a.out + (row * g.n + c) * 4) = o;
    } else {
      const uint32_t f = ni | ((flagged ? 0u : (uint32_t)rqf) << ib);
      if (CB == 16) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, f, 1);
        if (live && !(lane & 1)) reinterpret_cast<uint32_t*>(a.dst.codes + row * a.dst.row_bytes)[c >> 1] = f | (other << 16);
      } else {
        const int RW = CB;                             // words per row of 32 chunks (pairs have 16-bit fields)
        if (lane < RW) myrow[lane] = 0;
        __syncwarp();
        const int bit = lane * CB, wd = bit >> 5, s_ = bit & 31;
        atomicOr(&myrow[wd], f << s_);
        if (s_ + CB > 32) atomicOr(&myrow[wd + 1], f >> (32 - s_));
        __syncwarp();
        if (lane < RW) reinterpret_cast<uint32_t*>(a.dst.codes + row * a.dst.row_bytes)[lane] = myrow[lane];
        __syncwarp();
      }
      if (live && c == 0) {
        store_scale(a.dst, row, rmax);
        if (a.dst.flags) a.dst.flags[row] = pair ? (sub ? flag_word >> 16 : flag_word & 0xffffu) : flag_word;
      }
    }
  };
  // this warp's tokens up to w_end, the next one's chunks on their way
  int w_now = w0 + warp;
  Place now = place_of(min(w_now, W - 1));
  auto encode_tokens = [&](int w_end) {
    uint2 nxt = w_now < w_end ? fetch(now) : make_uint2(0u, 0u);
    while (w_now < w_end) {
      const uint2 raw = nxt;
      const bool live = is_live(now);
      const int64_t row = now.row;
      w_now += kEnc32Warps;
      advance(now);
      if (w_now < w_end) nxt = fetch(now);
      encode_token(raw, live, row);
    }
  };

  // ---- exact threshold: three levels of 11, 11 and 10 bits over the head's norms; the tokens in the waits ----------------------
  // Between a level's arrival and its wait a warp encodes a token as if nothing were flagged (a round of tokens takes 3600 to 4000
  // clocks, the wait would take about 2000); once the threshold is known the flagged chunks of those are put right, 650 clocks a
  // token, and the other tokens are encoded with it.  (All eight kept tokens ahead of the threshold: the last step alone 4400.)
  // Putting right reads x again: a dense tensor that is written over its own x has no token encoded ahead.
  bool usable = true;
  if (select) {
    const QRank qr = quantile_rank((uint64_t)g.B * g.T_new * g.n, a.quantile);
#pragma unroll
    for (int u = 0; u < kKeep; ++u) keys[u] |= __float_as_uint(norm_of(first[u]));
    const int early = min(a.early, (w1 - w0 + kEnc32Warps - 1) / kEnc32Warps);      // rounds of the warps
    uint32_t p0 = 0u, p1 = 0u, k0 = (uint32_t)qr.lo, k1 = (uint32_t)qr.hi;      // prefixes and ranks of the two statistics
#pragma unroll 1
    for (int level = 0; level < 3; ++level) {
      const int hs = level == 0 ? 31 : level == 1 ? 21 : 10, ds = level == 0 ? 21 : level == 1 ? 10 : 0;
      const uint32_t dm = level == 2 ? 0x3ffu : 0x7ffu, q0 = p0 >> hs, q1 = p1 >> hs;
      const bool same = q0 == q1;
      for (int i = threadIdx.x; i < 2 * kHistBins; i += blockDim.x) sh[i] = 0u;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kKeep; ++u) {
        const uint32_t top = keys[u] >> hs, dig = (keys[u] >> ds) & dm;
        if (top == q0) atomicAdd(&sh[dig], 1u);
        else if (top == q1) atomicAdd(&sh[kHistBins + dig], 1u);
      }
      if (w0 + warp + kKeep * kEnc32Warps < w1) {
       Place at = place_of(w0 + warp + kKeep * kEnc32Warps);
       for (int w = w0 + warp + kKeep * kEnc32Warps; w < w1; w += 4 * kEnc32Warps) {
        uint2 raw[4]; bool live[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          live[u] = w + u * kEnc32Warps < w1;
          if (live[u]) { raw[u] = fetch(at); live[u] = is_live(at); advance(at); }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (live[u]) {
            const uint32_t key = __float_as_uint(norm_of(raw[u])), top = key >> hs, dig = (key >> ds) & dm;
            if (top == q0) atomicAdd(&sh[dig], 1u);
            else if (top == q1) atomicAdd(&sh[kHistBins + dig], 1u);
          }
       }
      }
      __syncthreads();
      uint32_t* gl = a.hist + ((int64_t)h * 3 + level) * 2 * kHistBins;
      for (int i = threadIdx.x; i < (same ? 1 : 2) * kHistBins; i += blockDim.x)
        if (sh[i]) atomicAdd(&gl[i], sh[i]);
      // the head's CTAs meet: this one arrives ...
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) atomicAdd(&a.bars[h], 1u);
      if (level == 0) usable = tables();
      const int w_to = min(w1, w0 + ((level + 1) * early + 2) / 3 * kEnc32Warps);
      if (usable) encode_tokens(w_to);
      // ... and waits for the others
      if (threadIdx.x == 0) {
        const uint32_t want = (uint32_t)(a.cph * (level + 1));
        uint32_t polls = 0, seen;
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bars + h) : "memory");
        } while (seen < want && ++polls < kFusedPolls);
        if (seen < want) s_gave_up = 1u;
      }
      __syncthreads();
      // scan: two bins per thread, once for both statistics while they share a prefix; only the warp that holds a rank looks into
      // its bins (every thread's place by two scans of 32: 2100 clocks a level)
      for (int q = 0; q < (same ? 1 : 2); ++q) {
        const uint2 cnt = __ldcg(reinterpret_cast<const uint2*>(gl + q * kHistBins) + threadIdx.x);
        const uint32_t mine = cnt.x + cnt.y, sum = __reduce_add_sync(0xffffffffu, mine);
        if (lane == 0) s_warp[q][warp] = sum;
        __syncthreads();
        uint32_t ws = s_warp[q][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, ws, o); if (lane >= o) ws += y; }
        const uint32_t w_end = __shfl_sync(0xffffffffu, ws, warp), w_beg = w_end - sum;
        auto find = [&](uint32_t rank, int slot) {
          if (rank < w_beg || rank >= w_end) return;
          uint32_t incl = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
          const uint32_t before = w_beg + incl - mine;
          if (rank >= before && rank < before + mine) {
            const bool hi = rank >= before + cnt.x;
            s_sel[2 * slot] = (uint32_t)(2 * threadIdx.x + (hi ? 1 : 0));
            s_sel[2 * slot + 1] = rank - before - (hi ? cnt.x : 0u);
          }
        };
        if (q == 0) find(k0, 0);
        if (same || q == 1) find(k1, 1);
      }
      __syncthreads();
      p0 |= s_sel[0] << ds; k0 = s_sel[1]; p1 |= s_sel[2] << ds; k1 = s_sel[3];
      __syncthreads();
    }
    const float va = __uint_as_float(p0), vb = __uint_as_float(p1);
    const float med = qr.hi == qr.lo ? va : quantile_lerp(va, vb, qr.w);
    thr = __fmul_rn(med, a.C);
    if (part == 0 && threadIdx.x == 0 && a.med_out) a.med_out[h] = med;
    // the flagged chunks of the tokens encoded ahead
    if (usable && !s_gave_up && early) {
      // (what is read first, for all of them, then what is written: one by one the eight took 4000 clocks)
      uint2 was[DENSE ? kFusedEarly : 1];
      uint16_t code[DENSE ? 1 : kFusedEarly];
      Place at = place_of(min(w0 + warp, W - 1));
      const Place at0 = at;
      if constexpr (!DENSE) __syncwarp();        // (the rows were stored by other lanes)
#pragma unroll
      for (int u = 0; u < kFusedEarly; ++u) {
        if (keys[u] != 0xffffffffu && __uint_as_float(keys[u]) > thr) {
          if constexpr (DENSE) was[u] = *reinterpret_cast<const uint2*>(at.x);
          else if (CB == 16) code[u] = reinterpret_cast<const uint16_t*>(a.dst.codes + at.row * a.dst.row_bytes)[c];
        }
        advance(at);
      }
      at = at0;
#pragma unroll
      for (int u = 0; u < kFusedEarly; ++u) {
        const bool flagged = keys[u] != 0xffffffffu && __uint_as_float(keys[u]) > thr;
        const uint32_t word = __ballot_sync(0xffffffffu, flagged);
        n_fl += __popc(word);
        if constexpr (DENSE) {
          if (flagged) *reinterpret_cast<uint2*>(a.out + (at.row * g.n + c) * 4) = was[u];
        } else if (word) {
          uint32_t* rowp = reinterpret_cast<uint32_t*>(a.dst.codes + at.row * a.dst.row_bytes);
          if (flagged) {
            if (CB == 16) reinterpret_cast<uint16_t*>(rowp)[c] = (uint16_t)(code[u] & ((1u << ib) - 1u));
            else clear_radius(rowp, c, ib, CB - ib);
          }
          if (is_live(at) && c == 0 && a.dst.flags) a.dst.flags[at.row] = pair ? (sub ? word >> 16 : word & 0xffffu) : word;
        }
        advance(at);
      }
    }
  } else if (a.C > 0.f) {
    const float med = a.med_in[h];
    thr = __fmul_rn(med, a.C);
    if (part == 0 && threadIdx.x == 0 && a.med_out) a.med_out[h] = med;
  }
  if (!select) usable = tables();
  __syncthreads();
  if (usable && !s_gave_up) {
    encode_tokens(w1);
  } else {
    // a bounded wait ran out: what this CTA's tokens decode to is NaN (rows of index 0, nothing flagged), and the status says so
    if (threadIdx.x == 0) {
      atomicOr(a.status, 2u);
      if (part == 0 && a.med_out) a.med_out[h] = NAN;
    }
    Place at = place_of(min(w0 + warp, W - 1));
    for (int w = w0 + warp; w < w1; w += kEnc32Warps, advance(at)) {
      if (!is_live(at)) continue;
      if constexpr (DENSE) {
        *reinterpret_cast<uint2*>(a.out + (at.row * g.n + c) * 4) = make_uint2(0x7fff7fffu, 0x7fff7fffu);
      } else {
        for (int i = c; i < a.dst.row_bytes >> 2; i += g.n) reinterpret_cast<uint32_t*>(a.dst.codes + at.row * a.dst.row_bytes)[i] = 0u;
        if (c == 0) {
          store_scale(a.dst, at.row, NAN);
          if (a.dst.flags) a.dst.flags[at.row] = 0u;
        }
      }
    }
    return;
  }
  if (DENSE && a.n_flagged && a.C > 0.f) {
    if (lane == 0 && n_fl) atomicAdd(&s_flagged, n_fl);
    __syncthreads();
    if (threadIdx.x == 0 && s_flagged) atomicAdd(a.n_flagged, s_flagged);
  }
}
