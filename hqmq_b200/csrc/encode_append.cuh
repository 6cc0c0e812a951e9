// The decode-time append: ONE token per sequence, K and V of a layer, in one launch (included by encode.cu).
//
// What append_pair_kernel does for up to 32 blocks of tokens, cut down to the latency of its longest chain.  A head's chunks
// (at most 512) are held twice: group A of the CTA takes norms, threshold, flags, payload and offsets, group B searches
// the codewords (four dependent look-ups in L2) at the same time and packs the rows.  Offsets and payload come from
// registers and shared memory instead of being read back; only the token that completes a 16-token block runs the general
// scan and record code.  The heads of a tensor form one cluster where they can, so that the status word is cleared
// without a memset ahead of the launch.  11 us per append (4 sequences, 8 heads of 64) before.
struct AppendArgs { SmallArgs t[2]; Maps24 maps; int clear; };   // clear: the status words are cleared here (one cluster per tensor)
constexpr int kAppendMax = 512;                 // chunks per head

__device__ __forceinline__ void bar_group(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

__global__ void __launch_bounds__(2 * kAppendMax) append_one_kernel(const AppendArgs p) {
  __shared__ uint32_t keys[kAppendMax], fld[kAppendMax], tokmax[kAppendMax], tokfl[kAppendMax];
  __shared__ uint32_t rowbuf[kAppendMax * 2];     // packed rows [B][words]: at most 24 bits a chunk, a word at least
  __shared__ uint32_t shist[256], s_state[4], s_over;
  const SmallArgs& a = p.t[blockIdx.y];
  const EncGeom& g = a.g;
  const hqmq_packed& dst = a.dst;
  const int h = blockIdx.x, n = g.n, N = g.B * n, NP = blockDim.x >> 1, S = g.S;
  const bool grpA = (int)threadIdx.x < NP;
  const int i = grpA ? threadIdx.x : threadIdx.x - NP;           // this thread's chunk
  const bool live = i < N;
  const int b = live ? i / n : 0, c = i - b * n;
  const bool med = a.C > 0.f;
  const int rw = dst.row_bytes >> 2, cb = g.ib + g.rbits;
  for (int w = threadIdx.x; w < g.B * rw; w += blockDim.x) rowbuf[w] = 0u;
  if (grpA) { tokmax[i] = 0u; tokfl[i] = 0u; }
  for (int w = threadIdx.x; w < 256; w += blockDim.x) shist[w] = 0u;
  if (threadIdx.x == 0) { s_state[2] = 0u; s_state[3] = 0xffffffffu; s_over = 0u; }
  // (launched while the predecessor may still run: nothing before this line touches global memory)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  bool use_lut = false;
  LutView L = {};
  if (!grpA) {
    use_lut = a.lut && lut_head_valid(a.lut, h);
    if (use_lut) L = lut_global(a.lut, h, g.H, S, false);
  }
  if (p.clear) {
    if (h == 0 && threadIdx.x == 0) *a.status = 0u;
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // (waited for at the end)
  }
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) load_chunk(a.x, b * g.xs_b + h * g.xs_h + 4 * c, g.x_dtype, v);
  const float nrm = chunk_norm(v), radius = fmaxf(nrm, 1e-8f);
  const bool complete = ((a.t_start + 1) % HQMQ_OUT_BLOCK) == 0;     // this token completes a block: records are due
  const bool quick = a.scan && a.payload && !(complete && dst.ofrag);
  const int nb_cap = dst.T_cap / HQMQ_OUT_BLOCK + 1;
  __syncthreads();

  if (grpA) {
    uint32_t run = 0u, frun = 0u;
    const int64_t bh_tok = (int64_t)i * g.H + h;                     // (thread i < B also looks after sequence i)
    if (i < g.B && quick) {
      run = dst.out_count[bh_tok];
      if (dst.ofrag) frun = dst.ofrag_off[bh_tok * nb_cap + a.blk0];
    }
    const uint32_t key = __float_as_uint(nrm);
    if (live) {
      keys[i] = key;
      atomicMax(&tokmax[b], __float_as_uint(radius));
    }
    bar_group(1, NP);
    float thr = INFINITY;
    if (med) {
      const QRank qr = quantile_rank((uint64_t)N, a.quantile);
      const uint32_t lo = (uint32_t)qr.lo, hi = (uint32_t)qr.hi;
      uint32_t a_bits, b_bits;
      if (N <= 128) {
        // every thread counts the keys below its own: both order statistics name themselves
        uint32_t lt = 0u, le = 0u;
        for (int j = 0; j < N; ++j) { const uint32_t y = keys[j]; lt += y < key; le += y <= key; }
        if (live && lt <= lo && lo < le) s_state[0] = key;
        if (live && lt <= hi && hi < le) s_state[1] = key;
        bar_group(1, NP);
        a_bits = s_state[0]; b_bits = s_state[1];
      } else {
        uint32_t prefix = 0u, rank = lo;
        for (int pass = 0; pass < 4; ++pass) {
          const int shift = 24 - 8 * pass;
          if (live && (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8)))) atomicAdd(&shist[(key >> shift) & 0xffu], 1u);
          bar_group(1, NP);
          // every warp scans the digit counts for itself (eight per lane)
          const int lane = threadIdx.x & 31;
          uint32_t c8[8], mine = 0u;
#pragma unroll
          for (int q = 0; q < 8; ++q) { c8[q] = shist[lane * 8 + q]; mine += c8[q]; }
          uint32_t incl = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
          uint32_t acc = incl - mine;
          const bool own = rank >= acc && rank < incl;
          uint32_t digit = 0u;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (own && digit == 0u) {
              if (acc + c8[q] > rank) digit = (uint32_t)(lane * 8 + q) + 1u;
              else acc += c8[q];
            }
          }
          const int src = __ffs(__ballot_sync(0xffffffffu, own)) - 1;
          digit = __shfl_sync(0xffffffffu, digit, src);
          rank -= __shfl_sync(0xffffffffu, acc, src);
          prefix |= (digit - 1u) << shift;
          bar_group(1, NP);
          for (int w = threadIdx.x; w < 256; w += NP) shist[w] = 0u;
          bar_group(1, NP);
        }
        a_bits = prefix;
        if (live) {
          if (key <= a_bits) atomicAdd(&s_state[2], 1u);
          else atomicMin(&s_state[3], key);
        }
        bar_group(1, NP);
        b_bits = s_state[2] > hi ? a_bits : s_state[3];
      }
      const float va = __uint_as_float(a_bits), vb = __uint_as_float(b_bits);
      const float m = hi == lo ? va : quantile_lerp(va, vb, qr.w);
      thr = __fmul_rn(m, a.C);
      if (threadIdx.x == 0 && a.med_out) a.med_out[h] = m;
    }
    const bool flagged = med && live && nrm > thr;
    if (live) {
      const float rmax = fmaxf(__uint_as_float(tokmax[b]), 1e-8f), qmaxf = (float)g.qmax;
      const float scale = __fdiv_rn(rmax, qmaxf);
      const float rqf = fminf(fmaxf(rintf(__fdiv_rn(radius, scale)), 0.f), qmaxf);
      fld[i] = (flagged ? 0u : (uint32_t)rqf) << g.ib;
      if (flagged) atomicOr(&tokfl[b], 1u << c);
    }
    bar_group(1, NP);
    __threadfence_block();
    asm volatile("bar.arrive 2, %0;" ::"r"(2 * NP) : "memory");       // radius codes are there for group B
    if (i < g.B) {
      const int64_t row = bh_tok * dst.T_cap + a.t_start;
      store_scale(dst, row, fmaxf(__uint_as_float(tokmax[i]), 1e-8f));
      if (dst.flags) dst.flags[row] = tokfl[i];
      if (quick) {
        // offsets of the block (its first token starts it), running totals; records carry on
        const uint32_t total = run + __popc(tokfl[i]);
        uint32_t* off = dst.out_off + bh_tok * nb_cap;
        if (a.t_start % HQMQ_OUT_BLOCK == 0) off[a.blk0] = run;
        off[a.blk0 + 1] = total;
        dst.out_count[bh_tok] = total;
        if (dst.ofrag) dst.ofrag_off[bh_tok * nb_cap + a.blk0 + 1] = frun;
        keys[i] = run;                                                   // (the keys are done with)
        if (total > (uint32_t)dst.out_cap) s_over = 1u;
      }
    }
  } else {
    // ---- group B: nearest codeword --------------------------------------------------------------------------------------
    uint32_t ni = 0u;
    if (live) {
      const float4* joint = reinterpret_cast<const float4*>(a.joint) + (int64_t)h * 24 * S;
      const float4* qs = reinterpret_cast<const float4*>(a.qs) + (int64_t)h * S;
      const float inv_r = __frcp_rn(radius);
      const float u0 = v[0] * inv_r, u1 = v[1] * inv_r, u2 = v[2] * inv_r, u3 = v[3] * inv_r;
      if (!(use_lut && search_fold24(joint, L, S, u0, u1, u2, u3, ni))) {
        int sidx;
        const int q = search_exhaustive(qs, S, u0, u1, u2, u3, sidx);
        ni = code_of<false>(q, sidx, S, p.maps);
      }
    }
    bar_group(2, 2 * NP);
    if (live) {
      const uint32_t f = ni | fld[i];
      const int bit = c * cb, w = bit >> 5, sh = bit & 31;
      atomicOr(&rowbuf[b * rw + w], f << sh);
      if (sh + cb > 32) atomicOr(&rowbuf[b * rw + w + 1], f >> (32 - sh));
    }
    bar_group(3, NP);
    for (int w = i; w < g.B * rw; w += NP) {
      const int bb = w / rw;
      const int64_t row = ((int64_t)bb * g.H + h) * dst.T_cap + a.t_start;
      reinterpret_cast<uint32_t*>(dst.codes + row * dst.row_bytes)[w - bb * rw] = rowbuf[w];
    }
  }
  __syncthreads();
  if (p.clear) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (!a.scan) return;
  if (quick) {
    if (threadIdx.x == 0 && s_over) atomicOr(a.status, 1u);
    // ---- payload: the flagged chunk's own thread has its values and its place ---------------------------------------------
    if (grpA && live && ((tokfl[b] >> c) & 1u)) {
      const uint32_t pos = keys[b] + __popc(tokfl[b] & ((1u << c) - 1u));
      if (pos < (uint32_t)dst.out_cap) {
        const int64_t o = (((int64_t)b * g.H + h) * dst.out_cap + pos) * 4;
        if (dst.out_dtype == HQMQ_F32) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(dst.out_vals) + o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
          uint2 w;
          w.x = float_to_bits16(v[0], dst.out_dtype) | ((uint32_t)float_to_bits16(v[1], dst.out_dtype) << 16);
          w.y = float_to_bits16(v[2], dst.out_dtype) | ((uint32_t)float_to_bits16(v[3], dst.out_dtype) << 16);
          *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(dst.out_vals) + o) = w;
        }
      }
    }
    return;
  }
  // ---- the token completes a block (or only records are kept up): the general scan and side planes -------------------------
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int bb = warp; bb < g.B; bb += blockDim.x >> 5)
    scan_small_warp(dst, bb * g.H + h, a.t_start, 1, a.blk0, a.nblk, a.payload, a.status, lane);
  if (!a.side) return;
  __syncthreads();
  for (int bb = warp; bb < g.B; bb += blockDim.x >> 5)
    side_block(g, a.x, dst, a.t_start, a.blk0, a.nblk, bb * g.H + h, 0, lane);
}
