// Attention of many query positions over one compressed cache (a prompt, or a chunk of one): tensor cores, tcgen05.
//
// The decode kernels make every query position a unit of its own and decode K and V once per unit: right for one
// token, 2048 times the decoding for a 2048-token prompt chunk.  Here the cache is decoded ONCE per call into operand
// tiles, and the attention runs on the tensor cores over those:
//
//   expand   (prefill_expand_kernel) per (b, KV head) and 128-token tile: K and V as fp16 operand images in the 128-byte
//            swizzle that tcgen05.mma reads (tokens down, 64 elements of d across: K-major for Q K^T, MN-major for P V), so
//            that a tile is one contiguous bulk copy later.
//            A value is codeword * (rq * rs / qmax * 2^(10-e)), e the exponent of the largest scale of the (b, head), outliers
//            are x * 2^(10-e): everything lies below 2^10 and keeps its 11 bits down to 2^-24 of the largest token.
//   attend   (prefill_attn_kernel) persistent, one CTA per SM.  A unit is (b, KV head, up to 2 x 128 rows), a row one
//            (query position, head of the group): all heads of a group share the decoded tile.  Two row blocks ("streams")
//            alternate on the tensor cores: while the softmax warps of one stream work on S = Q K^T, the other stream's
//            P V and its next Q K^T run.  Warps 0-3 / 4-7: softmax of stream 0 / 1 (a thread owns a row: S comes out of
//            TMEM, P goes back as fp16 into the same columns, the accumulator is rescaled only when a row's maximum rises by
//            more than 2^8); warps 8 / 10 issue the MMAs of stream 0 / 1; warp 9 streams the tiles in through two-deep (four at
//            d_head 64) rings.
//            The tiles of all units form one flat sequence cut into equal pieces, one per CTA, whatever the mask leaves of
//            each unit; a unit that is cut leaves partials, merged by prefill_merge_kernel.
//
// Bound: per 256 rows x 128 keys, 2048 tensor clocks and as many of the exponential unit; 3110 clocks a tile with the two streams'
// softmax out of step.  Measured and left: part of the exponentials as a polynomial on the FMA pipe (3240 to 4000), P handed over
// after 96 keys instead of 64 (3100), two threads to a row (246 us against 236 for 2048 queries over 8192 keys).  A prompt of a few
// tiles pays for what a unit costs once: queries 3000 to 6000 clocks, output 4000, a first pass through cold code 1000.  Loads and
// stores in one small copy each, masks 32 columns at a time and the streams out of step from the start took the attention of
// 2048 causal tuple queries from 58 to 47 us, of 4 x 500 with heads of 64 from 45 to 33.
#include "attn_prefill.cuh"
#include "attn_ring.cuh"

namespace hqmq {
namespace attn {
namespace {

constexpr int kPfThreads = 384;             // 2 x 4 softmax warps; two MMA warps, a loader warp and an idle one (register shares are per 4 warps)
// registers per thread: the launch gives 384 x 168; the third warpgroup hands its share to the softmax warps (128 values of
// a row each): 256 x 208 + 128 x 80 <= 384 x 168
constexpr int kPfSoftmaxRegs = 208, kPfOtherRegs = 80;
static_assert(256 * kPfSoftmaxRegs + 128 * kPfOtherRegs <= kPfThreads * 168, "register split beyond the launch's share");
constexpr float kPfSlack = 8.f;             // log2 units a row's maximum may rise before its accumulator is rescaled
constexpr uint32_t kPfTmemCols = 512;
constexpr int kPfStaggerPolls = 64;
constexpr int kPfFirst = 64;                     // keys of a tile whose P is handed over first (32: 3800 clocks a tile; 64 and 96: 3110)

__host__ __device__ constexpr int pf_stages(int d) { return d == 128 ? 2 : 4; }
__host__ __device__ constexpr size_t pf_tile_bytes(int d) { return (size_t)d * 256; }
constexpr int kPfOutRow = 80;                // bytes of a row in a warp's output staging area: 64 + padding
__host__ __device__ constexpr size_t pf_smem_bytes(int d) { return (size_t)(2 + 2 * pf_stages(d)) * pf_tile_bytes(d) + 8 * 32 * kPfOutRow + 1024 + 256; }

// ---- work decomposition -------------------------------------------------------------------------------------------
// KV tiles [lo, lo + n) that the rows of unit m see (at least one, so that a fully masked unit still writes its zeros).
__host__ __device__ inline void pf_unit_tiles(const PrefillParams& p, int m, int& lo, int& n) {
  const int pos0 = m * p.streams * p.P;
  int pos1 = pos0 + p.streams * p.P - 1;
  if (pos1 >= p.Tq) pos1 = p.Tq - 1;
  int beg, end, beg1, end1;
  key_range(p.Tkv, p.Tq, p.causal, p.window, pos0, beg, end);
  key_range(p.Tkv, p.Tq, p.causal, p.window, pos1, beg1, end1);
  lo = beg / kPfTok;
  const int hi = (end1 + kPfTok - 1) / kPfTok, last = (p.Tkv - 1) / kPfTok;
  if (lo > last) lo = last;
  n = hi > lo ? hi - lo : 1;
}

struct PfPiece { int bh, m, tile0, n; bool head, tail; };
// The pieces of one CTA.  Cut mode (p.L > 0): its stretch [c * L, (c + 1) * L) of the flat tile sequence, unit by unit.
// Whole mode: units in order of m falling (with a causal mask: of length falling), dealt out to the CTAs to and fro.
struct PfIter {
  int left;                      // tiles left of the piece; whole mode: index of the next unit in the CTA's hand
  int bh, m, off, lo, n;
  __device__ __forceinline__ void init(const PrefillParams& p, int cta) {
    if (p.L == 0) { left = 0; return; }
    const int64_t pos = (int64_t)cta * p.L;
    left = (int)(p.total - pos < p.L ? p.total - pos : p.L);
    bh = (int)(pos / p.Wh);
    m = p.start_m[cta]; off = p.start_off[cta];
    pf_unit_tiles(p, m, lo, n);
  }
  __device__ __forceinline__ bool next(const PrefillParams& p, PfPiece& q) {
    if (p.L == 0) {
      const int G = (int)gridDim.x, c = (int)blockIdx.x;
      const int i = left * G + ((left & 1) ? G - 1 - c : c);
      if (i >= p.units_all) return false;
      ++left;
      const int n_bh = p.units_all / p.units_m, j = i / n_bh;
      q.bh = i - j * n_bh; q.m = p.units_m - 1 - j;
      pf_unit_tiles(p, q.m, q.tile0, q.n);
      q.head = q.tail = true;
      return true;
    }
    if (left <= 0) return false;
    if (off >= n) {
      off = 0;
      if (++m == p.units_m) { m = 0; ++bh; }
      pf_unit_tiles(p, m, lo, n);
    }
    q.bh = bh; q.m = m; q.tile0 = lo + off;
    q.n = n - off < left ? n - off : left;
    q.head = off == 0; q.tail = off + q.n == n;
    left -= q.n; off += q.n;
    return true;
  }
};

// ---- tcgen05 ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Issued inside `if (elect_one())` by a converged warp: the compiler then knows that one lane is active and that descriptors
// and addresses are uniform.  (Measured, 128 x 128 x 16: 64 clocks per MMA -- the tensor cores' own rate -- against 75 to 90
// from a branch on the lane number or with the instruction predicated.)
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0u;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
#define PF_R8(r, o) "=r"((r)[o]), "=r"((r)[o + 1]), "=r"((r)[o + 2]), "=r"((r)[o + 3]), "=r"((r)[o + 4]), "=r"((r)[o + 5]), \
                    "=r"((r)[o + 6]), "=r"((r)[o + 7])
#define PF_I8(r, o) "r"((r)[o]), "r"((r)[o + 1]), "r"((r)[o + 2]), "r"((r)[o + 3]), "r"((r)[o + 4]), "r"((r)[o + 5]), \
                    "r"((r)[o + 6]), "r"((r)[o + 7])
__device__ __forceinline__ void tc_ld32(uint32_t* r, uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : PF_R8(r, 0), PF_R8(r, 8), PF_R8(r, 16), PF_R8(r, 24) : "r"(addr));
}
__device__ __forceinline__ void tc_st32(uint32_t addr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(addr), PF_I8(r, 0), PF_I8(r, 8), PF_I8(r, 16), PF_I8(r, 24) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t addr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), PF_I8(r, 0), PF_I8(r, 8) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// K-major operand in the 128-byte swizzle: rows of 128 bytes, groups of eight rows 1024 bytes apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
// MN-major operand in the same swizzle: k rows of 128 bytes (64 elements across), groups of eight rows 1024 bytes apart, the
// next 64 elements across in a plane of 128 rows of their own.
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(16384 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
// kind::f16, fp16 operands (A K-major; B K-major, or MN-major), fp32 accumulators
__host__ __device__ constexpr uint32_t f16_idesc(int M, int N, bool b_mn = false) {
  return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Two fp32 operations per instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}

// ---- attend ----------------------------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kPfThreads, 1) prefill_attn_kernel(const PrefillParams p) {
  constexpr int NS = pf_stages(D);
  constexpr uint32_t TB = (uint32_t)pf_tile_bytes(D);
  extern __shared__ unsigned char smem_raw[];
  const uint32_t s_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base = smem_raw + (s_base - smem_u32(smem_raw));
  const uint32_t sQ = s_base, sK = sQ + 2 * TB, sV = sK + NS * TB, sO = sV + NS * TB, bars = sO + 8 * 32 * kPfOutRow;
  const uint32_t kfull = bars, kempty = kfull + 8 * NS, vfull = kempty + 8 * NS, vempty = vfull + 8 * NS;
  // per stream: queries written, S of a tile computed, either part of its P written, the unit's last P V done
  const uint32_t qfull = vempty + 8 * NS, sfull = qfull + 16, pfull = sfull + 16, odone = pfull + 32;
  volatile uint32_t* abort_word = reinterpret_cast<volatile uint32_t*>(base + (odone + 16 - s_base));
  volatile uint32_t* progress = abort_word + 2;      // units that stream 0 has half of its first P of (the word between is tcgen05.alloc's)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(kfull + 8 * i, 1); mbar_init(kempty + 8 * i, p.streams); mbar_init(vfull + 8 * i, 1); mbar_init(vempty + 8 * i, p.streams);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(qfull + 8 * s, 4); mbar_init(sfull + 8 * s, 1); mbar_init(odone + 8 * s, 1);
      mbar_init(pfull + 16 * s, 4); mbar_init(pfull + 16 * s + 8, 4);
    }
    *abort_word = 0u;
    *progress = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(odone + 20), "n"(kPfTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // (launched while the expansion still runs: nothing before this line touches what a kernel wrote)
  grid_dep_wait();
  grid_dep_launch();
  constexpr uint32_t tmem = 0u;               // an allocation of all columns starts at column 0
  // (a wait that runs out raises the abort word: every role then stops at its next wait.  No suspend hint: these waits are
  //  links of the per-tile chain, and a hinted wait was seen to wake late.)
  // A wait by parity takes a barrier that is two phases on for one that has not moved, so whoever waits has to have a part in the
  // next phase.  Tile g, unit u of the CTA:
  //   kfull, vfull    (MMA issuers)  the stage is filled again only after the commits of both streams for tile g
  //   kempty, vempty  (loader)       freed again only after the tile that the loader is about to put there
  //   qfull           (MMA issuer)   the next queries need S of the unit's last tile, which it issues after this wait
  //   qfull           (loader)       the first unit's, before K of its second tile
  //   sfull           (softmax)      the next S needs P of this one, or the next unit's queries, of all four warps
  //   pfull           (MMA issuer)   the next P needs the S that it issues after both parts of this one
  //   odone           (softmax)      the next unit's needs all four warps' P of that unit
  auto wait = [&](uint32_t bar, uint32_t parity) {
    for (uint32_t spins = 0; !mbar_try_wait(bar, parity);) {
      if (++spins > kWaitLimit || ((spins & 255u) == 0u && *abort_word)) { *abort_word = 1u; return false; }
    }
    return true;
  };
  if (warp >= 8) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPfOtherRegs));
  if (warp == 9) {
    // ================================ loader =====================================================================
    if (lane == 0) {
      PfIter it;
      PfPiece q;
      it.init(p, (int)blockIdx.x);
      uint32_t g = 0;          // tiles issued
      bool ok = true;
      while (ok && it.next(p, q)) {
        const unsigned char* kp = p.kimg + ((int64_t)q.bh * p.nt + (q.tile0 - p.kt0)) * TB;
        const unsigned char* vp = p.vimg + ((int64_t)q.bh * p.nt + (q.tile0 - p.kt0)) * TB;
        for (int i = 0; i < q.n; ++i, ++g) {
          const uint32_t st = g % NS, ph = (g / NS) & 1u;
          if (g >= NS && !wait(kempty + 8 * st, ph ^ 1u)) { ok = false; break; }
          mbar_expect_tx(kfull + 8 * st, TB);
          bulk_g2s(sK + st * TB, kp + (int64_t)i * TB, TB, kfull + 8 * st);
          // (all CTAs start at once, and the first S wants a tile of K and the queries: what is needed later waits for those, which is
          //  worth 0.1 to 0.6 % of a call, 2.6 of a causal prompt of 500, and costs 4 x 500 with heads of 64 0.3.  Only
          //  where the piece has a second tile: its K is issued behind this wait, so no stream gets to its next queries before.  Of a
          //  piece of one tile a stream does without V, its barrier is then two phases on, and this wait would never end.)
          if (g == 0 && q.n > 1) { wait(qfull, 0u); if (p.streams > 1) wait(qfull + 8, 0u); }
          if (g >= NS && !wait(vempty + 8 * st, ph ^ 1u)) {
            ok = false;
            uint32_t spins = 0;      // the K copy just issued must have landed before the CTA leaves
            while (!mbar_try_wait(kfull + 8 * st, ph) && ++spins < kWaitLimit) {}
            break;
          }
          mbar_expect_tx(vfull + 8 * st, TB);
          bulk_g2s(sV + st * TB, vp + (int64_t)i * TB, TB, vfull + 8 * st);
        }
      }
      // no copy may be in flight when the CTA exits (bounded)
      for (uint32_t k = 1; k <= (g < NS ? g : NS); ++k) {
        const uint32_t st = (g - k) % NS, ph = ((g - k) / NS) & 1u;
        uint32_t spins = 0;
        while (!mbar_try_wait(kfull + 8 * st, ph) && ++spins < kWaitLimit) {}
        while (!mbar_try_wait(vfull + 8 * st, ph) && ++spins < kWaitLimit) {}
      }
    }
  } else if ((warp - 8) / 2 < p.streams && (warp & 1) == 0) {
    // ================================ MMA issuers: one warp per stream, converged ====================================
    // (A ready wait costs its warp about 200 clocks; with one warp for both streams the tensor cores ran dry meanwhile.)
    const int s = (warp - 8) / 2;
    PfIter it;
    PfPiece q;
    it.init(p, (int)blockIdx.x);
    auto wait_w = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };   // one answer per warp
    constexpr uint32_t id_qk = f16_idesc(128, 128), id_pv = f16_idesc(128, D, true);
    // S of the tile in stage st; O += P V of a part of its keys
    auto qk = [&](uint32_t st) {
      const uint64_t a0 = sw128_desc(sQ + s * TB), b0 = sw128_desc(sK + st * TB);
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const uint32_t o = ((k >> 2) * 16384 + (k & 3) * 32) >> 4;
        tc_mma_ss(128 * s, a0 + o, b0 + o, id_qk, k > 0 ? 1u : 0u);
      }
      tc_commit(sfull + 8 * s);
      tc_commit(kempty + 8 * st);
    };
    auto pv = [&](uint32_t st, int part, bool acc) {
      const uint64_t b0 = sw128_mn_desc(sV + st * TB);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if ((16 * k < kPfFirst) == (part == 0))
          tc_mma_ts(256 + D * s, 128 * s + 8 * k, b0 + ((k * 16 * 128) >> 4), id_pv, acc || k > 0 ? 1u : 0u);
    };
    uint32_t g = 0, u = 0;     // tiles, units
    bool ok = true;
    while (ok && it.next(p, q)) {
      ok = wait_w(kfull + 8 * (g % NS), (g / NS) & 1u) && wait_w(qfull + 8 * s, u & 1u);
      if (!ok) break;
      // The second stream starts a unit half a tile behind the first, so that their softmax warps, which share the exponential
      // units, take turns from the first tile on.  In step they took 4600 clocks a tile; out of step, where they drift to after
      // five to fifteen tiles by themselves, 3070.  (A bound of a few thousand clocks, not a condition: nothing depends on it.)
      if (s == 1 && q.n > 1) {
        for (int spins = 0; (int)(*progress - (u + 1u)) < 0 && spins < kPfStaggerPolls; ++spins) {}
      }
      __syncwarp();
      tc_fence_after();
      if (elect_one()) qk(g % NS);
      for (int i = 0; i < q.n && ok; ++i, ++g) {
        const bool last = i + 1 == q.n;
        const uint32_t st = g % NS, ph = (g / NS) & 1u, st1 = (g + 1) % NS, ph1 = ((g + 1) / NS) & 1u;
        ok = wait_w(vfull + 8 * st, ph) && (last || wait_w(kfull + 8 * st1, ph1)) && wait_w(pfull + 16 * s, g & 1u);
        if (!ok) break;
        if (s == 0 && i == 0) *progress = u + 1u;
        tc_fence_after();
        if (elect_one()) pv(st, 0, i > 0);
        ok = wait_w(pfull + 16 * s + 8, g & 1u);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          pv(st, 1, true);
          if (last) tc_commit(odone + 8 * s);
          tc_commit(vempty + 8 * st);
          if (!last) qk(st1);
        }
      }
      ++u;
    }
    // the last commits must have arrived before the CTA's shared memory goes away
    if (ok && g > 0) {
      const uint32_t st = (g - 1) % NS, ph = ((g - 1) / NS) & 1u;
      if (wait(vempty + 8 * st, ph)) wait(kempty + 8 * st, ph);
    }
  }
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPfSoftmaxRegs));
  if ((warp >> 2) < p.streams) {
    // ================================ softmax: one thread per row ===================================================
    const int s = warp >> 2, row = threadIdx.x & 127;
    const int pl = row / p.G, gh = row - pl * p.G;
    const uint32_t lane_sel = (uint32_t)(warp & 3) << 21;               // TMEM lane 32 * (warp & 3), bits 31:16 of an address
    const uint32_t tS = tmem + 128 * s + lane_sel, tO = tmem + 256 + D * s + lane_sel;
    // The queries of a unit: a warp loads its 32 rows together, D / 8 lanes of 16 bytes to a row, eight loads in flight.  (Loads
    // and stores of every form, unrolled and in two places, were cold code of several thousand instructions at every unit.)
    constexpr int QL = D / 8, QR = 32 / QL;      // lanes per row, rows per warp-wide load
    const int c_q = lane % QL;
    const uint32_t g_inv = 65536u / (uint32_t)p.G + 1u;                   // rw / G = rw * g_inv >> 16 for rw < 128
    auto load_q = [&](const PfPiece& w) {
      const int bh = p.bh0 + w.bh, b = bh / p.Hkv, h = bh - b * p.Hkv;
      const int64_t qb = (int64_t)b * p.qs_b + (int64_t)(h * p.G) * p.qs_h + 8 * c_q;
      const int tq0 = (w.m * p.streams + s) * p.P;
      auto put = [&](int rw, uint4 v) {
        const uint32_t dst = sQ + s * TB + rw * 128 + (c_q >> 3) * 16384 + (((c_q & 7) ^ (rw & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
      };
      const int rw0 = (warp & 3) * 32 + lane / QL;
      if (p.q_vec) {
        // (offsets in the unit are 32-bit counts of 16 bytes: with 64-bit strides the addresses of eight loads took 1600 clocks)
        const uint4* qp = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.Q) + qb + (int64_t)tq0 * p.qs_t);
        const int st_h = (int)(p.qs_h >> 3), st_t = (int)(p.qs_t >> 3), n_pos = min(p.P, p.Tq - tq0);
#pragma unroll 1
        for (int k0 = 0; k0 < QL; k0 += 8) {
          uint4 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int rw = rw0 + (k0 + k) * QR, pw = (int)((uint32_t)rw * g_inv >> 16), gw = rw - pw * p.G;
            v[k] = make_uint4(0u, 0u, 0u, 0u);
            if (pw < n_pos) v[k] = __ldg(qp + (gw * st_h + pw * st_t));
          }
          const bool bf = p.q_dtype == HQMQ_BF16;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint32_t* w4 = reinterpret_cast<uint32_t*>(&v[k]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint32_t hv = pack_half2(__uint_as_float(w4[e] << 16), __uint_as_float(w4[e] & 0xffff0000u));
              w4[e] = bf ? hv : w4[e];
            }
            put(rw0 + (k0 + k) * QR, v[k]);
          }
        }
      } else {
#pragma unroll 1
        for (int k = 0; k < QL; ++k) {
          const int rw = rw0 + k * QR, pw = (int)((uint32_t)rw * g_inv >> 16), gw = rw - pw * p.G;
          const int64_t o = qb + (int64_t)gw * p.qs_h + (int64_t)(tq0 + pw) * p.qs_t;
          float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          if (pw < p.P && tq0 + pw < p.Tq) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = load_float(p.Q, o + e, p.q_dtype);
          }
          put(rw, make_uint4(pack_half2(f[0], f[1]), pack_half2(f[2], f[3]), pack_half2(f[4], f[5]), pack_half2(f[6], f[7])));
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the MMA reads it through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(qfull + 8 * s);
    };
    PfIter it;
    PfPiece q, nq;
    it.init(p, (int)blockIdx.x);
    uint32_t g = 0, u = 0;
    bool more = it.next(p, nq), ok = true;
    // (the expansion, complete by now, went on without a table somewhere: no row of the call is a result.  Units that are cut get
    //  their NaN from the merge.)
    const bool lost = __ldcg(p.status) == p.epoch;
    int tq = 0;
    bool live = false, w_live = false;
    float m_run = -INFINITY, vmul = 0.f;
    float2 l2 = make_float2(0.f, 0.f);
    for (bool first = true;; first = false) {
      // the last Q K^T of the unit is complete (or there is no unit yet): the next unit's queries may take their place
      if (more) load_q(nq);
      if (!first) {
        ok = wait(odone + 8 * s, u & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (w_live) {
          const int bh = p.bh0 + q.bh, b = bh / p.Hkv, h = bh - b * p.Hkv;
          const float l = l2.x + l2.y;
          const bool whole = q.head && q.tail;
          const float mul = whole ? (l != 0.f ? vmul / l : 0.f) : vmul;
          // a partial is stored four columns at a time ([d / 4][256 rows][4], then m and l of the rows), so that a lane stores 16 bytes
          // and its neighbours the next
          float* part0 = p.part + ((int64_t)blockIdx.x * 2 + (q.head ? 1 : 0)) * (256 * (D + 2)) + s * 128 + row;
          float* part = part0 + 3 * (s * 128 + row);
          const uint32_t stage = sO + warp * (32 * kPfOutRow);
          uint16_t* orow[4];                       // the rows this lane writes 16 bytes of (null: not a query)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int rw = (warp & 3) * 32 + 8 * k + (lane >> 2), pw = (int)((uint32_t)rw * g_inv >> 16), gw = rw - pw * p.G;
            const int tw = (q.m * p.streams + s) * p.P + pw;
            orow[k] = pw < p.P && tw < p.Tq ? reinterpret_cast<uint16_t*>(p.O) + (int64_t)b * p.os_b + (int64_t)(h * p.G + gw) * p.os_h +
                                                  (int64_t)tw * p.os_t + (lane & 3) * 8 : nullptr;
          }
          const bool bf = p.o_dtype == HQMQ_BF16;
          const float2 mul2v = make_float2(mul, mul);
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {        // (one small body: this code runs once or twice a call, from a cold instruction cache)
            uint32_t o[32];
            tc_ld32(o, tO + c);
            tc_wait_ld();
            float2 x[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = mul2(make_float2(__uint_as_float(o[2 * e]), __uint_as_float(o[2 * e + 1])), mul2v);
            if (!whole) {
#pragma unroll
              for (int e = 0; e < 16; e += 2)
                *reinterpret_cast<float4*>(part + (c + 2 * e) * 256) = make_float4(x[e].x, x[e].y, x[e + 1].x, x[e + 1].y);
            } else if (p.o_vec) {
              // through shared memory: four lanes of 16 bytes to a row's 32 columns
              uint32_t w[16];
              if (bf) {
#pragma unroll
                for (int e = 0; e < 16; ++e) { const __nv_bfloat162 t = __float22bfloat162_rn(x[e]); w[e] = *reinterpret_cast<const uint32_t*>(&t); }
              } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) { const __half2 t = __float22half2_rn(x[e]); w[e] = *reinterpret_cast<const uint32_t*>(&t); }
              }
              __syncwarp();
#pragma unroll
              for (int e = 0; e < 16; e += 4)
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(stage + lane * kPfOutRow + 4 * e), "r"(w[e]), "r"(w[e + 1]), "r"(w[e + 2]), "r"(w[e + 3]) : "memory");
              __syncwarp();
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                uint4 v;
                asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                             : "r"(stage + (8 * k + (lane >> 2)) * kPfOutRow + (lane & 3) * 16) : "memory");
                if (orow[k]) *reinterpret_cast<uint4*>(orow[k] + c) = v;
              }
            } else {
              // any strides, any type: parked in shared memory (fp32) and stored an element at a time
              const int64_t oo = (int64_t)b * p.os_b + (int64_t)(h * p.G + gh) * p.os_h + (int64_t)tq * p.os_t + c;
              float* mine = reinterpret_cast<float*>(base + (stage - s_base)) + lane;      // [16][32 lanes]: half of the columns at a time
#pragma unroll
              for (int e0 = 0; e0 < 32; e0 += 16) {
#pragma unroll
                for (int e = 0; e < 16; e += 2) { mine[e * 32] = x[(e0 + e) / 2].x; mine[(e + 1) * 32] = x[(e0 + e) / 2].y; }
#pragma unroll 1
                for (int e = 0; e < 16; ++e)
                  if (live) store_float(p.O, oo + e0 + e, mine[e * 32], p.o_dtype);
              }
            }
          }
          if (!whole) { part0[D * 256] = m_run; part0[(D + 1) * 256] = l; }
          __syncwarp();
          tc_fence_before();
        }
        ++u;
      }
      if (!more) break;
      q = nq;
      more = it.next(p, nq);
      tq = (q.m * p.streams + s) * p.P + pl;
      live = pl < p.P && tq < p.Tq;
      w_live = __any_sync(0xffffffffu, live);
      // this row's keys; the least and the most that a row of the warp sees.  (A row without a query is not written; its queries
      // are zero, and it takes whatever mask leaves the warp's loops alone.)
      int beg = 0, end = 0;
      if (live) key_range(p.Tkv, p.Tq, p.causal, p.window, tq, beg, end);
      const int beg_lo = __reduce_min_sync(0xffffffffu, live ? beg : 0x7fffffff), beg_hi = __reduce_max_sync(0xffffffffu, live ? beg : 0);
      const int end_lo = __reduce_min_sync(0xffffffffu, live ? end : 0x7fffffff), end_hi = __reduce_max_sync(0xffffffffu, live ? end : 0);
      if (!live) { beg = beg_lo; end = end_hi; }
      const float kmul = p.kmul[p.bh0 + q.bh];
      vmul = lost ? NAN : p.vmul[p.bh0 + q.bh];
      const float2 kmul2 = make_float2(kmul, kmul);
      m_run = -INFINITY;
      l2 = make_float2(0.f, 0.f);
      for (int i = 0; i < q.n; ++i, ++g) {
        ok = wait(sfull + 8 * s, g & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (w_live) {
          uint32_t r[128];
#pragma unroll
          for (int c = 0; c < 4; ++c) tc_ld32(r + 32 * c, tS + 32 * c);
          tc_wait_ld();
          const int t0 = (q.tile0 + i) * kPfTok;
          // Masks, 32 columns at a time and only where a row of the warp needs one: a warp's rows are a few neighbouring positions.
          // (Compared column by column against both ends a masked tile took 4200 clocks, an unmasked one 1850.)
          if (t0 < beg_hi || t0 + kPfTok > end_lo) {
#pragma unroll
            for (int gc = 0; gc < 4; ++gc) {
              const int tg = t0 + 32 * gc;
              if (tg < beg_hi || tg + 32 > end_lo) {
                const int hi = end - tg, lo = beg - tg;
                uint32_t see = hi >= 32 ? 0xffffffffu : hi <= 0 ? 0u : (1u << hi) - 1u;
                if (lo > 0) see &= lo >= 32 ? 0u : 0xffffffffu << lo;
#pragma unroll
                for (int e = 0; e < 32; ++e)
                  if (!(see & (1u << e))) r[32 * gc + e] = 0xff800000u;
              }
            }
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < 128; c += 8)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(r[c + 2 * e]), __uint_as_float(r[c + 2 * e + 1])));
          const float mc = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * kmul;
          if (__any_sync(0xffffffffu, mc > m_run + kPfSlack)) {
            const float m_new = fmaxf(m_run, mc);
            const float alpha = m_new == -INFINITY ? 1.f : fast_exp2(m_run - m_new);
            m_run = m_new;
            l2.x *= alpha; l2.y *= alpha;
            if (i > 0) {
              // (S of this tile was issued behind the previous tile's P V: the accumulator is complete)
#pragma unroll 1
              for (int c = 0; c < D; c += 32) {
                uint32_t o[32];
                tc_ld32(o, tO + c);
                tc_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                tc_st32(tO + c, o);
              }
            }
          }
          const float nb = m_run == -INFINITY ? 0.f : -m_run;
          const float2 nb2 = make_float2(nb, nb);
          // P goes to the tensor cores in two parts: the first part's P V runs under the other's exponentials
          auto pairs_of = [&](int grp, uint32_t* pk) {          // 32 keys
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float2 x = fma2(make_float2(__uint_as_float(r[32 * grp + 2 * e]), __uint_as_float(r[32 * grp + 2 * e + 1])), kmul2, nb2);
              x.x = fast_exp2(x.x); x.y = fast_exp2(x.y);
              const __half2 h = __float22half2_rn(x);
              // (the weights that are summed are the rounded ones the tensor cores see: the rounding cancels)
              l2 = add2(l2, __half22float2(h));
              pk[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
          };
          auto hand_over = [&](int part) {
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pfull + 16 * s + 8 * part);
          };
          if (t0 + 96 < end_hi && t0 + 32 > beg_lo) {
#pragma unroll
            for (int grp = 0; grp < 4; ++grp) {
              uint32_t pk[16];
              pairs_of(grp, pk);
              tc_st16(tS + 16 * grp, pk);
              if (32 * (grp + 1) == kPfFirst) hand_over(0);
            }
          } else {                               // 32 keys that no row of the warp sees have weights of zero
#pragma unroll
            for (int grp = 0; grp < 4; ++grp) {
              uint32_t pk[16];
              if (t0 + 32 * grp < end_hi && t0 + 32 * grp + 32 > beg_lo) {
                pairs_of(grp, pk);
              } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) pk[e] = 0u;
              }
              tc_st16(tS + 16 * grp, pk);
              if (32 * (grp + 1) == kPfFirst) hand_over(0);
            }
          }
          hand_over(1);
        } else {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) { mbar_arrive(pfull + 16 * s); mbar_arrive(pfull + 16 * s + 8); }
        }
      }
      if (!ok) break;
    }
    // A wait ran out: the rows of this unit and of the CTA's others become NaN (of a unit that is cut, the merge's do).
    for (bool left = !ok; left;) {
      const int bh = p.bh0 + q.bh, b = bh / p.Hkv, h = bh - b * p.Hkv, tn = (q.m * p.streams + s) * p.P + pl;
      if (q.head && q.tail && pl < p.P && tn < p.Tq) {
        const int64_t oo = (int64_t)b * p.os_b + (int64_t)(h * p.G + gh) * p.os_h + (int64_t)tn * p.os_t;
#pragma unroll 1
        for (int x = 0; x < D; ++x) store_float(p.O, oo + x, NAN, p.o_dtype);
      }
      left = more;
      q = nq;
      if (left) more = it.next(p, nq);
    }
  }
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_word) *p.status = p.epoch;
  if (warp == 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kPfTmemCols) : "memory");
  }
}

// ---- merge of the units that were cut between CTAs: blockIdx.x + 1 = a CTA whose piece starts inside a unit ----------------
// blockIdx.y = 32 rows of the unit: a lane per row, a warp per D / 8 columns; the result is turned in shared memory.
template <int D>
__global__ void __launch_bounds__(256) prefill_merge_kernel(const PrefillParams p) {
  constexpr int E = D / 8;
  __shared__ float tile[32][D + 1];
  const int c = blockIdx.x + 1;
  PfIter it;
  it.init(p, c);
  grid_dep_wait();                                          // (no CTA may outlive the kernel ahead of it)
  if (it.off == 0) return;                                  // the unit starts with the CTA
  const int64_t s_u = (int64_t)c * p.L - it.off;
  if ((int64_t)(c - 1) * p.L > s_u) return;                 // the unit's first boundary does the merge
  const int c0 = c - 1, n_parts = (int)((s_u + it.n - 1) / p.L) - c0 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.y * 32 + lane;
  const int bh = p.bh0 + it.bh, b = bh / p.Hkv, h = bh - b * p.Hkv;
  // the CTA that holds the unit's first tile wrote its second slot, the others their first
  constexpr int64_t kSlot = 256 * (D + 2);
  const float* part = p.part + (int64_t)c0 * 2 * kSlot + row;
  auto slot = [&](int k) { return part + k * 2 * kSlot + (k == 0 ? kSlot : 0); };
  float m = -INFINITY;
  for (int k = 0; k < n_parts; ++k) m = fmaxf(m, slot(k)[D * 256]);
  const float mu = m == -INFINITY ? 0.f : m;
  float l = 0.f, acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int k = 0; k < n_parts; ++k) {
    const float* pp = slot(k);
    const float w = fast_exp2(pp[D * 256] - mu);
    l = fmaf(pp[(D + 1) * 256], w, l);
    const float4* col = reinterpret_cast<const float4*>(pp - row) + warp * (E / 4) * 256 + row;
#pragma unroll
    for (int e = 0; e < E; e += 4) {
      const float4 v = col[e / 4 * 256];
      acc[e] = fmaf(v.x, w, acc[e]); acc[e + 1] = fmaf(v.y, w, acc[e + 1]);
      acc[e + 2] = fmaf(v.z, w, acc[e + 2]); acc[e + 3] = fmaf(v.w, w, acc[e + 3]);
    }
  }
  const bool failed = *p.status == p.epoch;                 // the attention kernel gave up on a wait
  const float inv = failed ? NAN : l != 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) tile[lane][warp * E + e] = acc[e] * inv;
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * D / 2; i += 256) {
    const int rl = i / (D / 2), x = 2 * (i - rl * (D / 2)), r = blockIdx.y * 32 + rl, s = r >> 7, pl = (r & 127) / p.G, gh = (r & 127) - pl * p.G;
    const int tq = (it.m * p.streams + s) * p.P + pl;
    if (s >= p.streams || pl >= p.P || tq >= p.Tq) continue;
    const int64_t oo = (int64_t)b * p.os_b + (int64_t)(h * p.G + gh) * p.os_h + (int64_t)tq * p.os_t + x;
    const float f0 = tile[rl][x], f1 = tile[rl][x + 1];
    if (p.o_vec)
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.O) + oo) =
          (uint32_t)float_to_bits16(f0, p.o_dtype) | ((uint32_t)float_to_bits16(f1, p.o_dtype) << 16);
    else { store_float(p.O, oo, f0, p.o_dtype); store_float(p.O, oo + 1, f1, p.o_dtype); }
  }
}

// ---- expand -------------------------------------------------------------------------------------------------------------------
// 2^(10 - e) and 2^(e - 10) for the largest scale of a (b, head), e its exponent (largest < 2^e)
__device__ __forceinline__ void pf_scale_of(float big, float& mul, float& inv) {
  int e = big > 0.f ? (int)((__float_as_uint(big) >> 23) & 255u) - 126 : 10;
  e = min(120, max(-110, e));
  mul = __uint_as_float((uint32_t)(10 - e + 127) << 23);
  inv = __uint_as_float((uint32_t)(e - 10 + 127) << 23);
}

// grid (tile chunks, (b, head) of the group, 2): blockIdx.z = 0 K, 1 V.  Eight warps; a warp takes the 16 tokens of one
// outlier block of a tile with a lane per chunk, and writes them straight to the image (the lanes of a token fill whole
// 128-byte rows).  Flagged chunks decode to zero (radius code 0) and are overwritten afterwards from a list of the block's
// entries, a lane per entry: the payload is then read in order, 32 entries at a time.  (Looked up chunk by chunk inside the
// decode loop they tripled its instructions: 46 us for 8192 tokens of 8 heads, K with 6 % flagged.)
// Bound: latency of a CTA's dependent loads (table, scales, rows, then payload): the issue slots are a quarter busy, DRAM
// less.  So the table comes by bulk copy, the scale scan and the first tile's rows are in flight with it, and a tile's rows are
// fetched while the payload of the one before is written.  8192 tokens of 8 heads, s96, K with 6 % flagged: 17.4 us (35 with V
// turned into a K-major image through shared memory, three barriers a tile and 68 KB a CTA); the tuple, 2048 tokens: 11.4 (24).
template <int N, int LAYOUT>
__global__ void __launch_bounds__(256, 4) prefill_expand_kernel(const ExpandParams e) {
  constexpr int D = 4 * N;
  constexpr uint32_t TB = (uint32_t)pf_tile_bytes(D);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint2* tbl = reinterpret_cast<uint2*>(smem_raw);
  __shared__ float s_big[8];
  __shared__ uint16_t s_list[8][16 * N];       // (token of the block) * 32 + chunk of the block's payload entries
  __shared__ __align__(8) uint64_t s_bar;
  grid_dep_launch();
  const bool is_v = blockIdx.z != 0;
  const hqmq_packed& pk = is_v ? e.V : e.K;
  const hqmq_ref_packed& rf = is_v ? e.Vr : e.Kr;
  const int bh = e.bh0 + blockIdx.y, b = bh / e.Hkv, h = bh - b * e.Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---- the head's table on its way: entries of four fp16 values by bulk copy where their address allows -----------------------
  const void* jt = is_v ? e.jV : e.jK;
  const uint2* src = (LAYOUT == 0 ? reinterpret_cast<const uint2*>(is_v ? e.tblV : e.tblK) : reinterpret_cast<const uint2*>(jt)) + (int64_t)h * e.table_rows;
  const uint32_t bar = smem_u32(&s_bar), tbytes = (uint32_t)e.table_rows * 8u;
  const bool bulk = (LAYOUT == 0 || e.j_dtype == HQMQ_F16) && ((reinterpret_cast<uintptr_t>(src) | tbytes) & 15u) == 0;
  if (bulk) {
    if (threadIdx.x == 0) {
      mbar_init(bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(bar, tbytes);
      bulk_g2s(smem_u32(tbl), src, tbytes, bar);
    }
  } else if (LAYOUT == 0) {
    for (int i = threadIdx.x; i < e.table_rows; i += 256) tbl[i] = src[i];
  } else if (e.j_dtype != HQMQ_F32 && (reinterpret_cast<uintptr_t>(src) & 7u) == 0) {
    for (int i = threadIdx.x; i < e.table_rows; i += 256) {
      const uint2 w = src[i];
      const float2 a = pair16_to_float2(w.x, e.j_dtype), d = pair16_to_float2(w.y, e.j_dtype);
      tbl[i] = make_uint2(pack_half2(a.x, a.y), pack_half2(d.x, d.y));
    }
  } else {
    for (int i = threadIdx.x; i < e.table_rows; i += 256) {
      const int64_t o = ((int64_t)h * e.table_rows + i) * 4;
      tbl[i] = make_uint2(pack_half2(load_float(jt, o, e.j_dtype), load_float(jt, o + 1, e.j_dtype)),
                          pack_half2(load_float(jt, o + 2, e.j_dtype), load_float(jt, o + 3, e.j_dtype)));
    }
  }

  // what this lane needs of the planes, as bases and 32-bit steps (a lane keeps its chunk for the whole kernel)
  const bool outl = LAYOUT == 0 && pk.flags != nullptr;
  constexpr int TPW = 32 / N;                 // tokens a warp takes at a time
  constexpr int NF = 16 / TPW;                // fields of a lane
  const int half = N == 32 ? 0 : lane >> 4, c = N == 32 ? lane : lane & 15;
  const uint32_t* rows = nullptr;
  int row_words = 0, w1 = 0, sh = 0;
  uint32_t imask = 0u, fmask = 0u;
  if constexpr (LAYOUT == 0) {
    const int cb = e.ib + pk.radius_bits, bit = c * cb;
    row_words = pk.row_bytes >> 2;
    rows = reinterpret_cast<const uint32_t*>(pk.codes + (int64_t)bh * pk.T_cap * pk.row_bytes) + (bit >> 5);
    sh = bit & 31; w1 = sh + cb > 32 ? 1 : 0;
    imask = (1u << e.ib) - 1u; fmask = (1u << cb) - 1u;
  }
  const unsigned char* vals = outl ? reinterpret_cast<const unsigned char*>(pk.out_vals) + (int64_t)bh * pk.out_cap * 8 : nullptr;   // (16-bit entries)
  const uint32_t cap = outl ? (uint32_t)pk.out_cap : 0u;
  const int out_dtype = pk.out_dtype;
  const uint32_t* flags = outl ? pk.flags + (int64_t)bh * pk.T_cap : nullptr;
  const uint32_t* offs = outl ? pk.out_off + (int64_t)bh * (pk.T_cap / HQMQ_OUT_BLOCK + 1) : nullptr;
  auto scale_of = [&](int t) {
    return LAYOUT == 0 ? load_scale(pk, (int64_t)bh * pk.T_cap + t)
                       : load_float(rf.rs, b * rf.rs_stride[0] + h * rf.rs_stride[1] + t, rf.rs_dtype);
  };
  // the rows of a tile's 16 tokens of this warp: fields (index | radius code << 16), lanes 0..15 the scale and flag word of a token
  uint32_t f[NF], myflag, run;
  float rs;
  auto fetch = [&](int tile) {
    const int tb = (e.kt0 + tile) * kPfTok + warp * 16;
    rs = 0.f; myflag = 0u; run = 0u;
    if (lane < 16 && tb + lane < e.Tkv) {
      rs = scale_of(tb + lane);
      if (outl) myflag = flags[tb + lane];
    }
    if (outl && tb < e.Tkv) run = offs[tb / HQMQ_OUT_BLOCK];
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      const int t = tb + k * TPW + half;
      f[k] = 0u;
      if (t < e.Tkv) {
        if constexpr (LAYOUT == 0) {
          const uint32_t* r = rows + t * row_words;
          const uint32_t raw = __funnelshift_r(r[0], r[w1], sh) & fmask;
          f[k] = (raw & imask) | ((raw >> e.ib) << 16);
        } else {
          const int64_t io = b * rf.idx_stride[0] + h * rf.idx_stride[1] + t * rf.idx_stride[2] + c;
          const int64_t ro = b * rf.rq_stride[0] + h * rf.rq_stride[1] + t * rf.rq_stride[2] + c;
          if (rf.idx_dtype == HQMQ_I32 && rf.rq_dtype == HQMQ_I32) {
            const int i = reinterpret_cast<const int32_t*>(rf.idx)[io], r = reinterpret_cast<const int32_t*>(rf.rq)[ro];
            f[k] = (uint32_t)min(max(i, 0), e.table_rows - 1) | ((uint32_t)min(max(r, 0), 1023) << 16);
          } else {
            long long i = load_int(rf.idx, io, rf.idx_dtype), r = load_int(rf.rq, ro, rf.rq_dtype);
            i = i < 0 ? 0 : (i >= e.table_rows ? e.table_rows - 1 : i);
            r = r < 0 ? 0 : (r > 1023 ? 1023 : r);
            f[k] = (uint32_t)i | ((uint32_t)r << 16);
          }
        }
      }
    }
  };
  const int tile_hi = min(e.nt, (int)(blockIdx.x + 1) * e.per);
  fetch(blockIdx.x * e.per);

  // ---- the largest scale of the keys in range -----------------------------------------------------------------------------
  const int t_first = e.kt0 * kPfTok, t_end = min(e.Tkv, (e.kt0 + e.nt) * kPfTok);
  float big = 0.f;
  if (LAYOUT == 0 && pk.scale_dtype != HQMQ_F32) {
    // eight 16-bit scales per load (they are positive: their bits order like their values)
    const uint16_t* rsp = reinterpret_cast<const uint16_t*>(pk.rs) + (int64_t)bh * pk.T_cap;
    uint32_t mx = 0u;
    for (int t = t_first + threadIdx.x * 8; t + 8 <= t_end; t += 256 * 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(rsp + t);
      mx = __vmaxu2(mx, __vmaxu2(__vmaxu2(v.x, v.y), __vmaxu2(v.z, v.w)));
    }
    big = fmaxf(bits16_to_float(mx & 0xffff, pk.scale_dtype), bits16_to_float(mx >> 16, pk.scale_dtype));
    const int t = (t_end & ~7) + (int)threadIdx.x;
    if (t < t_end) big = fmaxf(big, scale_of(t));
  } else {
    for (int t = t_first + threadIdx.x; t < t_end; t += 256) big = fmaxf(big, fabsf(scale_of(t)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (lane == 0) s_big[warp] = big;
  __syncthreads();                             // (the barrier word of the table's copy is initialised, too)
#pragma unroll
  for (int w = 0; w < 8; ++w) big = fmaxf(big, s_big[w]);
  float mul, inv;
  pf_scale_of(big, mul, inv);
  if (blockIdx.x == 0 && threadIdx.x == 0) (is_v ? e.vmul : e.kmul)[bh] = is_v ? inv : inv * e.qscale;
  if (bulk) {
    // (every thread waits: a CTA must not exit with a copy into it in flight.  Bounded: whoever goes on without the table raises the
    //  status word, and the rows of the whole call become NaN, see prefill_attn_kernel.)
    uint32_t spins = 0;
    while (!mbar_try_wait(bar, 0)) {
      if (++spins > kWaitLimit) { *e.status = e.epoch; break; }
    }
  }

  // four fp16 values of a chunk from its codeword and radius code
  auto value_of = [&](uint32_t fv, float fac) {
    const uint2 cw = tbl[fv & 0xffffu];
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&cw.x)), d = __half22float2(*reinterpret_cast<const __half2*>(&cw.y));
    fac *= (float)(fv >> 16);
    return make_uint2(pack_half2(a.x * fac, a.y * fac), pack_half2(d.x * fac, d.y * fac));
  };
  // ... of a flagged chunk from its payload entry (an entry the encoder dropped reads as 0)
  auto payload_of = [&](uint32_t slot) {
    if (slot >= cap) return make_uint2(0u, 0u);
    return *reinterpret_cast<const uint2*>(vals + (int64_t)slot * 8);
  };
  for (int tile = blockIdx.x * e.per; tile < tile_hi; ++tile) {
    unsigned char* dst = (is_v ? e.vimg : e.kimg) + ((int64_t)blockIdx.y * e.nt + tile) * TB;
    const float myfac = rs * e.vscale * mul;
    // the block's payload entries in order; the first 32 are fetched now
    uint32_t n_ent = 0u;
    const uint32_t run0 = run;
    uint2 ent = make_uint2(0u, 0u);
    if (outl) {
      uint32_t incl = __popc(myflag);
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
      n_ent = __shfl_sync(0xffffffffu, incl, 15);
      if (n_ent) {
        if (lane < n_ent) ent = payload_of(run0 + lane);
        uint32_t pos = incl - __popc(myflag);
        for (uint32_t w = myflag; w; w &= w - 1u) s_list[warp][pos++] = (uint16_t)(lane * 32 + __ffs(w) - 1);
      }
    }
    unsigned char* kd = dst + (c >> 4) * 16384 + (c & 1) * 8;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      const int tl = warp * 16 + k * TPW + half;
      const float fac = __shfl_sync(0xffffffffu, myfac, k * TPW + half);
      *reinterpret_cast<uint2*>(kd + tl * 128 + ((((c & 15) >> 1) ^ (tl & 7)) << 4)) = value_of(f[k], fac);
    }
    if (tile + 1 < tile_hi) fetch(tile + 1);
    if (n_ent) {
      __syncwarp();                            // (the list, and the zeros of the flagged chunks, were stored by other lanes)
      for (uint32_t i = lane; i < n_ent; i += 32) {
        if (i != lane) ent = payload_of(run0 + i);
        const uint32_t at = s_list[warp][i];
        const int tl = warp * 16 + (int)(at >> 5), cc = (int)(at & 31u);
        const float2 a = pair16_to_float2(ent.x, out_dtype), d = pair16_to_float2(ent.y, out_dtype);
        *reinterpret_cast<uint2*>(dst + (cc >> 4) * 16384 + tl * 128 + ((((cc & 15) >> 1) ^ (tl & 7)) << 4) + (cc & 1) * 8) =
            make_uint2(pack_half2(a.x * mul, a.y * mul), pack_half2(d.x * mul, d.y * mul));
      }
      __syncwarp();                            // (the next tile's list takes this one's place)
    }
  }
}

}  // namespace

// ---- host --------------------------------------------------------------------------------------------------------------------
// Workspace: status word (16 bytes) | kmul, vmul [B * H_kv] | K images, V images of a group of (b, head) | partials
bool prefill_plan(const hqmq_attn_args* a, PrefillPlan& pl) {
  const int G = a->H_q / a->H_kv;
  const int rows = a->layout == 0 ? 24 * a->K.S : a->K_size;
  if ((a->d != 64 && a->d != 128) || a->T_q < kPrefillMinQueries || a->T_kv < 1 || a->partials_only || a->kv_splits > 0) return false;
  if (rows > kPrefillMaxTable) return false;
  // Outliers are fp16 operands here: exact for a 16-bit side buffer, 11 of 24 bits of one in fp32, which the decode kernels
  // add in fp32.  The generic one of those also keeps fp32 queries for the outliers of K.  Such calls stay with them.
  if (a->layout == 0) {
    if ((a->K.flags && a->K.out_dtype == HQMQ_F32) || (a->V.flags && a->V.out_dtype == HQMQ_F32)) return false;
    if (a->K.flags && a->q_dtype == HQMQ_F32 && !staged_kernel(a)) return false;
  }
  PrefillParams& p = pl.p;
  memset(&p, 0, sizeof(p));
  p.Hkv = a->H_kv; p.G = G; p.Tq = a->T_q; p.Tkv = a->T_kv; p.causal = a->causal; p.window = a->window;
  p.P = 128 / G;
  p.streams = a->T_q > p.P ? 2 : 1;
  p.units_m = (a->T_q + p.streams * p.P - 1) / (p.streams * p.P);
  int kt1 = 0;
  for (int m = 0; m < p.units_m; ++m) {
    int lo, n;
    pf_unit_tiles(p, m, lo, n);
    if (m == 0) p.kt0 = lo;
    p.kt0 = lo < p.kt0 ? lo : p.kt0;
    kt1 = lo + n > kt1 ? lo + n : kt1;
    p.Wh += n;
  }
  p.nt = kt1 - p.kt0;
  const int bh_all = a->B * a->H_kv;
  const size_t tile = 2 * pf_tile_bytes(a->d);
  // the operand images of as many (b, head) at a time as kPrefillImageBytes hold
  int64_t gb = (int64_t)(kPrefillImageBytes / ((size_t)p.nt * tile));
  pl.group = gb < 1 ? 1 : gb > bh_all ? bh_all : (int)gb;
  // Whole units per CTA, or equal pieces of the flat sequence?  Costs in tiles: every unit about two (its queries, pipeline
  // fill, output), cut units one more for each partial, and the merge launch about six.
  const int n_units = pl.group * p.units_m;
  p.total = (int64_t)pl.group * p.Wh;
  const int64_t L = (p.total + kPfMaxCtas - 1) / kPfMaxCtas;
  const int grid_w = n_units < kPfMaxCtas ? n_units : kPfMaxCtas;
  int64_t whole = 0;
  for (int c = 0; c < grid_w; ++c) {
    int64_t t = 0;
    for (int k = 0;; ++k) {
      const int i = k * grid_w + ((k & 1) ? grid_w - 1 - c : c);
      if (i >= n_units) break;
      int lo, n;
      pf_unit_tiles(p, p.units_m - 1 - i / pl.group, lo, n);
      t += n + 2;
    }
    whole = t > whole ? t : whole;
  }
  const int64_t cut = L + 2 * ((n_units + kPfMaxCtas - 1) / kPfMaxCtas + 1) + 2 + 6;
  pl.whole = whole <= cut;
  pl.grid = pl.whole ? grid_w : (int)((p.total + (L < 1 ? 1 : L) - 1) / (L < 1 ? 1 : L));
  pl.off_mul = 16;
  pl.off_img = (16 + (size_t)bh_all * 8 + 255) & ~(size_t)255;
  pl.off_part = pl.off_img + (size_t)pl.group * p.nt * tile;
  pl.ws_bytes = pl.off_part + (pl.whole ? 0 : (size_t)pl.grid * 2 * 256 * (a->d + 2) * sizeof(float));
  return true;
}

// Launch that may start while its predecessor on the stream finishes (see grid_dep_wait).
static cudaError_t launch_dependent(const void* k, dim3 grid, int threads, void** args, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = &at; cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, k, args);
}
int prefill_launch(const hqmq_attn_args* a, const PrefillPlan& pl, void* workspace, float qscale, uint32_t epoch, cudaStream_t st) {
  PrefillParams p = pl.p;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  const int bh_all = a->B * a->H_kv, d = a->d;
  p.Q = a->Q; p.q_dtype = a->q_dtype; p.qs_b = a->q_stride[0]; p.qs_h = a->q_stride[1]; p.qs_t = a->q_stride[2];
  p.O = a->O; p.o_dtype = a->o_dtype; p.os_b = a->o_stride[0]; p.os_h = a->o_stride[1]; p.os_t = a->o_stride[2];
  auto vec = [](const void* ptr, const int64_t* s, int dt) {
    return dt != HQMQ_F32 && ((uintptr_t)ptr & 15) == 0 && s[0] % 8 == 0 && s[1] % 8 == 0 && s[2] % 8 == 0;
  };
  // (offsets inside a unit, up to 128 positions or heads away, are 32-bit counts of 16 bytes)
  auto near = [](int64_t st) { return st > -((int64_t)1 << 26) && st < ((int64_t)1 << 26); };
  p.q_vec = vec(a->Q, a->q_stride, a->q_dtype) && near(a->q_stride[1]) && near(a->q_stride[2]); p.o_vec = vec(a->O, a->o_stride, a->o_dtype);
  p.status = reinterpret_cast<uint32_t*>(ws); p.epoch = epoch;
  float* mul = reinterpret_cast<float*>(ws + pl.off_mul);
  p.kmul = mul; p.vmul = mul + bh_all;
  ExpandParams e;
  memset(&e, 0, sizeof(e));
  e.Hkv = a->H_kv; e.Tkv = a->T_kv; e.kt0 = p.kt0; e.nt = p.nt;
  e.qscale = qscale; e.vscale = 1.0f / (float)a->r_qmax;
  e.kmul = mul; e.vmul = mul + bh_all;
  e.status = p.status; e.epoch = epoch;
  if (a->layout == 0) {
    e.K = a->K; e.V = a->V; e.tblK = a->table_K; e.tblV = a->table_V;
    e.ib = idx_bits_for(a->K.S); e.table_rows = 24 * a->K.S;
  } else {
    e.Kr = a->K_ref; e.Vr = a->V_ref; e.jK = a->joint_K; e.jV = a->joint_V; e.j_dtype = a->joint_dtype;
    e.ib = 16; e.table_rows = a->K_size;
  }
  const size_t img_bytes = (size_t)pl.group * p.nt * pf_tile_bytes(d);
  e.kimg = ws + pl.off_img; e.vimg = e.kimg + img_bytes;
  p.kimg = e.kimg; p.vimg = e.vimg;
  p.part = reinterpret_cast<float*>(ws + pl.off_part);
  const int N = d / 4;
  const size_t esmem = (size_t)e.table_rows * 8;
  const void* ek = N == 32 ? (a->layout == 0 ? (const void*)&prefill_expand_kernel<32, 0> : (const void*)&prefill_expand_kernel<32, 1>)
                           : (a->layout == 0 ? (const void*)&prefill_expand_kernel<16, 0> : (const void*)&prefill_expand_kernel<16, 1>);
  const void* ak = d == 128 ? (const void*)&prefill_attn_kernel<128> : (const void*)&prefill_attn_kernel<64>;
  const void* mk = d == 128 ? (const void*)&prefill_merge_kernel<128> : (const void*)&prefill_merge_kernel<64>;
  HQMQ_CHECK_CUDA(raise_smem_limit(ek, esmem));
  HQMQ_CHECK_CUDA(raise_smem_limit(ak, pf_smem_bytes(d)));
  for (int bh0 = 0; bh0 < bh_all; bh0 += pl.group) {
    const int n_bh = bh_all - bh0 < pl.group ? bh_all - bh0 : pl.group;
    e.bh0 = p.bh0 = bh0;
    p.total = (int64_t)n_bh * p.Wh;
    p.units_all = n_bh * p.units_m;
    p.L = pl.whole ? 0 : (p.total + pl.grid - 1) / pl.grid;
    const int grid = pl.whole ? (p.units_all < pl.grid ? p.units_all : pl.grid) : (int)((p.total + p.L - 1) / p.L);
    // where every CTA's piece starts: its unit, and the tiles of the unit before it
    if (!pl.whole) {
      int64_t at = 0;                 // flat position of unit m of the current (b, head)
      int m = 0, lo, n;
      pf_unit_tiles(p, m, lo, n);
      for (int c = 0; c < grid; ++c) {
        const int64_t pos = (int64_t)c * p.L;
        if (pos - at >= p.Wh) at += (pos - at) / p.Wh * p.Wh;          // whole (b, head)s at once
        while (pos - at >= n) {
          at += n;
          if (++m == p.units_m) m = 0;
          pf_unit_tiles(p, m, lo, n);
        }
        p.start_m[c] = m; p.start_off[c] = (int)(pos - at);
      }
    }
    // Tiles per expand CTA: about six CTAs per SM in all (four at a time), so that a CTA's table and scale scan serve several tiles of a
    // long cache.  Six / four, us a call of 16 queries, 8 heads: 16 sequences of 300 keys 24.8 / 26.6, of 4000 167 / 160, of 16000 630 /
    // 639; one of 16000 81 / 74, of 65536 199 / 176 (eight 181, twelve 187).  Neither is the shorter one everywhere: what decides is how
    // the CTAs of a (b, head) divide its tiles, which the line does not look at.
    const int64_t per = ((int64_t)p.nt * n_bh * 2 + 6 * kPfMaxCtas - 1) / (6 * kPfMaxCtas);
    e.per = per < 1 ? 1 : per > p.nt ? p.nt : (int)per;
    void* ea[] = {&e};
    HQMQ_CHECK_CUDA(cudaLaunchKernel(ek, dim3((p.nt + e.per - 1) / e.per, n_bh, 2), dim3(256), ea, esmem, st));
    void* pa[] = {&p};
    HQMQ_CHECK_CUDA(launch_dependent(ak, dim3(grid), kPfThreads, pa, pf_smem_bytes(d), st));
    if (!pl.whole && grid > 1) HQMQ_CHECK_CUDA(launch_dependent(mk, dim3(grid - 1, 4 * p.streams), 256, pa, 0, st));
  }
  return HQMQ_OK;
}

}  // namespace attn
}  // namespace hqmq
