// KV-cache encoder for sm_100a: chunk norms, per-token-max radius codes, nearest codeword of
// the 24*S product codebook, Med3x median / flags / outlier side buffer, bit-packed rows.
//
// Arithmetic contract (bit-exact with the reference evaluated on the fp32 upcast of x):
//   norm   = sqrt(((x0^2 + x1^2) + x2^2) + x3^2), every op a separate IEEE fp32 op
//   radius = max(norm, 1e-8); r_max = max over the token's chunks (flagged ones included)
//   rq     = clamp(rint((radius / (r_max / qmax))), 0, qmax) with two IEEE divisions
//   idx    = argmax_k <x/radius, joint[k]>; exhaustive search evaluates, for every secondary
//            s, y = u * conj(q_s) and snaps y to the 24-cell in closed form
//   med    = torch.quantile(norms of the head, 0.5): the two middle order statistics a <= b,
//            med = a if N odd else b - (b - a) * 0.5; flag = norm > med * C (strict)
// A flagged chunk keeps its index but its stored radius code is 0: its values live in the side buffer.
#include <string.h>

#include <atomic>

#include "attn_prefill.cuh"      // raise_smem_limit
#include "common.cuh"

namespace hqmq {

namespace {

constexpr int kEncThreads = 512;
constexpr int kEncWarps = kEncThreads / 32;
constexpr int kEncIters = 8;      // token groups per block
constexpr int kHistBins = 2048;   // 11-bit digits: bits [31:21], [20:10], then 10 bits [9:0]
constexpr int kMaxRowWords = 20;
constexpr int kBandWords = 4;     // per head: thr_lo bits, thr_hi bits, undecided chunks seen, spare
constexpr int kUndCap = 4096;     // undecided chunks listed per head at least; more -> the fix-up re-scans x instead

// ---- nearest-codeword look-up table -------------------------------------------------------------------
// The joint codebook {p * q_s} is invariant under left multiplication by any of the 24 Hurwitz units g, so the
// unit direction u is first FOLDED by its nearest unit: v = conj(g) * u lies in the Voronoi cell of 1 among the 24
// units, which in the coordinates w = (v1, v2, v3) / v0 is the octahedron |w1| + |w2| + |w3| <= 1, and the nearest
// codeword of u is g times the nearest codeword of v (a 24 x 24 index table).  (Folding by the nearest unit is
// closed form: the larger of the largest |u_i| and (|u0|+|u1|+|u2|+|u3|)/2 names it; conj(g) * u is a signed
// permutation for an axis unit and sums of differences of the |u_i| for a half-integer unit.)
// A grid of n cells per axis covers the octahedron (only the cells that meet it are stored: a row table over
// (cx, cy) gives the first stored cz and where the row's cells start).  Each cell names every codeword that can be
// the nearest one for some direction in the (slightly grown) cell: all k not beaten over the whole cell by the
// winner at the cell's centre, minus those beaten over the whole cell by another listed one -- the comparison of
// two codewords is linear in w, so its extreme over the box is at a corner.  A cell with ONE possible winner stores
// it in its own word (no similarity is evaluated at all); the others point at a list, padded to a multiple of four,
// which is evaluated with the same fp32 dot product an exhaustive scan of the joint table would use.  At S = 96
// (n = 44) 39 % of the cells have one winner; a list holds 2.7 codewords on average (11 at most) and 5 % are longer than four.  S = 24
// (n = 48): 60 %, 2.3, 1 %; S = 192 (n = 36): 20 %, 3.2, 15 %.
constexpr int kLutNMax = 48;
constexpr int kLutRows = kLutNMax * kLutNMax;
constexpr int kLutCellCap = 24576;          // stored cells (23.4 k at n = 48), and the one that rows without cells point at
constexpr int kLutCandCap = 65528;          // candidate entries per head (list offsets / 4 are 15-bit cell words; every head's part a multiple of 16 bytes)
constexpr int kLutMaxList = 16;             // longest list a cell may have; longer -> exhaustive search there
constexpr float kLutBoxEps = 1e-5f;         // the boxes are grown by this much (cell assignment rounding)
constexpr float kLutMargin = 1e-5f;         // a codeword is dropped only if it loses by more than this
// device layout of a table (bytes): global header {n, n_cells, ...} | rows[kLutRows] uint32 = first cell (16 bits) |
// first stored cz (8; kLutNoCells: none, and the first cell is the last of all, 0xFFFF) | stored cells of the row - 1 (8) | per head: {total candidates, valid, -, -} uint32, then
// cells[kLutCellCap] uint16 (0xFFFF: exhaustive; bit 15: the single winner in bits 0..14; else list offset / 4),
// cands[kLutCandCap] uint16 (lists of a multiple of four entries; bit 15 of a list's first entry: there are at most four codewords,
// else bit 15 marks the last one) | Mul24Both
constexpr uint32_t kLutNoCells = 255u;
constexpr size_t kLutOffRows = 32;
constexpr size_t kLutOffHeads = kLutOffRows + (size_t)kLutRows * 4;
constexpr size_t kLutHeadBytes = 16 + (size_t)kLutCellCap * 2 + (size_t)kLutCandCap * 2;

// (fold unit g, primary p of the folded winner) -> what the codeword of g * p and secondary 0 is called: its native index, or its
// index in the joint table
struct Mul24 { uint16_t v[24][24]; };
struct Mul24Both { Mul24 native, ref; };

struct Maps24 { uint8_t ref_to_native[24]; };

struct EncGeom {
  int B, H, T_new, n, npl, tpw;  // npl = lanes per token (power of two >= n), tpw = tokens per warp
  int S, ib, rbits, qmax;
  int x_dtype;
  int64_t xs_b, xs_h, xs_t;
  // d_head 64 through the kernels written for 32 chunks per token: with the tokens contiguous in memory, an even
  // token count and an even first row, two consecutive tokens form one "token" of 32 chunks (T_new, xs_t and the
  // packed rows are then those of the pairs); what is per token -- the maximum radius, the scale, the flag word, the
  // row number -- is taken per half-warp (PAIR).
};

// Workspace layout (uint32 words)
struct EncWs {
  uint32_t* status;   // [4]
  uint32_t* hist;     // [H][3 levels][2 queries][kHistBins]
  uint32_t* sel;      // [H][8]: prefix_lo, rank_lo, prefix_hi, rank_hi, a_bits, b_bits, thr_bits, med_bits
};

__device__ __forceinline__ void load_chunk(const void* x, int64_t off, int dtype, float v[4]) {
  if (dtype == HQMQ_F32) {
    float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + off);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    uint2 r = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(x) + off);
    uint16_t a = r.x & 0xffff, b = r.x >> 16, c = r.y & 0xffff, d = r.y >> 16;
    v[0] = bits16_to_float(a, dtype); v[1] = bits16_to_float(b, dtype);
    v[2] = bits16_to_float(c, dtype); v[3] = bits16_to_float(d, dtype);
  }
}

__device__ __forceinline__ float chunk_norm(const float v[4]) {
  float s = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(v[0], v[0]), __fmul_rn(v[1], v[1])), __fmul_rn(v[2], v[2])),
                      __fmul_rn(v[3], v[3]));
  return __fsqrt_rn(s);
}

// Closed-form nearest 24-cell vertex to y: returns similarity and writes the reference
// primary index (axis candidates 0..7, half-integer candidates 8..23).
__device__ __forceinline__ float snap24(float y0, float y1, float y2, float y3, int& p) {
  float a0 = fabsf(y0), a1 = fabsf(y1), a2 = fabsf(y2), a3 = fabsf(y3);
  float best = a0; int ax = 0;
  if (a1 > best) { best = a1; ax = 1; }
  if (a2 > best) { best = a2; ax = 2; }
  if (a3 > best) { best = a3; ax = 3; }
  float yv = ax == 0 ? y0 : ax == 1 ? y1 : ax == 2 ? y2 : y3;
  p = 2 * ax + (yv < 0.f ? 1 : 0);
  float half = 0.5f * (((a0 + a1) + a2) + a3);
  if (half > best) {
    best = half;
    p = 8 + ((y0 < 0.f) << 3) + ((y1 < 0.f) << 2) + ((y2 < 0.f) << 1) + (y3 < 0.f);
  }
  return best;
}

// Exhaustive search: for every secondary quaternion q_s (shared memory, fp32), rotate the
// unit direction by conj(q_s) and snap.  Ties keep the smallest reference index p*S + s.
__device__ __forceinline__ int search_exhaustive(const float4* __restrict__ qs, int S, float u0, float u1, float u2,
                                                 float u3, int& best_s) {
  float best = -1.f; int bp = 0, bs = 0;
  for (int s = 0; s < S; ++s) {
    float4 q = qs[s];
    float y0 = u0 * q.x + u1 * q.y + u2 * q.z + u3 * q.w;
    float y1 = -u0 * q.y + u1 * q.x - u2 * q.w + u3 * q.z;
    float y2 = -u0 * q.z + u1 * q.w + u2 * q.x - u3 * q.y;
    float y3 = -u0 * q.w - u1 * q.z + u2 * q.y + u3 * q.x;
    int p;
    float sim = snap24(y0, y1, y2, y3, p);
    if (sim > best || (sim == best && p < bp)) { best = sim; bp = p; bs = s; }
  }
  best_s = bs;
  return bp;
}

// A table as a kernel sees it (global or shared memory).
struct LutView {
  const uint32_t* rows; const uint16_t* cells; const uint16_t* cands;
  const uint16_t* nm;    // [24][24], one of Mul24Both
  int n, step;           // cells per axis; what the next secondary adds to a codeword's index: 8 (native) or 1 (joint table)
  uint32_t k_row;        // 0x4B000000 * (n + 1): the exponents of two cell coordinates in n * cx + cy
  float hn, off;         // n / 2 less four parts per million, n / 2 + 2^23
  uint32_t s_mul;        // k / S = umulhi(2 k, s_mul) for k < 32768
};
__device__ __forceinline__ void lut_set(LutView& L, int n, int S, bool ref) {
  L.n = n; L.step = ref ? 1 : 8;
  L.k_row = 0x4B000000u * (uint32_t)(n + 1);
  // (the shrunk scale keeps |w| <= 1 inside the grid without a clamp; it moves a direction by 4e-6 of a box grown by 1e-5)
  L.hn = 0.5f * (float)n * (1.f - 4e-6f); L.off = 0.5f * (float)n + 8388608.f;
  L.s_mul = (0x80000000u + (uint32_t)S - 1u) / (uint32_t)S;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The order statistics torch.quantile(flat, q) interpolates between and its weight, with torch's own arithmetic
// (ATen quantile_compute: rank = fl32(fl32(q) * fl32(N - 1)), below = trunc, above = ceil, weight = rank - below;
// lerp with one fused multiply-add, a + w * (b - a) for w < 0.5, else b - (b - a) * (1 - w)).  q <= 0 names the
// median of Med3x with exact integer ranks: (N - 1) / 2 and N / 2, weight 0.5 for an even count.
struct QRank { uint64_t lo, hi; float w; };
__host__ __device__ inline QRank quantile_rank(uint64_t N, float q) {
  QRank r;
  if (!(q > 0.f)) { r.lo = (N - 1) / 2; r.hi = N / 2; r.w = (N & 1) ? 0.f : 0.5f; return r; }
  volatile float last = (float)(N - 1);
  volatile float rf = q * last;
  const float rfl = rf;
  r.lo = (uint64_t)rfl;
  r.hi = (uint64_t)ceilf(rfl);
  r.w = rfl - (float)r.lo;
  return r;
}
__device__ __forceinline__ float quantile_lerp(float a, float b, float w) {
  const float diff = __fsub_rn(b, a);
  return w < 0.5f ? __fmaf_rn(w, diff, a) : __fmaf_rn(-diff, __fsub_rn(1.f, w), b);
}

// Nearest codeword of the direction u through the table: writes its index (native or joint, by the view) and returns true, or
// false when the chunk has to take the exhaustive search (zero direction, one that is no number, a cell without a list).
// Every issue slot here is paid once per 32 chunks and bounds the encoders.  So there is one way through: what has to take the other
// search is found on the way (every look-up stays inside its table whatever the direction), not branched for.
__device__ __forceinline__ bool search_fold24(const float4* __restrict__ joint, const LutView& L, int S,
                                              float u0, float u1, float u2, float u3, uint32_t& code) {
  const float a0 = fabsf(u0), a1 = fabsf(u1), a2 = fabsf(u2), a3 = fabsf(u3);
  const float hs = ((a0 + a1) + a2) + a3;          // twice the similarity of the nearest half-integer unit
  bool found = hs > 0.f && hs < 4.f;                // (a direction has |u_0| + .. + |u_3| <= 2)
  const float m01 = fmaxf(a0, a1), m23 = fmaxf(a2, a3), am = fmaxf(m01, m23);
  // Both folds are taken and one is selected: the lanes of a warp need either and all four axes, and as branches they were a
  // quarter of the kernel's instructions (28 BRA, 30 BSSY / BSYNC of 411 per token).
  // g = (s0, s1, s2, s3) / 2 with s_i = sign(u_i); 2 conj(g) u in terms of s_i u_j (products with +-1 are exact, so every difference
  // is rounded once, on the FMA pipe)
  const uint32_t b0 = __float_as_uint(u0), b1 = __float_as_uint(u1), b2 = __float_as_uint(u2), b3 = __float_as_uint(u3);
  auto sign_of = [](uint32_t b) { return __uint_as_float((b & 0x80000000u) | 0x3f800000u); };
  const float s0 = sign_of(b0), s1 = sign_of(b1), s2 = sign_of(b2), s3 = sign_of(b3);
  const bool half = hs > 2.f * am;
  const float h1 = __fadd_rn(__fmaf_rn(s0, u1, -(s1 * u0)), __fmaf_rn(s3, u2, -(s2 * u3)));
  const float h2 = __fadd_rn(__fmaf_rn(s0, u2, -(s2 * u0)), __fmaf_rn(s1, u3, -(s3 * u1)));
  const float h3 = __fadd_rn(__fmaf_rn(s0, u3, -(s3 * u0)), __fmaf_rn(s2, u1, -(s1 * u2)));
  // g = the axis of the largest |u_i| (the first of equals) with its sign: conj(g) u swaps neighbours (o), pairs (w), and signs
  const bool w = m23 > m01, o = w ? a3 > a2 : a1 > a0;
  const uint32_t q0 = o ? b1 : b0, q1 = o ? b0 : b1, q2 = o ? b3 : b2, q3 = o ? b2 : b3;
  const uint32_t e0 = w ? q2 : q0, e1 = w ? q3 : q1, e2 = w ? q0 : q2, e3 = w ? q1 : q3;
  const uint32_t neg = e0 & 0x80000000u, f3 = o ? 0x80000000u : 0u, f2 = w ? 0x80000000u : 0u;
  const float v0 = half ? hs : am;
  const float v1 = half ? h1 : __uint_as_float(e1 ^ neg ^ (f2 ^ f3));
  const float v2 = half ? h2 : __uint_as_float(e2 ^ neg ^ f2);
  const float v3 = half ? h3 : __uint_as_float(e3 ^ neg ^ f3);
  const uint32_t signs = __funnelshift_l(b3, __funnelshift_l(b2, __funnelshift_l(b1, b0 >> 31, 1), 1), 1);
  const uint32_t gp = half ? 8u + signs : (w ? 4u : 0u) + (o ? 2u : 0u) + (neg >> 31);
  // Cell coordinates as the low bits of floats of 2^23 and more, rounded down; clamped once, for memory's sake.  A row without cells
  // has one that sends the chunk to the other search.  A cz outside its row's cells would be taken for the last of them, and none
  // is: a folded direction lies in the octahedron but for its roundings (the sums, the approximate reciprocal and the product, less
  // than 1e-6 of a coordinate) and the shrunk scale's 4e-6, and the cells are those whose boxes, grown by 1e-5, meet it.
  const float inv = rcp_approx(v0) * L.hn;
  const uint32_t cx = __float_as_uint(__fmaf_rd(v1, inv, L.off)), cy = __float_as_uint(__fmaf_rd(v2, inv, L.off)),
                 cz = __float_as_uint(__fmaf_rd(v3, inv, L.off));
  const uint32_t row = L.rows[min(cx * (uint32_t)L.n + (cy - L.k_row), (uint32_t)(L.n * L.n - 1))];
  const uint32_t zc = min(cz - 0x4B000000u - ((row >> 16) & 255u), row >> 24);
  const uint32_t cw = L.cells[(row & 0xffffu) + zc];
  found &= cw != 0xffffu;
  uint32_t bk = found ? cw & 0x7fffu : 0u;          // the single winner, if that is what the cell names
  if (cw < 0x8000u) {
    float best = -3.f;
    bk = 0;
    // Four at once, and the rest one by one: the warp goes on for its longest list, 5 or 6 codewords where a lane has more than 4
    // (a second group of four cost 45 instructions for what 12 or 24 do; s96: two thirds of the warps).
    const uint16_t* e = L.cands + cw * 4u;
    const uint2 kk = *reinterpret_cast<const uint2*>(e);
    const uint32_t k0 = kk.x & 0x7fff, k1 = kk.x >> 16, k2 = kk.y & 0xffff, k3 = kk.y >> 16;
    const float4 c0 = joint[k0], c1 = joint[k1], c2 = joint[k2], c3 = joint[k3];
    const float t0 = fmaf(v3, c0.w, fmaf(v2, c0.z, fmaf(v1, c0.y, v0 * c0.x)));
    const float t1 = fmaf(v3, c1.w, fmaf(v2, c1.z, fmaf(v1, c1.y, v0 * c1.x)));
    const float t2 = fmaf(v3, c2.w, fmaf(v2, c2.z, fmaf(v1, c2.y, v0 * c2.x)));
    const float t3 = fmaf(v3, c3.w, fmaf(v2, c3.z, fmaf(v1, c3.y, v0 * c3.x)));
    if (t0 > best) { best = t0; bk = k0; }
    if (t1 > best) { best = t1; bk = k1; }
    if (t2 > best) { best = t2; bk = k2; }
    if (t3 > best) { best = t3; bk = k3; }
    for (uint32_t last = kk.x; !(last & 0x8000u);) {
      last = e[4];
      ++e;
      const uint32_t k = last & 0x7fffu;
      const float4 c = joint[k];
      const float t = fmaf(v3, c.w, fmaf(v2, c.z, fmaf(v1, c.y, v0 * c.x)));
      if (t > best) { best = t; bk = k; }
    }
  }
  const uint32_t pf = __umulhi(2u * bk, L.s_mul);
  code = L.nm[gp * 24u + pf] + (bk - pf * (uint32_t)S) * (uint32_t)L.step;
  return found;
}
// The same index of the codeword that the exhaustive search names (ref: the one in the joint table).
template <bool REF>
__device__ __forceinline__ uint32_t code_of(int p, int sidx, int S, const Maps24& maps) {
  if (REF) return (uint32_t)(p * S + sidx);
  const int au = maps.ref_to_native[p];
  return (uint32_t)((((au >> 3) * S + sidx) << 3) | (au & 7));
}
// x / b for a small whole b, rounded to nearest: y = 1 / b rounded, a first quotient and one step with its exact remainder
// (P. Markstein, IBM J. Res. Dev. 34, 1990: correctly rounded where y is and nothing under- or overflows; checked against the
// division for every fraction and b = 1, 3, .., 255).  An infinite x takes the division.
template <int B>
__device__ __forceinline__ float div_whole(float x) {
  constexpr float y = 1.0f / (float)B;
  const float q = x * y;
  return x < 1e38f ? __fmaf_rn(__fmaf_rn(-q, (float)B, x), y, q) : __fdiv_rn(x, (float)B);
}

// Bytes of shared memory a kernel needs for a table of n cells per axis, n_cells stored cells and n_cand candidates.
__host__ __device__ inline size_t lut_smem_bytes(int n, int n_cells, int n_cand) {
  return (size_t)n * n * 4 + (((size_t)n_cells * 2 + 15) & ~(size_t)15) + (((size_t)n_cand * 2 + 15) & ~(size_t)15) + sizeof(Mul24);
}
// Copy head h's table into shared memory at `dst` (all threads of the CTA; the caller synchronises) and return the view.
__device__ __forceinline__ LutView lut_to_smem(const unsigned char* __restrict__ lut, int h, int H, int S, unsigned char* dst) {
  const uint32_t* gh = reinterpret_cast<const uint32_t*>(lut);
  const int n = (int)gh[0], n_cells = (int)gh[1];
  const unsigned char* head = lut + kLutOffHeads + (size_t)h * kLutHeadBytes;
  const uint32_t total = reinterpret_cast<const uint32_t*>(head)[0];
  uint32_t* rows = reinterpret_cast<uint32_t*>(dst);
  uint16_t* cells = reinterpret_cast<uint16_t*>(dst + (size_t)n * n * 4);
  uint16_t* cands = reinterpret_cast<uint16_t*>(dst + (size_t)n * n * 4 + (((size_t)n_cells * 2 + 15) & ~(size_t)15));
  uint16_t* snm = cands + (((size_t)total + 7) & ~(size_t)7);
  const uint32_t* grows = reinterpret_cast<const uint32_t*>(lut + kLutOffRows);
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) rows[i] = grows[i];
  const uint32_t* gc = reinterpret_cast<const uint32_t*>(head + 16);
  for (int i = threadIdx.x; i < (n_cells + 1) / 2; i += blockDim.x) reinterpret_cast<uint32_t*>(cells)[i] = gc[i];
  const uint32_t* gd = reinterpret_cast<const uint32_t*>(head + 16 + (size_t)kLutCellCap * 2);
  for (uint32_t i = threadIdx.x; i < (total + 1) / 2; i += blockDim.x) reinterpret_cast<uint32_t*>(cands)[i] = gd[i];
  const uint16_t* gn = reinterpret_cast<const uint16_t*>(lut + kLutOffHeads + (size_t)H * kLutHeadBytes);
  for (int i = threadIdx.x; i < 576; i += blockDim.x) snm[i] = gn[i];
  LutView L;
  L.rows = rows; L.cells = cells; L.cands = cands; L.nm = snm;
  lut_set(L, n, S, false);
  return L;
}
// The same table read in place from global memory (small calls).
__device__ __forceinline__ LutView lut_global(const unsigned char* __restrict__ lut, int h, int H, int S, bool ref) {
  const uint32_t* gh = reinterpret_cast<const uint32_t*>(lut);
  const unsigned char* head = lut + kLutOffHeads + (size_t)h * kLutHeadBytes;
  LutView L;
  L.rows = reinterpret_cast<const uint32_t*>(lut + kLutOffRows);
  L.cells = reinterpret_cast<const uint16_t*>(head + 16);
  L.cands = reinterpret_cast<const uint16_t*>(head + 16 + (size_t)kLutCellCap * 2);
  L.nm = reinterpret_cast<const uint16_t*>(lut + kLutOffHeads + (size_t)H * kLutHeadBytes) + (ref ? 576 : 0);
  lut_set(L, (int)gh[0], S, ref);
  return L;
}
__device__ __forceinline__ bool lut_head_valid(const unsigned char* __restrict__ lut, int h) {
  return reinterpret_cast<const uint32_t*>(lut + kLutOffHeads + (size_t)h * kLutHeadBytes)[1] == 1u;
}

template <bool LUT>
__global__ void __launch_bounds__(kEncThreads)
encode_main_kernel(EncGeom g, const void* __restrict__ x, const float* __restrict__ qs_all, hqmq_packed dst,
                   int t_start, uint32_t* __restrict__ hist, Maps24 maps, const float* __restrict__ joint_all,
                   const unsigned char* __restrict__ lut) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* qs = reinterpret_cast<float4*>(smem_raw);
  uint32_t* rows = reinterpret_cast<uint32_t*>(qs + g.S);            // [warps][tpw][kMaxRowWords]
  uint32_t* shist = rows + kEncWarps * g.tpw * kMaxRowWords;          // [kHistBins]
  float4* sjoint = reinterpret_cast<float4*>(shist + kHistBins);      // LUT: [24 S], then the table of the head

  const int bh = blockIdx.y;
  const int h = bh % g.H, b = bh / g.H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < g.S; i += blockDim.x) qs[i] = reinterpret_cast<const float4*>(qs_all)[(int64_t)h * g.S + i];
  if (hist) for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) shist[i] = 0;
  bool use_lut = false;
  LutView L = {};
  if constexpr (LUT) {
    use_lut = lut_head_valid(lut, h);
    if (use_lut) {
      for (int i = threadIdx.x; i < 24 * g.S; i += blockDim.x) sjoint[i] = reinterpret_cast<const float4*>(joint_all)[(int64_t)h * 24 * g.S + i];
      L = lut_to_smem(lut, h, g.H, g.S, reinterpret_cast<unsigned char*>(sjoint + 24 * g.S));
    }
  }
  __syncthreads();

  const int sub = lane / g.npl, c = lane % g.npl;
  const int rw = dst.row_bytes >> 2;
  const int cb = g.ib + g.rbits;
  uint32_t* myrow = rows + (warp * g.tpw + sub) * kMaxRowWords;
  const int tok_per_iter = kEncWarps * g.tpw;
  const int t_block0 = blockIdx.x * tok_per_iter * kEncIters;

  // the chunk of the next iteration is loaded before the current one is searched
  float vn[4] = {0.f, 0.f, 0.f, 0.f};
  {
    const int t = t_block0 + warp * g.tpw + sub;
    if (t < g.T_new && c < g.n) load_chunk(x, b * g.xs_b + h * g.xs_h + t * g.xs_t + 4 * c, g.x_dtype, vn);
  }
  for (int it = 0; it < kEncIters; ++it) {
    const int t = t_block0 + it * tok_per_iter + warp * g.tpw + sub;
    const bool tok_ok = t < g.T_new;
    const bool active = tok_ok && c < g.n;
    float v[4] = {vn[0], vn[1], vn[2], vn[3]};
    vn[0] = vn[1] = vn[2] = vn[3] = 0.f;
    if (it + 1 < kEncIters) {
      const int t2 = t + tok_per_iter;
      if (t2 < g.T_new && c < g.n) load_chunk(x, b * g.xs_b + h * g.xs_h + t2 * g.xs_t + 4 * c, g.x_dtype, vn);
    }
    const float nrm = chunk_norm(v);
    const float radius = fmaxf(nrm, 1e-8f);
    float rmax = active ? radius : 0.f;
    for (int o = g.npl >> 1; o > 0; o >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    rmax = fmaxf(rmax, 1e-8f);
    const float scale = __fdiv_rn(rmax, (float)g.qmax);
    float rqf = rintf(__fdiv_rn(radius, scale));
    rqf = fminf(fmaxf(rqf, 0.f), (float)g.qmax);

    for (int w = lane; w < g.tpw * kMaxRowWords; w += 32) rows[warp * g.tpw * kMaxRowWords + w] = 0;
    __syncwarp();
    if (active) {
      // the nearest codeword does not depend on the length of the chunk: search with a cheaply
      // normalised copy (keeps the values in range) instead of the reference's exact x / radius
      const float inv_r = __frcp_rn(radius);
      const float u0 = v[0] * inv_r, u1 = v[1] * inv_r, u2 = v[2] * inv_r, u3 = v[3] * inv_r;
      uint32_t ni;
      if (!(LUT && use_lut && search_fold24(sjoint, L, g.S, u0, u1, u2, u3, ni))) {
        int s;
        const int p = search_exhaustive(qs, g.S, u0, u1, u2, u3, s);
        ni = code_of<false>(p, s, g.S, maps);
      }
      const uint32_t f = ni | ((uint32_t)rqf << g.ib);
      const int bit = c * cb, w = bit >> 5, sh = bit & 31;
      atomicOr(&myrow[w], f << sh);
      if (sh + cb > 32) atomicOr(&myrow[w + 1], f >> (32 - sh));
      if (hist) atomicAdd(&shist[__float_as_uint(nrm) >> 21], 1u);
    }
    __syncwarp();
    if (tok_ok) {
      const int64_t row = (int64_t)bh * dst.T_cap + t_start + t;
      uint32_t* out = reinterpret_cast<uint32_t*>(dst.codes + row * dst.row_bytes);
      for (int w = c; w < rw; w += g.npl) out[w] = myrow[w];
      if (c == 0) {
        store_scale(dst, row, rmax);
        if (dst.flags) dst.flags[row] = 0u;
      }
    }
    __syncwarp();
  }
  if (hist) {
    __syncthreads();
    uint32_t* gh = hist + (int64_t)h * 3 * 2 * kHistBins;  // level 0, query 0
    for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) {
      uint32_t cnt = shist[i];
      if (cnt) atomicAdd(&gh[i], cnt);
    }
  }
}

// ---- small calls (decode-time appends) ------------------------------------------------------------------
// One CTA per head does the whole call: norms, per-token scale, nearest codeword (tables read straight from
// global memory: they sit in L2 and a handful of chunks per thread do not pay for staging them), the exact
// median by rank counting in shared memory, flags, packed rows.  It replaces the main pass, the three select
// levels and the flag pass by one launch when a head has at most kSmallMax chunks in the call; the offset
// scan and the side-plane kernel follow as usual.  Same arithmetic as the large-call kernels.
constexpr int kSmallMax = 2048;          // chunks per head and call
constexpr int kSmallThreads = 1024;
constexpr int kSmallTok = 512;           // tokens per head and call (kSmallMax / 4 chunks)

// (the body is shared by the kernel of one tensor, by the kernel that appends K and V of a layer in one launch, and -- DENSE:
// the fake-quantised values go to `out`, (B, H, T, 4 n) contiguous in the type of x, nothing is packed -- by the quantizer's
// quantize calls)
template <bool DENSE>
__device__ __forceinline__ void
encode_small_body(const EncGeom& g, const void* __restrict__ x, const float* __restrict__ qs_all, const hqmq_packed& dst,
                  int t_start, const Maps24& maps, const float* __restrict__ joint_all, const unsigned char* __restrict__ lut,
                  float C, float* __restrict__ med_out, float quantile,
                  void* __restrict__ out = nullptr, uint32_t* __restrict__ n_flagged = nullptr) {
  __shared__ uint32_t keys[kSmallMax];                    // norm bits of every chunk of the head
  __shared__ uint32_t tokmax[kSmallTok];                  // bits of the largest radius of a token
  __shared__ uint32_t tokflags[kSmallTok];
  __shared__ uint32_t rows[kSmallTok / 8][kMaxRowWords];   // packed rows, 64 tokens at a time
  const int h = blockIdx.x, NT = blockDim.x;              // at most two chunks per thread
  const int n = g.n, per_b = g.T_new * n;                 // chunks of one batch entry
  const int N = g.B * per_b, n_tok = g.B * g.T_new;
  const int S = g.S;
  const bool med = C > 0.f;
  const float qmaxf = (float)g.qmax;
  for (int i = threadIdx.x; i < n_tok; i += blockDim.x) { tokmax[i] = 0u; tokflags[i] = 0u; }
  __syncthreads();

  const bool use_lut = lut && lut_head_valid(lut, h);
  LutView L = {};
  if (use_lut) L = lut_global(lut, h, g.H, S, DENSE);
  const float4* joint = reinterpret_cast<const float4*>(joint_all) + (int64_t)h * 24 * S;
  const float4* qs = reinterpret_cast<const float4*>(qs_all) + (int64_t)h * S;

  // ---- phase A: norms, token maxima, nearest codewords ------------------------------------------------------
  float nrm[2], radius[2];
  uint32_t ni[2];          // native indices (DENSE: indices in the joint table)
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = threadIdx.x + k * NT;
    nrm[k] = 0.f; radius[k] = 0.f; ni[k] = 0u;
    if (i < N) {
      const int b = i / per_b, r = i - b * per_b, t = r / n, c = r - t * n;
      float v[4];
      load_chunk(x, b * g.xs_b + h * g.xs_h + t * g.xs_t + 4 * c, g.x_dtype, v);
      nrm[k] = chunk_norm(v);
      radius[k] = fmaxf(nrm[k], 1e-8f);
      keys[i] = __float_as_uint(nrm[k]);
      atomicMax(&tokmax[b * g.T_new + t], __float_as_uint(radius[k]));   // positive floats order like their bits
      const float inv_r = __frcp_rn(radius[k]);
      const float u0 = v[0] * inv_r, u1 = v[1] * inv_r, u2 = v[2] * inv_r, u3 = v[3] * inv_r;
      if (!(use_lut && search_fold24(joint, L, S, u0, u1, u2, u3, ni[k]))) {
        int sidx;
        const int p = search_exhaustive(qs, S, u0, u1, u2, u3, sidx);
        ni[k] = code_of<DENSE>(p, sidx, S, maps);
      }
    }
  }
  __syncthreads();

  // ---- phase B: the two middle order statistics: radix select (4 x 8 bits) of the lower one in shared memory,
  // the upper one is the same value or the next larger key ------------------------------------------------------
  float thr = 0.f;
  if (med) {
    __shared__ uint32_t shist[256];
    __shared__ uint32_t s_state[4];       // prefix, rank, keys <= a, smallest key > a
    const QRank qr = quantile_rank((uint64_t)N, quantile);
    const uint32_t lo = (uint32_t)qr.lo, hi = (uint32_t)qr.hi;
    uint32_t prefix = 0u, rank = lo;
    if (N <= 256) {
      // few keys: every thread counts the keys below its own; the one of rank `lo` is the key with at most lo below and
      // more than lo at or below it (no passes, two barriers)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int i = threadIdx.x + k * NT;
        if (i < N) {
          const uint32_t key = keys[i];
          uint32_t lt = 0u, le = 0u;
          for (int j = 0; j < N; ++j) { const uint32_t y = keys[j]; lt += y < key; le += y <= key; }
          if (lt <= lo && lo < le) s_state[0] = key;       // (every such key has the same bits)
        }
      }
      __syncthreads();
      prefix = s_state[0];
      __syncthreads();
    } else
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      if (threadIdx.x < 256) shist[threadIdx.x] = 0u;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int i = threadIdx.x + k * NT;
        if (i < N) {
          const uint32_t key = keys[i];
          if (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8))) atomicAdd(&shist[(key >> shift) & 0xffu], 1u);
        }
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        uint32_t c8[8], mine = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) { c8[q] = shist[lane * 8 + q]; mine += c8[q]; }
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        const uint32_t before = incl - mine;
        if (rank >= before && rank < incl) {      // exactly one lane: the rank is below the number of matching keys
          uint32_t acc = before; int digit = lane * 8 + 7;
          bool found = false;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (!found) {
              if (acc + c8[q] > rank) { digit = lane * 8 + q; found = true; }
              else acc += c8[q];
            }
          }
          s_state[0] = prefix | ((uint32_t)digit << shift);
          s_state[1] = rank - acc;
        }
      }
      __syncthreads();
      prefix = s_state[0]; rank = s_state[1];
    }
    const uint32_t a_bits = prefix;
    if (threadIdx.x == 0) { s_state[2] = 0u; s_state[3] = 0xffffffffu; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < N) {
        const uint32_t key = keys[i];
        if (key <= a_bits) atomicAdd(&s_state[2], 1u);
        else atomicMin(&s_state[3], key);
      }
    }
    __syncthreads();
    const uint32_t b_bits = s_state[2] > hi ? a_bits : s_state[3];
    const float a = __uint_as_float(a_bits), b2 = __uint_as_float(b_bits);
    const float m = hi == lo ? a : quantile_lerp(a, b2, qr.w);
    thr = __fmul_rn(m, C);
    if (threadIdx.x == 0 && med_out) med_out[h] = m;
  }

  if constexpr (DENSE) {
    // ---- the dense values: codeword * (rq * (rmax / qmax)), one rounding each, or the original chunk where flagged ----
    uint32_t fl = 0u;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < N) {
        const int b = i / per_b, r = i - b * per_b, t = r / n, c = r - t * n;
        const float rmax = fmaxf(__uint_as_float(tokmax[b * g.T_new + t]), 1e-8f);
        const float scale = __fdiv_rn(rmax, qmaxf);
        const float rqf = fminf(fmaxf(rintf(__fdiv_rn(radius[k], scale)), 0.f), qmaxf);
        const int64_t o = ((((int64_t)b * g.H + h) * g.T_new + t) * n + c) * 4;
        float v[4];
        if (med && nrm[k] > thr) {
          ++fl;
          load_chunk(x, b * g.xs_b + h * g.xs_h + t * g.xs_t + 4 * c, g.x_dtype, v);
        } else {
          const float rad = __fmul_rn(rqf, scale);
          const float4 cw = joint[ni[k]];
          v[0] = __fmul_rn(cw.x, rad); v[1] = __fmul_rn(cw.y, rad); v[2] = __fmul_rn(cw.z, rad); v[3] = __fmul_rn(cw.w, rad);
        }
        if (g.x_dtype == HQMQ_F32) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
          uint2 w;
          w.x = float_to_bits16(v[0], g.x_dtype) | ((uint32_t)float_to_bits16(v[1], g.x_dtype) << 16);
          w.y = float_to_bits16(v[2], g.x_dtype) | ((uint32_t)float_to_bits16(v[3], g.x_dtype) << 16);
          *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(out) + o) = w;
        }
      }
    }
    if (n_flagged && med) {
      fl = __reduce_add_sync(0xffffffffu, fl);
      if ((threadIdx.x & 31) == 0 && fl) atomicAdd(n_flagged, fl);
    }
  } else {

  // ---- phase C: radius codes, flags -------------------------------------------------------------------------
  uint32_t field[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = threadIdx.x + k * NT;
    field[k] = 0u;
    if (i < N) {
      const int b = i / per_b, r = i - b * per_b, t = r / n, c = r - t * n;
      const float rmax = fmaxf(__uint_as_float(tokmax[b * g.T_new + t]), 1e-8f);
      const float scale = __fdiv_rn(rmax, qmaxf);
      float rqf = rintf(__fdiv_rn(radius[k], scale));
      rqf = fminf(fmaxf(rqf, 0.f), qmaxf);
      if (med && nrm[k] > thr) {
        atomicOr(&tokflags[b * g.T_new + t], 1u << c);
        rqf = 0.f;          // a flagged chunk is stored in the side buffer: its radius code in the row is 0
      }
      field[k] = ni[k] | ((uint32_t)rqf << g.ib);
    }
  }
  __syncthreads();

  // ---- phase D: packed rows, 64 tokens at a time; scales and flag words ---------------------------------------
  const int cb = g.ib + g.rbits, rw = dst.row_bytes >> 2;
  for (int tok0 = 0; tok0 < n_tok; tok0 += kSmallTok / 8) {
    for (int w = threadIdx.x; w < (kSmallTok / 8) * kMaxRowWords; w += blockDim.x) (&rows[0][0])[w] = 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < N) {
        const int b = i / per_b, r = i - b * per_b, t = r / n, c = r - t * n;
        const int tok = b * g.T_new + t - tok0;
        if (tok >= 0 && tok < kSmallTok / 8) {
          const int bit = c * cb, w = bit >> 5, sh = bit & 31;
          atomicOr(&rows[tok][w], field[k] << sh);
          if (sh + cb > 32) atomicOr(&rows[tok][w + 1], field[k] >> (32 - sh));
        }
      }
    }
    __syncthreads();
    const int cnt = min(kSmallTok / 8, n_tok - tok0);
    for (int w = threadIdx.x; w < cnt * rw; w += blockDim.x) {
      const int tok = tok0 + w / rw, ww = w - (w / rw) * rw;
      const int b = tok / g.T_new, t = tok - b * g.T_new;
      const int64_t row = ((int64_t)b * g.H + h) * dst.T_cap + t_start + t;
      reinterpret_cast<uint32_t*>(dst.codes + row * dst.row_bytes)[ww] = rows[tok - tok0][ww];
    }
    __syncthreads();
  }
  for (int tok = threadIdx.x; tok < n_tok; tok += blockDim.x) {
    const int b = tok / g.T_new, t = tok - b * g.T_new;
    const int64_t row = ((int64_t)b * g.H + h) * dst.T_cap + t_start + t;
    store_scale(dst, row, fmaxf(__uint_as_float(tokmax[tok]), 1e-8f));
    if (dst.flags) dst.flags[row] = tokflags[tok];
  }
  }
}

// Everything one tensor of a small call needs; two of them make the K + V append of a layer.
struct SmallArgs {
  EncGeom g;
  const void* x;
  const float* qs;
  hqmq_packed dst;
  int t_start;
  const float* joint;
  const unsigned char* lut;
  float C;
  float* med_out;
  float quantile;
  uint32_t* status;     // first word of the tensor's workspace: cleared here, set by scan_kernel on an overflow
  int blk0, nblk, scan, payload, side;
  void* out;            // dense calls: the fake-quantised tensor, and the counter that its flagged chunks are added to
  uint32_t* n_flagged;
};
// Threads of a small call's CTA: two chunks each (fewer threads, cheaper barriers).
inline int small_threads(int64_t chunks) {
  return chunks <= 128 ? 128 : chunks <= 512 ? 256 : chunks <= 1024 ? 512 : kSmallThreads;
}
struct SmallPair { SmallArgs t[2]; Maps24 maps; };

__global__ void __launch_bounds__(kSmallThreads) encode_small_kernel(SmallArgs a, Maps24 maps) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.status = 0u;
  encode_small_body<false>(a.g, a.x, a.qs, a.dst, a.t_start, maps, a.joint, a.lut, a.C, a.med_out, a.quantile);
}

__global__ void __launch_bounds__(kSmallThreads) fake_quant_small_kernel(SmallArgs a, Maps24 maps) {
  encode_small_body<true>(a.g, a.x, a.qs, a.dst, a.t_start, maps, a.joint, a.lut, a.C, a.med_out, a.quantile, a.out, a.n_flagged);
}

// ---- main pass for the common geometry ------------------------------------------------------------------
// 32 chunks per token, 16-bit input, look-up-table search, compile-time field layout: one warp per token,
// one lane per chunk, no run-time geometry in the loop.  Results are the ones encode_main_kernel gives.
constexpr int kEnc32Threads = 1024;   // one CTA per SM (the tables fill half of shared memory): 32 warps hide the search latency
constexpr int kEnc32Warps = kEnc32Threads / 32;
// A two-level select over a sample of the tokens predicts the threshold statistic; this pass then does everything that needs x
// in its one read.  Per head, `bp` holds a range [R_lo, R_hi] of norm bits around the prediction (0.2 to 1.2 % either way, by the
// sample's size, see bracket_wanted) and the bounds thr_lo / thr_hi of the threshold that follow from it.  A chunk above thr_hi is flagged
// here (radius code 0, bit in the token's flag word), a chunk at or below thr_lo is not, the few in between are listed for
// the fix-up; the norms inside the range are appended to a list (one region per CTA and head) and the norms below it are
// counted, from which list_select_kernel takes the exact order statistics -- and finds out whether the prediction held: if
// not, it raises the gate word and the one-launch encoder, which otherwise returns at once, redoes the call.
struct BracketArgs {
  const uint32_t* bp;       // [H][8]: R_lo, R_hi, thr_lo, thr_hi (float bits), norms below R_lo, ...
  uint32_t* bp_count;       // same array, for the atomics
  uint32_t* band;           // [H][kBandWords]: word 2 counts the undecided chunks
  uint32_t* und;            // [H][und_cap] undecided chunks
  uint32_t* rcnt;           // [regions] norms appended per region (may exceed rcap: the list then overflowed)
  uint32_t* rlist;          // [regions][rcap]
  uint32_t* histA;          // [H][kHistBins] top digit of (norm bits - R_lo) of the norms inside the range
  int rcap, und_cap;
};
constexpr int kBpWords = 16;

template <int DT, int IB, int RB, bool PAIR>
__global__ void __launch_bounds__(kEnc32Threads, 1)
encode_main32_kernel(EncGeom g, const uint16_t* __restrict__ x, const float* __restrict__ qs_all, hqmq_packed dst,
                     int t_start, Maps24 maps, const float* __restrict__ joint_all, const unsigned char* __restrict__ lut,
                     int64_t per, BracketArgs br) {
  __shared__ uint32_t s_below, s_rcount;
  constexpr int CB = IB + RB;
  constexpr int RW = 32 * CB / 32;                       // words per row
  constexpr float qmaxf = (float)((1 << RB) - 1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* qs = reinterpret_cast<float4*>(smem_raw);
  uint32_t* rows = reinterpret_cast<uint32_t*>(qs + g.S);            // [warps][kMaxRowWords]
  uint32_t* shist = rows + kEnc32Warps * kMaxRowWords;                  // [kHistBins]
  float4* sjoint = reinterpret_cast<float4*>(shist + kHistBins);    // [24 S], then the look-up table of the head

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.S;
  uint32_t* myrow = rows + warp * kMaxRowWords;
  // The tokens of all heads form one sequence, head by head, cut into equal pieces, one per CTA and SM: the tables are
  // loaded once or twice per CTA, and all SMs finish together.  (Cut per (batch, head), 384 CTAs of 16 x 8 heads x 8192
  // tokens were 2.6 rounds with a table load and an exit each: 547 us.)
  const int64_t W = (int64_t)g.B * g.T_new, f1 = min((int64_t)g.H * W, (int64_t)(blockIdx.x + 1) * per);
  for (int64_t f0 = (int64_t)blockIdx.x * per; f0 < f1;) {
  const int h = (int)(f0 / W);
  const int64_t f_end = min(f1, (int64_t)(h + 1) * W);
  const int w0 = (int)(f0 - (int64_t)h * W), w1 = (int)(f_end - (int64_t)h * W);
  f0 = f_end;
  for (int i = threadIdx.x; i < S; i += blockDim.x) qs[i] = reinterpret_cast<const float4*>(qs_all)[(int64_t)h * S + i];
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) shist[i] = 0;
  for (int i = threadIdx.x; i < 24 * S; i += blockDim.x) sjoint[i] = reinterpret_cast<const float4*>(joint_all)[(int64_t)h * 24 * S + i];
  const LutView L = lut_to_smem(lut, h, g.H, S, reinterpret_cast<unsigned char*>(sjoint + 24 * S));
  const int region = blockIdx.x + h;              // (the next piece has the next CTA or the next head, or both)
  const uint32_t r_lo = br.bp[h * kBpWords + 0], r_hi = br.bp[h * kBpWords + 1], s1 = br.bp[h * kBpWords + 5];
  const float thr_lo = __uint_as_float(br.bp[h * kBpWords + 2]), thr_hi = __uint_as_float(br.bp[h * kBpWords + 3]);
  uint32_t n_below = 0u;
  if (threadIdx.x == 0) { s_below = 0u; s_rcount = 0u; }
  __syncthreads();

  // this warp's token w = b * T_new + t of the head, its chunks in x and its row, advanced by kEnc32Warps tokens
  const int rpt = PAIR ? 2 : 1;
  int w = w0 + warp;
  int b = w / g.T_new, t = w - b * g.T_new;
  const uint16_t* xp = x + b * g.xs_b + h * g.xs_h + (int64_t)t * g.xs_t + 4 * lane;
  int64_t row = ((int64_t)b * g.H + h) * dst.T_cap + t_start + (int64_t)rpt * t;
  const int64_t xstep = kEnc32Warps * g.xs_t, xwrap = g.xs_b - g.T_new * g.xs_t;
  const int64_t rwrap = (int64_t)g.H * dst.T_cap - (int64_t)rpt * g.T_new;
  uint2 raw_n = make_uint2(0u, 0u);
  if (w < w1) raw_n = *reinterpret_cast<const uint2*>(xp);
  for (int bn = b, tn = t; w < w1; w += kEnc32Warps, b = bn, t = tn) {
    const uint2 raw = raw_n;
    const int64_t row_now = row;
    tn += kEnc32Warps; xp += xstep; row += rpt * kEnc32Warps;
    while (tn >= g.T_new) { tn -= g.T_new; ++bn; xp += xwrap; row += rwrap; }
    if (w + kEnc32Warps < w1) raw_n = *reinterpret_cast<const uint2*>(xp);
    float v[4];
    v[0] = bits16_to_float(raw.x & 0xffff, DT); v[1] = bits16_to_float(raw.x >> 16, DT);
    v[2] = bits16_to_float(raw.y & 0xffff, DT); v[3] = bits16_to_float(raw.y >> 16, DT);
    const float nrm = chunk_norm(v);
    const float radius = fmaxf(nrm, 1e-8f);
    // (radii are positive: their bits order like the values)
    const float rmax = __uint_as_float(PAIR ? __reduce_max_sync(lane & 16 ? 0xffff0000u : 0xffffu, __float_as_uint(radius))
                                        : __reduce_max_sync(0xffffffffu, __float_as_uint(radius)));
    const float scale = div_whole<(1 << RB) - 1>(rmax);
    // radius code: the quotient is first taken with an approximate reciprocal; only a lane whose quotient
    // lies close to a rounding boundary repeats it with the IEEE division the contract names
    float quo = radius * rcp_approx(scale);
    float rqf = rintf(quo);
    if (fabsf(quo - rqf) > 0.499f) rqf = rintf(__fdiv_rn(radius, scale));
    rqf = fminf(fmaxf(rqf, 0.f), qmaxf);
    uint32_t flag_word;
    {
      const uint32_t key = __float_as_uint(nrm);
      const bool certain = nrm > thr_hi;
      if (certain) rqf = 0.f;                       // a flagged chunk's values live in the side buffer
      flag_word = __ballot_sync(0xffffffffu, certain);
      n_below += __popc(__ballot_sync(0xffffffffu, key < r_lo));       // (every lane keeps the warp's count)
      const bool in_range = key >= r_lo && key <= r_hi, undecided = !certain && nrm > thr_lo;
      if (__any_sync(0xffffffffu, in_range || undecided)) {
        const uint32_t m = __ballot_sync(0xffffffffu, in_range);
        uint32_t base = 0u;
        if (lane == 0) base = atomicAdd(&s_rcount, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (in_range) {
          const uint32_t pos = base + __popc(m & ((1u << lane) - 1u));
          if (pos < (uint32_t)br.rcap) br.rlist[(int64_t)region * br.rcap + pos] = key;
          atomicAdd(&shist[((key - r_lo) >> s1) & (kHistBins - 1)], 1u);
        }
        if (undecided) {                            // rare: settled against the exact threshold afterwards
          const uint32_t pos = atomicAdd(&br.band[h * kBandWords + 2], 1u);
          if (pos < (uint32_t)br.und_cap)
            br.und[(int64_t)h * br.und_cap + pos] =
                PAIR ? (uint32_t)(((int64_t)b * (2 * g.T_new) + 2 * t + (lane >> 4)) * 32 + (lane & 15))
                     : (uint32_t)(((int64_t)b * g.T_new + t) * 32 + lane);
        }
        __syncwarp();
      }
    }

    // ---- nearest codeword ---------------------------------------------------------------------------
    // (the nearest codeword does not depend on the chunk's length: a cheaply normalised copy keeps the
    // values in range)
    const float inv_r = rcp_approx(radius);
    const float u0 = v[0] * inv_r, u1 = v[1] * inv_r, u2 = v[2] * inv_r, u3 = v[3] * inv_r;
    uint32_t ni;
    if (!search_fold24(sjoint, L, S, u0, u1, u2, u3, ni)) {
      // zero direction (every similarity is 0, the first index wins) or a cell without a list
      int p = 0, sidx = 0;
      if (fmaxf(fmaxf(fabsf(u0), fabsf(u1)), fmaxf(fabsf(u2), fabsf(u3))) > 0.f) p = search_exhaustive(qs, S, u0, u1, u2, u3, sidx);
      ni = code_of<false>(p, sidx, S, maps);
    }
    const uint32_t f = ni | ((uint32_t)rqf << IB);

    // ---- packed row, scale, flag word ---------------------------------------------------------------------
    uint32_t* out = reinterpret_cast<uint32_t*>(dst.codes + row_now * dst.row_bytes);   // (pairs: two rows, contiguous)
    if constexpr (CB == 16) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, f, 1);
      if (!(lane & 1)) out[lane >> 1] = f | (other << 16);
    } else {
      if (lane < RW) myrow[lane] = 0;
      __syncwarp();
      const int bit = lane * CB, w = bit >> 5, sh = bit & 31;
      atomicOr(&myrow[w], f << sh);
      if (sh + CB > 32) atomicOr(&myrow[w + 1], f >> (32 - sh));
      __syncwarp();
      if (lane < RW) out[lane] = myrow[lane];
      __syncwarp();
    }
    if (lane == 0 || (PAIR && lane == 16)) {
      const int half = lane >> 4;
      store_scale(dst, row_now + half, rmax);
      if (dst.flags) dst.flags[row_now + half] = PAIR ? (half ? flag_word >> 16 : flag_word & 0xffffu) : flag_word;
    }
  }
  if (lane == 0 && n_below) atomicAdd(&s_below, n_below);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_below) atomicAdd(&br.bp_count[h * kBpWords + 4], s_below);
    br.rcnt[region] = s_rcount;
    if (s_rcount > (uint32_t)br.rcap) atomicOr(&br.bp_count[h * kBpWords + 10], 1u);
  }
  uint32_t* gA = br.histA + (int64_t)h * kHistBins;
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x)
    if (shist[i]) atomicAdd(&gA[i], shist[i]);
  __syncthreads();          // the next head's tables and counters replace these
  }
}

// Clear the radius code of chunk c in a packed row (atomics: other threads may own neighbouring chunks).
__device__ __forceinline__ void clear_radius(uint32_t* rowp, int c, int ib, int rbits) {
  const int cb = ib + rbits;
  const int lo = c * cb + ib, hi = (c + 1) * cb;   // bit range of the radius code
  const int w0 = lo >> 5, w1 = (hi - 1) >> 5;
  const uint32_t m0 = ~0u << (lo & 31);
  const uint32_t m1 = (hi & 31) ? ~(~0u << (hi & 31)) : ~0u;
  if (w0 == w1) atomicAnd(&rowp[w0], ~(m0 & m1));
  else { atomicAnd(&rowp[w0], ~m0); atomicAnd(&rowp[w1], ~m1); }
}

#include "encode_fused.cuh"

// ---- Med3x: radix select of the two middle order statistics ------------------------------
// Level 0 histogram (bits 31:21) is accumulated by encode_main_kernel into query slot 0.
// One level for head h by a CTA of 256 threads.  The histograms may have been completed by other CTAs of this launch.
__device__ __forceinline__ void select_level(const uint32_t* hist, uint32_t* sel, int h, int level, uint64_t N, float quantile) {
  __shared__ uint64_t wtot[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;   // launched with 256 threads
  uint32_t* st = sel + h * 8;
  const QRank qr = quantile_rank(N, quantile);
  const uint64_t lo = qr.lo, hi = qr.hi;
  const uint32_t* hl = hist + ((int64_t)h * 3 + level) * 2 * kHistBins;
  const int shift = level == 0 ? 21 : level == 1 ? 10 : 0;
  const int bins = level == 2 ? 1024 : kHistBins;
  const int per = bins / 256;         // bins per thread: 8 or 4
  for (int q = 0; q < 2; ++q) {
    const uint64_t rank = level == 0 ? (q == 0 ? lo : hi) : st[2 * q + 1];
    const uint32_t prefix = level == 0 ? 0u : st[2 * q];
    // level 0 has one histogram (slot 0); deeper levels have one per query
    const uint32_t* hq = hl + (level == 0 ? 0 : q * kHistBins);
    uint32_t cnt[8];
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (i < per) v = __ldcg(reinterpret_cast<const uint4*>(hq + tid * per + i));
      cnt[i] = v.x; cnt[i + 1] = v.y; cnt[i + 2] = v.z; cnt[i + 3] = v.w;
    }
    uint64_t mine = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) mine += cnt[i];
    uint64_t incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    __syncthreads();                  // the previous query's readers of wtot are done
    if (lane == 31) wtot[warp] = incl;
    __syncthreads();
    uint64_t base = 0;
    for (int w = 0; w < warp; ++w) base += wtot[w];
    incl += base;
    const uint64_t before = incl - mine;
    // the thread whose bins hold the rank (the last thread takes an out-of-range rank)
    const bool owner = (rank >= before && rank < incl) || (tid == 255 && rank >= incl);
    if (owner) {
      uint64_t acc = before; int bin = bins - 1;
      bool found = false;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < per && !found) {
          if (acc + cnt[i] > rank) { bin = tid * per + i; found = true; }
          else acc += cnt[i];
        }
      }
      st[2 * q] = prefix | ((uint32_t)bin << shift);
      st[2 * q + 1] = (uint32_t)(rank - acc);
    }
  }
  __syncthreads();
}
__global__ void __launch_bounds__(256)
select_kernel(const uint32_t* __restrict__ hist, uint32_t* __restrict__ sel, int level, uint64_t N, float C,
              float* __restrict__ med_out, float quantile) {
  const int h = blockIdx.x;
  select_level(hist, sel, h, level, N, quantile);
  if (threadIdx.x != 0) return;
  uint32_t* st = sel + h * 8;
  const QRank qr = quantile_rank(N, quantile);
  if (level == 2) {
    const float a = __uint_as_float(st[0]), b = __uint_as_float(st[2]);
    float med = qr.hi == qr.lo ? a : quantile_lerp(a, b, qr.w);
    const float thr = __fmul_rn(med, C);
    st[4] = st[0]; st[5] = st[2];
    st[6] = __float_as_uint(thr);
    st[7] = __float_as_uint(med);
    if (med_out) med_out[h] = med;
  }
}

// Levels 1 and 2: re-read x, recompute the norms, histogram the next digit of the keys that
// match each query's prefix.
__global__ void __launch_bounds__(256)
hist_kernel(EncGeom g, const void* __restrict__ x, uint32_t* __restrict__ hist, const uint32_t* __restrict__ sel,
            int level) {
  __shared__ uint32_t sh[2][kHistBins];
  const int bh = blockIdx.y;
  const int h = bh % g.H, b = bh / g.H;
  for (int i = threadIdx.x; i < 2 * kHistBins; i += blockDim.x) (&sh[0][0])[i] = 0;
  __syncthreads();
  const uint32_t p0 = sel[h * 8 + 0], p1 = sel[h * 8 + 2];
  // level 0 (used when the histograms of several GPUs are summed between the levels): nothing is fixed yet; a
  // norm has sign bit 0 and `sel` starts zeroed, so comparing bit 31 alone lets every key through
  const int hs = level == 0 ? 31 : level == 1 ? 21 : 10;   // bits already fixed are above hs
  const int ds = level == 0 ? 21 : level == 1 ? 10 : 0;
  const uint32_t dm = level == 2 ? 0x3ffu : 0x7ffu;
  const int64_t total = (int64_t)g.T_new * g.n;
  const int64_t per_block = (total + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = blockIdx.x * per_block, i1 = min(total, i0 + per_block);
  // four independent loads in flight per thread
  for (int64_t i = i0 + threadIdx.x; i < i1; i += 4 * blockDim.x) {
    float v[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t iu = i + (int64_t)u * blockDim.x;
      if (iu < i1) {
        int64_t off = b * g.xs_b + h * g.xs_h;
        if (g.xs_t == 4 * g.n) off += iu * 4;     // tokens are contiguous: the (t, chunk) grid is flat
        else { const uint32_t t = (uint32_t)iu / (uint32_t)g.n, c = (uint32_t)iu - t * (uint32_t)g.n; off += (int64_t)t * g.xs_t + 4 * c; }
        load_chunk(x, off, g.x_dtype, v[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i + (int64_t)u * blockDim.x < i1) {
        const uint32_t key = __float_as_uint(chunk_norm(v[u]));
        const uint32_t dig = (key >> ds) & dm;
        if ((key >> hs) == (p0 >> hs)) atomicAdd(&sh[0][dig], 1u);
        if ((key >> hs) == (p1 >> hs)) atomicAdd(&sh[1][dig], 1u);
      }
    }
  }
  __syncthreads();
  uint32_t* gh = hist + ((int64_t)h * 3 + level) * 2 * kHistBins;
  for (int i = threadIdx.x; i < 2 * kHistBins; i += blockDim.x) {
    uint32_t cnt = (&sh[0][0])[i];
    if (cnt) atomicAdd(&gh[i], cnt);
  }
}

// ---- Med3x passes for the common geometry -----------------------------------------------------------------
// 32 chunks per token (d_head 128), 16-bit inputs, token rows 16-byte aligned: one lane reads two chunks
// (16 bytes), half a warp reads a token.
struct Fast32 {
  const uint16_t* x;
  int64_t xs_b, xs_h, xs_t;
  int H, T_new;
  int pair;      // 1: every "token" here is two consecutive tokens of 16 chunks (d_head 64), see EncGeom
};

template <int DT>
__device__ __forceinline__ void norms_of_two(const uint4& r, float& n0, float& n1) {
  float a[4], b[4];
  a[0] = bits16_to_float(r.x & 0xffff, DT); a[1] = bits16_to_float(r.x >> 16, DT);
  a[2] = bits16_to_float(r.y & 0xffff, DT); a[3] = bits16_to_float(r.y >> 16, DT);
  b[0] = bits16_to_float(r.z & 0xffff, DT); b[1] = bits16_to_float(r.z >> 16, DT);
  b[2] = bits16_to_float(r.w & 0xffff, DT); b[3] = bits16_to_float(r.w >> 16, DT);
  n0 = chunk_norm(a); n1 = chunk_norm(b);
}

// Histogram of every kSampleStride-th token, and from it the two order statistics of the sample: level 0 (norm bits 31:21)
// finds their bins, level 1 (bits 20:10 of the sampled norms inside those) gives them to 22 bits, and the bracket of the
// main pass with them.  The last CTA of a head to arrive (a ticket, nobody waits) does the select.
// The order statistics a <= b of the whole call are expected inside [R_lo, R_hi] = [a_s (1 - delta), b_s (1 + delta)], where
// a_s / b_s are the sample's (low bits 0 / all ones).  The threshold is fl(lerp(a, b, w) * C) with lerp(a, b, w) in [a, b]
// and fl monotone, so it then lies in [fl(R_lo * C), fl(R_hi * C)].  Whether the expectation held is checked exactly by
// list_select_kernel.
constexpr int kSampleStride = 32;
struct SampleArgs {
  uint32_t* hist; uint32_t* sel; uint32_t* tickets;     // laid out like the full ones; [H][2] arrivals
  uint64_t N; float quantile, C, delta;
  uint32_t* bp; uint32_t* band;
};
template <int DT>
__global__ void __launch_bounds__(256) sample32_kernel(Fast32 f, const SampleArgs a, int level) {
  __shared__ uint32_t sh[2][kHistBins];
  __shared__ uint32_t s_last;
  const int bh = blockIdx.y;
  const int h = bh % f.H, b = bh / f.H;
  for (int i = threadIdx.x; i < 2 * kHistBins; i += blockDim.x) (&sh[0][0])[i] = 0;
  __syncthreads();
  const uint32_t q0 = level ? a.sel[h * 8 + 0] >> 21 : 0u, q1 = level ? a.sel[h * 8 + 2] >> 21 : 0u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l16 = lane & 15;
  const int n_s = (f.T_new + kSampleStride - 1) / kSampleStride;       // sampled tokens of this (b, h)
  const uint16_t* base = f.x + b * f.xs_b + h * f.xs_h + 8 * l16;
  for (int k = blockIdx.x * 16 + warp * 2 + (lane >> 4); k < n_s; k += gridDim.x * 16) {
    const uint4 r = *reinterpret_cast<const uint4*>(base + (int64_t)k * kSampleStride * f.xs_t);
    float n[2];
    norms_of_two<DT>(r, n[0], n[1]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t key = __float_as_uint(n[e]);
      if (level == 0) atomicAdd(&sh[0][key >> 21], 1u);
      else if ((key >> 21) == q0) atomicAdd(&sh[0][(key >> 10) & 0x7ffu], 1u);
      else if ((key >> 21) == q1) atomicAdd(&sh[1][(key >> 10) & 0x7ffu], 1u);
    }
  }
  __syncthreads();
  // laid out like the full histograms: level 0 has one slot, level 1 one per order statistic
  uint32_t* gh = a.hist + ((int64_t)h * 3 + level) * 2 * kHistBins;
  const bool same = q0 == q1;
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) {
    const uint32_t c0 = sh[0][i];
    if (c0) atomicAdd(&gh[i], c0);
    if (level) {
      const uint32_t c1 = same ? c0 : sh[1][i];
      if (c1) atomicAdd(&gh[kHistBins + i], c1);
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&a.tickets[2 * h + level], 1u) == gridDim.x * (gridDim.y / f.H) - 1u ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  select_level(a.hist, a.sel, h, level, a.N, a.quantile);
  if (level == 0 || threadIdx.x != 0) return;
  uint32_t* bp = a.bp + h * kBpWords;
  const float a_s = __uint_as_float(a.sel[h * 8 + 0]), b_s = __uint_as_float(a.sel[h * 8 + 2] | 0x3ffu);
  const float r_lo = __fmul_rn(a_s, 1.f - a.delta), r_hi = __fmul_rn(b_s, 1.f + a.delta);
  bp[0] = __float_as_uint(r_lo);
  bp[1] = __float_as_uint(r_hi);
  a.band[h * kBandWords + 0] = bp[2] = __float_as_uint(__fmul_rn(r_lo, a.C));
  a.band[h * kBandWords + 1] = bp[3] = __float_as_uint(__fmul_rn(r_hi, a.C));
  // top digit of (norm bits - R_lo): 2048 bins of 2^s1 keys cover the range (a range wider than 2^22 keys -- a
  // statistic next to zero -- is left to the one-launch encoder)
  const uint32_t width = __float_as_uint(r_hi) - __float_as_uint(r_lo);
  const int bits = 32 - __clz(width | 1u);
  bp[5] = (uint32_t)(bits > 11 ? bits - 11 : 0);
}

// ---- exact order statistics of a head from what the main pass left ---------------------------------------------
// The pass counted the norms below the range, histogrammed the top digit of (norm bits - R_lo) for the norms inside
// it (`histA`, 2048 bins of 2^s1 keys each) and listed those norms per region.  Every CTA of list_select_kernel checks that
// both order statistics of its head fall inside the range (else the prediction failed and the gate word is raised), finds
// the bin of the lower one and the next non-empty bin, and histograms the low s1 bits of one region's listed norms of
// those two bins; the last CTA of the head then has both statistics exactly and writes the select words (a, b, threshold,
// statistic) like the last level of select_kernel.  (As three launches, ranks found by one thread: 20 us.)
// bp words: 0 R_lo, 1 R_hi, 2 thr_lo, 3 thr_hi, 4 norms below R_lo, 5 s1, 6 arrivals, 10 a region overflowed
// Bin of `rank` in a histogram of at most 8 * 256 bins, the entries before it and the next non-empty bin (~0: none), by a
// CTA of 256 threads; s: 11 words.
__device__ __forceinline__ void block_find_rank(const uint32_t* hist, int nbins, uint32_t rank, uint32_t* s, int& bin,
                                                uint32_t& before, int& next_bin) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (nbins + 255) / 256;
  uint32_t c[8], mine = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int at = tid * per + i;
    c[i] = i < per && at < nbins ? __ldcg(hist + at) : 0u;
    mine += c[i];
  }
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
  if (lane == 31) s[warp] = incl;
  if (tid == 0) { s[8] = (uint32_t)nbins - 1u; s[9] = 0u; s[10] = 0xffffffffu; }
  __syncthreads();
  uint32_t acc = incl - mine;
  for (int w = 0; w < warp; ++w) acc += s[w];
  if (rank >= acc && rank < acc + mine) {
    bool found = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (!found && rank < acc + c[i]) { s[8] = (uint32_t)(tid * per + i); s[9] = acc; found = true; }
      acc += c[i];
    }
  }
  __syncthreads();
  bin = (int)s[8]; before = s[9];
#pragma unroll
  for (int i = 7; i >= 0; --i)
    if (c[i] && tid * per + i > bin) incl = (uint32_t)(tid * per + i), mine = 0xffffffffu;
  if (mine == 0xffffffffu) atomicMin(&s[10], incl);
  __syncthreads();
  next_bin = (int)s[10];
  __syncthreads();
}

// grid (CTAs of the main pass that can share a head, heads): one CTA per list region
__global__ void __launch_bounds__(256)
list_select_kernel(uint32_t* __restrict__ bp_all, const uint32_t* __restrict__ histA, const uint32_t* __restrict__ rcnt,
                   const uint32_t* __restrict__ rlist, int rcap, int64_t per, int64_t W, uint32_t* histB, uint64_t N, float C,
                   float quantile, uint32_t* __restrict__ sel, float* __restrict__ med_out, uint32_t* __restrict__ gate) {
  __shared__ uint32_t s_w[11], s_tot, s_last;
  const int h = blockIdx.y, tid = threadIdx.x;
  const int64_t cta0 = h * W / per, ctas = ((h + 1) * W - 1) / per - cta0 + 1;
  if ((int64_t)blockIdx.x >= ctas) return;
  uint32_t* bp = bp_all + h * kBpWords;
  const uint32_t* hA = histA + (int64_t)h * kHistBins;
  if (tid == 0) s_tot = 0u;
  __syncthreads();
  uint32_t mine = 0;
  for (int i = tid; i < kHistBins; i += 256) mine += hA[i];
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((tid & 31) == 0 && mine) atomicAdd(&s_tot, mine);
  __syncthreads();
  const QRank qr = quantile_rank(N, quantile);
  const uint64_t below = bp[4];
  const uint32_t r_lo = bp[0], s1 = bp[5];
  if (bp[10] || s1 > 11u || qr.lo < below || qr.hi >= below + s_tot) {
    if (tid == 0) atomicExch(gate, 1u);
    return;
  }
  int bin0, bin1; uint32_t before0;
  block_find_rank(hA, kHistBins, (uint32_t)(qr.lo - below), s_w, bin0, before0, bin1);
  const uint32_t rank = (uint32_t)(qr.lo - below) - before0;
  const uint32_t lowmask = (1u << s1) - 1u;
  const int region = (int)(cta0 + blockIdx.x) + h;
  uint32_t c = rcnt[region];
  if (c > (uint32_t)rcap) c = rcap;
  const uint32_t* keys = rlist + (int64_t)region * rcap;
  uint32_t* hB = histB + (int64_t)h * 2 * kHistBins;
  // (the bins hold few keys: straight to the global histograms)
  for (uint32_t i0 = tid; i0 < c; i0 += 8 * 256) {
    uint32_t k[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) k[u] = i0 + u * 256 < c ? keys[i0 + u * 256] : 0xffffffffu;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i0 + u * 256 < c) {
        const uint32_t off = k[u] - r_lo, top = off >> s1;
        if (top == (uint32_t)bin0) atomicAdd(&hB[off & lowmask], 1u);
        else if (top == (uint32_t)bin1) atomicAdd(&hB[kHistBins + (off & lowmask)], 1u);
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&bp[6], 1u) == (uint32_t)ctas - 1u ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int nb = 1 << s1;
  int bin, next_bin; uint32_t before;
  block_find_rank(hB, nb, rank, s_w, bin, before, next_bin);
  // smallest key of the next non-empty top bin (the upper statistic when a is the last key of its bin)
  int first1 = 0, dummy_n; uint32_t dummy_b;
  if (bin1 != -1) block_find_rank(hB + kHistBins, nb, 0u, s_w, first1, dummy_b, dummy_n);
  if (tid == 0) {
    const uint32_t a_bits = r_lo + ((uint32_t)bin0 << s1) + (uint32_t)bin;
    uint32_t b_bits = a_bits;
    if (qr.hi != qr.lo && before + __ldcg(hB + bin) <= rank + 1u) {      // the key after a's run of equal keys
      if (next_bin != -1) b_bits = r_lo + ((uint32_t)bin0 << s1) + (uint32_t)next_bin;
      else b_bits = r_lo + ((uint32_t)bin1 << s1) + (uint32_t)first1;      // (the statistic exists in the list)
    }
    const float a = __uint_as_float(a_bits), b = __uint_as_float(b_bits);
    const float med = qr.hi == qr.lo ? a : quantile_lerp(a, b, qr.w);
    uint32_t* st = sel + h * 8;
    st[4] = a_bits; st[5] = b_bits;
    st[6] = __float_as_uint(__fmul_rn(med, C));
    st[7] = __float_as_uint(med);
    if (med_out) med_out[h] = med;
  }
}

// Flag a chunk found to be an outlier after the provisional pass.
__device__ __forceinline__ void flag_late(const hqmq_packed& dst, int64_t row, int c, int ib, int rbits) {
  atomicOr(&dst.flags[row], 1u << c);
  clear_radius(reinterpret_cast<uint32_t*>(dst.codes + row * dst.row_bytes), c, ib, rbits);
}

// The undecided chunks of a head against the exact threshold, kFixupCtas CTAs per head: the listed ones, or, when the list
// overflowed, x is read again and every chunk between the two bounds settled.
constexpr int kFixupCtas = 32;
template <int DT>
__global__ void __launch_bounds__(256)
fixup_kernel(Fast32 f, hqmq_packed dst, int t_start, int ib, int rbits, int B, const uint32_t* __restrict__ sel,
             const uint32_t* __restrict__ band, const uint32_t* __restrict__ und, const uint32_t* __restrict__ gate, int und_cap) {
  if (*gate) return;                  // (the one-launch encoder redoes the call)
  const int h = blockIdx.y;
  const uint32_t n = band[h * kBandWords + 2];
  if (n == 0) return;
  const float thr = __uint_as_float(sel[h * 8 + 6]);
  if (n <= (uint32_t)und_cap) {
    const int tokens = f.pair ? 2 * f.T_new : f.T_new;
    const int64_t xs_t = f.pair ? f.xs_t / 2 : f.xs_t;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const uint32_t e = und[(int64_t)h * und_cap + i];
      const int c = e & 31;
      const int64_t bt = e >> 5;
      const int b = (int)(bt / tokens), t = (int)(bt - (int64_t)b * tokens);
      const uint2 raw = *reinterpret_cast<const uint2*>(f.x + b * f.xs_b + h * f.xs_h + (int64_t)t * xs_t + 4 * c);
      float v[4];
      v[0] = bits16_to_float(raw.x & 0xffff, DT); v[1] = bits16_to_float(raw.x >> 16, DT);
      v[2] = bits16_to_float(raw.y & 0xffff, DT); v[3] = bits16_to_float(raw.y >> 16, DT);
      if (chunk_norm(v) > thr) flag_late(dst, ((int64_t)b * f.H + h) * dst.T_cap + t_start + t, c, ib, rbits);
    }
    return;
  }
  const float thr_lo = __uint_as_float(band[h * kBandWords + 0]), thr_hi = __uint_as_float(band[h * kBandWords + 1]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l16 = lane & 15;
  for (int b = 0; b < B; ++b) {
    const uint16_t* base = f.x + b * f.xs_b + h * f.xs_h + 8 * l16;
    const int64_t row0 = ((int64_t)b * f.H + h) * dst.T_cap + t_start;
    for (int t = blockIdx.x * 16 + warp * 2 + (lane >> 4); t < f.T_new; t += gridDim.x * 16) {
      const uint4 r = *reinterpret_cast<const uint4*>(base + (int64_t)t * f.xs_t);
      float nv[2];
      norms_of_two<DT>(r, nv[0], nv[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (nv[e] > thr_lo && !(nv[e] > thr_hi) && nv[e] > thr) {
          const int c32 = 2 * l16 + e;
          if (f.pair) flag_late(dst, row0 + 2 * t + (c32 >> 4), c32 & 15, ib, rbits);
          else flag_late(dst, row0 + t, c32, ib, rbits);
        }
    }
  }
}

// Flags: one lane group per token.
__global__ void __launch_bounds__(256)
flags_kernel(EncGeom g, const void* __restrict__ x, hqmq_packed dst, int t_start, const uint32_t* __restrict__ sel) {
  const int bh = blockIdx.y;
  const int h = bh % g.H, b = bh / g.H;
  const float thr = __uint_as_float(sel[h * 8 + 6]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / g.npl, c = lane % g.npl;
  const int tok_per_iter = (blockDim.x >> 5) * g.tpw;
  for (int tb4 = blockIdx.x * tok_per_iter * 4; tb4 < g.T_new; tb4 += gridDim.x * tok_per_iter * 4) {
   float v4[4][4];
#pragma unroll
   for (int u = 0; u < 4; ++u) {   // four independent loads in flight per thread
     const int t = tb4 + u * tok_per_iter + warp * g.tpw + sub;
     v4[u][0] = v4[u][1] = v4[u][2] = v4[u][3] = 0.f;
     if (t < g.T_new && c < g.n) load_chunk(x, b * g.xs_b + h * g.xs_h + t * g.xs_t + 4 * c, g.x_dtype, v4[u]);
   }
#pragma unroll
   for (int u = 0; u < 4; ++u) {
    const int tb = tb4 + u * tok_per_iter;
    if (tb >= g.T_new) break;
    const int t = tb + warp * g.tpw + sub;
    const bool active = t < g.T_new && c < g.n;
    const float* v = v4[u];
    const bool f = active && chunk_norm(v) > thr;
    const uint32_t bal = __ballot_sync(0xffffffffu, f);
    if (f) {
      // A flagged chunk is stored in the side buffer: its radius code in the packed row becomes 0 so
      // that decoding the row contributes nothing for it.
      const int cb = g.ib + g.rbits;
      uint32_t* rowp = reinterpret_cast<uint32_t*>(dst.codes + ((int64_t)bh * dst.T_cap + t_start + t) * dst.row_bytes);
      const int lo = c * cb + g.ib, hi = (c + 1) * cb;   // bit range of the radius code
      const int w0 = lo >> 5, w1 = (hi - 1) >> 5;
      const uint32_t m0 = ~0u << (lo & 31);
      const uint32_t m1 = (hi & 31) ? ~(~0u << (hi & 31)) : ~0u;
      if (w0 == w1) atomicAnd(&rowp[w0], ~(m0 & m1));
      else { atomicAnd(&rowp[w0], ~m0); atomicAnd(&rowp[w1], ~m1); }
    }
    if (t < g.T_new && c == 0) {
      const uint32_t mask = g.npl == 32 ? 0xffffffffu : ((1u << g.npl) - 1u);
      const uint32_t word = (bal >> (sub * g.npl)) & mask;
      dst.flags[(int64_t)bh * dst.T_cap + t_start + t] = word;
    }
   }
  }
}

// Distinct flagged chunk positions of a 16-token block -> records the block owns (0 when it has none,
// or more than HQMQ_OFRAG_MAX_PER_TILE records would be needed).
__device__ __forceinline__ int ofrag_records_for(uint32_t any_c) {
  const int nd = __popc(any_c);
  const int ng = (nd + 3) >> 2;
  return ng <= HQMQ_OFRAG_MAX_PER_TILE ? ng : 0;
}

// Per (b,h), one CTA of 8 warps, one lane per 16-token block of this call: the block's flagged chunks are
// counted from its flag words and scanned into the payload offsets; with a fragment plane, also the record
// offsets (a block gets records in the call that completes it; a block whose records would pass the capacity,
// and every block after it in this call, gets none: the running total is monotone, so that is every block
// whose inclusive total exceeds the capacity).  `payload` = 0 on a call without Med3x (nothing flagged).
constexpr int kScanWarps = 8;
constexpr int kScanIters = 16;     // blocks per lane at most: 8 * 32 * 16 = 4096 blocks (64 k tokens) in one sweep
__device__ __forceinline__ void
scan_body(const hqmq_packed& dst, int t_start, int T_new, int blk0, int nblk, int payload, uint32_t* __restrict__ status) {
  __shared__ uint32_t w_tot[kScanWarps], w_ftot[kScanWarps], s_last_ok[kScanWarps];
  const int bh = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb_cap = dst.T_cap / HQMQ_OUT_BLOCK + 1;
  uint32_t* off = dst.out_off + (int64_t)bh * nb_cap;
  uint32_t* foff = dst.ofrag ? dst.ofrag_off + (int64_t)bh * nb_cap : nullptr;
  const uint32_t* fl = dst.flags + (int64_t)bh * dst.T_cap;
  uint32_t run = payload ? dst.out_count[bh] : 0u;
  uint32_t frun = foff ? foff[blk0] : 0u;
  const int t_end = t_start + T_new;
  // (no more blocks to a lane than it takes: with sixteen whatever the call, 8192 tokens were the work of one warp, 16.5 us)
  const int iters = min(kScanIters, (nblk + kScanWarps * 32 - 1) / (kScanWarps * 32)), sweep = kScanWarps * 32 * iters;
  bool full = false;       // a block of an earlier sweep did not fit the record capacity
  for (int s0 = 0; s0 < nblk; s0 += sweep) {
    // warp w owns the contiguous blocks [s0 + w * 32 * iters, ...): lane-major inside an iteration
    uint32_t c[kScanIters], fc[kScanIters];
    uint32_t wsum = 0, wfsum = 0;
#pragma unroll
    for (int it = 0; it < kScanIters; ++it) {
      const int i = s0 + (warp * iters + it) * 32 + lane, ba = blk0 + i;
      uint32_t cc = 0, any_c = 0;
      // (an iteration whose 32 blocks all lie past the call -- every one but the first in a one-token append --
      //  is skipped here and in the scan below: it would add zeros)
      if (it >= iters || i - lane >= nblk) { c[it] = fc[it] = 0u; continue; }
      if (i < nblk) {
        const int tb = ba * HQMQ_OUT_BLOCK;
#pragma unroll
        for (int q = 0; q < HQMQ_OUT_BLOCK / 4; ++q) {
          const uint4 w = *reinterpret_cast<const uint4*>(fl + tb + 4 * q);
          const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int t = tb + 4 * q + k;
            if (t >= t_start && t < t_end) cc += __popc(ww[k]);   // payload entries: tokens of this call only
            if (t < t_end) any_c |= ww[k];                          // records: every token the block holds
          }
        }
      }
      // a block gets its records in the call that completes it (all 16 tokens present), from flags and payload
      const bool complete = i < nblk && (ba + 1) * HQMQ_OUT_BLOCK <= t_end;
      c[it] = cc;
      fc[it] = foff && complete ? (uint32_t)ofrag_records_for(any_c) : 0u;
      wsum += cc; wfsum += fc[it];
    }
    wsum = __reduce_add_sync(0xffffffffu, wsum);
    wfsum = __reduce_add_sync(0xffffffffu, wfsum);
    if (lane == 0) { w_tot[warp] = wsum; w_ftot[warp] = wfsum; }
    __syncthreads();
    uint32_t base = run, fbase = frun, all = 0, fall = 0;
    for (int w = 0; w < kScanWarps; ++w) {
      if (w < warp) { base += w_tot[w]; fbase += w_ftot[w]; }
      all += w_tot[w]; fall += w_ftot[w];
    }
    uint32_t my_last_ok = frun;      // largest inclusive record total within the capacity seen by this warp
#pragma unroll
    for (int it = 0; it < kScanIters; ++it) {
      const int i = s0 + (warp * iters + it) * 32 + lane, ba = blk0 + i;
      if (it >= iters || i - lane >= nblk) continue;
      uint32_t incl = c[it], fincl = fc[it];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        const uint32_t fv = __shfl_up_sync(0xffffffffu, fincl, o);
        if (lane >= o) { incl += v; fincl += fv; }
      }
      if (payload) {
        // A block that already holds tokens from an earlier call keeps its offset.
        if (i < nblk && !(i == 0 && (t_start % HQMQ_OUT_BLOCK) != 0)) off[ba] = base + incl - c[it];
        base += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (foff) {
        fincl += fbase;
        const bool ok = !full && fincl <= (uint32_t)dst.ofrag_cap;
        fc[it] = ok ? fincl : 0xffffffffu;      // reused: the inclusive total, or "over the capacity"
        if (ok && i < nblk) my_last_ok = max(my_last_ok, fincl);
        fbase = __shfl_sync(0xffffffffu, fincl, 31);
      }
    }
    if (foff) {
      my_last_ok = __reduce_max_sync(0xffffffffu, my_last_ok);
      if (lane == 0) s_last_ok[warp] = my_last_ok;
      __syncthreads();
      uint32_t last_ok = frun;
      for (int w = 0; w < kScanWarps; ++w) last_ok = max(last_ok, s_last_ok[w]);
#pragma unroll
      for (int it = 0; it < kScanIters; ++it) {
        const int i = s0 + (warp * iters + it) * 32 + lane;
        if (it < iters && i < nblk) foff[blk0 + i + 1] = fc[it] != 0xffffffffu ? fc[it] : last_ok;
      }
      full = full || frun + fall > last_ok;   // some block of this sweep was over the capacity
      frun = last_ok;
    }
    run += all;
    __syncthreads();      // w_tot / s_last_ok are rewritten by the next sweep
  }
  if (payload && threadIdx.x == 0) {
    off[blk0 + nblk] = run;
    if (run > (uint32_t)dst.out_cap) atomicOr(&status[0], 1u);
    dst.out_count[bh] = run;
  }
}

__global__ void __launch_bounds__(kScanWarps * 32)
scan_kernel(hqmq_packed dst, int t_start, int T_new, int blk0, int nblk, int payload, uint32_t* __restrict__ status) {
  scan_body(dst, t_start, T_new, blk0, nblk, payload, status);
}

// Side planes of one 16-token block, one warp per block: the payload (original values of every flagged chunk,
// in (token, chunk) order) and, for a block that owns fragment records, the records (layout in
// include/hqmq_b200.h).  Lane l < 16 holds the flag word of token l of the block.
__device__ __forceinline__ void
side_block(const EncGeom& g, const void* __restrict__ x, const hqmq_packed& dst, int t_start, int blk0, int nblk, int bh, int i,
           int lane) {
  const int h = bh % g.H, b = bh / g.H;
  if (i >= nblk) return;
  const int ba = blk0 + i;
  const int nb_cap = dst.T_cap / HQMQ_OUT_BLOCK + 1;
  const int64_t row0 = (int64_t)bh * dst.T_cap + (int64_t)ba * HQMQ_OUT_BLOCK;
  const uint32_t fw = lane < HQMQ_OUT_BLOCK ? dst.flags[row0 + lane] : 0u;
  uint32_t any_c = __reduce_or_sync(0xffffffffu, fw);
  if (!any_c) return;
  const int64_t xbase = b * g.xs_b + h * g.xs_h;

  // ---- payload: lane pair (l, l + 16) shares token l; the pair takes the token's flagged chunks alternately ----
  uint32_t excl16;   // lanes 0..15: flagged chunks of the block's earlier tokens
  const uint32_t off0 = dst.out_off[(int64_t)bh * nb_cap + ba];
  const int esz = dst.out_dtype == HQMQ_F32 ? 4 : 2;
  unsigned char* base = reinterpret_cast<unsigned char*>(dst.out_vals) + (int64_t)bh * dst.out_cap * 4 * esz;
  {
    uint32_t incl = __popc(fw);
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if ((lane & 15) >= o) incl += v;
    }
    excl16 = incl - __popc(fw);
    const uint32_t before = __shfl_sync(0xffffffffu, excl16, lane & 15);
    uint32_t word = __shfl_sync(0xffffffffu, fw, lane & 15);
    const int t = ba * HQMQ_OUT_BLOCK + (lane & 15) - t_start;                         // token index within this call
    if (t >= 0 && t < g.T_new && word) {
      uint32_t pos = off0 + before;
      int k = 0;
      while (word) {
        const int c = __ffs(word) - 1;
        word &= word - 1;
        if ((k & 1) == (lane >> 4) && pos < (uint32_t)dst.out_cap) {
          float v[4];
          load_chunk(x, xbase + t * g.xs_t + 4 * c, g.x_dtype, v);
          if (dst.out_dtype == HQMQ_F32) {
            *reinterpret_cast<float4*>(base + (int64_t)pos * 16) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
            uint2 o;
            o.x = float_to_bits16(v[0], dst.out_dtype) | ((uint32_t)float_to_bits16(v[1], dst.out_dtype) << 16);
            o.y = float_to_bits16(v[2], dst.out_dtype) | ((uint32_t)float_to_bits16(v[3], dst.out_dtype) << 16);
            *reinterpret_cast<uint2*>(base + (int64_t)pos * 8) = o;
          }
        }
        ++pos; ++k;
      }
    }
  }

  // ---- fragment records: built from the flags and the payload, so that a block filled by several calls
  // (token-by-token appends) gets them too, in the call that completes it -------------------------------------
  if (!dst.ofrag) return;
  const uint32_t* off = dst.ofrag_off + (int64_t)bh * nb_cap;
  const uint32_t o0 = off[ba], o1 = off[ba + 1];
  if (o1 <= o0) return;
  __threadfence_block();
  __syncwarp();            // this call's payload entries of the block were written by other lanes of the warp
  const int j = lane & 3, r = lane >> 2;
  uint32_t fl[2], pre[2]; float inv[2];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    fl[nt] = __shfl_sync(0xffffffffu, fw, nt * 8 + r);
    pre[nt] = __shfl_sync(0xffffffffu, excl16, nt * 8 + r);
    inv[nt] = fl[nt] ? (float)g.qmax / load_scale(dst, row0 + nt * 8 + r) : 0.f;
  }
  for (uint32_t rec = o0; rec < o1; ++rec) {
    int cj = -1;
    uint32_t hdr = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = any_c ? __ffs(any_c) - 1 : -1;
      any_c &= any_c - 1;
      if (q == j) cj = c;
      hdr |= (uint32_t)(c & 0xff) << (8 * q);
    }
    uint32_t a[4] = {0u, 0u, 0u, 0u};
    if (cj >= 0) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        if ((fl[nt] >> cj) & 1u) {
          const uint32_t pos = off0 + pre[nt] + __popc(fl[nt] & ((1u << cj) - 1u));
          float v[4] = {0.f, 0.f, 0.f, 0.f};
          if (pos < (uint32_t)dst.out_cap) {     // (an entry dropped by an overflowing side buffer reads as 0)
            if (dst.out_dtype == HQMQ_F32) {
              const float4 f = *reinterpret_cast<const float4*>(base + (int64_t)pos * 16);
              v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            } else {
              const uint2 o = *reinterpret_cast<const uint2*>(base + (int64_t)pos * 8);
              v[0] = bits16_to_float(o.x & 0xffff, dst.out_dtype); v[1] = bits16_to_float(o.x >> 16, dst.out_dtype);
              v[2] = bits16_to_float(o.y & 0xffff, dst.out_dtype); v[3] = bits16_to_float(o.y >> 16, dst.out_dtype);
            }
          }
          const __half2 h01 = __floats2half2_rn(v[0] * inv[nt], v[1] * inv[nt]);
          const __half2 h23 = __floats2half2_rn(v[2] * inv[nt], v[3] * inv[nt]);
          a[nt] = *reinterpret_cast<const uint32_t*>(&h01);
          a[2 + nt] = *reinterpret_cast<const uint32_t*>(&h23);
        }
      }
    }
    unsigned char* recp = dst.ofrag + ((int64_t)bh * dst.ofrag_cap + rec) * HQMQ_OFRAG_BYTES;
    if (lane == 0) *reinterpret_cast<uint4*>(recp) = make_uint4(hdr, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(recp + 16 + lane * 16) = make_uint4(a[0], a[1], a[2], a[3]);
  }
}

// (grid (blocks / warps per CTA, B * H): one warp per block)
__device__ __forceinline__ void
side_body(const EncGeom& g, const void* __restrict__ x, const hqmq_packed& dst, int t_start, int blk0, int nblk) {
  side_block(g, x, dst, t_start, blk0, nblk, blockIdx.y, blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), threadIdx.x & 31);
}
__global__ void __launch_bounds__(256)
side_kernel(EncGeom g, const void* __restrict__ x, hqmq_packed dst, int t_start, int blk0, int nblk) {
  side_body(g, x, dst, t_start, blk0, nblk);
}

// The offset scan of scan_body for a call that touches at most 32 blocks of a (b, h): one warp, one lane per block, a
// single sweep.  Same results word for word (payload offsets of the blocks this call starts, record offsets of the
// blocks it completes with the capacity rule, the running totals).
constexpr int kScanSmallBlocks = 32;
__device__ __forceinline__ void
scan_small_warp(const hqmq_packed& dst, int bh, int t_start, int T_new, int blk0, int nblk, int payload,
                uint32_t* __restrict__ status, int lane) {
  const int nb_cap = dst.T_cap / HQMQ_OUT_BLOCK + 1;
  uint32_t* off = dst.out_off + (int64_t)bh * nb_cap;
  uint32_t* foff = dst.ofrag ? dst.ofrag_off + (int64_t)bh * nb_cap : nullptr;
  const uint32_t* fl = dst.flags + (int64_t)bh * dst.T_cap;
  // (the totals are read by one lane and handed round, so that the reads are done before lane 0 rewrites them)
  uint32_t run = 0u, frun = 0u;
  if (lane == 0) { run = payload ? dst.out_count[bh] : 0u; frun = foff ? foff[blk0] : 0u; }
  run = __shfl_sync(0xffffffffu, run, 0);
  frun = __shfl_sync(0xffffffffu, frun, 0);
  const int t_end = t_start + T_new;
  const int i = lane, ba = blk0 + i;
  uint32_t cc = 0, any_c = 0;
  if (i < nblk) {
    const int tb = ba * HQMQ_OUT_BLOCK;
#pragma unroll
    for (int q = 0; q < HQMQ_OUT_BLOCK / 4; ++q) {
      const uint4 w = *reinterpret_cast<const uint4*>(fl + tb + 4 * q);
      const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = tb + 4 * q + k;
        if (t >= t_start && t < t_end) cc += __popc(ww[k]);
        if (t < t_end) any_c |= ww[k];
      }
    }
  }
  const bool complete = i < nblk && (ba + 1) * HQMQ_OUT_BLOCK <= t_end;
  const uint32_t fcnt = foff && complete ? (uint32_t)ofrag_records_for(any_c) : 0u;
  uint32_t incl = cc, fincl = fcnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    const uint32_t fv = __shfl_up_sync(0xffffffffu, fincl, o);
    if (lane >= o) { incl += v; fincl += fv; }
  }
  if (payload && i < nblk && !(i == 0 && (t_start % HQMQ_OUT_BLOCK) != 0)) off[ba] = run + incl - cc;
  if (foff) {
    fincl += frun;
    const bool ok = fincl <= (uint32_t)dst.ofrag_cap;
    const uint32_t last_ok = __reduce_max_sync(0xffffffffu, ok && i < nblk ? fincl : frun);
    if (i < nblk) foff[ba + 1] = ok ? fincl : last_ok;
  }
  const uint32_t total = run + __shfl_sync(0xffffffffu, incl, 31);
  if (payload && lane == 0) {
    off[blk0 + nblk] = total;
    if (total > (uint32_t)dst.out_cap) atomicOr(&status[0], 1u);
    dst.out_count[bh] = total;
  }
}

// The same steps for one tensor or for K and V of a layer (blockIdx selects the tensor).
struct SideArgs {
  EncGeom g;
  const void* x;
  hqmq_packed dst;
  int t_start, T_new, blk0, nblk, payload;
  uint32_t* status;
};
struct SidePair { SideArgs t[2]; };
__global__ void __launch_bounds__(kScanWarps * 32) scan_pair_kernel(const SidePair p) {
  const SideArgs& a = p.t[blockIdx.y];
  if (!a.payload && !a.dst.ofrag) return;
  scan_body(a.dst, a.t_start, a.T_new, a.blk0, a.nblk, a.payload, a.status);
}
__global__ void __launch_bounds__(256) side_pair_kernel(const SidePair p) {
  const SideArgs& a = p.t[blockIdx.z];
  side_block(a.g, a.x, a.dst, a.t_start, a.blk0, a.nblk, blockIdx.y, blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), threadIdx.x & 31);
}
// Calls of at most kScanSmallBlocks blocks per (b, h): a CTA scans and writes the side planes, a warp per block.
__global__ void __launch_bounds__(kScanSmallBlocks * 32) side_small_kernel(const SidePair p, int side) {
  const SideArgs& a = p.t[blockIdx.y];
  if (!a.payload && !a.dst.ofrag) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) scan_small_warp(a.dst, blockIdx.x, a.t_start, a.T_new, a.blk0, a.nblk, a.payload, a.status, lane);
  if (!side) return;
  __syncthreads();
  side_block(a.g, a.x, a.dst, a.t_start, a.blk0, a.nblk, blockIdx.x, warp, lane);
}

// The K + V append of a layer in ONE launch, grid (H, 2): blockIdx.y = 0 the K tensor, 1 the V tensor (same batch,
// heads, tokens and head dim).  After the head's codes, scales and flags, the same CTA scans the offsets of its batch
// entries (a warp per entry) and writes their side planes (a warp per block) -- what scan_kernel and side_kernel do in
// two more launches of a single-tensor call.  For calls that touch at most kScanSmallBlocks blocks per (b, h).
// The status words are cleared by the host (a memset ahead of the launch): a CTA may report an overflow before
// another CTA has started.
__global__ void __launch_bounds__(kSmallThreads) append_pair_kernel(SmallPair p) {
  const SmallArgs& a = p.t[blockIdx.y];
  encode_small_body<false>(a.g, a.x, a.qs, a.dst, a.t_start, p.maps, a.joint, a.lut, a.C, a.med_out, a.quantile);
  if (!a.scan) return;
  __syncthreads();          // the head's flag words and scales are in global memory for the other warps of the CTA
  const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < a.g.B; b += (int)(blockDim.x >> 5))
    scan_small_warp(a.dst, b * a.g.H + h, a.t_start, a.g.T_new, a.blk0, a.nblk, a.payload, a.status, lane);
  if (!a.side) return;
  __syncthreads();          // ... and so are the offsets
  for (int w = warp; w < a.g.B * a.nblk; w += (int)(blockDim.x >> 5)) {
    const int b = w / a.nblk, i = w - b * a.nblk;
    side_block(a.g, a.x, a.dst, a.t_start, a.blk0, a.nblk, b * a.g.H + h, i, lane);
  }
}

#include "encode_append.cuh"

// ---- look-up table construction ---------------------------------------------------------------------
// Geometry (the same for every head): per (cx, cy) column the stored cz range = the cells whose grown box meets
// the octahedron |w1| + |w2| + |w3| <= 1, and the index of the column's first cell.
__device__ __forceinline__ float min_abs_over(float lo, float hi) { return (lo <= 0.f && hi >= 0.f) ? 0.f : fminf(fabsf(lo), fabsf(hi)); }
__global__ void __launch_bounds__(1024) lut_rows_kernel(int n, uint32_t* __restrict__ ghdr, uint32_t* __restrict__ rows) {
  __shared__ uint32_t s_cnt[kLutRows], s_min[kLutRows];
  const float step = 2.0f / (float)n;
  for (int col = threadIdx.x; col < n * n; col += blockDim.x) {
    const int cx = col / n, cy = col - cx * n;
    const float m1 = min_abs_over(cx * step - 1.f - kLutBoxEps, (cx + 1) * step - 1.f + kLutBoxEps);
    const float m2 = min_abs_over(cy * step - 1.f - kLutBoxEps, (cy + 1) * step - 1.f + kLutBoxEps);
    const float lim = 1.f + kLutBoxEps - m1 - m2;
    int zmin = n, zmax = -1;
    for (int cz = 0; cz < n; ++cz) {
      const float m3 = min_abs_over(cz * step - 1.f - kLutBoxEps, (cz + 1) * step - 1.f + kLutBoxEps);
      if (m3 <= lim) { zmin = min(zmin, cz); zmax = max(zmax, cz); }
    }
    s_cnt[col] = zmax >= zmin ? (uint32_t)(zmax - zmin + 1) : 0u;
    s_min[col] = zmax >= zmin ? (uint32_t)zmin : 0u;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0, all = 0;
    for (int col = 0; col < n * n; ++col) all += s_cnt[col];
    for (int col = 0; col < n * n; ++col) {
      rows[col] = s_cnt[col] ? run | (s_min[col] << 16) | ((s_cnt[col] - 1u) << 24) : all | (kLutNoCells << 16);
      run += s_cnt[col];
    }
    ghdr[0] = (uint32_t)n; ghdr[1] = all + 1u; ghdr[2] = ghdr[3] = 0u;
  }
}

// One CTA per ((cx, cy) column, head), walking the column's stored cells.  tmp: [H][kLutCellCap][kLutMaxList] uint16
// candidate lists (ascending), cnt: [H][kLutCellCap] list lengths (0 = too long: exhaustive search in that cell).
__global__ void __launch_bounds__(128)
lut_cells_kernel(const float* __restrict__ joint_all, int S, int n, const uint32_t* __restrict__ rows,
                 uint16_t* __restrict__ tmp, uint32_t* __restrict__ cnt) {
  __shared__ float s_best[4];
  __shared__ int s_bk[4];
  __shared__ int s_n;
  __shared__ uint16_t s_list[kLutMaxList];
  __shared__ float4 s_cw[kLutMaxList];
  __shared__ unsigned char s_drop[kLutMaxList];
  const int col = blockIdx.x, h = blockIdx.y, K = 24 * S;
  const float4* joint = reinterpret_cast<const float4*>(joint_all) + (int64_t)h * K;
  const uint32_t row = rows[col];
  const int zmin = (int)((row >> 16) & 255u), zcnt = (uint32_t)zmin == kLutNoCells ? 0 : (int)(row >> 24) + 1, base = (int)(row & 0xffffu);
  const int cx = col / n, cy = col - cx * n;
  const float step = 2.0f / (float)n;
  const float w1 = (cx + 0.5f) * step - 1.f, w2 = (cy + 0.5f) * step - 1.f;
  const float hh = 0.5f * step + kLutBoxEps;
  for (int zc = 0; zc < zcnt; ++zc) {
    const int cell = base + zc;
    const float w3 = (zmin + zc + 0.5f) * step - 1.f;
    // winner at the centre of the cell
    float best = -1e30f; int bk = 0;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      const float4 c = joint[k];
      const float sim = c.x + w1 * c.y + w2 * c.z + w3 * c.w;
      if (sim > best) { best = sim; bk = k; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
      if (ob > best || (ob == best && ok < bk)) { best = ob; bk = ok; }
    }
    if ((threadIdx.x & 31) == 0) { s_best[threadIdx.x >> 5] = best; s_bk[threadIdx.x >> 5] = bk; }
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    best = s_best[0]; bk = s_bk[0];
    for (int i = 1; i < 4; ++i)
      if (s_best[i] > best || (s_best[i] == best && s_bk[i] < bk)) { best = s_best[i]; bk = s_bk[i]; }
    const float4 cs = joint[bk];
    // every codeword that is not beaten by the centre's winner over the whole (grown) box
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      const float4 c = joint[k];
      const float d0 = c.x - cs.x, d1 = c.y - cs.y, d2 = c.z - cs.z, d3 = c.w - cs.w;
      const float ub = d0 + d1 * w1 + d2 * w2 + d3 * w3 + hh * (fabsf(d1) + fabsf(d2) + fabsf(d3));
      if (ub >= -kLutMargin) {
        const int pos = atomicAdd(&s_n, 1);
        if (pos < kLutMaxList) s_list[pos] = (uint16_t)k;
      }
    }
    __syncthreads();
    int m = s_n;
    if (m > kLutMaxList) m = 0;         // too long: this cell falls back to the exhaustive search
    if (threadIdx.x == 0) {
      for (int i = 1; i < m; ++i) {     // ascending order makes the table reproducible
        const uint16_t v = s_list[i];
        int q = i - 1;
        while (q >= 0 && s_list[q] > v) { s_list[q + 1] = s_list[q]; --q; }
        s_list[q + 1] = v;
      }
    }
    __syncthreads();
    if (threadIdx.x < m) s_cw[threadIdx.x] = joint[s_list[threadIdx.x]];
    __syncthreads();
    // second filter: drop a codeword that loses to some OTHER listed codeword over the whole box
    if (threadIdx.x < m) {
      const float4 ci = s_cw[threadIdx.x];
      bool drop = false;
      for (int q = 0; q < m && !drop; ++q) {
        if (q == threadIdx.x) continue;
        const float4 cq = s_cw[q];
        const float d0 = ci.x - cq.x, d1 = ci.y - cq.y, d2 = ci.z - cq.z, d3 = ci.w - cq.w;
        const float ub = d0 + d1 * w1 + d2 * w2 + d3 * w3 + hh * (fabsf(d1) + fabsf(d2) + fabsf(d3));
        drop = ub < -kLutMargin;
      }
      s_drop[threadIdx.x] = drop ? 1 : 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint16_t* dst = tmp + ((int64_t)h * kLutCellCap + cell) * kLutMaxList;
      int q = 0;
      for (int i = 0; i < m; ++i)
        if (!s_drop[i]) dst[q++] = s_list[i];
      cnt[(int64_t)h * kLutCellCap + cell] = (uint32_t)q;
    }
    __syncthreads();
  }
}

// Per head: cell words and the padded candidate lists.  A list of one needs no entry; longer ones are padded to a
// multiple of four with their last codeword.  Bit 15: on the first entry of a list of up to four, on the last codeword of a longer one.
__global__ void __launch_bounds__(1024)
lut_pack_kernel(const uint16_t* __restrict__ tmp, const uint32_t* __restrict__ cnt, unsigned char* __restrict__ lut, int S) {
  __shared__ uint32_t s_sum[1024];
  const int h = blockIdx.x;
  const uint32_t* gh = reinterpret_cast<const uint32_t*>(lut);
  const int n_cells = (int)gh[1];
  unsigned char* head = lut + kLutOffHeads + (size_t)h * kLutHeadBytes;
  uint16_t* cells = reinterpret_cast<uint16_t*>(head + 16);
  uint16_t* cands = reinterpret_cast<uint16_t*>(head + 16 + (size_t)kLutCellCap * 2);
  const int per = (n_cells + 1023) / 1024;
  const int c0 = threadIdx.x * per, c1 = min(n_cells, c0 + per);
  auto length = [&](int c) { return c == n_cells - 1 ? 0u : cnt[(int64_t)h * kLutCellCap + c]; };      // (the last: of rows without cells)
  uint32_t tot = 0;
  for (int c = c0; c < c1; ++c) {
    const uint32_t m = length(c);
    tot += m > 1 ? (m + 3u) & ~3u : 0u;
  }
  s_sum[threadIdx.x] = tot;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const uint32_t v = threadIdx.x >= o ? s_sum[threadIdx.x - o] : 0;
    __syncthreads();
    s_sum[threadIdx.x] += v;
    __syncthreads();
  }
  const uint32_t total = s_sum[1023];
  const bool valid = total <= (uint32_t)kLutCandCap && n_cells <= kLutCellCap && 24 * S < 32768;
  if (threadIdx.x == 0) {
    uint32_t* hh = reinterpret_cast<uint32_t*>(head);
    hh[0] = valid ? total : 0u; hh[1] = valid ? 1u : 0u; hh[2] = hh[3] = 0u;
  }
  if (!valid) return;
  uint32_t run = s_sum[threadIdx.x] - tot;
  for (int c = c0; c < c1; ++c) {
    const uint32_t m = length(c);
    const uint16_t* src = tmp + ((int64_t)h * kLutCellCap + c) * kLutMaxList;
    if (m == 0) cells[c] = 0xffffu;
    else if (m == 1) cells[c] = (uint16_t)(0x8000u | src[0]);
    else {
      const uint32_t pm = (m + 3u) & ~3u;
      cells[c] = (uint16_t)(run >> 2);
      for (uint32_t i = 0; i < pm; ++i) {
        uint16_t v = src[i < m ? i : m - 1];
        if (i == (m <= 4 ? 0u : m - 1)) v |= 0x8000u;
        cands[run + i] = v;
      }
      run += pm;
    }
  }
}

// (unit g) * (primary p) for all 24 units: the reference primary of the product
struct RefMul24 { uint8_t v[24][24]; };
RefMul24 make_mul24() {
  auto prim = [](int p, double v[4]) {
    for (int i = 0; i < 4; ++i) v[i] = 0;
    if (p < 8) v[p >> 1] = (p & 1) ? -1.0 : 1.0;
    else for (int i = 0; i < 4; ++i) v[i] = (((p - 8) >> (3 - i)) & 1) ? -0.5 : 0.5;
  };
  RefMul24 m;
  for (int g = 0; g < 24; ++g)
    for (int p = 0; p < 24; ++p) {
      double a[4], b[4], c[4];
      prim(g, a); prim(p, b);
      c[0] = a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3];
      c[1] = a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2];
      c[2] = a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1];
      c[3] = a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0];
      int ref = 0;
      for (int q = 0; q < 24; ++q) {
        double e[4];
        prim(q, e);
        double dd = 0;
        for (int i = 0; i < 4; ++i) dd += (e[i] - c[i]) * (e[i] - c[i]);
        if (dd < 1e-12) ref = q;
      }
      m.v[g][p] = (uint8_t)ref;
    }
  return m;
}
// What a codebook of S secondaries calls the products (see Mul24).
Mul24Both mul24_both(int S) {
  static const RefMul24 m = make_mul24();
  Mul24Both b;
  for (int g = 0; g < 24; ++g)
    for (int p = 0; p < 24; ++p) {
      const int ref = m.v[g][p], au = index_maps().ref_to_native[ref];
      b.native.v[g][p] = (uint16_t)((((au >> 3) * S) << 3) | (au & 7));
      b.ref.v[g][p] = (uint16_t)(ref * S);
    }
  return b;
}

inline size_t lut_bytes(int H) { return kLutOffHeads + (size_t)H * kLutHeadBytes + sizeof(Mul24Both); }   // (+ the index tables)
inline size_t lut_ws_bytes(int H) { return (size_t)H * kLutCellCap * 4 + (size_t)H * kLutCellCap * kLutMaxList * 2; }
// shared memory a main-pass kernel can give to a table next to its other arrays (fp32 joint table, histograms, rows)
inline size_t lut_smem_budget(int S) { return (size_t)226 * 1024 - (size_t)24 * S * 16 - (size_t)S * 16 - 3 * kHistBins * 4 - 4096; }

// Geometry of the main pass for the common case (d_head 128, 16-bit input): tokens per CTA, CTAs (one per SM).
struct MainGrid { int64_t per; int ctas; };
static MainGrid main_grid(int T_new, int B, int H) {
  MainGrid m;
  const int64_t total = (int64_t)T_new * B * H;
  m.per = (((total + 147) / 148 + kEnc32Warps - 1) / kEnc32Warps) * kEnc32Warps;
  m.ctas = (int)((total + m.per - 1) / m.per);
  return m;
}
// d_head 64 as pairs of tokens (see EncGeom): the call's geometry must allow it, and a token's row must be whole
// words without padding (16-bit fields; rows of 13- and 19-bit fields are padded, so two of them are not one longer row).
static bool pair16_of(const hqmq_encode_args& a) {
  return a.dst.n_chunks == 16 && (16 * (idx_bits_for(a.dst.S) + a.dst.radius_bits)) % 32 == 0 && is_half_dtype(a.x_dtype) && a.x_stride[2] == 64 && a.T_new >= 2 && a.T_new % 2 == 0 &&
         a.t_start % 2 == 0;
}
// The bracket pass pays when the sample predicts well: the statistic's sampling error falls with the square root of
// the sampled norms per head (a 1/32 sample of B * T_new tokens, 32 norms each), so the bracket's half-width is
// 3 / sqrt(norms) (about six standard errors of a median), at least 0.2 % and at most 1.2 %; calls too small for that,
// and quantiles out in the tails (few norms nearby: a much larger error), take the one-launch encoder.
// 65536 tokens are where 1.2 % still holds six standard errors.  One read / one launch, us a tensor, s96, 8 heads of 128 with some
// flagged: 65536 tokens a head 328 / 392, 98304 436 / 570, 131072 535 / 749 (s24, none flagged: 65536 304 / 351; four heads, s192:
// 331 / 353; heads of 64: 131072 326 / 432).  Below the line the one read is the shorter by little for 8 heads (32768: 201 / 208, 49152:
// 272 / 306) and the longer for four (230 / 223) and at 16384 (139 / 125); its bracket would hold four standard errors, three at 16384.
constexpr int64_t kBracketMinTokens = 65536;     // B * T_new per head (of 32 chunks each)
static bool bracket_wanted(const hqmq_encode_args& a) {
  const bool pair = pair16_of(a);
  const int T32 = pair ? a.T_new / 2 : a.T_new;
  return a.median_mult > 0.f && !a.med_in && (a.dst.n_chunks == 32 || pair) && is_half_dtype(a.x_dtype) &&
         (int64_t)a.dst.B * T32 >= kBracketMinTokens && T32 >= 1024 &&
         (a.quantile == 0.f || (a.quantile >= 0.25f && a.quantile <= 0.75f));
}

struct WsPlan {
  size_t status, hist, sel, hist_s, sel_s, tickets, gate, bp, histA, histB, band, und, sel_b, rcnt, rlist, zero_bytes, total;
  int blk0, nblk, rcap, und_cap;
};
WsPlan plan_ws(const hqmq_encode_args& a) {
  WsPlan w = {};
  const int H = a.dst.H;
  w.blk0 = a.t_start / HQMQ_OUT_BLOCK;
  w.nblk = a.T_new > 0 ? (a.t_start + a.T_new - 1) / HQMQ_OUT_BLOCK - w.blk0 + 1 : 0;
  size_t o = 0;
  w.status = o; o += 4;
  w.hist = o; o += (size_t)H * 3 * 2 * kHistBins;
  w.sel = o; o += (size_t)H * 8;
  w.zero_bytes = o * sizeof(uint32_t);
  if (bracket_wanted(a)) {
    const int T32 = pair16_of(a) ? a.T_new / 2 : a.T_new;
    const MainGrid mg = main_grid(T32, a.dst.B, H);
    const int regions = mg.ctas + H - 1;
    w.rcap = (int)(mg.per * 32 / 16);                  // a sixteenth of a CTA's chunks (the range holds about 2 %)
    w.hist_s = o; o += (size_t)H * 3 * 2 * kHistBins;   // the sample's histograms (two levels)
    w.sel_s = o; o += (size_t)H * 8;
    w.tickets = o; o += ((size_t)H * 2 + 3) & ~(size_t)3;
    w.gate = o; o += 4;
    w.bp = o; o += (size_t)H * kBpWords;
    w.histA = o; o += (size_t)H * kHistBins;
    w.histB = o; o += (size_t)H * 2 * kHistBins;
    w.band = o; o += (size_t)H * kBandWords;
    w.sel_b = o; o += (size_t)H * 8;
    w.rcnt = o; o += (size_t)regions;
    w.zero_bytes = o * sizeof(uint32_t);              // everything up to here starts at zero; the lists need not
    // (a few per mille of the chunks of a head with many outliers fall inside the bracket)
    const int64_t per_head = (int64_t)a.dst.B * T32 * 32;
    w.und_cap = (int)(per_head / 256 > kUndCap ? (per_head / 256 < (1 << 20) ? per_head / 256 : (1 << 20)) : kUndCap);
    w.und = o; o += (size_t)H * w.und_cap;
    w.rlist = o; o += (size_t)regions * w.rcap;
  }
  w.total = o * sizeof(uint32_t);
  return w;
}

}  // namespace

}  // namespace hqmq

using namespace hqmq;

static int validate_encode(const hqmq_encode_args* a) {
  if (!a || a->struct_size != sizeof(hqmq_encode_args)) return HQMQ_ERR_ARG;
  if ((!a->x && a->T_new != 0) || !a->qs || !a->joint) return HQMQ_ERR_ARG;   // an empty input has no address
  if (!is_float_dtype(a->x_dtype)) return HQMQ_ERR_DTYPE;
  const bool med = a->median_mult > 0.f;
  int rc = check_packed(a->dst, med);
  if (rc) return rc;
  if (a->T_new < 0 || a->t_start < 0) return HQMQ_ERR_SHAPE;
  if (!(a->quantile >= 0.f && a->quantile < 1.f)) return HQMQ_ERR_ARG;
  if ((int64_t)a->t_start + a->T_new > a->dst.T_cap) return HQMQ_ERR_CAPACITY;
  const int align = a->x_dtype == HQMQ_F32 ? 16 : 8;
  if ((uintptr_t)a->x & (align - 1)) return HQMQ_ERR_ALIGN;
  for (int i = 0; i < 3; ++i)
    if (a->x_stride[i] % 4) return HQMQ_ERR_ALIGN;
  if (((uintptr_t)a->qs & 15) || ((uintptr_t)a->joint & 15)) return HQMQ_ERR_ALIGN;
  return HQMQ_OK;
}

extern "C" size_t hqmq_encode_lut_bytes(int H, int S) {
  if (H < 1 || S < 1 || 24 * S > 65536) return 0;
  return lut_bytes(H);
}
extern "C" size_t hqmq_encode_lut_workspace_bytes(int H, int S) {
  if (H < 1 || S < 1 || 24 * S > 65536) return 0;
  return lut_ws_bytes(H);
}
// Largest per-head candidate total of a built table, its grid, and whether every head is valid (synchronises).
static int lut_read(const void* lut, int H, cudaStream_t st, int& n, int& n_cells, int& max_total, bool& valid) {
  uint32_t gh[4];
  HQMQ_CHECK_CUDA(cudaMemcpyAsync(gh, lut, 16, cudaMemcpyDeviceToHost, st));
  HQMQ_CHECK_CUDA(cudaStreamSynchronize(st));
  n = (int)gh[0]; n_cells = (int)gh[1];
  max_total = 0; valid = n >= 2 && n <= kLutNMax && n_cells <= kLutCellCap;
  for (int h = 0; h < H && valid; ++h) {
    uint32_t v[2];
    HQMQ_CHECK_CUDA(cudaMemcpyAsync(v, reinterpret_cast<const unsigned char*>(lut) + kLutOffHeads + (size_t)h * kLutHeadBytes, 8,
                                    cudaMemcpyDeviceToHost, st));
    HQMQ_CHECK_CUDA(cudaStreamSynchronize(st));
    if (v[1] != 1u) valid = false;
    if ((int)v[0] > max_total) max_total = (int)v[0];
  }
  return HQMQ_OK;
}
extern "C" int hqmq_encode_lut_build(const float* joint, int H, int S, void* lut, size_t lut_nbytes, void* workspace,
                                     size_t ws_nbytes, void* stream) {
  if (!joint || !lut || !workspace) return HQMQ_ERR_ARG;
  if (H < 1 || S < 1 || 24 * S > 65536) return HQMQ_ERR_SHAPE;
  if (lut_nbytes < lut_bytes(H) || ws_nbytes < lut_ws_bytes(H)) return HQMQ_ERR_WORKSPACE;
  if (((uintptr_t)joint & 15) || ((uintptr_t)lut & 15) || ((uintptr_t)workspace & 15)) return HQMQ_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* L = reinterpret_cast<unsigned char*>(lut);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(workspace);
  uint16_t* tmp = reinterpret_cast<uint16_t*>(cnt + (size_t)H * kLutCellCap);
  // the index tables of the fold units
  // (pageable memory: the copy has left it when the call returns)
  const Mul24Both products = mul24_both(S);
  HQMQ_CHECK_CUDA(cudaMemcpyAsync(L + kLutOffHeads + (size_t)H * kLutHeadBytes, &products, sizeof(products), cudaMemcpyHostToDevice, st));
  // the finest grid whose tables fit the encoder's shared memory next to this codebook
  for (int n = kLutNMax; n >= 16; n -= 4) {
    lut_rows_kernel<<<1, 1024, 0, st>>>(n, reinterpret_cast<uint32_t*>(L), reinterpret_cast<uint32_t*>(L + kLutOffRows));
    lut_cells_kernel<<<dim3(n * n, H), 128, 0, st>>>(joint, S, n, reinterpret_cast<const uint32_t*>(L + kLutOffRows), tmp, cnt);
    lut_pack_kernel<<<H, 1024, 0, st>>>(tmp, cnt, L, S);
    HQMQ_LAUNCH_CHECK();
    int nn, n_cells, max_total; bool valid;
    const int rc = lut_read(lut, H, st, nn, n_cells, max_total, valid);
    if (rc) return rc;
    if (valid && lut_smem_bytes(nn, n_cells, max_total) <= lut_smem_budget(S)) return HQMQ_OK;
    if (24 * S >= 32768) break;          // codeword ids need 15 bits: no table for this codebook
  }
  // no grid fits: mark every head invalid (the encoder then searches exhaustively)
  for (int h = 0; h < H; ++h) HQMQ_CHECK_CUDA(cudaMemsetAsync(L + kLutOffHeads + (size_t)h * kLutHeadBytes, 0, 16, st));
  return HQMQ_OK;
}
extern "C" int hqmq_encode_lut_footprint(const void* lut, int H, int* footprint, void* stream) {
  if (!lut || !footprint || H < 1) return HQMQ_ERR_ARG;
  int n, n_cells, max_total; bool valid;
  const int rc = lut_read(lut, H, (cudaStream_t)stream, n, n_cells, max_total, valid);
  if (rc) return rc;
  *footprint = valid ? (int)lut_smem_bytes(n, n_cells, max_total) : -1;
  return HQMQ_OK;
}

// ---- Med3x median of a head whose batch entries live on several GPUs ---------------------------------------
// State: [H][3 levels][2 queries][kHistBins] histograms, then [H][8] select words (the layout select_kernel uses).
namespace hqmq {
namespace {
inline size_t med3x_state_words(int H) { return (size_t)H * 3 * 2 * kHistBins + (size_t)H * 8; }

__global__ void thr_from_median_kernel(const float* __restrict__ med_in, float C, int H, uint32_t* __restrict__ sel,
                                       float* __restrict__ med_out) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= H) return;
  const float med = med_in[h];
  sel[h * 8 + 6] = __float_as_uint(__fmul_rn(med, C));   // thr = med * C in fp32, like the local select
  sel[h * 8 + 7] = __float_as_uint(med);
  if (med_out) med_out[h] = med;
}
}  // namespace
}  // namespace hqmq
using namespace hqmq;

extern "C" size_t hqmq_med3x_state_bytes(int H) { return H < 1 ? 0 : med3x_state_words(H) * 4; }

extern "C" int hqmq_med3x_hist(const hqmq_encode_args* a, int level, void* state, size_t state_bytes, void* stream) {
  int rc = validate_encode(a);
  if (rc) return rc;
  if (level < 0 || level > 2) return HQMQ_ERR_ARG;
  const hqmq_packed& d = a->dst;
  if (!state || state_bytes < med3x_state_words(d.H) * 4) return HQMQ_ERR_WORKSPACE;
  if ((uintptr_t)state & 15) return HQMQ_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t* hist = reinterpret_cast<uint32_t*>(state);
  uint32_t* sel = hist + (size_t)d.H * 3 * 2 * kHistBins;
  if (level == 0) HQMQ_CHECK_CUDA(cudaMemsetAsync(state, 0, med3x_state_words(d.H) * 4, st));
  if (a->T_new == 0) return HQMQ_OK;     // this GPU holds none of the head's tokens: its histograms stay zero
  EncGeom g;
  g.B = d.B; g.H = d.H; g.T_new = a->T_new; g.n = d.n_chunks;
  g.npl = 1; while (g.npl < g.n) g.npl <<= 1;
  g.tpw = 32 / g.npl;
  g.S = d.S; g.ib = idx_bits_for(d.S); g.rbits = d.radius_bits; g.qmax = (1 << d.radius_bits) - 1;
  g.x_dtype = a->x_dtype;
  g.xs_b = a->x_stride[0]; g.xs_h = a->x_stride[1]; g.xs_t = a->x_stride[2];
  const int bh_count = d.B * d.H;
  const int64_t per_bh = (int64_t)a->T_new * d.n_chunks;
  int hb = (148 * 16 + bh_count - 1) / bh_count;
  const int hb_max = (int)((per_bh + 256 * 16 - 1) / (256 * 16));
  if (hb > hb_max) hb = hb_max;
  if (hb < 1) hb = 1;
  hist_kernel<<<dim3(hb, bh_count), 256, 0, st>>>(g, a->x, hist, sel, level);
  HQMQ_LAUNCH_CHECK();
  return HQMQ_OK;
}

extern "C" int hqmq_med3x_select(int H, int level, uint64_t n_total, float median_mult, void* state, size_t state_bytes,
                                 float* med_out, void* stream) {
  if (H < 1 || level < 0 || level > 2 || n_total < 1 || !(median_mult > 0.f)) return HQMQ_ERR_ARG;
  if (!state || state_bytes < med3x_state_words(H) * 4) return HQMQ_ERR_WORKSPACE;
  if ((uintptr_t)state & 15) return HQMQ_ERR_ALIGN;
  uint32_t* hist = reinterpret_cast<uint32_t*>(state);
  uint32_t* sel = hist + (size_t)H * 3 * 2 * kHistBins;
  select_kernel<<<H, 256, 0, (cudaStream_t)stream>>>(hist, sel, level, n_total, median_mult, level == 2 ? med_out : nullptr, 0.f);
  HQMQ_LAUNCH_CHECK();
  return HQMQ_OK;
}

extern "C" size_t hqmq_encode_workspace_bytes(const hqmq_encode_args* a) {
  if (validate_encode(a) != HQMQ_OK) return 0;
  return plan_ws(*a).total;
}

static EncGeom geom_of(const hqmq_encode_args* a) {
  const hqmq_packed& d = a->dst;
  EncGeom g;
  g.B = d.B; g.H = d.H; g.T_new = a->T_new; g.n = d.n_chunks;
  g.npl = 1; while (g.npl < g.n) g.npl <<= 1;
  g.tpw = 32 / g.npl;
  g.S = d.S; g.ib = idx_bits_for(d.S); g.rbits = d.radius_bits; g.qmax = (1 << d.radius_bits) - 1;
  g.x_dtype = a->x_dtype;
  g.xs_b = a->x_stride[0]; g.xs_h = a->x_stride[1]; g.xs_t = a->x_stride[2];
  return g;
}

// Small calls (decode-time appends): one kernel per head does main pass, median and flags at once.
static bool small_call(const hqmq_encode_args* a) {
  const bool ext_med = a->median_mult > 0.f && a->med_in != nullptr;   // the median comes from the caller
  const int64_t tok = (int64_t)a->dst.B * a->T_new;
  return !ext_med && tok * a->dst.n_chunks <= kSmallMax && tok <= kSmallTok;
}

static int fill_small(const hqmq_encode_args* a, const WsPlan& wp, uint32_t* ws, SmallArgs& sa) {
  const hqmq_packed& d = a->dst;
  const bool med = a->median_mult > 0.f;
  const bool lut_ok = a->search == 0 && a->lut != nullptr && a->lut_footprint >= 0;
  sa.out = nullptr; sa.n_flagged = nullptr;
  if (lut_ok && ((uintptr_t)a->lut & 15)) return HQMQ_ERR_ALIGN;
  const unsigned char* lut_b = reinterpret_cast<const unsigned char*>(a->lut);
  sa.g = geom_of(a);
  sa.x = a->x; sa.qs = a->qs; sa.dst = d; sa.t_start = a->t_start; sa.joint = a->joint;
  sa.lut = lut_ok ? lut_b : nullptr;
  sa.C = a->median_mult; sa.med_out = a->med_out; sa.quantile = a->quantile;
  sa.status = ws + wp.status;
  sa.blk0 = wp.blk0; sa.nblk = wp.nblk;
  sa.scan = (med || d.ofrag) ? 1 : 0; sa.payload = med ? 1 : 0; sa.side = med ? 1 : 0;
  return HQMQ_OK;
}

// The one-launch encoder: whether a call takes it, and its launch.
static int sm_count() {
  static std::atomic<int> cached{0};
  int n = cached.load(std::memory_order_relaxed);
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    cached.store(n, std::memory_order_relaxed);
  }
  return n;
}
// Shared-memory bytes of the largest head's table, from hqmq_encode_lut_footprint (0 = unknown: the largest a table can be).
static size_t lut_foot_of(const hqmq_encode_args* a) {
  return a->lut_footprint > 0 ? ((size_t)a->lut_footprint + 15) & ~(size_t)15 : lut_smem_bytes(kLutNMax, kLutCellCap, kLutCandCap);
}
static bool fused_call(const hqmq_encode_args* a) {
  const hqmq_packed& d = a->dst;
  const int ib = idx_bits_for(d.S), rb = d.radius_bits;
  // (two 64-wide tokens per warp need rows of whole words, which 16-bit fields give)
  const bool geom = d.n_chunks == 32 || (d.n_chunks == 16 && ib + rb == 16);
  if (!geom || ib < 1 || ib + rb > kMaxRowWords || !is_half_dtype(a->x_dtype) || a->search != 0 || !a->lut || a->lut_footprint <= 0 || ((uintptr_t)a->lut & 15)) return false;
  if ((uint64_t)d.B * a->T_new * d.n_chunks >= ((uint64_t)1 << 32)) return false;
  return fused_smem_bytes(d.S, lut_foot_of(a)) <= (size_t)226 * 1024;
}
// Calls for the one-read main pass: token rows on 16-byte boundaries, and the one-launch encoder able to take over where the
// prediction fails.
static bool common_layout(const hqmq_encode_args* a) {
  const int ib = idx_bits_for(a->dst.S), rb = a->dst.radius_bits;
  return (ib == 10 && rb == 3) || (ib == 12 && rb == 4) || (ib == 13 && rb == 6);
}
static bool bracket_call(const hqmq_encode_args* a) {
  return bracket_wanted(*a) && common_layout(a) && fused_call(a) && ((uintptr_t)a->x & 15) == 0 && a->x_stride[0] % 8 == 0 && a->x_stride[1] % 8 == 0 &&
         a->x_stride[2] % 8 == 0;
}
// Whether the dense tensor of a call (16-bit values) shares memory with what the call reads of x.
static bool overlaps_x(const hqmq_encode_args* a, const void* out) {
  const hqmq_packed& d = a->dst;
  const int64_t last[3] = {d.B - 1, d.H - 1, (int64_t)a->T_new - 1};
  int64_t lo = 0, hi = 4 * (int64_t)d.n_chunks;
  for (int i = 0; i < 3; ++i) (a->x_stride[i] < 0 ? lo : hi) += last[i] * a->x_stride[i];
  const uintptr_t x = (uintptr_t)a->x, o = (uintptr_t)out;
  return o < x + 2 * hi && x + 2 * lo < o + 2 * ((int64_t)d.B * d.H * a->T_new * d.n_chunks * 4);
}
static void fill_fused(const hqmq_encode_args* a, int tensors, uint32_t* status, uint32_t* hist, uint32_t* bars, void* out, uint32_t* n_flagged,
                       FusedArgs& f) {
  const hqmq_packed& d = a->dst;
  f.g = geom_of(a);
  f.x = reinterpret_cast<const uint16_t*>(a->x); f.qs = a->qs; f.joint = a->joint;
  f.lut = reinterpret_cast<const unsigned char*>(a->lut);
  f.dst = d; f.t_start = a->t_start; f.out = reinterpret_cast<uint16_t*>(out); f.n_flagged = n_flagged;
  f.C = a->median_mult; f.quantile = a->quantile; f.med_in = a->med_in; f.med_out = a->med_out;
  f.hist = hist; f.bars = bars; f.status = status; f.gate = nullptr;
  // (the near-ties of the generic kernels, which divide with the rounded reciprocal, are kept where those used to run: other
  //  field widths, 64-wide tokens outside the paired geometry)
  f.rcp_rn = !common_layout(a) || (d.n_chunks == 16 && !(pair16_of(*a) && ((uintptr_t)a->x & 15) == 0 && a->x_stride[0] % 8 == 0 && a->x_stride[1] % 8 == 0));
  f.early = out && overlaps_x(a, out) ? 0 : kFusedEarly;
  // one CTA per SM in all, no fewer than a round of its warps each
  const int64_t W = (int64_t)d.B * (d.n_chunks == 16 ? (a->T_new + 1) / 2 : a->T_new);
  int64_t cph = sm_count() / (tensors * d.H);
  if (cph < 1) cph = 1;                 // (a CTA per head meets nobody: any number of them)
  if (cph > (W + kEnc32Warps - 1) / kEnc32Warps) cph = (W + kEnc32Warps - 1) / kEnc32Warps;
  f.per = (int)((W + cph - 1) / cph);
  f.cph = (int)((W + f.per - 1) / f.per);
  const uint32_t T2 = (uint32_t)(W / d.B);
  f.t2_mul = 0u; f.t2_sh = 0;
  if (T2 > 1) {
    int s = 1;
    while (((uint64_t)1 << s) < T2) ++s;
    f.t2_mul = (uint32_t)(((uint64_t)1 << (31 + s)) / T2 + 1); f.t2_sh = s - 1;
  }
}
// `tensors` of one geometry, element type and codebook size, each with its own threshold or all without.
static int launch_fused(const FusedPair& f, int tensors, int x_dtype, size_t lut_foot, cudaStream_t st) {
  const EncGeom& g = f.t[0].g;
  const bool h16 = x_dtype == HQMQ_F16, dense = f.t[0].out != nullptr;
  const void* k = nullptr;
#define HQMQ_PICK(IB_, RB_)                                                                                    \
  if (g.ib == IB_ && g.rbits == RB_)                                                                             \
    k = dense ? (h16 ? (const void*)&encode_fused_kernel<HQMQ_F16, IB_, RB_, true> : (const void*)&encode_fused_kernel<HQMQ_BF16, IB_, RB_, true>)   \
              : (h16 ? (const void*)&encode_fused_kernel<HQMQ_F16, IB_, RB_, false> : (const void*)&encode_fused_kernel<HQMQ_BF16, IB_, RB_, false>);
  HQMQ_PICK(10, 3) HQMQ_PICK(12, 4) HQMQ_PICK(13, 6)
#undef HQMQ_PICK
  if (!k)
    k = dense ? (h16 ? (const void*)&encode_fused_kernel<HQMQ_F16, 0, 0, true> : (const void*)&encode_fused_kernel<HQMQ_BF16, 0, 0, true>)
              : (h16 ? (const void*)&encode_fused_kernel<HQMQ_F16, 0, 0, false> : (const void*)&encode_fused_kernel<HQMQ_BF16, 0, 0, false>);
  const size_t smem = fused_smem_bytes(g.S, (lut_foot + 15) & ~(size_t)15);
  HQMQ_CHECK_CUDA(attn::raise_smem_limit(k, smem));
  Maps24 maps;
  memcpy(maps.ref_to_native, index_maps().ref_to_native, 24);
  void* args[] = {(void*)&f, &maps};
  const dim3 grid(f.t[0].cph * g.H, tensors);
  // (the CTAs of a head wait for one another only for a threshold of the call's own)
  const bool waits = f.t[0].C > 0.f && !f.t[0].med_in && f.t[0].cph > 1;
  if (waits) HQMQ_CHECK_CUDA(cudaLaunchCooperativeKernel(k, grid, dim3(kEnc32Threads), args, smem, st));
  else HQMQ_CHECK_CUDA(cudaLaunchKernel(k, grid, dim3(kEnc32Threads), args, smem, st));
  return HQMQ_OK;
}
// Offsets and side planes behind the main kernel, of one tensor or of two.
static int launch_side(const SidePair& sp, int tensors, bool med, cudaStream_t st) {
  const SideArgs& a = sp.t[0];
  const int bh = a.dst.B * a.dst.H;
  if (a.nblk <= kScanSmallBlocks) {
    side_small_kernel<<<dim3(bh, tensors), 32 * (med ? a.nblk : 1), 0, st>>>(sp, med ? 1 : 0);
  } else if (tensors == 1) {        // (arguments picked by blockIdx cost the side kernel a quarter of its time)
    scan_kernel<<<bh, kScanWarps * 32, 0, st>>>(a.dst, a.t_start, a.T_new, a.blk0, a.nblk, a.payload, a.status);
    if (med) side_kernel<<<dim3((a.nblk + 7) / 8, bh), 256, 0, st>>>(a.g, a.x, a.dst, a.t_start, a.blk0, a.nblk);
  } else {
    scan_pair_kernel<<<dim3(bh, tensors), kScanWarps * 32, 0, st>>>(sp);
    if (med) side_pair_kernel<<<dim3((a.nblk + 7) / 8, bh, tensors), 256, 0, st>>>(sp);
  }
  HQMQ_LAUNCH_CHECK();
  return HQMQ_OK;
}
static SideArgs side_args(const hqmq_encode_args* a, const WsPlan& wp, uint32_t* ws) {
  SideArgs s;
  s.g = geom_of(a); s.x = a->x; s.dst = a->dst; s.t_start = a->t_start; s.T_new = a->T_new; s.blk0 = wp.blk0; s.nblk = wp.nblk;
  s.payload = a->median_mult > 0.f ? 1 : 0; s.status = ws + wp.status;
  return s;
}

// ---- fake-quantised tensor straight from x ----------------------------------------------------------------------------
// words of a call's workspace: status [4], histograms, arrivals
static size_t fake_quant_ws_words(int H) { return 4 + (size_t)H * 3 * 2 * kHistBins + (size_t)H * 8; }
static int validate_fake_quant(const hqmq_encode_args* a) {
  if (!a || a->struct_size != sizeof(hqmq_encode_args) || a->dst.struct_size != sizeof(hqmq_packed)) return HQMQ_ERR_ARG;
  if (!a->x || !a->qs || !a->joint) return HQMQ_ERR_ARG;
  if (!is_float_dtype(a->x_dtype)) return HQMQ_ERR_DTYPE;
  const hqmq_packed& d = a->dst;
  if (d.B < 1 || d.H < 1 || d.n_chunks < 1 || d.n_chunks > 32 || d.S < 1 || 24 * d.S > 65536 || d.radius_bits < 1 || d.radius_bits > 8 ||
      a->T_new < 1 || a->t_start != 0)
    return HQMQ_ERR_SHAPE;
  if (!(a->quantile >= 0.f && a->quantile < 1.f)) return HQMQ_ERR_ARG;
  if ((uintptr_t)a->x & (a->x_dtype == HQMQ_F32 ? 15 : 7)) return HQMQ_ERR_ALIGN;
  for (int i = 0; i < 3; ++i)
    if (a->x_stride[i] % 4) return HQMQ_ERR_ALIGN;
  if (((uintptr_t)a->qs & 15) || ((uintptr_t)a->joint & 15)) return HQMQ_ERR_ALIGN;
  return small_call(a) || fused_call(a) ? HQMQ_OK : HQMQ_ERR_UNSUPPORTED;
}
extern "C" size_t hqmq_fake_quant_workspace_bytes(const hqmq_encode_args* a) {
  return validate_fake_quant(a) == HQMQ_OK ? fake_quant_ws_words(a->dst.H) * 4 : 0;
}
extern "C" int hqmq_fake_quant(const hqmq_encode_args* a, void* out, uint32_t* n_flagged, void* workspace, size_t workspace_bytes,
                               void* stream) {
  const int rc = validate_fake_quant(a);
  if (rc) return rc;
  if (!out || ((uintptr_t)out & 15)) return HQMQ_ERR_ARG;
  if (!workspace || workspace_bytes < fake_quant_ws_words(a->dst.H) * 4) return HQMQ_ERR_WORKSPACE;
  if ((uintptr_t)workspace & 15) return HQMQ_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t* ws = reinterpret_cast<uint32_t*>(workspace);
  const hqmq_packed& d = a->dst;
  if (small_call(a)) {
    WsPlan wp{};
    SmallArgs sa;
    const int e = fill_small(a, wp, ws, sa);
    if (e) return e;
    sa.out = out; sa.n_flagged = n_flagged;
    Maps24 maps;
    memcpy(maps.ref_to_native, index_maps().ref_to_native, 24);
    fake_quant_small_kernel<<<d.H, small_threads((int64_t)d.B * a->T_new * d.n_chunks), 0, st>>>(sa, maps);
    HQMQ_LAUNCH_CHECK();
    return HQMQ_OK;
  }
  uint32_t* hist = ws + 4;
  uint32_t* bars = hist + (size_t)d.H * 3 * 2 * kHistBins;
  if (a->median_mult > 0.f && !a->med_in) HQMQ_CHECK_CUDA(cudaMemsetAsync(ws, 0, fake_quant_ws_words(d.H) * 4, st));
  FusedPair f;
  fill_fused(a, 1, ws, hist, bars, out, n_flagged, f.t[0]);
  return launch_fused(f, 1, a->x_dtype, lut_foot_of(a), st);
}

extern "C" size_t hqmq_encode_pair_workspace_bytes(const hqmq_encode_args* k, const hqmq_encode_args* v) {
  const size_t wk = hqmq_encode_workspace_bytes(k), wv = hqmq_encode_workspace_bytes(v);
  if (!wk || !wv) return 0;
  return ((wk + 255) & ~(size_t)255) + wv;
}

extern "C" int hqmq_encode_pair(const hqmq_encode_args* k, const hqmq_encode_args* v, void* workspace, size_t workspace_bytes,
                                void* stream) {
  int rc = validate_encode(k);
  if (rc) return rc;
  rc = validate_encode(v);
  if (rc) return rc;
  const size_t wk = (plan_ws(*k).total + 255) & ~(size_t)255, wv = plan_ws(*v).total;
  if (!workspace || workspace_bytes < wk + wv) return HQMQ_ERR_WORKSPACE;
  if ((uintptr_t)workspace & 15) return HQMQ_ERR_ALIGN;
  unsigned char* wsb = reinterpret_cast<unsigned char*>(workspace);
  const hqmq_packed &dk = k->dst, &dv = v->dst;
  const bool same = dk.B == dv.B && dk.H == dv.H && dk.n_chunks == dv.n_chunks && k->T_new == v->T_new;
  if (!same || k->T_new == 0 || !small_call(k) || !small_call(v) || plan_ws(*k).nblk > kScanSmallBlocks ||
      plan_ws(*v).nblk > kScanSmallBlocks) {
    const bool med = k->median_mult > 0.f;
    if (same && k->T_new > 0 && !small_call(k) && fused_call(k) && fused_call(v) && !bracket_call(k) && !bracket_call(v) &&
        2 * dk.H <= sm_count() && dk.S == dv.S && dk.radius_bits == dv.radius_bits && k->x_dtype == v->x_dtype &&
        med == (v->median_mult > 0.f) && !k->med_in == !v->med_in && plan_ws(*k).nblk == plan_ws(*v).nblk) {
      // a prompt of ordinary length: both tensors in each launch
      cudaStream_t st = (cudaStream_t)stream;
      const WsPlan pk = plan_ws(*k), pv = plan_ws(*v);
      uint32_t *sk = reinterpret_cast<uint32_t*>(wsb), *sv = reinterpret_cast<uint32_t*>(wsb + wk);
      HQMQ_CHECK_CUDA(cudaMemset2DAsync(wsb, wk, 0, (pk.sel + (size_t)dk.H * 8) * sizeof(uint32_t), 2, st));
      FusedPair f;
      fill_fused(k, 2, sk + pk.status, sk + pk.hist, sk + pk.sel, nullptr, nullptr, f.t[0]);
      fill_fused(v, 2, sv + pv.status, sv + pv.hist, sv + pv.sel, nullptr, nullptr, f.t[1]);
      rc = launch_fused(f, 2, k->x_dtype, lut_foot_of(k) > lut_foot_of(v) ? lut_foot_of(k) : lut_foot_of(v), st);
      if (rc || !(med || dk.ofrag || dv.ofrag)) return rc;
      SidePair sp;
      sp.t[0] = side_args(k, pk, sk); sp.t[1] = side_args(v, pv, sv);
      return launch_side(sp, 2, med, st);
    }
    // no common launch shape: one tensor after the other, each with its part of the workspace
    rc = hqmq_encode(k, wsb, wk, stream);
    if (rc) return rc;
    return hqmq_encode(v, wsb + wk, wv, stream);
  }
  cudaStream_t st = (cudaStream_t)stream;
  SmallPair pr;
  rc = fill_small(k, plan_ws(*k), reinterpret_cast<uint32_t*>(wsb), pr.t[0]);
  if (rc) return rc;
  rc = fill_small(v, plan_ws(*v), reinterpret_cast<uint32_t*>(wsb + wk), pr.t[1]);
  if (rc) return rc;
  memcpy(pr.maps.ref_to_native, index_maps().ref_to_native, 24);
  const int64_t chunks = (int64_t)dk.B * k->T_new * dk.n_chunks;
  if (k->T_new == 1 && chunks <= kAppendMax) {
    // one token per sequence: the low-latency kernel; its status words are cleared inside where a tensor's heads fit a cluster
    AppendArgs ap;
    ap.t[0] = pr.t[0]; ap.t[1] = pr.t[1]; ap.maps = pr.maps; ap.clear = dk.H <= 8 ? 1 : 0;
    if (!ap.clear) HQMQ_CHECK_CUDA(cudaMemset2DAsync(wsb, wk, 0, sizeof(uint32_t), 2, st));
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = dk.H; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(dk.H, 2); cfg.blockDim = dim3(2 * (int)((chunks + 31) / 32 * 32)); cfg.stream = st;
    cfg.attrs = at; cfg.numAttrs = ap.clear ? 2 : 1;
    void* kargs[] = {&ap};
    HQMQ_CHECK_CUDA(cudaLaunchKernelExC(&cfg, (const void*)&append_one_kernel, kargs));
    return HQMQ_OK;
  }
  // one launch for the whole append; the two status words (first word of each tensor's part) are cleared ahead of it
  HQMQ_CHECK_CUDA(cudaMemset2DAsync(wsb, wk, 0, sizeof(uint32_t), 2, st));
  append_pair_kernel<<<dim3(dk.H, 2), small_threads((int64_t)dk.B * k->T_new * dk.n_chunks), 0, st>>>(pr);
  HQMQ_LAUNCH_CHECK();
  return HQMQ_OK;
}

extern "C" int hqmq_encode(const hqmq_encode_args* a, void* workspace, size_t workspace_bytes, void* stream) {
  int rc = validate_encode(a);
  if (rc) return rc;
  if (a->T_new == 0) return HQMQ_OK;   // appending nothing: the planes stay as they are, no workspace needed
  const WsPlan wp = plan_ws(*a);
  if (!workspace || workspace_bytes < wp.total) return HQMQ_ERR_WORKSPACE;
  if ((uintptr_t)workspace & 15) return HQMQ_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  const hqmq_packed& d = a->dst;
  const bool med = a->median_mult > 0.f;
  const EncGeom g = geom_of(a);

  uint32_t* ws = reinterpret_cast<uint32_t*>(workspace);
  Maps24 maps;
  memcpy(maps.ref_to_native, index_maps().ref_to_native, 24);

  const bool ext_med = med && a->med_in != nullptr;   // the median comes from the caller (batch of a head split over GPUs)
  if (small_call(a)) {
    SmallArgs sa;
    rc = fill_small(a, wp, ws, sa);
    if (rc) return rc;
    encode_small_kernel<<<d.H, small_threads((int64_t)d.B * a->T_new * d.n_chunks), 0, st>>>(sa, maps);      // (clears the status word itself)
    if (sa.scan) scan_kernel<<<d.B * d.H, kScanWarps * 32, 0, st>>>(d, a->t_start, a->T_new, wp.blk0, wp.nblk, sa.payload, ws + wp.status);
    if (sa.side) side_kernel<<<dim3((wp.nblk + 7) / 8, d.B * d.H), 256, 0, st>>>(g, a->x, d, a->t_start, wp.blk0, wp.nblk);
    HQMQ_LAUNCH_CHECK();
    return HQMQ_OK;
  }
  const bool bracket = bracket_call(a);
  if (fused_call(a) && !bracket) {
    // (status, histograms and select words are the first part of the workspace; the select words serve as arrival counters)
    HQMQ_CHECK_CUDA(cudaMemsetAsync(ws, 0, (wp.sel + (size_t)d.H * 8) * sizeof(uint32_t), st));
    FusedPair f;
    fill_fused(a, 1, ws + wp.status, ws + wp.hist, ws + wp.sel, nullptr, nullptr, f.t[0]);
    rc = launch_fused(f, 1, a->x_dtype, lut_foot_of(a), st);
    if (rc || !(med || d.ofrag)) return rc;
    SidePair sp;
    sp.t[0] = side_args(a, wp, ws);
    return launch_side(sp, 1, med, st);
  }
  HQMQ_CHECK_CUDA(cudaMemsetAsync(ws, 0, wp.zero_bytes, st));
  const uint64_t N = (uint64_t)d.B * a->T_new * d.n_chunks;
  const bool h16 = a->x_dtype == HQMQ_F16;
  if (bracket) {
    // A sample of the tokens predicts the threshold statistic, the main pass needs x only once; should the prediction fail,
    // the one-launch encoder (gated on a word that the check raises) redoes the call.
    const bool pair16 = pair16_of(*a);
    const int T32 = pair16 ? a->T_new / 2 : a->T_new;
    EncGeom g32 = g;
    if (pair16) { g32.n = 32; g32.npl = 32; g32.tpw = 1; g32.T_new = T32; g32.xs_t = 2 * g.xs_t; }
    const uint16_t* x16 = reinterpret_cast<const uint16_t*>(a->x);
    const unsigned char* lut_arg = reinterpret_cast<const unsigned char*>(a->lut);
    const Fast32 f32{x16, g.xs_b, g.xs_h, g32.xs_t, d.H, T32, pair16 ? 1 : 0};
    const int n_s = (T32 + kSampleStride - 1) / kSampleStride;
    int gs = (148 * 8 + d.B * d.H - 1) / (d.B * d.H);
    if (gs > (n_s + 15) / 16) gs = (n_s + 15) / 16;
    if (gs < 1) gs = 1;
    float delta = 3.0f / sqrtf((float)d.B * (float)n_s * 32.f);
    delta = delta < 0.002f ? 0.002f : delta > 0.012f ? 0.012f : delta;
    uint32_t* bp = ws + wp.bp;
    uint32_t* gate = ws + wp.gate;
    const SampleArgs sa{ws + wp.hist_s, ws + wp.sel_s, ws + wp.tickets, (uint64_t)d.B * n_s * 32, a->quantile, a->median_mult, delta, bp, ws + wp.band};
    for (int level = 0; level < 2; ++level) {
      if (h16) sample32_kernel<HQMQ_F16><<<dim3(gs, d.B * d.H), 256, 0, st>>>(f32, sa, level);
      else sample32_kernel<HQMQ_BF16><<<dim3(gs, d.B * d.H), 256, 0, st>>>(f32, sa, level);
    }
    const void* k = nullptr;
#define HQMQ_PICK(IB_, RB_, PAIR_) \
    if (g.ib == IB_ && g.rbits == RB_ && pair16 == PAIR_) k = h16 ? (const void*)&encode_main32_kernel<HQMQ_F16, IB_, RB_, PAIR_> : (const void*)&encode_main32_kernel<HQMQ_BF16, IB_, RB_, PAIR_>;
    HQMQ_PICK(10, 3, false) HQMQ_PICK(12, 4, false) HQMQ_PICK(13, 6, false) HQMQ_PICK(12, 4, true)
#undef HQMQ_PICK
    const size_t smem = (size_t)g.S * 16 + (size_t)kEnc32Warps * kMaxRowWords * 4 + kHistBins * 4 + (size_t)24 * g.S * 16 + lut_foot_of(a) + 16;
    HQMQ_CHECK_CUDA(attn::raise_smem_limit(k, smem));
    const MainGrid mg = main_grid(T32, d.B, d.H);
    int64_t per = mg.per;
    int t_start = a->t_start;
    BracketArgs br{bp, bp, ws + wp.band, ws + wp.und, ws + wp.rcnt, ws + wp.rlist, ws + wp.histA, wp.rcap, wp.und_cap};
    void* kargs[] = {(void*)&g32, (void*)&x16, (void*)&a->qs, (void*)&d, (void*)&t_start, (void*)&maps, (void*)&a->joint, (void*)&lut_arg,
                     (void*)&per, (void*)&br};
    HQMQ_CHECK_CUDA(cudaLaunchKernel(k, dim3(mg.ctas), dim3(kEnc32Threads), kargs, smem, st));
    const int64_t W32 = (int64_t)d.B * T32;
    const int shares = (int)((W32 + mg.per - 2) / mg.per) + 1;             // most CTAs that share a head
    list_select_kernel<<<dim3(shares, d.H), 256, 0, st>>>(bp, ws + wp.histA, ws + wp.rcnt, ws + wp.rlist, wp.rcap, mg.per, W32, ws + wp.histB, N,
                                                          a->median_mult, a->quantile, ws + wp.sel_b, a->med_out, gate);
    if (h16) fixup_kernel<HQMQ_F16><<<dim3(kFixupCtas, d.H), 256, 0, st>>>(f32, d, a->t_start, g.ib, g.rbits, d.B, ws + wp.sel_b, ws + wp.band, ws + wp.und, gate, wp.und_cap);
    else fixup_kernel<HQMQ_BF16><<<dim3(kFixupCtas, d.H), 256, 0, st>>>(f32, d, a->t_start, g.ib, g.rbits, d.B, ws + wp.sel_b, ws + wp.band, ws + wp.und, gate, wp.und_cap);
    FusedPair f;
    fill_fused(a, 1, ws + wp.status, ws + wp.hist, ws + wp.sel, nullptr, nullptr, f.t[0]);
    f.t[0].gate = gate;
    rc = launch_fused(f, 1, a->x_dtype, lut_foot_of(a), st);
    if (rc) return rc;
    SidePair sp;
    sp.t[0] = side_args(a, wp, ws);
    return launch_side(sp, 1, true, st);
  }

  // any other geometry: the main pass, then two more passes over x for the exact threshold and one for the flags
  const int tok_per_block = kEncWarps * g.tpw * kEncIters;
  dim3 grid((a->T_new + tok_per_block - 1) / tok_per_block, d.B * d.H);
  const size_t smem_base = (size_t)g.S * 16 + (size_t)kEncWarps * g.tpw * kMaxRowWords * 4 + kHistBins * 4;
  if (smem_base > 200 * 1024) return HQMQ_ERR_UNSUPPORTED;
  // look-up-table search when a table is given and it fits shared memory next to the joint codebook
  const size_t smem_lut = smem_base + (size_t)24 * g.S * 16 + lut_foot_of(a);
  const bool use_lut = a->search == 0 && a->lut != nullptr && a->lut_footprint >= 0 && smem_lut <= 226 * 1024;
  if (use_lut && (uintptr_t)a->lut & 15) return HQMQ_ERR_ALIGN;
  uint32_t* hist = ws + wp.hist;
  uint32_t* sel = ws + wp.sel;
  uint32_t* hist_arg = med && !ext_med ? hist : nullptr;
  if (use_lut) {
    if (smem_lut > 48 * 1024)
      HQMQ_CHECK_CUDA(cudaFuncSetAttribute(encode_main_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_lut));
    encode_main_kernel<true><<<grid, kEncThreads, smem_lut, st>>>(g, a->x, a->qs, d, a->t_start, hist_arg, maps, a->joint,
                                                                  reinterpret_cast<const unsigned char*>(a->lut));
  } else {
    if (smem_base > 48 * 1024)
      HQMQ_CHECK_CUDA(cudaFuncSetAttribute(encode_main_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_base));
    encode_main_kernel<false><<<grid, kEncThreads, smem_base, st>>>(g, a->x, a->qs, d, a->t_start, hist_arg, maps, a->joint, nullptr);
  }
  HQMQ_LAUNCH_CHECK();
  SidePair sp;
  sp.t[0] = side_args(a, wp, ws);
  // (without a threshold no chunk of this call is flagged: the record offsets of its blocks just carry the running total on)
  if (!med) return d.ofrag ? launch_side(sp, 1, false, st) : HQMQ_OK;

  const int64_t per_bh = (int64_t)a->T_new * d.n_chunks;
  // about 16 resident CTAs per SM in total; each CTA amortises zeroing and flushing its private histograms
  const int bh_count = d.B * d.H;
  int hb = (148 * 16 + bh_count - 1) / bh_count;
  const int hb_max = (int)((per_bh + 256 * 16 - 1) / (256 * 16));
  if (hb > hb_max) hb = hb_max;
  if (hb < 1) hb = 1;
  if (ext_med) {
    // threshold from the caller's medians, then the plain flag pass
    thr_from_median_kernel<<<(d.H + 63) / 64, 64, 0, st>>>(a->med_in, a->median_mult, d.H, sel, a->med_out);
  } else {
    select_kernel<<<d.H, 256, 0, st>>>(hist, sel, 0, N, a->median_mult, nullptr, a->quantile);
    hist_kernel<<<dim3(hb, bh_count), 256, 0, st>>>(g, a->x, hist, sel, 1);
    select_kernel<<<d.H, 256, 0, st>>>(hist, sel, 1, N, a->median_mult, nullptr, a->quantile);
    hist_kernel<<<dim3(hb, bh_count), 256, 0, st>>>(g, a->x, hist, sel, 2);
    select_kernel<<<d.H, 256, 0, st>>>(hist, sel, 2, N, a->median_mult, a->med_out, a->quantile);
  }
  const int tok_per_fblock = 8 * g.tpw;
  int fb = (a->T_new + 4 * tok_per_fblock - 1) / (4 * tok_per_fblock);
  const int fb_cap = (148 * 32 + bh_count - 1) / bh_count;
  if (fb > fb_cap) fb = fb_cap;
  if (fb < 1) fb = 1;
  flags_kernel<<<dim3(fb, bh_count), 256, 0, st>>>(g, a->x, d, a->t_start, sel);
  HQMQ_LAUNCH_CHECK();
  return launch_side(sp, 1, true, st);
}
