// Attention of many query positions over one compressed cache: parameters and the host entry points (attn_prefill.cu).
#pragma once
#include "attn_kernel.cuh"

namespace hqmq {
namespace attn {

constexpr int kPfTok = 128;                       // tokens per operand tile
constexpr int kPfMaxCtas = 148;                   // one CTA per SM
// Query positions from which a call decodes the cache once instead of once per position.  This path at 16 positions / the decode
// kernels at 15, us:
//   8 heads of 128, G 4, s96 with outliers, 1 sequence: 300 tokens 22.5 / 14.6, 1000 25.6 / 22.8, 4000 33 / 45, 16000 81 / 137, 64000
//   198 / 434; 16 sequences: 300 25 / 155, 4000 168 / 518, 16000 621 / 1884
//   4 heads, G 7, s192, 4 sequences: 1000 27 / 63, 16000 109 / 329;  8 heads of 64, G 8, 4 sequences: 1000 23 / 78
// (At 24 positions it costs what it costs at 16.  The decode kernels stay shorter while every position and head can have a cluster
// of its own, 148 in all, up to about 2000 tokens, and at 8 positions of one short sequence: 1000 tokens 18.  The line does not look
// at that, nor at 8 to 15 positions of many sequences, where this path would be the shorter: 16000 tokens of 16, 8 positions, 1014.)
constexpr int kPrefillMinQueries = HQMQ_ATTN_PROMPT_QUERIES;
constexpr int kPrefillMaxTable = 8192;            // codewords per head that fit the expand kernel's shared memory
constexpr size_t kPrefillImageBytes = (size_t)512 << 20;   // operand images held at a time; larger caches go by groups of (b, head)

struct PrefillParams {
  const void* Q; int q_dtype; int64_t qs_b, qs_h, qs_t;
  void* O; int o_dtype; int64_t os_b, os_h, os_t;
  int q_vec, o_vec;                               // 16-byte accesses to Q / O rows are aligned (16-bit types)
  int Hkv, G, Tq, Tkv, causal, window;
  int P, streams, units_m;                        // query positions per stream, row blocks per unit, units per (b, head)
  int kt0, nt;                                    // first KV tile that any query sees, tiles in the images
  int bh0;                                        // first (b, head) of the group
  int64_t Wh, total, L;                           // tiles per (b, head), in all, per CTA (0: whole units, not pieces)
  int units_all;                                  // units of the group
  const unsigned char* kimg; const unsigned char* vimg;
  const float* kmul; const float* vmul;           // [B * H_kv] what a score / an output is multiplied by
  float* part;                                    // [CTA][2][256 rows x (d + 2)]: [d / 4][256][4], m [256], l [256]
  uint32_t* status; uint32_t epoch;
  int start_m[kPfMaxCtas], start_off[kPfMaxCtas];  // first unit of every CTA's piece, the unit's tiles before it
};

struct ExpandParams {
  hqmq_packed K, V;
  hqmq_ref_packed Kr, Vr;
  const uint16_t* tblK; const uint16_t* tblV;
  const void* jK; const void* jV; int j_dtype;
  int ib, table_rows, Hkv, Tkv, kt0, nt, per, bh0;
  float qscale, vscale;                           // softmax scale * log2(e), 1 / qmax
  unsigned char* kimg; unsigned char* vimg;
  float* kmul; float* vmul;
  uint32_t* status; uint32_t epoch;
};

struct PrefillPlan {
  PrefillParams p;
  int group, grid;
  bool whole;                                     // units are not cut
  size_t off_mul, off_img, off_part, ws_bytes;
};

// The plan of a call that takes this path, or false.
bool prefill_plan(const hqmq_attn_args* a, PrefillPlan& pl);
int prefill_launch(const hqmq_attn_args* a, const PrefillPlan& pl, void* workspace, float qscale, uint32_t epoch, cudaStream_t st);
// The staged decode kernel that a call would take, or nullptr where that is the generic one (attn.cu).
const void* staged_kernel(const hqmq_attn_args* a);
// Raises a kernel's dynamic shared-memory limit to the device's maximum, once per kernel and device (attn.cu).
cudaError_t raise_smem_limit(const void* kernel, size_t smem);

}  // namespace attn
}  // namespace hqmq
