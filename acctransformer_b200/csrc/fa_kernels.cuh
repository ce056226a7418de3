// Parameter blocks and launchers of the attention kernels (internal to the library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace acct {

constexpr int kTile = 128;          // rows of a Q tile and of a K/V tile; also the band block
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// What a mask tensor of zeros and ones leaves to compute.  In a row that has an unmasked key anywhere, a masked position
// (-10000 added to its score) has a probability of exactly 0 (exp2 underflows) and adds nothing to O, dQ, dK and dV, as long
// as no score can make up for the -10000 and no operand is infinite or NaN.  Then a tile that is all 1 need not be computed,
// and in a mixed one a bit per position is all there is to read, without arithmetic on the scores.  The rows are checked
// on the mask (mask_bits_kernel, mask_plan_kernel), the operands through the largest squared row norms of q, k and v
// (plan_norms_kernel; by Cauchy-Schwarz |score| <= scale |q| |k|) and, in the backward, of dO and the row sums D.  Where
// the norms do not allow it, every tile is computed from the mask itself.
constexpr int kPlanTiles = 256;       // tiles per row and column a plan can describe (32 768 positions)
constexpr int kPlanWords = kPlanTiles / 32;
constexpr int kPlanBitWords = 1024;   // per tile: 128 x 128 bits by query row, then the same by key
struct alignas(16) MaskPlan {         // head of the plan; PlanParts lie behind it
  unsigned int q2, k2, v2;            // largest squared row norms, as bits (a NaN is larger than everything)
  unsigned int any;                   // the plan saves something
};
// The parts of a plan, all in one piece of device memory.
struct PlanParts {
  MaskPlan* head;
  uint32_t* need;                     // [mask_batch, tiles_q][kPlanWords]: bit j = this Q tile needs K/V tile j
  uint32_t* need_t;                   // [mask_batch, tiles_k][kPlanWords]: bit i = this K/V tile is needed by Q tile i
  uint32_t* seen;                     // [mask_batch, tiles_q][4]: bit r = row r has an unmasked key
  uint8_t* cls;                       // [mask_batch, tiles_q, tiles_k]: ScoreMods::mask_tiles, or 3 = take the bits
  uint32_t* bits;                     // [mask_batch, tiles_q, tiles_k][kPlanBitWords]: set = masked (tiles of class 3)
};
inline size_t plan_parts(void* base, int mask_batch, int S_q, int S_k, PlanParts* out) {
  const size_t mb = mask_batch, tq = (S_q + kTile - 1) / kTile, tk = (S_k + kTile - 1) / kTile;
  uint8_t* at = static_cast<uint8_t*>(base);
  auto take = [&](size_t bytes) { uint8_t* here = at; at += (bytes + 15) / 16 * 16; return here; };
  out->head = reinterpret_cast<MaskPlan*>(take(sizeof(MaskPlan)));
  out->need_t = reinterpret_cast<uint32_t*>(take(mb * tk * kPlanWords * 4));
  out->seen = reinterpret_cast<uint32_t*>(take(mb * tq * 16));
  out->need = reinterpret_cast<uint32_t*>(take(mb * tq * kPlanWords * 4));
  out->cls = take(mb * tq * tk);
  out->bits = reinterpret_cast<uint32_t*>(take(mb * tq * tk * kPlanBitWords * 4));
  return static_cast<size_t>(at - static_cast<uint8_t*>(base));
}
// With scores within +-4800 a masked one ends at least 400 below the largest of its row; exp() of that, and of up to 8 / log2e
// more (the forward's stale maximum), is 0 in fp32: it is from -104 down.
constexpr float kPlanMaxScore = 4800.0f;
constexpr float kPlanMaxNorm2 = 1e30f;

__device__ __forceinline__ bool plan_holds(const MaskPlan* plan, float scale) {
  const float q2 = __uint_as_float(plan->q2), k2 = __uint_as_float(plan->k2), v2 = __uint_as_float(plan->v2);
  return q2 < kPlanMaxNorm2 && k2 < kPlanMaxNorm2 && v2 < kPlanMaxNorm2 &&      // (false for NaN)
         sqrtf(q2) * sqrtf(k2) * scale < kPlanMaxScore;
}

// What the softmax stage must look at besides the raw scores.
struct ScoreMods {
  int causal;
  int prev_block_num, next_block_num;
  int mask_kind, mask_dtype, mask_batch;
  const void* mask;
  const uint8_t* mask_tiles;        // optional [mask_batch, ceil(S_q/128), ceil(S_k/128)]: 0 = tile all 0 (not read),
                                    // 2 = tile all 1 (fill value added, not read), 1 = read; null = read every tile
  const void* drop;
  int drop_dtype;
  float drop_scale;                 // 1/keep_prob for uint8 masks, 1 for pre-scaled 16-bit masks
  const void* alibi;                // [B,N,1,S_k] in the tensor dtype
  const float* alibi_slopes;        // [N]
  const int* seq_lens;              // [B]
  int tri_block;                    // > 0: query row r sees keys < (r / tri_block + 1) * tri_block only
  PlanParts plan;                   // of a mask tensor, or plan.head == null: none
  int drop_philox;                  // 1: dropout decided in the kernel (DropoutRng), `drop` is null, drop_scale = 256/threshold
  unsigned int drop_seed_lo, drop_seed_hi, drop_offset, drop_threshold;
};

struct alignas(64) FwdParams {
  CUtensorMap map_q, map_k, map_v, map_o;
  void* o;
  float* lse;
  int64_t o_stride_b, o_stride_h, o_stride_s;
  int B, N, S_q, S_k, D;
  int kv_group;                     // query heads per key/value head (1 unless grouped-query attention)
  int unit_group;                   // (batch, head) slices whose thread blocks are interleaved, heaviest tile pairs first
  float scale, scale_log2;          // scale_log2 = scale * log2(e)
  ScoreMods mods;
  unsigned int* status;
};

struct alignas(64) BwdParams {
  CUtensorMap map_q, map_k, map_v, map_do;
  CUtensorMap map_dq;               // fp32 dQ accumulator [B,N,S_q,D], box 32 x 128
  CUtensorMap map_dk, map_dv;       // 16-bit dk, dv [B,N_kv,S_k,D], box 64 x 128 (unused with fp32 gradients and above head_dim 160)
  const float* lse;                 // [B,N,S_q]
  const float* delta;               // [B,N,S_q]  rowsum(dO * O)
  float* dq_acc;                    // [B,N,S_q,D] fp32, zeroed before launch
  unsigned int* dq_order;           // [B,N,ceil(S_q/128)] turn counters (x 2 for head_dim > 128), zeroed before launch;
                                    // nullptr = any order
  const unsigned int* plan_stats;   // with mods.plan: largest squared row norm of dO and largest |D| of this call, as bits
  unsigned int* work_counter;       // one word, zeroed before launch: the next work item of the persistent CTAs
  void* dk;
  void* dv;
  int grads_f32;
  int B, N, S_q, S_k, D;
  int kv_group;                     // query heads per key/value head; dk, dv are [B, N / kv_group, S_k, D]
  float scale;                      // multiplies dS for dQ and dK
  float scale_log2;
  ScoreMods mods;
  unsigned int* status;
};

struct DecodeParams {
  const void* q;
  const void* k;
  const void* v;
  void* y;
  const int* seq_lens;
  float* part_acc;                  // [B*N, splits, D]
  float* part_ml;                   // [B*N, splits, 2]
  int64_t kv_stride_b, kv_stride_h, kv_stride_s;
  int B, N, S_max, D;
  int kv_group;                     // query heads per key/value head: 1..16 (head_dim <= 128), else 1, 2, 4 or 8
  const int* block_table;           // [B, max_pages] page numbers, or nullptr: contiguous caches
  int page_shift, max_pages;        // rows per page = 1 << page_shift; kv_stride_b is then the page stride
  int splits;
  int clustered;                    // 1: the parts of a slice are one thread-block cluster and merge through its shared memory
  float scale_log2;
};

// counts into *mismatch the elements of a [batch, S_q, S_k] mask that differ from the causal mask (key > query)
cudaError_t launch_mask_check(const void* mask, int dtype, int batch, int S_q, int S_k, unsigned int* mismatch,
                              cudaStream_t stream);

// writes one class byte per 128x128 tile of a [batch, S_q, S_k] mask into tiles[batch, ceil(S_q/128), ceil(S_k/128)]:
// 0 = all elements 0, 2 = all elements 1, 1 = anything else (ScoreMods::mask_tiles)
cudaError_t launch_mask_classify(const void* mask, int dtype, int batch, int S_q, int S_k, uint8_t* tiles,
                                 cudaStream_t stream);

// Fills a plan for a mask with its tile classes `tiles` and for q [B,N,S_q,D], k and v [B,N_kv,S_k,D] with element strides
// (B, N, S); at most kPlanTiles tiles per dimension.  `norms` (may be null): a head outside the plan whose norms are written
// as well, or, if `norms_known`, taken instead of a pass over q, k and v.
struct PlanOperand {
  const void* ptr;
  int64_t stride[3];
  int heads, rows;
};
cudaError_t launch_mask_plan(const void* mask, int mask_dtype, int mask_batch, const uint8_t* tiles, int S_q, int S_k,
                             const PlanOperand (&qkv)[3], int B, int D, bool bf16, const PlanParts& plan, MaskPlan* norms,
                             bool norms_known, cudaStream_t stream);

// Raises a kernel's dynamic shared memory limit, once per thread, kernel and device (the call costs the host about as
// much as a launch argument block, and every operator call would repeat it).
cudaError_t allow_smem(const void* kernel, size_t bytes);

// Launchers: return cudaGetLastError() of the launch.
cudaError_t launch_fa_fwd(const FwdParams& p, bool bf16, int sm_count, cudaStream_t stream);
cudaError_t launch_fa_bwd(const BwdParams& p, bool bf16, int sm_count, cudaStream_t stream);
// head_dim in (64, 128], dQ in any order, no mask tensor, alibi, band, valid lengths or dropout, row groups of whole tiles:
// like launch_fa_bwd with 64-row boxes of the Q, dO and dQ maps
cudaError_t launch_fa_bwd_pair(const BwdParams& p, bool bf16, int sm_count, cudaStream_t stream);
// head_dim in (128, 256]: Q / dO maps with 64-row boxes, the dQ map with a 32 x 64 box, two turn counters per Q tile
cudaError_t launch_fa_bwd_wide(const BwdParams& p, bool bf16, cudaStream_t stream);
// head_dim in (128, 160], dQ in any order: like the above with a 32 x 32 box of the dQ map, and dk, dv maps
constexpr int kMidHeadDim = 160;
cudaError_t launch_fa_bwd_mid(const BwdParams& p, bool bf16, cudaStream_t stream);
// writes the {0,1} mask the kernels' in-kernel dropout uses, [units, S_q, S_k] uint8 (units = B*N)
cudaError_t launch_dropout_mask(unsigned char* mask, int units, int S_q, int S_k, unsigned int seed_lo, unsigned int seed_hi,
                                unsigned int offset, unsigned int threshold, cudaStream_t stream);
// delta = rowsum(dO * O); the same pass zero-fills the packed fp32 dQ accumulator zero_acc[rows, D] and the counters, and
// raises plan_stats (if given: zeroed by the caller) to the largest squared row norm of dO and the largest |delta|
cudaError_t launch_bwd_delta(const void* o, const void* d_o, float* delta, int64_t rows, int D, const int64_t (&o_stride)[3],
                             const int64_t (&do_stride)[3], int N, int S_q, bool bf16, cudaStream_t stream,
                             float* zero_acc, unsigned int* counters, int64_t n_counters, unsigned int* plan_stats);
cudaError_t launch_bwd_convert_dq(const float* dq_acc, void* dq, int64_t n_elems, bool bf16, bool f32_out,
                                  cudaStream_t stream);
// (with `resident` nothing is launched: see launch_parts)
cudaError_t launch_decode(const DecodeParams& p, bool bf16, cudaStream_t stream, int* resident = nullptr);
// split kernel for 2..16 query heads per cache head at head_dim <= 128 (tensor-core path, decode_gqa.cu)
cudaError_t launch_decode_gqa_split(const DecodeParams& p, bool bf16, cudaStream_t stream, int* resident);
#ifndef ACCT_DECODE_GQA_MIN_GROUP
#define ACCT_DECODE_GQA_MIN_GROUP 2
#endif
constexpr int kDecodeGqaMinGroup = ACCT_DECODE_GQA_MIN_GROUP;   // groups of at least this many heads take that path

}  // namespace acct
