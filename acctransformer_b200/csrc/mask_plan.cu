// What a mask tensor leaves to compute (MaskPlan in fa_kernels.cuh).
//
// Packed documents, padding and block-sparse masks consist mostly of 128x128 tiles that are all 1.  Adding -10000 to such
// a tile and computing it costs as much as any other tile; 3 000 tokens of four documents need a third of their tiles.  And a
// mixed tile costs a pass over its scores in tensor memory and, where rows are not 16-byte aligned, 128 loads per thread,
// for every head.  Three small passes find out once per call what counts: one turns the mixed tiles into bits (by query for
// the forward, whose threads own score rows, by key for the backward) and notes which rows have an unmasked key, one draws
// up the tiles that each Q tile and each K/V tile needs, one bounds q, k and v (it returns at once if nothing is saved).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fa_common.cuh"
#include "fa_kernels.cuh"

namespace acct {

namespace {

constexpr int kPlanThreads = 256;
constexpr int kPlanWarps = kPlanThreads / 32;

// One block per 128x128 tile; warp w takes rows w, w + 8, ..
__global__ void __launch_bounds__(kPlanThreads) mask_bits_kernel(const void* mask, int dtype, int S_q, int S_k,
                                                                 const uint8_t* tiles, PlanParts plan) {
  __shared__ uint32_t words[kTile][4];
  __shared__ uint32_t seen[4];
  const int j = blockIdx.x, i = blockIdx.y, mb = blockIdx.z;
  const int64_t row_of_tiles = static_cast<int64_t>(mb) * gridDim.y + i, tile = row_of_tiles * gridDim.x + j;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = tiles[tile];
  if (c == 0 || c == 2) {                            // (any other byte: the tile is read)
    if (tid == 0) plan.cls[tile] = static_cast<uint8_t>(c);
    if (c == 0 && tid < 4) atomicOr(&plan.seen[row_of_tiles * 4 + tid], 0xffffffffu);
    return;
  }
  if (tid < 4) seen[tid] = 0u;
  __syncthreads();
  int other = 0;                                     // a value that is neither 0 nor 1
#pragma unroll 4
  for (int r = warp; r < kTile; r += kPlanWarps) {
    const int row = min(i * kTile + r, S_q - 1);     // (a row past the end repeats the last one: nobody looks at it)
    const int64_t at = (static_cast<int64_t>(mb) * S_q + row) * S_k;
    bool zero = false;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int col = j * kTile + x * 32 + lane;
      const float v = col < S_k ? load_mask_value(mask, dtype, at + col) : 1.f;     // (keys past the end: masked)
      zero |= v == 0.f;
      other |= v != 0.f && v != 1.f;
      const uint32_t w = __ballot_sync(0xffffffffu, v != 0.f);
      if (lane == 0) words[r][x] = w;
    }
    if (__any_sync(0xffffffffu, zero) && lane == 0) atomicOr(&seen[r >> 5], 1u << (r & 31));
  }
  other = __syncthreads_or(other);
  if (tid == 0) plan.cls[tile] = other ? 1 : 3;
  if (tid < 4) atomicOr(&plan.seen[row_of_tiles * 4 + tid], seen[tid]);
  if (other) return;
  uint32_t* out = plan.bits + tile * kPlanBitWords;
  for (int t = tid; t < kTile * 4; t += kPlanThreads) out[t] = words[t >> 2][t & 3];
  // by key: 32 x 32 blocks transposed with ballots; block (x, y) = columns 32x.., rows 32y..
  for (int blk = warp; blk < 16; blk += kPlanWarps) {
    const int x = blk & 3, y = blk >> 2;
    const uint32_t w = words[y * 32 + lane][x];
    uint32_t mine = 0u;
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      const uint32_t col = __ballot_sync(0xffffffffu, (w >> e) & 1u);
      if (lane == e) mine = col;
    }
    out[kTile * 4 + (x * 32 + lane) * 4 + y] = mine;
  }
}

// One block per (Q tile, mask of the batch), one thread per K/V tile.  `norms`: see launch_mask_plan.
__global__ void __launch_bounds__(kPlanThreads) mask_plan_kernel(int S_q, int S_k, PlanParts plan, MaskPlan* norms, bool norms_known) {
  if (norms != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    if (norms_known) {
      plan.head->q2 = norms->q2; plan.head->k2 = norms->k2; plan.head->v2 = norms->v2;
    } else {
      norms->q2 = norms->k2 = norms->v2 = norms->any = 0u;      // (raised by the next kernel)
    }
  }
  const int i = blockIdx.x, mb = blockIdx.y, tiles_q = gridDim.x, tiles_k = (S_k + kTile - 1) / kTile;
  const int64_t row_of_tiles = static_cast<int64_t>(mb) * tiles_q + i;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool there = tid < tiles_k;
  const int c = there ? plan.cls[row_of_tiles * tiles_k + tid] : 0;
  bool open = false;                                 // row tid of the tile exists and sees no key: leave the Q tile as it is
  if (tid < kTile) open = i * kTile + tid < S_q && ((plan.seen[row_of_tiles * 4 + (tid >> 5)] >> (tid & 31)) & 1u) == 0u;
  const int uncovered = __syncthreads_or(open);
  if (there && uncovered && c == 3) plan.cls[row_of_tiles * tiles_k + tid] = 1;
  const bool need = there && (c != 2 || uncovered);
  const uint32_t word = __ballot_sync(0xffffffffu, need);
  if (lane == 0) plan.need[row_of_tiles * kPlanWords + warp] = word;
  if (need) atomicOr(&plan.need_t[(static_cast<int64_t>(mb) * tiles_k + tid) * kPlanWords + (i >> 5)], 1u << (i & 31));
  if (__syncthreads_or(c >= 2 && !uncovered) && tid == 0) atomicOr(&plan.head->any, 1u);
}

struct NormOperands {
  PlanOperand t[3];
};

// Largest squared row norm of each operand.  16 bytes per lane, LPR lanes per row; compared as bits, so that a NaN wins.
template <bool BF16, int LPR>
__global__ void plan_norms_kernel(const __grid_constant__ NormOperands ops, int B, int D, MaskPlan* plan, MaskPlan* copy) {
  if (plan->any == 0u) return;
  __shared__ unsigned int block_max;
  const PlanOperand& t = ops.t[blockIdx.y];
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  if (threadIdx.x == 0) block_max = 0u;
  __syncthreads();
  const int64_t rows = static_cast<int64_t>(B) * t.heads * t.rows;
  const int64_t step = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32) * RPW;
  unsigned int most = 0u;
#pragma unroll 4
  for (int64_t row0 = (static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5)) * RPW; row0 < rows; row0 += step) {
    const int64_t row = row0 + lane / LPR;
    float acc = 0.f;
    if (row < rows && sub * 8 < D) {
      const uint32_t bh = static_cast<uint32_t>(row / t.rows);
      const uint4 a = *reinterpret_cast<const uint4*>(
          reinterpret_cast<const uint16_t*>(t.ptr) + static_cast<int64_t>(bh / t.heads) * t.stride[0] +
          static_cast<int64_t>(bh % t.heads) * t.stride[1] + (row % t.rows) * t.stride[2] + sub * 8);
      acc = dot8<BF16>(a, a, 0.f);
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    most = max(most, __float_as_uint(acc) & 0x7fffffffu);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) atomicMax(&block_max, most);
  __syncthreads();
  if (threadIdx.x != 0) return;
  atomicMax(blockIdx.y == 0 ? &plan->q2 : blockIdx.y == 1 ? &plan->k2 : &plan->v2, block_max);
  if (copy != nullptr) atomicMax(blockIdx.y == 0 ? &copy->q2 : blockIdx.y == 1 ? &copy->k2 : &copy->v2, block_max);
}

}  // namespace

cudaError_t launch_mask_plan(const void* mask, int mask_dtype, int mask_batch, const uint8_t* tiles, int S_q, int S_k,
                             const PlanOperand (&qkv)[3], int B, int D, bool bf16, const PlanParts& plan, MaskPlan* norms,
                             bool norms_known, cudaStream_t stream) {
  const int tiles_q = (S_q + kTile - 1) / kTile, tiles_k = (S_k + kTile - 1) / kTile;
  // head, need_t and seen are added into; they come first
  const size_t zeroed = reinterpret_cast<uint8_t*>(plan.need) - reinterpret_cast<uint8_t*>(plan.head);
  cudaError_t e = cudaMemsetAsync(plan.head, 0, zeroed, stream);
  if (e != cudaSuccess) return e;
  mask_bits_kernel<<<dim3(tiles_k, tiles_q, mask_batch), kPlanThreads, 0, stream>>>(mask, mask_dtype, S_q, S_k, tiles, plan);
  mask_plan_kernel<<<dim3(tiles_q, mask_batch), kPlanThreads, 0, stream>>>(S_q, S_k, plan, norms, norms_known);
  e = cudaGetLastError();
  if (e != cudaSuccess || norms_known) return e;
  NormOperands ops;
  for (int i = 0; i < 3; ++i) ops.t[i] = qkv[i];
  auto kern = D <= 64 ? (bf16 ? plan_norms_kernel<true, 8> : plan_norms_kernel<false, 8>)
              : D <= 128 ? (bf16 ? plan_norms_kernel<true, 16> : plan_norms_kernel<false, 16>)
                         : (bf16 ? plan_norms_kernel<true, 32> : plan_norms_kernel<false, 32>);
  kern<<<dim3(148 * 4, 3), 256, 0, stream>>>(ops, B, D, plan.head, norms);
  return cudaGetLastError();
}

}  // namespace acct
