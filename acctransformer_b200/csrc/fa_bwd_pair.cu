// FlashAttention-2 backward for head_dim in (64, 128] on pairs of thread blocks (sm_100a, cta_group::2).
//
// A work item is two neighbouring 128-row K/V tiles of one (batch, head) slice and the Q tiles that touch either.  The two
// blocks of a cluster hold one tile each and walk the Q tiles together; every product is one M = 256 (dQ: M = 128) MMA over
// both, issued by the block of rank 0.  Per 128 queries and 128 keys the one-block kernel (fa_bwd.cu) moves 480 KB through
// its shared memory (operands 256, Q and dO in 64, dS^T 32, dQ out 2 x 64: 3 840 clk at 128 B/clk, against 2 560 clk of
// products) and adds 64 KB of dQ in L2, which alone takes it some 4 000 clk of its 4 800 per step.  Here a block reads only
// its half of every B operand, and dQ is summed over both tiles inside the product:
//   S^T  = K Q^T         M 256 keys  N 128 queries  B: 64 queries per block   (K-major)
//   dP^T = V dO^T        the same
//   dV  += P^T dO    M 256 keys  N 128 columns  A: tensor memory, B: 64 columns per block (MN-major)
//   dK  += dS^T Q        the same
//   dQ   = dS K          M 128 queries, N 128 columns, contraction over 256 keys: A: dS^T of this block's 64 queries (half of
//                        it copied over by the peer), B: 64 columns of both K tiles
// 384 KB and 32 KB of dQ per block.  A block of rank r keeps, of Q and dO: rows [64r, 64r+64) of the tile (for S^T, dP^T) and
// columns [64r, 64r+64) (for dK, dV), each with one buffer that is refilled as soon as its product has finished.
//
// The first Q tiles of a head may need the first K/V tile alone (under a causal mask one, at the end of a row group several;
// all of them where there is no second tile).  In those steps the second tile has no part in any product's result: dQ
// contracts over the first 128 keys, and dV and dK write the first block's rows only, or into the second's accumulators what
// its first step with a part overwrites.  That its P and dS are 0 there would not do: 0 times a NaN or infinity of a key or
// query that do not see one another is NaN.
//
// Tensor memory (512 columns): X = S^T | Y = dP^T | dK | dV, 128 each.  P^T goes over columns 0-31 and 96-127 of X (each half
// of the compute warps over its own), dS^T likewise in Y; dQ (64 columns of a block: its 64 rows, columns 0-63 in lanes 0-63,
// columns 64-127 in lanes 64-127) takes columns 32-95 of X, which are free from when S^T is in registers until the
// next S^T.  So dP^T of the next tile waits for nothing but dK, and dQ drains under it.  Tensor-pipe order per Q tile n:
//   dV(n), S^T(n+1) | dK(n), dP^T(n+1) | dQ(n)
// Warp roles (four warpgroups, registers re-split): warps 0-7 compute (thread = one key row x 64 queries), 8-11 drain dQ (and
// dV at the end of an item), 12 TMA producer, 13 MMA issuer (rank 0) or relay (rank 1).  Work items, mailboxes, statistics
// and the write-out are those of the one-block kernel, which this one replaces where it applies (bwd_on_pairs).
//
// Barriers: what the MMA warp waits for lives in rank 0's shared memory, both blocks' TMA loads complete on it and a lane of
// each warp of both arrives there; what the MMA warp signals is committed to both blocks.  No hand-off of a step releases or
// acquires at cluster scope, which costs some 1 000 clk each: tensor memory needs its own fences only, and what goes into the
// other block's shared memory goes there by an asynchronous copy (plain and st.async stores of the same 16 KB took 1 400 and
// 3 000 clk).
//
// 2 x 32 heads of 128, 8 192 tokens, causal, against the one-block kernel: backward call 3 416 -> 2 583 us, forward and backward
// 4 421 -> 3 933; a step 4 800 -> 4 100 clk (cycle counters; with the register split of before).  The tensor pipe is busy 59 % of
// the time (43 %).  What bounds it now: the compute warps (S^T -> P^T -> dS^T, 3 500 clk of a step), whose two halves wait for
// one another through the tensor pipe.
//
// Follows the reference's backward (train/acctransformer/flash_attention/ops/flash_attention/flash_attention_bwd.py:259-415)
// like the one-block kernel does.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fa_common.cuh"
#include "fa_kernels.cuh"
#include "fa_bwd_helpers.cuh"
#include "ptx.cuh"

namespace acct {

namespace {

constexpr int kPThreads = 512;
constexpr int kPComputeThreads = 256;
constexpr int kPDrainWarp0 = 8, kPProducerWarp = 12, kPMmaWarp = 13;     // (warp 13 of rank 1: the relay)
constexpr int kPUnitGroup = 8;          // (batch, head) slices whose items are interleaved, heaviest tiles first
// 256 x 168 + 128 x 96 + 128 x 80 = 512 x 128.  Backward call, 2 x 32 heads, 8 192 tokens causal: 2 590 us; 176 / 88 / 72 2 639;
// 176 / 104 / 56, where the MMA warp spills, 2 741.
constexpr int kPRegsCompute = 168, kPRegsDrain = 96, kPRegsControl = 80;
constexpr uint32_t kPTile = 32768;      // 128 rows x 128 columns of 16-bit values
constexpr uint32_t kPHalf = 16384;      // 64 rows x 128 columns, or 128 rows x 64 columns

struct PairItem {
  int w;                         // its number; >= the number of items: none is left
  int n_iter;                    // steps: Q tiles x query heads of the group
  uint16_t bh_kv, jp, i_lo, n_per;   // slice, pair of K/V tiles, first Q tile, Q tiles per query head
  uint16_t n_first;              // how many of those, from the first on, need the first K/V tile alone
};

struct PairShared {
  uint64_t item_full[2], item_empty[2];   // producer <-> the other roles of its block: item[] (two slots)
  uint64_t w_full[2], w_empty[2];         // rank 0's producer <-> rank 1's: w_next[]
  // rank 0's count (TMA loads of both blocks, one lane of each warp of both)
  uint64_t qk_full, qm_full;     // Q rows (first step of an item: and K) / Q columns (first step: and the columns of both K tiles)
  uint64_t dok_full, dom_full;   // dO rows (first step: and V) / dO columns
  uint64_t p_half, p_ready;      // P^T of the first 32, of all 64 queries of each half is in tensor memory
  uint64_t s_read;               // S^T is in registers
  uint64_t ds_tmem;              // dS^T is in tensor memory
  uint64_t ds_peer;              // rank 1's dS^T for dQ is complete
  uint64_t dq_read;              // drain: dQ is in registers
  uint64_t acc_free;             // compute, drain: dK and dV of the item are in registers
  // committed to both blocks
  uint64_t st_full, dp_full, dq_full;
  uint64_t ds_in;                // this block's dS^T for dQ: its own half written, the peer's arrived
  uint64_t stats_ready;          // the next step's statistics are in shared memory
  uint64_t store_done;           // both blocks' dK stores have read their dS^T areas
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
  uint32_t w_next[2];
  PairItem item[2];
  alignas(16) float nlse2[2][kTile];      // -L * log2(e) per query of the tile (-inf for rows past S_q)
  alignas(16) float ndelta[2][kTile];     // -D
};
constexpr size_t kPSmem = 3 * kPTile + 4 * kPHalf + kPTile + 2 * kPHalf + sizeof(PairShared);
static_assert(kPSmem <= 232448, "shared memory of a thread block");

// Q tiles i that need K/V tile j (decode_item of the one-block kernel, without a band or valid lengths)
__device__ __forceinline__ void q_range(const BwdParams& p, int j, int& lo, int& hi) {
  const ScoreMods& mods = p.mods;
  lo = 0;
  hi = (p.S_q + kTile - 1) / kTile - 1;
  if (mods.causal) lo = max(lo, j);
  if (mods.tri_block > 0) lo = max(lo, (((j * kTile) / mods.tri_block) * mods.tri_block) / kTile);
}

// Item number -> item: inside a group of kPUnitGroup slices the heaviest pairs of all slices first (decode_item of the
// one-block kernel).
__device__ __forceinline__ PairItem decode_pair(const BwdParams& p, int w) {
  PairItem it;
  it.w = w;
  const int n_j = (p.S_k + kTile - 1) / kTile, n_jp = (n_j + 1) / 2;
  const int n_units = p.B * (p.N / p.kv_group);
  const int per_group = n_jp * kPUnitGroup;
  const int grp = w / per_group, within = w % per_group;
  const int g_units = min(kPUnitGroup, n_units - grp * kPUnitGroup);
  const int jp = within / g_units, bh_kv = grp * kPUnitGroup + within % g_units;
  int lo, hi;
  q_range(p, 2 * jp, lo, hi);
  const int n_per = max(0, hi - lo + 1);
  // (the second tile needs no Q tile that the first does not, and the same last one)
  int lo1 = hi + 1, hi1;
  if (2 * jp + 1 < n_j) q_range(p, 2 * jp + 1, lo1, hi1);
  it.n_first = static_cast<uint16_t>(min(n_per, max(0, lo1 - lo)));
  it.bh_kv = static_cast<uint16_t>(bh_kv);
  it.jp = static_cast<uint16_t>(jp);
  it.i_lo = static_cast<uint16_t>(n_per > 0 ? lo : 0);
  it.n_per = static_cast<uint16_t>(n_per);
  it.n_iter = n_per * p.kv_group;
  return it;
}

// A block's k-th item (next_item of the one-block kernel: this wait does not look at the abort flag, because all threads of
// a role must see the same item and the producer always publishes one, after a failure the end marker).
__device__ __forceinline__ PairItem next_pair(PairShared& sh, int k, volatile uint32_t* abort_flag, unsigned int* status,
                                              bool whole_warp = false) {
  uint64_t* bar = &sh.item_full[k & 1];
  const uint32_t parity = (k >> 1) & 1;
  uint32_t polls = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (++polls >= (kWaitPollLimit << 2)) {
      *abort_flag = 1u;
      atomicMax(status, DEV_TIMEOUT_SYNC);
      break;
    }
  }
  const PairItem it = sh.item[k & 1];
  if (whole_warp) __syncwarp();
  if (!whole_warp || (threadIdx.x & 31) == 0) mbar_arrive(&sh.item_empty[k & 1]);
  return it;
}

// P = exp2(s*scale + bias - L) for 32 consecutive queries of one key row, two per instruction; the roundings are those of
// p_fast.
template <bool DIAG>
__device__ __forceinline__ void p_pairwise(const uint32_t (&s)[32], const float* nlse2c, uint64_t scale2, uint64_t bias2, int kv_idx,
                                           int q0, float (&pr)[32]) {
#pragma unroll
  for (int e4 = 0; e4 < 8; ++e4) {
    const ulonglong2 L = *reinterpret_cast<const ulonglong2*>(nlse2c + 4 * e4);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = 4 * e4 + 2 * u;
      float x0, x1;
      f2_unpack(f2_add(f2_fma(f2_pack(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), scale2, bias2), u == 0 ? L.x : L.y), x0, x1);
      const float v0 = ex2(x0), v1 = ex2(x1);
      pr[e] = DIAG && kv_idx > q0 + e ? 0.f : v0;
      pr[e + 1] = DIAG && kv_idx > q0 + e + 1 ? 0.f : v1;
    }
  }
}

}  // namespace

template <bool BF16>
__global__ void __launch_bounds__(kPThreads, 1) __cluster_dims__(2, 1, 1) fa_bwd_pair_kernel(const __grid_constant__ BwdParams p) {
  constexpr uint32_t kColX = 0, kColY = 128, kColDK = 256, kColDV = 384, kColDQ = 32;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;                              // own K tile: two blocks of 64 columns
  uint8_t* sV = sK + kPTile;
  uint8_t* sKm = sV + kPTile;                      // columns [64 rank, +64) of both K tiles
  uint8_t* sQk = sKm + kPTile;                     // rows [64 rank, +64) of the Q tile: two blocks of 64 columns
  uint8_t* sQm = sQk + kPHalf;                     // columns [64 rank, +64) of the Q tile
  uint8_t* sDOk = sQm + kPHalf;
  uint8_t* sDOm = sDOk + kPHalf;
  uint8_t* sDS = sDOm + kPHalf;                    // dS^T: 256 keys x this block's 64 queries; dK leaves through it
  uint8_t* sOut = sDS + kPTile;                    // dS^T of the peer's queries, on its way there
  uint8_t* sStage = sOut + kPHalf;                 // dQ staging: 2 chunks of 64 rows x 32 fp32; dV leaves through it
  PairShared& sh = *reinterpret_cast<PairShared*>(sStage + kPHalf);

  const int tid = threadIdx.x;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const int lane = tid & 31;
  const int rank = static_cast<int>(cluster_rank());
  const ScoreMods& mods = p.mods;
  const int n_kv = p.N / p.kv_group;
  const int n_j = (p.S_k + kTile - 1) / kTile;
  const int total_items = ((n_j + 1) / 2) * p.B * n_kv;

  if ((smem_u32(smem) & 1023u) != 0u) {            // (the same in both blocks)
    if (tid == 0) atomicMax(p.status, DEV_BAD_SMEM_BASE);
    return;
  }

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh.item_full[s], 1);
      mbar_init(&sh.item_empty[s], 1 + kTile + kPComputeThreads);
      mbar_init(&sh.w_full[s], 1);
      mbar_init(&sh.w_empty[s], 1);
    }
    mbar_init(&sh.qk_full, 1); mbar_init(&sh.qm_full, 1); mbar_init(&sh.dok_full, 1); mbar_init(&sh.dom_full, 1);
    mbar_init(&sh.p_half, 16); mbar_init(&sh.p_ready, 16); mbar_init(&sh.s_read, 16);
    mbar_init(&sh.ds_tmem, 16); mbar_init(&sh.ds_peer, 1); mbar_init(&sh.ds_in, 5);
    mbar_init(&sh.dq_read, 8);
    mbar_init(&sh.acc_free, 24);
    mbar_init(&sh.st_full, 1); mbar_init(&sh.dp_full, 1); mbar_init(&sh.dq_full, 1);
    mbar_init(&sh.stats_ready, 4);
    mbar_init(&sh.store_done, 2);
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  cluster_sync();                                  // the peer has started (its tensor memory may be reached), its barriers exist
  if (warp == kPProducerWarp) tmem_alloc_pair(&sh.tmem_base, 512);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();                                  // both have their columns
  tc_fence_after_sync();
  const uint32_t tmem = warp_uniform(sh.tmem_base);
  volatile uint32_t* abort_flag = &sh.abort_flag;
  // one lane of a converged warp arrives on rank 0's barrier for the whole warp
  auto arrive_for_warp = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive_pair(cluster_map(bar, 0));
  };

  if (warp >= kPProducerWarp) {
    // ------------------------------------------------------------------ control warpgroup
    reg_dealloc<kPRegsControl>();
    if (warp == kPProducerWarp) {
      // ---------------------------------------------------------------- TMA producer (and keeper of the work list)
      if (elect_one()) {
        prefetch_tmap(&p.map_q); prefetch_tmap(&p.map_k); prefetch_tmap(&p.map_v); prefetch_tmap(&p.map_do);
        const uint32_t qk_full = cluster_map(&sh.qk_full, 0), qm_full = cluster_map(&sh.qm_full, 0);
        const uint32_t dok_full = cluster_map(&sh.dok_full, 0), dom_full = cluster_map(&sh.dom_full, 0);
        // rank 0 counts the bytes of both blocks' loads
        auto expect = [&](uint64_t* bar, uint32_t bytes) { if (rank == 0) mbar_expect_tx(bar, 2 * bytes); };
        // rows [64 rank, +64) / columns [64 rank, +64) of Q tile i (the maps have boxes of 64 rows x 64 columns)
        auto load_rows = [&](uint8_t* dst, const CUtensorMap* map, uint32_t bar, int i, int h, int b) {
          for (int nb = 0; nb < 2; ++nb) tma_load_4d_pair(dst + nb * 8192, map, bar, nb * 64, i * kTile + rank * 64, h, b);
        };
        auto load_cols = [&](uint8_t* dst, const CUtensorMap* map, uint32_t bar, int i, int h, int b) {
          for (int half = 0; half < 2; ++half) tma_load_4d_pair(dst + half * 8192, map, bar, rank * 64, i * kTile + half * 64, h, b);
        };
        // The number of item k: rank 0 draws it and passes it to rank 1, both decode it for their block's roles.
        auto fetch = [&](int k) {
          const int slot = k & 1;
          if (k >= 2) mbar_wait(&sh.item_empty[slot], ((k - 2) >> 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          int w;
          if (rank == 0) {
            w = *abort_flag == 0u ? static_cast<int>(atomicAdd(p.work_counter, 1u)) : total_items;
            if (k >= 2) mbar_wait_cluster(&sh.w_empty[slot], ((k - 2) >> 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
            cluster_store(cluster_map(&sh.w_next[slot], 1), static_cast<uint32_t>(w));
            mbar_arrive_cluster(cluster_map(&sh.w_full[slot], 1));
          } else {
            const bool ok = mbar_wait_cluster(&sh.w_full[slot], (k >> 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
            w = ok ? static_cast<int>(*const_cast<volatile uint32_t*>(&sh.w_next[slot])) : total_items;
            mbar_arrive_cluster(cluster_map(&sh.w_empty[slot], 0));
          }
          PairItem it;
          if (w < total_items) it = decode_pair(p, w);
          else { it.w = total_items; it.n_iter = 0; it.bh_kv = it.jp = it.i_lo = it.n_per = it.n_first = 0; }
          sh.item[slot] = it;
          mbar_arrive(&sh.item_full[slot]);
          return it;
        };
        PairItem it = fetch(0);
        int g0 = 0;
        for (int k = 0; it.w < total_items; ++k) {
          PairItem nxt;
          bool fetched = false;
          if (it.n_iter > 0 && *abort_flag == 0u) {
            const int b = it.bh_kv / n_kv, h_kv = it.bh_kv % n_kv, h0 = h_kv * p.kv_group;
            const int j0 = 2 * it.jp, j = j0 + rank;
            const int i0 = it.i_lo;
            // first step: K and V with the rows of Q and dO (S^T and dP^T of the item before have finished: waited for below),
            // the columns of K, Q and dO once all of its products have
            expect(&sh.qk_full, kPTile + kPHalf);
            for (int nb = 0; nb < 2; ++nb) tma_load_4d_pair(sK + nb * 16384, &p.map_k, qk_full, nb * 64, j * kTile, h_kv, b);
            load_rows(sQk, &p.map_q, qk_full, i0, h0, b);
            expect(&sh.dok_full, kPTile + kPHalf);
            for (int nb = 0; nb < 2; ++nb) tma_load_4d_pair(sV + nb * 16384, &p.map_v, dok_full, nb * 64, j * kTile, h_kv, b);
            load_rows(sDOk, &p.map_do, dok_full, i0, h0, b);
            if (g0 > 0) mbar_wait(&sh.dq_full, (g0 - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
            if (*abort_flag == 0u) {       // (a barrier must not be told to expect loads twice in one phase)
              expect(&sh.dom_full, kPHalf);
              load_cols(sDOm, &p.map_do, dom_full, i0, h0, b);
              expect(&sh.qm_full, kPTile + kPHalf);
              load_cols(sQm, &p.map_q, qm_full, i0, h0, b);
              for (int t = 0; t < 2; ++t) tma_load_4d_pair(sKm + t * 16384, &p.map_k, qm_full, rank * 64, (j0 + t) * kTile, h_kv, b);
            }
            int i = i0, h = h0, m1 = 0;            // Q tile and head of step n; number of the next step's tile in its head
            for (int n = 0; n < it.n_iter; ++n) {
              const int g = g0 + n;
              const bool more = n + 1 < it.n_iter;
              int h1 = h;
              if (++m1 == it.n_per) { m1 = 0; ++h1; }
              const int i1 = more ? it.i_lo + m1 : 0;
              // S^T(n) has finished: so has dV(n-1), which was issued before it
              mbar_wait(&sh.st_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
              if (*abort_flag != 0u) break;
              if (n > 0) { expect(&sh.dom_full, kPHalf); load_cols(sDOm, &p.map_do, dom_full, i, h, b); }
              if (more) { expect(&sh.qk_full, kPHalf); load_rows(sQk, &p.map_q, qk_full, i1, h1, b); }
              // dP^T(n) has finished, and dK(n-1) before it
              mbar_wait(&sh.dp_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
              if (*abort_flag != 0u) break;
              if (more) { expect(&sh.dok_full, kPHalf); load_rows(sDOk, &p.map_do, dok_full, i1, h1, b); }
              // (dQ(n-1) is seen before dQ(n) can finish, for which this load is needed: a barrier that is two phases ahead of
              // a wait looks like one that has yet to complete)
              if (n > 0) {
                mbar_wait(&sh.dq_full, (g - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
                if (*abort_flag != 0u) break;
                expect(&sh.qm_full, kPHalf);
                load_cols(sQm, &p.map_q, qm_full, i, h, b);
              }
              if (n == (it.n_iter >= 2 ? it.n_iter - 2 : 0)) { nxt = fetch(k + 1); fetched = true; }
              i = i1; h = h1;
            }
            g0 += it.n_iter;
          }
          if (!fetched) nxt = fetch(k + 1);
          it = nxt;
        }
      }
    } else if (warp == kPMmaWarp && rank == 0) {
      // ---------------------------------------------------------------- MMA issuer
      const uint32_t idesc_s = make_idesc(BF16, 256, 128, false, false);     // S^T, dP^T
      const uint32_t idesc_kv = make_idesc(BF16, 256, 128, false, true);     // dV, dK
      const uint32_t idesc_dq = make_idesc(BF16, 128, 128, true, true);      // dQ
      const uint64_t kmajor = make_sdesc_base(16, 1024);
      const uint64_t mnmajor = make_sdesc_base(16384, 1024);
      const uint32_t k_hi = static_cast<uint32_t>(kmajor >> 32), k_lo = static_cast<uint32_t>(kmajor);
      const uint32_t mn_hi = static_cast<uint32_t>(mnmajor >> 32), mn_lo = static_cast<uint32_t>(mnmajor);
      auto lo_of = [](uint32_t base_lo, const uint8_t* ptr) { return base_lo | ((smem_u32(ptr) >> 4) & 0x3fffu); };
      const uint32_t kK = lo_of(k_lo, sK), kV = lo_of(k_lo, sV), kQ = lo_of(k_lo, sQk), kDO = lo_of(k_lo, sDOk);
      const uint32_t mKm = lo_of(mn_lo, sKm), mQ = lo_of(mn_lo, sQm), mDO = lo_of(mn_lo, sDOm), mDS = lo_of(mn_lo, sDS);

      auto scores = [&](uint32_t col, uint32_t a, uint32_t bb, uint64_t* full) {      // S^T or dP^T
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_pair_ss(tmem + col, a + (kk >> 2) * 1024u + (kk & 3) * 2u, k_hi, bb + (kk >> 2) * 512u + (kk & 3) * 2u, k_hi, idesc_s,
                         kk > 0);
          umma_commit_pair(full);
        }
      };
      // queries 16 kk .. + 15 of P^T / dS^T: over columns 0-31 for the first 64 queries, 96-127 for the others
      auto packed_col = [](int kk) { return static_cast<uint32_t>(kk < 4 ? kk * 8 : 64 + kk * 8); };
      // dV or dK += (P^T or dS^T) (dO or Q) over the queries 16 (4 x + y) .. + 15, x < 2, from <= y < to, in the steps that are not
      // alike for both blocks, out of the way of the others: without a part of the second block (both = false), or the first one
      // with a part of it, which starts its sum.
      auto one_by_one = [&](uint32_t d, uint32_t a, uint32_t bb, int from, int to, bool both) {
#pragma unroll 1
        for (int x = 0; x < 2; ++x)
#pragma unroll 1
          for (int y = from; y < to; ++y) {
            const int kk = 4 * x + y;
            if (both && kk > 0) {
              umma_pair_ts(d, a + packed_col(kk), bb + kk * 128u, mn_hi, idesc_kv, true);
            } else {
              umma_pair_ts_one(0, d, a + packed_col(kk), bb + kk * 128u, mn_hi, idesc_kv, true);
              if (both) umma_pair_ts_one(1, d, a + packed_col(kk), bb + kk * 128u, mn_hi, idesc_kv, false);
            }
          }
      };

      int g0 = 0, live = 0;
      for (int k = 0;; ++k) {
        const PairItem it = next_pair(sh, k, abort_flag, p.status, true);
        if (it.w >= total_items) break;
        if (it.n_iter == 0) continue;
        mbar_wait(&sh.qk_full, g0 & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
        if (g0 > 0) mbar_wait(&sh.dq_read, (g0 - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
        scores(kColX, kK, kQ, &sh.st_full);
        mbar_wait(&sh.dok_full, g0 & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
        scores(kColY, kV, kDO, &sh.dp_full);
        bool acc1 = false;
        for (int n = 0, m = 0; n < it.n_iter; ++n) {
          const int g = g0 + n;
          const bool more = n + 1 < it.n_iter;
          const bool both = m >= it.n_first;
          // (before its first step with a part, what the second block sums up is of no account: that step starts over)
          const bool regular = both ? acc1 == (n > 0) : !acc1;
          if (++m == it.n_per) m = 0;
          // dV += P^T dO, in two parts as P^T arrives
          mbar_wait(&sh.dom_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
          if (n == 0 && live > 0) mbar_wait(&sh.acc_free, (live - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            mbar_wait(part == 0 ? &sh.p_half : &sh.p_ready, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
            tc_fence_after_sync();
            if (elect_one()) {
              if (regular) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const int kk = (u >> 1) * 4 + part * 2 + (u & 1);
                  umma_pair_ts(tmem + kColDV, tmem + kColX + packed_col(kk), mDO + kk * 128u, mn_hi, idesc_kv, n > 0 || kk > 0);
                }
              } else {
                one_by_one(tmem + kColDV, tmem + kColX, mDO, part * 2, part * 2 + 2, both);
              }
            }
          }
          // S^T of the next tile, behind the dV that read P^T and once dQ of the tile before this one is out of its columns
          if (more) {
            mbar_wait(&sh.qk_full, (g + 1) & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
            if (g > 0) mbar_wait(&sh.dq_read, (g - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
            scores(kColX, kK, kQ, &sh.st_full);
          }
          // dK += dS^T Q
          mbar_wait(&sh.qm_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
          mbar_wait(&sh.ds_tmem, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          tc_fence_after_sync();
          if (elect_one()) {
            if (regular) {
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)
                umma_pair_ts(tmem + kColDK, tmem + kColY + packed_col(kk), mQ + kk * 128u, mn_hi, idesc_kv, n > 0 || kk > 0);
            } else {
              one_by_one(tmem + kColDK, tmem + kColY, mQ, 0, 4, both);
            }
          }
          acc1 = acc1 || both;
          // dP^T of the next tile behind it
          if (more) {
            mbar_wait(&sh.dok_full, (g + 1) & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
            scores(kColY, kV, kDO, &sh.dp_full);
          }
          // dQ = dS K into X, whose S^T has been read (of the last tile: whose P^T has been consumed and the dQ before drained)
          if (lane == 0 && *abort_flag == 0u) mbar_expect_tx(&sh.ds_in, kPHalf);
          mbar_wait(&sh.ds_in, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          mbar_wait(&sh.ds_peer, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          if (more) mbar_wait(&sh.s_read, (g + 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          else if (g > 0) mbar_wait(&sh.dq_read, (g - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          __syncwarp();
          tc_fence_after_sync();
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_pair_ss(tmem + kColX + kColDQ, mDS + kk * 128u, mn_hi, mKm + kk * 128u, mn_hi, idesc_dq, kk > 0);
            if (both) {
#pragma unroll
              for (int kk = 8; kk < 16; ++kk)
                umma_pair_ss(tmem + kColX + kColDQ, mDS + kk * 128u, mn_hi, mKm + kk * 128u, mn_hi, idesc_dq, true);
            }
            umma_commit_pair(&sh.dq_full);
          }
        }
        g0 += it.n_iter;
        ++live;
      }
    } else if (warp == kPMmaWarp) {
      // ---------------------------------------------------------------- relay of rank 1: its dS^T for dQ is complete -> MMA warp
      const uint32_t ds_peer = cluster_map(&sh.ds_peer, 0);
      int g = 0;
      for (int k = 0;; ++k) {
        const PairItem it = next_pair(sh, k, abort_flag, p.status, true);
        if (it.w >= total_items) break;
        for (int n = 0; n < it.n_iter; ++n, ++g) {
          if (lane == 0 && *abort_flag == 0u) mbar_expect_tx(&sh.ds_in, kPHalf);
          mbar_wait(&sh.ds_in, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          if (lane == 0) mbar_arrive_pair(ds_peer);
        }
      }
    }
  } else if (warp >= kPDrainWarp0) {
    // ------------------------------------------------------------------ drain warpgroup: this block's 64 rows of dQ out of tensor
    // memory (thread t: row t % 64, columns 64 (t / 64) .. + 63), through the swizzled staging area, into the fp32
    // accumulator by TMA reduce-add
    reg_dealloc<kPRegsDrain>();
    const int t = tid - kPDrainWarp0 * 32;
    const int row = t & 63, half = t >> 6;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool elected = (t == 0);
    int g0 = 0;
    for (int k = 0;; ++k) {
      const PairItem it = next_pair(sh, k, abort_flag, p.status);
      if (it.w >= total_items) break;
      const int b = it.bh_kv / n_kv, h_kv = it.bh_kv % n_kv;
      int h = h_kv * p.kv_group, m = 0;
      for (int n = 0; n < it.n_iter; ++n) {
        const int g = g0 + n;
        const int row0 = (it.i_lo + m) * kTile + rank * 64;
        mbar_wait(&sh.dq_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
        tc_fence_after_sync();
        uint32_t dq[2][32];
        tmem_ld32(tmem + lane_base + kColX + kColDQ, dq[0]);
        tmem_ld32(tmem + lane_base + kColX + kColDQ + 32, dq[1]);
        tmem_wait_ld();
        tc_fence_before_sync();
        arrive_for_warp(&sh.dq_read);
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {          // 32 of this thread's columns at a time
          // the staging area is free once the reduce before has read it
          if (elected) tma_store_wait_read();
          named_barrier(3, kTile);
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            *reinterpret_cast<float4*>(sStage + half * 8192u + swz128(row, q4)) =
                make_float4(__uint_as_float(dq[cc][4 * q4]) * p.scale, __uint_as_float(dq[cc][4 * q4 + 1]) * p.scale,
                            __uint_as_float(dq[cc][4 * q4 + 2]) * p.scale, __uint_as_float(dq[cc][4 * q4 + 3]) * p.scale);
          fence_proxy_async_smem();
          named_barrier(3, kTile);
          if (elected) {
            if (row0 < p.S_q)
              for (int x = 0; x < 2; ++x)
                if ((2 * x + cc) * 32 < p.D) tma_reduce_add_4d(&p.map_dq, sStage + x * 8192, (2 * x + cc) * 32, row0, h, b);
            tma_store_commit();
          }
        }
        if (++m == it.n_per) { m = 0; ++h; }
      }
      // dV of the item (16-bit gradients) through the staging area, 64 columns at a time, while the compute warps write dK.
      // Thread t owns key row t here.
      const int j = 2 * it.jp + rank;
      const bool summed = it.n_iter > 0 && (rank == 0 || it.n_first < it.n_per);
      if (!p.grads_f32) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          if ((c & 1) == 0) {
            if (elected) tma_store_wait_read();
            named_barrier(3, kTile);
          }
          uint32_t dv[32];
          if (summed) { tmem_ld32(tmem + lane_base + kColDV + c * 32, dv); tmem_wait_ld(); }
          else {
#pragma unroll
            for (int e = 0; e < 32; ++e) dv[e] = 0u;
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(sStage + swz128(t, (c & 1) * 4 + q4)) =
                make_uint4(pack2<BF16>(__uint_as_float(dv[8 * q4]), __uint_as_float(dv[8 * q4 + 1])),
                           pack2<BF16>(__uint_as_float(dv[8 * q4 + 2]), __uint_as_float(dv[8 * q4 + 3])),
                           pack2<BF16>(__uint_as_float(dv[8 * q4 + 4]), __uint_as_float(dv[8 * q4 + 5])),
                           pack2<BF16>(__uint_as_float(dv[8 * q4 + 6]), __uint_as_float(dv[8 * q4 + 7])));
          if (c == 3) {
            tc_fence_before_sync();
            if (it.n_iter > 0) arrive_for_warp(&sh.acc_free);
          }
          if ((c & 1) != 0) {
            fence_proxy_async_smem();
            named_barrier(3, kTile);
            if (elected) {
              if (j < n_j) tma_store_4d(&p.map_dv, sStage, (c >> 1) * 64, j * kTile, h_kv, b);
              tma_store_commit();
            }
          }
        }
      } else if (it.n_iter > 0) {
        arrive_for_warp(&sh.acc_free);             // fp32 gradients: the compute warps write both tiles out
      }
      g0 += it.n_iter;
    }
    if (elected) tma_store_wait_all();
  } else {
    // ------------------------------------------------------------------ compute warps
    reg_alloc<kPRegsCompute>();
    const int hf = warp >> 2;                      // which half of the query columns / of head_dim
    const int r = (warp & 3) * 32 + lane;          // key row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_x = tmem + lane_base + kColX, t_y = tmem + lane_base + kColY;
    const uint32_t t_pack = hf * 96;               // this half's packed P^T / dS^T columns
    // dS^T of this half's queries goes to the block whose rows of dQ they are: its own dS^T area, or by way of sOut the peer's
    const bool remote = hf != rank;
    uint8_t* my_ds = remote ? sOut : sDS + rank * 16384u;
    const uint32_t warp_rows = (warp & 3) * 4096u;            // this warp's 32 rows of it
    const uint32_t peer_ds = cluster_map(sDS + rank * 16384u + warp_rows, rank ^ 1), peer_ds_in = cluster_map(&sh.ds_in, rank ^ 1);
    const uint64_t scale2 = f2_pack(p.scale_log2, p.scale_log2);
    int g0 = 0;
    uint32_t stores = 0;            // dK stores whose reads have been waited for
    bool ds_stage_busy = false;     // a dK store may still be reading the dS^T areas
    // what an item needs from global memory before its first step is requested before the write-out of the item before it
    float pre_lse = 0.f, pre_dlt = 0.f;
    auto request_first = [&](const PairItem& t) {
      const int b = t.bh_kv / n_kv, h0 = (t.bh_kv % n_kv) * p.kv_group;
      if (t.n_iter <= 0) return;
      if (hf == 0) {
        const int64_t idx = (static_cast<int64_t>(b) * p.N + h0) * p.S_q + min(t.i_lo * kTile + r, p.S_q - 1);
        pre_lse = p.lse[idx];
        pre_dlt = p.delta[idx];
      }
    };
    auto park = [&](int g, int q_row, float lse, float dlt) {       // statistics of step g (threads of half 0)
      const bool q_ok = q_row < p.S_q;
      sh.nlse2[g & 1][r] = q_ok ? -(lse * kLog2e) : -INFINITY;
      sh.ndelta[g & 1][r] = q_ok ? -dlt : 0.f;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.stats_ready);
    };
    PairItem it_next = next_pair(sh, 0, abort_flag, p.status);
    if (it_next.w < total_items) request_first(it_next);
    for (int k = 0; it_next.w < total_items; ++k) {
      const PairItem it = it_next;
      bool next_known = false;
      const int n_per = it.n_per, n_iter = it.n_iter;
      const int b = it.bh_kv / n_kv, h_kv = it.bh_kv % n_kv;
      const int j = 2 * it.jp + rank;
      // Q tile and query head of the step, and of the next one (counted on: divisions here took some 600 clk a step)
      int i = n_iter > 0 ? it.i_lo : 0, h = h_kv * p.kv_group, m1 = 0;
      const int kv_idx = j * kTile + r;
      const float bias = kv_idx < p.S_k ? 0.f : kNegInf;       // -inf removes a key row that does not exist
      const uint64_t bias2 = f2_pack(bias, bias);
      // Statistics go through shared memory, double-buffered by step: parked at the end of the step before (buffer g & 1 was
      // last read for step g - 2, whose dS part every thread finished before dP^T of step g - 1 could be issued).
      if (hf == 0 && n_iter > 0) park(g0, i * kTile + r, pre_lse, pre_dlt);

      for (int n = 0; n < n_iter; ++n) {
        const int q_base = i * kTile;
        const int g = g0 + n;
        const bool more = n + 1 < n_iter;
        int h1 = h;
        if (++m1 == n_per) { m1 = 0; ++h1; }
        const int i1 = more ? it.i_lo + m1 : 0;
        // the next step's statistics, left raw until they are parked
        float nxt_lse = 0.f, nxt_dlt = 0.f;
        if (hf == 0 && more) {
          const int64_t idx = (static_cast<int64_t>(b) * p.N + h1) * p.S_q + min(i1 * kTile + r, p.S_q - 1);
          nxt_lse = p.lse[idx];
          nxt_dlt = p.delta[idx];
        }
        const float* nlse2 = sh.nlse2[g & 1];
        const float* ndlt = sh.ndelta[g & 1];
        const bool diag = mods.causal && (q_base < j * kTile + kTile - 1);

        // ---- P part
        mbar_wait(&sh.stats_ready, g & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
        if (n == 0) named_barrier(4, kPComputeThreads);      // (later steps: no warp parks for g + 1 before all have seen S^T(g))
        mbar_wait(&sh.st_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
        tc_fence_after_sync();
        float pr[2][32];
        {
          uint32_t s[2][32];
          tmem_ld32(t_x + (hf * 2) * 32, s[0]);
          tmem_ld32(t_x + (hf * 2 + 1) * 32, s[1]);
          tmem_wait_ld();
          tc_fence_before_sync();
          arrive_for_warp(&sh.s_read);
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int c = hf * 2 + cc;
            if (diag) p_pairwise<true>(s[cc], nlse2 + c * 32, scale2, bias2, kv_idx, q_base + c * 32, pr[cc]);
            else p_pairwise<false>(s[cc], nlse2 + c * 32, scale2, bias2, kv_idx, q_base + c * 32, pr[cc]);
            uint32_t pk[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) pk[e] = pack2<BF16>(pr[cc][2 * e], pr[cc][2 * e + 1]);
            tmem_st16(t_x + t_pack + cc * 16, pk);
            tmem_wait_st();
            tc_fence_before_sync();
            arrive_for_warp(cc == 0 ? &sh.p_half : &sh.p_ready);
          }
        }

        // ---- dS part: dS^T = P^T * (dP^T - D)
        if (ds_stage_busy) {       // first step after a write-out: both blocks' dK stores have read their dS^T areas
          if (tid == 0) {
            tma_store_wait_read();
            mbar_arrive_pair(cluster_map(&sh.store_done, 0));
            mbar_arrive_pair(cluster_map(&sh.store_done, 1));
          }
          mbar_wait(&sh.store_done, stores & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          __syncwarp();
          ++stores;
          ds_stage_busy = false;
        }
        mbar_wait(&sh.dp_full, g & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
        tc_fence_after_sync();
        uint32_t ds[2][16];
        {
          uint32_t dp[2][32];
          tmem_ld32(t_y + (hf * 2) * 32, dp[0]);
          tmem_ld32(t_y + (hf * 2 + 1) * 32, dp[1]);
          tmem_wait_ld();
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int c = hf * 2 + cc;
#pragma unroll
            for (int e4 = 0; e4 < 8; ++e4) {
              const ulonglong2 nd = *reinterpret_cast<const ulonglong2*>(ndlt + c * 32 + 4 * e4);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int e = 4 * e4 + 2 * u;
                float d0, d1;
                f2_unpack(f2_mul(f2_pack(pr[cc][e], pr[cc][e + 1]),
                                 f2_add(f2_pack(__uint_as_float(dp[cc][e]), __uint_as_float(dp[cc][e + 1])), u == 0 ? nd.x : nd.y)),
                          d0, d1);
                ds[cc][e >> 1] = pack2<BF16>(d0, d1);
              }
            }
            tmem_st16(t_y + t_pack + cc * 16, ds[cc]);
          }
        }
        tmem_wait_st();
        tc_fence_before_sync();
        arrive_for_warp(&sh.ds_tmem);
        // into shared memory for dQ, once the dQ before has read what is there (in both blocks, so sOut has been copied too)
        if (g > 0) mbar_wait(&sh.dq_full, (g - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(my_ds + swz128(r, cc * 4 + q4)) =
                make_uint4(ds[cc][4 * q4], ds[cc][4 * q4 + 1], ds[cc][4 * q4 + 2], ds[cc][4 * q4 + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        // (after a failure neither: without the barrier's owner they would overrun its phase)
        if (lane == 0 && *abort_flag == 0u) {
          if (remote) cluster_copy_async(peer_ds, sOut + warp_rows, 4096u, peer_ds_in);
          else mbar_arrive(&sh.ds_in);
        }
        if (hf == 0 && more) park(g + 1, i1 * kTile + r, nxt_lse, nxt_dlt);
        // the next item has been published since this item's last step but one: request what its first step needs
        if (!more) {
          it_next = next_pair(sh, k + 1, abort_flag, p.status);
          next_known = true;
          if (it_next.w < total_items) request_first(it_next);
        }
        i = i1; h = h1;
      }

      // write-out of dK (scaled) and, with fp32 gradients, dV; each half writes its half of head_dim
      const bool summed = n_iter > 0 && (rank == 0 || it.n_first < n_per);      // (else nothing has been written there)
      if (n_iter > 0) mbar_wait(&sh.dq_full, (g0 + n_iter - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
      tc_fence_after_sync();
      if (!next_known) {      // (an item without steps)
        it_next = next_pair(sh, k + 1, abort_flag, p.status);
        if (it_next.w < total_items) request_first(it_next);
      }
      if (!p.grads_f32) {
        // through this block's dS^T area (the last dQ has read it) and one TMA store
        if (ds_stage_busy) {     // (an item without steps right after another write-out)
          if (tid == 0) tma_store_wait_read();
          named_barrier(4, kPComputeThreads);
        }
#pragma unroll 1
        for (int cq = 0; cq < 2; ++cq) {
          const int c = hf * 2 + cq;
          uint32_t v[32];
          if (summed) { tmem_ld32(tmem + lane_base + kColDK + c * 32, v); tmem_wait_ld(); }
          else {
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = 0u;
          }
          uint8_t* blk = sDS + (c >> 1) * 16384u;
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack2<BF16>(__uint_as_float(v[8 * q4 + 2 * e]) * p.scale, __uint_as_float(v[8 * q4 + 2 * e + 1]) * p.scale);
            *reinterpret_cast<uint4*>(blk + swz128(r, (c & 1) * 4 + q4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        tc_fence_before_sync();
        if (n_iter > 0) arrive_for_warp(&sh.acc_free);
        fence_proxy_async_smem();
        named_barrier(4, kPComputeThreads);
        if (tid == 0) {
          if (j < n_j)
            for (int nb = 0; nb < 2; ++nb) tma_store_4d(&p.map_dk, sDS + nb * 16384, nb * 64, j * kTile, h_kv, b);
          tma_store_commit();
        }
        ds_stage_busy = true;
      } else {
        const bool row_ok = kv_idx < p.S_k;
        const int64_t row_off = (static_cast<int64_t>(it.bh_kv) * p.S_k + kv_idx) * p.D;
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          const uint32_t t_src = tmem + lane_base + (which == 0 ? kColDK : kColDV);
          const float mul = which == 0 ? p.scale : 1.0f;
          float* dst = reinterpret_cast<float*>(which == 0 ? p.dk : p.dv) + row_off;
#pragma unroll 1
          for (int cq = 0; cq < 2; ++cq) {
            const int c = hf * 2 + cq;
            uint32_t v[32];
            if (summed) { tmem_ld32(t_src + c * 32, v); tmem_wait_ld(); }
            else {
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = 0u;
            }
            if (!row_ok) continue;
#pragma unroll
            for (int q4 = 0; q4 < 8; ++q4) {
              const int col = c * 32 + q4 * 4;
              if (col + 4 <= p.D)
                *reinterpret_cast<float4*>(dst + col) =
                    make_float4(__uint_as_float(v[4 * q4]) * mul, __uint_as_float(v[4 * q4 + 1]) * mul,
                                __uint_as_float(v[4 * q4 + 2]) * mul, __uint_as_float(v[4 * q4 + 3]) * mul);
            }
          }
        }
        tc_fence_before_sync();
        if (n_iter > 0) arrive_for_warp(&sh.acc_free);
      }
      g0 += n_iter;
    }
    if (ds_stage_busy && tid == 0) tma_store_wait_read();   // shared memory must outlive the last store's read of it
  }

  linger_after_abort(abort_flag);
  __syncthreads();
  __syncwarp();
  cluster_sync();                                  // neither block leaves while the other may still reach its memory
  if (warp == kPProducerWarp) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem, 512);
  }
  __syncwarp();
  cluster_sync();                                  // (nor while the other frees its half of the pair's tensor memory)
}

cudaError_t launch_fa_bwd_pair(const BwdParams& p, bool bf16, int sm_count, cudaStream_t stream) {
  const long long items = static_cast<long long>(((p.S_k + kTile - 1) / kTile + 1) / 2) * p.B * (p.N / p.kv_group);
  const long long pairs = items < sm_count / 2 ? items : sm_count / 2;
  void (*kern)(const BwdParams) = bf16 ? fa_bwd_pair_kernel<true> : fa_bwd_pair_kernel<false>;
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), kPSmem);
  if (e != cudaSuccess) return e;
  kern<<<static_cast<unsigned>(2 * pairs), kPThreads, kPSmem, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace acct
