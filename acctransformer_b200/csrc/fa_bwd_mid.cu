// FlashAttention-2 backward for head_dim in (128, 160] on sm_100a.
//
// Up to 160 columns the dK and dV accumulators of a 128-row K/V tile (2 x 160 columns of tensor memory) leave room for
// S^T, dP^T and dQ^T of 64 queries, and three 64-column blocks of K, V and of two stages of Q and dO fit shared memory:
// one CTA does the whole width, where the kernel for head_dim up to 256 has two that both recompute S^T and dP^T over 256
// padded columns with single-buffered Q and dO.  Per step of 64 queries (m), tensor-pipe order
//   dP^T(m) | dV(m), S^T(m+1) | dK(m), dQ^T(m)
//   S^T  = K Q^T, dP^T = V dO^T            10 steps of 16 columns, M = 128 keys, N = 64 queries
//   dV  += (P^T*M) dO, dK += dS^T Q        N = 160, A from tensor memory (written over S^T / dP^T), B MN-major
//   dQ^T = K^T dS^T                        two M = 128 blocks of head_dim columns: 0-127 into columns of their own,
//                                          128-159 over dP^T (dS^T in it has been consumed by dK by then)
// Tensor memory: S^T 64 | dP^T 64 | dQ^T 64 | dK 160 | dV 160.  Shared memory: K, V 2 x 48 KB, Q and dO two stages of
// 24 KB each, dS^T 16 KB, dQ staging 4 x 4 KB (one per drain warp, which then need no barrier among themselves).
// What bounds it: the chain of hand-offs of a step, as in the narrow kernel, with half the queries per step.
// 8 x 8 heads of 160, 1 024 tokens, forward and backward: 957 us with the split-width kernel, 300 us with this one (backward 194).
//
// Warp roles: warps 0-7 compute (thread = one key row x 32 of the 64 queries), warps 8-11 drain dQ^T (warp w = head_dim
// columns 32w..32w+31, warp 0 also 128..159), warp 12 TMA producer, warp 13 MMA issuer.  MODE 0: no mask tensor, dropout
// or row groups; 1: in-kernel dropout; 2: everything, element by element.
//
// Follows the reference's backward (train/acctransformer/flash_attention/ops/flash_attention/
// flash_attention_bwd.py:259-415) like the narrow kernel does.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fa_bwd_helpers.cuh"
#include "fa_common.cuh"
#include "fa_kernels.cuh"
#include "ptx.cuh"

namespace acct {

namespace {

constexpr int kMThreads = 512;
constexpr int kMComputeThreads = 256;
constexpr int kMDrainWarp0 = 8, kMProducerWarp = 12, kMMmaWarp = 13;
constexpr int kSub = 64;                          // query rows per step
constexpr int kMRegsCompute = 152, kMRegsDrain = 152, kMRegsControl = 56;
constexpr int kMWidth = 160;                      // head_dim columns of the accumulators
constexpr uint32_t kMKvBytes = 3 * 16384u;        // 128 rows x 192 columns, three 64-column blocks
constexpr uint32_t kMSubBytes = 3 * 8192u;        // 64 rows x 192 columns
constexpr int kMStages = 2;                       // of Q and of dO

struct MidShared {
  uint64_t kv_full;
  uint64_t q_full[kMStages], q_empty[kMStages];    // q_empty: drain (on dq_full) -> producer
  uint64_t do_full[kMStages], do_empty[kMStages];  // do_empty: the dV product (and dP^T before it) has finished
  uint64_t st_full, dp_full;       // MMA -> compute
  uint64_t p_ready, ds_ready;      // compute -> MMA
  uint64_t dq_full, dq_read;       // MMA -> drain -> MMA
  uint64_t stats_ready;
  uint32_t tmem_base;
  volatile uint32_t abort_flag;
  alignas(16) float lse2[2][kSub];
  alignas(16) float delta[2][kSub];
};
constexpr size_t kMSmem = 2 * kMKvBytes + 2 * kMStages * kMSubBytes + 2 * 16384 + sizeof(MidShared);
static_assert(kMSmem <= 232448, "shared memory of a thread block");

}  // namespace

template <bool BF16, int MODE>
__global__ void __launch_bounds__(kMThreads, 1) fa_bwd_mid_kernel(const __grid_constant__ BwdParams p) {
  constexpr uint32_t kColST = 0, kColDP = 64, kColDQ = 128, kColDK = 192, kColDV = 192 + kMWidth;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + kMKvBytes;
  uint8_t* sQ = sV + kMKvBytes;                    // kMStages sub-tiles; dK leaves through them at the end
  uint8_t* sDO = sQ + kMStages * kMSubBytes;       // kMStages sub-tiles; dV leaves through them
  uint8_t* sDS = sDO + kMStages * kMSubBytes;      // dS^T: 128 key rows x 64 queries (one 128-byte-row block)
  uint8_t* sStage = sDS + 16384;                   // dQ^T staging: per drain warp 32 query rows x 32 fp32
  MidShared& sh = *reinterpret_cast<MidShared*>(sStage + 16384);

  const int tid = threadIdx.x;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const int lane = tid & 31;
  const int n_kv = p.N / p.kv_group;
  const int bh_kv = blockIdx.y;
  const int b = bh_kv / n_kv, h_kv = bh_kv % n_kv;
  const int j = blockIdx.x;
  const ScoreMods& mods = p.mods;

  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) atomicMax(p.status, DEV_BAD_SMEM_BASE);
    return;
  }

  int kv_len = p.S_k;
  if (mods.seq_lens != nullptr) kv_len = min(p.S_k, max(0, mods.seq_lens[b]));

  // 128-row Q tiles i that need K/V tile j (same predicate as the narrow kernel), each walked as two 64-row steps
  const int tiles_q = (p.S_q + kTile - 1) / kTile;
  int i_lo = 0, i_hi = tiles_q - 1;
  if (mods.next_block_num < 65536) i_lo = max(i_lo, j - mods.next_block_num);
  if (mods.prev_block_num < 65536) i_hi = min(i_hi, j + mods.prev_block_num);
  if (mods.causal) i_lo = max(i_lo, j);
  if (mods.tri_block > 0) i_lo = max(i_lo, (((j * kTile) / mods.tri_block) * mods.tri_block) / kTile);
  if (j * kTile >= kv_len) i_hi = i_lo - 1;
  const int n_per = max(0, i_hi - i_lo + 1);
  const int per_head = 2 * n_per;                  // steps per query head
  const int n_steps = per_head * p.kv_group;
  auto head_of = [&](int m) { return h_kv * p.kv_group + m / max(per_head, 1); };
  auto tile_of = [&](int m) { return i_lo + (m % max(per_head, 1)) / 2; };
  auto qbase_of = [&](int m) { return tile_of(m) * kTile + (m & 1) * kSub; };

  if (tid == 0) {
    mbar_init(&sh.kv_full, 1);
    for (int s = 0; s < kMStages; ++s) {
      mbar_init(&sh.q_full[s], 1); mbar_init(&sh.q_empty[s], 1);
      mbar_init(&sh.do_full[s], 1); mbar_init(&sh.do_empty[s], 1);
    }
    mbar_init(&sh.st_full, 1); mbar_init(&sh.dp_full, 1);
    mbar_init(&sh.p_ready, kMComputeThreads); mbar_init(&sh.ds_ready, kMComputeThreads);
    mbar_init(&sh.dq_full, 1); mbar_init(&sh.dq_read, 4);
    mbar_init(&sh.stats_ready, kSub);
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kMProducerWarp) { tmem_alloc(&sh.tmem_base, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = warp_uniform(sh.tmem_base);
  volatile uint32_t* abort_flag = &sh.abort_flag;

  if (warp >= kMProducerWarp) {
    reg_dealloc<kMRegsControl>();
    if (warp == kMProducerWarp) {
      // ---------------------------------------------------------------- TMA producer
      if (n_steps > 0 && elect_one()) {
        prefetch_tmap(&p.map_q); prefetch_tmap(&p.map_k); prefetch_tmap(&p.map_v); prefetch_tmap(&p.map_do);
        prefetch_tmap(&p.map_dq);
        mbar_expect_tx(&sh.kv_full, 2 * kMKvBytes);
        for (int nb = 0; nb < 3; ++nb) tma_load_4d(sK + nb * 16384, &p.map_k, &sh.kv_full, nb * 64, j * kTile, h_kv, b);
        for (int nb = 0; nb < 3; ++nb) tma_load_4d(sV + nb * 16384, &p.map_v, &sh.kv_full, nb * 64, j * kTile, h_kv, b);
        for (int m = 0; m < n_steps; ++m) {
          const int q0 = qbase_of(m), h = head_of(m), st = m % kMStages;
          const uint32_t reuse_parity = ((m / kMStages) - 1) & 1;
          uint8_t* dstq = sQ + st * kMSubBytes;
          uint8_t* dstd = sDO + st * kMSubBytes;
          if (m >= kMStages) mbar_wait(&sh.q_empty[st], reuse_parity, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          mbar_expect_tx(&sh.q_full[st], kMSubBytes);
          for (int nb = 0; nb < 3; ++nb) tma_load_4d(dstq + nb * 8192, &p.map_q, &sh.q_full[st], nb * 64, q0, h, b);
          if (m >= kMStages) mbar_wait(&sh.do_empty[st], reuse_parity, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          mbar_expect_tx(&sh.do_full[st], kMSubBytes);
          for (int nb = 0; nb < 3; ++nb) tma_load_4d(dstd + nb * 8192, &p.map_do, &sh.do_full[st], nb * 64, q0, h, b);
        }
      }
    } else if (warp == kMMmaWarp) {
      // ---------------------------------------------------------------- MMA issuer
      if (n_steps > 0) {
        const uint32_t idesc_s = make_idesc(BF16, 128, kSub, false, false);    // S^T, dP^T
        const uint32_t idesc_kv = make_idesc(BF16, 128, kMWidth, false, true);  // dV, dK
        const uint32_t idesc_dq = make_idesc(BF16, 128, kSub, true, true);     // dQ^T, one block of 128 columns
        const uint64_t kmajor = make_sdesc_base(16, 1024);
        const uint64_t mn_kv = make_sdesc_base(16384, 1024);    // 64-column blocks of a 128-row tile
        const uint64_t mn_sub = make_sdesc_base(8192, 1024);    // 64-column blocks of a 64-row sub-tile
        const uint32_t k_hi = static_cast<uint32_t>(kmajor >> 32), k_lo = static_cast<uint32_t>(kmajor);
        const uint32_t mkv_hi = static_cast<uint32_t>(mn_kv >> 32), mkv_lo = static_cast<uint32_t>(mn_kv);
        const uint32_t msub_hi = static_cast<uint32_t>(mn_sub >> 32), msub_lo = static_cast<uint32_t>(mn_sub);
        auto lo_of = [](uint32_t base_lo, const uint8_t* ptr) { return base_lo | ((smem_u32(ptr) >> 4) & 0x3fffu); };
        const uint32_t kK = lo_of(k_lo, sK), kV = lo_of(k_lo, sV), kQ0 = lo_of(k_lo, sQ), kDO0 = lo_of(k_lo, sDO);
        const uint32_t mK = lo_of(mkv_lo, sK);                       // A operand of dQ^T
        const uint32_t mQ0 = lo_of(msub_lo, sQ), mDO0 = lo_of(msub_lo, sDO), mDS = lo_of(msub_lo, sDS);
        constexpr uint32_t kSubUnits = kMSubBytes >> 4;
        constexpr int kSteps = kMWidth / 16;

        auto issue_st = [&](int st) {   // S^T = K Q^T
          const uint32_t kQ = kQ0 + st * kSubUnits;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk)
              umma_ss_lohi(tmem + kColST, kK + (kk >> 2) * 1024u + (kk & 3) * 2u, k_hi, kQ + (kk >> 2) * 512u + (kk & 3) * 2u,
                           k_hi, idesc_s, kk > 0);
            umma_commit(&sh.st_full);
          }
        };
        mbar_wait(&sh.kv_full, 0, abort_flag, p.status, DEV_TIMEOUT_TMA);
        mbar_wait(&sh.q_full[0], 0, abort_flag, p.status, DEV_TIMEOUT_TMA);
        tc_fence_after_sync();
        issue_st(0);
        for (int m = 0; m < n_steps; ++m) {
          const uint32_t par = m & 1;
          const int st = m % kMStages, stn = (m + 1) % kMStages;
          // dP^T = V dO^T, over the columns that the drain has taken dQ^T of the step before out of
          mbar_wait(&sh.do_full[st], (m / kMStages) & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
          if (m > 0) mbar_wait(&sh.dq_read, (m - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t kDO = kDO0 + st * kSubUnits;
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk)
              umma_ss_lohi(tmem + kColDP, kV + (kk >> 2) * 1024u + (kk & 3) * 2u, k_hi, kDO + (kk >> 2) * 512u + (kk & 3) * 2u,
                           k_hi, idesc_s, kk > 0);
            umma_commit(&sh.dp_full);
          }
          // dV += P^T dO: P^T of queries [32h, 32h+32) sits in S^T columns [32h, 32h+16)
          mbar_wait(&sh.p_ready, par, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t mDO = mDO0 + st * kSubUnits;
#pragma unroll
            for (int kk = 0; kk < kSub / 16; ++kk)
              umma_ts_lohi(tmem + kColDV, tmem + kColST + (kk >> 1) * 32 + (kk & 1) * 8, mDO + kk * 128u, msub_hi, idesc_kv,
                           m > 0 || kk > 0);
            umma_commit(&sh.do_empty[st]);
          }
          if (m + 1 < n_steps) {
            mbar_wait(&sh.q_full[stn], ((m + 1) / kMStages) & 1, abort_flag, p.status, DEV_TIMEOUT_TMA);
            tc_fence_after_sync();
            issue_st(stn);
          }
          // dK += dS^T Q, then dQ^T = K^T dS^T: columns 128-159 go over dP^T (the rows of that block past 191 are
          // whatever follows K in shared memory: lanes that nobody reads)
          mbar_wait(&sh.ds_ready, par, abort_flag, p.status, DEV_TIMEOUT_SYNC);
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t mQ = mQ0 + st * kSubUnits;
#pragma unroll
            for (int kk = 0; kk < kSub / 16; ++kk)
              umma_ts_lohi(tmem + kColDK, tmem + kColDP + (kk >> 1) * 32 + (kk & 1) * 8, mQ + kk * 128u, msub_hi, idesc_kv,
                           m > 0 || kk > 0);
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)
              umma_ss_lohi(tmem + kColDQ, mK + kk * 128u, mkv_hi, mDS + kk * 128u, msub_hi, idesc_dq, kk > 0);
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)
              umma_ss_lohi(tmem + kColDP, mK + 2048u + kk * 128u, mkv_hi, mDS + kk * 128u, msub_hi, idesc_dq, kk > 0);
            umma_commit(&sh.dq_full);
          }
        }
      }
    }
  } else if (warp >= kMDrainWarp0) {
    // ------------------------------------------------------------------ drain: dQ^T (lane = head_dim column, 64 query
    // columns) through 4 KB of swizzled staging per warp, 32 queries at a time, into the fp32 accumulator by TMA
    // reduce-add.  Warp w owns head_dim columns 32w .. 32w+31, warp 0 also 128 .. 159.
    reg_alloc<kMRegsDrain>();
    const int w = warp & 3;
    const uint32_t lanes = static_cast<uint32_t>(w * 32) << 16;
    uint8_t* stage = sStage + w * 4096;
    uint8_t* dst = stage + (lane & 3) * 4;
    const uint32_t ch = lane >> 2;
    for (int m = 0; m < n_steps; ++m) {
      const int q0 = qbase_of(m);
      const int h = head_of(m);
      mbar_wait(&sh.dq_full, m & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
      tc_fence_after_sync();
      if (w == 3 && lane == 0) mbar_arrive(&sh.q_empty[m % kMStages]);    // every product of the step has finished
      uint32_t dq[4][32];
      tmem_ld32(tmem + lanes + kColDQ, dq[0]);
      tmem_ld32(tmem + lanes + kColDQ + 32, dq[1]);
      if (w == 0) {
        tmem_ld32(tmem + kColDP, dq[2]);
        tmem_ld32(tmem + kColDP + 32, dq[3]);
      }
      tmem_wait_ld();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.dq_read);
#pragma unroll
      for (int rd = 0; rd < 4; ++rd) {
        if (rd < 2 || w == 0) {
          if (lane == 0) tma_store_wait_read();      // the piece before has been read out of the staging area
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 32; ++e)               // query row e of the piece; (row & 7) == (e & 7)
            *reinterpret_cast<float*>(dst + e * 128 + ((ch ^ (e & 7)) << 4)) = __uint_as_float(dq[rd][e]) * p.scale;
          fence_proxy_async_smem();
          __syncwarp();
          const int col = rd < 2 ? w * 32 : 128, row = q0 + (rd & 1) * 32;
          if (lane == 0) {
            if (col < p.D && row < p.S_q) tma_reduce_add_4d(&p.map_dq, stage, col, row, h, b);
            tma_store_commit();
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_all();
  } else {
    // ------------------------------------------------------------------ compute warps
    reg_alloc<kMRegsCompute>();
    const int hf = warp >> 2;                            // which 32 of the step's 64 queries
    const int r = (warp & 3) * 32 + lane;                // key row inside the tile
    const int kv_idx = j * kTile + r;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_st = tmem + lane_base + kColST + hf * 32;
    const uint32_t t_dp = tmem + lane_base + kColDP + hf * 32;
    const bool kv_ok = kv_idx < kv_len;
    const int kv_c = min(kv_idx, p.S_k - 1);
    auto bias_of = [&](int h) {
      float v = kNegInf;
      if (kv_ok) {
        v = 0.f;
        if (mods.alibi != nullptr) v = load16<BF16>(mods.alibi, (static_cast<int64_t>(b) * p.N + h) * p.S_k + kv_idx) * kLog2e;
        else if (mods.alibi_slopes != nullptr) v = mods.alibi_slopes[h] * static_cast<float>(kv_idx) * kLog2e;
      }
      return v;
    };
    float bias = kNegInf;
    const bool stats_thread = hf == 0 && r < kSub;      // warps 0 and 1: one thread per query of the step

    float nxt_lse = 0.f, nxt_dlt = 0.f;
    bool nxt_ok = false;
    if (stats_thread && n_steps > 0) {
      const int q_row = qbase_of(0) + r;
      const bool q_ok = q_row < p.S_q;
      const int64_t idx = (static_cast<int64_t>(b) * p.N + head_of(0)) * p.S_q + min(q_row, p.S_q - 1);
      sh.lse2[0][r] = q_ok ? p.lse[idx] * kLog2e : INFINITY;
      sh.delta[0][r] = q_ok ? p.delta[idx] : 0.f;
      mbar_arrive(&sh.stats_ready);
    }

    for (int m = 0; m < n_steps; ++m) {
      [[maybe_unused]] const int i = tile_of(m);
      const int q0 = qbase_of(m) + hf * 32;              // first of this thread's 32 queries
      [[maybe_unused]] const int bh = b * p.N + head_of(m);
      if (m % max(per_head, 1) == 0) bias = bias_of(head_of(m));
      // ---- P part
      mbar_wait(&sh.st_full, m & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
      tc_fence_after_sync();
      if (stats_thread && m > 0) {
        sh.lse2[m & 1][r] = nxt_ok ? nxt_lse * kLog2e : INFINITY;
        sh.delta[m & 1][r] = nxt_ok ? nxt_dlt : 0.f;
        mbar_arrive(&sh.stats_ready);
      }
      if (stats_thread && m + 1 < n_steps) {
        const int q_row = qbase_of(m + 1) + r;
        nxt_ok = q_row < p.S_q;
        const int64_t idx = (static_cast<int64_t>(b) * p.N + head_of(m + 1)) * p.S_q + min(q_row, p.S_q - 1);
        nxt_lse = p.lse[idx];
        nxt_dlt = p.delta[idx];
      }
      mbar_wait(&sh.stats_ready, m & 1, abort_flag, p.status, DEV_TIMEOUT_SYNC);
      const float* lse2 = sh.lse2[m & 1] + hf * 32;
      const float* dlt = sh.delta[m & 1] + hf * 32;
      [[maybe_unused]] const bool use_mask = (mods.mask_kind == 1) || (mods.mask_kind == 2 && i == j);
      const bool diag = mods.causal && (q0 < j * kTile + kTile - 1);

      uint32_t s[32];
      tmem_ld32(t_st, s);
      // dropout: bit e = query q0 + e keeps this key
      [[maybe_unused]] uint32_t keep_bits = 0xffffffffu;
      if constexpr (MODE != 0) if (mods.drop_philox != 0) keep_bits = philox_keep_column(mods, bh, q0, p.S_q - 1, kv_idx, lane);
      tmem_wait_ld();
      float pr[32];
      uint32_t pk[16];
      if constexpr (MODE == 2) {
  #pragma unroll
        for (int e = 0; e < 32; ++e) {
          const int q = q0 + e;
          float x = fmaf(__uint_as_float(s[e]), p.scale_log2, bias) - lse2[e];
          if (use_mask) {
            const int qc = min(q, p.S_q - 1);
            const float mv = mods.mask_kind == 1
                                 ? load_mask_value(mods.mask, mods.mask_dtype,
                                                   (static_cast<int64_t>(mods.mask_batch > 1 ? b : 0) * p.S_q + qc) * p.S_k + kv_c)
                                 : load_mask_value(mods.mask, mods.mask_dtype, static_cast<int64_t>(q - i * kTile) * kTile + r);
            x = fmaf(mv, -10000.0f * kLog2e, x);
          }
          float v = ex2(x);
          if (diag && kv_idx > q) v = 0.f;
          if (mods.tri_block > 0 && kv_idx >= (q / mods.tri_block + 1) * mods.tri_block) v = 0.f;
          pr[e] = v;
        }
      } else {
        if (diag) p_fast<true>(s, lse2, p.scale_log2, bias, kv_idx, q0, pr);
        else p_fast<false>(s, lse2, p.scale_log2, bias, kv_idx, q0, pr);
      }
      [[maybe_unused]] float fac[32];     // dropout factors, 0 or the rescale value (1 without dropout)
      if constexpr (MODE == 0) {
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack2<BF16>(pr[2 * e], pr[2 * e + 1]);
      } else {
        if (MODE == 2 && mods.drop != nullptr) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            fac[e] = load_mask_value(mods.drop, mods.drop_dtype,
                                     (static_cast<int64_t>(bh) * p.S_q + min(q0 + e, p.S_q - 1)) * p.S_k + kv_c) * mods.drop_scale;
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) fac[e] = ((keep_bits >> e) & 1u) ? mods.drop_scale : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack2<BF16>(pr[2 * e] * fac[2 * e], pr[2 * e + 1] * fac[2 * e + 1]);
      }
      tmem_st16(t_st, pk);     // over the first 16 of this half's own 32 S^T columns
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&sh.p_ready);

      // ---- dS part
      mbar_wait(&sh.dp_full, m & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
      tc_fence_after_sync();
      uint32_t dp[32];
      tmem_ld32(t_dp, dp);
      tmem_wait_ld();
      uint32_t ds[16];
#pragma unroll
      for (int e4 = 0; e4 < 8; ++e4) {
        const float4 Dl = *reinterpret_cast<const float4*>(dlt + 4 * e4);
        const float dl[4] = {Dl.x, Dl.y, Dl.z, Dl.w};
        float d[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = 4 * e4 + u;
          if constexpr (MODE == 0) d[u] = pr[e] * (__uint_as_float(dp[e]) - dl[u]);
          else d[u] = pr[e] * fmaf(__uint_as_float(dp[e]), fac[e], -dl[u]);
        }
        ds[2 * e4] = pack2<BF16>(d[0], d[1]);
        ds[2 * e4 + 1] = pack2<BF16>(d[2], d[3]);
      }
      tmem_st16(t_dp, ds);     // A operand of the dK product
#pragma unroll
      for (int g = 0; g < 4; ++g)   // and row r of the dS^T block in shared memory (B operand of dQ^T)
        *reinterpret_cast<uint4*>(sDS + swz128(r, hf * 4 + g)) = make_uint4(ds[4 * g], ds[4 * g + 1], ds[4 * g + 2], ds[4 * g + 3]);
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(&sh.ds_ready);
    }

    // epilogue: warps 0-3 write dK (scaled), warps 4-7 dV, one key row per thread: 16-bit gradients through the Q and dO
    // stages, which every product has finished reading, and one TMA store each (it drops rows past S_k and columns past D)
    if (n_steps > 0) mbar_wait(&sh.dq_full, (n_steps - 1) & 1, abort_flag, p.status, DEV_TIMEOUT_MMA);
    tc_fence_after_sync();
    const uint32_t t_src = tmem + lane_base + (hf == 0 ? kColDK : kColDV);
    const float mul = hf == 0 ? p.scale : 1.0f;
    uint8_t* stage = hf == 0 ? sQ : sDO;
    float* dst = reinterpret_cast<float*>(hf == 0 ? p.dk : p.dv) + (static_cast<int64_t>(bh_kv) * p.S_k + kv_idx) * p.D;
#pragma unroll 1
    for (int c = 0; c < kMWidth / 32; ++c) {
      uint32_t v[32];
      if (n_steps > 0) { tmem_ld32(t_src + c * 32, v); tmem_wait_ld(); }
      else {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = 0u;
      }
      if (p.grads_f32) {
        if (kv_idx >= p.S_k) continue;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const int col = c * 32 + g * 4;
          if (col + 4 <= p.D)
            *reinterpret_cast<float4*>(dst + col) =
                make_float4(__uint_as_float(v[4 * g]) * mul, __uint_as_float(v[4 * g + 1]) * mul,
                            __uint_as_float(v[4 * g + 2]) * mul, __uint_as_float(v[4 * g + 3]) * mul);
        }
      } else {
        uint8_t* blk = stage + (c >> 1) * 16384u;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t wv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            wv[e] = pack2<BF16>(__uint_as_float(v[8 * g + 2 * e]) * mul, __uint_as_float(v[8 * g + 2 * e + 1]) * mul);
          *reinterpret_cast<uint4*>(blk + swz128(r, (c & 1) * 4 + g)) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        }
      }
    }
    if (!p.grads_f32) {
      fence_proxy_async_smem();
      named_barrier(1 + hf, 128);
      if (r == 0) {
        for (int nb = 0; nb < 3; ++nb)
          if (nb * 64 < p.D) tma_store_4d(hf == 0 ? &p.map_dk : &p.map_dv, stage + nb * 16384, nb * 64, j * kTile, h_kv, b);
        tma_store_commit();
        tma_store_wait_read();      // shared memory must outlive the store's read of it
      }
    }
    tc_fence_before_sync();
  }

  linger_after_abort(abort_flag);
  __syncthreads();
  if (warp == kMProducerWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

cudaError_t launch_fa_bwd_mid(const BwdParams& p, bool bf16, cudaStream_t stream) {
  dim3 grid((p.S_k + kTile - 1) / kTile, p.B * (p.N / p.kv_group));
  // (row groups of a multiple of 128 rows never cut a tile: the tile ranges alone take care of them)
  const bool general = p.mods.mask_kind != 0 || p.mods.drop != nullptr || (p.mods.tri_block > 0 && p.mods.tri_block % kTile != 0);
  const int mode = general ? 2 : (p.mods.drop_philox != 0 ? 1 : 0);
  void (*kern)(const BwdParams) =
      mode == 0 ? (bf16 ? fa_bwd_mid_kernel<true, 0> : fa_bwd_mid_kernel<false, 0>)
      : mode == 1 ? (bf16 ? fa_bwd_mid_kernel<true, 1> : fa_bwd_mid_kernel<false, 1>)
                  : (bf16 ? fa_bwd_mid_kernel<true, 2> : fa_bwd_mid_kernel<false, 2>);
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), kMSmem);
  if (e != cudaSuccess) return e;
  kern<<<grid, kMThreads, kMSmem, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace acct
