// Warp-specialised flash-attention backward for sm_100a, head dim 64 or 128 (included by
// attention_sm100.cu inside namespace nkb).
//
// One CTA per (128-key block, batch*head) looping over query blocks, 16 warps:
//   warps 0-7   two compute warpgroups.  Scores are produced transposed (S^T = K Q^T,
//               dP^T = V dO^T), so a thread owns one KEY row (TMEM lane); warpgroup w takes
//               query columns [64w, 64w+64).  It forms P^T = exp2(S^T c - lse), written
//               back to TMEM as bf16 pairs (A operand of dV += P^T dO, read straight from
//               TMEM), and dS^T = P^T (dP^T - delta), written to shared memory (A operand of
//               dK += dS^T Q as K-major and of dQ = dS K as MN-major).
//   warps 8-11  dQ writer: TMEM -> registers -> swizzled fp32 tile in shared memory ->
//               one TMA reduce-add into the fp32 dQ accumulator (no per-thread atomics).
//   warp 12     TMA producer (K, V once; Q and dO in stages).
//   warp 13     tcgen05.mma issuer.
//   warps 14-15 idle (they complete the fourth warpgroup for setmaxnreg).
//
// TMEM (512 columns) decides what can overlap.  Head dim 64: S^T of even blocks [0,128), of odd
// blocks [128,256); once both warpgroups have read it, P^T of warpgroup w over its columns
// [32w, 32w+32) and dQ over [64,128); dP^T [256,384), dV [384,448), dK [448,512).  S^T and dP^T
// of block i+1 are issued before the issuer waits for the compute warpgroups' block i, so these
// go from block to block without a gap while dV, dK and dQ run behind them.
// Head dim 128: S^T [0,128) (P^T over [0,64)), dP^T [128,256), later dQ of the same block,
// dV [256,384), dK [384,512).  S^T of block i+1 follows dV of block i, so the exponentials
// of block i+1 run under dQ and dK of block i; dP^T waits until dQ has been read.
//
// What bounds it: the chain tensor core -> compute -> tensor core of a block.  With the next
// block's S^T issued after dV and dK a block took 7.6 k cycles (head dim 64), of which the
// compute is about 2.1 k and the 32 MMAs (at least 60 cycles each) about 2 k.  Causal, 8 x 16
// heads, 1024 positions, head dim 64: 167 -> 112 us; full, 3 x 12, 1111: 111 -> 73 us; causal,
// 2 x 32, 2048, head dim 128: 568 (one tile at a time, dQ by atomics) -> 338 us.  With packed pairs in the
// compute warps (the staged lse and delta negated for it) another 2 % with head dim 64 (106.8 -> 105.0,
// 69.3 -> 67.9 us in later timings), nothing with 128.
//
// lse / delta of the query block are staged in shared memory (they index columns here),
// fetched one block ahead.  All waits are bounded.  The reference has no attention layer.
#pragma once

constexpr int BWD2_THREADS = 512;
// setmaxnreg budget: the CTA owns threads x 128 registers (the compile-time cap)
static_assert(256 * 176 + 128 * 96 + 128 * 64 <= BWD2_THREADS * 128, "register budget");

template <int D>
struct AttnBwd2Smem {
  static constexpr int TILE = 128 * D * 2;       // bf16 tile: 64-column sub-tiles of 16 KB
  static constexpr int QST = D == 64 ? 3 : 2;    // Q: in use, next (, on the way)
  static constexpr int OST = D == 64 ? 3 : 1;    // dO is free early with head dim 128
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = TILE;
  static constexpr int Q_OFF = 2 * TILE;
  static constexpr int DO_OFF = Q_OFF + QST * TILE;
  static constexpr int DS_OFF = DO_OFF + OST * TILE;  // 32 KB (dS^T, two 64-query sub-tiles)
  static constexpr int DQ_OFF = DS_OFF + 32768;   // 32 KB fp32 staging (two 32-column sub-tiles)
  static constexpr int LD_OFF = DQ_OFF + 32768;   // [2][256] floats: -lse*log2e | -delta
  static constexpr int BAR_OFF = LD_OFF + 2048;
  // the buffer starts on 1024 bytes (checked in the kernel): there is no room for slack
  static constexpr int BYTES = BAR_OFF + 256;
  static_assert(BYTES <= 232448, "shared memory");
};

template <int D>
__global__ void __launch_bounds__(BWD2_THREADS, 1)
attn_bwd_pp_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmDQ, const AttnBwdArgs a) {
  using L = AttnBwd2Smem<D>;
  constexpr int TILE = L::TILE, NKD = D / 64;
  constexpr int QST = L::QST, OST = L::OST;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t S_STEP = D == 64 ? 128 : 0;  // S^T of odd blocks
  constexpr uint32_t DPT_COL = D == 64 ? 256 : 128, DV_COL = D == 64 ? 384 : 256,
                     DK_COL = D == 64 ? 448 : 384;
  constexpr uint32_t DQ_COL = D == 64 ? 64 : 128;  // + S_STEP for odd blocks
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    if (!grid_dep_wait()) return;
    if (threadIdx.x == 0 && a.status) atomicCAS(a.status, 0, (int)NKB_ERR_BOUNDS);
    return;
  }
  uint8_t* sK = smem + L::K_OFF;
  uint8_t* sV = smem + L::V_OFF;
  uint8_t* sQ = smem + L::Q_OFF;
  uint8_t* sDO = smem + L::DO_OFF;
  uint8_t* sDS = smem + L::DS_OFF;
  uint8_t* sDQ = smem + L::DQ_OFF;
  float* sLD = reinterpret_cast<float*>(smem + L::LD_OFF);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;     // [QST]
  uint64_t* q_empty = bars + 4;    // [QST]
  uint64_t* s_full = bars + 7;
  uint64_t* s_read = bars + 8;     // S^T in registers (8 compute warps)
  uint64_t* dp_full = bars + 9;
  uint64_t* dp_read = bars + 10;   // dP^T in registers (8 compute warps)
  uint64_t* pds_full = bars + 11;  // 8 compute warps
  uint64_t* dq_full = bars + 12;   // dQ written, dS^T in shared memory free
  uint64_t* dq_free = bars + 13;   // 4 dQ-writer warps
  uint64_t* acc_full = bars + 14;
  uint64_t* ld_ready = bars + 15;  // [2] lse / delta of a query block staged (256 threads)
  uint64_t* stg_free = bars + 17;  // dQ staging tile reusable
  uint64_t* stg_full = bars + 18;  // dQ staging tile written (128 threads)
  uint64_t* do_full = bars + 19;   // [OST]
  uint64_t* do_empty = bars + 22;  // [OST]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 25);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (a.S + 127) / 128;
  const int j = blockIdx.y;  // key block; early key blocks have the most work and go first
  const int bh = blockIdx.x;
  const int b = bh / a.H, h = bh % a.H;
  const int i0 = a.causal ? j : 0;
  const int niter = nq - i0;
  const long long bh_off = ((long long)b * a.H + h) * a.S;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < QST; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < OST; ++i) {
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_read, 8);
    mbar_init(dp_full, 1);
    mbar_init(dp_read, 8);
    mbar_init(pds_full, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 4);
    mbar_init(acc_full, 1);
    mbar_init(&ld_ready[0], 256);
    mbar_init(&ld_ready[1], 256);
    mbar_init(stg_free, 1);
    mbar_init(stg_full, 128);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!grid_dep_wait()) return;

  if (warp >= 12) {
    // =================================================================== control
    reg_alloc_dec<64>();
    if (warp == 12 && lane == 0) {
      // ------------------------------------------------------------ TMA producer
      auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row0) {
#pragma unroll
        for (int kd = 0; kd < NKD; ++kd) tma_load_4d(dst + kd * 16384, tm, bar, kd * 64, h, row0, b);
      };
      mbar_expect_tx(kv_full, 2 * TILE);
      load_tile(sK, &tmK, kv_full, j * 128);
      load_tile(sV, &tmV, kv_full, j * 128);
      for (int it = 0; it < niter; ++it) {
        const int q = it % QST, o = it % OST;
        if (!mbar_wait(&q_empty[q], ((it / QST) & 1) ^ 1, abort_flag)) {
          att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
          break;
        }
        mbar_expect_tx(&q_full[q], TILE);
        load_tile(sQ + q * TILE, &tmQ, &q_full[q], (i0 + it) * 128);
        if (!mbar_wait(&do_empty[o], ((it / OST) & 1) ^ 1, abort_flag)) {
          att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
          break;
        }
        mbar_expect_tx(&do_full[o], TILE);
        load_tile(sDO + o * TILE, &tmDO, &do_full[o], (i0 + it) * 128);
      }
      grid_dep_trigger();
    } else if (warp == 13 && lane == 0) {
      // -------------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);  // S^T, dP^T
      constexpr uint32_t idesc_ts = umma_idesc_bf16(128, D, 0, 1);   // dV (A from TMEM), dK
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, D, 1, 1);   // dQ: both MN-major
      // descriptors are built once; per MMA only the start-address field (16-byte units) moves.
      // Their upper words are all the same, so a register each holds the lower one.
      constexpr uint64_t DESC_HI = (uint64_t)((1024u >> 4) | 1u << 14 | 2u << 29) << 32;
      auto lo = [](uint64_t d) { return (uint32_t)d; };
      auto dsc = [](uint32_t l) { return DESC_HI | l; };
      const uint32_t dK_k = lo(umma_desc_sw128(smem_u32(sK), 16, 1024));      // K, K-major (A of S^T)
      const uint32_t dV_k = lo(umma_desc_sw128(smem_u32(sV), 16, 1024));      // V, K-major (A of dP^T)
      const uint32_t dK_mn = lo(umma_desc_sw128(smem_u32(sK), 16384, 1024));  // K, MN-major (B of dQ)
      const uint32_t dQ_k0 = lo(umma_desc_sw128(smem_u32(sQ), 16, 1024));     // Q, K-major (B of S^T)
      const uint32_t dDO_k0 = lo(umma_desc_sw128(smem_u32(sDO), 16, 1024));
      const uint32_t dQ_mn0 = lo(umma_desc_sw128(smem_u32(sQ), 16384, 1024));   // Q, MN-major (B of dK)
      const uint32_t dDO_mn0 = lo(umma_desc_sw128(smem_u32(sDO), 16384, 1024));
      const uint32_t dDS_mn = lo(umma_desc_sw128(smem_u32(sDS), 16384, 1024));  // dS^T, A of dQ
      const uint32_t dDS_k = lo(umma_desc_sw128(smem_u32(sDS), 16, 1024));      // dS^T, A of dK
      auto issue_s = [&](int it) -> bool {  // S^T = K Q^T
        const int q = it % QST;
        if (!mbar_wait(&q_full[q], (it / QST) & 1, abort_flag)) {
          att_error(a.status, abort_flag, NKB_ERR_TMA_WAIT);
          return false;
        }
        tc_fence_after();
        const uint32_t off = (uint32_t)q * (TILE >> 4);
#pragma unroll
        for (int k = 0; k < 4 * NKD; ++k) {
          const uint32_t ko = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
          umma_bf16_ss(tmem_base + (it & 1) * S_STEP, dsc(dK_k + ko), dsc(dQ_k0 + off + ko),
                       idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full);
        return true;
      };
      auto issue_dp = [&](int it) -> bool {  // dP^T = V dO^T
        const int o = it % OST;
        if (!mbar_wait(&do_full[o], (it / OST) & 1, abort_flag)) {
          att_error(a.status, abort_flag, NKB_ERR_TMA_WAIT);
          return false;
        }
        tc_fence_after();
        const uint32_t off = (uint32_t)o * (TILE >> 4);
#pragma unroll
        for (int k = 0; k < 4 * NKD; ++k) {
          const uint32_t ko = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
          umma_bf16_ss(tmem_base + DPT_COL, dsc(dV_k + ko), dsc(dDO_k0 + off + ko), idesc_s,
                       k > 0 ? 1u : 0u);
        }
        umma_commit(dp_full);
        return true;
      };
      // dV += P^T dO ; dK += dS^T Q (contraction over the 128 queries, 16 per MMA: 8 columns of
      // bf16 pairs of P^T, 32 bytes of a row of dS^T) ; dQ = dS K (16 keys per MMA)
      auto issue_dv = [&](int it) {
        const uint32_t off = (uint32_t)(it % OST) * (TILE >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts(tmem_base + DV_COL, tmem_base + (it & 1) * S_STEP + k * 8,
                       dsc(dDO_mn0 + off + k * 128), idesc_ts, (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(&do_empty[it % OST]);
      };
      auto issue_dk = [&](int it) {
        const uint32_t off = (uint32_t)(it % QST) * (TILE >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + DK_COL, dsc(dDS_k + (k >> 2) * (16384 >> 4) + (k & 3) * 2),
                       dsc(dQ_mn0 + off + k * 128), idesc_ts, (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(&q_empty[it % QST]);
      };
      auto issue_dq = [&](int it) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + (it & 1) * S_STEP + DQ_COL, dsc(dDS_mn + k * 128),
                       dsc(dK_mn + k * 128), idesc_dq, k > 0 ? 1u : 0u);
      };
      auto wait_for = [&](uint64_t* bar, int phase, int code) -> bool {
        if (mbar_wait(bar, phase, abort_flag)) return true;
        att_error(a.status, abort_flag, code);
        return false;
      };
      bool ok = wait_for(kv_full, 0, NKB_ERR_TMA_WAIT) && niter > 0 && issue_s(0) && issue_dp(0);
      for (int it = 0; it < niter && ok; ++it) {
        const bool more = it + 1 < niter;
        if constexpr (D == 64) {
          // A barrier that may be two phases ahead of one of its waiters would look like one
          // that has not moved: S^T(it+1) waits until every warp has seen S^T(it), and dQ(it) until
          // its writer has seen dQ(it-1).  The latter also frees the buffer of S^T(it+1), which
          // holds dQ(it-1) and P^T(it-1) (consumed by MMAs issued before: the pipe runs in order).
          ok = it == 0 || wait_for(dq_free, (it - 1) & 1, NKB_ERR_ACC_FREE);
          if (ok && more)
            ok = wait_for(s_read, it & 1, NKB_ERR_ACC_FREE) && issue_s(it + 1) &&
                 wait_for(dp_read, it & 1, NKB_ERR_ACC_FREE) && issue_dp(it + 1);
          if (!ok) break;
          if (!(ok = wait_for(pds_full, it & 1, NKB_ERR_ACC_WAIT))) break;
          tc_fence_after();
          issue_dv(it);
          issue_dk(it);
          issue_dq(it);
          umma_commit(dq_full);
        } else {
          // (every warp has read dP^T(it) before it reports pds_full)
          if (!(ok = wait_for(pds_full, it & 1, NKB_ERR_ACC_WAIT))) break;
          tc_fence_after();
          issue_dv(it);
          if (more && !(ok = issue_s(it + 1))) break;
          issue_dq(it);
          issue_dk(it);
          umma_commit(dq_full);
          if (more) {
            if (!(ok = wait_for(dq_free, it & 1, NKB_ERR_ACC_FREE))) break;
            if (!(ok = issue_dp(it + 1))) break;
          }
        }
      }
      if (ok) umma_commit(acc_full);
    }
  } else if (warp >= 8) {
    // ================================================================= dQ writer
    reg_alloc_dec<96>();
    const int r = (warp & 3) * 32 + lane;  // query row inside the block (TMEM lane)
    const uint32_t t_lane = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    for (int it = 0; it < niter; ++it) {
      if (!mbar_wait(dq_full, it & 1, abort_flag)) {
        att_error(a.status, abort_flag, NKB_ERR_ACC_WAIT);
        break;
      }
      tc_fence_after();
      bool ok = true;
#pragma unroll
      for (int hf = 0; hf < NKD; ++hf) {  // 64 columns at a time
        uint32_t v[64];
        tmem_ld_32x32(t_lane + (it & 1) * S_STEP + DQ_COL + hf * 64, v);
        tmem_ld_32x32(t_lane + (it & 1) * S_STEP + DQ_COL + hf * 64 + 32, v + 32);
        tmem_ld_wait();
        if (hf == NKD - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_free);
        }
        // the previous reduce must have finished reading the staging tile
        const int n = it * NKD + hf;
        if (threadIdx.x == 256) {
          tma_store_wait_read<0>();
          mbar_arrive(stg_free);
        }
        if (!mbar_wait(stg_free, n & 1, abort_flag)) {
          att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
          ok = false;
          break;
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) {  // 16-byte chunk c of the row: sub-tile c>>3, chunk c&7
          float4 f = make_float4(__uint_as_float(v[4 * c]) * a.scale, __uint_as_float(v[4 * c + 1]) * a.scale,
                                 __uint_as_float(v[4 * c + 2]) * a.scale, __uint_as_float(v[4 * c + 3]) * a.scale);
          *reinterpret_cast<float4*>(sDQ + (c >> 3) * 16384 + sw128_off(r, c & 7)) = f;
        }
        fence_proxy_async_smem();
        mbar_arrive(stg_full);
        if (threadIdx.x == 256) {
          if (!mbar_wait(stg_full, n & 1, abort_flag)) {
            att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
            ok = false;
            break;
          }
          tma_reduce_add_3d(&tmDQ, sDQ, hf * 64, (i0 + it) * 128, bh);
          tma_reduce_add_3d(&tmDQ, sDQ + 16384, hf * 64 + 32, (i0 + it) * 128, bh);
          tma_store_commit();
        }
      }
      if (!ok) break;
    }
    if (threadIdx.x == 256) tma_store_wait<0>();
  } else {
    // =================================================================== compute
    reg_alloc_inc<176>();
    const int w = warp >> 2;                 // warpgroup: query columns [64w, 64w+64)
    const int r = (warp & 3) * 32 + lane;    // key row inside the block (TMEM lane)
    const int tid = threadIdx.x;             // 0..255
    const uint32_t t_lane = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    // -lse * log2(e) (threads 0-127) / -delta (threads 128-255) of query (block, tid & 127)
    auto fetch_ld = [&](int it) -> float {
      const int qi = (i0 + it) * 128 + (tid & 127);
      if (qi >= a.S) return tid < 128 ? -INFINITY : 0.f;
      return tid < 128 ? -(a.lse[bh_off + qi] * LOG2E) : -a.delta[bh_off + qi];
    };
    if (niter > 0) {
      sLD[tid] = fetch_ld(0);
      mbar_arrive(&ld_ready[0]);
    }
    bool ok = true;
    for (int it = 0; it < niter; ++it) {
      const int i = i0 + it;
      float nxt = 0.f;
      if (it + 1 < niter) nxt = fetch_ld(it + 1);
      if (!mbar_wait(&ld_ready[it & 1], (it >> 1) & 1, abort_flag)) {  // lse / delta staged
        att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
        ok = false;
        break;
      }
      const float* sL = sLD + (it & 1) * 256 + w * 64;
      const float* sDl = sL + 128;
      if (!mbar_wait(s_full, it & 1, abort_flag)) {
        att_error(a.status, abort_flag, NKB_ERR_ACC_WAIT);
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t t_s = t_lane + (it & 1) * S_STEP;
      uint32_t s[64];
      tmem_ld_32x32(t_s + w * 64, s);
      tmem_ld_32x32(t_s + w * 64 + 32, s + 32);
      tmem_ld_wait();
      // P^T of either warpgroup overwrites scores that the first one reads
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_read);
      const bool diag = a.causal && i == j;
      const f32x2_t scale2 = f2_pack(a.scale_log2, a.scale_log2);
      float p[64];
#pragma unroll
      for (int e = 0; e < 64; e += 4) {
        const float4 l4 = *reinterpret_cast<const float4*>(sL + e);
        float x0, x1, x2, x3;
        f2_unpack(f2_fma(f2_pack(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), scale2,
                         f2_pack(l4.x, l4.y)), x0, x1);
        f2_unpack(f2_fma(f2_pack(__uint_as_float(s[e + 2]), __uint_as_float(s[e + 3])), scale2,
                         f2_pack(l4.z, l4.w)), x2, x3);
        p[e] = ex2_f32(x0);
        p[e + 1] = ex2_f32(x1);
        p[e + 2] = ex2_f32(x2);
        p[e + 3] = ex2_f32(x3);
      }
      if (diag) {  // key r may only see queries >= r
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (r > w * 64 + e) p[e] = 0.f;
      }
      // Keys behind the last one: their scores are 0, so a query whose scores are all far below
      // 0 would give them P = exp2(-lse) = inf, and inf * 0 in dQ = dS K
      if (j * 128 + r >= a.S) {
#pragma unroll
        for (int e = 0; e < 64; ++e) p[e] = 0.f;
      }
      if (!mbar_wait(s_read, it & 1, abort_flag)) {
        att_error(a.status, abort_flag, NKB_ERR_ACC_WAIT);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack_bf16x2(p[hf * 32 + 2 * e], p[hf * 32 + 2 * e + 1]);
        tmem_st_32x16(t_s + w * 32 + hf * 16, pk);
      }
      if (!mbar_wait(dp_full, it & 1, abort_flag)) {
        att_error(a.status, abort_flag, NKB_ERR_ACC_WAIT);
        ok = false;
        break;
      }
      tc_fence_after();
      // dK and dQ of the block before have read the shared dS^T
      if (it > 0 && !mbar_wait(dq_full, (it - 1) & 1, abort_flag)) {
        att_error(a.status, abort_flag, NKB_ERR_EMPTY_WAIT);
        ok = false;
        break;
      }
      uint8_t* ds_tile = sDS + w * 16384;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {  // halves: a thread has 128 registers
        uint32_t dp[32];
        tmem_ld_32x32(t_lane + DPT_COL + w * 64 + hf * 32, dp);
        tmem_ld_wait();
        if (D == 64 && hf == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dp_read);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* pe = p + hf * 32 + q * 8;
          const float4 d0 = *reinterpret_cast<const float4*>(sDl + hf * 32 + q * 8);
          const float4 d1 = *reinterpret_cast<const float4*>(sDl + hf * 32 + q * 8 + 4);
          const uint32_t* v = dp + q * 8;
          auto ds2 = [&](int e, float n0, float n1) {  // P^T (dP^T - delta), two columns
            return f2_to_bf16x2(f2_mul(
                f2_pack(pe[e], pe[e + 1]),
                f2_add(f2_pack(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), f2_pack(n0, n1))));
          };
          *reinterpret_cast<uint4*>(ds_tile + sw128_off(r, hf * 4 + q)) =
              make_uint4(ds2(0, d0.x, d0.y), ds2(2, d0.z, d0.w), ds2(4, d1.x, d1.y),
                         ds2(6, d1.z, d1.w));
        }
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      if (it + 1 < niter) {
        sLD[((it + 1) & 1) * 256 + tid] = nxt;
        mbar_arrive(&ld_ready[(it + 1) & 1]);
      }
    }
    if (ok && niter > 0 && mbar_wait(acc_full, 0, abort_flag)) {
      tc_fence_after();
      // dV, dK: warpgroup w stores half of the head-dim columns of key row r
      const int ki = j * 128 + r;
      const long long off = (long long)b * a.sb + (long long)h * a.sh + (long long)ki * a.ss;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const float mul = which == 0 ? 1.f : a.scale;
#pragma unroll
        for (int c = w * (D / 2); c < w * (D / 2) + D / 2; c += 32) {
          __nv_bfloat16* dst = (which == 0 ? a.dv : a.dk) + off + c;
          uint32_t v[32];
          tmem_ld_32x32(t_lane + (which == 0 ? DV_COL : DK_COL) + c, v);
          tmem_ld_wait();
          if (ki < a.S) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(
                  pack_bf16x2(__uint_as_float(v[8 * q]) * mul, __uint_as_float(v[8 * q + 1]) * mul),
                  pack_bf16x2(__uint_as_float(v[8 * q + 2]) * mul, __uint_as_float(v[8 * q + 3]) * mul),
                  pack_bf16x2(__uint_as_float(v[8 * q + 4]) * mul, __uint_as_float(v[8 * q + 5]) * mul),
                  pack_bf16x2(__uint_as_float(v[8 * q + 6]) * mul, __uint_as_float(v[8 * q + 7]) * mul));
          }
        }
      }
    } else if (ok && niter > 0) {
      att_error(a.status, abort_flag, NKB_ERR_ACC_WAIT);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    if (*abort_flag)
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}
