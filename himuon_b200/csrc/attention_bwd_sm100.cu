// Flash attention backward, dK/dV pass, in the transposed formulation.
//
// CTA = (KV block of 128 positions, head, batch).  K_j and V_j stay in shared memory; Q and dO stream through in
// sub-blocks of 64 query positions.  The score tile is computed transposed,
//     S^T = K Q^T  and  dP^T = V dO^T        (128 key rows on the TMEM lanes, 64 query columns),
// so that after the softmax threads turn it into P^T and dS^T (bf16, written back over the same TMEM columns) those
// tiles are already in the layout of a tensor-memory A operand:
//     dV += P^T dO   and   dK += dS^T Q      (A from TMEM, B = the streamed tile read along the head dimension).
// Nothing but Q/dO/K/V touches shared memory, which leaves room for four streamed stages, and the two S^T/dP^T
// buffers let the tensor core work on sub-block i+1 while the softmax threads work on sub-block i.
//
// TMEM (512 columns): S^T buffers at 0 and 64 (P^T over columns 0-15 and 32-47 of each), dP^T buffers at 128 and 192
// (dS^T likewise), dV at 256, dK at 384.
// Any sequence length: rows past S arrive as zeros (TMA) with a log-sum-exp of +inf, so their probabilities are 0, and
// are not stored.  The per-row statistics (log-sum-exp, delta) arrive by bulk copies with the Q/dO stage when S is a
// multiple of 64 (every sub-block is then whole and starts on 16 bytes); otherwise (RAGGED) the softmax groups fetch
// their sub-block's values themselves, ahead of the wait for the scores.
//
// What bounds both kernels (clock readings in one block, heads of 128): a sub-block takes 1480 cycles here and 1210 in the dQ
// pass, against 1280 and 1020 that the tensor core needs (a 128 x 64 x 16 product from shared memory is bound by the 6 KB of
// its operands, 48 cycles).  The rest is some 10000 cycles a block: set-up and first loads 5000-7000, the last products 2000,
// the epilogue 1400-2900.  Descriptors that are one addition each, 16 softmax warps, the first loads ahead of the set-up, the
// staged epilogue and delta by rows of lanes took, dK/dV and dQ: 4 x 2048 tokens, 16 heads over 8, 167 and 156 -> 145 and
// 133 us; 2 x 1024, 32 over 8, 61 and 58 -> 53 and 47; 8 x 512, 10 heads of 64, 24.5 and 22.5 -> 22 and 19.
// Measured, whole backward pass on ragged lengths against the unpipelined kernels that served them before: 5 x 777 tokens
// with 16 heads over 8 191 -> 139 us, 4 x 1000 with 32 over 8 373 -> 270 us, 2 x 1984 with 16 over 8 304 -> 205 us;
// 4 x 1024 (whole sub-blocks) 149 us before and after.
#include "attention_common.cuh"

#include <string>

namespace himuon {

namespace {

constexpr int BQ = 64;                               // query positions per streamed sub-block
constexpr uint32_t Q_HALF = BQ * 128;                // one 64-column half of a sub-block: 8 KB
constexpr int NST = 4;                               // streamed stages of (Q, dO, lse, delta)
constexpr uint32_t STAT_BYTES = 2 * BQ * 4;          // lse[64] then delta[64]
// warp 0: TMA producer, warp 1: MMA issue, warps 2-17: four softmax groups of 128 threads (one per TMEM lane).  Groups 0 and
// 2 share the even sub-blocks, 32 of the 64 columns each, 1 and 3 the odd ones.  A sub-block's chain of TMEM load, exponential
// and TMEM store has to stay shorter than the products of the sub-block before, which are issued ahead of it.
constexpr int BWD_THREADS = 576;
// A packed bf16 tile lies over the fp32 columns that its writers have read themselves: columns 0-15 and 32-47 of its buffer.
__device__ __forceinline__ uint32_t packed_col(int ks) { return static_cast<uint32_t>((ks >> 1) * 32 + (ks & 1) * 8); }

struct DkvBars {
  uint64_t kv_full, qd_full[NST], qd_empty[NST], s_full[2], p_ready[2], stat_ready[2], acc_done;
  uint32_t tmem_slot;
  int abort_flag;
};

__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

}  // namespace

template <int NH, bool RAGGED>
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dkv_t_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, AttnDev p) {
  constexpr uint32_t TILE_BYTES = NH * HALF_BYTES, Q_TILE = NH * Q_HALF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_up_1024(smem_raw);
  uint8_t* sK = smem;
  uint8_t* sV = smem + TILE_BYTES;
  uint8_t* sQ = smem + 2 * TILE_BYTES;                 // NST x 16 KB
  uint8_t* sDO = sQ + NST * Q_TILE;                    // NST x 16 KB
  float* sStat = reinterpret_cast<float*>(sDO + NST * Q_TILE);   // NST x (lse[64], delta[64])
  DkvBars* bars = reinterpret_cast<DkvBars*>(reinterpret_cast<uint8_t*>(sStat) + NST * STAT_BYTES);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = warp_id(), lane = threadIdx.x & 31;
  int kb, hy, b;
  attn_block_coords(kb, hy, b);        // early KV blocks (attended by the most query blocks) start first
  const int Gall = p.Hq / p.Hkv;
  const int G = p.split_heads ? 1 : Gall;
  const int hk = p.split_heads ? hy / Gall : hy;
  const int h_first = p.split_heads ? hy : hk * Gall;
  const int out_head = p.split_heads ? hy : hk;
  const int nsub = (p.S - kb * AT + BQ - 1) / BQ;      // query sub-blocks from the diagonal to the end
  const int iters = G * nsub;

  auto load_stage = [&](int it, uint32_t e) {
    const int g = it / nsub;
    const int h = h_first + g;
    const int q0 = kb * AT + (it - g * nsub) * BQ;
    const int st = it % NST;
    mbar_expect_tx(&bars->qd_full[st], 2 * Q_TILE + (RAGGED ? 0 : STAT_BYTES), e);
    load_head_tile<NH>(sQ + st * Q_TILE, Q_HALF, &tmQ, &bars->qd_full[st], h, q0, b, e);
    load_head_tile<NH>(sDO + st * Q_TILE, Q_HALF, &tmDO, &bars->qd_full[st], h, q0, b, e);
    if (!RAGGED) {
      const long long stat_idx = (static_cast<long long>(b) * p.Hq + h) * p.S + q0;
      if (e) bulk_load_1d(sStat + st * 2 * BQ, p.lse + stat_idx, BQ * 4, &bars->qd_full[st]);
      if (e) bulk_load_1d(sStat + st * 2 * BQ + BQ, p.delta + stat_idx, BQ * 4, &bars->qd_full[st]);
    }
  };
  if (warp == 0) {                     // the first loads are on their way while the block sets itself up
    if (lane == 0) {
      mbar_init(&bars->kv_full, 1);
      for (int i = 0; i < NST; ++i) { mbar_init(&bars->qd_full[i], 1); mbar_init(&bars->qd_empty[i], 1); }
      for (int i = 0; i < 2; ++i) { mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_ready[i], 256); mbar_init(&bars->stat_ready[i], 256); }
      mbar_init(&bars->acc_done, 1);
      bars->abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
    const uint32_t e = elect_one();
    mbar_expect_tx(&bars->kv_full, 2 * TILE_BYTES, e);
    load_head_tile<NH>(sK, HALF_BYTES, &tmK, &bars->kv_full, hk, kb * AT, b, e);
    load_head_tile<NH>(sV, HALF_BYTES, &tmV, &bars->kv_full, hk, kb * AT, b, e);
    for (int it = 0; it < NST && it < iters; ++it) load_stage(it, e);
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);
  const uint32_t tS = tmem, tDP = tmem + 128, tDV = tmem + 256, tDK = tmem + 384;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    const uint32_t e = elect_one();
    for (int it = NST; it < iters; ++it) {
      if (!mbar_wait_warp(&bars->qd_empty[it % NST], ((it / NST) & 1) ^ 1, abort_flag, p.status, 4)) break;
      load_stage(it, e);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BQ, false, false);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, 64 * NH, false, true);
      const uint64_t k_desc = kmajor_desc(sK), v_desc = kmajor_desc(sV), q_desc = kmajor_desc(sQ), do_desc = kmajor_desc(sDO);
      const uint64_t q_mn = mnmajor_desc(sQ, Q_HALF), do_mn = mnmajor_desc(sDO, Q_HALF);
      bool ok = mbar_wait_warp(&bars->kv_full, 0, abort_flag, p.status, 4);
      auto issue_sp = [&](int it) -> bool {
        const int st = it % NST, buf = it & 1;
        if (!mbar_wait_warp(&bars->qd_full[st], (it / NST) & 1, abort_flag, p.status, 4)) return false;
        tc_fence_after();
        // The buffer's previous contents (P^T, dS^T of sub-block it-2) were consumed by MMAs issued earlier, which
        // the tensor core executes in order before these.
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tS + buf * BQ, desc_at(k_desc, kmajor_off(HALF_BYTES, ks)), desc_at(q_desc, st * Q_TILE + kmajor_off(Q_HALF, ks)), idesc_s, ks > 0 ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tDP + buf * BQ, desc_at(v_desc, kmajor_off(HALF_BYTES, ks)), desc_at(do_desc, st * Q_TILE + kmajor_off(Q_HALF, ks)), idesc_s, ks > 0 ? 1u : 0u, e);
        umma_commit(&bars->s_full[buf], e);
        return true;
      };
      if (ok) ok = issue_sp(0);
      for (int it = 0; ok && it < iters; ++it) {
        if (it + 1 < iters) { ok = issue_sp(it + 1); if (!ok) break; }
        const int st = it % NST, buf = it & 1;
        if (!mbar_wait_warp(&bars->p_ready[buf], (it >> 1) & 1, abort_flag, p.status, 4)) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)
          umma_ts(tDV, tS + buf * BQ + packed_col(ks), desc_at(do_mn, st * Q_TILE + mnmajor_off(ks)), idesc_acc, (it > 0 || ks > 0) ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)
          umma_ts(tDK, tDP + buf * BQ + packed_col(ks), desc_at(q_mn, st * Q_TILE + mnmajor_off(ks)), idesc_acc, (it > 0 || ks > 0) ? 1u : 0u, e);
        umma_commit(&bars->qd_empty[st], e);
      }
      if (ok) umma_commit(&bars->acc_done, e);
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue: one thread per key row
    const int wg = (warp - 2) >> 2, buf = wg & 1, part = wg >> 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int kv_idx = kb * AT + row;
    const f32x2 nscale = pack2(-p.scale_log2, -p.scale_log2), minus = pack2(-1.f, -1.f);
    bool ok = true;
    for (int it = buf; it < iters; it += 2) {
      const int g = it / nsub;
      const int q0 = kb * AT + (it - g * nsub) * BQ;
      const int st = it % NST;
      // RAGGED: sub-block `it` has statistics slot it % NST, so the two groups of a buffer alternate between two slots of
      // their own, which the first of them fills.  It rewrites a slot two of its sub-blocks later, past the groups' barrier of
      // the one between, at which every thread of both arrives only after it has read this one.  They meet on an mbarrier,
      // because a thread may leave the loop on its own when a bounded wait runs out: the others then give up here as well.
      if (RAGGED) {
        if (part == 0) {
          const int qi = q0 + (row & (BQ - 1));
          const long long stat_idx = (static_cast<long long>(b) * p.Hq + h_first + g) * p.S + qi;
          const bool want_lse = row < BQ;
          float v = want_lse ? INFINITY : 0.f;
          if (qi < p.S) v = want_lse ? p.lse[stat_idx] : p.delta[stat_idx];
          sStat[st * 2 * BQ + row] = v;
        }
        mbar_arrive(&bars->stat_ready[buf]);
        if (!mbar_wait(&bars->stat_ready[buf], (it >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      }
      if (!mbar_wait(&bars->qd_full[st], (it / NST) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      if (!mbar_wait(&bars->s_full[buf], (it >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const float* lse_s = sStat + st * 2 * BQ;
      const float* delta_s = lse_s + BQ;
      const bool diag = q0 < kb * AT + AT;               // some keys of this block lie after some of these queries
      const uint32_t col = buf * BQ + part * 32 + lane_off;
#pragma unroll
      for (int c = 0; c < 32; c += 16) {                    // 32 at once would take more than the 96 registers there are
        uint32_t sv[16], dv[16], pk[8], dk[8];
        tmem_ld16(tS + col + c, sv);
        tmem_ld16(tDP + col + c, dv);
        tmem_ld_wait();
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(lse_s + part * 32 + c + t);
          const float4 d4 = *reinterpret_cast<const float4*>(delta_s + part * 32 + c + t);
          const f32x2 lv[2] = {pack2(l4.x, l4.y), pack2(l4.z, l4.w)}, dl[2] = {pack2(d4.x, d4.y), pack2(d4.z, d4.w)};
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int j = t + 2 * u, q = q0 + part * 32 + c + j;
            float x0, x1, s0, s1;
            unpack2(fma2(pack2(sv[j], sv[j + 1]), nscale, lv[u]), x0, x1);         // log-sum-exp minus score
            float p0 = exp2f(-x0), p1 = exp2f(-x1);
            if (diag && (q < kv_idx)) p0 = 0.f;
            if (diag && (q + 1 < kv_idx)) p1 = 0.f;
            // the softmax scale is applied to dK once, at the end
            unpack2(mul2(pack2(p0, p1), fma2(dl[u], minus, pack2(dv[j], dv[j + 1]))), s0, s1);
            pk[j >> 1] = pack_bf16x2(p0, p1);
            dk[j >> 1] = pack_bf16x2(s0, s1);
          }
        }
        tmem_st8(tS + col + c / 2, pk);                     // over columns that this thread has read (packed_col)
        tmem_st8(tDP + col + c / 2, dk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars->p_ready[buf]);
    }
    if (ok && mbar_wait(&bars->acc_done, 0, abort_flag, p.status, 4)) {
      tc_fence_after();
      // groups 0 and 2 store dV, 1 and 3 dK, half of the columns each
      const long long ld = buf == 0 ? p.ld_dv : p.ld_dk;
      const int row0 = kb * AT + (warp & 3) * 32;
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(buf == 0 ? p.dv : p.dk) + (static_cast<long long>(b) * p.S + row0) * ld +
                           out_head * p.hd + part * NH * 32;
      const uint32_t t_src = (buf == 0 ? tDV : tDK) + lane_off;
      const float out_scale = buf == 0 ? 1.f : p.scale;
      uint8_t* stage = smem + (warp - 2) * (NH * 2048);     // over K and V: every product has been computed
#pragma unroll 1
      for (int c = 0; c < NH; ++c) {
        uint32_t v[32];
        tmem_ld32(t_src + (part * NH + c) * 32, v);
        tmem_ld_wait();
        stage_head32<4 * NH>(stage, lane, c, v, out_scale);
      }
      store_staged<4 * NH>(dst, ld, stage, lane, p.S - row0, p.hd - part * NH * 32);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ================================================================================================ backward: dQ
// CTA = (query block of 128 positions, head, batch).  Q_i and dO_i stay in shared memory; K and V stream through in
// sub-blocks of 64 positions.  S = Q K^T and dP = dO V^T land in one of two TMEM buffer pairs; the softmax threads
// (two per query row) write dS as bf16 over half of the dP buffer's columns, which are then the tensor-memory
// A operand of dQ += dS K.  Also produces delta = rowsum(O * dO) for the dK/dV pass.
// TMEM: S buffers at 0 and 64, dP buffers at 128 and 192, dQ at 256.
struct DqBars {
  uint64_t qd_full, kv_full[NST], kv_empty[NST], s_full[2], p_ready[2], acc_done;
  uint32_t tmem_slot;
  int abort_flag;
  float delta[AT];
};

template <int NH>
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dq_t_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, AttnDev p) {
  constexpr uint32_t TILE_BYTES = NH * HALF_BYTES, Q_TILE = NH * Q_HALF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_up_1024(smem_raw);
  uint8_t* sQ = smem;
  uint8_t* sDO = smem + TILE_BYTES;
  uint8_t* sK = smem + 2 * TILE_BYTES;                 // NST x 16 KB
  uint8_t* sV = sK + NST * Q_TILE;                     // NST x 16 KB
  uint8_t* sTerm = sV + NST * Q_TILE;                  // what delta is summed from, 16 bytes for each 8 columns of a row
  DqBars* bars = reinterpret_cast<DqBars*>(sTerm + TILE_BYTES);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = warp_id(), lane = threadIdx.x & 31;
  int sblk, h, b;
  attn_block_coords(sblk, h, b);
  const int qb = gridDim.x - 1 - sblk;                 // heavy (late) query blocks first
  const int hk = h / (p.Hq / p.Hkv);
  int nkv = (qb + 1) * (AT / BQ);                      // KV sub-blocks up to and including the diagonal
  const int nkv_all = (p.S + BQ - 1) / BQ;
  if (nkv > nkv_all) nkv = nkv_all;

  auto load_stage = [&](int j, uint32_t e) {
    const int st = j % NST;
    mbar_expect_tx(&bars->kv_full[st], 2 * Q_TILE, e);
    load_head_tile<NH>(sK + st * Q_TILE, Q_HALF, &tmK, &bars->kv_full[st], hk, j * BQ, b, e);
    load_head_tile<NH>(sV + st * Q_TILE, Q_HALF, &tmV, &bars->kv_full[st], hk, j * BQ, b, e);
  };
  if (warp == 0) {                     // the first loads are on their way while the block sets itself up
    if (lane == 0) {
      mbar_init(&bars->qd_full, 1);
      for (int i = 0; i < NST; ++i) { mbar_init(&bars->kv_full[i], 1); mbar_init(&bars->kv_empty[i], 1); }
      for (int i = 0; i < 2; ++i) { mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_ready[i], 256); }
      mbar_init(&bars->acc_done, 1);
      bars->abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
    const uint32_t e = elect_one();
    mbar_expect_tx(&bars->qd_full, 2 * TILE_BYTES, e);
    load_head_tile<NH>(sQ, HALF_BYTES, &tmQ, &bars->qd_full, h, qb * AT, b, e);
    load_head_tile<NH>(sDO, HALF_BYTES, &tmDO, &bars->qd_full, h, qb * AT, b, e);
    for (int j = 0; j < NST && j < nkv; ++j) load_stage(j, e);
  }
  // delta = sum over the head of o * dO.  The 16 warps take 8 rows of o each, LPR lanes to a row, and find dO in shared memory
  // later.  One thread to a row, reading both rows 16 bytes at a time, took 9000 of the 50000 cycles of the longest block.
  // What one thread to a row still does is the sum, from shared memory: pairs of columns, first to last, so that delta is the
  // same for every split of the loads.  (Summed over the lanes instead, its last bit moved one dS in some thousand across a
  // bf16 boundary.)
  constexpr int LPR = 8 * NH, PASSES = LPR / 4;
  uint4 o4[PASSES];
  if (warp >= 2) {
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int r = qb * AT + (warp - 2) * 8 + (i * 32 + lane) / LPR, c = (lane % LPR) * 8;
      o4[i] = make_uint4(0, 0, 0, 0);
      if (r < p.S && c < p.hd)
        o4[i] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.o_in) + (static_cast<long long>(b) * p.S + r) * p.ld_o + h * p.hd + c);
    }
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);
  const uint32_t tS = tmem, tDP = tmem + 128, tDQ = tmem + 256;

  if (warp == 0) {
    const uint32_t e = elect_one();
    for (int j = NST; j < nkv; ++j) {
      if (!mbar_wait_warp(&bars->kv_empty[j % NST], ((j / NST) & 1) ^ 1, abort_flag, p.status, 4)) break;
      load_stage(j, e);
    }
  } else if (warp == 1) {
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BQ, false, false);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, 64 * NH, false, true);
      const uint64_t q_desc = kmajor_desc(sQ), do_desc = kmajor_desc(sDO), k_desc = kmajor_desc(sK), v_desc = kmajor_desc(sV);
      const uint64_t k_mn = mnmajor_desc(sK, Q_HALF);
      bool ok = mbar_wait_warp(&bars->qd_full, 0, abort_flag, p.status, 4);
      auto issue_sp = [&](int j) -> bool {
        const int st = j % NST, buf = j & 1;
        if (!mbar_wait_warp(&bars->kv_full[st], (j / NST) & 1, abort_flag, p.status, 4)) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tS + buf * BQ, desc_at(q_desc, kmajor_off(HALF_BYTES, ks)), desc_at(k_desc, st * Q_TILE + kmajor_off(Q_HALF, ks)), idesc_s, ks > 0 ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tDP + buf * BQ, desc_at(do_desc, kmajor_off(HALF_BYTES, ks)), desc_at(v_desc, st * Q_TILE + kmajor_off(Q_HALF, ks)), idesc_s, ks > 0 ? 1u : 0u, e);
        umma_commit(&bars->s_full[buf], e);
        return true;
      };
      if (ok) ok = issue_sp(0);
      for (int j = 0; ok && j < nkv; ++j) {
        if (j + 1 < nkv) { ok = issue_sp(j + 1); if (!ok) break; }
        const int st = j % NST, buf = j & 1;
        if (!mbar_wait_warp(&bars->p_ready[buf], (j >> 1) & 1, abort_flag, p.status, 4)) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)
          umma_ts(tDQ, tDP + buf * BQ + packed_col(ks), desc_at(k_mn, st * Q_TILE + mnmajor_off(ks)), idesc_acc, (j > 0 || ks > 0) ? 1u : 0u, e);
        umma_commit(&bars->kv_empty[st], e);
      }
      if (ok) umma_commit(&bars->acc_done, e);
    }
  } else {
    const int wg = (warp - 2) >> 2, buf = wg & 1, part = wg >> 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int q_idx = qb * AT + row;
    const long long stat_idx = (static_cast<long long>(b) * p.Hq + h) * p.S + q_idx;
    const bool row_ok = q_idx < p.S;
    const float lse2 = row_ok ? p.lse[stat_idx] : INFINITY;
    bool ok = mbar_wait(&bars->qd_full, 0, abort_flag, p.status, 4);
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int r = (warp - 2) * 8 + (i * 32 + lane) / LPR, c = lane % LPR;
      const uint4 g4 = *reinterpret_cast<const uint4*>(sDO + (c >> 3) * HALF_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4));
      const uint32_t ow[4] = {o4[i].x, o4[i].y, o4[i].z, o4[i].w}, gw[4] = {g4.x, g4.y, g4.z, g4.w};
      float t[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) t[q] = bf16_lo(ow[q]) * bf16_lo(gw[q]) + bf16_hi(ow[q]) * bf16_hi(gw[q]);
      *reinterpret_cast<float4*>(sTerm + staged_at<LPR>(r, c)) = make_float4(t[0], t[1], t[2], t[3]);
    }
    named_barrier(1, 512);                                // all groups: the terms are in shared memory
    if (wg == 0) {
      float d = 0.f;
#pragma unroll
      for (int c = 0; c < LPR; ++c) {
        const float4 t = *reinterpret_cast<const float4*>(sTerm + staged_at<LPR>(row, c));
        d += t.x; d += t.y; d += t.z; d += t.w;
      }
      bars->delta[row] = d;
      if (row_ok) p.delta[stat_idx] = d;
    }
    named_barrier(1, 512);                                // and the block's delta values
    const float delta = bars->delta[row];
    const f32x2 nscale = pack2(-p.scale_log2, -p.scale_log2), lse_2 = pack2(lse2, lse2), ndelta = pack2(-delta, -delta);
    for (int j = buf; ok && j < nkv; j += 2) {
      if (!mbar_wait(&bars->s_full[buf], (j >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const int kv0 = j * BQ;
      const bool diag = (kv0 + BQ - 1 > qb * AT);
      const uint32_t col = buf * BQ + part * 32 + lane_off;
      uint32_t sv[32], dv[32];
      tmem_ld32(tS + col, sv);
      tmem_ld32(tDP + col, dv);
      tmem_ld_wait();
      uint32_t dk[16];
#pragma unroll
      for (int t = 0; t < 32; t += 2) {
        float x0, x1, s0, s1;
        unpack2(fma2(pack2(sv[t], sv[t + 1]), nscale, lse_2), x0, x1);             // log-sum-exp minus score
        float p0 = exp2f(-x0), p1 = exp2f(-x1);
        if (diag && (kv0 + part * 32 + t > q_idx)) p0 = 0.f;
        if (diag && (kv0 + part * 32 + t + 1 > q_idx)) p1 = 0.f;
        unpack2(mul2(pack2(p0, p1), add2(pack2(dv[t], dv[t + 1]), ndelta)), s0, s1);
        dk[t >> 1] = pack_bf16x2(s0, s1);
      }
      tmem_st16(tDP + col, dk);                             // over columns that this thread has read (packed_col)
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars->p_ready[buf]);
    }
    if (ok && mbar_wait(&bars->acc_done, 0, abort_flag, p.status, 4)) {
      tc_fence_after();
      // the groups store 32 dQ columns each (two of them where the head is one half wide); dS was left unscaled, so the
      // softmax scale lands here
      if (wg < 2 * NH) {
        const int row0 = qb * AT + (warp & 3) * 32;
        uint8_t* stage = smem + (warp - 2) * 2048;          // over Q and dO: every product has been computed
        uint32_t v[32];
        tmem_ld32(tDQ + lane_off + wg * 32, v);
        tmem_ld_wait();
        stage_head32<4>(stage, lane, 0, v, p.scale);
        store_staged<4>(reinterpret_cast<__nv_bfloat16*>(p.dq) + (static_cast<long long>(b) * p.S + row0) * p.ld_dq + h * p.hd + wg * 32,
                        p.ld_dq, stage, lane, p.S - row0, p.hd - wg * 32);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int NH, bool RAGGED>
static void launch_dkv_t(const AttnArgs& a, const AttnDev& p, int heads_y, cudaStream_t s) {
  constexpr size_t SMEM = 1024 + 2 * NH * HALF_BYTES + 2 * NST * NH * Q_HALF + NST * STAT_BYTES + sizeof(DkvBars) + 64;
  static bool attr = false;
  if (!attr) { cudaFuncSetAttribute(flash_bwd_dkv_t_kernel<NH, RAGGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); attr = true; }
  const CUtensorMap tq = head_tmap(a.q, a.B, a.S, a.Hq, a.hd, a.ld_q, BQ), tk = head_tmap(a.k, a.B, a.S, a.Hkv, a.hd, a.ld_k),
                    tv = head_tmap(a.v, a.B, a.S, a.Hkv, a.hd, a.ld_v), tdo = head_tmap(a.d_o, a.B, a.S, a.Hq, a.hd, a.ld_do, BQ);
  flash_bwd_dkv_t_kernel<NH, RAGGED><<<dim3(p.nblk, heads_y, a.B), BWD_THREADS, SMEM, s>>>(tq, tk, tv, tdo, p);
}
// `p` carries the output pointers and the split_heads flag chosen by the caller; the grid's y extent is the number of
// query heads (split_heads) or KV heads.
void flash_bwd_dkv_t(const AttnArgs& a, const AttnDev& p, int heads_y, cudaStream_t s) {
  const bool whole = a.S % BQ == 0 && (reinterpret_cast<uintptr_t>(a.lse) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.delta) & 15) == 0;
  if (head_halves(a.hd) == 1) {
    if (whole) launch_dkv_t<1, false>(a, p, heads_y, s);
    else launch_dkv_t<1, true>(a, p, heads_y, s);
  } else {
    if (whole) launch_dkv_t<2, false>(a, p, heads_y, s);
    else launch_dkv_t<2, true>(a, p, heads_y, s);
  }
}

template <int NH>
static void launch_dq_t(const AttnArgs& a, const AttnDev& p, cudaStream_t s) {
  constexpr size_t SMEM = 1024 + 3 * NH * HALF_BYTES + 2 * NST * NH * Q_HALF + sizeof(DqBars) + 64;
  static_assert(SMEM <= 232448, "shared memory budget of one CTA exceeded");
  static bool attr = false;
  if (!attr) { cudaFuncSetAttribute(flash_bwd_dq_t_kernel<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); attr = true; }
  const CUtensorMap tq = head_tmap(a.q, a.B, a.S, a.Hq, a.hd, a.ld_q), tk = head_tmap(a.k, a.B, a.S, a.Hkv, a.hd, a.ld_k, BQ),
                    tv = head_tmap(a.v, a.B, a.S, a.Hkv, a.hd, a.ld_v, BQ), tdo = head_tmap(a.d_o, a.B, a.S, a.Hq, a.hd, a.ld_do);
  flash_bwd_dq_t_kernel<NH><<<dim3(p.nblk, a.Hq, a.B), BWD_THREADS, SMEM, s>>>(tq, tk, tv, tdo, p);
}
void flash_bwd_dq_t(const AttnArgs& a, const AttnDev& p, cudaStream_t s) {
  if (head_halves(a.hd) == 1) launch_dq_t<1>(a, p, s);
  else launch_dq_t<2>(a, p, s);
}

}  // namespace himuon
