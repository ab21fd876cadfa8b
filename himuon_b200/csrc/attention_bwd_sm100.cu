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
// TMEM (512 columns): S^T buffers at 0 and 64 (P^T over the first 32 columns of each), dP^T buffers at 128 and 192
// (dS^T likewise), dV at 256, dK at 384.
// Any sequence length: rows past S arrive as zeros (TMA) with a log-sum-exp of +inf, so their probabilities are 0, and
// are not stored.  The per-row statistics (log-sum-exp, delta) arrive by bulk copies with the Q/dO stage when S is a
// multiple of 64 (every sub-block is then whole and starts on 16 bytes); otherwise (RAGGED) each softmax group fetches
// its sub-block's values itself, ahead of the wait for the scores.
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
// warp 0: TMA producer, warp 1: MMA issue, warps 2-5 and 6-9: two softmax groups of 128 threads (one per TMEM
// lane) that take alternate sub-blocks, so two warps per scheduler hide each other's MUFU and TMEM latencies
constexpr int BWD_THREADS = 320;

struct DkvBars {
  uint64_t kv_full, qd_full[NST], qd_empty[NST], s_full[2], p_ready[2], stat_ready[2], acc_done;
  uint32_t tmem_slot;
  int abort_flag;
};

__device__ __forceinline__ uint64_t sub_desc_kmajor(uint32_t base, int ks) {   // [64 q][128 hd] as the K-major B operand
  return umma_smem_desc(base + (ks >> 2) * Q_HALF + (ks & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t sub_desc_mnmajor(uint32_t base, int ks) {  // the same bytes read along the head dim
  return umma_smem_desc(base + ks * 2048, Q_HALF, 1024);
}
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

  if (threadIdx.x == 0) {
    mbar_init(&bars->kv_full, 1);
    for (int i = 0; i < NST; ++i) { mbar_init(&bars->qd_full[i], 1); mbar_init(&bars->qd_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_ready[i], 128); mbar_init(&bars->stat_ready[i], 128); }
    mbar_init(&bars->acc_done, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);
  const uint32_t tS = tmem, tDP = tmem + 128, tDV = tmem + 256, tDK = tmem + 384;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    {
      const uint32_t e = elect_one();
      mbar_expect_tx(&bars->kv_full, 2 * TILE_BYTES, e);
      load_head_tile<NH>(sK, HALF_BYTES, &tmK, &bars->kv_full, hk, kb * AT, b, e);
      load_head_tile<NH>(sV, HALF_BYTES, &tmV, &bars->kv_full, hk, kb * AT, b, e);
      for (int it = 0; it < iters; ++it) {
        const int g = it / nsub;
        const int h = h_first + g;
        const int q0 = kb * AT + (it - g * nsub) * BQ;
        const int st = it % NST;
        if (!mbar_wait_warp(&bars->qd_empty[st], ((it / NST) & 1) ^ 1, abort_flag, p.status, 4)) break;
        mbar_expect_tx(&bars->qd_full[st], 2 * Q_TILE + (RAGGED ? 0 : STAT_BYTES), e);
        uint8_t* q_dst = sQ + st * Q_TILE;
        uint8_t* do_dst = sDO + st * Q_TILE;
        load_head_tile<NH>(q_dst, Q_HALF, &tmQ, &bars->qd_full[st], h, q0, b, e);
        load_head_tile<NH>(do_dst, Q_HALF, &tmDO, &bars->qd_full[st], h, q0, b, e);
        if (!RAGGED) {
          const long long stat_idx = (static_cast<long long>(b) * p.Hq + h) * p.S + q0;
          if (e) bulk_load_1d(sStat + st * 2 * BQ, p.lse + stat_idx, BQ * 4, &bars->qd_full[st]);
          if (e) bulk_load_1d(sStat + st * 2 * BQ + BQ, p.delta + stat_idx, BQ * 4, &bars->qd_full[st]);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BQ, false, false);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, 64 * NH, false, true);
      const uint32_t k_base = smem_u32(sK), v_base = smem_u32(sV), q_base = smem_u32(sQ), do_base = smem_u32(sDO);
      bool ok = mbar_wait_warp(&bars->kv_full, 0, abort_flag, p.status, 4);
      auto issue_sp = [&](int it) -> bool {
        const int st = it % NST, buf = it & 1;
        if (!mbar_wait_warp(&bars->qd_full[st], (it / NST) & 1, abort_flag, p.status, 4)) return false;
        tc_fence_after();
        // The buffer's previous contents (P^T, dS^T of sub-block it-2) were consumed by MMAs issued earlier, which
        // the tensor core executes in order before these.
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tS + buf * BQ, desc_kmajor(k_base, ks), sub_desc_kmajor(q_base + st * Q_TILE, ks), idesc_s, ks > 0 ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tDP + buf * BQ, desc_kmajor(v_base, ks), sub_desc_kmajor(do_base + st * Q_TILE, ks), idesc_s, ks > 0 ? 1u : 0u, e);
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
          umma_ts(tDV, tS + buf * BQ + ks * 8, sub_desc_mnmajor(do_base + st * Q_TILE, ks), idesc_acc, (it > 0 || ks > 0) ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)
          umma_ts(tDK, tDP + buf * BQ + ks * 8, sub_desc_mnmajor(q_base + st * Q_TILE, ks), idesc_acc, (it > 0 || ks > 0) ? 1u : 0u, e);
        umma_commit(&bars->qd_empty[st], e);
      }
      if (ok) umma_commit(&bars->acc_done, e);
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue: one thread per key row
    const int wg = (warp - 2) >> 2;                       // 0: even sub-blocks (buffer 0), 1: odd sub-blocks (buffer 1)
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int kv_idx = kb * AT + row;
    const int buf = wg;
    bool ok = true;
    for (int it = wg; it < iters; it += 2) {
      const int g = it / nsub;
      const int q0 = kb * AT + (it - g * nsub) * BQ;
      const int st = it % NST;
      // RAGGED: sub-block `it` has statistics slot it % NST, so a group alternates between two slots of its own.  A
      // thread rewrites a slot two of its sub-blocks later, past the group's barrier of the one between, at which every
      // thread of the group arrives only after it has read this one.  The group meets on an mbarrier, because a thread
      // may leave the loop on its own when a bounded wait runs out: the others then give up here as well.
      if (RAGGED) {
        const int qi = q0 + (row & (BQ - 1));
        const long long stat_idx = (static_cast<long long>(b) * p.Hq + h_first + g) * p.S + qi;
        const bool want_lse = row < BQ;
        float v = want_lse ? INFINITY : 0.f;
        if (qi < p.S) v = want_lse ? p.lse[stat_idx] : p.delta[stat_idx];
        sStat[st * 2 * BQ + row] = v;
        mbar_arrive(&bars->stat_ready[wg]);
        if (!mbar_wait(&bars->stat_ready[wg], (it >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      }
      if (!mbar_wait(&bars->qd_full[st], (it / NST) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      if (!mbar_wait(&bars->s_full[buf], (it >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const float* lse_s = sStat + st * 2 * BQ;
      const float* delta_s = lse_s + BQ;
      const bool diag = q0 < kb * AT + AT;               // some keys of this block lie after some of these queries
#pragma unroll
      for (int c = 0; c < BQ / 32; ++c) {
        uint32_t sv[32], dv[32];
        tmem_ld32(tS + buf * BQ + lane_off + c * 32, sv);
        tmem_ld32(tDP + buf * BQ + lane_off + c * 32, dv);
        tmem_ld_wait();
        uint32_t pk[16], dk[16];
#pragma unroll
        for (int t = 0; t < 32; t += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(lse_s + c * 32 + t);
          const float4 d4 = *reinterpret_cast<const float4*>(delta_s + c * 32 + t);
          const float lv[4] = {l4.x, l4.y, l4.z, l4.w}, dl[4] = {d4.x, d4.y, d4.z, d4.w};
          float pr[4], ds[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float pv = exp2f(fmaf(__uint_as_float(sv[t + u]), p.scale_log2, -lv[u]));
            if (diag && (q0 + c * 32 + t + u < kv_idx)) pv = 0.f;
            pr[u] = pv;
            ds[u] = pv * (__uint_as_float(dv[t + u]) - dl[u]);      // the softmax scale is applied to dK once, at the end
          }
          pk[t >> 1] = pack_bf16x2(pr[0], pr[1]);
          pk[(t >> 1) + 1] = pack_bf16x2(pr[2], pr[3]);
          dk[t >> 1] = pack_bf16x2(ds[0], ds[1]);
          dk[(t >> 1) + 1] = pack_bf16x2(ds[2], ds[3]);
        }
        // The bf16 tiles occupy the first 32 columns of their buffers, i.e. only columns of the first fp32 chunk,
        // which this thread has already read: 16 packed columns per chunk.
        tmem_st16(tS + buf * BQ + lane_off + c * 16, pk);
        tmem_st16(tDP + buf * BQ + lane_off + c * 16, dk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars->p_ready[buf]);
    }
    if (ok && mbar_wait(&bars->acc_done, 0, abort_flag, p.status, 4)) {
      tc_fence_after();
      // group 0 stores dV, group 1 stores dK
      __nv_bfloat16* dst0 = reinterpret_cast<__nv_bfloat16*>(wg == 0 ? p.dv : p.dk) +
                            (static_cast<long long>(b) * p.S + kv_idx) * (wg == 0 ? p.ld_dv : p.ld_dk) + out_head * p.hd;
      const uint32_t t_src = (wg == 0 ? tDV : tDK) + lane_off;
      const float out_scale = wg == 0 ? 1.f : p.scale;
#pragma unroll 1
      for (int c = 0; c < 2 * NH; ++c) {
        uint32_t v[32];
        tmem_ld32(t_src + c * 32, v);
        tmem_ld_wait();
        if (kv_idx < p.S) store_head32(dst0, c * 32, p.hd, v, out_scale);
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

// ================================================================================================ backward: dQ
// CTA = (query block of 128 positions, head, batch).  Q_i and dO_i stay in shared memory; K and V stream through in
// sub-blocks of 64 positions.  S = Q K^T and dP = dO V^T land in one of two TMEM buffer pairs; the softmax threads
// (one per query row) write dS as bf16 over the first 32 columns of the dP buffer, which is then the tensor-memory
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
  DqBars* bars = reinterpret_cast<DqBars*>(sV + NST * Q_TILE);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = warp_id(), lane = threadIdx.x & 31;
  int sblk, h, b;
  attn_block_coords(sblk, h, b);
  const int qb = gridDim.x - 1 - sblk;                 // heavy (late) query blocks first
  const int hk = h / (p.Hq / p.Hkv);
  int nkv = (qb + 1) * (AT / BQ);                      // KV sub-blocks up to and including the diagonal
  const int nkv_all = (p.S + BQ - 1) / BQ;
  if (nkv > nkv_all) nkv = nkv_all;

  if (threadIdx.x == 0) {
    mbar_init(&bars->qd_full, 1);
    for (int i = 0; i < NST; ++i) { mbar_init(&bars->kv_full[i], 1); mbar_init(&bars->kv_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_ready[i], 128); }
    mbar_init(&bars->acc_done, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);
  const uint32_t tS = tmem, tDP = tmem + 128, tDQ = tmem + 256;

  if (warp == 0) {
    {
      const uint32_t e = elect_one();
      mbar_expect_tx(&bars->qd_full, 2 * TILE_BYTES, e);
      load_head_tile<NH>(sQ, HALF_BYTES, &tmQ, &bars->qd_full, h, qb * AT, b, e);
      load_head_tile<NH>(sDO, HALF_BYTES, &tmDO, &bars->qd_full, h, qb * AT, b, e);
      for (int j = 0; j < nkv; ++j) {
        const int st = j % NST;
        if (!mbar_wait_warp(&bars->kv_empty[st], ((j / NST) & 1) ^ 1, abort_flag, p.status, 4)) break;
        mbar_expect_tx(&bars->kv_full[st], 2 * Q_TILE, e);
        uint8_t* k_dst = sK + st * Q_TILE;
        uint8_t* v_dst = sV + st * Q_TILE;
        load_head_tile<NH>(k_dst, Q_HALF, &tmK, &bars->kv_full[st], hk, j * BQ, b, e);
        load_head_tile<NH>(v_dst, Q_HALF, &tmV, &bars->kv_full[st], hk, j * BQ, b, e);
      }
    }
  } else if (warp == 1) {
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BQ, false, false);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, 64 * NH, false, true);
      const uint32_t q_base = smem_u32(sQ), do_base = smem_u32(sDO), k_base = smem_u32(sK), v_base = smem_u32(sV);
      bool ok = mbar_wait_warp(&bars->qd_full, 0, abort_flag, p.status, 4);
      auto issue_sp = [&](int j) -> bool {
        const int st = j % NST, buf = j & 1;
        if (!mbar_wait_warp(&bars->kv_full[st], (j / NST) & 1, abort_flag, p.status, 4)) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tS + buf * BQ, desc_kmajor(q_base, ks), sub_desc_kmajor(k_base + st * Q_TILE, ks), idesc_s, ks > 0 ? 1u : 0u, e);
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tDP + buf * BQ, desc_kmajor(do_base, ks), sub_desc_kmajor(v_base + st * Q_TILE, ks), idesc_s, ks > 0 ? 1u : 0u, e);
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
          umma_ts(tDQ, tDP + buf * BQ + ks * 8, sub_desc_mnmajor(k_base + st * Q_TILE, ks), idesc_acc, (j > 0 || ks > 0) ? 1u : 0u, e);
        umma_commit(&bars->kv_empty[st], e);
      }
      if (ok) umma_commit(&bars->acc_done, e);
    }
  } else {
    const int wg = (warp - 2) >> 2;                       // 0: even KV sub-blocks (buffer 0), 1: odd (buffer 1)
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int q_idx = qb * AT + row;
    const long long stat_idx = (static_cast<long long>(b) * p.Hq + h) * p.S + q_idx;
    const bool row_ok = q_idx < p.S;
    const float lse2 = row_ok ? p.lse[stat_idx] : INFINITY;
    if (wg == 0) {
      float d = 0.f;
      const __nv_bfloat16* op = reinterpret_cast<const __nv_bfloat16*>(p.o_in) + (static_cast<long long>(b) * p.S + q_idx) * p.ld_o + h * p.hd;
      const __nv_bfloat16* gp = reinterpret_cast<const __nv_bfloat16*>(p.d_o) + (static_cast<long long>(b) * p.S + q_idx) * p.ld_do + h * p.hd;
      if (row_ok) {
        d = row_delta(op, gp, p.hd);
        p.delta[stat_idx] = d;
      }
      bars->delta[row] = d;
    }
    named_barrier(1, 256);                                // both groups: the block's delta values are in shared memory
    const float delta = bars->delta[row];
    const int buf = wg;
    bool ok = true;
    for (int j = wg; j < nkv; j += 2) {
      if (!mbar_wait(&bars->s_full[buf], (j >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const int kv0 = j * BQ;
      const bool diag = (kv0 + BQ - 1 > qb * AT);
#pragma unroll
      for (int c = 0; c < BQ / 32; ++c) {
        uint32_t sv[32], dv[32];
        tmem_ld32(tS + buf * BQ + lane_off + c * 32, sv);
        tmem_ld32(tDP + buf * BQ + lane_off + c * 32, dv);
        tmem_ld_wait();
        uint32_t dk[16];
#pragma unroll
        for (int t = 0; t < 32; t += 2) {
          float p0 = exp2f(fmaf(__uint_as_float(sv[t]), p.scale_log2, -lse2));
          float p1 = exp2f(fmaf(__uint_as_float(sv[t + 1]), p.scale_log2, -lse2));
          if (diag && (kv0 + c * 32 + t > q_idx)) p0 = 0.f;
          if (diag && (kv0 + c * 32 + t + 1 > q_idx)) p1 = 0.f;
          dk[t >> 1] = pack_bf16x2(p0 * (__uint_as_float(dv[t]) - delta), p1 * (__uint_as_float(dv[t + 1]) - delta));
        }
        tmem_st16(tDP + buf * BQ + lane_off + c * 16, dk);  // dS over columns of the first dP chunk (already read)
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars->p_ready[buf]);
    }
    if (ok && mbar_wait(&bars->acc_done, 0, abort_flag, p.status, 4)) {
      tc_fence_after();
      // each group stores one half of the dQ columns; dS was left unscaled, so the softmax scale lands here
      __nv_bfloat16* dqp = reinterpret_cast<__nv_bfloat16*>(p.dq) + (static_cast<long long>(b) * p.S + q_idx) * p.ld_dq + h * p.hd;
#pragma unroll 1
      for (int c = wg * NH; c < (wg + 1) * NH; ++c) {
        uint32_t v[32];
        tmem_ld32(tDQ + lane_off + c * 32, v);
        tmem_ld_wait();
        if (row_ok) store_head32(dqp, c * 32, p.hd, v, p.scale);
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
  constexpr size_t SMEM = 1024 + 2 * NH * HALF_BYTES + 2 * NST * NH * Q_HALF + sizeof(DqBars) + 64;
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
