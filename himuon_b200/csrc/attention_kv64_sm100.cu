// Flash attention forward with 64-wide KV blocks.
//
// K/V arrive in blocks of 64 positions: shared memory stays at 96 KB and the TMEM footprint at 256 columns, so two
// CTAs run on every SM and one CTA's tensor-core work overlaps the other's softmax.
#include "attention_common.cuh"

#include <string>

namespace himuon {

constexpr int BKV = 64;                              // KV positions per block
constexpr uint32_t KV_HALF = BKV * 128;              // one 64-column half of a K or V block: 8 KB

// ================================================================================================ forward, P in TMEM
// CTA = (128 query rows, head, batch); loops over 64-wide KV blocks up to the diagonal; S(j+1) = Q K^T is issued
// before P(j) V so the tensor core overlaps the softmax; O stays in TMEM and is rescaled lazily (only when a row max
// grows by > 2^8).  The probabilities never touch shared memory: the softmax threads write P (bf16) over the first 32
// columns of the S buffer they just read and P·V runs with the A operand in tensor memory.  The two S buffers
// therefore double-buffer P as well, the wait for the previous P·V is only needed on the rare O rescale, S is read
// from TMEM once, and K and V each have two 16 KB stages.
// A parity wait can only tell a phase from its neighbours, and the softmax threads skip most phases of `o_done`, so there
// is one per S buffer: whoever waits for P(i)·V has seen S(i), which the tensor core finishes after P(i-2)·V, the phase
// before it on the same barrier.  The end of the last product has a barrier of its own (`acc_done`, one phase): a warp
// that is done with its softmax gets there while P(nkv-2)·V may still be running.
struct Fwd64TBars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_done[2], acc_done;
  uint32_t tmem_slot;
  int abort_flag;
};

template <int NH>
__global__ void __launch_bounds__(192, 2)
flash_fwd64_t_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, AttnDev p) {
  constexpr uint32_t TILE_BYTES = NH * HALF_BYTES, KV_TILE = NH * KV_HALF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_up_1024(smem_raw);
  uint8_t* sQ = smem;                          // 32 KB
  uint8_t* sK = smem + TILE_BYTES;             // 2 stages x 16 KB
  uint8_t* sV = sK + 2 * KV_TILE;              // 2 stages x 16 KB
  Fwd64TBars* bars = reinterpret_cast<Fwd64TBars*>(sV + 2 * KV_TILE);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = warp_id(), lane = threadIdx.x & 31;
  int sblk, h, b;
  attn_block_coords(sblk, h, b);
  const int qb = gridDim.x - 1 - sblk;         // heavy (late) query blocks first
  const int hk = h / (p.Hq / p.Hkv);
  int nkv = (qb + 1) * (AT / BKV);             // KV blocks up to and including the diagonal
  const int nkv_all = (p.S + BKV - 1) / BKV;
  if (nkv > nkv_all) nkv = nkv_all;

  auto load_k = [&](int j, uint32_t e) {
    const int st = j & 1;
    mbar_expect_tx(&bars->k_full[st], KV_TILE, e);
    load_head_tile<NH>(sK + st * KV_TILE, KV_HALF, &tmK, &bars->k_full[st], hk, j * BKV, b, e);
  };
  auto load_v = [&](int j, uint32_t e) {
    const int st = j & 1;
    mbar_expect_tx(&bars->v_full[st], KV_TILE, e);
    load_head_tile<NH>(sV + st * KV_TILE, KV_HALF, &tmV, &bars->v_full[st], hk, j * BKV, b, e);
  };
  if (warp == 0) {                             // the first loads are on their way while the block sets itself up
    if (lane == 0) {
      mbar_init(&bars->q_full, 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&bars->k_full[i], 1); mbar_init(&bars->k_empty[i], 1);
        mbar_init(&bars->v_full[i], 1); mbar_init(&bars->v_empty[i], 1);
        mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_ready[i], 128);
      }
      for (int i = 0; i < 2; ++i) mbar_init(&bars->o_done[i], 1);
      mbar_init(&bars->acc_done, 1);
      bars->abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
    const uint32_t e = elect_one();
    mbar_expect_tx(&bars->q_full, TILE_BYTES, e);
    load_head_tile<NH>(sQ, HALF_BYTES, &tmQ, &bars->q_full, h, qb * AT, b, e);
    for (int j = 0; j < 2 && j < nkv; ++j) { load_k(j, e); load_v(j, e); }
  }
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_slot, 0);
  const uint32_t tS0 = tmem, tO = tmem + 128;   // S / P buffers at columns 0 and 64, O at 128

  if (warp == 0) {
    const uint32_t e = elect_one();
    for (int j = 2; j < nkv; ++j) {
      const uint32_t par = ((j >> 1) & 1) ^ 1;
      if (!mbar_wait_warp(&bars->k_empty[j & 1], par, abort_flag, p.status, 4)) break;
      load_k(j, e);
      if (!mbar_wait_warp(&bars->v_empty[j & 1], par, abort_flag, p.status, 4)) break;
      load_v(j, e);
    }
  } else if (warp == 1) {
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BKV, false, false);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, 64 * NH, false, true);
      const uint64_t q_desc = kmajor_desc(sQ), k_desc = kmajor_desc(sK), v_mn = mnmajor_desc(sV, KV_HALF);
      bool ok = mbar_wait_warp(&bars->q_full, 0, abort_flag, p.status, 4);
      auto issue_s = [&](int j) -> bool {
        const int st = j & 1;
        if (!mbar_wait_warp(&bars->k_full[st], (j >> 1) & 1, abort_flag, p.status, 4)) return false;
        tc_fence_after();
        // buffer st held S(j-2) / P(j-2): the softmax threads are done with it (p_ready(j-2) was waited for) and the
        // P(j-2)·V MMAs were issued earlier, which the tensor core executes in order before these
#pragma unroll
        for (int ks = 0; ks < 4 * NH; ++ks)
          umma_ss(tS0 + st * BKV, desc_at(q_desc, kmajor_off(HALF_BYTES, ks)), desc_at(k_desc, st * KV_TILE + kmajor_off(KV_HALF, ks)), idesc_s, ks > 0 ? 1u : 0u, e);
        umma_commit(&bars->k_empty[st], e);
        umma_commit(&bars->s_full[st], e);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; ok && j < nkv; ++j) {
        if (j + 1 < nkv) { ok = issue_s(j + 1); if (!ok) break; }
        const int st = j & 1;
        if (!mbar_wait_warp(&bars->p_ready[st], (j >> 1) & 1, abort_flag, p.status, 4)) break;
        if (!mbar_wait_warp(&bars->v_full[st], (j >> 1) & 1, abort_flag, p.status, 4)) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < BKV / 16; ++ks)
          umma_ts(tO, tS0 + st * BKV + ks * 8, desc_at(v_mn, st * KV_TILE + mnmajor_off(ks)), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u, e);
        umma_commit(&bars->v_empty[st], e);
        umma_commit(&bars->o_done[st], e);
      }
      if (ok) umma_commit(&bars->acc_done, e);
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue: one thread per query row
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int q_idx = qb * AT + row;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      const int st = j & 1;
      if (!mbar_wait(&bars->s_full[st], (j >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const uint32_t tS = tS0 + st * BKV + lane_off;
      const int kv0 = j * BKV;
      const bool diag = (kv0 + BKV - 1 > qb * AT);       // the block reaches past the first row of this query tile
      uint32_t v0[32], v1[32];
      tmem_ld32(tS, v0);
      tmem_ld32(tS + 32, v1);
      tmem_ld_wait();
      float mx = -INFINITY;
#pragma unroll
      for (int t = 0; t < 32; ++t) {
        float s0 = __uint_as_float(v0[t]) * p.scale_log2, s1 = __uint_as_float(v1[t]) * p.scale_log2;
        if (diag && (kv0 + t > q_idx)) s0 = -INFINITY;
        if (diag && (kv0 + 32 + t > q_idx)) s1 = -INFINITY;
        v0[t] = __float_as_uint(s0);
        v1[t] = __float_as_uint(s1);
        mx = fmaxf(mx, fmaxf(s0, s1));
      }
      const float m_new = fmaxf(m_used, mx);
      const bool need = (j > 0) && (m_new - m_used > 8.f);
      const bool warp_need = __any_sync(0xffffffffu, need);
      if (j == 0) {
        m_used = m_new;
      } else if (warp_need) {
        // O (and l) move to the new maximum: the previous P·V must have landed in O first
        const float alpha = exp2f(m_used - m_new);
        m_used = m_new;
        if (!mbar_wait(&bars->o_done[st ^ 1], ((j - 1) >> 1) & 1, abort_flag, p.status, 4)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 2 * NH; ++c) {
          uint32_t v[32];
          tmem_ld32(tO + lane_off + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 32; ++t) v[t] = __float_as_uint(__uint_as_float(v[t]) * alpha);
          tmem_st32(tO + lane_off + c * 32, v);
        }
        l *= alpha;
      }
      uint32_t pk[32];
      float rs = 0.f;
#pragma unroll
      for (int t = 0; t < 32; t += 2) {
        // masked entries are -inf: exp2 gives exactly 0
        pk[t >> 1] = pack_bf16x2(exp2f(__uint_as_float(v0[t]) - m_used), exp2f(__uint_as_float(v0[t + 1]) - m_used));
        pk[16 + (t >> 1)] = pack_bf16x2(exp2f(__uint_as_float(v1[t]) - m_used), exp2f(__uint_as_float(v1[t + 1]) - m_used));
        rs += bf16_lo(pk[t >> 1]) + bf16_hi(pk[t >> 1]) + bf16_lo(pk[16 + (t >> 1)]) + bf16_hi(pk[16 + (t >> 1)]);
      }
      l += rs;
      tmem_st32(tS, pk);                     // P over the first 32 columns of the S buffer just read
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars->p_ready[st]);
    }
    if (ok && mbar_wait(&bars->acc_done, 0, abort_flag, p.status, 4)) {
      tc_fence_after();
      const float inv = 1.f / l;
      const int row0 = qb * AT + (warp & 3) * 32;
      __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.o) + (static_cast<long long>(b) * p.S + row0) * p.ld_o + h * p.hd;
      uint8_t* stage = smem + (warp & 3) * (NH * 4096);    // over Q: every product has been computed
      // Half a tile of rows or less: a thread stores its own, because turning them around takes longer than it saves (128 x 64
      // tokens, 16 heads of 128: 34.4 us, 39.0 staged; 8 x 96 already 6.5 against 6.4).  Heads of 64 gain less than the branch
      // costs their longer sequences (64 x 64 tokens 15.7 -> 15.1, but 16 x 128 6.6 -> 6.9).
      const bool few = NH == 2 && p.S - qb * AT <= AT / 2;
#pragma unroll 1
      for (int c = 0; c < 2 * NH; ++c) {
        uint32_t v[32];
        tmem_ld32(tO + lane_off + c * 32, v);
        tmem_ld_wait();
        if (few) {
          if (q_idx < p.S) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (c * 32 + q * 8 < p.hd) *reinterpret_cast<uint4*>(out + lane * p.ld_o + c * 32 + q * 8) = head8(v + 8 * q, inv);
          }
        } else {
          stage_head32<8 * NH>(stage, lane, c, v, inv);
        }
      }
      if (!few) store_staged<8 * NH>(out, p.ld_o, stage, lane, p.S - row0, p.hd);
      if (q_idx < p.S) p.lse[(static_cast<long long>(b) * p.Hq + h) * p.S + q_idx] = m_used + log2f(l);   // base-2 log-sum-exp of the scaled scores
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ================================================================================================ host
static AttnDev make_dev(const AttnArgs& a) {
  AttnDev p{};
  p.o = a.o; p.lse = a.lse; p.delta = a.delta; p.o_in = a.o; p.d_o = a.d_o; p.dq = a.dq; p.dk = a.dk; p.dv = a.dv;
  p.hd = a.hd;
  p.B = a.B; p.S = a.S; p.Hq = a.Hq; p.Hkv = a.Hkv;
  p.ld_o = a.ld_o; p.ld_do = a.ld_do; p.ld_dq = a.ld_dq; p.ld_dk = a.ld_dk; p.ld_dv = a.ld_dv;
  p.nblk = (a.S + AT - 1) / AT;
  p.scale = a.scale; p.scale_log2 = a.scale * kLog2e;
  p.status = status_word_ptr();
  return p;
}

template <int NH>
static void launch_fwd(const AttnArgs& a, cudaStream_t s) {
  constexpr size_t SMEM = 1024 + NH * HALF_BYTES + 4 * NH * KV_HALF + 256;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(flash_fwd64_t_kernel<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    attr = true;
  }
  const AttnDev p = make_dev(a);
  const CUtensorMap tq = head_tmap(a.q, a.B, a.S, a.Hq, a.hd, a.ld_q), tk = head_tmap(a.k, a.B, a.S, a.Hkv, a.hd, a.ld_k, BKV),
                    tv = head_tmap(a.v, a.B, a.S, a.Hkv, a.hd, a.ld_v, BKV);
  flash_fwd64_t_kernel<NH><<<dim3(p.nblk, a.Hq, a.B), 192, SMEM, s>>>(tq, tk, tv, p);
}
void flash_fwd_kv64(const AttnArgs& a, cudaStream_t s) {
  if (head_halves(a.hd) == 1) launch_fwd<1>(a, s);
  else launch_fwd<2>(a, s);
}

}  // namespace himuon
