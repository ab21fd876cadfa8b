// Causal grouped-query flash attention for head widths up to 128 on sm_100a: the host entry points (flash_attn_fwd,
// flash_attn_bwd).  The forward kernel lives in attention_kv64_sm100.cu, the backward kernels in attention_bwd_sm100.cu.
//
// Every score / value product runs on tcgen05 tensor cores with TMEM accumulators; Q, K, V and dO tiles arrive by
// TMA (128-byte swizzle, no multicast).  One thread owns one row of a 128-row tile, so row max / row sum need no
// shuffles; grouped heads need no atomics.
//
// The reference reaches attention through HF `sdpa` (PyTorch library kernels); it ships no attention code of its own.
#include "attention_common.cuh"


namespace himuon {

// ================================================================================================ host
static void check_attn(const AttnArgs& a) {
  if (a.S <= 0 || a.B <= 0 || a.Hq <= 0 || a.Hkv <= 0 || a.Hq % a.Hkv) throw std::runtime_error("himuon attention: bad sizes");
  if (a.hd <= 0 || a.hd > 128 || a.hd % 8) throw std::runtime_error("himuon attention: head_dim must be a multiple of 8 up to 128");
  if (a.ld_q % 8 || a.ld_k % 8 || a.ld_v % 8 || a.ld_o % 8) throw std::runtime_error("himuon attention: token strides must be multiples of 8");
}

void flash_attn_fwd(const AttnArgs& a, cudaStream_t s) {
  check_attn(a);
  flash_fwd_kv64(a, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("himuon flash_attn_fwd launch failed: ") + cudaGetErrorString(e));
}

void flash_attn_bwd(const AttnArgs& a, cudaStream_t s) {
  check_attn(a);
  if (a.ld_do % 8 || a.ld_dq % 8 || a.ld_dk % 8 || a.ld_dv % 8) throw std::runtime_error("himuon attention: gradient strides must be multiples of 8");
  AttnDev p{};
  p.lse = a.lse; p.delta = a.delta; p.o_in = a.o; p.d_o = a.d_o; p.dq = a.dq; p.dk = a.dk; p.dv = a.dv;
  p.B = a.B; p.S = a.S; p.Hq = a.Hq; p.Hkv = a.Hkv; p.hd = a.hd;
  p.ld_o = a.ld_o; p.ld_do = a.ld_do; p.ld_dq = a.ld_dq; p.ld_dk = a.ld_dk; p.ld_dv = a.ld_dv;
  p.nblk = (a.S + AT - 1) / AT;
  p.scale = a.scale; p.scale_log2 = a.scale * kLog2e;
  p.status = status_word_ptr();
  flash_bwd_dq_t(a, p, s);
  const int G = a.Hq / a.Hkv;
  if (G > 1 && a.dk_part != nullptr && a.dv_part != nullptr) {
    // one CTA per (KV block, query head): G times more CTAs, balanced across the SMs; the per-head partial
    // gradients are then summed over each group
    AttnDev ps = p;
    ps.split_heads = 1;
    ps.dk = a.dk_part; ps.dv = a.dv_part; ps.ld_dk = a.ld_part; ps.ld_dv = a.ld_part;
    flash_bwd_dkv_t(a, ps, a.Hq, s);
    const long long tokens = static_cast<long long>(a.B) * a.S;
    group_sum_heads(a.dk_part, a.dk, tokens, a.Hkv, G, a.hd, a.ld_part, a.ld_dk, s);
    group_sum_heads(a.dv_part, a.dv, tokens, a.Hkv, G, a.hd, a.ld_part, a.ld_dv, s);
  } else {
    flash_bwd_dkv_t(a, p, a.Hkv, s);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("himuon flash_attn_bwd launch failed: ") + cudaGetErrorString(e));
}

}  // namespace himuon
