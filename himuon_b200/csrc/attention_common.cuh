// Definitions shared by the attention kernels (128-wide and 64-wide KV-block variants).
#pragma once

#include "himuon.h"
#include "sm100_common.cuh"
#include "tma_host.h"

namespace himuon {

constexpr int AT = 128;                 // tile rows (queries) and tile columns (keys)
constexpr uint32_t HALF_BYTES = 16384;  // [128 rows][64 columns] bf16
// The kernels are instantiated for NH = 1 or 2 halves of 64 head columns.  A head narrower than 64 * NH (any multiple
// of 8) is filled up with zeros by the TMA loads (its tensor map ends at the head's own width) and cut off again by
// the epilogues, so no padded copy of q, k, v, o or their gradients exists in memory.  Heads of 64 take NH = 1: half
// the tensor work, shared memory and operand traffic of the 128-wide instantiation.
// Measured on a training step of the 220M Llama (8 x 512 tokens, heads of 64), together with the 64-wide rotary kernel:
// 9.9 -> 6.5 ms; before, q, k, v, o and their gradients were padded to 128 columns in memory.
inline int head_halves(int hd) { return hd <= 64 ? 1 : 2; }
constexpr float kLog2e = 1.4426950408889634f;

// Byte offsets of k-step ks (16 deep) in a tile of swizzled halves of 64 columns: read K-major (along the columns, halves
// `half` bytes apart) and MN-major (along the rows).
__device__ __forceinline__ constexpr uint32_t kmajor_off(uint32_t half, int ks) { return (ks >> 2) * half + (ks & 3) * 32; }
__device__ __forceinline__ constexpr uint32_t mnmajor_off(int ks) { return ks * 2048; }
__device__ __forceinline__ uint64_t kmajor_desc(const void* tile) { return umma_smem_desc(smem_u32(tile), 16, 1024); }
__device__ __forceinline__ uint64_t mnmajor_desc(const void* tile, uint32_t half) { return umma_smem_desc(smem_u32(tile), half, 1024); }

struct AttnDev {
  void* o; float* lse; float* delta;
  const void* o_in; const void* d_o;
  void* dq; void* dk; void* dv;
  int B, S, Hq, Hkv, nblk;
  int hd;               // head width in memory (<= 64 * NH)
  int split_heads;      // dkv kernel: 1 = one CTA per (KV block, query head) writing per-head partials
  long long ld_o, ld_do, ld_dq, ld_dk, ld_dv;
  float scale_log2, scale;
  int* status;
};

// 4-D tensor map over a (B, S, H, hd) view: box = 64 head-dim columns x `rows` sequence positions of one head.
inline CUtensorMap head_tmap(const void* ptr, int B, int S, int H, int hd, long long ld, int rows = AT) {
  // dims (innermost first): head_dim, heads, sequence, batch
  const uint64_t dims[4] = {static_cast<uint64_t>(hd), static_cast<uint64_t>(H), static_cast<uint64_t>(S), static_cast<uint64_t>(B)};
  const uint64_t strides[3] = {static_cast<uint64_t>(hd) * 2, static_cast<uint64_t>(ld) * 2, static_cast<uint64_t>(ld) * 2 * static_cast<uint64_t>(S)};
  const uint32_t box[4] = {64, 1, static_cast<uint32_t>(rows), 1};
  return make_tmap(ptr, 4, dims, strides, box, 2, true);
}


// CTAs start in linear block order (x fastest).  The causal work of a CTA depends only on its position along the
// sequence, so that position is decoded as the slowest coordinate: all the heaviest blocks start first and the
// light ones fill the tail of the launch (longest-processing-time order).  `sblk` counts from 0 = first started.
__device__ __forceinline__ void attn_block_coords(int& sblk, int& head, int& batch) {
  const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int per = gridDim.y * gridDim.z;
  sblk = lin / per;
  const int r = lin - sblk * per;
  batch = r / gridDim.y;
  head = r - batch * gridDim.y;
}

// Loads `rows` positions (NH halves of `half_bytes` each) of one head into a swizzled tile (a converged warp's elected lane).
template <int NH>
__device__ __forceinline__ void load_head_tile(uint8_t* dst, uint32_t half_bytes, const CUtensorMap* tm, uint64_t* bar,
                                               int head, int s0, int b, uint32_t e) {
#pragma unroll
  for (int j = 0; j < NH; ++j) tma_load_4d(dst + j * half_bytes, tm, bar, j * 64, head, s0, b, e);
}
// Eight accumulator columns, scaled, as bf16.
__device__ __forceinline__ uint4 head8(const uint32_t* v, float f) {
  return make_uint4(pack_bf16x2(__uint_as_float(v[0]) * f, __uint_as_float(v[1]) * f), pack_bf16x2(__uint_as_float(v[2]) * f, __uint_as_float(v[3]) * f),
                    pack_bf16x2(__uint_as_float(v[4]) * f, __uint_as_float(v[5]) * f), pack_bf16x2(__uint_as_float(v[6]) * f, __uint_as_float(v[7]) * f));
}
// The epilogues go through shared memory: a thread has one row of the accumulator, and a warp that stores 32 rows of 16 bytes
// touches 32 lines with every instruction (3000-4000 cycles for the dK and dV of a block).  Each warp turns its own 32 rows
// around in a buffer of its own, 16-byte chunks exchanged within a row so that neither side meets a bank conflict, and stores
// whole row pieces.  CHUNKS = 16-byte chunks per row: 4, 8 or 16.
template <int CHUNKS>
__device__ __forceinline__ uint32_t staged_at(int row, int c) {
  return (row * CHUNKS + (c ^ (CHUNKS == 4 ? (row >> 1) & 3 : row & 7))) * 16;
}
// 32 accumulator columns of this lane's row, scaled, as bf16: chunks 4 * part .. 4 * part + 3.
template <int CHUNKS>
__device__ __forceinline__ void stage_head32(uint8_t* buf, int lane, int part, const uint32_t (&v)[32], float f) {
#pragma unroll
  for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(buf + staged_at<CHUNKS>(lane, part * 4 + q)) = head8(v + 8 * q, f);
}
// The warp's 32 rows from `first` (the row and column that buf starts with), cut off at `rows` rows and `cols` columns.
template <int CHUNKS>
__device__ __forceinline__ void store_staged(__nv_bfloat16* first, long long ld, const uint8_t* buf, int lane, int rows, int cols) {
  __syncwarp();
// (16 in a row cost a short kernel more in fetched instructions than they save: 8 x 128 tokens 6.9 us, 6.5 with four at a time;
// 8 in a row, heads of 64, are the better way, 8 x 512 tokens 12.8 against 13.1)
#pragma unroll(CHUNKS > 8 ? 4 : CHUNKS)
  for (int i = 0; i < CHUNKS; ++i) {
    const int row = (i * 32 + lane) / CHUNKS, c = (i * 32 + lane) % CHUNKS;
    if (row < rows && c * 8 < cols)
      *reinterpret_cast<uint4*>(first + row * ld + c * 8) = *reinterpret_cast<const uint4*>(buf + staged_at<CHUNKS>(row, c));
  }
}

// Forward (two CTAs per SM); dK/dV and dQ in the pipelined formulation of attention_bwd_sm100.cu.
void flash_fwd_kv64(const AttnArgs& a, cudaStream_t s);
void flash_bwd_dkv_t(const AttnArgs& a, const AttnDev& p, int heads_y, cudaStream_t s);
void flash_bwd_dq_t(const AttnArgs& a, const AttnDev& p, cudaStream_t s);

}  // namespace himuon
