// Persistent batched bf16 GEMM for sm_100a:  C[b] = alpha * op(A[b]) * op(B[b]) + beta * Aux[b]
//
//   * operands are staged by TMA (128-byte swizzle, no multicast) into a shared-memory ring,
//   * one elected thread issues tcgen05.mma (M=128, N=BN, K=16) into TMEM accumulators,
//   * eight epilogue warps, two groups of four that take alternate 64-column slabs of the tile, read TMEM with
//     tcgen05.ld and combine into shared-memory slabs; one thread of its own (the slab warp) stores the finished slabs
//     by TMA and hands the drained ones out again, with the next aux tile already in them,
//   * two TMEM accumulators (2 x BN columns) let the epilogue of tile i overlap the MMAs of tile i+1.
//
// Why two groups: a 128 x 256 x 512 tile (Newton-Schulz on 512 tiles) is 3 us of MMA, and one group of four warps
// needed 6.6 us to drain it - the epilogue, not the main loop, bound every short-K product.
// Measured with two: optimizer step on 2300 tiles of 512 15.1 -> 12.8 ms, on 28 of them 346 -> 287 us, 128 tiles through
// newton_schulz 853 -> 756 us, when tiles of 512 ran here; ns_pair_sm100.cu takes them now (475 us), and the products of larger
// tiles and of layers keep this epilogue.
//
// Either operand may be K-major (reduction dim contiguous) or MN-major (M/N contiguous),
// so forward (x W^T), dgrad (dy W) and wgrad (dy^T x) all run without a transpose pass.
// This one kernel replaces the reference's three Triton GEMM kernels
// (src/himuon/triton_kernels/XXT.py:12-75, ba_plus_cAA.py:12-89, fused_bmm_add.py:12-96)
// and the cuBLAS calls behind F.linear / torch.addmm.
#include "gemm_epilogue.cuh"
#include "himuon.h"
#include "sm100_common.cuh"
#include "tma_host.h"

#include <type_traits>

namespace himuon {

__device__ int g_status_word = 0;

// AUX_TMA (bf16 output with an aux operand): the aux tile arrives by TMA in the very staging slab that its output slab
// leaves from.  NSTG slabs rotate through load -> combine in place -> store, with the loads issued NSTG - 1 slabs ahead
// (across tile boundaries), so the epilogue threads never wait on global memory.
// Three operand stages and four slabs (256-wide tiles) serve short reductions, whose epilogue is the longer part; four
// stages and two slabs serve long plain ones in numbers (`long_plain()`).
constexpr int GEMM_THREADS = 384;             // warps 0-3: TMA, MMA, TMEM allocation, slabs; 4-11: epilogue
template <int BN, int STAGES, int NSTG, bool A_MN, bool B_MN, bool AUX_TMA>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX, GemmDev p) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN * BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t CHUNK_BYTES = BK * 128;  // one 64-wide MN chunk of an MN-major tile

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_up_1024(smem_raw);
  uint8_t* sC = smem + STAGES * STAGE_BYTES;                      // staging slabs of the TMA-store epilogue
  uint64_t* bars = reinterpret_cast<uint64_t*>(sC + NSTG * SLAB_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* slab_open = tempty + 2;           // one per slab: free (and, with AUX_TMA, holding its aux tile)
  uint64_t* slab_done = slab_open + NSTG;     // one per slab: combined by the 128 threads of a group
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(slab_done + NSTG);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_id();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 8);
    }
    for (int a = 0; a < NSTG; ++a) { mbar_init(&slab_open[a], 1); mbar_init(&slab_done[a], 128); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    {
      const uint32_t e = elect_one();
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
        const WorkItem w = decode_item(p, item);
        const TileCoord tc = decode_tile(p, w.tile, BN / BM);
        const int b = tc.b, mt = tc.mt, nt = tc.nt;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, p.status, 1)) { ok = false; break; }
          uint8_t* sA = smem + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          mbar_expect_tx(&full[stage], STAGE_BYTES, e);
          if (!A_MN) {
            tma_load_3d(sA, &tmA, &full[stage], kb * BK, mt * BM, b, e);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_3d(sA + j * CHUNK_BYTES, &tmA, &full[stage], mt * BM + j * 64, kb * BK, b, e);
          }
          if (!B_MN) {
            tma_load_3d(sB, &tmB, &full[stage], kb * BK, nt * BN, b, e);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_3d(sB + j * CHUNK_BYTES, &tmB, &full[stage], nt * BN + j * 64, kb * BK, b, e);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    {
      const uint32_t e = elect_one();
      constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
        const WorkItem w = decode_item(p, item);
        if (!mbar_wait_warp(&tempty[acc], acc_phase ^ 1, abort_flag, p.status, 2)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait_warp(&full[stage], phase, abort_flag, p.status, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_base = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t b_base = a_base + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t adesc = A_MN ? umma_smem_desc(a_base + k * 2048, CHUNK_BYTES, 1024)
                                        : umma_smem_desc(a_base + k * 32, 16, 1024);
            const uint64_t bdesc = B_MN ? umma_smem_desc(b_base + k * 2048, CHUNK_BYTES, 1024)
                                        : umma_smem_desc(b_base + k * 32, 16, 1024);
            umma_ss(d_tmem, adesc, bdesc, idesc, (kb > w.kb0 || k > 0) ? 1u : 0u, e);
          }
          umma_commit(&empty[stage], e);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tfull[acc], e);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------ slab warp: aux loads and output stores
    if (lane == 0 && p.tma_store) {
      tma_prefetch_desc(&tmC);
      if (AUX_TMA) tma_prefetch_desc(&tmX);
      const int sw = p.out_fp32 ? 32 : 64;                  // columns of a slab (128 bytes)
      // Two cursors over the slabs of this CTA in the order the epilogue visits them: `op` opens slabs, `st` stores them.
      struct Cursor { int item, col, left; TileCoord tc; } op, st;
      auto enter_tile = [&](Cursor& c) {
        if (c.item >= p.total_items) return;
        c.tc = decode_tile(p, c.item, BN / BM);
        c.col = c.tc.nt * BN;
        const int n = min(BN, p.N - c.col);
        c.left = (n + sw - 1) / sw;
      };
      auto advance = [&](Cursor& c) {
        c.col += sw;
        if (--c.left == 0) { c.item += gridDim.x; enter_tile(c); }
      };
      op.item = st.item = blockIdx.x;
      enter_tile(op);
      enter_tile(st);
      uint32_t opened = 0, seq = 0;
      auto open_next = [&]() {
        if (op.item >= p.total_items) return;
        const uint32_t buf = opened & (NSTG - 1);
        if (AUX_TMA) {
          mbar_expect_tx(&slab_open[buf], SLAB_BYTES);
          tma_load_3d(sC + buf * SLAB_BYTES, &tmX, &slab_open[buf], op.col, op.tc.mt * BM, op.tc.b);
        } else {
          mbar_arrive(&slab_open[buf]);
        }
        ++opened;
        advance(op);
      };
      for (int a = 0; a < NSTG - 1; ++a) open_next();
      // `tail`: the last slab of a row of tiles ends in columns that TMA does not store.  They leave from this thread, in a
      // loop of its own: a branch in the epilogue threads or in the loop of whole slabs cost the short products 1 %.
      auto store_slabs = [&](auto tail) {
        while (st.item < p.total_items) {
          const uint32_t buf = seq & (NSTG - 1);
          if (!mbar_wait(&slab_done[buf], (seq / NSTG) & 1, abort_flag, p.status, 5)) break;
          const uint8_t* slab = sC + buf * SLAB_BYTES;
          if (!tail.value || st.col < p.n_store) tma_store_3d(&tmC, slab, st.col, st.tc.mt * BM, st.tc.b);
          if (tail.value && st.col + sw > p.n_store) {
            const long long off = static_cast<long long>(st.tc.b) * p.strideC + static_cast<long long>(st.tc.mt) * BM * p.ldc + p.n_store;
            const int rows = min(BM, p.M - st.tc.mt * BM), n = p.N - p.n_store, group = (p.n_store - st.col) * 8 / sw;
            if (p.out_fp32) store_tail(reinterpret_cast<float*>(p.C) + off, p.ldc, rows, n, slab, group);
            else store_tail(reinterpret_cast<__nv_bfloat16*>(p.C) + off, p.ldc, rows, n, slab, group);
          }
          tma_store_commit();
          tma_store_wait_read<1>();        // the slab stored before this one is drained: it is the next to be opened
          open_next();
          ++seq;
          advance(st);
        }
      };
      if (p.n_store == p.N) store_slabs(std::false_type{});
      else store_slabs(std::true_type{});
      tma_store_wait_read<0>();          // no store may still be reading shared memory at exit
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ epilogue (two groups of four warps -> TMEM lanes 0..127)
    const int ew = warp & 3;
    const uint32_t eg = static_cast<uint32_t>(warp - 4) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t seq = 0;                        // slabs of this CTA so far; group eg takes those of its parity
    const int row_in_tile = ew * 32 + lane;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
      const TileCoord tc = decode_tile(p, item, BN / BM);
      const int b = tc.b, mt = tc.mt, nt = tc.nt;
      if (!mbar_wait(&tfull[acc], acc_phase, abort_flag, p.status, 3)) break;
      tc_fence_after();
      if (p.tma_store) {
        const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + static_cast<uint32_t>(acc * BN);
        const int row = mt * BM + row_in_tile;
        const long long aux_row = static_cast<long long>(b) * p.strideAux + static_cast<long long>(row) * p.ldaux;
        __nv_bfloat16* mirror_c = tc.mirror ? reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(b) * p.strideC : nullptr;
        const bool fp32_out = !AUX_TMA && p.out_fp32;
        const int sw = fp32_out ? 32 : 64;
#pragma unroll 1
        for (int col = nt * BN; col < nt * BN + BN && col < p.N; col += sw, ++seq) {
          if ((seq & 1) != eg) continue;
          const uint32_t buf = seq & (NSTG - 1);
          uint8_t* my_row = sC + buf * SLAB_BYTES + row_in_tile * 128;
          const uint32_t t_slab = t_acc + static_cast<uint32_t>(col - nt * BN);
          uint4 xa[8];
          if (!AUX_TMA) {
            if (fp32_out) load_aux_slab<true>(p.aux, aux_row + col, row < p.M, p.N - col, xa);
            else load_aux_slab<false>(p.aux, aux_row + col, row < p.M, p.N - col, xa);
          }
          if (!mbar_wait(&slab_open[buf], (seq / NSTG) & 1, abort_flag, p.status, 5)) { ok = false; break; }
          if (fp32_out) slab_fp32(t_slab, my_row, row_in_tile, xa, p.alpha, p.beta);
          else slab_bf16<AUX_TMA>(t_slab, my_row, row_in_tile, xa, p.alpha, p.beta, p.round_acc, mirror_c, p.ldc, col, row, p.N);
          fence_proxy_async_smem();
          mbar_arrive(&slab_done[buf]);
        }
        if (!ok) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
        continue;
      }
      const int row = mt * BM + ew * 32 + lane;
      const bool row_ok = row < p.M;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + static_cast<uint32_t>(acc * BN);
      const long long c_off = static_cast<long long>(b) * p.strideC + static_cast<long long>(row) * p.ldc;
      const long long x_off = static_cast<long long>(b) * p.strideAux + static_cast<long long>(row) * p.ldaux;
#pragma unroll 1
      for (int c0 = static_cast<int>(eg) * 32; c0 < BN; c0 += 64) {
        const int col = nt * BN + c0;
        if (col >= p.N) break;  // uniform over the warp
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(t_row + c0, v);
        tmem_ld_wait();
        const bool full_vec = (col + 32 <= p.N);
        if (!row_ok) {
          // rows past M hold padding; nothing to store
        } else if (p.out_fp32) {
          float* cp = reinterpret_cast<float*>(p.C) + c_off + col;
          const float* xp = p.aux ? reinterpret_cast<const float*>(p.aux) + x_off + col : nullptr;
          if (full_vec && ((reinterpret_cast<uintptr_t>(cp) & 15) == 0) &&
              (!xp || (reinterpret_cast<uintptr_t>(xp) & 15) == 0)) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              float4 o;
              o.x = p.alpha * __uint_as_float(v[j + 0]);
              o.y = p.alpha * __uint_as_float(v[j + 1]);
              o.z = p.alpha * __uint_as_float(v[j + 2]);
              o.w = p.alpha * __uint_as_float(v[j + 3]);
              if (xp) {
                const float4 e = *reinterpret_cast<const float4*>(xp + j);
                o.x += p.beta * e.x; o.y += p.beta * e.y; o.z += p.beta * e.z; o.w += p.beta * e.w;
              }
              *reinterpret_cast<float4*>(cp + j) = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (col + j < p.N) {
                float o = p.alpha * __uint_as_float(v[j]);
                if (xp) o += p.beta * xp[j];
                cp[j] = o;
              }
            }
          }
        } else {
          __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + c_off + col;
          const __nv_bfloat16* xp = p.aux ? reinterpret_cast<const __nv_bfloat16*>(p.aux) + x_off + col : nullptr;
          if (full_vec && ((reinterpret_cast<uintptr_t>(cp) & 15) == 0) &&
              (!xp || (reinterpret_cast<uintptr_t>(xp) & 15) == 0)) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float f[8];
#pragma unroll
              for (int t = 0; t < 8; ++t) f[t] = p.alpha * __uint_as_float(v[j + t]);
              if (xp) {
                const uint4 e = *reinterpret_cast<const uint4*>(xp + j);
                const uint32_t ew4[4] = {e.x, e.y, e.z, e.w};
                if (p.round_acc) {
#pragma unroll
                  for (int t = 0; t < 8; t += 2) round_bf16x2(f[t], f[t + 1]);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  f[2 * t] += p.beta * bf16_lo(ew4[t]);
                  f[2 * t + 1] += p.beta * bf16_hi(ew4[t]);
                }
              }
              uint4 o;
              o.x = pack_bf16x2(f[0], f[1]);
              o.y = pack_bf16x2(f[2], f[3]);
              o.z = pack_bf16x2(f[4], f[5]);
              o.w = pack_bf16x2(f[6], f[7]);
              *reinterpret_cast<uint4*>(cp + j) = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (col + j < p.N) {
                float o = p.alpha * __uint_as_float(v[j]);
                if (xp) {
                  if (p.round_acc) o = round_bf16(o);
                  o += p.beta * __bfloat162float(xp[j]);
                }
                cp[j] = __float2bfloat16_rn(o);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// C can be written by TMA stores
static bool c_rows_aligned(const GemmArgs& a) {
  const int row_align = a.out_fp32 ? 4 : 8;
  return a.N >= row_align && a.ldc % row_align == 0 && (a.batch == 1 || a.strideC % row_align == 0) && reinterpret_cast<uintptr_t>(a.C) % 16 == 0;
}

// bf16 output with a bf16 aux tile that TMA can fetch (16-byte aligned base, rows and batches)
static bool aux_tma_ok(const GemmArgs& a) {
  // (broadcast rows or batches, strides of 0, take the plain loads)
  return a.aux != nullptr && !a.out_fp32 && a.ldaux % 8 == 0 && a.ldaux >= a.N &&
         (a.batch == 1 || (a.strideAux % 8 == 0 && a.strideAux > 0)) &&
         reinterpret_cast<uintptr_t>(a.aux) % 16 == 0 && c_rows_aligned(a);
}

template <int BN, int STAGES, int NSTG, bool A_MN, bool B_MN, bool AUX_TMA>
static void launch_gemm(const GemmArgs& a, cudaStream_t stream) {
  constexpr uint32_t STAGE_BYTES = (BM + BN) * BK * 2;
  constexpr size_t SMEM = 1024 + STAGES * STAGE_BYTES + NSTG * SLAB_BYTES + 256;
  static_assert(SMEM <= 232448, "shared memory budget of one CTA exceeded");
  auto kern = gemm_bf16_kernel<BN, STAGES, NSTG, A_MN, B_MN, AUX_TMA>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM));
    attr_done = true;
  }
  // A: K-major storage (M rows x K) or MN-major storage (K rows x M).
  uint64_t dimsA[3], strA[2], dimsB[3], strB[2];
  uint32_t boxA[3], boxB[3];
  if (!A_MN) { dimsA[0] = a.K; dimsA[1] = a.M; boxA[0] = BK; boxA[1] = BM; }
  else       { dimsA[0] = a.M; dimsA[1] = a.K; boxA[0] = 64; boxA[1] = BK; }
  dimsA[2] = a.batch; boxA[2] = 1;
  strA[0] = static_cast<uint64_t>(a.lda) * 2;
  strA[1] = a.batch > 1 ? static_cast<uint64_t>(a.strideA) * 2 : strA[0] * dimsA[1];
  if (!B_MN) { dimsB[0] = a.K; dimsB[1] = a.N; boxB[0] = BK; boxB[1] = BN; }
  else       { dimsB[0] = a.N; dimsB[1] = a.K; boxB[0] = 64; boxB[1] = BK; }
  dimsB[2] = a.batch; boxB[2] = 1;
  strB[0] = static_cast<uint64_t>(a.ldb) * 2;
  strB[1] = a.batch > 1 ? static_cast<uint64_t>(a.strideB) * 2 : strB[0] * dimsB[1];
  CUtensorMap tmA = make_tmap(a.A, 3, dimsA, strA, boxA, 2, true);
  CUtensorMap tmB = make_tmap(a.B, 3, dimsB, strB, boxB, 2, true);

  GemmDev p{};
  p.C = a.C; p.aux = a.aux;
  p.M = a.M; p.N = a.N; p.K = a.K; p.batch = a.batch;
  p.ldc = a.ldc; p.ldaux = a.ldaux; p.strideC = a.strideC; p.strideAux = a.strideAux;
  p.alpha = a.alpha; p.beta = a.beta; p.out_fp32 = a.out_fp32; p.round_acc = a.round_acc;
  p.tiles_m = (a.M + BM - 1) / BM;
  p.tiles_n = (a.N + BN - 1) / BN;
  p.kblocks = (a.K + BK - 1) / BK;
  p.status = status_word_ptr();
  // C tensor map for the TMA-store epilogue: rows of 128 bytes (64 bf16 / 32 fp32 columns) per slab.
  const int esz = a.out_fp32 ? 4 : 2;
  p.tma_store = c_rows_aligned(a) ? 1 : 0;
  p.n_store = a.N / (16 / esz) * (16 / esz);
  CUtensorMap tmC = tmA;
  if (p.tma_store) {
    const uint64_t dimsC[3] = {static_cast<uint64_t>(p.n_store), static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.batch)};
    const uint64_t strC[2] = {static_cast<uint64_t>(a.ldc) * esz,
                              a.batch > 1 ? static_cast<uint64_t>(a.strideC) * esz : static_cast<uint64_t>(a.ldc) * esz * a.M};
    const uint32_t boxC[3] = {static_cast<uint32_t>(128 / esz), BM, 1};
    tmC = make_tmap(a.C, 3, dimsC, strC, boxC, esz, true);
  }
  CUtensorMap tmX = tmC;
  if (AUX_TMA) {
    const uint64_t dimsX[3] = {static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.batch)};
    const uint64_t strX[2] = {static_cast<uint64_t>(a.ldaux) * 2,
                              a.batch > 1 ? static_cast<uint64_t>(a.strideAux) * 2 : static_cast<uint64_t>(a.ldaux) * 2 * a.M};
    const uint32_t boxX[3] = {64, BM, 1};
    tmX = make_tmap(a.aux, 3, dimsX, strX, boxX, 2, true);
  }
  long long total = static_cast<long long>(p.tiles_m) * p.tiles_n * a.batch;
  // Symmetric output: needs square bf16 C reachable by TMA stores and a tile width that is a whole number of tile
  // heights; otherwise every tile is computed (same result).
  p.sym = (a.symmetric && a.M == a.N && !a.out_fp32 && p.tma_store && BN % BM == 0 && p.tiles_n > 1) ? 1 : 0;
  p.sym_tiles = 0;
  if (p.sym) {
    for (int nt = 0; nt < p.tiles_n; ++nt) p.sym_tiles += p.tiles_m - nt * (BN / BM);
    total = static_cast<long long>(p.sym_tiles) * a.batch;
  }
  int sms = a.max_ctas > 0 ? a.max_ctas : num_sms();
  p.full_items = p.total_items = static_cast<int>(total);
  p.nslices = 1;
  const int grid = static_cast<int>(p.total_items < sms ? p.total_items : sms);
  kern<<<grid, GEMM_THREADS, SMEM, stream>>>(tmA, tmB, tmC, tmX, p);
}

int num_sms() {
  static int sms[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  return sms[dev];
}

// Tiles of width bn that the one-CTA kernel computes for this problem (launch_gemm's own count).
static long long tile_count(const GemmArgs& a, int bn) {
  const int tm = (a.M + BM - 1) / BM, tn = (a.N + bn - 1) / bn;
  long long per = static_cast<long long>(tm) * tn;
  if (a.symmetric && a.M == a.N && !a.out_fp32 && c_rows_aligned(a) && tn > 1) {
    per = 0;
    for (int nt = 0; nt < tn; ++nt) per += tm - nt * (bn / BM);
  }
  return per * a.batch;
}
// Tile width for outputs wider than 192 columns: 256, unless tiles of 128 need clearly fewer rounds over the SMs.  Two
// narrow tiles cost about 4 % more than a wide one (128 products of 512^3, which fill the chip either way: 755 and 786 us
// for newton_schulz), and narrow symmetric tiles mirror a larger share of the output with 2-byte stores (396 tiles of
// 256: 5 % slower than wide ones).  So a narrow round counts 0.7 of a wide one: at 0.55 and 0.65 those 396 tiles went narrow
// and the step that holds them took 4.5 % longer.  Narrow tiles win where the wide ones do not fill the chip (6 matrices of
// 333 x 500: 211 -> 179 us for the whole newton_schulz call) or just overflow it (symmetric products of 28 tiles of 512: 168 wide
// tiles are two rounds, 280 narrow ones two rounds of half the length; the optimizer step went from 277 to 250 us).
// Tiles up to 512 have since gone to ns_pair_sm100.cu; the figures are of the GEMM launches, which shapes it declines still take.
constexpr double kNarrowRound = 0.7;
static long long rounds(long long tiles, long long slots) { return (tiles + slots - 1) / slots; }
static int tile_width(const GemmArgs& a) {
  const long long sms = a.max_ctas > 0 ? a.max_ctas : num_sms();
  return rounds(tile_count(a, 128), sms) * kNarrowRound < static_cast<double>(rounds(tile_count(a, 256), sms)) ? 128 : 256;
}

// 256-wide tiles without an aux operand that need the longer operand ring: many rounds of tiles with a reduction so long
// that the main loop, not the epilogue, sets the pace, and outputs that leave by plain stores and use no slabs at all.  The
// shapes that arrive here are those that pairs_win() declines; measured, four stages and two slabs against three and four:
//   * batches of at most 128 rows, and matrices that the pairs' tiles would pad: 150 of 264 x 1024 x 1024 107 / 115 us, x 768
//     88.3 / 88.4, x 504 82 / 83; 320 x 150000 x 1536 146 / 157, x 384 56 / 55; 300 of 100 x 1024 x 2040 237 / 244;
//   * symmetric products, whose epilogue also writes the mirrored tile: 120 of 1024 x 1024 x 1024 162 / 153, x 1280 183 / 184, x 1536
//     205 / 211 and 215; 400 of 512 x 512 x 1792 241 / 257;
//   * fp32, short ones only where M > 128 (an fp32 slab takes half the columns: more stages help earlier, and the pairs have the
//     longer ones): 4096 x 8192 x 384 39.4 / 42.3, x 504 60.1 / 64.9; 64 of 128 x 4096 x 384 66 / 60, x 504 69 / 66, x 768 86 / 86, x 2040
//     204 / 209.
// With few rounds the slabs win at any length: 1895 x 2560 x 1984 (two rounds) 30.7 / 33.4, symmetric 128 x 512 x 512 x 1280 (six)
// 71.3 / 73.3.
static bool long_plain(const GemmArgs& a) {
  if (!c_rows_aligned(a)) return true;
  const long long sms = a.max_ctas > 0 ? a.max_ctas : num_sms();
  return a.K >= (a.out_fp32 ? (a.M > BM ? 384 : 768) : (a.symmetric ? 1280 : 1024)) && rounds(tile_count(a, 256), sms) > 6;
}

void gemm_bf16(const GemmArgs& a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0 || a.batch <= 0) return;
  if (a.K <= 0) throw std::runtime_error("himuon gemm: K must be positive");
  if (gemm2_supported(a)) {
    gemm2_bf16(a, stream);
    return;
  }
  const int best_bn = a.N <= 128 ? 128 : (a.N <= 192 ? 192 : tile_width(a));
  const int sel = (a.a_mn ? 2 : 0) | (a.b_mn ? 1 : 0);
#define HM_LAUNCH(BN_, ST_, SL_, AX_)                                              \
  switch (sel) {                                                                   \
    case 0: launch_gemm<BN_, ST_, SL_, false, false, AX_>(a, stream); break;       \
    case 1: launch_gemm<BN_, ST_, SL_, false, true, AX_>(a, stream); break;        \
    case 2: launch_gemm<BN_, ST_, SL_, true, false, AX_>(a, stream); break;        \
    default: launch_gemm<BN_, ST_, SL_, true, true, AX_>(a, stream); break;        \
  }
  if (aux_tma_ok(a)) {
    if (best_bn == 128) { HM_LAUNCH(128, 5, 4, true) }
    else if (best_bn == 192) { HM_LAUNCH(192, 4, 4, true) }
    else { HM_LAUNCH(256, 3, 4, true) }
  } else if (best_bn == 192) { HM_LAUNCH(192, 4, 4, false) }
  else if (best_bn == 128) { HM_LAUNCH(128, 5, 4, false) }
  else if (long_plain(a)) { HM_LAUNCH(256, 4, 2, false) }
  else { HM_LAUNCH(256, 3, 4, false) }
#undef HM_LAUNCH
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("himuon gemm launch failed: ") + cudaGetErrorString(e));
}

int* status_word_ptr() {
  static int* ptrs[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (ptrs[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess)
      throw std::runtime_error("himuon: cannot resolve the device status word");
    ptrs[dev] = static_cast<int*>(p);
  }
  return ptrs[dev];
}

int read_status_word(bool reset) {
  int v = 0;
  cudaMemcpy(&v, status_word_ptr(), sizeof(int), cudaMemcpyDeviceToHost);
  if (reset && v != 0) cudaMemset(status_word_ptr(), 0, sizeof(int));
  return v;
}

}  // namespace himuon
