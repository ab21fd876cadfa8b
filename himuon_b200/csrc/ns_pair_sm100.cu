// All products of the quintic Newton-Schulz iteration on a batch of matrices in one launch, for matrices that do not fit one
// CTA (ns5_sm100.cu) and whose short side is at most 512.
//
// A CTA pair (or a cluster of two or four pairs) takes a matrix through every iteration:
//     A = X X^T,   B = c A A + b A,   X' = bf16(B X) + a X          (X with its sides exchanged where it is tall)
// in tasks of one 256 x 256 block each (tcgen05.mma.cta_group::2, K = 64 a stage).  Of the symmetric products only the blocks
// on and below the diagonal are computed; the others are read as their transposes, through the operand's major mode, so
// nothing is mirrored.  Intermediates stay in a scratch of three or four buffers per resident matrix, each of X's padded size
// (116 MB for 512 x 512 matrices on every pair).  The L2 mostly serves that much: 512 matrices of 512 x 512 read 850 MB from HBM,
// 268 of them the input, and write 2.9 GB, as lines are written back before they are overwritten (of 19.5 GB that pass the L2 in
// 1447 us; the tensor pipe is busy for 70 % of it).  Long matrices overflow it, as two of them are resident on a pair: 148 of
// 256 x 2048 have 465 MB of scratch, tall ones 620 (the GEMM launches 194).  As fifteen GEMM launches the same products stream
// every intermediate through HBM both ways, and each launch pays its ramp and tail.
//
// Scratch layout: chunks of 64 columns, each [rows][64] with its rows one after the other.  A TMA box of it is one run of
// memory, and the same 128-byte-swizzled shared-memory image serves as K-major and as MN-major operand.
//
// Tasks of different pairs, and of the two CTAs of a pair, hand on through `done` barriers: behind its outputs' completion
// (cp.async.bulk.wait_group, then a fence of the cluster) a CTA arrives on the barrier of that task in every CTA of the cluster,
// and whoever loads the block waits there, with a proxy fence between the wait and the TMA loads (aux values are a CTA's
// own stores, which one proxy orders).  Between a block and its first reader lies at least one other task and a half, in
// which its drain, store and hand-on (4000-7000 cycles) are hidden but for 1000-2000; with one matrix block per phase
// (short and long side up to 256) a pair interleaves up to four matrices instead.
// What is overwritten: a buffer's readers are loads of earlier tasks, whose products a pair issues in order, and with
// several pairs A, B and the two X have a buffer each, so that a block's writer depends on all of its readers.
//
// What bounds it: with all pairs busy the power limit (592 matrices of 512 x 512: 1.2 PFLOP/s against 1.36 of cuBLAS
// sustained), alone the 64 bytes per clock that an SM takes in (operands, aux values) and the hand-on between phases.
// Measured, this kernel against the GEMM launches, us: 592 of 512 x 512 1656 / 2485, 128 of them 384 / 664, 28 127 / 234,
// 396 of 256 x 256 309 / 563, 6 of 336 x 504 110 / 165, 64 of 256 x 1024 139 / 270.  The results have the same bits.
#include "himuon.h"
#include "pair_common.cuh"
#include "sm100_common.cuh"
#include "tma_host.h"

namespace himuon {

constexpr int NSP_STAGES = 5;
constexpr int NSP_THREADS = 384;              // warp 0: operands, 1: MMA, 2: output stores, 3: aux loads, 4-11: epilogue
constexpr uint32_t NSP_OPERAND = 16384;       // 128 rows x 64 columns of one operand of one CTA
constexpr uint32_t NSP_STAGE = 2 * NSP_OPERAND;
constexpr uint32_t NSP_SLAB = 16384;          // 128 rows x 64 columns of a tile on their way in (aux) and out
constexpr int NSP_MAXP = 4;                   // CTA pairs of a cluster
constexpr int NSP_RING = 32;                  // completion barriers per pair

struct NsPairDev {
  long long n_mats, clusters;
  int m, n;                 // stored shape
  int nb, nc;               // 256-wide blocks of the short and of the long side
  int ks, kl;               // 64-wide blocks of the short and of the long side
  int steps, W, bufs;       // W: matrices that a cluster interleaves
  int rpx, rpa;             // padded rows of an X buffer and of A / B
  int rows_buf;             // 128-byte rows of a buffer
  int cx, ca;               // 64-column chunks of a buffer laid out as X and as A
  int* status;
};
struct NsPairMaps { CUtensorMap in_k, in_mn, s_k, s_x, s_a, out; };

struct NsTask {
  int mat, it, phase, w, wc, i, j;
  uint32_t l;               // number of the task among those of its pair
};

// Block tasks of a phase are dealt to the pairs in turn, the same block always to the same pair.  Of n, pair q has:
template <int P> __device__ __forceinline__ uint32_t ns_share(uint32_t n, uint32_t q) { return (n + P - 1 - q) / P; }

// Calls f(task, base) for the tasks of `pair`; base[q]: number of pair q's first task of the group of matrices.
template <int P, class F>
__device__ __forceinline__ void ns_walk(const NsPairDev& p, int cluster, uint32_t pair, F&& f) {
  const long long m0 = p.n_mats * cluster / p.clusters, share = p.n_mats * (cluster + 1) / p.clusters - m0;
  const int groups = static_cast<int>((share + p.W - 1) / p.W);
  const uint32_t t1 = p.nb * (p.nb + 1) / 2, t3 = p.nb * p.nc;
  uint32_t base[P];
#pragma unroll
  for (int q = 0; q < P; ++q) base[q] = 0;
  NsTask t;
  t.l = 0;
  for (int q = 0; q < groups; ++q) {
    const int first = static_cast<int>(m0 + share * q / groups);
    t.wc = static_cast<int>(m0 + share * (q + 1) / groups) - first;
    for (t.it = 0; t.it < p.steps; ++t.it)
      for (t.phase = 0; t.phase < 3; ++t.phase) {
        uint32_t turn = 0;
        for (t.w = 0; t.w < t.wc; ++t.w) {
          t.mat = first + t.w;
          for (t.i = 0; t.i < p.nb; ++t.i) {
            const int cols = t.phase < 2 ? t.i + 1 : p.nc;
            for (t.j = 0; t.j < cols; ++t.j) {
              if (P == 1 || turn == pair) {
                if (!f(t, base)) return;
                ++t.l;
              }
              if (++turn == P) turn = 0;
            }
          }
        }
      }
#pragma unroll
    for (int r = 0; r < P; ++r) base[r] += p.steps * (2 * ns_share<P>(t.wc * t1, r) + ns_share<P>(t.wc * t3, r));
  }
}

// mbar_wait_warp for a barrier on which other CTAs of the cluster arrive behind their outputs.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  bool ok = true;
  for (;;) {
    uint32_t there;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(there)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (there) break;
    if ((++spins & 0xFFu) == 0) {
      if (*abort_flag) { ok = false; break; }
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > kWaitLimitNs) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
        ok = false;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}
// Arrives on a barrier of a CTA of the cluster behind a fence of the cluster.
__device__ __forceinline__ void mbar_arrive_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// Where the 128 rows and 128 columns of a task go that one CTA and column half holds.
struct NsPlace { int row0, col0, rp, chunks; bool live; };
template <bool TALL>
__device__ __forceinline__ NsPlace ns_place(const NsPairDev& p, const NsTask& t, uint32_t rank, int half) {
  const bool transposed = TALL && t.phase == 2;
  const int rb = transposed ? t.j : t.i, cb = transposed ? t.i : t.j;
  NsPlace o;
  o.row0 = rb * 256 + static_cast<int>(rank) * 128;
  o.col0 = cb * 256 + half * 128;
  o.rp = t.phase < 2 ? p.rpa : p.rpx;
  const int row_lim = 64 * (transposed ? p.kl : p.ks), col_lim = 64 * (t.phase == 2 && !TALL ? p.kl : p.ks);
  // Rows and columns past the last 64 of the matrix are never read as reduction indices: nothing to store.  A CTA without
  // any such output takes the task's slab round with nothing in it, so that no warp of it runs ahead of the others.
  o.chunks = o.row0 >= row_lim ? 0 : max(0, min(2, (col_lim - o.col0 + 63) >> 6));
  o.live = o.chunks > 0;
  if (!o.live && half == 0) o.chunks = 1;
  return o;
}

// 64 columns of one accumulator row -> bf16 in the slab, which holds the aux values.
// PHASE 0: acc; 1: c*acc + b*aux; 2: bf16(acc) + a*aux.  Everything is fetched before the arithmetic begins, and conversions
// go two at a time: single ones run at an eighth of the rate (2300 -> 1000 cycles for the chunks of PHASE 2).
template <int PHASE>
__device__ __forceinline__ void ns_slab(uint32_t t_row, uint8_t* my_row, int lane) {
  constexpr float ca = 3.4445f, cb = -4.7750f, cc = 2.0315f;
  uint32_t v[2][32];
  tmem_ld32(t_row, v[0]);
  tmem_ld32(t_row + 32, v[1]);
  uint4 x[8];
  if (PHASE > 0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = *reinterpret_cast<const uint4*>(my_row + ((q ^ (lane & 7)) << 4));
  }
  tmem_ld_wait();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t e[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
    uint32_t o[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float f0 = __uint_as_float(v[q >> 2][8 * (q & 3) + 2 * t]), f1 = __uint_as_float(v[q >> 2][8 * (q & 3) + 2 * t + 1]);
      if (PHASE == 1) { f0 = cc * f0 + cb * bf16_lo(e[t]); f1 = cc * f1 + cb * bf16_hi(e[t]); }
      if (PHASE == 2) {
        const uint32_t r = pack_bf16x2(f0, f1);
        f0 = bf16_lo(r) + ca * bf16_lo(e[t]);
        f1 = bf16_hi(r) + ca * bf16_hi(e[t]);
      }
      o[t] = pack_bf16x2(f0, f1);
    }
    *reinterpret_cast<uint4*>(my_row + ((q ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// An operand of 128 rows and 64 reduction indices, and the step to the next 64.
struct NsOperand { const CUtensorMap* tm; int x, y, z, dx, dy; bool two; };

template <bool TALL, int P>
__global__ void __launch_bounds__(NSP_THREADS, 1)
ns_pair_kernel(const __grid_constant__ NsPairMaps maps, const __grid_constant__ NsPairDev p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_up_1024(smem_raw);
  uint8_t* slabs = smem + NSP_STAGES * NSP_STAGE;                 // two per column half
  uint64_t* full = reinterpret_cast<uint64_t*>(slabs + 4 * NSP_SLAB);
  uint64_t* empty = full + NSP_STAGES;
  uint64_t* tfull = empty + NSP_STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* slab_free = tempty + 2;           // one per slab [column half][64 columns]: stored
  uint64_t* slab_open = slab_free + 4;        // one per slab: free, and holding its aux values
  uint64_t* slab_done = slab_open + 4;        // one per slab: combined by the four warps of a column half
  uint64_t* done = slab_done + 4;             // [P][NSP_RING]: tasks whose outputs are in memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + P * NSP_RING);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_id(), lane = threadIdx.x & 31;
  const uint32_t crank = __shfl_sync(0xffffffffu, cluster_ctarank(), 0);
  const uint32_t pair = crank >> 1, rank = crank & 1, lead_cta = crank & ~1u;
  const int cluster = blockIdx.x / (2 * P);
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSP_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 16); }
    for (int a = 0; a < 4; ++a) { mbar_init(&slab_free[a], 1); mbar_init(&slab_open[a], 1); mbar_init(&slab_done[a], 4); }
    for (int a = 0; a < P * NSP_RING; ++a) mbar_init(&done[a], 2);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc2(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const int buf0 = cluster * p.W * p.bufs;                        // this cluster's first scratch buffer
  constexpr bool THREE = P == 1 && !TALL;
  // buffers of a matrix: A and X take 0 and 1 in turn, B has 2 (THREE), or A has 0, X 1 and 2 in turn, B 3
  auto buf_a = [&](const NsTask& t) { return buf0 + t.w * p.bufs + (THREE ? (t.it & 1) : 0); };
  auto buf_b = [&](const NsTask& t) { return buf0 + t.w * p.bufs + (THREE ? 2 : 3); };
  auto buf_x = [&](const NsTask& t, int it) { return buf0 + t.w * p.bufs + (THREE ? (it & 1) ^ 1 : 1 + (it & 1)); };   // X of iteration it >= 1

  if (warp == 0) {
    // ------------------------------------------------------------ operand loads (both CTAs of the pair)
    const uint32_t e = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t t1 = p.nb * (p.nb + 1) / 2, t3 = p.nb * p.nc;
    uint32_t seen[P];
#pragma unroll
    for (int q = 0; q < P; ++q) seen[q] = 0;
    bool ok = true;
    ns_walk<P>(p, cluster, pair, [&](const NsTask& t, const uint32_t (&base)[P]) {
      bool waited = false;
      auto reach = [&](uint32_t q, uint32_t l) {                  // the first l tasks of pair q are complete
#pragma unroll
        for (int r = 0; r < P; ++r) {
          if (P > 1 && static_cast<uint32_t>(r) != q) continue;
          while (ok && seen[r] < l) {
            ok = mbar_wait_cluster(&done[r * NSP_RING + seen[r] % NSP_RING], (seen[r] / NSP_RING) & 1, abort_flag, p.status, 5);
            ++seen[r];
            waited = true;
          }
        }
      };
      // the task with index `idx` in phase `ph` of iteration `it`
      auto require = [&](int it, int ph, uint32_t idx) {
        const uint32_t q = idx % P;
        const uint32_t c1 = ns_share<P>(t.wc * t1, q), c3 = ns_share<P>(t.wc * t3, q);
        uint32_t b = 0;
#pragma unroll
        for (int r = 0; r < P; ++r) if (static_cast<uint32_t>(r) == q) b = base[r];
        reach(q, b + it * (2 * c1 + c3) + ph * c1 + idx / P + 1);
      };
      // A barrier tells a phase only from its neighbours: this bounds how far behind the completions `seen` may be.
      if (P == 1) {
        if (t.l >= NSP_RING / 2) reach(0, t.l - NSP_RING / 2);
      } else {
#pragma unroll
        for (int q = 0; q < P; ++q) {                             // all phases before the last one
          const uint32_t c1 = ns_share<P>(t.wc * t1, q), c3 = ns_share<P>(t.wc * t3, q), sum = 2 * c1 + c3;
          reach(q, base[q] + (t.phase == 0 ? (t.it > 0 ? t.it * sum - c3 : 0) : t.phase == 1 ? t.it * sum : t.it * sum + c1));
        }
      }
      const bool diag = t.phase < 2 && t.i == t.j;
      const int ri = t.i * 256 + static_cast<int>(rank) * 128, rj = t.j * 256 + static_cast<int>(rank) * 128;
      const int nk = t.phase == 0 ? p.kl : p.ks;
      const int ba = buf_a(t), bb = buf_b(t), bx = buf_x(t, t.it);
      auto x_op = [&](bool mn, int idx, int kb) {
        NsOperand o;
        if (t.it == 0) {
          if (mn) o = {&maps.in_mn, idx, kb * 64, t.mat, 0, 64, true};
          else o = {&maps.in_k, kb * 64, idx, t.mat, 64, 0, false};
        } else {
          if (mn) o = {&maps.s_x, 0, kb * 64, bx * p.cx + (idx >> 6), 0, 64, false};
          else o = {&maps.s_k, 0, bx * p.rows_buf + kb * p.rpx + idx, 0, 0, p.rpx, false};
        }
        return o;
      };
      auto a_op = [&](int b, bool mn, int idx, int kb) {
        NsOperand o;
        if (mn) o = {&maps.s_a, 0, kb * 64, b * p.ca + (idx >> 6), 0, 64, false};
        else o = {&maps.s_k, 0, b * p.rows_buf + kb * p.rpa + idx, 0, 0, p.rpa, false};
        return o;
      };
      for (int kc = 0; kc * 4 < nk; ++kc) {
        const int kb0 = kc * 4, kb1 = min(nk, kb0 + 4);
        NsOperand oa, ob;
        if (t.phase == 0) {
          if (t.it > 0) { require(t.it - 1, 2, t.w * t3 + t.i * p.nc + kc); if (!diag) require(t.it - 1, 2, t.w * t3 + t.j * p.nc + kc); }
          oa = x_op(TALL, ri, kb0);
          ob = x_op(TALL, rj, kb0);
        } else if (t.phase == 1) {
          const int ha = max(t.i, kc), la = min(t.i, kc), hb = max(t.j, kc), lb = min(t.j, kc);
          require(t.it, 0, t.w * t1 + ha * (ha + 1) / 2 + la);
          if (!diag) require(t.it, 0, t.w * t1 + hb * (hb + 1) / 2 + lb);
          oa = a_op(ba, kc > t.i, ri, kb0);
          ob = a_op(ba, kc > t.j, rj, kb0);
        } else {
          const int h = max(t.i, kc), lo = min(t.i, kc);
          require(t.it, 1, t.w * t1 + h * (h + 1) / 2 + lo);
          if (t.it > 0) require(t.it - 1, 2, t.w * t3 + kc * p.nc + t.j);
          if (!TALL) { oa = a_op(bb, kc > t.i, ri, kb0); ob = x_op(true, rj, kb0); }
          else { oa = x_op(false, rj, kb0); ob = a_op(bb, kc > t.i, ri, kb0); }
        }
        if (waited) fence_proxy_async_global();       // what the waits have shown, for the loads that follow
        waited = false;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!ok || !mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, p.status, 5)) return ok = false;
          uint8_t* sA = smem + stage * NSP_STAGE;
          mbar_expect_tx(&full[stage], (diag ? 2 : 4) * NSP_OPERAND, leader ? e : 0);
          tma2_load_3d(sA, oa.tm, &full[stage], oa.x, oa.y, oa.z, e);
          if (oa.two) tma2_load_3d(sA + 8192, oa.tm, &full[stage], oa.x + 64, oa.y, oa.z, e);
          if (!diag) {
            tma2_load_3d(sA + NSP_OPERAND, ob.tm, &full[stage], ob.x, ob.y, ob.z, e);
            if (ob.two) tma2_load_3d(sA + NSP_OPERAND + 8192, ob.tm, &full[stage], ob.x + 64, ob.y, ob.z, e);
          }
          oa.x += oa.dx; oa.y += oa.dy; ob.x += ob.dx; ob.y += ob.dy;
          if (++stage == NSP_STAGES) { stage = 0; phase ^= 1; }
        }
      }
      return ok;
    });
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader)
    if (leader) {
      const uint32_t e = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      const uint32_t own = map_to_cta(smem_u32(full), lead_cta) - smem_u32(full), peer = map_to_cta(smem_u32(full), lead_cta + 1) - smem_u32(full);
      const uint64_t desc_k = umma_smem_desc(0, 16, 1024), desc_mn = umma_smem_desc(0, NSP_OPERAND / 2, 1024);
      ns_walk<P>(p, cluster, pair, [&](const NsTask& t, const uint32_t (&)[P]) {
        const uint32_t acc = t.l & 1;
        if (!mbar_wait_warp(&tempty[acc], ((t.l >> 1) & 1) ^ 1, abort_flag, p.status, 5)) return false;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        const bool diag = t.phase < 2 && t.i == t.j;
        const int nk = t.phase == 0 ? p.kl : p.ks;
        for (int kb = 0; kb < nk; ++kb) {
          const int kc = kb >> 2;
          bool mn_a, mn_b;
          if (t.phase == 0) { mn_a = mn_b = TALL; }
          else if (t.phase == 1) { mn_a = kc > t.i; mn_b = kc > t.j; }
          else if (!TALL) { mn_a = kc > t.i; mn_b = true; }
          else { mn_a = false; mn_b = kc > t.i; }
          const uint32_t a_base = smem_u32(smem + stage * NSP_STAGE) & 0x3FFFFu, b_base = diag ? a_base : a_base + NSP_OPERAND;
          const uint64_t adesc = (mn_a ? desc_mn : desc_k) + (a_base >> 4), bdesc = (mn_b ? desc_mn : desc_k) + (b_base >> 4);
          const uint32_t astep = mn_a ? 2048 >> 4 : 32 >> 4, bstep = mn_b ? 2048 >> 4 : 32 >> 4;
          const uint32_t idesc = umma_idesc_bf16(256, 256, false, false) | (mn_a ? 1u << 15 : 0u) | (mn_b ? 1u << 16 : 0u);
          if (!mbar_wait_warp(&full[stage], phase, abort_flag, p.status, 5)) return false;
          tc_fence_after();
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) umma2_ss(d_tmem, adesc + k * astep, bdesc + k * bstep, idesc, (kb > 0 || k > 0) ? 1u : 0u, e);
          const uint32_t bar = smem_u32(&empty[stage]);
          umma2_commit(bar + own, e);
          umma2_commit(bar + peer, e);
          if (++stage == NSP_STAGES) { stage = 0; phase ^= 1; }
        }
        const uint32_t bar = smem_u32(&tfull[acc]);
        umma2_commit(bar + own, e);
        umma2_commit(bar + peer, e);
        return true;
      });
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ output stores, completions
    const uint32_t e = elect_one();
    uint32_t stored[2][2] = {};
    ns_walk<P>(p, cluster, pair, [&](const NsTask& t, const uint32_t (&)[P]) {
      const bool last = t.phase == 2 && t.it == p.steps - 1;
      const int b = t.phase == 1 ? buf_b(t) : t.phase == 0 ? buf_a(t) : buf_x(t, t.it + 1);
      const NsPlace o[2] = {ns_place<TALL>(p, t, rank, 0), ns_place<TALL>(p, t, rank, 1)};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (c >= o[half].chunks) continue;
          if (!mbar_wait_warp(&slab_done[half * 2 + c], stored[half][c] & 1, abort_flag, p.status, 5)) return false;
          ++stored[half][c];
          const uint8_t* slab = slabs + (half * 2 + c) * NSP_SLAB;
          const int col = o[half].col0 + c * 64;
          if (e && o[half].live) {
            if (last) tma_store_3d(&maps.out, slab, col, o[half].row0, t.mat);
            else tma_store_3d(&maps.s_k, slab, 0, b * p.rows_buf + (col >> 6) * o[half].rp + o[half].row0, 0);
          }
          __syncwarp();
        }
        if (e) tma_store_commit();
        __syncwarp();
      }
      if (e) {
        tma_store_wait_read<1>();
        for (int half = 0; half < 2; ++half) if (0 < o[half].chunks) mbar_arrive(&slab_free[half * 2]);
        tma_store_wait_read<0>();
        for (int half = 0; half < 2; ++half) if (1 < o[half].chunks) mbar_arrive(&slab_free[half * 2 + 1]);
        tma_store_wait_all();
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        const uint32_t d = smem_u32(&done[pair * NSP_RING + t.l % NSP_RING]);
#pragma unroll
        for (int q = 0; q < 2 * P; ++q) mbar_arrive_relaxed(map_to_cta(d, q));
      }
      __syncwarp();
      return true;
    });
  } else if (warp == 3) {
    // ------------------------------------------------------------ aux loads into the slabs
    const uint32_t e = elect_one();
    const uint32_t t1 = p.nb * (p.nb + 1) / 2, t3 = p.nb * p.nc;
    uint32_t opened[2][2] = {};
    ns_walk<P>(p, cluster, pair, [&](const NsTask& t, const uint32_t (&)[P]) {
      // the task that wrote the aux values, if the slabs may be free before its outputs are in memory
      const uint32_t c1 = ns_share<P>(t.wc * t1, pair), c3 = ns_share<P>(t.wc * t3, pair), back = t.phase == 1 ? c1 : 2 * c1 + c3;
      if (t.phase > 0 && (t.phase == 1 || t.it > 0) && back == 1) {
        const uint32_t from = t.l - 1;
        if (!mbar_wait_cluster(&done[pair * NSP_RING + from % NSP_RING], (from / NSP_RING) & 1, abort_flag, p.status, 5)) return false;
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const NsPlace o = ns_place<TALL>(p, t, rank, half);
          if (c >= o.chunks) continue;
          const int s = half * 2 + c, col = o.col0 + c * 64;
          if (!mbar_wait_warp(&slab_free[s], (opened[half][c] & 1) ^ 1, abort_flag, p.status, 5)) return false;
          ++opened[half][c];
          if (e) {
            if (t.phase == 0 || !o.live) {
              mbar_arrive(&slab_open[s]);
            } else {
              mbar_expect_tx(&slab_open[s], NSP_SLAB);
              if (t.phase == 2 && t.it == 0) {
                tma_load_3d(slabs + s * NSP_SLAB, &maps.in_k, &slab_open[s], col, o.row0, t.mat);
              } else {
                const int b = t.phase == 1 ? buf_a(t) : buf_x(t, t.it);
                tma_load_3d(slabs + s * NSP_SLAB, &maps.s_k, &slab_open[s], 0, b * p.rows_buf + (col >> 6) * o.rp + o.row0, 0);
              }
            }
          }
          __syncwarp();
        }
      }
      return true;
    });
  } else {
    // ------------------------------------------------------------ epilogue: two groups of four warps, one per column half
    const int ew = warp & 3, half = (warp - 4) >> 2, row = ew * 32 + lane;
    uint8_t* my_row = slabs + half * 2 * NSP_SLAB + row * 128;
    uint64_t* open = slab_open + half * 2;
    uint64_t* combined = slab_done + half * 2;
    uint32_t used[2] = {0, 0};
    const uint32_t tempty_lead = map_to_cta(smem_u32(tempty), lead_cta);
    ns_walk<P>(p, cluster, pair, [&](const NsTask& t, const uint32_t (&)[P]) {
      const NsPlace o = ns_place<TALL>(p, t, rank, half);
      const uint32_t acc = t.l & 1;
      if (!mbar_wait_warp(&tfull[acc], (t.l >> 1) & 1, abort_flag, p.status, 5)) return false;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(ew * 32) << 16) + acc * 256 + half * 128;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (c < o.chunks) {
          if (!mbar_wait_warp(&open[c], used[c] & 1, abort_flag, p.status, 5)) return false;
          ++used[c];
          if (!o.live) {}
          else if (t.phase == 0) ns_slab<0>(t_row + c * 64, my_row + c * NSP_SLAB, lane);
          else if (t.phase == 1) ns_slab<1>(t_row + c * 64, my_row + c * NSP_SLAB, lane);
          else ns_slab<2>(t_row + c * 64, my_row + c * NSP_SLAB, lane);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&combined[c]);
        }
        if (c == 1) {                                             // the accumulator is drained
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(tempty_lead + acc * 8);
        }
      }
      return true;
    });
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                           // a wait ran out: copies and products in flight end before the CTA does
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000) {}
  }
  cluster_sync_all();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
}

constexpr size_t NSP_SMEM = 1024 + NSP_STAGES * NSP_STAGE + 4 * NSP_SLAB + 2048;
static_assert(NSP_SMEM <= 232448, "shared memory budget of one CTA exceeded");

using NsPairKernel = void (*)(NsPairMaps, NsPairDev);
static NsPairKernel nsp_kernel(bool tall, int P) {
  switch (P) {
    case 1: return tall ? ns_pair_kernel<true, 1> : ns_pair_kernel<false, 1>;
    case 2: return tall ? ns_pair_kernel<true, 2> : ns_pair_kernel<false, 2>;
    case 4: return tall ? ns_pair_kernel<true, 4> : ns_pair_kernel<false, 4>;
    default: throw std::runtime_error("himuon ns_pair: one, two or four pairs per matrix");
  }
}

static cudaLaunchConfig_t nsp_config(int clusters, int P, cudaLaunchAttribute* attr, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * 2 * P));
  cfg.blockDim = dim3(NSP_THREADS);
  cfg.dynamicSmemBytes = NSP_SMEM;
  cfg.stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = static_cast<unsigned>(2 * P);
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

static int nsp_max_clusters(int P) {
  static int cache[64][NSP_MAXP + 1] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cache[dev][P] == 0) {
    for (int tall = 0; tall < 2; ++tall)
      cudaFuncSetAttribute(nsp_kernel(tall, P), cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(NSP_SMEM));
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = nsp_config(num_sms() / (2 * P), P, &attr, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, nsp_kernel(false, P), &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = num_sms() / (4 * P); }
    cache[dev][P] = n;
  }
  return cache[dev][P];
}

// Pairs per matrix and matrices interleaved per cluster, or false where the GEMM launches are the better path.
//   * Short sides above 512 stay with the GEMMs: 4 matrices of 1024 x 1024 took 248 us there, 389 here (28 of them 779 / 608, but no
//     rule is drawn from one figure).  So do more than 1024 columns in two blocks (one matrix of 512 x 2048 191 / 207), 2048
//     in one.  Short sides up to 128 use half of a block's rows, so the GEMMs catch up with many matrices.
//   * As many pairs per matrix as all matrices at once leave, while they have work: 4 of 336 x 504 with 1, 2, 4 pairs 145,
//     112, 107 us, of 256 x 1024 120, 101, 101, of 256 x 512 91, 85, 89, of 256 x 256 77, 80, 84.
//   * One block per phase leaves nothing to hide the hand-on behind but other matrices: 396 of 256 x 256 interleaved by
//     1, 2, 3, 4: 480, 381, 345, 309 us; with several blocks two are enough (296 of 256 x 512: 266 with two, 311 with four).
//   * More matrices than pairs take whole rounds, where the GEMMs' time goes with the number: ns_rounds_pay.
//   * One to four matrices that half-fill eight blocks: 384 x 1024 135 us there, 139 here (264 x 1024 139 / 135).
// Below, time here / there, from one round of matrices (74) to four.
static bool ns_rounds_pay(long long n_mats, int s, int l, bool tall, long long slots) {
  const int nb = (s + 255) / 256, nc = (l + 255) / 256;
  const long long rounds = (n_mats + slots - 1) / slots;
  auto filled = [&](int percent) { return n_mats * 100 >= percent * rounds * slots; };
  if (rounds == 1) return true;
  if (s <= 128) {
    if (n_mats > 4 * slots) return false;             // 64 x 2000: 100 matrices 257 / 348
    // wide: 16 x 512 75-148 matrices 0.79-0.82, 150-296 1.04-1.10; 128 x 768 92 1.04, 100 0.95, 150-296 1.03-1.15; 16 x 1024
    // 75-148 1.03-1.15.  The GEMMs are slower on tall ones: 512 x 128 150-296 0.92-0.99, 264 x 16 0.88-0.93, but 264 x 128 1.01-1.08;
    // 768 x 128 185-296 0.92-0.97, 640 x 128 1.01-1.09, 1024 x 16 75-148 0.83-0.95, 150-260 0.99-1.08.
    if (nc == 1) return true;
    if (!tall) return rounds == 2 && (nc == 2 || (nc == 3 && filled(66)));
    return rounds == 2 || (nc < 4 && (l * 10 >= nc * 2304 || (nc == 2 && s <= 64)));
  }
  if (nb == 1 || nc < 3) return true;                 // 256 x 2048 75 matrices 0.94; 384 x 512 75 1.00, 150 0.94
  // Two block rows, the second up to half full: 264 x 768 75 matrices 1.11, 100 0.90, 150 1.01, 185 0.87, 223 0.91; 384 x 1024 75
  // 1.20, 100 0.99, 150 1.17; 264 x 1024 165 1.06, 185 0.95; tall 768 x 264 75 0.94, 150 0.83, but 1024 x 384 92 1.11.  More than
  // half: 512 x 1024 75 1.01, 84 0.97; 448 x 768 0.69-0.89.
  if (s > 384) return nc == 3 || filled(54);
  return (tall && s <= 288) || filled(rounds == 2 ? 66 : nc == 3 ? 72 : 80);
}
bool ns_pair_plan(long long n_mats, int m, int n, int* P, int* W) {
  const int s = m < n ? m : n, l = m < n ? n : m, nb = (s + 255) / 256, nc = (l + 255) / 256;
  if (n_mats <= 0 || m <= 0 || n <= 0 || m % 8 || n % 8 || nb > 2 || nc > (nb == 2 || s <= 128 ? 4 : 8)) return false;
  if (!ns_rounds_pay(n_mats, s, l, m > n, nsp_max_clusters(1)) || (nc == 4 && nb == 2 && s > 288 && n_mats < 5)) return false;
  *P = n_mats <= nsp_max_clusters(4) && nb * nc >= 4 ? 4 : n_mats <= nsp_max_clusters(2) && nb * nc >= 2 ? 2 : 1;
  const long long each = (n_mats + nsp_max_clusters(1) - 1) / nsp_max_clusters(1), most = nc == 1 ? 4 : 2;
  *W = nb == 2 || *P > 1 ? 1 : static_cast<int>(each < most ? each : most);
  return true;
}

static NsPairDev nsp_shape(long long n_mats, int m, int n, int P, int W) {
  NsPairDev d{};
  d.n_mats = n_mats; d.m = m; d.n = n; d.W = W;
  const int s = m < n ? m : n, l = m < n ? n : m;
  d.nb = (s + 255) / 256; d.nc = (l + 255) / 256; d.ks = (s + 63) / 64; d.kl = (l + 63) / 64;
  d.rpa = d.nb * 256; d.rpx = m > n ? d.nc * 256 : d.nb * 256;
  d.rows_buf = d.nb * 256 * d.nc * 4;
  d.cx = d.rows_buf / d.rpx; d.ca = d.rows_buf / d.rpa;
  d.bufs = P == 1 && m <= n ? 3 : 4;
  const long long cap = nsp_max_clusters(P);
  d.clusters = n_mats < cap ? n_mats : cap;
  return d;
}
long long ns_pair_scratch_bytes(long long n_mats, int m, int n, int P, int W) {
  const NsPairDev d = nsp_shape(n_mats, m, n, P, W);
  return d.clusters * W * d.bufs * d.rows_buf * 128;
}

// `out` may be `in` from two steps on: the input is read in the first one only.
void ns_pair(const void* in, void* out, void* scratch, long long n_mats, int m, int n, int steps, int P, int W, cudaStream_t s) {
  if (n_mats <= 0 || steps <= 0) return;
  if (n_mats >= (1LL << 31)) throw std::runtime_error("himuon ns_pair: too many matrices");
  NsPairDev d = nsp_shape(n_mats, m, n, P, W);
  // a barrier of the ring has to be seen before it comes round: three phases of tasks of one pair at most (NSP_RING)
  const int t1 = W * d.nb * (d.nb + 1) / 2, t3 = W * d.nb * d.nc;
  if (P > 1 && 2 * ((t1 + P - 1) / P) + (t3 + P - 1) / P >= NSP_RING) throw std::runtime_error("himuon ns_pair: too many blocks per pair");
  d.steps = steps;
  d.status = status_word_ptr();
  NsPairMaps t;
  const uint64_t dims_io[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(m), static_cast<uint64_t>(n_mats)};
  const uint64_t str_io[2] = {static_cast<uint64_t>(n) * 2, static_cast<uint64_t>(n) * 2 * m};
  const uint32_t box128[3] = {64, 128, 1}, box64[3] = {64, 64, 1}, box64x2[3] = {64, 64, 2};
  t.in_k = make_tmap(in, 3, dims_io, str_io, box128, 2, true);
  t.in_mn = make_tmap(in, 3, dims_io, str_io, box64, 2, true);
  t.out = make_tmap(out, 3, dims_io, str_io, box128, 2, true);
  const uint64_t bufs = static_cast<uint64_t>(d.clusters) * W * d.bufs, rows = bufs * d.rows_buf;
  const uint64_t dims_s[3] = {64, rows, 1}, str_s[2] = {128, rows * 128};
  t.s_k = make_tmap(scratch, 3, dims_s, str_s, box128, 2, true);
  const uint64_t dims_x[3] = {64, static_cast<uint64_t>(d.rpx), bufs * d.cx}, str_x[2] = {128, static_cast<uint64_t>(d.rpx) * 128};
  const uint64_t dims_a[3] = {64, static_cast<uint64_t>(d.rpa), bufs * d.ca}, str_a[2] = {128, static_cast<uint64_t>(d.rpa) * 128};
  t.s_x = make_tmap(scratch, 3, dims_x, str_x, box64x2, 2, true);
  t.s_a = make_tmap(scratch, 3, dims_a, str_a, box64x2, 2, true);
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = nsp_config(static_cast<int>(d.clusters), P, &attr, s);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, nsp_kernel(m > n, P), t, d);
  if (e != cudaSuccess) throw std::runtime_error(std::string("himuon ns_pair launch failed: ") + cudaGetErrorString(e));
}

}  // namespace himuon
