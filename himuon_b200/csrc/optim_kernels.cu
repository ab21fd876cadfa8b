// Multi-tensor optimizer kernels (HBM-bound): each runs ONE launch over every matrix of a
// bucket, driven by a device-resident entry table.
//
//   momentum_tile : sum of gradient replicas (this rank's and, under sharding, the peers' through
//                   peer pointers) -> scale -> momentum update -> Nesterov -> zero-padded tile layout
//                   (the reference's separate launches: src/himuon/optimizers/himuon.py:350-357, 713-719)
//   ns_normalize  : per-tile Frobenius normalisation (himuon.py:241 / triton_kernels/ns5_smem.py:84-88)
//   untile_apply  : untile + crop + lr-scale + decoupled weight decay + parameter update
//                   (himuon.py:315-348, 215-228) with lr / wd read from a device table, so a captured
//                   CUDA graph follows the LR schedule without recapture
//   adamw_multi   : the three AdamW conventions used by the optimizers (himuon.py:359-372,
//                   muon.py:171-193, adamw.py:86-116)
#include "himuon.h"
#include "sm100_common.cuh"

namespace himuon {

constexpr int kRowsPerUnit = 16;

int momentum_tile_units(int R, int C, int Th) { return R * C * ((Th + kRowsPerUnit - 1) / kRowsPerUnit); }

template <typename Entry>
__device__ __forceinline__ int find_entry(const Entry* e, int n, long long unit) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (static_cast<long long>(e[mid].unit_begin) <= unit) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// One 16-byte access of a gradient, momentum or parameter tensor: 8 bf16 or 4 fp32 elements.
template <typename T> struct Vec16 {
  static constexpr int N = 16 / sizeof(T);
  __device__ static __forceinline__ void unpack(const uint4& v, float (&f)[N]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if constexpr (sizeof(T) == 2) { f[2 * q] = bf16_lo(w[q]); f[2 * q + 1] = bf16_hi(w[q]); }
      else f[q] = __uint_as_float(w[q]);
    }
  }
  __device__ static __forceinline__ uint4 pack(const float (&f)[N]) {
    if constexpr (sizeof(T) == 2)
      return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
    else
      return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};
// N elements (8 or 4) of the bf16 tile buffer.
template <int N> __device__ __forceinline__ void store_tile(__nv_bfloat16* p, const float (&f)[N]) {
  if constexpr (N == 8) *reinterpret_cast<uint4*>(p) = Vec16<__nv_bfloat16>::pack(f);
  else *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
}
template <int N> __device__ __forceinline__ void load_tile(const __nv_bfloat16* p, float (&f)[N]) {
  if constexpr (N == 8) Vec16<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(p), f);
  else {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x); f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
  }
}
template <int N> __device__ __forceinline__ bool tiles_aligned(const __nv_bfloat16* tiles) {
  return (reinterpret_cast<uintptr_t>(tiles) & (2 * N - 1)) == 0;
}

// ------------------------------------------------------------------------------------------------
// Bound by HBM: gradient(s), momentum in and out, tile out.  The 16-byte path takes every matrix whose rows and row
// widths are whole 16-byte vectors on aligned tensors (anything else goes element by element: a parameter or gradient
// may be a view that starts anywhere): U vectors per thread and pass with their loads issued together, 2 of 8 bf16
// elements or 4 of 4 fp32 elements.
// Measured on fp32 matrices of a 640-wide model with tile 256 (19 M elements) and an embedding of 27 M: optimizer step
// 1103 -> 846 us with this path for fp32 here, in untile_apply and in adamw_multi; bf16 is unchanged.
// For bf16 the four conversions of an element bound it as long as they went one at a time: 604 M elements in tiles of 512
// 1050 -> 940 us with pairs (740 at the copy rate).  fp32 gained by reading the entry in place: 77.7 -> 62.3 us.
// Four vectors of bf16 in flight are slower (1340 us), and so are streaming hints (1160) and units in bands across tiles (1095).
template <typename G>
__global__ void __launch_bounds__(256)
momentum_tile_kernel(const MomTileEntry* __restrict__ entries, int n_entries, int total_units, int Th, int Tw,
                     __nv_bfloat16* __restrict__ tiles, float mu, int nesterov, float gscale, int n_src) {
  constexpr int VN = Vec16<G>::N, U = sizeof(G) == 2 ? 2 : 4;
  const int row_blocks = (Th + kRowsPerUnit - 1) / kRowsPerUnit;
  for (int unit = blockIdx.x; unit < total_units; unit += gridDim.x) {
    const int ei = find_entry(entries, n_entries, unit);
    const MomTileEntry& e = entries[ei];                  // not a copy: its indexed source pointers would live in local memory
    const int local = unit - e.unit_begin;
    const int t = local / row_blocks;
    const int rb = local - t * row_blocks;
    const int tr = t / e.C, tc = t - tr * e.C;
    __nv_bfloat16* out = tiles + (e.tile_base + t) * static_cast<long long>(Th) * Tw;
    G* mom = reinterpret_cast<G*>(e.mom);
    const int i0 = rb * kRowsPerUnit;
    const int i1 = min(Th, i0 + kRowsPerUnit);
    bool vec = (Tw % VN == 0) && (e.ld % VN == 0) && (e.w % VN == 0) && tiles_aligned<VN>(tiles);
    if (vec) {
      uintptr_t addr = reinterpret_cast<uintptr_t>(e.mom);
      for (int s = 0; s < n_src; ++s) addr |= reinterpret_cast<uintptr_t>(e.grad[s]);
      vec = (addr & 15) == 0;
    }
    if (vec) {
      const int vec_per_row = Tw / VN;
      const int nvec = (i1 - i0) * vec_per_row;
      for (int x0 = threadIdx.x; x0 < nvec; x0 += U * blockDim.x) {
        bool live[U], inside[U];
        int ii[U], jj[U];
        long long off[U], moff[U];
        float g[U][VN];
        uint4 mv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int x = x0 + u * static_cast<int>(blockDim.x);
          live[u] = x < nvec;
          ii[u] = i0 + x / vec_per_row;
          jj[u] = (x % vec_per_row) * VN;
          const int gi = tr * Th + ii[u], gj = tc * Tw + jj[u];
          inside[u] = live[u] && gi < e.h && gj < e.w;
          off[u] = static_cast<long long>(gi) * e.ld + gj;
          moff[u] = static_cast<long long>(gi) * e.w + gj;
#pragma unroll
          for (int q = 0; q < VN; ++q) g[u][q] = 0.f;
          mv[u] = make_uint4(0, 0, 0, 0);
          if (inside[u]) mv[u] = *reinterpret_cast<const uint4*>(mom + moff[u]);
        }
        for (int sidx = 0; sidx < n_src; ++sidx) {
          uint4 gv[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            gv[u] = make_uint4(0, 0, 0, 0);
            if (inside[u]) gv[u] = *reinterpret_cast<const uint4*>(reinterpret_cast<const G*>(e.grad[sidx]) + off[u]);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            float f[VN];
            Vec16<G>::unpack(gv[u], f);
#pragma unroll
            for (int q = 0; q < VN; ++q) g[u][q] += f[q];
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!live[u]) continue;
          float r[VN], m[VN];
#pragma unroll
          for (int q = 0; q < VN; ++q) r[q] = 0.f;
          if (inside[u]) {
            Vec16<G>::unpack(mv[u], m);
#pragma unroll
            for (int q = 0; q < VN; q += 2) {
              float g0 = g[u][q] * gscale, g1 = g[u][q + 1] * gscale, b0, b1;
              if constexpr (sizeof(G) == 2) {
                // the gradient as the optimizer would see it (stored precision), then buf = mu*buf + g
                round_bf16x2(g0, g1);
                float m0 = m[q] * mu, m1 = m[q + 1] * mu;
                round_bf16x2(m0, m1);
                b0 = m0 + g0;
                b1 = m1 + g1;
                round_bf16x2(b0, b1);
              } else {
                b0 = m[q] * mu + g0;
                b1 = m[q + 1] * mu + g1;
              }
              m[q] = b0;
              m[q + 1] = b1;
              r[q] = nesterov ? g0 + mu * b0 : b0;         // rounded to bf16 as it is stored
              r[q + 1] = nesterov ? g1 + mu * b1 : b1;
            }
            *reinterpret_cast<uint4*>(mom + moff[u]) = Vec16<G>::pack(m);
          }
          store_tile<VN>(out + static_cast<long long>(ii[u]) * Tw + jj[u], r);
        }
      }
    } else {
      const int n = (i1 - i0) * Tw;
      for (int x = threadIdx.x; x < n; x += blockDim.x) {
        const int i = i0 + x / Tw;
        const int j = x % Tw;
        const int gi = tr * Th + i, gj = tc * Tw + j;
        float r = 0.f;
        if (gi < e.h && gj < e.w) {
          const long long off = static_cast<long long>(gi) * e.ld + gj;
          float g = 0.f;
          for (int s = 0; s < n_src; ++s) g += ldf(reinterpret_cast<const G*>(e.grad[s]) + off);
          g *= gscale;
          const long long moff = static_cast<long long>(gi) * e.w + gj;
          float b;
          if (sizeof(G) == 2) {
            g = round_bf16(g);
            b = round_bf16(round_bf16(ldf(mom + moff) * mu) + g);
            r = nesterov ? round_bf16(g + mu * b) : b;
          } else {
            b = ldf(mom + moff) * mu + g;
            r = nesterov ? g + mu * b : b;
          }
          stf(mom + moff, b);
        }
        out[static_cast<long long>(i) * Tw + j] = __float2bfloat16_rn(r);
      }
    }
  }
}

void momentum_tile(const MomTileEntry* entries, int n_entries, int total_units, int Th, int Tw, void* tiles,
                   float momentum, int nesterov, float grad_scale, int n_src, int grad_fp32, cudaStream_t stream) {
  if (total_units <= 0) return;
  const int grid = total_units < num_sms() * 16 ? total_units : num_sms() * 16;
  if (grad_fp32)
    momentum_tile_kernel<float><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, Th, Tw,
                                                          reinterpret_cast<__nv_bfloat16*>(tiles), momentum, nesterov,
                                                          grad_scale, n_src);
  else
    momentum_tile_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, Th, Tw,
                                                                  reinterpret_cast<__nv_bfloat16*>(tiles), momentum,
                                                                  nesterov, grad_scale, n_src);
}

// ------------------------------------------------------------------------------------------------
// Decay, rounded to the parameter's type, then one multiply-add: spelled out, so that every path rounds alike.
template <typename P>
__device__ __forceinline__ void apply_update(float& p0, float& p1, bool has_decay, float decay, float step, float u0, float u1) {
  if (has_decay) {
    p0 = __fmul_rn(p0, decay);
    p1 = __fmul_rn(p1, decay);
    if (sizeof(P) == 2) round_bf16x2(p0, p1);
  }
  p0 = __fmaf_rn(-step, u0, p0);
  p1 = __fmaf_rn(-step, u1, p1);
}
template <typename P>
__device__ __forceinline__ float apply_update(float p, bool has_decay, float decay, float step, float u) {
  float unused = 0.f;
  apply_update<P>(p, unused, has_decay, decay, step, u, 0.f);
  return p;
}
template <typename P>
__global__ void __launch_bounds__(256)
untile_apply_kernel(const ApplyEntry* __restrict__ entries, int n_entries, int total_units, int Th, int Tw,
                    const __nv_bfloat16* __restrict__ tiles, const float* __restrict__ hyper) {
  constexpr int VN = Vec16<P>::N, U = sizeof(P) == 2 ? 2 : 4;
  const int row_blocks = (Th + kRowsPerUnit - 1) / kRowsPerUnit;
  for (int unit = blockIdx.x; unit < total_units; unit += gridDim.x) {
    const int ei = find_entry(entries, n_entries, unit);
    const ApplyEntry e = entries[ei];
    const float lr = hyper[8 * e.group], wd = hyper[8 * e.group + 1];
    const float decay = wd > 0.f ? 1.f - lr * wd : 1.f;
    const float step = lr * e.scale;
    const int local = unit - e.unit_begin;
    const int t = local / row_blocks;
    const int rb = local - t * row_blocks;
    const int tr = t / e.C, tc = t - tr * e.C;
    const __nv_bfloat16* in = tiles + (e.tile_base + t) * static_cast<long long>(Th) * Tw;
    P* param = reinterpret_cast<P*>(e.param);
    const int i0 = rb * kRowsPerUnit;
    const int i1 = min(Th, i0 + kRowsPerUnit);
    const bool vec = (Tw % VN == 0) && (e.ld % VN == 0) && (e.w % VN == 0) && tiles_aligned<VN>(tiles) &&
                     (reinterpret_cast<uintptr_t>(e.param) & 15) == 0;
    if (vec) {
      const int vec_per_row = Tw / VN;
      const int nvec = (i1 - i0) * vec_per_row;
      for (int x0 = threadIdx.x; x0 < nvec; x0 += U * blockDim.x) {
        bool inside[U];
        P* pp[U];
        uint4 pv[U];
        float uf[U][VN];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int x = x0 + u * static_cast<int>(blockDim.x);
          const int i = i0 + x / vec_per_row;
          const int j = (x % vec_per_row) * VN;
          const int gi = tr * Th + i, gj = tc * Tw + j;
          inside[u] = x < nvec && gi < e.h && gj < e.w;
          pp[u] = param + static_cast<long long>(gi) * e.ld + gj;
          pv[u] = make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int q = 0; q < VN; ++q) uf[u][q] = 0.f;
          if (inside[u]) {
            load_tile<VN>(in + static_cast<long long>(i) * Tw + j, uf[u]);
            pv[u] = *reinterpret_cast<const uint4*>(pp[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!inside[u]) continue;
          float f[VN];
          Vec16<P>::unpack(pv[u], f);
#pragma unroll
          for (int q = 0; q < VN; q += 2) apply_update<P>(f[q], f[q + 1], wd > 0.f, decay, step, uf[u][q], uf[u][q + 1]);
          *reinterpret_cast<uint4*>(pp[u]) = Vec16<P>::pack(f);
        }
      }
    } else {
      const int n = (i1 - i0) * Tw;
      for (int x = threadIdx.x; x < n; x += blockDim.x) {
        const int i = i0 + x / Tw;
        const int j = x % Tw;
        const int gi = tr * Th + i, gj = tc * Tw + j;
        if (gi >= e.h || gj >= e.w) continue;
        const float u = __bfloat162float(in[static_cast<long long>(i) * Tw + j]);
        P* pp = param + static_cast<long long>(gi) * e.ld + gj;
        stf(pp, apply_update<P>(ldf(pp), wd > 0.f, decay, step, u));
      }
    }
  }
}

void untile_apply(const ApplyEntry* entries, int n_entries, int total_units, int Th, int Tw, const void* tiles,
                  const float* hyper, int param_fp32, cudaStream_t stream) {
  if (total_units <= 0) return;
  const int grid = total_units < num_sms() * 16 ? total_units : num_sms() * 16;
  if (param_fp32)
    untile_apply_kernel<float><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, Th, Tw,
                                                         reinterpret_cast<const __nv_bfloat16*>(tiles), hyper);
  else
    untile_apply_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, Th, Tw,
                                                                 reinterpret_cast<const __nv_bfloat16*>(tiles), hyper);
}

// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (warp == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// Adds the squares of eight bf16 elements to a chain of sums.
__device__ __forceinline__ void add_squares8(float& ss, const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float a = bf16_lo(w[q]), b = bf16_hi(w[q]); ss += a * a + b * b; }
}

__global__ void __launch_bounds__(1024)
ns_normalize_kernel(const __nv_bfloat16* tiles, __nv_bfloat16* out, long long n_tiles, long long tile_elems, float eps) {
  __shared__ float red[32];
  for (long long t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const __nv_bfloat16* x = tiles + t * tile_elems;
    __nv_bfloat16* y = out + t * tile_elems;             // may alias x (in place)
    float ss = 0.f;
    if ((tile_elems & 7) == 0) {
      const long long nv = tile_elems >> 3;
      const uint4* xv = reinterpret_cast<const uint4*>(x);
      long long i = threadIdx.x;
      for (; i + 3 * blockDim.x < nv; i += 4 * blockDim.x) {      // four independent loads in flight per thread
        uint4 v4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v4[u] = xv[i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < 4; ++u) add_squares8(ss, v4[u]);
      }
      for (; i < nv; i += blockDim.x) add_squares8(ss, xv[i]);
    } else {
      for (long long i = threadIdx.x; i < tile_elems; i += blockDim.x) { const float a = __bfloat162float(x[i]); ss += a * a; }
    }
    const float tot = block_sum(ss, red);
    // an all-zero (padding) tile stays exactly zero (inv = 0 also covers the out-of-place copy); uniform over the block
    if (tot == 0.f && y == x) continue;
    const float inv = tot == 0.f ? 0.f : 1.f / (sqrtf(tot) + eps);
    if ((tile_elems & 7) == 0) {
      const long long nv = tile_elems >> 3;
      const uint4* xv = reinterpret_cast<const uint4*>(x);
      uint4* yv = reinterpret_cast<uint4*>(y);
      long long i = threadIdx.x;
      for (; i + 3 * blockDim.x < nv; i += 4 * blockDim.x) {
        uint4 v4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v4[u] = xv[i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t w[4] = {v4[u].x, v4[u].y, v4[u].z, v4[u].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(bf16_lo(w[q]) * inv, bf16_hi(w[q]) * inv);
          yv[i + u * blockDim.x] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      for (; i < nv; i += blockDim.x) {
        uint4 v = xv[i];
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(bf16_lo(w[q]) * inv, bf16_hi(w[q]) * inv);
        yv[i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    } else {
      for (long long i = threadIdx.x; i < tile_elems; i += blockDim.x) y[i] = __float2bfloat16_rn(__bfloat162float(x[i]) * inv);
    }
  }
}

// Normalisation of tiles of 64 Ki elements and more: a cluster of eight CTAs per tile, for launches of few large tiles,
// which one CTA per tile spread over too few SMs.  The sum of squares is built in the order of the kernel above (1024
// chains, chain c adding the vectors c, c + 1024, ...; then a tree over the chains of each warp and one over the 32
// warps), so that a tile's result does not depend on how many tiles share its launch: CTA r owns chains 128 r ... 128 r +
// 127, one thread each, and the 32 warp sums meet in the distributed shared memory of every CTA.  A chain is serial, so the
// bytes in flight come from a ring of kNormRing vectors per chain that asynchronous copies fill ahead of it; a tile whose chains
// fit the ring is read once.  All threads of the CTA share the second pass.
constexpr int kNormCluster = 8, kNormChains = 1024, kNormOwn = kNormChains / kNormCluster, kNormThreads = 512, kNormGroup = 8;
constexpr int kNormRing = 32;                              // 64 KB
__device__ __forceinline__ uint4 scale8(const uint4& v, float f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = pack_bf16x2(bf16_lo(w[q]) * f, bf16_hi(w[q]) * f);
  return make_uint4(o[0], o[1], o[2], o[3]);
}
template <bool ONCE>     // the chains fit the ring
__global__ void __cluster_dims__(kNormCluster, 1, 1) __launch_bounds__(kNormThreads, ONCE ? 3 : 2)
ns_normalize_cluster_kernel(const uint4* tiles, uint4* out, long long nv, float eps) {
  extern __shared__ uint4 ring[];                          // [kNormRing][kNormOwn]
  __shared__ float red[kNormChains / 32];
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // waited for before the first remote store
  const uint32_t rank = blockIdx.x % kNormCluster;         // clusters are runs of consecutive blocks
  const long long t = blockIdx.x / kNormCluster;
  const uint4* x = tiles + t * nv;
  uint4* y = out + t * nv;                                 // may alias x (in place)
  const long long base = static_cast<long long>(rank) * kNormOwn;
  const int len = static_cast<int>((nv + kNormChains - 1) / kNormChains);  // vectors of the longest chain
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float ss = 0.f;
  if (threadIdx.x < kNormOwn) {
    const long long first = base + threadIdx.x;
    auto fetch = [&](int g) {                              // one group of copies; zeros past the end
#pragma unroll
      for (int u = 0; u < kNormGroup; ++u) {
        const int k = g * kNormGroup + u;
        const long long i = first + static_cast<long long>(k) * kNormChains;
        const uint32_t dst = smem_u32(ring + (k % kNormRing) * kNormOwn + threadIdx.x);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(x + (i < nv ? i : 0)), "r"(i < nv ? 16 : 0)
                     : "memory");
      }
    };
    const int groups = (len + kNormGroup - 1) / kNormGroup;
    for (int g = 0; g < kNormRing / kNormGroup; ++g) {
      if (g < groups) fetch(g);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int g = 0; g < groups; ++g) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kNormRing / kNormGroup - 1) : "memory");
#pragma unroll
      for (int u = 0; u < kNormGroup; ++u) add_squares8(ss, ring[((g * kNormGroup + u) % kNormRing) * kNormOwn + threadIdx.x]);
      if (g + kNormRing / kNormGroup < groups) fetch(g + kNormRing / kNormGroup);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // every CTA of the cluster has started
  if (threadIdx.x < kNormOwn && lane < kNormCluster) {     // hand the warp's sum to every CTA of the cluster
    uint32_t dst;
    const uint32_t local = smem_u32(&red[rank * (kNormOwn / 32) + warp]);
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(local), "r"(lane));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(ss) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  float tot = red[lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  // an all-zero (padding) tile stays exactly zero (inv = 0 also covers the out-of-place copy); uniform over the cluster
  if (tot == 0.f && y == x) return;
  const float inv = tot == 0.f ? 0.f : 1.f / (sqrtf(tot) + eps);
  const int c = threadIdx.x % kNormOwn;
  constexpr int kStep = kNormThreads / kNormOwn;
  if (ONCE) {
    for (int k = threadIdx.x / kNormOwn; k < len; k += kStep) {
      const long long i = base + c + static_cast<long long>(k) * kNormChains;
      if (i < nv) y[i] = scale8(ring[k * kNormOwn + c], inv);
    }
    return;
  }
  for (int k0 = threadIdx.x / kNormOwn; k0 < len; k0 += kStep * kNormGroup) {
    uint4 v[kNormGroup];                                   // loads together, ahead of the stores, which may alias them
#pragma unroll
    for (int u = 0; u < kNormGroup; ++u) {
      const long long i = base + c + static_cast<long long>(k0 + u * kStep) * kNormChains;
      if (i < nv) v[u] = x[i];
    }
#pragma unroll
    for (int u = 0; u < kNormGroup; ++u) {
      const long long i = base + c + static_cast<long long>(k0 + u * kStep) * kNormChains;
      if (i < nv) y[i] = scale8(v[u], inv);
    }
  }
}

void ns_normalize(void* tiles, long long n_tiles, long long tile_elems, float eps, cudaStream_t stream, void* out) {
  if (n_tiles <= 0) return;
  // A cluster per tile where one CTA per tile would leave half of the SMs idle.  Measured with clusters, and with one CTA
  // per tile where that is known: 28 tiles of 512 6.4 us (17), 74 of them 13.7 (75 of them with one CTA each: 17.5), 8 of
  // 1024 x 3072 32, 74 of 1024 72 (75: 88), 74 of 256 6.9 (75: 6.0).  The clusters are still level or ahead at the line;
  // past it one CTA per tile fills the chip by itself.  From 256 x 256 elements every thread has eight loads or more.
  if (tile_elems % 8 == 0 && tile_elems >= 65536 && tile_elems < (1LL << 40) && n_tiles * 2 <= num_sms()) {
    constexpr int smem = kNormRing * kNormOwn * 16;
    const bool once = tile_elems <= 8LL * kNormChains * kNormRing;
    auto kern = once ? ns_normalize_cluster_kernel<true> : ns_normalize_cluster_kernel<false>;
    static bool attr[2][64] = {};                          // per device: the one-CTA kernel runs on any of them without a word
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !attr[once][dev]) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (dev < 64) attr[once][dev] = true;
    }
    kern<<<static_cast<unsigned>(n_tiles * kNormCluster), kNormThreads, smem, stream>>>(
        reinterpret_cast<const uint4*>(tiles), reinterpret_cast<uint4*>(out ? out : tiles), tile_elems / 8, eps);
    return;
  }
  const long long cap = static_cast<long long>(num_sms()) * 2;
  const int grid = static_cast<int>(n_tiles < cap ? n_tiles : cap);
  const int threads = tile_elems >= 8192 ? 1024 : 256;
  ns_normalize_kernel<<<grid, threads, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(tiles),
                                                    reinterpret_cast<__nv_bfloat16*>(out ? out : tiles), n_tiles, tile_elems, eps);
}

// ------------------------------------------------------------------------------------------------
// Newton-Schulz on sides that are no multiples of 8: (B, sm, sn) of S -> (B, dm, dn) of D, rows and columns past the
// source filled with zeros, those past the destination dropped, element type converted on the way, and matrix b divided by
// norm[b] + eps where norms are given (IEEE division, as PyTorch divides).  One launch on each side of the iteration and
// one for the scaling, in place of the cast, pad, divide, cast, copy and crop launches of PyTorch.  Odd rows have no common
// alignment, so accesses are single elements, coalesced along the row.  `src` may be `dst` when the sizes are the same.
template <typename S, typename D>
__global__ void __launch_bounds__(256)
repad_kernel(const S* src, D* dst, int sm, int sn, int dm, int dn, const float* norm, float eps) {
  const S* s = src + static_cast<long long>(blockIdx.y) * sm * sn;
  D* d = dst + static_cast<long long>(blockIdx.y) * dm * dn;
  const float div = norm ? __fadd_rn(norm[blockIdx.y], eps) : 1.f;
  for (int i = blockIdx.x; i < dm; i += gridDim.x)
    for (int j = threadIdx.x; j < dn; j += blockDim.x) {
      const float v = (i < sm && j < sn) ? ldf(s + static_cast<long long>(i) * sn + j) : 0.f;
      stf(d + static_cast<long long>(i) * dn + j, norm ? __fdiv_rn(v, div) : v);
    }
}
void ns_repad(const void* src, void* dst, long long batch, int sm, int sn, int dm, int dn, int src_fp32, int dst_fp32,
              cudaStream_t stream, const float* norm, float eps) {
  if (batch <= 0 || dm <= 0 || dn <= 0) return;
  for (long long b0 = 0; b0 < batch; b0 += 65535) {       // grid.y limit
    const unsigned nb = static_cast<unsigned>(batch - b0 < 65535 ? batch - b0 : 65535);
    const int want = num_sms() * 8 / static_cast<int>(nb) + 1;
    const dim3 grid(static_cast<unsigned>(dm < want ? dm : want), nb);
    auto sp = static_cast<const char*>(src) + b0 * sm * sn * (src_fp32 ? 4 : 2);
    auto dp = static_cast<char*>(dst) + b0 * dm * dn * (dst_fp32 ? 4 : 2);
    const float* np = norm ? norm + b0 : nullptr;
    using bf = __nv_bfloat16;
    if (src_fp32) repad_kernel<float, bf><<<grid, 256, 0, stream>>>((const float*)sp, (bf*)dp, sm, sn, dm, dn, np, eps);
    else if (dst_fp32) repad_kernel<bf, float><<<grid, 256, 0, stream>>>((const bf*)sp, (float*)dp, sm, sn, dm, dn, np, eps);
    else repad_kernel<bf, bf><<<grid, 256, 0, stream>>>((const bf*)sp, (bf*)dp, sm, sn, dm, dn, np, eps);
  }
}

// ------------------------------------------------------------------------------------------------
constexpr int kAdamUnit = 4096;  // elements per work unit

// The three parameter-update conventions (0: HiMuon's fallback, 1: Muon / MuonFsdp, 2: plain AdamW, decay after the step).
__device__ __forceinline__ float adam_apply(int mode, float pi, float mi, float vi, float lr, float wd, float eps,
                                            float bc1, float bc2) {
  if (mode == 0) {
    const float u = (mi / bc1) / (sqrtf(vi) / sqrtf(bc2) + eps);
    if (wd > 0.f) pi *= 1.f - lr * wd;
    pi -= lr * u;
  } else if (mode == 1) {
    const float u = mi / (eps + sqrtf(vi));
    const float scale = bc1 / sqrtf(bc2);
    if (wd > 0.f) pi *= 1.f - lr * wd;
    pi -= (lr / scale) * u;
  } else {
    const float u = mi / (sqrtf(vi) + eps);
    pi -= lr * sqrtf(bc2) / bc1 * u;
    if (wd > 0.f) pi -= lr * wd * pi;
  }
  return pi;
}

template <typename P, typename S>
__global__ void __launch_bounds__(256)
adamw_multi_kernel(const AdamEntry* __restrict__ entries, int n_entries, long long total_units,
                   const float* __restrict__ hyper, const float* __restrict__ step_ptr, int mode) {
  const float t = *step_ptr + 1.f;  // this step's index; the counter itself is advanced by adamw_step_advance
  for (long long unit = blockIdx.x; unit < total_units; unit += gridDim.x) {
    int lo = 0, hi = n_entries - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (entries[mid].unit_begin <= unit) lo = mid; else hi = mid - 1;
    }
    const AdamEntry e = entries[lo];
    const float* h = hyper + 8 * e.group;
    const float lr = h[0], wd = h[1], b1 = h[2], b2 = h[3], eps = h[4];
    const float bc1 = 1.f - powf(b1, t), bc2 = 1.f - powf(b2, t);
    const long long base = (unit - e.unit_begin) * kAdamUnit;
    const long long end = min(e.numel, base + kAdamUnit);
    P* p = reinterpret_cast<P*>(e.param);
    const S* g = reinterpret_cast<const S*>(e.grad);
    S* m = reinterpret_cast<S*>(e.m);
    S* v = reinterpret_cast<S*>(e.v);
    long long scalar_from = base;
    if (sizeof(P) == sizeof(S) &&
        ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
          reinterpret_cast<uintptr_t>(v)) & 15) == 0) {
      // one storage type: 16 bytes per thread and access (units start on multiples of 4096 elements)
      constexpr int VN = Vec16<S>::N;
      const long long nvec = (end - base) / VN;
      for (long long k = threadIdx.x; k < nvec; k += blockDim.x) {
        const long long i = base + k * VN;
        float gf[VN], mf[VN], vf[VN], pf[VN];
        Vec16<S>::unpack(*reinterpret_cast<const uint4*>(g + i), gf);
        Vec16<S>::unpack(*reinterpret_cast<const uint4*>(m + i), mf);
        Vec16<S>::unpack(*reinterpret_cast<const uint4*>(v + i), vf);
        Vec16<S>::unpack(*reinterpret_cast<const uint4*>(reinterpret_cast<const S*>(e.param) + i), pf);
#pragma unroll
        for (int q = 0; q < VN; ++q) {
          mf[q] = mf[q] + (gf[q] - mf[q]) * (1.f - b1);
          vf[q] = vf[q] + (gf[q] * gf[q] - vf[q]) * (1.f - b2);
          // (one at a time here: pairs gain 1-3 % on an embedding alone, 866 -> 843 us for 389 M elements, and lose 2 % on 60 matrices
          // of 1024 x 1024, 156 -> 160)
          if (sizeof(S) == 2) { mf[q] = round_bf16(mf[q]); vf[q] = round_bf16(vf[q]); }
          pf[q] = adam_apply(mode, pf[q], mf[q], vf[q], lr, wd, eps, bc1, bc2);
        }
        *reinterpret_cast<uint4*>(m + i) = Vec16<S>::pack(mf);
        *reinterpret_cast<uint4*>(v + i) = Vec16<S>::pack(vf);
        *reinterpret_cast<uint4*>(reinterpret_cast<S*>(e.param) + i) = Vec16<S>::pack(pf);
      }
      scalar_from = base + nvec * VN;
    }
    for (long long i = scalar_from + threadIdx.x; i < end; i += blockDim.x) {
      const float gi = ldf(g + i);
      float mi = ldf(m + i), vi = ldf(v + i);
      mi = mi + (gi - mi) * (1.f - b1);
      vi = vi + (gi * gi - vi) * (1.f - b2);
      if (sizeof(S) == 2) { mi = round_bf16(mi); vi = round_bf16(vi); }
      stf(m + i, mi);
      stf(v + i, vi);
      stf(p + i, adam_apply(mode, ldf(p + i), mi, vi, lr, wd, eps, bc1, bc2));
    }
  }
}

__global__ void adamw_step_advance_kernel(float* step) { *step += 1.f; }

void adamw_step_advance(float* step, cudaStream_t stream) { adamw_step_advance_kernel<<<1, 1, 0, stream>>>(step); }

void adamw_multi(const AdamEntry* entries, int n_entries, long long total_units, const float* hyper, float* step,
                 int mode, int param_fp32, int state_fp32, cudaStream_t stream) {
  if (total_units <= 0) return;
  const long long cap = static_cast<long long>(num_sms()) * 16;
  const int grid = static_cast<int>(total_units < cap ? total_units : cap);
  if (param_fp32 && state_fp32)
    adamw_multi_kernel<float, float><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, hyper, step, mode);
  else if (!param_fp32 && !state_fp32)
    adamw_multi_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, hyper, step, mode);
  else if (!param_fp32 && state_fp32)
    adamw_multi_kernel<__nv_bfloat16, float><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, hyper, step, mode);
  else
    adamw_multi_kernel<float, __nv_bfloat16><<<grid, 256, 0, stream>>>(entries, n_entries, total_units, hyper, step, mode);
}

}  // namespace himuon
