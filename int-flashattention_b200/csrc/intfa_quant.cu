// Fused quantisation prologue (HBM-bound): fp16 -> int8 with absmax scales.
//
// Bit-exact restatement of the reference quantisers, whose arithmetic follows the fp16
// input dtype (benchmark.py:96-107):
//   amax  = max |x|                       (exact in fp16)
//   scale = fp16( fp32(amax) / 127 )      (IEEE fp32 division, then round-to-nearest fp16)
//   q     = int8( rint( fp16( fp32(x) / fp32(scale) ) ) )   (rint = half-to-even, as torch.round)
// The per-element division is one product with the reciprocal of the row's or channel's scale, which gives the same
// bytes (see quant_pair).
// Scales are written as fp32 holding the fp16-representable value.  amax == 0 gives
// scale 0 and q 0 (the reference computes 0/0 there).
//
// Each row of D fp16 is read by D/8 lanes with one 128-bit load per lane; the row/column
// maxima are reduced with warp shuffles.  Per-token: one pass.  V (per-channel or
// per-(batch,head)): one pass where a cluster of CTAs holds a slab in registers (v_slab), else a column-absmax pass, then the
// quantising pass.  The fused entry (quant_qkv) runs small calls as ONE launch; larger ones take the Q and the K rows first and V
// second, where V has two passes the column-absmax one with the first launch (partial maxima per chunk, plain stores).  The stand-alone V entries: partial maxima as well (intfa_quant_v_partial, which the Python
// operators call), or atomicMax into a small array (intfa_quant_v, intfa_v_colmax, intfa_quant_v_static).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "intfa_internal.h"
#include "intfa_ptx.cuh"

namespace intfa {

__device__ __forceinline__ float scale_from_amax(float amax) {
  return __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
}
// fp16(RN32(x / s)) without a division per element: with r = RN32(1/s), fp16(RN32(x*r)) is the same number.  x and s are
// fp16 values, so x/s = (X/S) * 2^k with X, S < 2^11.  Where rounding to fp16 can turn -- at a midpoint m of two fp16
// numbers, whose significand M is odd and below 2^12 -- x/s is never equal to m (M would have to divide X) and at least
// 1/(M*S) > 1.0007 * 2^-23 away from it, relative to m; RN32(x*r) is at most 2^-23 + 2^-48 away from x/s, hence on the same
// side of m, and so is RN32(x/s).  (Below the fp16 normal range the result is rounded to 0 in any case.)
// Then rint() done IN fp16 by adding 1536 = 1.5*2^10 (the sum has an ulp of 1, so its round-to-nearest-even is rint, and
// its bit pattern is 0x6600 + n: the two's-complement integer is the low byte).  Everything runs two elements per
// instruction (packed fp32, fp16x2): these kernels are as much bound by instruction issue as by HBM.
// A zero scale (an all-zero row or channel; the reference computes 0/0 there) is given the reciprocal 0, which makes
// every quotient 0.
__device__ __forceinline__ float safe_rcp(float s) { return s == 0.f ? 0.f : __frcp_rn(s); }
// two fp16 inputs -> two int8 in bytes 0 and 2 of the result; r: the reciprocals of their scales
__device__ __forceinline__ uint32_t quant_pair(__half2 x, uint64_t r) {
  const float2 f = __half22float2(x);
  float qa, qb;
  f2_unpack(f2_mul(f2_pack(f.x, f.y), r), qa, qb);
  const __half2 u = __hadd2(__floats2half2_rn(qa, qb), __half2(__ushort_as_half(0x6600), __ushort_as_half(0x6600)));
  return *reinterpret_cast<const uint32_t*>(&u);
}
// the absmax of the even and of the odd elements
__device__ __forceinline__ __half2 amax8(const uint4& v) {
  const __half2* h = reinterpret_cast<const __half2*>(&v);
  return __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
}
__device__ __forceinline__ __half2 shfl_xor_h2(__half2 x, int o) {
  const uint32_t y = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&x), o);
  return *reinterpret_cast<const __half2*>(&y);
}
// k[i]: the reciprocals of the scales of elements 2i, 2i+1 of the 8
__device__ __forceinline__ uint2 quant8(const uint4& v, const uint64_t (&k)[4]) {
  const __half2* h2 = reinterpret_cast<const __half2*>(&v);
  const uint32_t u0 = quant_pair(h2[0], k[0]), u1 = quant_pair(h2[1], k[1]);
  const uint32_t u2 = quant_pair(h2[2], k[2]), u3 = quant_pair(h2[3], k[3]);
  return make_uint2(__byte_perm(u0, u1, 0x6420), __byte_perm(u2, u3, 0x6420));
}

// L2 residency hints.  The first launch of the fused prologue reads V for its column maxima and the second reads it
// again to quantise it: V is loaded "evict last" there and everything that is touched once (Q, K, every int8 store)
// "evict first", and the second launch walks the (batch, head) slabs in the opposite order, so that the slabs read
// last -- as much of V as the L2 holds -- are served from L2 instead of HBM.
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ld_hint(const void* p, uint64_t policy) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(policy));
  return v;
}
__device__ __forceinline__ void st_hint(void* p, uint2 v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.v2.u32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(v.x), "r"(v.y), "l"(policy) : "memory");
}

constexpr int kQuantUnroll = 4;    // independent 128-bit loads in flight per lane

// Scales of the four rows that the LPR lanes of a row group hold 8 elements of each (m: absmax of each lane's part): s[u] and
// its reciprocal k[u].  The division, the rounding and the reciprocal cost more instructions than the quantisation of a
// load itself, so no lane does them for all four rows: the rows' maxima are reduced as two fp16 pairs, the first step
// of the butterfly leaves each lane one pair, and lane `sub` ends with the scale of row 2*(sub & 1) + (sub >> 1 & 1)
// (returned), whose reciprocal the others fetch from it.
template <int LPR>
__device__ __forceinline__ float row_scales(const __half2 (&m)[4], int lane, float (&k)[4]) {
  static_assert(kQuantUnroll == 4 && LPR >= 4, "one lane per row");
  const __half2 p01 = __hmax2(__lows2half2(m[0], m[1]), __highs2half2(m[0], m[1]));
  const __half2 p23 = __hmax2(__lows2half2(m[2], m[3]), __highs2half2(m[2], m[3]));
  const bool odd = lane & 1;
  __half2 p = __hmax2(odd ? p23 : p01, shfl_xor_h2(odd ? p01 : p23, 1));
#pragma unroll
  for (int o = 2; o < LPR; o <<= 1) p = __hmax2(p, shfl_xor_h2(p, o));
  const float s = scale_from_amax((lane & 2) ? __high2float(p) : __low2float(p));
  const float r = safe_rcp(s);
#pragma unroll
  for (int u = 0; u < 4; ++u) k[u] = __shfl_sync(0xffffffffu, r, (u >> 1) | ((u & 1) << 1), LPR);
  return s;
}

// Per-token quantisation of the rows that CTA `cta` of `ncta` owns (a grid-stride loop over groups of rows).
template <int D, bool CONTIG>
__device__ __forceinline__ void pertoken_rows(const __half* __restrict__ x, long long sB, long long sH, long long sN,
                                              int8_t* __restrict__ x8, float* __restrict__ scale, int H, int N,
                                              long long total_rows, int cta, int ncta) {
  constexpr int LPR = D / 8;         // lanes per row
  constexpr int RPW = 32 / LPR;      // rows per warp and load
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPR;
  const long long warp_g = (long long)cta * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = (long long)ncta * (blockDim.x >> 5);
  const uint64_t once = l2_policy_evict_first();
  for (long long row0 = warp_g * (RPW * kQuantUnroll); row0 < total_rows; row0 += nwarps * (RPW * kQuantUnroll)) {
    uint4 v[kQuantUnroll];
    long long rows[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const long long row = row0 + u * RPW + lane / LPR;
      rows[u] = row;
      v[u] = make_uint4(0, 0, 0, 0);
      if (row < total_rows) {
        if (CONTIG) {
          v[u] = ld_hint(x + row * D + sub * 8, once);      // [B,H,N,D] contiguous: the row index is the address
        } else {
          // total_rows < 2^31 (checked by the host): 32-bit divisions
          const unsigned int r32 = (unsigned int)row;
          const unsigned int bh = r32 / (unsigned int)N;
          const unsigned int n = r32 - bh * (unsigned int)N;
          const unsigned int b = bh / (unsigned int)H, h = bh - b * (unsigned int)H;
          v[u] = ld_hint(x + (long long)b * sB + (long long)h * sH + (long long)n * sN + sub * 8, once);
        }
      }
    }
    float k[kQuantUnroll];
    if constexpr (LPR >= 4) {
      const __half2 m[4] = {amax8(v[0]), amax8(v[1]), amax8(v[2]), amax8(v[3])};
      const float s = row_scales<LPR>(m, lane, k);
      const long long row = row0 + (2 * (sub & 1) + (sub >> 1 & 1)) * RPW + lane / LPR;
      if (sub < 4 && row < total_rows) scale[row] = s;
    } else {
#pragma unroll
      for (int u = 0; u < kQuantUnroll; ++u) {
        __half2 m = amax8(v[u]);
        m = __hmax2(m, shfl_xor_h2(m, 1));
        const float s = scale_from_amax(fmaxf(__low2float(m), __high2float(m)));
        k[u] = safe_rcp(s);
        if (sub == 0 && rows[u] < total_rows) scale[rows[u]] = s;
      }
    }
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      if (rows[u] < total_rows) {
        const uint64_t k1 = f2_pack(k[u], k[u]);
        const uint64_t kk[4] = {k1, k1, k1, k1};
        st_hint(x8 + rows[u] * D + sub * 8, quant8(v[u], kk), once);
      }
    }
  }
}

template <int D, bool CONTIG>
__global__ void __launch_bounds__(256) quant_pertoken_kernel(const __half* __restrict__ x, long long sB, long long sH,
                                                             long long sN, int8_t* __restrict__ x8,
                                                             float* __restrict__ scale, int H, int N,
                                                             long long total_rows) {
  pdl_wait();
  pdl_launch();
  pertoken_rows<D, CONTIG>(x, sB, sH, sN, x8, scale, H, N, total_rows, blockIdx.x, gridDim.x);
}

// Column absmax of chunk `chunk` (rows_per_cta rows) of the (batch, head) slab `bh`.  ATOMIC: atomicMax on the bit
// patterns of non-negative floats into colmax[bh*D + ch] (the caller has zeroed it); otherwise a plain store into
// row `chunk` of a [chunks][B*H][D] array of partial maxima (nothing to clear, nothing to order).
template <int D, bool ATOMIC>
__device__ __forceinline__ void colmax_chunk(const __half* __restrict__ x, long long sB, long long sH, long long sN,
                                             unsigned int* __restrict__ colmax, int H, int N, int rows_per_cta,
                                             int chunk, int bh, int BH) {
  constexpr int LPR = D / 8;
  constexpr int RPW = 32 / LPR;
  __shared__ float red[8][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane % LPR;
  const int b = bh / H, h = bh - b * H;
  const __half* base = x + b * sB + h * sH + sub * 8;
  const int r_begin = chunk * rows_per_cta;
  const int r_end = min(N, r_begin + rows_per_cta);
  const uint64_t keep = l2_policy_evict_last();
  __half2 m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = __float2half2_rn(0.f);
  for (int r0 = r_begin + warp * RPW + lane / LPR; r0 < r_end; r0 += nw * RPW * kQuantUnroll) {
    uint4 v[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const int r = r0 + u * nw * RPW;
      v[u] = r < r_end ? ld_hint(base + r * sN, keep) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const __half2* hv = reinterpret_cast<const __half2*>(&v[u]);
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], __habs2(hv[i]));
    }
  }
  float f[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __low2float(m[i]);
    f[2 * i + 1] = __high2float(m[i]);
  }
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = fmaxf(f[i], __shfl_xor_sync(0xffffffffu, f[i], o));
  if (lane < LPR)
#pragma unroll
    for (int i = 0; i < 8; ++i) red[warp][sub * 8 + i] = f[i];
  __syncthreads();
  for (int ch = threadIdx.x; ch < D; ch += blockDim.x) {
    float a = 0.f;
    for (int w = 0; w < nw; ++w) a = fmaxf(a, red[w][ch]);
    if (ATOMIC) atomicMax(colmax + (long long)bh * D + ch, __float_as_uint(a));
    else colmax[((long long)chunk * BH + bh) * D + ch] = __float_as_uint(a);
  }
}

template <int D, bool ATOMIC>
__global__ void __launch_bounds__(256) v_colmax_kernel(const __half* __restrict__ x, long long sB, long long sH,
                                                       long long sN, unsigned int* __restrict__ colmax, int H, int N,
                                                       int rows_per_cta) {
  pdl_wait();
  pdl_launch();
  colmax_chunk<D, ATOMIC>(x, sB, sH, sN, colmax, H, N, rows_per_cta, blockIdx.x, blockIdx.y, gridDim.y);
}

// V of one (batch, head) in one pass: the CTAs of a cluster take its rows in equal chunks, keep them in registers (U loads a
// thread), exchange their channels' maxima through distributed shared memory and quantise what they hold.  V is read once,
// there are no partial maxima in memory, and one launch does it.  Bound by memory; `early` (V is older than the kernel before
// this one on the stream): loads before pdl_wait.
template <int D, int U>
__device__ __forceinline__ void v_slab(const __half* __restrict__ x, long long sB, long long sH, long long sN, int8_t* __restrict__ x8,
                                       float* __restrict__ scale, int per_channel, int H, int N, int rows_per_cta, int bh, int early) {
  constexpr int LPR = D / 8;
  constexpr int RPC = 256 / LPR;         // rows that the CTA loads at a time
  __shared__ float red[8][D];
  __shared__ float s_max[D];             // the chunk's maxima, read by the other CTAs of the cluster
  __shared__ float s_scale[D];
  __shared__ float s_all[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = threadIdx.x % LPR;
  const int b = bh / H, h = bh - b * H;
  const uint32_t rank = cluster_rank(), ncta = cluster_size();
  const int r0 = (int)rank * rows_per_cta + threadIdx.x / LPR;
  const int r_end = min(N, ((int)rank + 1) * rows_per_cta);
  const __half* base = x + b * sB + h * sH + sub * 8;
  const uint64_t once = l2_policy_evict_first();
  if (!early) {
    pdl_wait();
    pdl_launch();
  }
  uint4 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int r = r0 + u * RPC;
    v[u] = r < r_end ? ld_hint(base + r * sN, once) : make_uint4(0, 0, 0, 0);
  }
  if (early) {
    pdl_wait();
    pdl_launch();
  }
  __half2 m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = __float2half2_rn(0.f);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const __half2* hv = reinterpret_cast<const __half2*>(&v[u]);
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], __habs2(hv[i]));
  }
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = __hmax2(m[i], shfl_xor_h2(m[i], o));
  if (lane < LPR) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      red[warp][sub * 8 + 2 * i] = __low2float(m[i]);
      red[warp][sub * 8 + 2 * i + 1] = __high2float(m[i]);
    }
  }
  __syncthreads();
  const int ch = threadIdx.x;
  if (ch < D) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) a = fmaxf(a, red[w][ch]);
    s_max[ch] = a;
  }
  cluster_arrive();
  cluster_wait();
  float a = 0.f;
  if (ch < D)
    for (uint32_t c = 0; c < ncta; ++c) a = fmaxf(a, ld_peer(s_max + ch, c));
  cluster_arrive();                      // (the CTA must not end before its peers have read its maxima: waited for below)
  if (!per_channel) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    if (lane == 0) s_all[warp] = a;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) a = fmaxf(a, s_all[w]);
  }
  if (ch < D) {
    const float s = scale_from_amax(a);
    s_scale[ch] = safe_rcp(s);
    if (rank == 0) {
      if (per_channel) scale[(long long)bh * D + ch] = s;
      else if (ch == 0) scale[bh] = s;
    }
  }
  __syncthreads();
  uint64_t k[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) k[i] = f2_pack(s_scale[sub * 8 + 2 * i], s_scale[sub * 8 + 2 * i + 1]);
  int8_t* o = x8 + (long long)bh * N * D + sub * 8;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int r = r0 + u * RPC;
    if (r < r_end) st_hint(o + (long long)r * D, quant8(v[u], k), once);
  }
  cluster_wait();
}
// CTAs of a cluster at most (16 hold longer slabs, but wait for one another longer: 128 slabs of 2048 x 128 24.9 -> 27.9 us, 256 of
// 2048 x 64 22.4 -> 37.4)
constexpr int kSlabCluster = 8;
__host__ __device__ constexpr int slab_ctas_per_sm(int U) { return U == 16 ? 3 : U == 4 ? 6 : 4; }
template <int D, int U>
__global__ void __launch_bounds__(256, slab_ctas_per_sm(U)) v_slab_kernel(const __half* __restrict__ x, long long sB, long long sH, long long sN,
                                                     int8_t* __restrict__ x8, float* __restrict__ scale, int per_channel, int H, int N,
                                                     int rows_per_cta, int early) {
  v_slab<D, U>(x, sB, sH, sN, x8, scale, per_channel, H, N, rows_per_cta, blockIdx.x / cluster_size(), early);
}

// The first launch of the fused prologue: one grid over three jobs -- CTAs [0, gq) quantise the rows of Q,
// [gq, gq+gk) those of K (both per token, contiguous tensors), the rest take one (chunk, batch*head) piece of V each and
// store its column absmax as a partial result.  Nothing is shared between the jobs, so no ordering is needed.
struct QkvJob {
  const __half* q; int8_t* q8; float* qs; long long q_rows; int gq;
  const __half* k; int8_t* k8; float* ks; long long k_rows; int gk;
  const __half* v; long long vB, vH, vN; unsigned int* partial; int Hkv, Nk, rows_per_cta, chunks, BHkv;
};
// Small calls: all of it in one launch.  CTAs [0, gv) are the clusters of v_slab, then as above; only where every CTA is resident at
// once, because v_slab's registers leave room for fewer of the others than their loads need to fill the memory.
struct SlabJob {
  int8_t* v8; float* vs; int per_channel, gv;
};
template <int D, int U>
__global__ void __launch_bounds__(256) quant_qkv_slab_kernel(const QkvJob j, const SlabJob s) {
  const int cta = (int)blockIdx.x - s.gv;
  if (cta < 0) {
    v_slab<D, U>(j.v, j.vB, j.vH, j.vN, s.v8, s.vs, s.per_channel, j.Hkv, j.Nk, j.rows_per_cta, blockIdx.x / cluster_size(), 0);
    return;
  }
  pdl_wait();
  pdl_launch();
  if (cta < j.gq) pertoken_rows<D, true>(j.q, 0, 0, 0, j.q8, j.qs, 1, 1, j.q_rows, cta, j.gq);
  else if (cta < j.gq + j.gk) pertoken_rows<D, true>(j.k, 0, 0, 0, j.k8, j.ks, 1, 1, j.k_rows, cta - j.gq, j.gk);
}

template <int D>
__global__ void __launch_bounds__(256) quant_qkv_kernel(const QkvJob j) {
  const int cta = blockIdx.x;
  pdl_wait();
  pdl_launch();
  if (cta < j.gq) {
    pertoken_rows<D, true>(j.q, 0, 0, 0, j.q8, j.qs, 1, 1, j.q_rows, cta, j.gq);
  } else if (cta < j.gq + j.gk) {
    pertoken_rows<D, true>(j.k, 0, 0, 0, j.k8, j.ks, 1, 1, j.k_rows, cta - j.gq, j.gk);
  } else {
    const int i = cta - j.gq - j.gk;
    colmax_chunk<D, false>(j.v, j.vB, j.vH, j.vN, j.partial, j.Hkv, j.Nk, j.rows_per_cta, i % j.chunks, i / j.chunks, j.BHkv);
  }
}

// The V quantising pass.  Its start is a serial chain (maxima -> scales -> reciprocals), so every thread takes part in
// reducing the partial maxima (one warp doing it cost 5 us of latency at 8 chunks), and `early` (the kernel before this one
// on the stream is the column-absmax pass, so V is older) has the first rows on their way meanwhile.
template <int D>
__global__ void __launch_bounds__(256) v_quant_kernel(const __half* __restrict__ x, long long sB, long long sH,
                                                      long long sN, const unsigned int* __restrict__ colmax,
                                                      int8_t* __restrict__ x8, float* __restrict__ scale,
                                                      int per_channel, int H, int N, int rows_per_cta, int nparts, int early) {
  constexpr int LPR = D / 8;
  constexpr int RPW = 32 / LPR;
  constexpr int PG = 256 / D;            // partial maxima in parallel
  __shared__ float s_max[PG][D];
  __shared__ float s_scale[D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane % LPR;
  const int bh = gridDim.y - 1 - blockIdx.y;     // last slab first: the column-absmax pass read it last
  const int b = bh / H, h = bh - b * H;
  const uint64_t once = l2_policy_evict_first();
  const __half* base = x + b * sB + h * sH + sub * 8;
  int8_t* obase = x8 + (long long)bh * N * D + sub * 8;
  const int r_begin = blockIdx.x * rows_per_cta;
  const int r_end = min(N, r_begin + rows_per_cta);
  int r0 = r_begin + warp * RPW + lane / LPR;
  uint4 v[kQuantUnroll];
  auto load = [&]() {
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const int r = r0 + u * nw * RPW;
      v[u] = r < r_end ? ld_hint(base + r * sN, once) : make_uint4(0, 0, 0, 0);
    }
  };
  if (early) load();
  pdl_wait();
  pdl_launch();
  if (!early) load();
  {
    // every channel's absmax (colmax is [nparts][B*H][D]: one row, or the partial maxima of the pass before)
    const int ch = threadIdx.x % D;
    float a = 0.f;
#pragma unroll 4
    for (int c = threadIdx.x / D; c < nparts; c += PG) a = fmaxf(a, __uint_as_float(__ldcg(colmax + ((long long)c * gridDim.y + bh) * D + ch)));
    s_max[threadIdx.x / D][ch] = a;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // ... and for the per-(batch,head) mode their maximum
    constexpr int CPL = (D + 31) / 32;     // channels per lane
    float a[CPL];
    float all = 0.f;
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
      a[i] = 0.f;
      if (lane + 32 * i < D)
#pragma unroll
        for (int c = 0; c < PG; ++c) a[i] = fmaxf(a[i], s_max[c][lane + 32 * i]);
      all = fmaxf(all, a[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all = fmaxf(all, __shfl_xor_sync(0xffffffffu, all, o));
#pragma unroll
    for (int i = 0; i < CPL; ++i)
      if (lane + 32 * i < D) s_scale[lane + 32 * i] = scale_from_amax(per_channel ? a[i] : all);
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    if (per_channel) {
      for (int ch = threadIdx.x; ch < D; ch += blockDim.x) scale[(long long)bh * D + ch] = s_scale[ch];
    } else if (threadIdx.x == 0) {
      scale[bh] = s_scale[0];
    }
  }
  uint64_t k[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) k[i] = f2_pack(safe_rcp(s_scale[sub * 8 + 2 * i]), safe_rcp(s_scale[sub * 8 + 2 * i + 1]));
  while (r0 < r_end) {
    uint4 w[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) w[u] = v[u];
    const int r1 = r0;
    r0 += nw * RPW * kQuantUnroll;
    if (r0 < r_end) load();
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const int r = r1 + u * nw * RPW;
      if (r < r_end) st_hint(obase + (long long)r * D, quant8(w[u], k), once);
    }
  }
}

__global__ void scales_f16_to_f32_kernel(const __half* __restrict__ src, float* __restrict__ dst, long long n) {
  pdl_wait();
  pdl_launch();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __half2float(src[i]);
}

// head dims of the reference's ops (flash_atten_full_int8.py:193): one instantiation each
#define INTFA_D_SWITCH(D, CALL)                 \
  switch (D) {                                  \
    case 16: { constexpr int DD = 16; CALL; } break;   \
    case 32: { constexpr int DD = 32; CALL; } break;   \
    case 64: { constexpr int DD = 64; CALL; } break;   \
    case 128: { constexpr int DD = 128; CALL; } break; \
    default: { constexpr int DD = 256; CALL; } break;  \
  }

int quant_pertoken(const void* x, const int64_t* st, void* x8, float* scale, int B, int H, int N, int D,
                   cudaStream_t stream) {
  const long long rows = (long long)B * H * N;
  const int rpw = 32 / (D / 8) * kQuantUnroll;
  if (rows >= (1LL << 31)) return set_error(INTFA_ERR_TOO_LARGE, "quant_pertoken: B*H*N must be below 2^31");
  // CTAs of 8 warps, one row group a warp: no loop, so a CTA's stores never hold back its own next loads (with a grid of 8
  // CTAs an SM in a loop 18.6 us at 262144 rows of 128, now 16.7; at 1048576 rows 80 -> 67 us)
  const int grid = (int)((rows + 8LL * rpw - 1) / (8LL * rpw));
  const bool contig = st[2] == D && st[1] == (int64_t)N * D && st[0] == (int64_t)H * N * D;
  int rc = INTFA_OK;
#define INTFA_QPT(CC) \
  rc = launch_kernel("quant_pertoken", quant_pertoken_kernel<DD, CC>, dim3(grid), 256, 0, stream, (const __half*)x, (long long)st[0], \
                     (long long)st[1], (long long)st[2], (int8_t*)x8, scale, H, N, rows)
  INTFA_D_SWITCH(D, if (contig) INTFA_QPT(true); else INTFA_QPT(false))
#undef INTFA_QPT
  return rc;
}

static int v_grid(int BH, int N, int sms, int* rows_per_cta) {
  // chunks per (batch, head): enough CTAs to fill the machine a few times over, at least 256 rows each
  int chunks = (sms * 8 + BH - 1) / BH;
  const int max_chunks = (N + 255) / 256;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  *rows_per_cta = (N + chunks - 1) / chunks;
  return chunks;
}

// V in one pass (v_slab): where the registers of a cluster hold a (batch, head), that is up to 262144/D rows.  rows_per_cta: equal
// chunks over as many CTAs as have 4 loads a thread to make; U of them rounded up to what is compiled.  (A CTA takes registers for U
// loads: rounded up to 16, 9 and 10 of them left three CTAs an SM where 10 leave four, 128 heads of 1152 x 128 18.9 -> 14.4 us, 222 of
// 2049 x 64 29.5 -> 22.8.)  Two passes before -> now, quantise V alone: 4 heads of 512 x 64 11.9 -> 7.9 us, 128 x 1024 x 64 10.6 -> 9.1,
// 256 x 2048 x 64 30.2 -> 22.4, 256 x 4096 x 64 58.9 -> 49.3, 2048 x 64 x 128 20.9 -> 10.1.
// Two passes stay where they are the faster ones.  Their second one reads V out of L2, so that is where there are several waves of
// clusters, which wait for one another within themselves (256 channels, `in_qkv` even at the best fill: there Q and K fill up the first
// pass), and more so where a part of the loads is padding; and single heads of the narrowest rows, for which 8 CTAs are few.  One pass:
//   512 heads of 256 x 256 29.8 -> 30.4 us; 222 of 513 x 128 15.7 -> 16.6, 512 of 1025 x 64 37.9 -> 38.9 (29.7 -> 38.9
//   with V in L2), 300 of 257 x 256 20.0 -> 23.6; 1 of 16384 x 16 4.3 -> 5.0
//   in_qkv: 512 x 256 x 256 55.4 -> 61.2; 512 x 512 x 128 56.1 -> 58.3; 300 x 768 x 128 49.6 -> 51.0; 300 x 1025 x 64 34.8 -> 37.9
// One side is left where the two differ: V alone, several waves, 50 MB and more.  Out of L2 one pass is faster (128 x 2048 x 128 28 ->
// 25 us, 512 x 512 x 128 29.8 -> 27.3), with V in L2 slower (23.6 -> 24.9, 23.3 -> 26.3); the call cannot know, and after Q and K of the
// same size V is in L2 no more.
struct Slab {
  int cluster = 0, rows_per_cta = 0, U = 0;
};
static Slab slab_plan(int N, int D, long long heads, int sms, bool in_qkv) {
  Slab s;
  const int rpc = 256 / (D / 8);                        // rows of one load
  if (N > kSlabCluster * 16 * rpc) return s;
  int cluster = (N + 4 * rpc - 1) / (4 * rpc);
  if (cluster > kSlabCluster) cluster = kSlabCluster;
  s.rows_per_cta = (N + cluster - 1) / cluster;
  const int loads = (s.rows_per_cta + rpc - 1) / rpc;
  s.U = loads <= 4 ? 4 : loads <= 8 ? 8 : loads <= 10 ? 10 : 16;
  const double waves = (double)heads * cluster / ((double)sms * slab_ctas_per_sm(s.U));
  const bool padded = loads == 5;
  const bool two = in_qkv ? (D == 256 && waves > 1.75) || (D == 128 && ((s.U == 4 && waves > 1.6) || (s.U == 8 && loads < 8 && waves > 3.5))) ||
                                (padded && waves > 2.5)
                          : (D == 256 && s.U == 4 && cluster > 4 && waves > 2.8) || (padded && waves > (D >= 128 ? 2.5 : 3.5)) ||
                                (D <= 32 && loads > 13 && heads <= 4);
  if (!two) s.cluster = cluster;
  return s;
}
#define INTFA_U_SWITCH(U, CALL)                       \
  switch (U) {                                        \
    case 4: { constexpr int UU = 4; CALL; } break;    \
    case 8: { constexpr int UU = 8; CALL; } break;    \
    case 10: { constexpr int UU = 10; CALL; } break;  \
    default: { constexpr int UU = 16; CALL; } break;  \
  }
static int v_slab_launch(const Slab& sl, const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
                         bool early, cudaStream_t stream) {
  const int pc = mode == INTFA_VSCALE_PER_CHANNEL;
  int rc = INTFA_OK;
  INTFA_D_SWITCH(D, INTFA_U_SWITCH(sl.U, (rc = launch_clusters("v_slab", v_slab_kernel<DD, UU>, dim3(sl.cluster * B * H), sl.cluster, 256, 0, stream,
                 (const __half*)v, (long long)st[0], (long long)st[1], (long long)st[2], (int8_t*)v8, scale, pc, H, N, sl.rows_per_cta, early ? 1 : 0))))
  return rc;
}

int v_colmax(const void* v, const int64_t* st, void* colmax, int B, int H, int N, int D, cudaStream_t stream) {
  const int sms = sm_count_cached();
  if (sms <= 0) return set_error(INTFA_ERR_CUDA, "cannot query SM count");
  int rows_per_cta;
  dim3 grid(v_grid(B * H, N, sms, &rows_per_cta), B * H);
  int rc = INTFA_OK;
  INTFA_D_SWITCH(D, (rc = launch_kernel("v_colmax", v_colmax_kernel<DD, true>, grid, 256, 0, stream, (const __half*)v, (long long)st[0],
                                        (long long)st[1], (long long)st[2], (unsigned int*)colmax, H, N, rows_per_cta)))
  return rc;
}

static int v_quant_launch(const void* v, const int64_t* st, const void* colmax, int nparts, bool early, void* v8, float* scale, int mode,
                          int B, int H, int N, int D, cudaStream_t stream) {
  const int sms = sm_count_cached();
  if (sms <= 0) return set_error(INTFA_ERR_CUDA, "cannot query SM count");
  int rows_per_cta;
  dim3 grid(v_grid(B * H, N, sms, &rows_per_cta), B * H);
  const int pc = mode == INTFA_VSCALE_PER_CHANNEL;
  int rc = INTFA_OK;
  INTFA_D_SWITCH(D, (rc = launch_kernel("v_quant", v_quant_kernel<DD>, grid, 256, 0, stream, (const __half*)v, (long long)st[0], (long long)st[1],
                                        (long long)st[2], (const unsigned int*)colmax, (int8_t*)v8, scale, pc, H, N, rows_per_cta, nparts, early ? 1 : 0)))
  return rc;
}

int v_quant_from_colmax(const void* v, const int64_t* st, const void* colmax, void* v8, float* scale, int mode, int B,
                        int H, int N, int D, cudaStream_t stream) {
  return v_quant_launch(v, st, colmax, 1, false, v8, scale, mode, B, H, N, D, stream);
}

// ---------------------------------------------------------------------------------------------
// fused prologue: Q, K (per token) and V (per channel / per batch-head) in one or two launches, no memset
// ---------------------------------------------------------------------------------------------
size_t quant_qkv_workspace_bytes(int B, int Hkv, int Nk, int D) {
  const int sms = sm_count_cached();
  int rows_per_cta;
  const int chunks = v_grid(B * Hkv, Nk, sms > 0 ? sms : 148, &rows_per_cta);
  return (size_t)chunks * B * Hkv * D * sizeof(unsigned int);
}

int quant_qkv(const void* q, const void* k, const void* v, const int64_t* v_st, void* q8, void* k8, void* v8, float* qs,
              float* ks, float* vs, int mode, int B, int H, int Hkv, int Nq, int Nk, int D, void* workspace,
              cudaStream_t stream) {
  const int sms = sm_count_cached();
  if (sms <= 0) return set_error(INTFA_ERR_CUDA, "cannot query SM count");
  QkvJob j;
  j.q = (const __half*)q; j.q8 = (int8_t*)q8; j.qs = qs; j.q_rows = (long long)B * H * Nq;
  j.k = (const __half*)k; j.k8 = (int8_t*)k8; j.ks = ks; j.k_rows = (long long)B * Hkv * Nk;
  if (j.q_rows >= (1LL << 31) || j.k_rows >= (1LL << 31)) return set_error(INTFA_ERR_TOO_LARGE, "quant_qkv: B*H*N must be below 2^31");
  const int rpw = 32 / (D / 8) * kQuantUnroll;
  auto ctas = [&](long long rows) {
    const long long want = (rows + 8LL * rpw - 1) / (8LL * rpw);
    const long long cap = (long long)sms * 8;
    return (int)(want < cap ? (want < 1 ? 1 : want) : cap);
  };
  j.gq = ctas(j.q_rows);
  j.gk = ctas(j.k_rows);
  j.v = (const __half*)v; j.partial = (unsigned int*)workspace; j.Hkv = Hkv; j.Nk = Nk; j.BHkv = B * Hkv;
  j.chunks = 0; j.rows_per_cta = 0; j.vB = j.vH = j.vN = 0;
  int gv = 0;
  if (v) {
    const Slab sl = slab_plan(Nk, D, (long long)B * Hkv, sms, true);
    if (sl.cluster > 0) {
      int rc = INTFA_OK;
      const int slabs = sl.cluster * B * Hkv;
      if (slabs + j.gq + j.gk <= 2 * sms) {
        j.vB = v_st[0]; j.vH = v_st[1]; j.vN = v_st[2];
        j.rows_per_cta = sl.rows_per_cta;
        const SlabJob s = {(int8_t*)v8, vs, mode == INTFA_VSCALE_PER_CHANNEL, slabs};
        const int grid = (slabs + j.gq + j.gk + sl.cluster - 1) / sl.cluster * sl.cluster;
        INTFA_D_SWITCH(D, INTFA_U_SWITCH(sl.U, (rc = launch_clusters("quant_qkv", quant_qkv_slab_kernel<DD, UU>, dim3(grid), sl.cluster, 256, 0, stream, j, s))))
        return rc;
      }
      INTFA_D_SWITCH(D, (rc = launch_kernel("quant_qkv", quant_qkv_kernel<DD>, dim3(j.gq + j.gk), 256, 0, stream, j)))
      return rc ? rc : v_slab_launch(sl, v, v_st, v8, vs, mode, B, Hkv, Nk, D, true, stream);
    }
    j.vB = v_st[0]; j.vH = v_st[1]; j.vN = v_st[2];
    j.chunks = v_grid(B * Hkv, Nk, sms, &j.rows_per_cta);
    gv = j.chunks * B * Hkv;
  }
  const int grid = j.gq + j.gk + gv;
  int rc = INTFA_OK;
  INTFA_D_SWITCH(D, (rc = launch_kernel("quant_qkv", quant_qkv_kernel<DD>, dim3(grid), 256, 0, stream, j)))
  if (rc || !v) return rc;
  return v_quant_launch(v, v_st, workspace, j.chunks, true, v8, vs, mode, B, Hkv, Nk, D, stream);
}

int quant_v_partial(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D, void* workspace,
                    cudaStream_t stream) {
  const int sms = sm_count_cached();
  if (sms <= 0) return set_error(INTFA_ERR_CUDA, "cannot query SM count");
  const Slab sl = slab_plan(N, D, (long long)B * H, sms, false);
  if (sl.cluster > 0) return v_slab_launch(sl, v, st, v8, scale, mode, B, H, N, D, false, stream);
  int rows_per_cta;
  const int chunks = v_grid(B * H, N, sms, &rows_per_cta);
  dim3 grid(chunks, B * H);
  int rc = INTFA_OK;
  INTFA_D_SWITCH(D, (rc = launch_kernel("v_colmax", v_colmax_kernel<DD, false>, grid, 256, 0, stream, (const __half*)v, (long long)st[0],
                                        (long long)st[1], (long long)st[2], (unsigned int*)workspace, H, N, rows_per_cta)))
  if (rc) return rc;
  return v_quant_launch(v, st, workspace, chunks, true, v8, scale, mode, B, H, N, D, stream);
}

int quant_v(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
            void* workspace, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(workspace, 0, (size_t)B * H * D * sizeof(unsigned int), stream);
  if (e != cudaSuccess) return set_error(INTFA_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  int rc = v_colmax(v, st, workspace, B, H, N, D, stream);
  if (rc) return rc;
  return v_quant_from_colmax(v, st, workspace, v8, scale, mode, B, H, N, D, stream);
}

// ---------------------------------------------------------------------------------------------
// V quantisation for callers that must not allocate (intfa_quant_v_static)
// ---------------------------------------------------------------------------------------------
// Column-absmax scratch that lives in the library image instead of in a caller-provided buffer.
// Every GPU that loads the library keeps these kStaticColmaxWords*4 bytes until the process exits.
// In host code `g_static_colmax` is only a handle for the symbol, not a device address, so the
// address is looked up once per device with cudaGetSymbolAddress and that pointer is what the
// kernels are given.
__device__ __align__(256) static unsigned int g_static_colmax[kStaticColmaxWords];

static unsigned int* static_colmax_ptr(int* rc) {
  static std::atomic<unsigned int*> ptr[64];     // host threads may race to be first: each stores the same address
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    *rc = set_error(INTFA_ERR_CUDA, "cannot query the current device");
    return nullptr;
  }
  unsigned int* q = ptr[dev].load(std::memory_order_acquire);
  if (!q) {
    void* sym = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&sym, g_static_colmax);     // with device `dev` current
    if (e != cudaSuccess || sym == nullptr) {
      *rc = set_error(INTFA_ERR_CUDA, "cudaGetSymbolAddress(static colmax scratch): %s", cudaGetErrorString(e));
      return nullptr;
    }
    q = static_cast<unsigned int*>(sym);
    ptr[dev].store(q, std::memory_order_release);
  }
  *rc = INTFA_OK;
  return q;
}

int quant_v_static(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
                   cudaStream_t stream) {
  const long long words = (long long)B * H * D;
  if (words > kStaticColmaxWords)
    return set_error(INTFA_ERR_TOO_LARGE, "B*H*D = %lld exceeds the built-in scratch of %d words; use intfa_quant_v",
                     words, kStaticColmaxWords);
  int rc;
  unsigned int* scratch = static_colmax_ptr(&rc);
  if (!scratch) return rc;
  // the scratch keeps the previous call's maxima: clear the part this call uses
  cudaError_t e = cudaMemsetAsync(scratch, 0, (size_t)words * sizeof(unsigned int), stream);
  if (e != cudaSuccess) return set_error(INTFA_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  rc = v_colmax(v, st, scratch, B, H, N, D, stream);
  if (rc) return rc;
  return v_quant_from_colmax(v, st, scratch, v8, scale, mode, B, H, N, D, stream);
}

int scales_f16_to_f32(const void* src, float* dst, long long n, cudaStream_t stream) {
  if (n <= 0) return INTFA_OK;
  long long blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  return launch_kernel("scales_f16_to_f32", scales_f16_to_f32_kernel, dim3((int)blocks), 256, 0, stream, (const __half*)src, dst, n);
}

}  // namespace intfa
