// Attention of a few query rows against a long K/V cache (decode), and of short prompts: where 128-row tiles are mostly
// padding or too few to fill the GPU.  With one row a head this path is bound by reading K and V once.
//
// The 128-row kernel gives such a call one CTA per (batch, query head) whose 128 rows are nearly all padding: it re-reads
// K/V once per query head of a group and leaves most SMs without work (batch 1, 32/8 heads, 32768 keys, fp16 V: 369 us for
// 102 MB, 0.28 TB/s).  Here
//   * the query rows of all heads that share a K/V head are packed into one tile of 8 or 16 rows (R = (H/H_kv)*Nq rows,
//     so K and V are read once for all of them; more than 16 rows take several tiles, which share K/V through L2);
//   * the keys are split over as many CTAs as fill the GPU, and over the warps of a CTA;
//   * the products run on m16n8 warp-level MMAs straight from registers: a warp-level tile is 8 or 16 rows tall where the
//     smallest tcgen05 tile is 64, and operands go from global memory to the MMA without a shared-memory stage.  The
//     order of the k index is free in a product, so every lane loads 16 contiguous bytes of a row and calls them its
//     fragment; for P V the lane transposes the few keys it holds with byte permutes.
//
// full-int8: P is rounded to int8 against the RUNNING maximum of the row (keys taken G at a time, ascending), so the
// maxima must be known before P: `scores_kernel` computes s = (fp32(S32)*s_q)*s_k, keeps it (fp32, in the order in which
// the next kernel's lanes want it) and the maximum of each 64 keys; `pv_full_kernel` takes the prefix maximum at its
// first group, and from there on does what the one-pass kernel does: m' = max(m, groupmax*c), p = exp2(s*c - m'), P8, O_j
// (with s*c - m' as one fma on masked groups too, where that kernel rounds s*c first).  The final maximum is known too, so that every partial result is scaled to it at once
// (acc += exp2(m_j - m_final) * O_j) and the splits add up without weights.  Where the splits of a K/V head fit a cluster of CTAs one
// kernel may do both passes and the sum (`fused_full_kernel`; `fused_is_faster` says where).
// half-int8: P is fp16, whose rounding is relative: every warp keeps a running maximum of its own and the partial results
// are combined with their weights (`pv_half_kernel`: scores and P V in one pass over K and V).
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "intfa_internal.h"
#include "intfa_ptx.cuh"

namespace intfa {

namespace {

constexpr int kThreads = 128, kWarps = 4;
constexpr int kMaxCluster = 8;            // CTAs of a cluster that every GPU grants
constexpr int kMaxLocalUnits = 128;       // 64-key units per CTA of pv_full_kernel (their maxima sit in shared memory)
constexpr float kMagicF = 12582912.0f;    // 1.5*2^23: added to an int32 below 2^22 as a bit pattern, it reads as fp32 1.5*2^23 + value
constexpr int kMagicI = 0x4B400000;

struct DParams {
  const int8_t* q; const int8_t* k; const void* v; void* o;
  long long qB, qH, qN, kB, kH, kN, vB, vH, vN, oB, oH, oN;
  const void* qs; const void* ks; const void* vs;
  long long qsB, qsH, ksB, ksH, vsB, vsH, vsD;
  int scale_f16, o_bf16, causal;
  int H, Hkv, ratio, Nq, R, tiles;        // R = ratio*Nq rows per K/V head, in `tiles` tiles of RT rows
  int unit0;                              // the launch's first unit (its scratch begins with this one)
  int nvis;                               // keys that some row sees
  long long limit0;                       // causal: row n sees the keys <= limit0 + n
  float c;                                // sm_scale * log2(e)
  int G, groups, splits, per_split;       // per_split: groups (full) or 64-key units (half) per split
  float* lse;
  float* scores; float* gmax;             // [unit][key tile of 8][NT][32 lanes][2]; [unit][64-key units][RT]
  float* part; float* part_ml;            // [unit][splits][RT][D]; [unit][splits][RT][2]
};

__device__ __forceinline__ float scale_at(const void* s, long long i, int f16) {
  return f16 ? __half2float(static_cast<const __half*>(s)[i]) : static_cast<const float*>(s)[i];
}
// streaming 16-byte load
__device__ __forceinline__ uint4 ld16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld8(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float unmagic(int x) { return __int_as_float(x) - kMagicF; }
template <bool B>
struct Const {
  static constexpr bool value = B;
};
template <int N>
struct Int {
  static constexpr int value = N;
};
// one (batch, K/V head, row tile)
struct Unit {
  int id, b, hk, tile;                    // id: counted from the launch's first, as scratch is
};
__device__ __forceinline__ Unit unit_of(const DParams& p, int id) {
  Unit u;
  u.id = id;
  id += p.unit0;
  u.tile = id % p.tiles;
  const int bh = id / p.tiles;
  u.b = bh / p.Hkv;
  u.hk = bh - u.b * p.Hkv;
  return u;
}

// Q fragments of a lane (g = lane/4, t = lane%4), its row scales and the last key its rows see.  Rows past R: zero.
// Word i of chunk ch of row half hr sits at qf[ch][hr][i]: bytes ch*64 + t*16 + 4i of row g + 8*hr.
template <int D, int NT>
struct QRows {
  static constexpr int CH = D / 64;
  uint32_t w[CH][NT][4];
  float s[NT];
  int last[NT];
  __device__ __forceinline__ void load(const DParams& p, const Unit& u, int g, int t) {
#pragma unroll
    for (int hr = 0; hr < NT; ++hr) {
      const int r = u.tile * (8 * NT) + g + 8 * hr;
      s[hr] = 0.f;
      last[hr] = p.nvis - 1;
#pragma unroll
      for (int c = 0; c < CH; ++c) w[c][hr][0] = w[c][hr][1] = w[c][hr][2] = w[c][hr][3] = 0u;
      if (r < p.R) {
        const int h = u.hk * p.ratio + r / p.Nq, n = r % p.Nq;
        const int8_t* q = p.q + u.b * p.qB + h * p.qH + n * p.qN + t * 16;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const uint4 x = *reinterpret_cast<const uint4*>(q + c * 64);
          w[c][hr][0] = x.x; w[c][hr][1] = x.y; w[c][hr][2] = x.z; w[c][hr][3] = x.w;
        }
        s[hr] = scale_at(p.qs, u.b * p.qsB + h * p.qsH + n, p.scale_f16 & INTFA_SCALE_F16_Q);
        if (p.causal && p.limit0 + n < last[hr]) last[hr] = (int)(p.limit0 + n);
      }
    }
  }
};

// S^T for 8 keys: kw[c] = bytes c*64 + t*16 .. +15 of key g.  Result: rows g (d[0], d[1]) and g+8 (d[2], d[3]), keys 2t, 2t+1.
template <int D, int NT>
__device__ __forceinline__ void qk_tile(const QRows<D, NT>& q, const uint4 (&kw)[D / 64], int (&d)[4]) {
  d[0] = d[1] = d[2] = d[3] = kMagicI;
#pragma unroll
  for (int c = 0; c < D / 64; ++c) {
    const uint32_t z = 0u;
    mma_s8(d, q.w[c][0][0], NT > 1 ? q.w[c][NT - 1][0] : z, q.w[c][0][1], NT > 1 ? q.w[c][NT - 1][1] : z, kw[c].x, kw[c].y);
    mma_s8(d, q.w[c][0][2], NT > 1 ? q.w[c][NT - 1][2] : z, q.w[c][0][3], NT > 1 ? q.w[c][NT - 1][3] : z, kw[c].z, kw[c].w);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// full-int8, first pass: scores and maxima.  One warp takes 64 keys at a time, 32 in flight; CTAs fill one wave.
// Bound by reading K (67 MB at batch 16, 8 K/V heads, 4097 keys).
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NT>
__global__ void __launch_bounds__(kThreads) scores_kernel(const DParams p, int splits) {
  constexpr int RT = 8 * NT, CH = D / 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const Unit u = unit_of(p, blockIdx.x % (gridDim.x / splits));
  const int split = blockIdx.x / (gridDim.x / splits);
  pdl_wait();
  pdl_launch();
  QRows<D, NT> q;
  q.load(p, u, g, t);
  const int8_t* kb = p.k + u.b * p.kB + u.hk * p.kH + t * 16;
  const long long ksb = u.b * p.ksB + u.hk * p.ksH;
  const int kf16 = p.scale_f16 & INTFA_SCALE_F16_K;
  const int units64 = p.groups * (p.G / 64), ktiles = units64 * 8;
  float2* sc = reinterpret_cast<float2*>(p.scores) + (long long)u.id * ktiles * NT * 32 + lane;
  float* gm = p.gmax + (long long)u.id * units64 * RT;
  for (int un = split * kWarps + warp; un < units64; un += splits * kWarps) {
    float mx[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) mx[i] = -INFINITY;
#pragma unroll 1
    for (int kt = un * 8; kt < un * 8 + 8; kt += 4) {
      uint4 kw[4][CH];
      float k0[4], k1[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int8_t* row = kb + (long long)min((kt + i) * 8 + g, p.nvis - 1) * p.kN;
#pragma unroll
        for (int c = 0; c < CH; ++c) kw[i][c] = ld16(row + c * 64);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int key = (kt + i) * 8 + 2 * t;
        k0[i] = scale_at(p.ks, ksb + min(key, p.nvis - 1), kf16);
        k1[i] = scale_at(p.ks, ksb + min(key + 1, p.nvis - 1), kf16);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        int d[4];
        qk_tile<D, NT>(q, kw[i], d);
        const int key = (kt + i) * 8 + 2 * t;
#pragma unroll
        for (int hr = 0; hr < NT; ++hr) {
          float2 s;
          // (what a row does not see: the next pass scales it by sm_scale, so no finite number would do)
          s.x = key <= q.last[hr] ? unmagic(d[2 * hr]) * q.s[hr] * k0[i] : -INFINITY;
          s.y = key + 1 <= q.last[hr] ? unmagic(d[2 * hr + 1]) * q.s[hr] * k1[i] : -INFINITY;
          mx[hr] = max3(mx[hr], s.x, s.y);
          sc[((kt + i) * NT + hr) * 32] = s;
        }
      }
    }
#pragma unroll
    for (int hr = 0; hr < NT; ++hr) {
      mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 1));
      mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 2));
      if (t == 0) gm[un * RT + g + 8 * hr] = mx[hr];
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// output of one CTA: the 4 warps' results of RT rows x D channels are in red (weights applied), l and m in ml
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void store_row4(const DParams& p, const Unit& u, int r, int ch, const float (&x)[4]) {
  const int h = u.hk * p.ratio + r / p.Nq, n = r % p.Nq;
  __half* o = static_cast<__half*>(p.o) + u.b * p.oB + h * p.oH + n * p.oN + ch;
  uint2 w;
  if (p.o_bf16) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]), b = __floats2bfloat162_rn(x[2], x[3]);
    w.x = *reinterpret_cast<const uint32_t*>(&a);
    w.y = *reinterpret_cast<const uint32_t*>(&b);
  } else {
    const __half2 a = __floats2half2_rn(x[0], x[1]), b = __floats2half2_rn(x[2], x[3]);
    w.x = *reinterpret_cast<const uint32_t*>(&a);
    w.y = *reinterpret_cast<const uint32_t*>(&b);
  }
  *reinterpret_cast<uint2*>(o) = w;
}
// o = acc * (s_v/127) / l for 4 channels of row r
template <bool FULL>
__device__ __forceinline__ void finish_row4(const DParams& p, const Unit& u, int r, int ch, float4 a, float l) {
  const float inv = 1.0f / l;
  float x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (FULL) x[i] *= scale_at(p.vs, u.b * p.vsB + u.hk * p.vsH + (ch + i) * p.vsD, p.scale_f16 & INTFA_SCALE_F16_V) / 127.0f;
    x[i] *= inv;
  }
  store_row4(p, u, r, ch, x);
}
__device__ __forceinline__ void store_lse(const DParams& p, const Unit& u, int r, float m, float l) {
  const int h = u.hk * p.ratio + r / p.Nq, n = r % p.Nq;
  if (p.lse) p.lse[((long long)u.b * p.H + h) * p.Nq + n] = m + log2f(l);
}
template <bool FULL, int D, int NT>
__device__ __forceinline__ void cta_out(const DParams& p, const Unit& u, int split, const float* red, const float (*ml)[2]) {
  constexpr int RT = 8 * NT;
#pragma unroll
  for (int e = threadIdx.x; e < RT * D / 4; e += kThreads) {
    const int r = e / (D / 4), ch = e % (D / 4) * 4, row = u.tile * RT + r;
    if (row >= p.R) continue;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float4 x = *reinterpret_cast<const float4*>(red + (w * RT + r) * (D + 4) + ch);
      a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
    }
    if (p.splits == 1) {
      finish_row4<FULL>(p, u, row, ch, a, ml[r][1]);
      if (ch == 0) store_lse(p, u, row, ml[r][0], ml[r][1]);
    } else {
      const long long pr = ((long long)u.id * p.splits + split) * RT + r;
      *reinterpret_cast<float4*>(p.part + pr * D + ch) = a;
      if (ch == 0) *reinterpret_cast<float2*>(p.part_ml + pr * 2) = make_float2(ml[r][0], ml[r][1]);
    }
  }
}

// The work of one CTA in the second pass, on `nun` units of 64 keys from group g0 on (upg units a group): mg holds the running maximum
// (scaled) at the group of each, ends[1] the final maximum; score(key tile of 8, row tile) is what this lane wants of the scores.
// One warp takes 64 keys at a time, 32 in flight ahead of the arithmetic.
template <int D, int NT>
struct PvFull {
  static constexpr int RT = 8 * NT, VB = D / 8, MT = D / 16;       // VB: bytes (channels) of a key that a lane holds; MT: 16-channel tiles
  static constexpr int W = VB / 4;                                 // ... in words
  const DParams& p;
  const int8_t* vb;
  const int lane, warp, g, t, g0, upg, nun;
  uint32_t vn[8][W];
  float acc[NT][MT][4], lsum[NT];
  __device__ __forceinline__ PvFull(const DParams& p, const Unit& u, int g0, int upg, int nun)
      : p(p), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), g(lane >> 2), t(lane & 3), g0(g0), upg(upg), nun(nun) {
    vb = static_cast<const int8_t*>(p.v) + u.b * p.vB + u.hk * p.vH + g * VB;
  }
  // this lane's 8 keys of a 32-key step: 2t, 2t+1 of each of the four 8-key tiles
  __device__ __forceinline__ void load_v(int key0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int key = min(key0 + (i >> 1) * 8 + 2 * t + (i & 1), p.nvis - 1);
      const int8_t* a = vb + (long long)key * p.vN;
      if constexpr (W == 4) {
        const uint4 x = ld16(a);
        vn[i][0] = x.x; vn[i][1] = x.y; vn[i][2] = x.z; vn[i][3] = x.w;
      } else {
        const uint2 x = ld8(a);
        vn[i][0] = x.x; vn[i][1] = x.y;
      }
    }
  }
  __device__ __forceinline__ void load_first() {
    if (warp < nun) load_v((g0 * upg + warp) * 64);
  }
  template <typename Score>
  __device__ __forceinline__ void run(const float* mg, const float (*ends)[RT], Score score) {
    float m_fin[NT][2], m_fin_g[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      lsum[n] = 0.f;
      m_fin[n][0] = ends[1][n * 8 + 2 * t];
      m_fin[n][1] = ends[1][n * 8 + 2 * t + 1];
      m_fin_g[n] = ends[1][n * 8 + g];
#pragma unroll
      for (int i = 0; i < MT; ++i) acc[n][i][0] = acc[n][i][1] = acc[n][i][2] = acc[n][i][3] = 0.f;
    }
#pragma unroll 1
    for (int un = warp; un < nun; un += kWarps) {
      float nm[NT], w_g[NT], rs[NT];
      int o[NT][MT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const float m = mg[un * RT + n * 8 + g];
        nm[n] = -m;
        w_g[n] = ex2_approx(m - m_fin_g[n]);
        rs[n] = 0.f;
#pragma unroll
        for (int i = 0; i < MT; ++i) o[n][i][0] = o[n][i][1] = o[n][i][2] = o[n][i][3] = kMagicI;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int key0 = (g0 * upg + un) * 64 + half * 32;
        uint32_t vc[8][W];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < W; ++j) vc[i][j] = vn[i][j];
        float2 s[NT][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int n = 0; n < NT; ++n) s[n][i] = score(key0 / 8 + i, n);
        if (half == 0) load_v(key0 + 32);
        else if (un + kWarps < nun) load_v(key0 - 32 + kWarps * 64);
        // P8 of this lane's keys: trunc(fp16(fp16(fp16(p)*127) + 0.5)), as in the 128-row kernel
        uint32_t b[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float2 x = s[n][2 * q], y = s[n][2 * q + 1];
            const float p0 = ex2_approx(fmaf(x.x, p.c, nm[n])), p1 = ex2_approx(fmaf(x.y, p.c, nm[n]));
            const float p2 = ex2_approx(fmaf(y.x, p.c, nm[n])), p3 = ex2_approx(fmaf(y.y, p.c, nm[n]));
            rs[n] += (p0 + p1) + (p2 + p3);
            const __half2 h01 = __floats2half2_rn(p0, p1), h23 = __floats2half2_rn(p2, p3);
            const uint32_t z01 = h2_fma(*reinterpret_cast<const uint32_t*>(&h01), 0x57F057F0u, 0x38003800u);
            const uint32_t z23 = h2_fma(*reinterpret_cast<const uint32_t*>(&h23), 0x57F057F0u, 0x38003800u);
            uint32_t u0, u1, u2, u3;
            h2_floor_add(z01, kMagicF, u0, u1);
            h2_floor_add(z23, kMagicF, u2, u3);
            b[n][q] = __byte_perm(__byte_perm(u0, u1, 0x0040), __byte_perm(u2, u3, 0x0040), 0x5410);
          }
        // O^T (channels x rows): the 4 keys of a quad transposed, so that a word holds one channel's 4 keys
#pragma unroll
        for (int j = 0; j < W; ++j) {
          uint32_t chn[4][2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint32_t x0 = vc[4 * q][j], x1 = vc[4 * q + 1][j], x2 = vc[4 * q + 2][j], x3 = vc[4 * q + 3][j];
            const uint32_t a = __byte_perm(x0, x1, 0x5140), c = __byte_perm(x0, x1, 0x7362);
            const uint32_t d = __byte_perm(x2, x3, 0x5140), e = __byte_perm(x2, x3, 0x7362);
            chn[0][q] = __byte_perm(a, d, 0x5410);
            chn[1][q] = __byte_perm(a, d, 0x7632);
            chn[2][q] = __byte_perm(c, e, 0x5410);
            chn[3][q] = __byte_perm(c, e, 0x7632);
          }
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            mma_s8(o[n][2 * j], chn[0][0], chn[1][0], chn[0][1], chn[1][1], b[n][0], b[n][1]);
            mma_s8(o[n][2 * j + 1], chn[2][0], chn[3][0], chn[2][1], chn[3][1], b[n][0], b[n][1]);
          }
        }
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        lsum[n] = fmaf(w_g[n], rs[n], lsum[n]);
        const float w0 = ex2_approx(mg[un * RT + n * 8 + 2 * t] - m_fin[n][0]), w1 = ex2_approx(mg[un * RT + n * 8 + 2 * t + 1] - m_fin[n][1]);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          acc[n][i][0] = fmaf(unmagic(o[n][i][0]), w0, acc[n][i][0]);
          acc[n][i][1] = fmaf(unmagic(o[n][i][1]), w1, acc[n][i][1]);
          acc[n][i][2] = fmaf(unmagic(o[n][i][2]), w0, acc[n][i][2]);
          acc[n][i][3] = fmaf(unmagic(o[n][i][3]), w1, acc[n][i][3]);
        }
      }
    }
  }
  // the warps' results into red; the sum of the CTA's l on top of what is in ml (written before a barrier)
  __device__ __forceinline__ void results(float* red, float (*ml)[2]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      // tile i of the lane: channel g*VB + 2i (entries 0, 1) and + 1 (2, 3) of rows 2t (0, 2) and 2t+1 (1, 3)
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        float* d = red + (warp * RT + n * 8 + 2 * t) * (D + 4) + g * VB + 2 * i;
        *reinterpret_cast<float2*>(d) = make_float2(acc[n][i][0], acc[n][i][2]);
        *reinterpret_cast<float2*>(d + D + 4) = make_float2(acc[n][i][1], acc[n][i][3]);
      }
      float l = lsum[n];
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      // (one warp after the other, so that the sum has one order)
      for (int w = 0; w < kWarps; ++w) {
        if (w == warp && t == 0) ml[n * 8 + g][1] += l;
        __syncthreads();
      }
    }
  }
};

// ---------------------------------------------------------------------------------------------------------------
// full-int8, second pass: P from the kept scores, O = P V.  Bound by reading V.
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NT>
constexpr int pv_full_ctas() { return NT == 1 ? (D == 64 ? 4 : 3) : 2; }   // of an SM
template <int D, int NT>
__global__ void __launch_bounds__(kThreads, (pv_full_ctas<D, NT>())) pv_full_kernel(const DParams p) {
  constexpr int RT = 8 * NT;
  __shared__ __align__(16) float red[kWarps * RT * (D + 4)];
  __shared__ __align__(16) float mg[kMaxLocalUnits * RT];   // running maximum (scaled) at the group of each 64-key unit of this CTA
  __shared__ __align__(16) float ends[2][RT];               // prefix before the first group; final maximum
  __shared__ float ml[RT][2];
  const int tid = threadIdx.x;
  const int units = gridDim.x / p.splits;
  const Unit u = unit_of(p, blockIdx.x % units);
  const int split = blockIdx.x / units;
  const int g0 = split * p.per_split, g1 = min(p.groups, g0 + p.per_split);
  const int upg = p.G / 64, nun = (g1 - g0) * upg;          // 64-key units of this CTA
  PvFull<D, NT> pv(p, u, g0, upg, nun);
  // (V is older than the first pass)
  pv.load_first();
  pdl_wait();
  pdl_launch();

  // ---- running maxima of this CTA's groups and the final maximum
  {
    const int units64 = p.groups * upg, u0 = g0 * upg;
    const float* gm = p.gmax + (long long)u.id * units64 * RT;
    constexpr int Q4 = RT / 4;                               // threads across a group's rows, 4 rows each
    const int rq = tid % Q4 * 4;
    float4 pre = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY), all = pre;
#pragma unroll 4
    for (int i = tid / Q4; i < units64; i += kThreads / Q4) {
      const float4 x = *reinterpret_cast<const float4*>(gm + i * RT + rq);
      all.x = fmaxf(all.x, x.x); all.y = fmaxf(all.y, x.y); all.z = fmaxf(all.z, x.z); all.w = fmaxf(all.w, x.w);
      if (i < u0) {
        pre.x = fmaxf(pre.x, x.x); pre.y = fmaxf(pre.y, x.y); pre.z = fmaxf(pre.z, x.z); pre.w = fmaxf(pre.w, x.w);
      } else if (i < u0 + nun) {
        *reinterpret_cast<float4*>(mg + (i - u0) * RT + rq) = x;
      }
    }
    float4* sp = reinterpret_cast<float4*>(red);             // (red is free until the end)
    sp[tid] = pre;
    sp[kThreads + tid] = all;
    __syncthreads();
    if (tid < 2 * RT) {
      const int which = tid / RT, r = tid % RT;
      float m = -INFINITY;
#pragma unroll 8
      for (int i = 0; i < kThreads / Q4; ++i) m = fmaxf(m, red[(which * kThreads + i * Q4) * 4 + r]);
      ends[which][r] = m * p.c;
    }
    __syncthreads();
    if (tid < RT) {
      float m = ends[0][tid];
      for (int i = 0; i < nun; i += upg) {
        float x = mg[i * RT + tid];
        if (upg == 2) x = fmaxf(x, mg[(i + 1) * RT + tid]);
        m = fmaxf(m, x * p.c);
        mg[i * RT + tid] = m;
        if (upg == 2) mg[(i + 1) * RT + tid] = m;
      }
    }
    __syncthreads();
  }

  const float2* sc = reinterpret_cast<const float2*>(p.scores) + ((long long)u.id * p.groups * (p.G / 8) * NT) * 32 + (tid & 31);
  pv.run(mg, ends, [&](int kt, int n) { return sc[(kt * NT + n) * 32]; });
  if (tid < RT) {
    ml[tid][0] = ends[1][tid];
    ml[tid][1] = 0.f;
  }
  __syncthreads();
  pv.results(red, ml);
  cta_out<true, D, NT>(p, u, split, red, ml);
}

// ---------------------------------------------------------------------------------------------------------------
// full-int8, both passes in one kernel: a unit's splits are a cluster.  Each CTA computes the scores of its keys and keeps them in
// shared memory; the CTAs exchange their maxima, which gives each the running maximum before its first key and the final one, and then
// their results, of which every CTA adds up and writes some rows -- both through distributed shared memory.  The scores make no way
// through L2 (a quarter of the bytes of K at 4 rows a head), there is no scratch, and one launch instead of three.  Bound by reading K
// and V, 12 warps an SM (fused_is_faster says what it gives and where).
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NT>
struct FusedCfg {
  static constexpr int RT = 8 * NT;
  // Scores of a CTA in bytes.  The CTAs of an SM must not need more than 196 KB of its shared memory: the next larger setting, 228 KB,
  // leaves 28 KB of L1, through which the loads in flight go (12 K/V heads of 128 channels, 8118 keys: 1984 keys a CTA 59 us, three
  // kernels 42; every call takes half as long again with that setting).  Three CTAs an SM, 60 KB each beside their static 4 KB.
  static constexpr int MAX_SCORES = NT == 1 ? 60 << 10 : 100 << 10;
  static constexpr int RED_BYTES = kWarps * RT * (D + 4) * 4;
  // Dynamic shared memory of a CTA.  At 64 channels the registers leave room for four an SM: where those would need the 228 KB
  // setting the size is rounded up to one of which three fit (320 heads of 1367 keys 28.3 -> 20.2 us, 400 of 4097 73 -> 61).
  static int smem_bytes(int keys) {
    const int b = keys * NT * 32;
    if (D == 64 && NT == 1 && b > (43 << 10) && b < (52 << 10)) return 52 << 10;
    return b < RED_BYTES ? RED_BYTES : b;
  }
};
template <int D, int NT>
__global__ void __launch_bounds__(kThreads, NT == 1 ? 3 : 2) fused_full_kernel(const DParams p) {
  constexpr int RT = 8 * NT, CH = D / 64;
  extern __shared__ __align__(16) uint8_t dyn[];
  __shared__ __align__(16) float mg[kMaxLocalUnits * RT];
  __shared__ __align__(16) float ends[2][RT];
  __shared__ float cmax[RT];                                // this CTA's maximum (scaled), for its peers
  __shared__ float ml[RT][2];
  float2* sc = reinterpret_cast<float2*>(dyn);              // [key tile of 8][NT][32 lanes]; afterwards the results
  float* red = reinterpret_cast<float*>(dyn);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const uint32_t rank = cluster_rank();
  const Unit u = unit_of(p, blockIdx.x / p.splits);
  const int g0 = (int)rank * p.per_split, g1 = min(p.groups, g0 + p.per_split);
  const int upg = p.G / 64, nun = (g1 - g0) * upg;
  pdl_wait();
  pdl_launch();
  {
    QRows<D, NT> q;
    q.load(p, u, g, t);
    const int8_t* kb = p.k + u.b * p.kB + u.hk * p.kH + t * 16;
    const long long ksb = u.b * p.ksB + u.hk * p.ksH;
    const int kf16 = p.scale_f16 & INTFA_SCALE_F16_K;
    // 64 keys in two halves, one loaded while the other is computed
    struct Half {
      uint4 kw[4][CH];
      float k0[4], k1[4];
    } a, b;
    auto load_k = [&](int kt, Half& x) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int8_t* row = kb + (long long)min((kt + i) * 8 + g, p.nvis - 1) * p.kN;
#pragma unroll
        for (int c = 0; c < CH; ++c) x.kw[i][c] = ld16(row + c * 64);
        const int key = (kt + i) * 8 + 2 * t;
        x.k0[i] = scale_at(p.ks, ksb + min(key, p.nvis - 1), kf16);
        x.k1[i] = scale_at(p.ks, ksb + min(key + 1, p.nvis - 1), kf16);
      }
    };
    const int kt0 = g0 * upg * 8;
    float mx[NT];
    auto scores = [&](int kt, const Half& x) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        int d[4];
        qk_tile<D, NT>(q, x.kw[i], d);
        const int key = (kt0 + kt + i) * 8 + 2 * t;
#pragma unroll
        for (int hr = 0; hr < NT; ++hr) {
          float2 s;
          s.x = key <= q.last[hr] ? unmagic(d[2 * hr]) * q.s[hr] * x.k0[i] : -INFINITY;
          s.y = key + 1 <= q.last[hr] ? unmagic(d[2 * hr + 1]) * q.s[hr] * x.k1[i] : -INFINITY;
          mx[hr] = max3(mx[hr], s.x, s.y);
          sc[((kt + i) * NT + hr) * 32 + lane] = s;
        }
      }
    };
    if (warp < nun) load_k(kt0 + warp * 8, a);
#pragma unroll 1
    for (int un = warp; un < nun; un += kWarps) {
#pragma unroll
      for (int i = 0; i < NT; ++i) mx[i] = -INFINITY;
      load_k(kt0 + un * 8 + 4, b);
      scores(un * 8, a);
      if (un + kWarps < nun) load_k(kt0 + (un + kWarps) * 8, a);
      scores(un * 8 + 4, b);
#pragma unroll
      for (int hr = 0; hr < NT; ++hr) {
        mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 1));
        mx[hr] = fmaxf(mx[hr], __shfl_xor_sync(0xffffffffu, mx[hr], 2));
        if (t == 0) mg[un * RT + g + 8 * hr] = mx[hr];
      }
    }
  }
  PvFull<D, NT> pv(p, u, g0, upg, nun);
  pv.load_first();
  __syncthreads();
  if (tid < RT) {
    float m = -INFINITY;
    for (int i = 0; i < nun; i += upg) {
      float x = mg[i * RT + tid];
      if (upg == 2) x = fmaxf(x, mg[(i + 1) * RT + tid]);
      m = fmaxf(m, x * p.c);
      mg[i * RT + tid] = m;
      if (upg == 2) mg[(i + 1) * RT + tid] = m;
    }
    cmax[tid] = m;
  }
  cluster_arrive();
  cluster_wait();
  if (tid < RT) {
    float pre = -INFINITY, all = -INFINITY;
    for (uint32_t c = 0; c < (uint32_t)p.splits; ++c) {
      const float x = ld_peer(&cmax[tid], c);
      all = fmaxf(all, x);
      if (c < rank) pre = fmaxf(pre, x);
    }
    ends[0][tid] = pre;
    ends[1][tid] = all;
    ml[tid][0] = all;
    ml[tid][1] = 0.f;
  }
  __syncthreads();
  for (int i = tid; i < nun * RT; i += kThreads) mg[i] = fmaxf(mg[i], ends[0][i % RT]);
  __syncthreads();
  const int kt0 = g0 * upg * 8;
  pv.run(mg, ends, [&](int kt, int n) { return sc[((kt - kt0) * NT + n) * 32 + lane]; });
  __syncthreads();                                          // (the scores are done with)
  pv.results(red, ml);
#pragma unroll
  for (int e = tid; e < RT * D / 4; e += kThreads) {
    float4* x = reinterpret_cast<float4*>(red + e / (D / 4) * (D + 4) + e % (D / 4) * 4);
    float4 a = x[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) {
      const float4 y = x[w * RT * (D + 4) / 4];
      a.x += y.x; a.y += y.y; a.z += y.z; a.w += y.w;
    }
    x[0] = a;
  }
  cluster_arrive();
  cluster_wait();
  for (int e = tid; e < RT * D / 4; e += kThreads) {
    const int r = e / (D / 4), ch = e % (D / 4) * 4, row = u.tile * RT + r;
    if (r % p.splits != (int)rank || row >= p.R) continue;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (uint32_t c = 0; c < (uint32_t)p.splits; ++c) {
      const float4 y = ld_peer4(red + r * (D + 4) + ch, c);
      a.x += y.x; a.y += y.y; a.z += y.z; a.w += y.w;
      l += ld_peer(&ml[r][1], c);
    }
    finish_row4<true>(p, u, row, ch, a, l);
    if (ch == 0) store_lse(p, u, row, ml[r][0], l);
  }
  cluster_arrive();                                         // (no CTA ends while a peer reads from it)
  cluster_wait();
}

// ---------------------------------------------------------------------------------------------------------------
// half-int8: scores, softmax and P V in one pass; one warp takes 32 keys at a time, with a running maximum of its own
// ---------------------------------------------------------------------------------------------------------------
template <int D, int NT>
__global__ void __launch_bounds__(kThreads, D == 64 ? 3 : 2) pv_half_kernel(const DParams p) {
  constexpr int RT = 8 * NT, CH = D / 64, MT = D / 16;
  __shared__ __align__(16) float red[kWarps * RT * (D + 4)];
  __shared__ float wml[kWarps][RT][2];
  __shared__ float ml[RT][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int units = gridDim.x / p.splits;
  const Unit u = unit_of(p, blockIdx.x % units);
  const int split = blockIdx.x / units;
  const int k_begin = split * p.per_split * 64, k_end = min(p.nvis, k_begin + p.per_split * 64);
  pdl_wait();
  pdl_launch();
  QRows<D, NT> q;
  q.load(p, u, g, t);
  const int8_t* kb = p.k + u.b * p.kB + u.hk * p.kH + t * 16;
  const __half* vb = static_cast<const __half*>(p.v) + u.b * p.vB + u.hk * p.vH + g * 8;
  const long long ksb = u.b * p.ksB + u.hk * p.ksH;
  const int kf16 = p.scale_f16 & INTFA_SCALE_F16_K;
  float acc[NT][MT][4], m[NT], l[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    m[n] = -INFINITY;
    l[n] = 0.f;
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[n][i][0] = acc[n][i][1] = acc[n][i][2] = acc[n][i][3] = 0.f;
  }
  uint4 kw[4][CH];
  float k0[4], k1[4];
  auto load_k = [&](int key0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int8_t* row = kb + (long long)min(key0 + i * 8 + g, p.nvis - 1) * p.kN;
#pragma unroll
      for (int c = 0; c < CH; ++c) kw[i][c] = ld16(row + c * 64);
      const int key = key0 + i * 8 + 2 * t;
      k0[i] = scale_at(p.ks, ksb + min(key, p.nvis - 1), kf16);
      k1[i] = scale_at(p.ks, ksb + min(key + 1, p.nvis - 1), kf16);
    }
  };
  const int first = k_begin + warp * 32;
  if (first < k_end) load_k(first);
  // One step of 32 keys.  TAIL: fewer of them; P of the missing ones is 0, and so must V be (the last key in their place may
  // hold an infinity).  A body of its own: any test of the kind in the common one costs its loads their overlap (32768 keys of
  // 8 K/V heads, one row: 22.6 -> 24.1 to 25.1 us).
  auto step = [&](int key0, auto tail) {
    constexpr bool TAIL = decltype(tail)::value;
    // V of the first 16 keys is on its way while the scores are computed
    uint4 v[4][CH];
    auto load_v = [&](int h) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int key = key0 + h * 16 + (i >> 1) * 8 + 2 * t + (i & 1);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          if (TAIL) v[i][c] = make_uint4(0, 0, 0, 0);
          if (!TAIL || key < p.nvis) v[i][c] = ld16(vb + (long long)key * p.vN + c * 64);
        }
      }
    };
    load_v(0);
    float x[NT][4][2], mx[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) mx[n] = m[n];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int d[4];
      qk_tile<D, NT>(q, kw[i], d);
      const int key = key0 + i * 8 + 2 * t;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        x[n][i][0] = key <= q.last[n] ? unmagic(d[2 * n]) * q.s[n] * k0[i] * p.c : -1.0e30f;
        x[n][i][1] = key + 1 <= q.last[n] ? unmagic(d[2 * n + 1]) * q.s[n] * k1[i] * p.c : -1.0e30f;
        mx[n] = max3(mx[n], x[n][i][0], x[n][i][1]);
      }
    }
    if (key0 + kWarps * 32 < k_end) load_k(key0 + kWarps * 32);
    bool moved = false;
    float al[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      mx[n] = fmaxf(mx[n], __shfl_xor_sync(0xffffffffu, mx[n], 1));
      mx[n] = fmaxf(mx[n], __shfl_xor_sync(0xffffffffu, mx[n], 2));
      mx[n] = fmaxf(mx[n], -1.0e29f);           // (a row that has seen no key yet: its p are 0)
      al[n] = ex2_approx(m[n] - mx[n]);
      moved |= mx[n] != m[n];
      m[n] = mx[n];
    }
    if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        l[n] *= al[n];
        const float a0 = __shfl_sync(0xffffffffu, al[n], 8 * t), a1 = __shfl_sync(0xffffffffu, al[n], 8 * t + 4);   // rows 2t, 2t+1
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          acc[n][i][0] *= a0;
          acc[n][i][1] *= a1;
          acc[n][i][2] *= a0;
          acc[n][i][3] *= a1;
        }
      }
    }
    uint32_t b[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float p0 = ex2_approx(x[n][i][0] - m[n]), p1 = ex2_approx(x[n][i][1] - m[n]);
        l[n] += p0 + p1;
        const __half2 h = __floats2half2_rn(p0, p1);
        b[n][i] = *reinterpret_cast<const uint32_t*>(&h);
      }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // O^T (channels x rows): two keys of one channel in a word
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const uint32_t* x0 = reinterpret_cast<const uint32_t*>(&v[0][c]);
        const uint32_t* x1 = reinterpret_cast<const uint32_t*>(&v[1][c]);
        const uint32_t* x2 = reinterpret_cast<const uint32_t*>(&v[2][c]);
        const uint32_t* x3 = reinterpret_cast<const uint32_t*>(&v[3][c]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t a0 = __byte_perm(x0[j], x1[j], 0x5410), a1 = __byte_perm(x0[j], x1[j], 0x7632);
          const uint32_t a2 = __byte_perm(x2[j], x3[j], 0x5410), a3 = __byte_perm(x2[j], x3[j], 0x7632);
#pragma unroll
          for (int n = 0; n < NT; ++n) mma_f16(acc[n][c * 4 + j], a0, a1, a2, a3, b[n][2 * h], b[n][2 * h + 1]);
        }
      }
      if (h == 0) load_v(1);
    }
  };
  int key0 = first;
  // (a CTA of few keys fetches one of the two bodies only: 6.5 -> 6.0 us for a call of a few hundred keys)
  if ((k_end & 31) == 0 || k_end - k_begin > 512) {
#pragma unroll 1
    for (; key0 + 32 <= k_end; key0 += kWarps * 32) step(key0, Const<false>());
  }
#pragma unroll 1
  for (; key0 < k_end; key0 += kWarps * 32) step(key0, Const<true>());
  // ---- the warps' results, scaled to the CTA's maximum
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    l[n] += __shfl_xor_sync(0xffffffffu, l[n], 1);
    l[n] += __shfl_xor_sync(0xffffffffu, l[n], 2);
    if (t == 0) {
      wml[warp][n * 8 + g][0] = m[n];
      wml[warp][n * 8 + g][1] = l[n];
    }
  }
  __syncthreads();
  auto cta_max = [&](int r) { return fmaxf(fmaxf(wml[0][r][0], wml[1][r][0]), fmaxf(wml[2][r][0], wml[3][r][0])); };
  static_assert(kWarps == 4, "cta_max");
  if (tid < RT) {
    const float mm = cta_max(tid);
    float ls = 0.f;
    for (int w = 0; w < kWarps; ++w) ls += wml[w][tid][1] * (wml[w][tid][0] == -INFINITY ? 0.f : ex2_approx(wml[w][tid][0] - mm));
    ml[tid][0] = mm;
    ml[tid][1] = ls;
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    float w01[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = n * 8 + 2 * t + e;
      w01[e] = wml[warp][r][0] == -INFINITY ? 0.f : ex2_approx(wml[warp][r][0] - cta_max(r));
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      float* d = red + (warp * RT + n * 8 + 2 * t) * (D + 4) + (i / 4) * 64 + g * 8 + 2 * (i % 4);
      *reinterpret_cast<float2*>(d) = make_float2(acc[n][i][0] * w01[0], acc[n][i][2] * w01[0]);
      *reinterpret_cast<float2*>(d + D + 4) = make_float2(acc[n][i][1] * w01[1], acc[n][i][3] * w01[1]);
    }
  }
  __syncthreads();
  cta_out<false, D, NT>(p, u, split, red, ml);
}

// Sum of the splits' results, one CTA of D/4 threads per row.  (full: all on the final maximum already; half: weighted.)
// For up to few_splits() of them: two latencies at most.
constexpr int few_splits(bool full) { return full ? 4 : 2; }
template <bool FULL, int D>
__global__ void __launch_bounds__(D / 4) combine_kernel(const DParams p, int RT) {
  const Unit u = unit_of(p, blockIdx.x / RT);
  const int r = blockIdx.x % RT, row = u.tile * RT + r, ch = threadIdx.x * 4;
  pdl_wait();
  pdl_launch();
  if (row >= p.R) return;
  const long long base = (long long)u.id * p.splits * RT + r;
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml);
  float m = -INFINITY;
  if constexpr (FULL) {
    m = ml[base].x;
  } else {
#pragma unroll 8
    for (int s = 0; s < p.splits; ++s) m = fmaxf(m, ml[base + (long long)s * RT].x);
  }
  float l = 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int s = 0; s < p.splits; ++s) {
    const long long pr = base + (long long)s * RT;
    const float2 x = ml[pr];
    const float4 y = *reinterpret_cast<const float4*>(p.part + pr * D + ch);
    const float w = FULL ? 1.f : (x.x == -INFINITY ? 0.f : ex2_approx(x.x - m));
    l = fmaf(w, x.y, l);
    a.x = fmaf(w, y.x, a.x); a.y = fmaf(w, y.y, a.y); a.z = fmaf(w, y.z, a.z); a.w = fmaf(w, y.w, a.w);
  }
  finish_row4<FULL>(p, u, row, ch, a, l);
  if (ch == 0) store_lse(p, u, row, m, l);
}

// The same for more splits.  A chain of L2 latencies, so the splits are spread over groups of D/4 threads, 4 splits in flight
// in each, whose first loads do not wait for the maxima (half-int8: 37 splits, the call 26.4 -> 22.3 us; 6 splits 40.6 -> 39.3;
// 4 splits 23.1 -> 22.0; full-int8: 3 splits 24.4 -> 25.4).  No more groups than the splits fill: many short rows are bound by
// the number of warps.
constexpr int kCombineThreads = 256;
inline int combine_threads(int D, int splits) {
  int threads = D / 4 < 32 ? 32 : D / 4;
  while (threads < kCombineThreads && threads / (D / 4) * 4 < splits) threads *= 2;
  return threads;
}
template <bool FULL, int D>
__global__ void __launch_bounds__(kCombineThreads) combine_many_kernel(const DParams p, int RT) {
  constexpr int C4 = D / 4, U = 4;
  __shared__ float4 red[kCombineThreads];
  const int CG = blockDim.x / C4;
  const Unit u = unit_of(p, blockIdx.x / RT);
  const int r = blockIdx.x % RT, row = u.tile * RT + r, c4 = threadIdx.x % C4, grp = threadIdx.x / C4, lane = threadIdx.x & 31;
  pdl_wait();
  pdl_launch();
  if (row >= p.R) return;
  const long long base = (long long)u.id * p.splits * RT + r;
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + base;
  const float* part = p.part + base * D + c4 * 4;
  float4 y[U];
  float mx[U];
  auto load = [&](int s0) {
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int s = s0 + i * CG;
      y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      mx[i] = -INFINITY;
      if (s < p.splits) {
        y[i] = *reinterpret_cast<const float4*>(part + (long long)s * RT * D);
        if (!FULL) mx[i] = ml[s * RT].x;
      }
    }
  };
  load(grp);
  // every warp for itself: the maximum and l
  const float2 x0 = lane < p.splits ? ml[lane * RT] : make_float2(-INFINITY, 0.f);
  float m = x0.x;
  for (int s = lane + 32; s < p.splits; s += 32) m = fmaxf(m, ml[s * RT].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  auto weight = [&](float x) { return x == -INFINITY ? 0.f : FULL ? 1.f : ex2_approx(x - m); };
  float l = x0.y * weight(x0.x);
  for (int s = lane + 32; s < p.splits; s += 32) l = fmaf(weight(ml[s * RT].x), ml[s * RT].y, l);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = grp; s0 < p.splits; s0 += U * CG) {
    if (s0 != grp) load(s0);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const float w = FULL ? 1.f : weight(mx[i]);
      a.x = fmaf(w, y[i].x, a.x); a.y = fmaf(w, y[i].y, a.y); a.z = fmaf(w, y[i].z, a.z); a.w = fmaf(w, y[i].w, a.w);
    }
  }
  red[threadIdx.x] = a;
  __syncthreads();
  if (grp > 0) return;
  for (int i = 1; i < CG; ++i) {
    const float4 b = red[i * C4 + c4];
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
  }
  finish_row4<FULL>(p, u, row, c4 * 4, a, l);
  if (c4 == 0) store_lse(p, u, row, m, l);
}

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------
struct Plan {
  bool use = false, full = false, fused = false;           // fused: one kernel, the splits of a unit are a cluster
  int NT = 1, tiles = 1, units = 0, slice = 0, nvis = 0, groups = 0, splits = 1, per_split = 1, score_splits = 1;
  size_t off_gmax = 0, off_part = 0, off_ml = 0, bytes = 0;
};

// Scratch of one call, unless one unit needs more.  The scores of full-int8 are fp32 and padded to 8 or 16 rows, up to as much
// again as K and V, so a call that needs more takes its units in slices that share it, one after the other.  (Half of this
// bound cuts up calls of few units, which then leave SMs idle: 128 units of 16384 keys 91 -> 104 to 110 us.)
constexpr size_t kMaxScratch = (size_t)256 << 20;

// Which path?  Times in microseconds, fitted to 3 781 calls that were timed on both (1 to 256 rows a head, 50 to 16384 keys, 1 to
// 512 heads in all; B200).  The kernels timed were earlier ones of both paths: the 128-row kernel has become 4 to 32 % faster since,
// full-int8 here up to 30 % where one kernel does for three, which the model does not know: near the line the slower
// path may be taken.
//   here       `fixed` and `combine` for the launches; `unit` per 64 keys of a row tile and SM (times `one_half` for tiles of 8
//              rows); `wave` for each further wave of CTAs
//   128 rows   `fill`, then `step` per KV step of G keys and `next` for each further work item of an SM.  The work items of
//              these calls are of one length, so an SM has a whole number of them.
// Typical error 5 to 15 %.  Over those calls, on those kernels, the choice cost 0.3 % against the better path each time, and 48 of them
// more than 10 %.  (One step time for any G and head dim, and no term for waves, before: 0.5 %, 72 of 1 610 calls more than 10 %, up
// to twice the time for half-int8 with 64-column steps.)
struct FewTimes {
  double fixed, combine, unit, one_half, wave;
};
struct TileTimes {
  double fill, step, next;
};
constexpr FewTimes kFew[2][2] = {{{5.41, 3.22, 0.267, 1.04, 1.40}, {6.14, 3.35, 0.490, 1.02, 3.27}},        // half-int8: d = 64, 128
                                 {{7.52, 1.93, 0.386, 0.73, 3.01}, {8.70, 1.80, 0.540, 0.81, 4.46}}};       // full-int8
constexpr TileTimes kTiles[2][2][2] = {{{{8.99, 0.694, 6.59}, {6.92, 1.179, 2.21}},                         // half-int8, d = 64: G = 64, 128
                                        {{9.23, 0.765, 6.47}, {7.49, 1.235, 2.46}}},
                                       {{{8.71, 0.838, 4.72}, {7.01, 1.432, 2.71}}, {{10.43, 0.962, 7.97}, {8.72, 1.359, 3.80}}}};
bool faster_than_tiles(const IntfaFwdParams* a, const Plan& pl, int wave, int sms) {
  const FewTimes& f = kFew[pl.full][a->D == 128];
  const TileTimes& t = kTiles[pl.full][a->D == 128][a->G == 128];
  const int slices = (pl.units + pl.slice - 1) / pl.slice;
  const double waves = (double)pl.slice * pl.splits / wave;
  const double here = (f.fixed + (pl.splits > 1 ? f.combine : 0.0) + (waves > 1 ? f.wave * (waves - 1) : 0.0)) * slices +
                      f.unit * (pl.NT == 1 ? f.one_half : 1.0) * (double)pl.units * ((pl.nvis + 63) / 64) / sms;
  const long long items = (long long)a->B * a->H * ((a->Nq + 127) / 128);
  const double rounds = (double)((items + sms - 1) / sms);
  const double steps = (double)((pl.nvis + a->G - 1) / a->G);
  double mean = a->causal ? steps - 0.5 * a->Nq / a->G : steps;             // steps of an average work item
  if (mean < 1) mean = 1;
  return here < t.fill + t.step * (rounds > 1 ? rounds * mean : steps) + t.next * (rounds - 1);
}

// Clusters of n CTAs of fused_full_kernel that the current device holds at once; 0: none, or it cannot be asked.  Not SMs * CTAs an SM / n:
// a cluster stays within a group of SMs, which n need not divide (three CTAs an SM, n = 3 to 8: 426, 416, 410, 426, 392, 384 CTAs of
// 444).  Asked once per device, kernel and n, for CTAs of up to 40 KB and for the largest.
template <int D, int NT>
int fused_places_of(int n, int smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)n;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaFuncSetAttribute(fused_full_kernel<D, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, FusedCfg<D, NT>::MAX_SCORES) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, fused_full_kernel<D, NT>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return clusters;
}
int fused_places(int D, int NT, int n, int keys) {
  static std::atomic<int> cache[64][2][2][kMaxCluster + 1][2];           // number + 1; 0: not asked yet
  constexpr int kSmall = 40 << 10;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  const int large = keys * NT * 32 > kSmall;
  std::atomic<int>& c = cache[dev][D == 128][NT - 1][n][large];
  int v = c.load(std::memory_order_relaxed);
  if (v == 0) {
    auto ask = [&](auto d, auto nt) {
      using F = FusedCfg<decltype(d)::value, decltype(nt)::value>;
      return fused_places_of<decltype(d)::value, decltype(nt)::value>(n, large ? F::MAX_SCORES : kSmall);
    };
    v = 1 + (D == 128 ? (NT == 2 ? ask(Int<128>(), Int<2>()) : ask(Int<128>(), Int<1>()))
                      : (NT == 2 ? ask(Int<64>(), Int<2>()) : ask(Int<64>(), Int<1>())));
    c.store(v, std::memory_order_relaxed);
  }
  return v - 1;
}

// Is fused_full_kernel with clusters of n CTAs and `keys` keys a CTA faster than the three kernels of `pl`?  `wave`: the CTAs it is
// laid out for, `wave3`: the resident ones of pv_full_kernel; `fewest`: no CTA has more keys than a split is given at least.  Fitted to
// 1 893 calls timed on both, inputs in and out of L2 (1 to 16 rows a head, 6 to 15 164 keys, 1 to 4 448 units).  Of these it takes 1 174:
// 8 % faster at the median, 5 of them slower by more than 4 %.  Of the others most would be slower, by up to 83 %; 55 would be faster by
// more than 5 %, chiefly some with 16 rows.
bool fused_is_faster(int D, const Plan& pl, int n, int keys, int wave, int wave3, bool fewest) {
  const int places = fused_places(D, pl.NT, n, keys);
  if (places <= 0) return false;
  const long long ctas = (long long)pl.units * n;
  auto full = [](long long have, long long of, int percent) { return have * 100 >= of * percent; };
  if (pl.units <= places) {              // one wave
    // 128 channels, more than 256 keys a CTA: a warp has more than one unit in each pass, which few CTAs do not make up for (two units
    // of 443 keys 6.7 -> 7.1 us; 16 rows, 8 units of 501 keys 9.7 -> 10.5)
    const bool chain = D == 128 && keys > 256;
    // 16 rows, 8 warps an SM to read with: where a CTA has the fewest keys (2 x 2048 keys, 8 rows a head 15.0 -> 14.0; 1 500 keys a
    // CTA 34.8 -> 37.2)
    if (pl.NT == 2) return fewest && !(chain && (ctas < 24 || (n <= 2 && ctas <= 60)));
    // Many keys in fewer CTAs than there is room for do not keep the memory busy, while the scores' kernel fills the chip with any
    // number of units: 64 channels, 112 units of 3260 keys 18.8 -> 20.1, 108 of 2960 17.4 -> 15.2, 224 of 1490 17.2 -> 19.6; 128
    // channels, 244 of 1610 28.0 -> 32.8, 429 of 1720 40.4 -> 37.1
    if (D == 64) return n == 1 ? keys <= 1408 || full(ctas, wave, 60) : keys <= 768 || keys >= 1408 || full(ctas, wave, n == 2 ? 80 : 91);
    if (chain && (n > 1 ? pl.units == 1 : pl.units < 36)) return false;
    if (n == 1) return full(ctas, wave, 85) || keys <= 512 || (keys <= 1280 && full(ctas, wave, 55));
    return keys <= 1536;                 // (more leave less L1: 132 units of 4809 keys 35.7 -> 36.8)
  }
  if (pl.NT == 2) return false;          // (248 units of 1636 keys 36.0 -> 43.2)
  // Several waves: where the last one is nearly full, and the three kernels are not well off with one or two
  const int slices = (pl.units + pl.slice - 1) / pl.slice;
  const long long ctas3 = (long long)pl.slice * pl.splits, waves3 = (ctas3 + wave3 - 1) / wave3;
  const long long waves = (pl.units + places - 1) / places, waves_up = (ctas + wave - 1) / wave;
  if (n > 3) return false;                                               // (72 units of 9216 keys 24.5 -> 37.0)
  if (n > 1 && slices == 1 && waves3 == 1 && full(ctas3, wave3, D == 64 ? 55 : 70)) return false;     // (144 units of 4980 keys 38.9 -> 58.1)
  if (D == 64) {
    if (n == 1 && keys <= 1280) return true;                             // (560 units of 701 keys 19.7 -> 14.3)
    if (slices == 1 && waves3 == 2 && full(ctas3, 2 * wave3, 93)) return false;                       // (1 184 units of 1304 keys 48.2 -> 54.4)
    return full(pl.units, waves * places, 83) || full(ctas, waves_up * wave, 83);
  }
  if (keys <= 64 && waves > 2) return false;                             // (one warp of four works: 2 499 units of 61 keys 33.5 -> 35.6)
  // (512 units of 4097 keys 135 -> 115, 1 104 of 1711 108 -> 102, 556 of 984 36.9 -> 38.5)
  return full(pl.units, waves * places, waves > 2 ? 80 : 83);
}

Plan make_plan(const IntfaFwdParams* a, int sms) {
  Plan pl;
  const int Hkv = a->H_kv > 0 ? a->H_kv : a->H;
  pl.full = a->variant == INTFA_VARIANT_FULL;
  // Options that the 128-row kernel keeps: head dims 16, 32, 256, fp8 V (its rounding of P follows the running maximum, too),
  // carried state, KV tiles last to first, per-tile V scales, RNE rounding, the debug tap, rows that see no key at all.
  // Calls of more than kDecodeRows rows a head stay there too: a pass continued through carried state is the same as one pass
  // bit for bit only where both run the same kernel, and that is what long sequences are cut up for.
  constexpr int kDecodeRows = 256;
  if (a->Nq > kDecodeRows || (a->D != 64 && a->D != 128) || (!pl.full && a->variant != INTFA_VARIANT_HALF) || (a->G != 64 && a->G != 128)) return pl;
  if (a->state_in || a->state_out || !a->write_o || a->kv_order || a->vs_stride_blk || (pl.full && a->p_round) || a->dbg_s || a->debug_skip_k_load) return pl;
  if (!(a->sm_scale > 0.f) || (a->causal && a->q_offset < a->kv_offset)) return pl;
  pl.nvis = a->Nk;
  if (a->causal) {
    const long long vis = a->q_offset + a->Nq - a->kv_offset;
    if (vis < pl.nvis) pl.nvis = (int)vis;
  }
  const long long R = (long long)(a->H / Hkv) * a->Nq;
  pl.NT = R > 8 ? 2 : 1;
  const int RT = 8 * pl.NT;
  pl.tiles = (int)((R + RT - 1) / RT);
  const long long units = (long long)a->B * Hkv * pl.tiles;
  if (units > (1 << 22)) return pl;
  pl.units = pl.slice = (int)units;
  pl.groups = (pl.nvis + a->G - 1) / a->G;
  // Splits: one wave of resident CTAs, as the kernels' launch bounds have it (full-int8 at 8 rows and 128 channels: two CTAs an SM or
  // four 35 -> 44 us at batch 16, 4097 keys; at 64 channels four, planned for three 264 heads of 6000 keys 65.8, for four 50.0; half-int8
  // at 128 channels: three 26.5 -> 30 us at 32768 keys)
  const int wave = sms * (pl.full ? (pl.NT == 2 ? pv_full_ctas<64, 2>() : a->D == 64 ? pv_full_ctas<64, 1>() : pv_full_ctas<128, 1>())
                                  : pl.NT == 1 && a->D == 64 ? 3 : 2);
  const int key_units = (pl.nvis + 63) / 64;
  size_t per_unit_scores = 0, per_unit_max = 0;
  if (pl.full) {
    if (pl.nvis > (1 << 27)) return pl;                                    // (the kernels count a unit's scores in 32 bits)
    per_unit_scores = (size_t)pl.groups * (a->G / 8) * pl.NT * 32 * 8;
    per_unit_max = (size_t)pl.groups * (a->G / 64) * RT * 4;
    const size_t most = (kMaxScratch - (8u << 20)) / (per_unit_scores + per_unit_max);       // (the rest: the splits' results)
    const int fit = most < 1 ? 1 : most > (1u << 22) ? 1 << 22 : (int)most, least = (pl.units + fit - 1) / fit;
    // As few slices as fit, or up to three more where their CTAs fill the waves better (16 rows, 512 units of 8192 keys, one
    // slice 301 us: 3 slices 380, 4 308, 5 328, 6 305; 8 rows, 512 units of 16384 keys, one slice 470: 448, 440, 419, 414)
    double best = 0;
    for (int n = least; n <= least + 3 && (n == 1 || least > 1); ++n) {
      const int slice = (pl.units + n - 1) / n, ctas = slice < wave ? wave / slice * slice : slice;
      const double fill = (double)ctas / ((ctas + wave - 1) / wave * wave);
      if (fill > best * 1.02) {
        best = fill;
        pl.slice = slice;
      }
    }
  }
  const int items = pl.full ? pl.groups : key_units;          // what a split is counted in
  const int per_min = pl.full ? 512 / a->G : 8;               // at least 512 keys per CTA: fewer are not worth the combine launch
  int splits = wave / pl.slice < 1 ? 1 : wave / pl.slice;
  int per = (items + splits - 1) / splits;
  if (per < per_min) per = per_min;
  if (pl.full && per > kMaxLocalUnits * 64 / a->G) per = kMaxLocalUnits * 64 / a->G;
  pl.per_split = per;
  pl.splits = (items + per - 1) / per;
  const int score_ctas = sms * (a->D == 128 ? 5 : 6);                      // resident at their register counts
  pl.score_splits = score_ctas / pl.slice < 1 ? 1 : score_ctas / pl.slice;
  const int score_cap = (pl.groups * (a->G / 64) + kWarps - 1) / kWarps;
  if (pl.score_splits > score_cap) pl.score_splits = score_cap;
  if ((long long)pl.slice * pl.splits > 0x7fffffffLL || (long long)pl.slice * pl.score_splits > 0x7fffffffLL) return pl;
  if (!faster_than_tiles(a, pl, wave, sms)) return pl;
  // One kernel (fused_full_kernel) where the splits of a unit make a cluster whose CTAs hold their scores, if need be more of them than
  // fill one wave.  No scratch to speak of, so nothing is cut into slices.
  if (pl.full) {
    const int max_keys = (pl.NT == 1 ? FusedCfg<128, 1>::MAX_SCORES : FusedCfg<128, 2>::MAX_SCORES) / (pl.NT * 32);
    const int fill = sms * (pl.NT == 1 ? 3 : 2);              // CTAs to share the work out to
    int n = fill / (int)units < 1 ? 1 : fill / (int)units;
    per = (items + n - 1) / n;
    if (per < per_min) per = per_min;
    if (per > max_keys / a->G) per = max_keys / a->G;
    n = (items + per - 1) / per;
    per = (items + n - 1) / n;
    n = (items + per - 1) / per;
    if (n <= kMaxCluster && fused_is_faster(a->D, pl, n, per * a->G, fill, wave, per <= per_min)) {
      pl.fused = true;
      pl.per_split = per;
      pl.splits = n;
      pl.slice = pl.units;
    }
  }
  size_t used = 0;
  auto take = [&](size_t bytes) {
    const size_t r = used;
    used += (bytes + 255) / 256 * 256;
    return r;
  };
  if (pl.fused) {
    take(1);                    // (none is used; but a call that brings no scratch at all runs on 128-row tiles, as ever)
    pl.bytes = used;
    pl.use = true;
    return pl;
  }
  if (pl.full) {
    take(pl.slice * per_unit_scores);                                      // scores, at 0
    pl.off_gmax = take(pl.slice * per_unit_max);
  }
  if (pl.splits > 1) {
    pl.off_part = take((size_t)pl.slice * pl.splits * RT * a->D * 4);
    pl.off_ml = take((size_t)pl.slice * pl.splits * RT * 8);
  }
  pl.bytes = used;
  pl.use = true;
  return pl;
}

template <int D, int NT>
int run_fused(const Plan& pl, const DParams& p, cudaStream_t stream) {
  using F = FusedCfg<D, NT>;
  static std::atomic<bool> attr_done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return set_error(INTFA_ERR_CUDA, "cannot query the current device");
  if (!attr_done[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(fused_full_kernel<D, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, F::MAX_SCORES);
    if (e != cudaSuccess) return set_error(INTFA_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_done[dev].store(true, std::memory_order_release);
  }
  return launch_clusters("decode", fused_full_kernel<D, NT>, pl.units * pl.splits, pl.splits, kThreads, F::smem_bytes(pl.per_split * p.G), stream, p);
}
template <int D, int NT>
int run_slice(const Plan& pl, int units, const DParams& p, cudaStream_t stream) {
  int rc;
  const int grid = units * pl.splits;
  if (pl.full) {
    if ((rc = launch_kernel("decode scores", scores_kernel<D, NT>, units * pl.score_splits, kThreads, 0, stream, p, pl.score_splits))) return rc;
    if ((rc = launch_kernel("decode P V", pv_full_kernel<D, NT>, grid, kThreads, 0, stream, p))) return rc;
  } else {
    if ((rc = launch_kernel("decode", pv_half_kernel<D, NT>, grid, kThreads, 0, stream, p))) return rc;
  }
  if (pl.splits == 1) return INTFA_OK;
  const int rows = units * 8 * NT;
  auto combine = [&](auto few, auto many) {
    return pl.splits <= few_splits(pl.full) ? launch_kernel("decode combine", few, rows, D / 4, 0, stream, p, 8 * NT)
                                   : launch_kernel("decode combine", many, rows, combine_threads(D, pl.splits), 0, stream, p, 8 * NT);
  };
  return pl.full ? combine(combine_kernel<true, D>, combine_many_kernel<true, D>) : combine(combine_kernel<false, D>, combine_many_kernel<false, D>);
}
// (Slices share scratch: each kernel waits for the one before it on the stream before it writes any.)
template <int D, int NT>
int run(const Plan& pl, DParams p, cudaStream_t stream) {
  if (pl.fused) {
    p.unit0 = 0;
    return run_fused<D, NT>(pl, p, stream);
  }
  for (p.unit0 = 0; p.unit0 < pl.units; p.unit0 += pl.slice)
    if (const int rc = run_slice<D, NT>(pl, pl.units - p.unit0 < pl.slice ? pl.units - p.unit0 : pl.slice, p, stream)) return rc;
  return INTFA_OK;
}

}  // namespace

size_t decode_workspace_bytes(const IntfaFwdParams* a) {
  const int sms = sm_count_cached();
  return make_plan(a, sms > 0 ? sms : 148).bytes;
}

bool decode_dispatch(const IntfaFwdParams* a, cudaStream_t stream, int* rc) {
  const int sms = sm_count_cached();
  if (sms <= 0) return false;
  const Plan pl = make_plan(a, sms);
  if (!pl.use || a->workspace_bytes < pl.bytes || (pl.bytes > 0 && !a->workspace)) return false;
  DParams p;
  p.q = static_cast<const int8_t*>(a->q); p.k = static_cast<const int8_t*>(a->k); p.v = a->v; p.o = a->o;
  p.qB = a->q_stride[0]; p.qH = a->q_stride[1]; p.qN = a->q_stride[2];
  p.kB = a->k_stride[0]; p.kH = a->k_stride[1]; p.kN = a->k_stride[2];
  p.vB = a->v_stride[0]; p.vH = a->v_stride[1]; p.vN = a->v_stride[2];
  p.oB = a->o_stride[0]; p.oH = a->o_stride[1]; p.oN = a->o_stride[2];
  p.qs = a->q_scale; p.ks = a->k_scale; p.vs = a->v_scale;
  p.qsB = a->qs_stride[0]; p.qsH = a->qs_stride[1]; p.ksB = a->ks_stride[0]; p.ksH = a->ks_stride[1];
  p.vsB = a->vs_stride[0]; p.vsH = a->vs_stride[1]; p.vsD = a->vs_stride[2];
  p.scale_f16 = a->scale_f16;
  p.o_bf16 = a->o_dtype == INTFA_OUT_BF16;
  p.causal = a->causal ? 1 : 0;
  p.H = a->H; p.Hkv = a->H_kv > 0 ? a->H_kv : a->H; p.ratio = p.H / p.Hkv; p.Nq = a->Nq;
  p.R = p.ratio * p.Nq; p.tiles = pl.tiles;
  p.nvis = pl.nvis;
  p.limit0 = a->q_offset - a->kv_offset;
  p.c = a->sm_scale * 1.44269504f;
  p.G = a->G; p.groups = pl.groups; p.splits = pl.splits; p.per_split = pl.per_split;
  p.lse = a->lse_out;
  char* ws = static_cast<char*>(a->workspace);
  p.scores = reinterpret_cast<float*>(ws);
  p.gmax = reinterpret_cast<float*>(ws + pl.off_gmax);
  p.part = reinterpret_cast<float*>(ws + pl.off_part);
  p.part_ml = reinterpret_cast<float*>(ws + pl.off_ml);
  *rc = a->D == 128 ? (pl.NT == 2 ? run<128, 2>(pl, p, stream) : run<128, 1>(pl, p, stream))
                    : (pl.NT == 2 ? run<64, 2>(pl, p, stream) : run<64, 1>(pl, p, stream));
  return true;
}

}  // namespace intfa
