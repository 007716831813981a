// Green's function, overlap and 16-bit operands of the mixed-precision path, one CTA per walker
// (wavefunctions.py:478-501 rhf, 658-692 uhf).

#include "afq_common.cuh"
#include "afq_kernels.cuh"
#include "afq_launch.cuh"
#include "afq_mixed_dev.cuh"
#include "afq_prof.cuh"

namespace afq {

// Threads per walker: with 256 every size measured slower (norb 60 / 512 walkers 32.7 us instead of
// 18.5, norb 198 / 256 walkers 107 instead of 88): the serial Gauss-Jordan holds the CTA's slots.
constexpr int kGreenThreads = 128;

// Row stride (complex elements) of the walker copy: a multiple of 4 columns rounded so that
// stride / 2 is odd (16-byte aligned rows; reads of one column of consecutive rows then hit
// each shared-memory bank at most twice per half warp).
__host__ __device__ constexpr int green_s_ld(int o) {
  return ((((o + 3) & ~3) >> 1) & 1) ? ((o + 3) & ~3) : ((o + 3) & ~3) + 2;
}

// Read once: keep it out of L1, which the trial and rot_h1 (shared by all walkers) need.
__device__ __forceinline__ float2 ld_once(const float2* p) {
  float2 v;
  asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// dst[(e / o) * ld + e % o] = src[e] for e < n * o, 8 loads in flight per thread, the row and
// column advanced incrementally (no division per element)
template <int NT>
__device__ __forceinline__ void copy_rows(float2* dst, const float2* __restrict__ src, int n, int o, int ld) {
  const int total = n * o, dq = NT / o, dr = NT - dq * o;
  int p = threadIdx.x / o, k = threadIdx.x - p * o;
  for (int base = threadIdx.x; base < total; base += 8 * NT) {
    float2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = base + u * NT;
      if (e < total) v[u] = ld_once(src + e);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = base + u * NT;
      if (e < total) dst[p * ld + k] = v[u];
      p += dq;
      k += dr;
      if (k >= o) {
        k -= o;
        ++p;
      }
    }
  }
}

// Shared memory: per slab the walker [n][ld] (G overwrites it row by row) and S / S^-1 [OM][OM + 1].
__host__ __device__ constexpr size_t green_slab_bytes(int n, int o) {
  return ((size_t)n * green_s_ld(o) * 8 + 15) & ~(size_t)15;
}
static size_t green_smem(const MixedDev& md, int om) {
  size_t b = 0;
  for (int s = 0; s < md.nslab; ++s) b += green_slab_bytes(md.n, md.o_slab[s]) + (size_t)om * (om + 1) * 8 + 16;
  return b;
}

// (x, y) scaled by a power of two, as 16-bit pairs hi = (x_hi, y_hi) and lo
__device__ __forceinline__ void split16_pair(float x, float y, bool bf, uint32_t& hi, uint32_t& lo) {
  if (bf) {
    uint16_t hx, lx, hy, ly;
    split16(x, true, hx, lx);
    split16(y, true, hy, ly);
    hi = (uint32_t)hx | ((uint32_t)hy << 16);
    lo = (uint32_t)lx | ((uint32_t)ly << 16);
  } else {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  }
}

// The order of every sum below is part of the mixed path's results: resampling compares sums of weights
// with the comb's teeth, and a weight that moves by one FP32 rounding exchanges a whole walker wherever a tooth
// lies that close to a boundary. (With the orbitals of S dealt to several threads, populations of 2048 walkers on 64 sites
// came out with another walker on one of twelve inputs.) So an element of S sums the orbitals in their order, the
// elimination divides the pivot row before the other rows take their multiples of it, and a thread sums
// the one-body energy of an orbital; the roundings are spelled out (mul_rn).
//
// What bounds it: instruction issue and latency, not arithmetic (0.35 M FP32 FMAs per walker at
// norb 120, 20 electrons, are 2.8 k of an SM's cycles). The phases:
//  * S = C^T W in register blocks of RI x CK elements, sized so that one pass takes most of the threads;
//  * Gauss-Jordan by one warp per slab with a matrix row per lane (two rows above 32) in
//    registers. Partial pivoting is implicit: no rows move, the pivot of step j is the unused
//    row with the largest |re| + |im| in column j (ties to the lower row; its index rides in the
//    low bits of the key). The columns rotate by one register each step, so that the pivot
//    column is always register 0 and one step's code serves all; the pivot lane publishes its
//    row through shared memory, where a lane per element multiplies it by 1 / pivot. S is padded to OM with an
//    identity block. The working matrix ends as P^T S^-1 P^T for the pivot order P: row r is row step(r) of S^-1,
//    column c its column piv(c); det(S) = sign(P) prod(pivots), the product in FP64.
//    (A thread block per matrix with a barrier per pivot took 1200 cycles a step where five
//    walkers shared an SM.)
//  * G = (W S^-1)^T: a walker row per thread in registers, G written over it;
//  * the power-of-two scale of G, its 16-bit operands (two orbitals per store) and
//    ene1 = sum G * rot_h1.
// Against the kernel with a block-wide elimination, the same bits: 64 x 28 electrons, 2048 walkers 190 -> 130 us;
// 198 x 33, 256 walkers 208 -> 70 us; 60 x 10 and 60 x 8, 512 walkers 27 -> 18 us; 120 x 20, 1024 walkers
// 76 -> 61 us. (Sums in any order: 111, 64, 18, 48 us.)
template <int OM, int NT>
__global__ void __launch_bounds__(NT, (OM <= 24 ? 640 : OM <= 32 ? 512 : 256) / NT)
    k_green_mixed(const MixedDev md, const float2* __restrict__ wu, const float2* __restrict__ wd,
                  double2* __restrict__ ovl, int flags) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr int NW = NT / 32, RR = OM > 32 ? 2 : 1;
  constexpr unsigned RM = RR == 1 ? 31u : 63u;  // row index in the low bits of the pivot key
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = md.n;
  const bool do_g = (flags & kGreenG) != 0, bf = md.bf16 != 0;
  unsigned char* at = sm;
  float2* Wsl[2];
  float2* Sm[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    Wsl[s] = reinterpret_cast<float2*>(at);
    if (s < md.nslab) at += green_slab_bytes(n, md.o_slab[s]);
    Sm[s] = reinterpret_cast<float2*>(at);
    if (s < md.nslab) at += (size_t)OM * (OM + 1) * 8 + ((OM * (OM + 1)) & 1 ? 8 : 0);
  }
  __shared__ __align__(16) float2 prow[2][2][OM];  // [slab][step parity]: the pivot row
  __shared__ float2 pivv[2][OM];
  __shared__ int piv_s[2][OM];
  __shared__ int odd_s[2];
  __shared__ float2 e1w[NW], e1l[NW];
  __shared__ float fred[NW];

  for (int s = 0; s < md.nslab; ++s) {
    const int o = md.o_slab[s], o4 = (o + 3) & ~3, ld = green_s_ld(o);
    if (o4 != o)
      for (int pp = tid; pp < n; pp += NT)
        for (int k = o; k < o4; ++k) Wsl[s][pp * ld + k] = make_float2(0.f, 0.f);
    copy_rows<NT>(Wsl[s], (s == 0 ? wu : wd) + (size_t)w * n * o, n, o, ld);
  }
  __syncthreads();
  if (flags & kGreenWT) {  // walker operand of the exp_h1 products: row (w, 2k + c), column p
    for (int s = 0; s < md.nslab; ++s) {
      const int o = md.o_slab[s], ld = green_s_ld(o);
      uint16_t* hi = md.wt[s][0] + (size_t)w * md.R[s] * md.nk;
      uint16_t* lo = md.wt[s][1] + (size_t)w * md.R[s] * md.nk;
      for (int k = warp; k < o; k += NW)
        for (int p = 2 * lane; p < n; p += 64) {  // column n of an odd n is padding and stays zero
          const float2 a = Wsl[s][p * ld + k], b = p + 1 < n ? Wsl[s][(p + 1) * ld + k] : make_float2(0.f, 0.f);
          uint32_t h, l;
          split16_pair(a.x, b.x, bf, h, l);
          *reinterpret_cast<uint32_t*>(hi + (size_t)(2 * k) * md.nk + p) = h;
          *reinterpret_cast<uint32_t*>(lo + (size_t)(2 * k) * md.nk + p) = l;
          split16_pair(a.y, b.y, bf, h, l);
          *reinterpret_cast<uint32_t*>(hi + (size_t)(2 * k + 1) * md.nk + p) = h;
          *reinterpret_cast<uint32_t*>(lo + (size_t)(2 * k + 1) * md.nk + p) = l;
        }
    }
  }
  // S: blocks of RI trial columns x CK walker columns, an element's sum over the orbitals in their order
  constexpr int CK = OM <= 8 ? 1 : OM <= 20 ? 2 : 4, RI = OM <= 16 ? 1 : OM <= 32 ? 2 : 4;
  for (int s = 0; s < md.nslab; ++s) {
    const int o = md.o_slab[s], o4 = (o + 3) & ~3, ld = green_s_ld(o), nk = (o + CK - 1) / CK, ni = (o + RI - 1) / RI;
    for (int e = tid; e < ni * nk; e += NT) {
      const int bi = e / nk, i0 = bi * RI, k0 = (e - bi * nk) * CK;
      const float* __restrict__ C = md.trial32[s] + i0;  // [n][o4], the same for every walker (L1); columns o.. are zero
      auto load = [&](float (&c)[RI], const float* src) {
        if constexpr (RI == 1) {
          c[0] = __ldg(src);
        } else if constexpr (RI == 2) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(src));
          c[0] = v.x;
          c[1] = v.y;
        } else {
          const float4 v = __ldg(reinterpret_cast<const float4*>(src));
          c[0] = v.x;
          c[1] = v.y;
          c[2] = v.z;
          c[3] = v.w;
        }
      };
      const float2* W = Wsl[s] + k0;
      float2 acc[RI][CK];
#pragma unroll
      for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int k = 0; k < CK; ++k) acc[i][k] = make_float2(0.f, 0.f);
      auto row = [&](const float (&c)[RI], const float2* wp) {
        float2 wv[CK];
        if constexpr (CK >= 2) {
#pragma unroll
          for (int k = 0; k < CK; k += 2) {
            const float4 x = *reinterpret_cast<const float4*>(wp + k);
            wv[k] = make_float2(x.x, x.y);
            wv[k + 1] = make_float2(x.z, x.w);
          }
        } else {
          wv[0] = wp[0];
        }
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
          for (int k = 0; k < CK; ++k) {
            acc[i][k].x = fmaf(c[i], wv[k].x, acc[i][k].x);
            acc[i][k].y = fmaf(c[i], wv[k].y, acc[i][k].y);
          }
      };
      constexpr int U = 8;  // the trial rows of a batch in flight together
      int p = 0;
      for (; p + U <= n; p += U) {
        float c[U][RI];
#pragma unroll
        for (int u = 0; u < U; ++u) load(c[u], C + (p + u) * o4);
#pragma unroll
        for (int u = 0; u < U; ++u) row(c[u], W + (p + u) * ld);
      }
      for (; p < n; ++p) {
        float c[RI];
        load(c, C + p * o4);
        row(c, W + p * ld);
      }
#pragma unroll
      for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int k = 0; k < CK; ++k)
          if (i0 + i < o && k0 + k < o) Sm[s][(i0 + i) * (OM + 1) + k0 + k] = acc[i][k];
    }
    for (int e = tid; e < OM * OM; e += NT) {  // identity beyond the electrons
      const int i = e / OM, k = e - i * OM;
      if (i >= o || k >= o) Sm[s][i * (OM + 1) + k] = make_float2(i == k ? 1.f : 0.f, 0.f);
    }
  }
  __syncthreads();

  if (warp < md.nslab) {
    const int s = warp, o = md.o_slab[s];
    float2 a[RR][OM];
    bool used[RR];
    int step[RR];
#pragma unroll
    for (int rr = 0; rr < RR; ++rr) {
      const int row = lane + 32 * rr;
      used[rr] = row >= o;
      step[rr] = 0;
#pragma unroll
      for (int k = 0; k < OM; ++k) a[rr][k] = row < OM ? Sm[s][row * (OM + 1) + k] : make_float2(0.f, 0.f);
    }
    unsigned long long open = (1ull << o) - 1ull;  // rows without a pivot
    int odd = 0;
#pragma unroll 1
    for (int j = 0; j < o; ++j) {  // column c ends in register OM - o + c
      float2* pw = prow[s][j & 1];
      unsigned key = 0u;
#pragma unroll
      for (int rr = 0; rr < RR; ++rr) {
        const float mag = fabsf(a[rr][0].x) + fabsf(a[rr][0].y);
        const unsigned kc = used[rr] ? 0u : ((__float_as_uint(mag) & ~RM) | (RM - (unsigned)(lane + 32 * rr)));
        key = max(key, kc);
      }
      const int pr = (int)(RM - (__reduce_max_sync(0xffffffffu, key) & RM));
      // every row's own 1 / a0 while the reduction runs: conj(a0) / |a0|^2, scaled by a power of
      // two near 1 / |a0| (no overflow)
      float2 rin[RR];
#pragma unroll
      for (int rr = 0; rr < RR; ++rr) {
        const float m = fmaxf(fabsf(a[rr][0].x), fabsf(a[rr][0].y));
        const int ef = min(max((int)(__float_as_uint(m) >> 23), 1), 253);
        const float sc = __uint_as_float((unsigned)(254 - ef) << 23);
        const float px = a[rr][0].x * sc, py = a[rr][0].y * sc;
        const float dd = __frcp_rn(fmaf(px, px, __fmul_rn(py, py))) * sc;
        rin[rr] = make_float2(px * dd, -py * dd);
      }
      bool own[RR];
#pragma unroll
      for (int rr = 0; rr < RR; ++rr) {
        own[rr] = lane + 32 * rr == pr;
        if (own[rr]) {
          used[rr] = true;
          step[rr] = j;
          pivv[s][j] = a[rr][0];
          piv_s[s][j] = pr;
          pw[0] = rin[rr];
          pw[1] = a[rr][1];
#pragma unroll
          for (int k = 2; k < OM; k += 2)
            *reinterpret_cast<float4*>(pw + k) = make_float4(a[rr][k].x, a[rr][k].y, a[rr][k + 1].x, a[rr][k + 1].y);
          a[rr][0] = make_float2(-1.f, 0.f);  // 0 - (-1) (row / pv) is the pivot row's new value
#pragma unroll
          for (int k = 1; k < OM; ++k) a[rr][k] = make_float2(0.f, 0.f);
        }
      }
      __syncwarp();
      const float2 inv = pw[0];
      float2 sp[RR];  // the pivot row over the pivot, an element per lane
#pragma unroll
      for (int rr = 0; rr < RR; ++rr)
        if (lane + 32 * rr < OM) sp[rr] = mul_rn(pw[lane + 32 * rr], inv);
      __syncwarp();
#pragma unroll
      for (int rr = 0; rr < RR; ++rr)
        if (lane + 32 * rr < OM && lane + 32 * rr > 0) pw[lane + 32 * rr] = sp[rr];
      __syncwarp();
      float2 f[RR];
#pragma unroll
      for (int rr = 0; rr < RR; ++rr) f[rr] = a[rr][0];
#pragma unroll
      for (int k = 0; k < OM; k += 2) {
        const float4 v = *reinterpret_cast<const float4*>(pw + k);
#pragma unroll
        for (int rr = 0; rr < RR; ++rr) {
          if (k > 0) a[rr][k - 1] = sub_rn(a[rr][k], mul_rn(f[rr], make_float2(v.x, v.y)));
          a[rr][k] = sub_rn(a[rr][k + 1], mul_rn(f[rr], make_float2(v.z, v.w)));
        }
      }
#pragma unroll
      for (int rr = 0; rr < RR; ++rr) a[rr][OM - 1] = sub_rn(make_float2(0.f, 0.f), mul_rn(f[rr], inv));
      odd += __popcll(open & ((1ull << pr) - 1ull));  // later pivots in lower rows
      open &= ~(1ull << pr);
    }
    __syncwarp();
    if (lane == 0) odd_s[s] = odd;
    if (do_g) {  // S^-1 [k][i], row stride OM, over S
#pragma unroll
      for (int rr = 0; rr < RR; ++rr)
        if (lane + 32 * rr < OM) {
#pragma unroll
          for (int k = 0; k < OM; ++k) {
            if (lane + 32 * rr >= o) Sm[s][(lane + 32 * rr) * OM + k] = make_float2(0.f, 0.f);
            else if (k >= OM - o) Sm[s][step[rr] * OM + piv_s[s][k - (OM - o)]] = a[rr][k];
          }
        }
    }
  }
  __syncthreads();
  if (warp == NW - 1) {  // det: FP64 product of the pivots (a shuffle tree), while the others form G
    double2 det = c2(1.0, 0.0);
    for (int s = 0; s < md.nslab; ++s) {
      double2 pd = c2(1.0, 0.0);
#pragma unroll
      for (int rr = 0; rr < RR; ++rr)
        if (lane + 32 * rr < md.o_slab[s])
          pd = cmul(pd, c2((double)pivv[s][lane + 32 * rr].x, (double)pivv[s][lane + 32 * rr].y));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        pd = cmul(pd, c2(__shfl_xor_sync(0xffffffffu, pd.x, off), __shfl_xor_sync(0xffffffffu, pd.y, off)));
      det = cmul(det, (odd_s[s] & 1) ? c2(-pd.x, -pd.y) : pd);
    }
    if (lane == 0 && ovl) ovl[w] = md.restricted_square ? cmul(det, det) : det;
  }
  if (!do_g) return;

  float mx = 0.f;
  for (int s = 0; s < md.nslab; ++s) {
    const int o = md.o_slab[s], ld = green_s_ld(o);
    const bool sum = md.nblk == 1 && s == 1;  // RHF two slabs: G = G_up + G_dn, in slab 0
    for (int p = tid; p < n; p += NT) {
      float2* row = Wsl[s] + p * ld;
      float2 wr[OM];
#pragma unroll
      for (int k = 0; k < OM; k += 2) {
        const float4 v = k < o ? *reinterpret_cast<const float4*>(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        wr[k] = make_float2(v.x, v.y);
        wr[k + 1] = make_float2(v.z, v.w);
      }
      // four columns i at a time: independent accumulation chains, 16-byte reads of S^-1
#pragma unroll 1
      for (int i0 = 0; i0 < o; i0 += 4) {
        float2 g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) g[u] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < OM; ++k) {
          const float4 s01 = *reinterpret_cast<const float4*>(&Sm[s][k * OM + i0]);
          const float4 s23 = *reinterpret_cast<const float4*>(&Sm[s][k * OM + i0 + 2]);
          g[0] = add_rn(g[0], mul_rn(wr[k], make_float2(s01.x, s01.y)));
          g[1] = add_rn(g[1], mul_rn(wr[k], make_float2(s01.z, s01.w)));
          g[2] = add_rn(g[2], mul_rn(wr[k], make_float2(s23.x, s23.y)));
          g[3] = add_rn(g[3], mul_rn(wr[k], make_float2(s23.z, s23.w)));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 + u < o) {
            float2* dst = (sum ? Wsl[0] + p * ld : row) + i0 + u;
            if (sum) g[u] = add_rn(g[u], *dst);
            *dst = g[u];
            if (md.nblk == 2 || s + 1 == md.nslab) mx = fmaxf(mx, fmaxf(fabsf(g[u].x), fabsf(g[u].y)));
          }
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if (lane == 0) fred[warp] = mx;
  __syncthreads();
  float mall = fred[0];
#pragma unroll
  for (int q = 1; q < NW; ++q) mall = fmaxf(mall, fred[q]);
  const float scl = pow2_scale(mall);
  if (tid == 0) md.g_inv[w] = 1.0f / scl;

  const int gtot = md.o_blk[0] + md.o_blk[1];
  float e1x = 0.f, e1y = 0.f;  // per-thread partials of <= 64 terms, an orbital a thread; FP64 across warps
  for (int p = tid; p < n; p += NT)
    for (int b = 0; b < md.nblk; ++b) {
      const int o = md.o_blk[b];
      const float2* G = Wsl[b] + p * green_s_ld(md.o_slab[b]);
      const float* __restrict__ rh = md.rh1_32[b] + p;
#pragma unroll 4
      for (int i = 0; i < o; ++i) {
        const float2 g = G[i];
        const float r1 = __ldg(rh + (size_t)i * n);
        e1x = fmaf(g.x, r1, e1x);
        e1y = fmaf(g.y, r1, e1y);
      }
    }
  const bool even = (n & 1) == 0;
  for (int ii = warp; ii < gtot; ii += NW) {
    const int b = (md.nblk == 2 && ii >= md.o_blk[0]) ? 1 : 0, i = ii - b * md.o_blk[0];
    const int ld = green_s_ld(md.o_slab[b]);
    const float2* G = Wsl[b] + i;
    uint16_t* fh[2] = {md.g_fb[0] + (size_t)(2 * w) * md.ldfb + (size_t)ii * n,
                       md.g_fb[1] + (size_t)(2 * w) * md.ldfb + (size_t)ii * n};
    uint16_t* kh[2] = {nullptr, nullptr};  // per-block operand (exchange / Coulomb of each spin separately)
    if (md.nblk == 2)
      for (int q = 0; q < 2; ++q) kh[q] = md.g_blk[b][q] + (size_t)(2 * w) * md.ldkb[b] + (size_t)i * n;
    if (even) {
      float2 g0[4], g1[4];  // n <= 256
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int p = 2 * lane + 64 * u;
        if (p < n) {
          g0[u] = G[p * ld];
          g1[u] = G[(p + 1) * ld];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int p = 2 * lane + 64 * u;
        if (p >= n) break;
        uint32_t rhi, rlo, ihi, ilo;
        split16_pair(g0[u].x * scl, g1[u].x * scl, bf, rhi, rlo);
        split16_pair(g0[u].y * scl, g1[u].y * scl, bf, ihi, ilo);
        *reinterpret_cast<uint32_t*>(fh[0] + p) = rhi;
        *reinterpret_cast<uint32_t*>(fh[1] + p) = rlo;
        *reinterpret_cast<uint32_t*>(fh[0] + md.ldfb + p) = ihi;
        *reinterpret_cast<uint32_t*>(fh[1] + md.ldfb + p) = ilo;
        if (md.nblk == 2) {
          *reinterpret_cast<uint32_t*>(kh[0] + p) = rhi;
          *reinterpret_cast<uint32_t*>(kh[1] + p) = rlo;
          *reinterpret_cast<uint32_t*>(kh[0] + md.ldkb[b] + p) = ihi;
          *reinterpret_cast<uint32_t*>(kh[1] + md.ldkb[b] + p) = ilo;
        }
      }
    } else {  // rows of the operands start at odd elements
      for (int p = lane; p < n; p += 32) {
        const float2 g = G[p * ld];
        uint16_t hr, lr, hi, li;
        split16(g.x * scl, bf, hr, lr);
        split16(g.y * scl, bf, hi, li);
        fh[0][p] = hr;
        fh[1][p] = lr;
        fh[0][md.ldfb + p] = hi;
        fh[1][md.ldfb + p] = li;
        if (md.nblk == 2) {
          kh[0][p] = hr;
          kh[1][p] = lr;
          kh[0][md.ldkb[b] + p] = hi;
          kh[1][md.ldkb[b] + p] = li;
        }
      }
    }
  }
  // warp sums as unevaluated float pairs (hi + lo, Knuth's TwoSum at every level)
  float lx = 0.f, ly = 0.f;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float ox = __shfl_xor_sync(0xffffffffu, e1x, off), oy = __shfl_xor_sync(0xffffffffu, e1y, off);
    const float olx = __shfl_xor_sync(0xffffffffu, lx, off), oly = __shfl_xor_sync(0xffffffffu, ly, off);
    float sx = e1x + ox, bx = sx - e1x;
    lx += olx + ((e1x - (sx - bx)) + (ox - bx));
    e1x = sx;
    float sy = e1y + oy, by = sy - e1y;
    ly += oly + ((e1y - (sy - by)) + (oy - by));
    e1y = sy;
  }
  if (lane == 0) {
    e1w[warp] = make_float2(e1x, e1y);
    e1l[warp] = make_float2(lx, ly);
  }
  __syncthreads();
  if (tid == 0) {
    double2 t = c2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < NW; ++q)
      t = c2(t.x + ((double)e1w[q].x + (double)e1l[q].x), t.y + ((double)e1w[q].y + (double)e1l[q].y));
    md.ene1[w] = t;
  }
}

template <int OM>
static int green_launch(const MixedDev& md, const float2* wu, const float2* wd, double2* ovl, int flags,
                        cudaStream_t st) {
  constexpr int NT = kGreenThreads;
  const size_t smem = green_smem(md, OM);
  if (int rc = check_smem_optin(smem + sizeof(float2) * 6 * OM + 1024,
                                "mixed Green's-function kernel (norb x electrons too large for one CTA)"))
    return rc;
  auto kfn = k_green_mixed<OM, NT>;
  // a refused attribute surfaces as the launch error checked by the caller
  raise_smem_limit((const void*)kfn, smem);
  launch_pdl(kfn, md.nw, NT, smem, st, md, wu, wd, ovl, flags);
  return 0;
}

int launch_green_mixed(const MixedDev& md, const float2* wu, const float2* wd, double2* ovl, int flags,
                       cudaStream_t st) {
  const int omax = md.o_slab[0] > md.o_slab[1] ? md.o_slab[0] : md.o_slab[1];
  ProfScope _ps(K_GREEN, st);
  switch ((omax + 3) / 4) {
    case 0:
    case 1: return green_launch<4>(md, wu, wd, ovl, flags, st);
    case 2: return green_launch<8>(md, wu, wd, ovl, flags, st);
    case 3: return green_launch<12>(md, wu, wd, ovl, flags, st);
    case 4: return green_launch<16>(md, wu, wd, ovl, flags, st);
    case 5: return green_launch<20>(md, wu, wd, ovl, flags, st);
    case 6: return green_launch<24>(md, wu, wd, ovl, flags, st);
    case 7: return green_launch<28>(md, wu, wd, ovl, flags, st);
    case 8: return green_launch<32>(md, wu, wd, ovl, flags, st);
    case 9: return green_launch<36>(md, wu, wd, ovl, flags, st);
    default: return green_launch<40>(md, wu, wd, ovl, flags, st);
  }
}

}  // namespace afq
