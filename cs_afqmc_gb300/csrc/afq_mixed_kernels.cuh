// Device code of the mixed-precision path: GEMM epilogues (fused field
// shifts, vhs scatter into the Taylor layout, exp_h1 products, exchange/Coulomb energy),
// the per-walker tcgen05 Taylor kernel, and one-time operand preparation.
#pragma once
#include "afq_mixed_dev.cuh"

namespace afq {

constexpr int kGreenMaxO = 40;  // occupied orbitals per slab (S is at most 40 x 40)

// dst[map(e)] = src[e] for e < n by a block of NT threads, 8 independent loads in flight per
// thread before the shared-memory stores (the copies are latency-bound otherwise)
template <int NT, class T, class Map>
__device__ __forceinline__ void copy_batched(T* dst, const T* __restrict__ src, int n, Map map) {
  for (int base = threadIdx.x; base < n; base += 8 * NT) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = base + u * NT;
      if (e < n) v[u] = src[e];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = base + u * NT;
      if (e < n) dst[map(e)] = v[u];
    }
  }
}

// ======================================================================================
// Force-bias GEMM epilogue: rows (w, re/im) of fb = alpha * G . rot_chol^T, fused with the
// field shifts of propagation.py:121-127 (writes the shifted-field operand and per-tile
// partial sums of shift_term and fb_term), or, for calc_force_bias, the plain force bias.
// ======================================================================================

struct EpiFB {
  struct Params {
    const double* fields;
    const double2* mf;
    const float* rc_inv;
    const float* g_inv;
    float alpha, sqdt;
    int nw, nchol, ldg, ntiles, bf16;
    uint16_t* xt_hi;
    uint16_t* xt_lo;
    double2* part_shift;
    double2* part_fbt;
    double2* fb_out;  // non-null: write the force bias instead
  };
  static constexpr int kSmemBytes = 0;
  __device__ static void run(const Params& p, int m0, int n0, int bn, uint32_t tmem, int q, int lane,
                             unsigned char*, bool) {
    const int R = m0 + q * 32 + lane, w = R >> 1, c = R & 1;
    const bool valid = w < p.nw;
    const float gi = valid ? p.g_inv[w] : 0.f;
    const bool bf = p.bf16 != 0;
    float shx = 0.f, shy = 0.f, fbx = 0.f, fby = 0.f;
#pragma unroll 1
    for (int c0 = 0; c0 < bn; c0 += 16) {
      float v[16];
      ptx::tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + c0, v);
      ptx::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int g = n0 + c0 + j;
        const bool gv = g < p.nchol;
        const float val = v[j] * p.alpha * gi * (gv ? p.rc_inv[g] : 0.f);
        const float other = __shfl_xor_sync(0xffffffffu, val, 1);
        if (!valid || !gv) continue;
        const float fr = c ? other : val, fi = c ? val : other;
        if (p.fb_out) {
          if (c == 0) p.fb_out[(size_t)w * p.nchol + g] = c2(fr, fi);
          continue;
        }
        const double2 mfd = p.mf[g];
        const float mfr = (float)mfd.x, mfi = (float)mfd.y;
        const float sr = -p.sqdt * (-fi - mfr), si = -p.sqdt * (fr - mfi);
        const float x = (float)p.fields[(size_t)w * p.nchol + g];
        const float xtr = x - sr, xti = -si;
        uint16_t h, l;
        split16(c ? xti : xtr, bf, h, l);
        p.xt_hi[(size_t)R * p.ldg + g] = h;
        p.xt_lo[(size_t)R * p.ldg + g] = l;
        if (c == 0) {
          shx += xtr * mfr - xti * mfi;
          shy += xtr * mfi + xti * mfr;
          fbx += x * sr - 0.5f * (sr * sr - si * si);
          fby += x * si - sr * si;
        }
      }
    }
    if (valid && c == 0 && !p.fb_out) {
      p.part_shift[(size_t)w * p.ntiles + blockIdx.x] = c2(shx, shy);
      p.part_fbt[(size_t)w * p.ntiles + blockIdx.x] = c2(fbx, fby);
    }
  }
};

// Force bias from the K-split partials of fb = G . rot_chol^T (rows (w, re/im)), one CTA
// per walker: sums the partials in split order, then the same scaling, field shifts and
// shift_term / fb_term sums as EpiFB (propagation.py:121-127), the sums reduced over all
// Cholesky vectors (part_shift / part_fbt hold one entry per walker).
struct FbReduce {
  const float* part;  // [ksplit][2 nw][ldp]
  int ksplit, nw, nchol, ldg, bf16;
  long ldp, sst;
  const double* fields;
  const double2* mf;
  const float* rc_inv;
  const float* g_inv;
  float alpha, sqdt;
  uint16_t* xt_hi;
  uint16_t* xt_lo;
  double2* part_shift;  // [nw]
  double2* part_fbt;    // [nw]
  double2* fb_out;      // non-null: write the force bias instead
};

__global__ void __launch_bounds__(256, 3) k_fb_reduce(const FbReduce r) {
  __shared__ double red[32];
  pdl_enter();
  const int w = blockIdx.x;
  const float gi = r.g_inv[w];
  const bool bf = r.bf16 != 0;
  float shx = 0.f, shy = 0.f, fbx = 0.f, fby = 0.f;
  const float* pr = r.part + (long)(2 * w) * r.ldp;
  const float* pi = pr + r.ldp;
  // four Cholesky indices per thread at a time, all loads issued before any store (the
  // 16-bit stores may alias the loads for the compiler)
  for (int g0 = threadIdx.x; g0 < r.nchol; g0 += 4 * blockDim.x) {
    float ar[4], ai[4], rc[4], xv[4];
    double2 mfv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int g = g0 + u * blockDim.x;
      ar[u] = ai[u] = rc[u] = xv[u] = 0.f;
      mfv[u] = c2(0.0, 0.0);
      if (g < r.nchol) {
        for (int ks = 0; ks < r.ksplit; ++ks) {
          ar[u] += pr[(long)ks * r.sst + g];
          ai[u] += pi[(long)ks * r.sst + g];
        }
        rc[u] = r.rc_inv[g];
        if (!r.fb_out) {
          xv[u] = (float)r.fields[(size_t)w * r.nchol + g];
          mfv[u] = r.mf[g];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int g = g0 + u * blockDim.x;
      if (g >= r.nchol) continue;
      const float fr = ar[u] * r.alpha * gi * rc[u], fi = ai[u] * r.alpha * gi * rc[u];
      if (r.fb_out) {
        r.fb_out[(size_t)w * r.nchol + g] = c2(fr, fi);
        continue;
      }
      const float mfr = (float)mfv[u].x, mfi = (float)mfv[u].y;
      const float sr = -r.sqdt * (-fi - mfr), si = -r.sqdt * (fr - mfi);
      const float x = xv[u];
      const float xtr = x - sr, xti = -si;
      uint16_t h, l;
      split16(xtr, bf, h, l);
      r.xt_hi[(size_t)(2 * w) * r.ldg + g] = h;
      r.xt_lo[(size_t)(2 * w) * r.ldg + g] = l;
      split16(xti, bf, h, l);
      r.xt_hi[(size_t)(2 * w + 1) * r.ldg + g] = h;
      r.xt_lo[(size_t)(2 * w + 1) * r.ldg + g] = l;
      shx += xtr * mfr - xti * mfi;
      shy += xtr * mfi + xti * mfr;
      fbx += x * sr - 0.5f * (sr * sr - si * si);
      fby += x * si - sr * si;
    }
  }
  if (r.fb_out) return;
  // the four sums reduced together: warp shuffles on unevaluated float pairs (hi + lo,
  // Knuth's TwoSum at every level: no FP64 on the shuffle path), then one FP64 pass over the
  // warps in shared memory
  float v[4] = {shx, shy, fbx, fby}, vl[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float o = __shfl_xor_sync(0xffffffffu, v[j], off), ol = __shfl_xor_sync(0xffffffffu, vl[j], off);
      const float sum = v[j] + o, bb = sum - v[j];
      vl[j] += ol + ((v[j] - (sum - bb)) + (o - bb));
      v[j] = sum;
    }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < 4; ++j) red[4 * wid + j] = (double)v[j] + (double)vl[j];
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int i = 0; i < nwarp; ++i) t += red[4 * i + threadIdx.x];
    red[threadIdx.x] = t;  // each thread wrote only its own slot of warp 0's row
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    r.part_shift[w] = c2(red[0], red[1]);
    r.part_fbt[w] = c2(red[2], red[3]);
  }
}

// ======================================================================================
// vhs GEMM epilogue (propagation.py:265-271): rows (w, re/im) of xt . chol give
// V = i sqrt(dt) xt . chol = sqrt(dt) (-(xt_i.L) + i (xt_r.L)); write the Taylor A operand
// [Vr | Vi] (hi and lo) for each walker of the chunk. Columns are (p, q) with q padded to nq.
// ======================================================================================

struct EpiVHS {
  struct Params {
    uint16_t* v_hi;
    uint16_t* v_lo;
    int n, nq, rows, bf16, want_lo;
    float sqdt;
    int sym;  // split GEMM only: columns are the packed (p, q) pairs of sym_decode
    int mr;   // rows per walker of the V operand (128, or 256 for norb > 128)
  };
  static constexpr int kSmemBytes = 0;
  __device__ static void run(const Params& p, int m0, int n0, int bn, uint32_t tmem, int q, int lane,
                             unsigned char*, bool) {
    const int R = m0 + q * 32 + lane, wl = R >> 1, c = R & 1;
    const bool bf = p.bf16 != 0;
    const float scale = c == 0 ? p.sqdt : -p.sqdt;
#pragma unroll 1
    for (int c0 = 0; c0 < bn; c0 += 16) {
      float v[16];
      ptx::tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + c0, v);
      ptx::tmem_ld_wait();
      const int col = n0 + c0, pr = col / p.nq, q0 = col % p.nq;
      if (R >= p.rows || pr >= p.n) continue;
      const size_t off = ((size_t)wl * p.mr + pr) * (2 * p.nq) + (c == 0 ? p.nq : 0) + q0;
      uint32_t hw[8], lw[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint16_t h0, l0, h1, l1;
        split16(v[2 * j] * scale, bf, h0, l0);
        split16(v[2 * j + 1] * scale, bf, h1, l1);
        hw[j] = (uint32_t)h0 | ((uint32_t)h1 << 16);
        lw[j] = (uint32_t)l0 | ((uint32_t)l1 << 16);
      }
      uint4* dh = reinterpret_cast<uint4*>(p.v_hi + off);
      dh[0] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
      dh[1] = make_uint4(hw[4], hw[5], hw[6], hw[7]);
      if (p.want_lo) {
        uint4* dl = reinterpret_cast<uint4*>(p.v_lo + off);
        dl[0] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        dl[1] = make_uint4(lw[4], lw[5], lw[6], lw[7]);
      }
    }
  }
};

// The same scatter for the persistent split GEMM: row R of the chunk, 128 columns from col0.
struct EpiVHSSplit {
  using Params = EpiVHS::Params;
  static constexpr bool kWarpStore = true;
  // Rows R0 + lane (walker R / 2, real (even R) or imaginary part) and 128 columns col0.. of
  // vhs, i.e. (orbital pr, q) pairs, into the Taylor operand V = [Vr | Vi] per walker. Per 32
  // columns each lane converts its row to fp16 hi / lo (two values per conversion
  // instruction) and stages one plane at a time in shared memory (80-byte rows), then four
  // lanes store each row's 64 contiguous bytes: a warp's stores cover 8 rows x 64 B instead of
  // 32 separate 16-byte pieces. A 32-column group never crosses a row run (runs are multiples
  // of 32 long and start at multiples of 32), so (pr, q0) is decoded once per tile and then
  // advanced.
  __device__ __forceinline__ static void store_warp(const Params& p, int R0, int lane, int col0, const float* v, int,
                                                    unsigned char* stage) {
    const int R = R0 + lane;
    const bool bf = p.bf16 != 0;
    const float scale = (R & 1) == 0 ? p.sqdt : -p.sqdt;
    int pr, q0;
    if (p.sym)
      sym_decode(p.n, p.nq, col0, pr, q0);
    else {
      pr = col0 / p.nq;
      q0 = col0 % p.nq;
    }
#pragma unroll
    for (int c32 = 0; c32 < 128; c32 += 32) {
      if (pr >= p.n) break;  // warp-uniform
      uint32_t hw[16], lw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a = v[c32 + 2 * j] * scale, b = v[c32 + 2 * j + 1] * scale;
        if (bf) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
          const float2 hf = __bfloat1622float2(h);
          const __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
          hw[j] = *reinterpret_cast<const uint32_t*>(&h);
          lw[j] = *reinterpret_cast<const uint32_t*>(&l);
        } else {
          const __half2 h = __floats2half2_rn(a, b);
          const float2 hf = __half22float2(h);
          const __half2 l = __floats2half2_rn(a - hf.x, b - hf.y);
          hw[j] = *reinterpret_cast<const uint32_t*>(&h);
          lw[j] = *reinterpret_cast<const uint32_t*>(&l);
        }
      }
#pragma unroll
      for (int plane = 0; plane < 2; ++plane) {
        if (plane == 1 && !p.want_lo) break;
        const uint32_t* src = plane ? lw : hw;
        uint4* srow = reinterpret_cast<uint4*>(stage + lane * kSplitStageRow);
#pragma unroll
        for (int u = 0; u < 4; ++u) srow[u] = make_uint4(src[4 * u], src[4 * u + 1], src[4 * u + 2], src[4 * u + 3]);
        __syncwarp();
        uint16_t* base = plane ? p.v_lo : p.v_hi;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int t = lane + 32 * u, row = t >> 2, part = t & 3, Rr = R0 + row;
          if (Rr < p.rows) {
            const int wl = Rr >> 1, c = Rr & 1;
            const size_t off = ((size_t)wl * p.mr + pr) * (2 * p.nq) + (c == 0 ? p.nq : 0) + q0 + part * 8;
            *reinterpret_cast<uint4*>(base + off) =
                *reinterpret_cast<const uint4*>(stage + row * kSplitStageRow + part * 16);
          }
        }
        __syncwarp();
      }
      // next 32 columns: same row run, or the start of the next row's run
      q0 += 32;
      if (q0 >= p.nq) {
        ++pr;
        q0 = p.sym ? 32 * (pr >> 5) : 0;
      }
    }
  }
};

// vhs B operand for symmetric vectors: chol [nchol][n*n] -> lop[c][g] for the packed columns
// c = (p, q) of sym_decode, 32 x 32 tiles through shared memory
__global__ void k_prep_lop_sym(const double* __restrict__ chol, int nchol, int n, int nq, int total, int ldg,
                               int bf16, uint16_t* __restrict__ hi, uint16_t* __restrict__ lo) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, g0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  int pp = n, qq = 0;
  if (c0 + tx < total) sym_decode(n, nq, c0 + tx, pp, qq);
  for (int r = ty; r < 32; r += 8) {
    const int g = g0 + r;
    tile[r][tx] = (g < nchol && pp < n && qq < n) ? (float)chol[(size_t)g * n * n + (size_t)pp * n + qq] : 0.f;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int c = c0 + r, g = g0 + tx;
    if (c < total && g < nchol) {
      uint16_t h, l;
      split16(tile[tx][r], bf16 != 0, h, l);
      hi[(size_t)c * ldg + g] = h;
      lo[(size_t)c * ldg + g] = l;
    }
  }
}

// ======================================================================================
// exp_h1 products: D[p][(w, 2k + c)] = ((E - I) X)[p][k].c for the walker (X = W) or the
// Taylor sum (X = acc). First product: W1 = W + D into the Taylor B operand (hi/lo);
// last product: W_new = acc + D back into the FP32 walker slab. propagation.py:73, 91.
// ======================================================================================

struct EpiExp {
  struct Params {
    float* w;                 // walker slab [nw][n][o] complex64
    const uint16_t* acc_hi;   // last product: Taylor sum operand [nw*R][nk]
    const uint16_t* acc_lo;
    uint16_t* t0_hi;          // first product: Taylor B operand [nw][NT][2nq]
    uint16_t* t0_lo;
    int n, o, R, nk, nq, NT, nw, bf16, last;
  };
  static constexpr int kSmemBytes = 0;
  // Walker-major: R (a multiple of 16) columns per walker, so each walker is R/16 whole
  // TMEM chunks; thread p handles orbital row p of every walker of the tile.
  __device__ static void run(const Params& p, int m0, int n0, int bn, uint32_t tmem, int q, int lane,
                             unsigned char*, bool) {
    const int pr = m0 + q * 32 + lane;
    const bool bf = p.bf16 != 0;
    const int wpt = bn / p.R, w0 = n0 / p.R;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
#pragma unroll 1
    for (int wl = 0; wl < wpt; ++wl) {
      float v[64];
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 16) {
        if (c0 < p.R) {
          float t[16];
          ptx::tmem_ld16(tmem + lane_off + (uint32_t)(wl * p.R + c0), t);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[c0 + j] = t[j];
        }
      }
      ptx::tmem_ld_wait();
      const int w = w0 + wl;
      if (pr >= p.n || w >= p.nw) continue;
      float2* wrow = reinterpret_cast<float2*>(p.w) + ((size_t)w * p.n + pr) * p.o;
      // loads are issued 8 orbitals at a time before the stores of those orbitals (the stores
      // may alias the loads for the compiler, which would otherwise wait one load latency per k)
      if (p.last) {
        const size_t ab = (size_t)w * p.R * p.nk + pr;
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 8) {
          if (k0 < p.o) {
            uint16_t ah[16], al[16];
#pragma unroll
            for (int r = 0; r < 16; ++r)
              if (2 * k0 + r < 2 * p.o) {
                ah[r] = p.acc_hi[ab + (size_t)(2 * k0 + r) * p.nk];
                al[r] = p.acc_lo[ab + (size_t)(2 * k0 + r) * p.nk];
              }
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const int k = k0 + kk;
              if (k < p.o) {
                const float ar = h2f(ah[2 * kk], bf) + h2f(al[2 * kk], bf);
                const float ai = h2f(ah[2 * kk + 1], bf) + h2f(al[2 * kk + 1], bf);
                wrow[k] = make_float2(ar + v[2 * k], ai + v[2 * k + 1]);
              }
            }
          }
        }
      } else {
        const size_t base = (size_t)w * p.NT * 2 * p.nq;
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 8) {
          if (k0 < p.o) {
            float2 xw[8];
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              if (k0 + kk < p.o) xw[kk] = wrow[k0 + kk];
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const int k = k0 + kk;
              if (k < p.o) {
                const float wr = xw[kk].x + v[2 * k], wi = xw[kk].y + v[2 * k + 1];
                uint16_t hr, lr, hi_, li, hn, ln;
                split16(wr, bf, hr, lr);
                split16(wi, bf, hi_, li);
                split16(-wi, bf, hn, ln);
                const size_t r0 = base + (size_t)(2 * k) * 2 * p.nq, r1 = r0 + 2 * p.nq;
                // row 2k: [Tr | -Ti], row 2k+1: [Ti | Tr]
                p.t0_hi[r0 + pr] = hr;
                p.t0_lo[r0 + pr] = lr;
                p.t0_hi[r0 + p.nq + pr] = hn;
                p.t0_lo[r0 + p.nq + pr] = ln;
                p.t0_hi[r1 + pr] = hi_;
                p.t0_lo[r1 + pr] = li;
                p.t0_hi[r1 + p.nq + pr] = hr;
                p.t0_lo[r1 + p.nq + pr] = lr;
              }
            }
          }
        }
      }
    }
  }
};

// ======================================================================================
// Exchange epilogue of the split GEMM, on the transposed product D = G U (U symmetric):
// D[(w, re/im)][(i,q)] = Z_w[(i,q)] = sum_(k,p) U[(i,q),(k,p)] G_w[k,p] with
// U[(i,q),(k,p)] = sum_g rot_chol_g[i,p] rot_chol_g[k,q], so that the exchange sum of
// wavefunctions.py:539 (and 737-738), exc = sum_g sum_ik f_g[i,k] f_g[k,i] with
// f_g = rot_chol_g G^T, equals sum_(i,q) Z_w[(i,q)] G_w[i,q]. A thread holds row (w, part)
// of D over 128 consecutive (i,q): it reads the same 128 entries of G_w's re and im rows
// (contiguous 16-byte loads, hi + lo) and forms Z_part . G_re and Z_part . G_im; the
// neighbouring lane (the other part of the same walker) completes the complex product. The
// walker's partial of exc for these 128 columns and this K range goes, scaled, to slot
// ks * n128 + col0 / 128 of its row of partials: exc is linear in Z, so K-split partials
// need no separate reduction, and the final energy kernel sums the slots in a fixed order.
// ======================================================================================

struct EpiExcSplit {
  static constexpr bool kWarpStore = true;
  struct Params {
    const uint16_t* g_hi;  // [2 nw][ldk] Green operand (rows 2w, 2w+1 = re, im)
    const uint16_t* g_lo;
    const float* g_inv;    // [nw]
    float u_inv;
    int kb, ldk, nw, bf16;
    int n128, slots;       // 128-column groups of kb; partial slots per walker (K splits * n128)
    double2* exc_part;     // [nw][slots]
  };
  __device__ __forceinline__ static void store_warp(const Params& p, int row0, int lane, int col0, const float* v,
                                                    int ks, unsigned char*) {
    if (row0 >= 2 * p.nw || col0 >= p.kb) return;  // warp-uniform: padding rows / columns of the last tiles
    const int R = row0 + lane, w = R >> 1;
    const bool rv = R < 2 * p.nw, bf = p.bf16 != 0;
    // Z_part . G_re and Z_part . G_im: 8-column chunk sums added with Kahan compensation
    float a_re = 0.f, a_im = 0.f, k_re = 0.f, k_im = 0.f;
    if (rv) {
      const uint16_t* gr_h = p.g_hi + (size_t)(2 * w) * p.ldk;
      const uint16_t* gr_l = p.g_lo + (size_t)(2 * w) * p.ldk;
      const uint16_t* gi_h = gr_h + p.ldk;
      const uint16_t* gi_l = gr_l + p.ldk;
#pragma unroll
      for (int c8 = 0; c8 < 128; c8 += 8) {
        const int c = col0 + c8;
        if (c < p.kb) {  // 8 columns at a time (c + 8 <= ldk: rows padded to multiples of 8)
          const uint4 rh = *reinterpret_cast<const uint4*>(gr_h + c), rl = *reinterpret_cast<const uint4*>(gr_l + c);
          const uint4 ih = *reinterpret_cast<const uint4*>(gi_h + c), il = *reinterpret_cast<const uint4*>(gi_l + c);
          const uint32_t rhw[4] = {rh.x, rh.y, rh.z, rh.w}, rlw[4] = {rl.x, rl.y, rl.z, rl.w};
          const uint32_t ihw[4] = {ih.x, ih.y, ih.z, ih.w}, ilw[4] = {il.x, il.y, il.z, il.w};
          float s_re = 0.f, s_im = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int sh = 16 * (e & 1);
            const float gre = h2f((uint16_t)(rhw[e >> 1] >> sh), bf) + h2f((uint16_t)(rlw[e >> 1] >> sh), bf);
            const float gim = h2f((uint16_t)(ihw[e >> 1] >> sh), bf) + h2f((uint16_t)(ilw[e >> 1] >> sh), bf);
            if (c + e < p.kb) {  // the row's padding columns are never written
              s_re = fmaf(v[c8 + e], gre, s_re);
              s_im = fmaf(v[c8 + e], gim, s_im);
            }
          }
          const float y_re = s_re - k_re, t_re = a_re + y_re;
          k_re = (t_re - a_re) - y_re;
          a_re = t_re;
          const float y_im = s_im - k_im, t_im = a_im + y_im;
          k_im = (t_im - a_im) - y_im;
          a_im = t_im;
        }
      }
      a_re -= k_re;
      a_im -= k_im;
    }
    // lane 2k: Z_re . G (part 0), lane 2k + 1: Z_im . G (part 1)
    const float o_re = __shfl_xor_sync(0xffffffffu, a_re, 1), o_im = __shfl_xor_sync(0xffffffffu, a_im, 1);
    if (rv && (R & 1) == 0) {
      const double sc = (double)p.g_inv[w] * (double)p.g_inv[w] * (double)p.u_inv;
      const double ex = (double)a_re - (double)o_im, ey = (double)a_im + (double)o_re;
      p.exc_part[(size_t)w * p.slots + ks * p.n128 + col0 / 128] = c2(ex * sc, ey * sc);
    }
  }
};

}  // namespace afq
