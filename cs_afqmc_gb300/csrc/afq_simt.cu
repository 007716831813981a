// SIMT kernels of the AFQMC hot path: Green's function / overlap (FP64 Gauss-Jordan),
// complex x real GEMMs (FP64), field shifts, Taylor propagator (FP64), phaseless weights,
// local energy (FP64), Householder QR (FP64, LAPACK convention), comb SR, Philox RNG.
//
// Every kernel is templated on the walker storage type WT (double -> complex128 slabs,
// float -> complex64 slabs); arithmetic is FP64 throughout this file.

#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <mutex>

#include "afq_common.cuh"
#include "afq_kernels.cuh"
#include "afq_launch.cuh"
#include "afq_prof.cuh"

namespace afq {

// ======================================================================================
// Green's function and overlap.
// Above 32 electrons per spin (up to there: afq_green64.cu). One CTA per walker. For each stored slab s: S = C_s^T W_s (C real), Gauss-Jordan with
// partial pivoting on [S | I] gives det(S) and S^-1, then G_s = (W_s S^-1)^T.
// wavefunctions.py:478-501 (rhf), 658-692 (uhf).
// ======================================================================================

template <typename WT>
__global__ void k_green_overlap(const afq_ctx_dev c, const WT* __restrict__ w_up,
                                const WT* __restrict__ w_dn, double2* __restrict__ green,
                                double2* __restrict__ overlap, int write_green) {
  using CT = typename CplxOf<WT>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wlk = blockIdx.x;
  const int norb = c.norb;
  const int tid = threadIdx.x, nt = blockDim.x;
  __shared__ double red[32];
  __shared__ int piv_sh;
  __shared__ double2 det_sh;
  __shared__ double2 colj[64];
  // smem: W [norb][kmax] double2, Aug [o][2o] double2, C [norb][kmax] double
  double2* Ws = reinterpret_cast<double2*>(smem_raw);
  double2* Aug = Ws + (size_t)norb * c.kmax;
  double* Cs = reinterpret_cast<double*>(Aug + (size_t)c.kmax * 2 * c.kmax);

  double2 ovl = c2(1.0, 0.0);
  for (int s = 0; s < c.nslab; ++s) {
    const int ks = c.kslab[s];
    const int o = c.nocc_slab[s];  // occupied columns used from this slab
    const CT* W = reinterpret_cast<const CT*>(s == 0 ? w_up : w_dn) + (size_t)wlk * norb * ks;
    const double* C = c.trial[s];
    for (int i = tid; i < norb * o; i += nt) {
      int p = i / o, k = i % o;
      Ws[i] = ld_c(W + (size_t)p * ks + k);
      Cs[i] = C[(size_t)p * o + k];
    }
    __syncthreads();
    // S[i][k] = sum_p C[p][i] W[p][k];  Aug = [S | I]
    for (int e = tid; e < o * o; e += nt) {
      int i = e / o, k = e % o;
      double2 acc = c2(0, 0);
      for (int p = 0; p < norb; ++p) {
        double cv = Cs[p * o + i];
        double2 wv = Ws[p * o + k];
        acc.x += cv * wv.x;
        acc.y += cv * wv.y;
      }
      Aug[i * 2 * o + k] = acc;
      Aug[i * 2 * o + o + k] = c2(i == k ? 1.0 : 0.0, 0.0);
    }
    if (tid == 0) det_sh = c2(1.0, 0.0);
    __syncthreads();
    // Gauss-Jordan with partial pivoting (|re|+|im| pivot choice, as LAPACK izamax)
    for (int j = 0; j < o; ++j) {
      if (tid < 32) {
        double best = -1.0;
        int bi = j;
        for (int r = j + tid; r < o; r += 32) {
          double2 v = Aug[r * 2 * o + j];
          double m = fabs(v.x) + fabs(v.y);
          if (m > best) { best = m; bi = r; }
        }
        for (int off = 16; off > 0; off >>= 1) {
          double ob = __shfl_xor_sync(0xffffffffu, best, off);
          int oi = __shfl_xor_sync(0xffffffffu, bi, off);
          if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (tid == 0) piv_sh = bi;
      }
      __syncthreads();
      const int pr = piv_sh;
      if (pr != j) {
        for (int e = tid; e < 2 * o; e += nt) {
          double2 t = Aug[j * 2 * o + e];
          Aug[j * 2 * o + e] = Aug[pr * 2 * o + e];
          Aug[pr * 2 * o + e] = t;
        }
      }
      __syncthreads();
      const double2 pv = Aug[j * 2 * o + j];
      if (tid == 0) {
        double2 d = cmul(det_sh, pv);
        det_sh = (pr != j) ? c2(-d.x, -d.y) : d;
      }
      const double2 inv = cdiv(c2(1.0, 0.0), pv);
      __syncthreads();
      for (int e = tid; e < 2 * o; e += nt) Aug[j * 2 * o + e] = cmul(Aug[j * 2 * o + e], inv);
      // snapshot the multipliers (column j) before any thread overwrites them
      for (int r = tid; r < o; r += nt) colj[r] = Aug[r * 2 * o + j];
      __syncthreads();
      for (int e = tid; e < o * 2 * o; e += nt) {
        int r = e / (2 * o), col = e % (2 * o);
        if (r == j) continue;
        Aug[e] = csub(Aug[e], cmul(colj[r], Aug[j * 2 * o + col]));
      }
      __syncthreads();
    }
    ovl = cmul(ovl, det_sh);
    if (c.nslab == 1 && c.restricted_square) ovl = cmul(ovl, det_sh);  // RHF restricted: det^2
    if (write_green) {
      // G[i][p] = sum_k W[p][k] Sinv[k][i]; Sinv[k][i] = Aug[k][o + i]
      const int gblk = (c.nspin_g == 2) ? s : 0;
      double2* Gw = green + (size_t)wlk * c.ktot + (size_t)gblk * c.nocc_slab[0] * norb;
      for (int e = tid; e < o * norb; e += nt) {
        int i = e / norb, p = e % norb;
        double2 acc = c2(0, 0);
        for (int k = 0; k < o; ++k) acc = cadd(acc, cmul(Ws[p * o + k], Aug[k * 2 * o + o + i]));
        if (c.nspin_g == 1 && s == 1) acc = cadd(acc, Gw[e]);  // RHF two-slab: G_up + G_dn
        Gw[e] = acc;
      }
    }
    __syncthreads();
  }
  if (tid == 0 && overlap) overlap[wlk] = ovl;
}

// ======================================================================================
// Complex x real GEMM, FP64, on the FP64 units: C[m][n] = alpha * sum_k A[m][k] * B(k, n)
// B_KN: B(k,n) = B[k*ldb + n]; otherwise B(k,n) = B[n*ldb + k].
// For the entry points without a workspace and contexts that ask for the FP64 units; the others use the
// digit GEMM (afq_digits.cuh).
// ======================================================================================

template <bool B_KN>
__global__ void __launch_bounds__(256) k_gemm_cr(int M, int N, int K, const double2* __restrict__ A,
                                                 long lda, const double* __restrict__ B, long ldb,
                                                 double2* __restrict__ C, long ldc, double2 alpha) {
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ double2 As[BK][BM + 1];
  __shared__ double Bs[BK][BN + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = c2(0, 0);
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      int e = tid + l * 256;
      int r = e >> 4, cc = e & 15;  // A: row r of 64, col cc of 16
      int gm = m0 + r, gk = k0 + cc;
      As[cc][r] = (gm < M && gk < K) ? A[(long)gm * lda + gk] : c2(0, 0);
      if (B_KN) {
        int br = e >> 6, bc = e & 63;  // k row br of 16, n col bc of 64
        int bk = k0 + br, bn = n0 + bc;
        Bs[br][bc] = (bk < K && bn < N) ? B[(long)bk * ldb + bn] : 0.0;
      } else {
        int bc = e >> 4, br = e & 15;  // n col bc of 64, k row br of 16
        int bk = k0 + br, bn = n0 + bc;
        Bs[br][bc] = (bk < K && bn < N) ? B[(long)bn * ldb + bk] : 0.0;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double2 a[4];
      double b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j].x = fma(a[i].x, b[j], acc[i][j].x);
          acc[i][j].y = fma(a[i].y, b[j], acc[i][j].y);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gm = m0 + ty + 16 * i, gn = n0 + tx + 16 * j;
      if (gm < M && gn < N) C[(long)gm * ldc + gn] = cmul(alpha, acc[i][j]);
    }
}

// ======================================================================================
// Field shifts (propagation.py:121-127):
//   s = -sqrt(dt) (i fb - mf);  xt = x - s;  shift = sum xt*mf;  fbt = sum x*s - s^2/2
// One CTA per walker.
// ======================================================================================

__global__ void k_field_shifts(int nchol, double sqdt, const double* __restrict__ fields,
                               const double2* __restrict__ fb, const double2* __restrict__ mf,
                               double2* __restrict__ xt, double2* __restrict__ shift,
                               double2* __restrict__ fbt) {
  pdl_enter();
  __shared__ double red[32];
  const int w = blockIdx.x;
  double sx = 0, sy = 0, fx = 0, fy = 0;
  for (int g = threadIdx.x; g < nchol; g += blockDim.x) {
    double2 f = fb[(long)w * nchol + g];
    double2 m = mf[g];
    // i*fb - mf = (-f.y - m.x, f.x - m.y)
    double2 s = c2(-sqdt * (-f.y - m.x), -sqdt * (f.x - m.y));
    double x = fields[(long)w * nchol + g];
    double2 t = c2(x - s.x, -s.y);
    xt[(long)w * nchol + g] = t;
    double2 tm = cmul(t, m);
    sx += tm.x;
    sy += tm.y;
    double2 s2 = cmul(s, s);
    fx += x * s.x - 0.5 * s2.x;
    fy += x * s.y - 0.5 * s2.y;
  }
  sx = block_sum(sx, red);
  sy = block_sum(sy, red);
  fx = block_sum(fx, red);
  fy = block_sum(fy, red);
  if (threadIdx.x == 0) {
    shift[w] = c2(sx, sy);
    fbt[w] = c2(fx, fy);
  }
}

// ======================================================================================
// Taylor propagator, FP64 (propagation.py:67-92):
//   W <- E W;  W <- W + sum_{m=1}^{nterms-1} V^m W / m!;  W <- E W
// One CTA per (walker in chunk, slab). V read from the chunk's vhs buffer (L2-resident).
// ======================================================================================

constexpr int TAYLOR_MAXPT = 32;  // accumulator entries per thread (norb*k <= 32*blockDim)

template <typename WT>
__global__ void __launch_bounds__(256) k_taylor_f64(const afq_ctx_dev c, int w0,
                                                    const double2* __restrict__ vhs,
                                                    WT* __restrict__ w_up, WT* __restrict__ w_dn) {
  pdl_enter();
  using CT = typename CplxOf<WT>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wl = blockIdx.x, s = blockIdx.y;
  const int wlk = w0 + wl;
  const int norb = c.norb, ks = c.kslab[s];
  const int n = norb * ks;
  const int tid = threadIdx.x, nt = blockDim.x;
  double2* Ta = reinterpret_cast<double2*>(smem_raw);
  double2* Tb = Ta + n;
  const double* E = c.exp_h1[s];
  const double2* V = vhs + (size_t)wl * norb * norb;
  CT* W = reinterpret_cast<CT*>(s == 0 ? w_up : w_dn) + (size_t)wlk * n;
  for (int i = tid; i < n; i += nt) Ta[i] = ld_c(W + i);
  __syncthreads();
  double2 acc[TAYLOR_MAXPT];
  // Tb = E Ta ; acc = Tb
#pragma unroll
  for (int j = 0; j < TAYLOR_MAXPT; ++j) {
    int i = tid + j * nt;
    if (i < n) {
      int p = i / ks, col = i % ks;
      double2 a = c2(0, 0);
      for (int q = 0; q < norb; ++q) {
        double e = E[(size_t)p * norb + q];
        double2 t = Ta[q * ks + col];
        a.x = fma(e, t.x, a.x);
        a.y = fma(e, t.y, a.y);
      }
      Tb[i] = a;
      acc[j] = a;
    }
  }
  __syncthreads();
  double fact = 1.0;
  double2* src = Tb;
  double2* dst = Ta;
  for (int m = 1; m < c.n_exp_terms; ++m) {
    fact *= (double)m;
    const double invf = 1.0 / fact;
#pragma unroll
    for (int j = 0; j < TAYLOR_MAXPT; ++j) {
      int i = tid + j * nt;
      if (i < n) {
        int p = i / ks, col = i % ks;
        double2 a = c2(0, 0);
        const double2* Vr = V + (size_t)p * norb;
        for (int q = 0; q < norb; ++q) a = cadd(a, cmul(Vr[q], src[q * ks + col]));
        dst[i] = a;
        acc[j] = cadd(acc[j], cscale(a, invf));
      }
    }
    __syncthreads();
    double2* t = src;
    src = dst;
    dst = t;
  }
  // acc -> Ta, then W = E Ta
#pragma unroll
  for (int j = 0; j < TAYLOR_MAXPT; ++j) {
    int i = tid + j * nt;
    if (i < n) Ta[i] = acc[j];
  }
  __syncthreads();
  for (int i = tid; i < n; i += nt) {
    int p = i / ks, col = i % ks;
    double2 a = c2(0, 0);
    for (int q = 0; q < norb; ++q) {
      double e = E[(size_t)p * norb + q];
      double2 t = Ta[q * ks + col];
      a.x = fma(e, t.x, a.x);
      a.y = fma(e, t.y, a.y);
    }
    st_c(W + i, a);
  }
}

// The same for small slabs (norb * k <= kTaylorSmall, what its static shared memory holds): four lanes per element,
// each a quarter of the sum over q, so that a product of a few hundred elements is a few dependent FMAs long
// instead of norb. A step against an element per thread: 16 x 3 electrons, 50 walkers 38 -> 13 us; 20 x 5, 50 walkers
// 44 -> 27, 400 walkers 130 -> 68; 32 x 8 98 -> 72; 40 x 12 195 -> 169; 64 x 8 323 -> 233.

__global__ void __launch_bounds__(256) k_taylor_small(const afq_ctx_dev c, int w0, const double2* __restrict__ vhs,
                                                      double2* __restrict__ w_up, double2* __restrict__ w_dn) {
  pdl_enter();
  __shared__ double2 Ta[kTaylorSmall], Tb[kTaylorSmall], Acc[kTaylorSmall];
  const int wl = blockIdx.x, s = blockIdx.y, norb = c.norb, ks = c.kslab[s], n = norb * ks, tid = threadIdx.x;
  const int part = tid & 3;
  const double* __restrict__ E = c.exp_h1[s];
  const double2* __restrict__ V = vhs + (size_t)wl * norb * norb;
  double2* W = (s == 0 ? w_up : w_dn) + (size_t)(w0 + wl) * n;
  for (int i = tid; i < n; i += 256) Ta[i] = W[i];
  __syncthreads();
  // dot products over q by four lanes, summed by two shuffles; every lane gets the sum
  auto sum4 = [&](double2 a) {
#pragma unroll
    for (int off = 1; off < 4; off <<= 1)
      a = cadd(a, c2(__shfl_xor_sync(0xffffffffu, a.x, off), __shfl_xor_sync(0xffffffffu, a.y, off)));
    return a;
  };
  auto exp_row = [&](const double2* src, int i) {
    double2 a = c2(0, 0);
    if (i < n) {
      const int p = i / ks, col = i - p * ks;
#pragma unroll 4
      for (int q = part; q < norb; q += 4) {
        const double e = __ldg(E + (size_t)p * norb + q);
        const double2 t = src[q * ks + col];
        a = c2(fma(e, t.x, a.x), fma(e, t.y, a.y));
      }
    }
    return sum4(a);
  };
  for (int i0 = 0; i0 < n; i0 += 64) {
    const int i = i0 + (tid >> 2);
    const double2 a = exp_row(Ta, i);
    if (i < n && part == 0) Tb[i] = Acc[i] = a;
  }
  __syncthreads();
  double fact = 1.0;
  double2 *src = Tb, *dst = Ta;
  for (int m = 1; m < c.n_exp_terms; ++m) {
    fact *= (double)m;
    const double invf = 1.0 / fact;
    for (int i0 = 0; i0 < n; i0 += 64) {
      const int i = i0 + (tid >> 2);
      double2 a = c2(0, 0), b = c2(0, 0);  // real and imaginary factors of V apart: shorter chains
      if (i < n) {
        const int p = i / ks, col = i - p * ks;
#pragma unroll 4
        for (int q = part; q < norb; q += 4) {
          const double2 v = __ldg(V + (size_t)p * norb + q), t = src[q * ks + col];
          a = c2(fma(v.x, t.x, a.x), fma(v.x, t.y, a.y));
          b = c2(fma(-v.y, t.y, b.x), fma(v.y, t.x, b.y));
        }
      }
      a = sum4(cadd(a, b));
      if (i < n && part == 0) {
        dst[i] = a;
        Acc[i] = c2(fma(a.x, invf, Acc[i].x), fma(a.y, invf, Acc[i].y));
      }
    }
    __syncthreads();
    double2* t = src;
    src = dst;
    dst = t;
  }
  for (int i0 = 0; i0 < n; i0 += 64) {
    const int i = i0 + (tid >> 2);
    const double2 a = exp_row(Acc, i);
    if (i < n && part == 0) W[i] = a;
  }
}

// ======================================================================================
// Phaseless importance function and weights (propagation.py:133-164).
// ======================================================================================

struct WeightArgs {
  int nw, ntiles;
  double dt;
  double2 h0_prop;
  const double2 *shift, *fbt, *ovl_new;
  double2* ovl;
  double *weights, *scalars;
  const int* status;  // may be NULL
};

// The tensor-core pipelines' guard word joins scalars[AFQ_S_STATUS], so that callers see a wait that ran
// out or a bad operand in the state (status may be NULL)
AFQ_D void fold_status(double* scalars, const int* status) {
  if (status && *status != 0) scalars[AFQ_S_STATUS] = (double)((int)scalars[AFQ_S_STATUS] | *status);
}

__global__ void k_fold_status(double* scalars, const int* status) {
  pdl_enter();
  fold_status(scalars, status);
}

// NaN over results that a call returns without a state to report in
__global__ void k_poison(long n, double2* out, const int* status) {
  pdl_enter();
  if (*status == 0) return;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = c2(nan(""), nan(""));
}

// One walker's new weight and overlap
AFQ_D double weight_step(const WeightArgs& g, int w, double pcs) {
  const double sqdt = sqrt(g.dt);
  double2 ratio = cdiv(g.ovl_new[w], g.ovl[w]);
  double2 sh = c2(0, 0), fb = c2(0, 0);
  for (int t = 0; t < g.ntiles; ++t) {
    sh = cadd(sh, g.shift[(size_t)w * g.ntiles + t]);
    fb = cadd(fb, g.fbt[(size_t)w * g.ntiles + t]);
  }
  // |I| cos(angle(ph)) with I = exp(arg) O'/O and ph = exp(-sqrt(dt) shift) O'/O equals
  // exp(Re arg) Re(exp(i Im(-sqrt(dt) shift)) O'/O): one exp and one sincos instead of two
  // complex exponentials, atan2, hypot and cos (the same quantity; FP64 transcendentals are
  // slow on this part)
  const double re_arg = -sqdt * sh.x + fb.x + g.dt * (pcs + g.h0_prop.x);
  double sn, cs;
  sincos(-sqdt * sh.y, &sn, &cs);
  double v = exp(re_arg) * (cs * ratio.x - sn * ratio.y);
  if (isnan(v)) v = 0.0;
  if (v < 1.0e-3) v = 0.0;
  if (v > 100.0) v = 0.0;
  double nwgt = v * g.weights[w];
  if (nwgt > 100.0) nwgt = 0.0;
  g.weights[w] = nwgt;
  g.ovl[w] = g.ovl_new[w];
  return nwgt;
}

// pop_control_ene_shift = e_estimate - 0.1 log(sum w / nw) / dt (propagation.py:161-163)
AFQ_D void pop_control(const WeightArgs& g, double sum) {
  g.scalars[AFQ_S_POP_CONTROL_SHIFT] = g.scalars[AFQ_S_E_ESTIMATE] - 0.1 * log(sum / (double)g.nw) / g.dt;
  fold_status(g.scalars, g.status);
}

__global__ void k_weights(const WeightArgs g) {
  pdl_enter();
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < g.nw) weight_step(g, w, g.scalars[AFQ_S_POP_CONTROL_SHIFT]);
}

__global__ void k_pop_control(const WeightArgs g) {
  pdl_enter();
  __shared__ double red[32];
  double sum = 0.0;
  for (int w = threadIdx.x; w < g.nw; w += blockDim.x) sum += g.weights[w];
  sum = block_sum(sum, red);
  if (threadIdx.x == 0) pop_control(g, sum);
}

// Both in one launch: a cluster of eight CTAs, so that the walkers' exponentials still run on eight SMs'
// FP64 units, and their sums meet in the first CTA's shared memory. Against two launches: 512 walkers
// 10.9 -> 9.1 us, 1024 11.9 -> 10.7, and a launch less in the chain of a step (ten steps of 64 walkers 787 -> 774 us).
// Above 1024 walkers an SM would run more than four warps of FP64 exponentials, 1.8 us each.
// The weights are summed as the two launches do, a warp of 32 consecutive walkers and then the 32 warps.
constexpr int kWeightsCluster = 1024, kWeightsCtas = 8;

__global__ void __cluster_dims__(kWeightsCtas, 1, 1) __launch_bounds__(128) k_weights_pop(const WeightArgs g) {
  namespace cg = cooperative_groups;
  __shared__ double part[32];
  const cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < 32) part[threadIdx.x] = 0.0;
  cl.sync();  // every CTA runs: its shared memory may be written from here on
  pdl_enter();
  const int w = (int)cl.block_rank() * blockDim.x + threadIdx.x;
  const double pcs = g.scalars[AFQ_S_POP_CONTROL_SHIFT];
  const double v = warp_sum(w < g.nw ? weight_step(g, w, pcs) : 0.0);
  if ((threadIdx.x & 31) == 0) *cl.map_shared_rank(&part[w >> 5], 0) = v;
  cl.sync();  // all have read the old shift, too
  if (cl.block_rank() == 0 && threadIdx.x < 32) {
    const double sum = warp_sum(part[threadIdx.x]);
    if (threadIdx.x == 0) pop_control(g, sum);
  }
}

// ======================================================================================
// Local energy, FP64 (wavefunctions.py:529-561, 711-743).
// Pass 1: CTA per (walker, chunk of g): f_g = RC_g G^T, c_g = tr f_g,
//         exc_g = sum_ik f_g[i,k] f_g[k,i]; per-chunk partial sums.
// Pass 2: CTA per walker: reduce chunks, add ene1 = sum G * rot_h1 and h0.
// Partial slots: RHF: [sum c^2, sum exc]; UHF: [sum cu^2, sum cd^2, sum cu cd, exc_u, exc_d].
// ======================================================================================

__global__ void __launch_bounds__(256) k_energy_f64_part(const afq_ctx_dev c, int gchunk,
                                                         const double2* __restrict__ green,
                                                         double2* __restrict__ epart) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int w = blockIdx.x, ch = blockIdx.y;
  const int norb = c.norb, tid = threadIdx.x, nt = blockDim.x;
  double2* Gs = reinterpret_cast<double2*>(smem_raw);            // [ktot]
  double2* F = Gs + c.ktot;                                      // [2][omax*omax]
  __shared__ double red[32];
  const int omax = c.kmax;
  for (int i = tid; i < c.ktot; i += nt) Gs[i] = green[(size_t)w * c.ktot + i];
  __syncthreads();
  double2 acc[5];
  for (int q = 0; q < 5; ++q) acc[q] = c2(0, 0);
  const int g0 = ch * gchunk, g1 = min(c.nchol, g0 + gchunk);
  for (int g = g0; g < g1; ++g) {
    double2 cc[2], ex[2];
    for (int s = 0; s < c.nspin_g; ++s) {
      const int o = c.gocc[s];
      const double* RC = c.rot_chol[s] + (size_t)g * o * norb;
      const double2* Gsp = Gs + (size_t)s * c.gocc[0] * norb;
      double2* Fs = F + s * omax * omax;
      for (int e = tid; e < o * o; e += nt) {
        int i = e / o, k = e % o;
        double2 a = c2(0, 0);
        const double* rr = RC + (size_t)i * norb;
        const double2* gg = Gsp + (size_t)k * norb;
        for (int p = 0; p < norb; ++p) {
          a.x = fma(rr[p], gg[p].x, a.x);
          a.y = fma(rr[p], gg[p].y, a.y);
        }
        Fs[e] = a;
      }
      __syncthreads();
      double tr_x = 0, tr_y = 0, ex_x = 0, ex_y = 0;
      for (int e = tid; e < o * o; e += nt) {
        int i = e / o, k = e % o;
        double2 p = cmul(Fs[i * o + k], Fs[k * o + i]);
        ex_x += p.x;
        ex_y += p.y;
        if (i == k) { tr_x += Fs[e].x; tr_y += Fs[e].y; }
      }
      tr_x = block_sum(tr_x, red);
      tr_y = block_sum(tr_y, red);
      ex_x = block_sum(ex_x, red);
      ex_y = block_sum(ex_y, red);
      cc[s] = c2(tr_x, tr_y);
      ex[s] = c2(ex_x, ex_y);
    }
    if (c.nspin_g == 1) {
      acc[0] = cadd(acc[0], cmul(cc[0], cc[0]));
      acc[1] = cadd(acc[1], ex[0]);
    } else {
      acc[0] = cadd(acc[0], cmul(cc[0], cc[0]));
      acc[1] = cadd(acc[1], cmul(cc[1], cc[1]));
      acc[2] = cadd(acc[2], cmul(cc[0], cc[1]));
      acc[3] = cadd(acc[3], ex[0]);
      acc[4] = cadd(acc[4], ex[1]);
    }
  }
  if (tid == 0) {
    for (int q = 0; q < 5; ++q) epart[((size_t)w * gridDim.y + ch) * 5 + q] = acc[q];
  }
}

__global__ void k_energy_final(const afq_ctx_dev c, int nchunks, const double2* __restrict__ green,
                               const double2* __restrict__ epart, double2* __restrict__ energy) {
  __shared__ double red[32];
  const int w = blockIdx.x, norb = c.norb;
  // ene1
  double e1x = 0, e1y = 0;
  for (int s = 0; s < c.nspin_g; ++s) {
    const int o = c.gocc[s];
    const double2* G = green + (size_t)w * c.ktot + (size_t)s * c.gocc[0] * norb;
    const double* R = c.rot_h1[s];
    for (int e = threadIdx.x; e < o * norb; e += blockDim.x) {
      e1x += G[e].x * R[e];
      e1y += G[e].y * R[e];
    }
  }
  e1x = block_sum(e1x, red);
  e1y = block_sum(e1y, red);
  if (threadIdx.x == 0) {
    double2 a[5];
    for (int q = 0; q < 5; ++q) a[q] = c2(0, 0);
    for (int ch = 0; ch < nchunks; ++ch)
      for (int q = 0; q < 5; ++q) a[q] = cadd(a[q], epart[((size_t)w * nchunks + ch) * 5 + q]);
    double2 e2, e1 = c2(e1x, e1y);
    if (c.energy_mode == 0) {  // RHF restricted: 2 sum c^2 - exc ; ene1 x2
      e2 = csub(cscale(a[0], 2.0), a[1]);
      e1 = cscale(e1, 2.0);
    } else if (c.energy_mode == 1) {  // RHF two-slab (G = G_up + G_dn): sum c^2 - exc
      e2 = csub(a[0], a[1]);
    } else {  // UHF
      e2 = cscale(csub(cadd(cadd(a[0], a[1]), cscale(a[2], 2.0)), cadd(a[3], a[4])), 0.5);
    }
    energy[w] = cadd(cadd(e2, e1), c2(c.h0, 0.0));
  }
}

// ======================================================================================
// Householder QR of FP64 walkers, LAPACK zgeqr2 + zung2r conventions (R has a real diagonal,
// beta = -sign(Re alpha) * |(alpha, x)|), linalg_utils.py:51-65 (jnp.linalg.qr, reduced mode). One CTA
// per (walker, slab) with the slab in shared memory (odd row stride: conflict-free column walks), a thread
// per row up to eight warps, Q over W.
//
// What bounds it: latency in FP64 chains, then the FP64 units (a warp instruction takes some 18 cycles
// whatever its lanes do; 10 m k^2 of them, with 32 elements each). So a column is one reduction, a few scalar
// steps by one warp and one update: the squares of column j are one more of the sums over its raw elements,
// v^H a_c = a_jc + conj(scale) sum, the divisions are lanes of one instruction, tau goes into the sums
// (conj(tau) conj(scale) = -1 / b).
// Row j right of the diagonal (R) is never read again and is left alone.
// Against a warp per slab with a pass for the norm: 40 x 7 and 40 x 6 electrons, 200 walkers 71 -> 57 us; 60 x 10 and
// 60 x 8, 512 walkers 186 -> 207 us; a block of five steps with one QR, 120 x 20, 256 walkers 7.82 -> 7.46 ms.
// rdiag (optional, [nslab][nw]): prod(diag R) per walker slab (linalg_utils.py:51-65 returns
// it as the norm factor; the free-projection step multiplies its norms by it)
// ======================================================================================

// y[c] = mul sum_{r > j} conj(A[r][j]) A[r][c] for c in [c_lo, k): lpc lanes (a power of two) per column.
// Short chains, the four products of a complex one in their own: two chains of eight rows at a time. Q
// against extended precision, walkers of 120 x 20 and 60 x 28: 3.10e-16 and 3.74e-16 with a sum over 32 lanes, 4.45e-16
// at 120 x 20 with chains over all rows of a lane and the update below as an FMA chain, 3.26e-16 and 3.97e-16 with
// two products a chain, now (with the reflector's scale to one rounding) 2.98e-16 and 3.65e-16.
AFQ_D void qr64_sums(const double2* A, int ld, int m, int k, int j, int c_lo, double2 mul, double2* y) {
  const int nc = k - c_lo, tid = threadIdx.x, nt = blockDim.x;
  int sh = 0;
  while (sh < 5 && (nc << (sh + 1)) <= nt) ++sh;
  const int lpc = 1 << sh, part = tid & (lpc - 1);
  for (int c0 = 0; c0 < nc; c0 += nt >> sh) {
    const int c = c_lo + c0 + (tid >> sh);
    double2 sum = c2(0, 0);
    if (c < k) {
      for (int r0 = j + 1 + part; r0 < m; r0 += 16 * lpc) {
        const int r1 = min(m, r0 + 16 * lpc);
        // sums of x.x v.x and x.y v.x (a, b), of x.y v.y and x.x v.y (e, f)
        double2 a = c2(0, 0), b = a, e = a, f = a;
        int r = r0;
#pragma unroll 4
        for (; r + lpc < r1; r += 2 * lpc) {
          const double2 x = A[r * ld + c], v = A[r * ld + j];
          const double2 x2 = A[(r + lpc) * ld + c], v2 = A[(r + lpc) * ld + j];
          a = c2(fma(x.x, v.x, a.x), fma(x.y, v.x, a.y));
          e = c2(fma(x.y, v.y, e.x), fma(x.x, v.y, e.y));
          b = c2(fma(x2.x, v2.x, b.x), fma(x2.y, v2.x, b.y));
          f = c2(fma(x2.y, v2.y, f.x), fma(x2.x, v2.y, f.y));
        }
        if (r < r1) {
          const double2 x = A[r * ld + c], v = A[r * ld + j];
          a = c2(fma(x.x, v.x, a.x), fma(x.y, v.x, a.y));
          e = c2(fma(x.y, v.y, e.x), fma(x.x, v.y, e.y));
        }
        a = cadd(a, b);
        e = cadd(e, f);
        sum = cadd(sum, c2(a.x + e.x, a.y - e.y));
      }
    }
    for (int off = 1; off < lpc; off <<= 1)
      sum = cadd(sum, c2(__shfl_xor_sync(0xffffffffu, sum.x, off), __shfl_xor_sync(0xffffffffu, sum.y, off)));
    if (c < k && part == 0) y[c] = cmul(mul, sum);
  }
}

// row[c] -= v z[c] for c > j. The product is rounded before it meets the element (an FMA chain onto the
// element rounds twice at its size).
AFQ_D void qr64_row(double2* row, int k, int j, double2 v, const double2* z) {
#pragma unroll 4
  for (int c = j + 1; c < k; ++c) {
    const double2 x = z[c], a = row[c];
    row[c] = c2(a.x - fma(v.x, x.x, -v.y * x.y), a.y - fma(v.x, x.y, v.y * x.x));
  }
}

__global__ void __launch_bounds__(256) k_qr_f64(const afq_ctx_dev c, double2* __restrict__ w_up,
                                                double2* __restrict__ w_dn, double2* __restrict__ rdiag) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double2 scale;
  const int wlk = blockIdx.x, s = blockIdx.y, tid = threadIdx.x, nt = blockDim.x;
  const int m = c.norb, k = c.kslab[s], ld = k | 1;
  double2* A = reinterpret_cast<double2*>(smem_raw);  // [m][ld]
  double2* y = A + (size_t)m * ld;                    // [k]
  double2* tau = y + k;                               // [k]
  double2* W = (s == 0 ? w_up : w_dn) + (size_t)wlk * m * k;
  for (int i = tid; i < m * k; i += nt) {
    const int r = i / k;
    A[r * ld + (i - r * k)] = W[i];
  }
  double2 rprod = c2(1.0, 0.0);  // warp 0
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    qr64_sums(A, ld, m, k, j, j, c2(1.0, 0.0), y);
    __syncthreads();
    if (tid < 32) {
      const double2 alpha = A[j * ld + j];
      const double xn = y[j].x;
      double2 t = c2(0, 0), scl = c2(1, 0), beta = alpha;
      double nib = 0.0;  // -1 / b = conj(tau) conj(scale)
      if (!(xn == 0.0 && alpha.y == 0.0)) {
        const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn);
        const double b = alpha.x >= 0.0 ? -nrm : nrm, dx = alpha.x - b, d2 = dx * dx + alpha.y * alpha.y;
        // tau = (b - alpha) / b, scale = 1 / (alpha - b) and -1 / b, a quotient per lane
        const double num = tid == 0 ? -dx : tid == 2 ? dx : tid == 4 ? -1.0 : -alpha.y;
        const double q = num / (tid == 2 || tid == 3 ? d2 : b);
        t = c2(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
        scl = c2(__shfl_sync(0xffffffffu, q, 2), __shfl_sync(0xffffffffu, q, 3));
        nib = __shfl_sync(0xffffffffu, q, 4);
        beta = c2(b, 0);
        // a Newton step: its relative error is that of the whole reflector, and 1 / d2 alone has three roundings
        const double h = alpha.y * scl.x, l = fma(alpha.y, scl.x, -h);
        const double ex = fma(alpha.y, scl.y, fma(-dx, scl.x, 1.0)), ey = fma(-dx, scl.y, -h) - l;
        scl = c2(scl.x + fma(scl.x, ex, -(scl.y * ey)), scl.y + fma(scl.x, ey, scl.y * ex));
      }
      // conj(tau) v^H a = conj(tau) a_j - sum / b
      for (int i = j + 1 + tid; i < k; i += 32) {
        const double2 p = cmul(cconj(t), A[j * ld + i]);
        y[i] = c2(fma(nib, y[i].x, p.x), fma(nib, y[i].y, p.y));
      }
      if (tid == 0) {
        rprod = cmul(rprod, beta);
        tau[j] = t;
        scale = scl;
      }
    }
    __syncthreads();
    const double2 scl = scale;
    for (int r = j + 1 + tid; r < m; r += nt) {
      double2* row = A + r * ld;
      const double2 v = cmul(row[j], scl);
      row[j] = v;
      qr64_row(row, k, j, v, y);
    }
    __syncthreads();
  }
  if (tid == 0 && rdiag) rdiag[(size_t)s * c.nw + wlk] = rprod;
  // form Q (zung2r): columns from last to first; row j of the columns behind j is still zero
  for (int j = k - 1; j >= 0; --j) {
    const double2 t = tau[j];
    qr64_sums(A, ld, m, k, j, j + 1, t, y);
    __syncthreads();
    for (int r = tid; r < m; r += nt) {
      double2* row = A + r * ld;
      if (r < j) {
        row[j] = c2(0, 0);
      } else if (r == j) {
        row[j] = c2(1.0 - t.x, -t.y);
        for (int i = j + 1; i < k; ++i) row[i] = c2(-y[i].x, -y[i].y);
      } else {
        const double2 v = row[j];
        qr64_row(row, k, j, v, y);
        row[j] = cmul(c2(-t.x, -t.y), v);
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < m * k; i += nt) {
    const int r = i / k;
    W[i] = A[r * ld + (i - r * k)];
  }
}

// ======================================================================================
// Comb stochastic reconfiguration (sr.py:24-47). One CTA computes the indices from the
// cumulative sum as numpy/jnp.cumsum rounds it (in index order), then a gather.
// ======================================================================================

// Serial sums cum[i] = |w_0| + ... + |w_i| from i on, a = the sum before (one thread).
AFQ_D void sr_serial(int i, int n, double a, const double* weights, double* cum) {
  for (; i + 16 <= n; i += 16) {  // sixteen loads ahead of the chain of adds
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = fabs(weights[i + u]);
#pragma unroll
    for (int u = 0; u < 16; ++u) cum[i + u] = a = a + v[u];
  }
  for (; i < n; ++i) cum[i] = a = a + fabs(weights[i]);
}

// The same rounded sums, bit for bit, a chunk of the block's threads at a time. While the sum a stays between
// two powers of two it is a multiple of u, its last bit's weight, and adding w moves it by w / u rounded to
// an integer, halves to the even sum. The integer depends on a by its parity only (and by that only at a
// half), so an element is a pair of steps, one for each parity it may meet, and pairs compose: an integer
// scan gives every sum. The element that takes a past the power of two is added in FP64 and the next
// chunk starts behind it, with twice the u.
// Serial adds take 50 ns each here, a chunk about 2 us, and some log2(nw / 32) + nw / 1024 chunks are needed.
// The whole kernel, against serial sums: 2048 walkers 108.8 -> 28.2 us, 1024 56.6 -> 24.4, 256 16.3 -> 15.2 (the line; 64
// walkers take 6.1 serially).
constexpr int kSrScanMin = 256, kSrHead = 32;  // populations from here on; elements summed serially first

AFQ_D void sr_scan(int nw, const double* weights, double* cum) {
  __shared__ long long tot[32][2];
  __shared__ int first[2];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x;  // 1024 threads
  if (tid == 0) sr_serial(0, kSrHead, 0.0, weights, cum);
  if (tid < 2) first[tid] = nt;
  __syncthreads();
  int i = kSrHead, turn = 0;
  double a = cum[kSrHead - 1];
  while (i < nw) {
    const int be = (int)((unsigned long long)__double_as_longlong(a) >> 52);  // sign and biased exponent
    if (be < 1 || be >= 2047) {  // zero, denormal or not finite
      if (tid == 0) sr_serial(i, nw, a, weights, cum);
      return;
    }
    // |w| = mw 2^(ew - 1075), so that w / u = mw 2^-sh (integers: FP64 instructions of 32 warps take longer)
    const int at = i + tid;
    const long long bits = at < nw ? __double_as_longlong(weights[at]) & 0x7fffffffffffffffll : 0;
    const int ew = (int)(bits >> 52), sh = be - max(ew, 1);
    const long long mw = (bits & 0xfffffffffffffll) | (ew ? 1ll << 52 : 0ll);
    const bool big = sh <= 0 && mw != 0;  // past the power of two for sure (or not finite)
    const bool some = sh > 0 && sh < 54;
    const long long n = some ? mw >> sh : 0, rem = some ? mw - (n << sh) : 0, half = some ? 1ll << (sh - 1) : 1;
    long long s0 = n + ((rem > half || (rem == half && (n & 1))) ? 1 : 0);   // from an even sum
    long long s1 = n + ((rem > half || (rem == half && !(n & 1))) ? 1 : 0);  // from an odd one
    auto join = [](long long& x0, long long& x1, long long y0, long long y1) {  // x, then y
      x0 += (x0 & 1) ? y1 : y0;
      x1 += (x1 & 1) ? y0 : y1;
    };
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      long long p0 = __shfl_up_sync(0xffffffffu, s0, o), p1 = __shfl_up_sync(0xffffffffu, s1, o);
      if (lane >= o) {
        join(p0, p1, s0, s1);
        s0 = p0;
        s1 = p1;
      }
    }
    if (lane == 31) {
      tot[wid][0] = s0;
      tot[wid][1] = s1;
    }
    __syncthreads();
    if (tid == 0) first[turn ^ 1] = nt;  // read for the last time before this barrier
    long long b0 = tot[lane][0], b1 = tot[lane][1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      long long p0 = __shfl_up_sync(0xffffffffu, b0, o), p1 = __shfl_up_sync(0xffffffffu, b1, o);
      if (lane >= o) {
        join(p0, p1, b0, b1);
        b0 = p0;
        b1 = p1;
      }
    }
    b0 = __shfl_sync(0xffffffffu, b0, (wid + 31) & 31);
    b1 = __shfl_sync(0xffffffffu, b1, (wid + 31) & 31);
    if (wid == 0) b0 = b1 = 0;
    join(b0, b1, s0, s1);
    const long long m = (__double_as_longlong(a) & 0xfffffffffffffll) | (1ll << 52);  // a / u
    const long long c = m + ((m & 1) ? b1 : b0);
    const bool past = big || c >= (1ll << 53);
    const unsigned votes = __ballot_sync(0xffffffffu, past);
    if (votes && lane == 0) atomicMin(&first[turn], wid * 32 + __ffs((int)votes) - 1);
    // valid as far as no element before is past; the others' values are written again below
    if (at < nw && !past) cum[at] = __longlong_as_double(((long long)be << 52) | (c & 0xfffffffffffffll));
    __syncthreads();
    const int f = first[turn];
    turn ^= 1;
    if (f >= nt) {
      i += nt;
      if (i < nw) a = cum[i - 1];
    } else {
      if (f > 0) a = cum[i + f - 1];
      a += fabs(weights[i + f]);
      __syncthreads();
      if (tid == 0) cum[i + f] = a;
      i += f + 1;
    }
  }
}

// in_smem: the sums stay in shared memory, where they are searched
__global__ void __launch_bounds__(1024) k_sr_indices(int nw, const double* __restrict__ zeta,
                                                     double* __restrict__ weights, double* __restrict__ cum_g,
                                                     int32_t* __restrict__ idx, int in_smem) {
  pdl_enter();
  extern __shared__ double cum_s[];
  double* cum = in_smem ? cum_s : cum_g;
  if (nw >= kSrScanMin) sr_scan(nw, weights, cum);
  else if (threadIdx.x == 0) sr_serial(0, nw, 0.0, weights, cum);
  __syncthreads();
  __shared__ double w_new;
  const double tw = cum[nw - 1];
  const double z0 = zeta[0];
  if (threadIdx.x == 0) w_new = tw / (double)nw;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    const double z = tw * ((double)i + z0) / (double)nw;
    // sums are not negative, so they compare as their bits do (a NaN: as nothing below)
    const long long zb = isnan(z) ? 0 : __double_as_longlong(z);
    int lo = 0, hi = nw;  // first index with cum >= z
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (__double_as_longlong(cum[mid]) < zb) lo = mid + 1; else hi = mid;
    }
    idx[i] = min(lo, nw - 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nw; i += blockDim.x) weights[i] = w_new;
}

template <typename WT>
__global__ void k_gather_slab(int slab_elems, const int32_t* __restrict__ idx,
                              const WT* __restrict__ src, WT* __restrict__ dst) {
  pdl_enter();
  using CT = typename CplxOf<WT>::type;
  const int w = blockIdx.x;
  const CT* s = reinterpret_cast<const CT*>(src) + (size_t)idx[w] * slab_elems;
  CT* d = reinterpret_cast<CT*>(dst) + (size_t)w * slab_elems;
  for (int i = threadIdx.x; i < slab_elems; i += blockDim.x) d[i] = s[i];
}

// ======================================================================================
// Block statistics (sampling.py:74-91) and the sampler total (sampling.py:337-341).
// ======================================================================================

__global__ void k_block_stats(int nw, double dt, const double2* __restrict__ energy,
                              const double* __restrict__ weights, double* __restrict__ scalars,
                              double* __restrict__ be_out, double* __restrict__ bw_out,
                              const int* __restrict__ status) {
  pdl_enter();
  if (threadIdx.x == 0) fold_status(scalars, status);
  __shared__ double red[32];
  const double e_est = scalars[AFQ_S_E_ESTIMATE];
  const double lim = sqrt(2.0 / dt);
  double sw = 0, swe = 0, nz = 0;
  for (int w = threadIdx.x; w < nw; w += blockDim.x) {
    double e = energy[w].x;
    if (fabs(e - e_est) > lim) e = e_est;
    double wt = weights[w];
    sw += wt;
    swe += e * wt;
    nz += (wt != 0.0) ? 1.0 : 0.0;
  }
  sw = block_sum(sw, red);
  swe = block_sum(swe, red);
  nz = block_sum(nz, red);
  if (threadIdx.x == 0) {
    double be = swe / sw;
    scalars[AFQ_S_N_KILLED] += (double)nw - nz;
    scalars[AFQ_S_BLOCK_ENERGY] = be;
    scalars[AFQ_S_BLOCK_WEIGHT] = sw;
    scalars[AFQ_S_POP_CONTROL_SHIFT] = 0.9 * scalars[AFQ_S_POP_CONTROL_SHIFT] + 0.1 * be;
    if (be_out) *be_out = be;
    if (bw_out) *bw_out = sw;
  }
}

// en_samples (corr_sample.py:482-491): Re(E) clamped to e_estimate beyond sqrt(2/dt)
__global__ void k_clamped_energies(int nw, double dt, const double2* __restrict__ energy,
                                   const double* __restrict__ scalars, double* __restrict__ out) {
  pdl_enter();
  const double e_est = scalars[AFQ_S_E_ESTIMATE];
  const double lim = sqrt(2.0 / dt);
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
    const double e = energy[w].x;
    out[w] = (fabs(e - e_est) > lim) ? e_est : e;
  }
}

// corr_otler_rm (corr_sample.py:557-594) + the weighted sums of cs_step (673-694), one CTA.
// mean and population std in two passes, as jnp.mean / jnp.std; the larger z-score selected
// with jnp.where(z1 > z2, z1, z2) semantics (a NaN z1 selects z2).
__global__ void k_cs_outlier(int nw, double z_thresh, double* __restrict__ w1, double* __restrict__ w2,
                             const double* __restrict__ e1, const double* __restrict__ e2,
                             double* __restrict__ sums) {
  pdl_enter();
  __shared__ double red[32];
  double s1 = 0, s2 = 0;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    s1 += w1[i];
    s2 += w2[i];
  }
  const double m1 = block_sum(s1, red) / nw, m2 = block_sum(s2, red) / nw;
  double v1 = 0, v2 = 0;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    v1 += (w1[i] - m1) * (w1[i] - m1);
    v2 += (w2[i] - m2) * (w2[i] - m2);
  }
  const double sd1 = sqrt(block_sum(v1, red) / nw), sd2 = sqrt(block_sum(v2, red) / nw);
  double a1 = 0, b1 = 0, a2 = 0, b2 = 0;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    const double z1 = fabs(w1[i] - m1) / sd1, z2 = fabs(w2[i] - m2) / sd2;
    const double z = (z1 > z2) ? z1 : z2;
    double x1 = w1[i], x2 = w2[i];
    if (z > z_thresh) {
      x1 = 0.0;
      x2 = 0.0;
    }
    w1[i] = x1;
    w2[i] = x2;
    a1 += e1[i] * x1;
    b1 += x1;
    a2 += e2[i] * x2;
    b2 += x2;
  }
  a1 = block_sum(a1, red);
  b1 = block_sum(b1, red);
  a2 = block_sum(a2, red);
  b2 = block_sum(b2, red);
  if (threadIdx.x == 0) {
    sums[0] = a1;
    sums[1] = b1;
    sums[2] = a2;
    sums[3] = b2;
  }
}

__global__ void k_phaseless_begin(double* scalars) {
  pdl_enter();
  scalars[AFQ_S_N_KILLED] = 0.0;
  scalars[AFQ_S_POP_CONTROL_SHIFT] = scalars[AFQ_S_E_ESTIMATE];
}

__global__ void k_phaseless_end(int nblk, double denom, const double* __restrict__ be,
                                const double* __restrict__ bw, double* __restrict__ scalars,
                                double* __restrict__ energy) {
  pdl_enter();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int i = 0; i < nblk; ++i) {
      a += be[i] * bw[i];
      b += bw[i];
    }
    *energy = a / b;
    scalars[AFQ_S_N_KILLED] /= denom;
  }
}

// driver.py:252 (block weight before QR/SR) and driver.py:308 (e_estimate update)
__global__ void k_driver_update(int nw, const double* __restrict__ weights,
                                const double* __restrict__ energy, double* __restrict__ scalars,
                                double* __restrict__ wsum) {
  pdl_enter();
  __shared__ double red[32];
  double s = 0.0;
  for (int w = threadIdx.x; w < nw; w += blockDim.x) s += weights[w];
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    *wsum = s;
    scalars[AFQ_S_E_ESTIMATE] = 0.9 * scalars[AFQ_S_E_ESTIMATE] + 0.1 * energy[0];
  }
}

// ======================================================================================
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) + Box-Muller.
// ======================================================================================

AFQ_D void philox_round(uint32_t& c0, uint32_t& c1, uint32_t& c2_, uint32_t& c3, uint32_t k0,
                        uint32_t k1) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  uint32_t hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
  uint32_t hi1 = __umulhi(M1, c2_), lo1 = M1 * c2_;
  uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
  c0 = n0; c1 = n1; c2_ = n2; c3 = n3;
}

AFQ_D uint4 philox4x32(uint64_t ctr, uint64_t key) {
  uint32_t c0 = (uint32_t)ctr, c1 = (uint32_t)(ctr >> 32), c2_ = 0x5851F42Du, c3 = 0x14057B7Eu;
  uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    philox_round(c0, c1, c2_, c3, k0, k1);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return make_uint4(c0, c1, c2_, c3);
}

// 53-bit uniform in (0, 1] from two words
AFQ_D double u53(uint32_t a, uint32_t b) {
  uint64_t v = ((uint64_t)(a >> 5) << 26) | (uint64_t)(b >> 6);
  return ((double)v + 1.0) * (1.0 / 9007199254740992.0);
}

__global__ void k_fill_normal(double* out, int64_t n, uint64_t seed, uint64_t offset) {
  int64_t pair = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t i0 = 2 * pair;
  if (i0 >= n) return;
  uint64_t ctr = (offset >> 1) + (uint64_t)pair;
  uint4 r = philox4x32(ctr, seed);
  // Box-Muller in FP32 arithmetic (FP64 transcendentals are slow on this part); u1 uses
  // 32 random bits in (0, 1], so the radius reaches 6.7 sigma
  const float u1 = ((float)r.x + 1.0f) * 2.3283064365386963e-10f;
  const float u2 = (float)(r.z >> 8) * 5.9604644775390625e-08f;
  const float rad = sqrtf(-2.0f * logf(u1));
  float s, co;
  sincospif(2.0f * u2, &s, &co);
  out[i0] = (double)(rad * co);
  if (i0 + 1 < n) out[i0 + 1] = (double)(rad * s);
}

__global__ void k_fill_uniform(double* out, int64_t n, uint64_t seed, uint64_t offset) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint4 r = philox4x32(offset + (uint64_t)i, seed ^ 0x5bd1e995ull);
  out[i] = u53(r.x, r.y) - (1.0 / 9007199254740992.0);
}

// ======================================================================================
// host launchers
// ======================================================================================

static inline int launch_err(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    afq_set_error("%s: %s", what, cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

int check_smem_optin(size_t smem, const char* what) {
  int dev = 0, lim = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;  // no limit known here: the launch reports it
  }
  if (smem > (size_t)lim) {
    afq_set_error("%s: needs %zu bytes of shared memory per block, the device allows %d", what, smem, lim);
    return -2;
  }
  return 0;
}

cudaError_t raise_smem_limit(const void* kernel, size_t smem) {
  static std::mutex m;
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess || (size_t)a.maxDynamicSharedSizeBytes >= smem) return e;
  std::lock_guard<std::mutex> lock(m);
  e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess || (size_t)a.maxDynamicSharedSizeBytes >= smem) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <typename WT>
int launch_green(const afq_ctx_dev& c, const void* wu, const void* wd, double2* green,
                 double2* ovl, bool write_green, cudaStream_t st) {
  if (c.kmax <= 32) {
    launch_green_f64(c, wu, wd, green, ovl, write_green, st);
    return launch_err("green_f64");
  }
  const size_t smem = green_f64_smem(c.norb, c.kmax);
  if (int rc = check_smem_optin(smem, "green_overlap (norb x occupied orbitals too large)")) return rc;
  auto kfn = k_green_overlap<WT>;
  cudaError_t ea = raise_smem_limit((const void*)kfn, smem);
  if (ea != cudaSuccess) {
    afq_set_error("green_overlap: shared-memory attribute: %s", cudaGetErrorString(ea));
    return (int)ea;
  }
  {
    ProfScope _ps(K_GREEN, st);
    kfn<<<c.nw, 256, smem, st>>>(c, (const WT*)wu, (const WT*)wd, green, ovl, write_green ? 1 : 0);
  }
  return launch_err("green_overlap");
}

int launch_gemm_cr(bool b_kn, int M, int N, int K, const double2* A, long lda, const double* B,
                   long ldb, double2* C, long ldc, double2 alpha, cudaStream_t st) {
  dim3 grid((N + 63) / 64, (M + 63) / 64);
  ProfScope _ps(b_kn ? K_VHS : K_FB, st);
  if (b_kn)
    k_gemm_cr<true><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha);
  else
    k_gemm_cr<false><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, alpha);
  return launch_err("gemm_cr");
}

int launch_field_shifts(const afq_ctx_dev& c, const double* fields, const double2* fb,
                        double2* xt, double2* shift, double2* fbt, cudaStream_t st) {
  {
    ProfScope _ps(K_FIELD, st);
    launch_pdl(k_field_shifts, c.nw, 256, 0, st, c.nchol, sqrt(c.dt), fields, fb, c.mf, xt, shift, fbt);
  }
  return launch_err("field_shifts");
}

template <typename WT>
int launch_taylor_f64(const afq_ctx_dev& c, int w0, int nwc, const double2* vhs, void* wu, void* wd,
                      cudaStream_t st) {
  if (c.norb * c.kmax <= kTaylorSmall) {
    {
      ProfScope _ps(K_TAYLOR, st);
      launch_pdl(k_taylor_small, dim3(nwc, c.nslab), 256, 0, st, c, w0, vhs, (double2*)wu, (double2*)wd);
    }
    return launch_err("taylor_small");
  }
  size_t smem = 2 * (size_t)c.norb * c.kmax * sizeof(double2);
  auto kfn = k_taylor_f64<WT>;
  raise_smem_limit((const void*)kfn, smem);
  {
    ProfScope _ps(K_TAYLOR, st);
    kfn<<<dim3(nwc, c.nslab), 256, smem, st>>>(c, w0, vhs, (WT*)wu, (WT*)wd);
  }
  return launch_err("taylor_f64");
}

int launch_weights(const afq_ctx_dev& c, const double2* shift, const double2* fbt, int ntiles,
                   const double2* ovl_new, double2* ovl, double* weights, double* scalars,
                   cudaStream_t st, const int* status) {
  const WeightArgs g = {c.nw, ntiles, c.dt, c2(c.h0_prop_re, c.h0_prop_im), shift, fbt, ovl_new, ovl, weights, scalars, status};
  if (c.nw <= kWeightsCluster) {
    ProfScope _ps(K_WEIGHTS, st);
    const int per = (c.nw + kWeightsCtas - 1) / kWeightsCtas;
    launch_pdl(k_weights_pop, kWeightsCtas, (per + 31) / 32 * 32, 0, st, g);
    return launch_err("weights_pop");
  }
  {
    ProfScope _ps(K_WEIGHTS, st);
    // FP64 transcendentals per walker: 8 walkers per CTA spread them over the SMs' FP64 units
    launch_pdl(k_weights, (c.nw + 7) / 8, 8, 0, st, g);
  }
  {
    ProfScope _ps(K_WEIGHTS, st);
    launch_pdl(k_pop_control, 1, 1024, 0, st, g);
  }
  return launch_err("weights");
}

int launch_energy_f64(const afq_ctx_dev& c, int nchunks, int gchunk, const double2* green,
                      double2* epart, double2* energy, cudaStream_t st) {
  size_t smem = (size_t)c.ktot * sizeof(double2) + 2 * (size_t)c.kmax * c.kmax * sizeof(double2);
  raise_smem_limit((const void*)k_energy_f64_part, smem);
  {
    ProfScope _ps(K_ENERGY, st);
    k_energy_f64_part<<<dim3(c.nw, nchunks), 256, smem, st>>>(c, gchunk, green, epart);
  }
  int e = launch_err("energy_part");
  if (e) return e;
  {
    ProfScope _ps(K_ENERGY_FIN, st);
    k_energy_final<<<c.nw, 256, 0, st>>>(c, nchunks, green, epart, energy);
  }
  return launch_err("energy_final");
}

int launch_qr_f64(const afq_ctx_dev& c, void* wu, void* wd, cudaStream_t st, double2* rdiag) {
  size_t smem = 0;
  for (int s = 0; s < c.nslab; ++s)
    smem = std::max(smem, ((size_t)c.norb * (c.kslab[s] | 1) + 2 * c.kslab[s]) * sizeof(double2));
  raise_smem_limit((const void*)k_qr_f64, smem);
  {
    ProfScope _ps(K_QR, st);
    launch_pdl(k_qr_f64, dim3(c.nw, c.nslab), 32 * std::min(8, (c.norb + 31) / 32), smem, st, c, (double2*)wu, (double2*)wd, rdiag);
  }
  return launch_err("qr_f64");
}

template <typename WT>
int launch_sr(const afq_ctx_dev& c, const double* zeta, double* weights, double* cum, int32_t* idx,
              void* wu, void* wd, void* wcopy, cudaStream_t st) {
  {
    ProfScope _ps(K_SR, st);
    const int in_smem = c.nw * 8 <= 46 * 1024 ? 1 : 0;  // with the static part inside the default 48 KB
    launch_pdl(k_sr_indices, 1, 1024, in_smem ? c.nw * 8 : 0, st, c.nw, zeta, weights, cum, idx, in_smem);
  }
  int e = launch_err("sr_indices");
  if (e) return e;
  using CT = typename CplxOf<WT>::type;
  size_t off = 0;
  for (int s = 0; s < c.nslab; ++s) {
    void* w = s == 0 ? wu : wd;
    size_t elems = (size_t)c.norb * c.kslab[s];
    size_t bytes = elems * c.nw * sizeof(CT);
    char* cp = (char*)wcopy + off;
    cudaMemcpyAsync(cp, w, bytes, cudaMemcpyDeviceToDevice, st);
    {
      ProfScope _ps(K_SR, st);
      launch_pdl(k_gather_slab<WT>, c.nw, 256, 0, st, (int)elems, idx, (const WT*)cp, (WT*)w);
    }
    off += bytes;
  }
  return launch_err("sr_gather");
}

int launch_block_stats(const afq_ctx_dev& c, const double2* energy, const double* weights,
                       double* scalars, double* be, double* bw, cudaStream_t st, const int* status) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_block_stats, 1, 1024, 0, st, c.nw, c.dt, energy, weights, scalars, be, bw, status);
  }
  return launch_err("block_stats");
}

int launch_clamped_energies(const afq_ctx_dev& c, const double2* energy, const double* scalars,
                            double* out, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_clamped_energies, (c.nw + 255) / 256, 256, 0, st, c.nw, c.dt, energy, scalars, out);
  }
  return launch_err("clamped_energies");
}

int launch_cs_outlier(double* w1, double* w2, const double* e1, const double* e2, int nw,
                      double z_thresh, double* sums, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_cs_outlier, 1, 1024, 0, st, nw, z_thresh, w1, w2, e1, e2, sums);
  }
  return launch_err("cs_outlier");
}

int launch_fold_status(double* scalars, const int* status, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_fold_status, 1, 1, 0, st, scalars, status);
  }
  return launch_err("fold_status");
}

int launch_poison(long n, double2* out, const int* status, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_poison, (unsigned)std::min((n + 255) / 256, 1024l), 256, 0, st, n, out, status);
  }
  return launch_err("poison");
}

int launch_phaseless_begin(double* scalars, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_phaseless_begin, 1, 1, 0, st, scalars);
  }
  return launch_err("phaseless_begin");
}

int launch_phaseless_end(int nblk, double denom, const double* be, const double* bw,
                         double* scalars, double* energy, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_phaseless_end, 1, 32, 0, st, nblk, denom, be, bw, scalars, energy);
  }
  return launch_err("phaseless_end");
}

int launch_driver_update(const afq_ctx_dev& c, const double* weights, const double* energy,
                         double* scalars, double* wsum, cudaStream_t st) {
  {
    ProfScope _ps(K_STATS, st);
    launch_pdl(k_driver_update, 1, 1024, 0, st, c.nw, weights, energy, scalars, wsum);
  }
  return launch_err("driver_update");
}

int launch_fill_normal(double* out, int64_t n, uint64_t seed, uint64_t offset, cudaStream_t st) {
  if (offset & 1ull) {
    afq_set_error("afq_fill_normal: offset must be even");
    return -1;
  }
  int64_t pairs = (n + 1) / 2;
  if (pairs == 0) return 0;
  {
    ProfScope _ps(K_RNG, st);
    k_fill_normal<<<(unsigned)((pairs + 255) / 256), 256, 0, st>>>(out, n, seed, offset);
  }
  return launch_err("fill_normal");
}

int launch_fill_uniform(double* out, int64_t n, uint64_t seed, uint64_t offset, cudaStream_t st) {
  if (n == 0) return 0;
  {
    ProfScope _ps(K_RNG, st);
    k_fill_uniform<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n, seed, offset);
  }
  return launch_err("fill_uniform");
}

template int launch_green<double>(const afq_ctx_dev&, const void*, const void*, double2*, double2*, bool, cudaStream_t);
template int launch_taylor_f64<double>(const afq_ctx_dev&, int, int, const double2*, void*, void*, cudaStream_t);
template int launch_sr<double>(const afq_ctx_dev&, const double*, double*, double*, int32_t*, void*, void*, void*, cudaStream_t);
template int launch_sr<float>(const afq_ctx_dev&, const double*, double*, double*, int32_t*, void*, void*, void*, cudaStream_t);

}  // namespace afq
