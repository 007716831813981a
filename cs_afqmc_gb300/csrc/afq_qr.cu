// QR of FP32 walker slabs (propagation.py:251-253 -> linalg_utils.py:51-65): the LAPACK Householder
// factorisation (zgeqr2) and explicit Q (zung2r). Q overwrites W.

#include "afq_common.cuh"
#include "afq_kernels.cuh"
#include "afq_launch.cuh"
#include "afq_prof.cuh"

namespace afq {

// The order of every sum below is part of the mixed path's results: resampling compares sums of weights
// with the comb's teeth, and a weight that moves by one FP32 rounding exchanges a whole walker wherever a
// tooth lies that close (64 sites, 2048 walkers: with the slab in registers and its column sums split over
// eight row groups, one of twelve populations came out with another walker). So a
// column is summed as it always was, which costs 64 x 28 electrons, 2048 slabs 131 -> 174 us; 120 x 20, 1024 slabs
// 114 -> 127; 198 x 33, 256 slabs 161 -> 215; 60 x 10 and 60 x 8, 512 walkers 16 -> 30.

// v y of a rank-1 update and -tau v of a column of Q (the compiler's contractions of the first version)
AFQ_D float2 qr_vy(float2 v, float2 y) {
  return make_float2(fmaf(v.x, y.x, -__fmul_rn(v.y, y.y)), fmaf(v.y, y.x, __fmul_rn(v.x, y.y)));
}
AFQ_D float2 qr_mtau(float2 t, float2 v) {
  return make_float2(fmaf(t.y, v.y, -__fmul_rn(t.x, v.x)), fmaf(-t.y, v.x, -__fmul_rn(t.x, v.y)));
}
// a - f (v y)
AFQ_D float2 qr_update(float2 a, float2 f, float2 v, float2 y) { return sub_rn(a, mul_rn(f, qr_vy(v, y))); }

// tau, the scale of the reflector and the new diagonal element of a column with the element alpha on the
// diagonal and the squares xn below it (|alpha - b| >= |Im alpha|). FUSED: the divisor in one rounding
template <bool FUSED>
AFQ_D void qr_reflector(float2 alpha, float xn, float2& tau, float2& scl, float2& beta) {
  if (xn == 0.f && alpha.y == 0.f) {
    tau = make_float2(0.f, 0.f);
    scl = make_float2(1.f, 0.f);
    beta = alpha;
    return;
  }
  const float nrm = sqrtf(__fadd_rn(abs2_rn(alpha), xn)), b = alpha.x >= 0.f ? -nrm : nrm;
  tau = make_float2((b - alpha.x) / b, -alpha.y / b);
  const float dx = alpha.x - b, r = alpha.y / dx;
  const float den = FUSED ? fmaf(alpha.y, r, dx) : __fadd_rn(dx, __fmul_rn(alpha.y, r));
  scl = make_float2(1.f / den, -r / den);
  beta = make_float2(b, 0.f);
}

// One warp per slab with the slab in shared memory (row stride k | 1: conflict-free column walks) and only
// warp-level synchronisation. Column sums (the reflector applied to the trailing columns) are owned by
// lanes per column (qr_colsum); the rank-1 updates by lane = row. The squared norm below the diagonal
// is accumulated as a float pair.
// Slabs per CTA: one of four waits for room for all four (64 x 28, 2048 slabs: 12 instead of 14 on an SM and a second,
// nearly empty wave, 254 us instead of 174).
constexpr int kQrWarps = 1;

__host__ __device__ constexpr int qr_ld(int k) { return k | 1; }

// y[c] = sum_{r >= j} conj(A[r][c]) A[r][j] for c in (j, k) by one warp: lpc = the largest
// power of two with lpc * (k - j - 1) <= 32 lanes per column, each summing every lpc-th row,
// combined by shuffles (the rows of a column are the serial part otherwise).
__device__ __forceinline__ void qr_colsum(const float2* A, int ld, int m, int k, int j, int lane, float2* y) {
  const int nc = k - j - 1;
  if (nc <= 0) return;
  int lpc = 1;
  while (lpc * 2 * nc <= 32) lpc *= 2;
  const int col = j + 1 + lane / lpc, part = lane % lpc;
  const bool active = lane < lpc * nc;
  float yx = 0.f, yy = 0.f;
  if (active) {
#pragma unroll 4
    for (int r = j + part; r < m; r += lpc) {
      const float2 pr = mulc_rn(A[r * ld + col], A[r * ld + j]);
      yx = __fadd_rn(yx, pr.x);
      yy = __fadd_rn(yy, pr.y);
    }
  }
  for (int off = 1; off < lpc; off <<= 1) {  // lpc is warp-uniform
    yx += __shfl_xor_sync(0xffffffffu, yx, off);
    yy += __shfl_xor_sync(0xffffffffu, yy, off);
  }
  if (active && part == 0) y[col] = make_float2(yx, yy);
}

__global__ void __launch_bounds__(32 * kQrWarps) k_qr_warp(const afq_ctx_dev c, int s0, float2* __restrict__ w_up,
                                                          float2* __restrict__ w_dn) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char qsm_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wlk = blockIdx.x * kQrWarps + warp, s = s0 + blockIdx.y, m = c.norb, k = c.kslab[s];
  if (wlk >= c.nw) return;  // warp-level work only: no block barrier below
  const int ld = qr_ld(k);
  float2* A = reinterpret_cast<float2*>(qsm_raw) + (size_t)warp * ((size_t)m * ld + 64);
  float2* y = A + (size_t)m * ld;
  float2* tau = y + 32;
  float2* W = (s == 0 ? w_up : w_dn) + (size_t)wlk * m * k;
  for (int i = lane; i < m * k; i += 32) {
    const int r = i / k;
    A[r * ld + (i - r * k)] = W[i];
  }
  __syncwarp();
  // ---- factorisation
  for (int j = 0; j < k; ++j) {
    // squared norm below the diagonal as an unevaluated float pair (TwoSum per term and per
    // shuffle level): FP64-class accuracy without the FP64 pipe
    float xh = 0.f, xl = 0.f;
    for (int r = j + 1 + lane; r < m; r += 32) {
      const float a2 = abs2_rn(A[r * ld + j]), sum = xh + a2, bb = sum - xh;
      xl += (xh - (sum - bb)) + (a2 - bb);
      xh = sum;
    }
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_xor_sync(0xffffffffu, xh, off), ol = __shfl_xor_sync(0xffffffffu, xl, off);
      const float sum = xh + o, bb = sum - xh;
      xl += ol + ((xh - (sum - bb)) + (o - bb));
      xh = sum;
    }
    const float2 alpha = A[j * ld + j];
    const float xn = xh + xl;
    float2 t, scl, beta;
    qr_reflector<true>(alpha, xn, t, scl, beta);
    __syncwarp();
    for (int r = j + 1 + lane; r < m; r += 32) A[r * ld + j] = mul_rn(A[r * ld + j], scl);
    if (lane == 0) {
      A[j * ld + j] = make_float2(1.f, 0.f);
      tau[j] = t;
    }
    __syncwarp();
    qr_colsum(A, ld, m, k, j, lane, y);
    __syncwarp();
    const float2 ct = make_float2(t.x, -t.y);
    for (int r = j + lane; r < m; r += 32) {
      const float2 v = A[r * ld + j];
#pragma unroll 4
      for (int cc = j + 1; cc < k; ++cc)
        A[r * ld + cc] = qr_update(A[r * ld + cc], ct, v, y[cc]);
    }
    __syncwarp();
    if (lane == 0) A[j * ld + j] = beta;
    __syncwarp();
  }
  // ---- form Q (zung2r): columns from last to first
  for (int j = k - 1; j >= 0; --j) {
    const float2 t = tau[j];
    if (j < k - 1) {
      if (lane == 0) A[j * ld + j] = make_float2(1.f, 0.f);
      __syncwarp();
      qr_colsum(A, ld, m, k, j, lane, y);
      __syncwarp();
      for (int r = j + lane; r < m; r += 32) {
        const float2 v = A[r * ld + j];
#pragma unroll 4
        for (int cc = j + 1; cc < k; ++cc)
          A[r * ld + cc] = qr_update(A[r * ld + cc], t, v, y[cc]);
      }
      __syncwarp();
    }
    for (int r = j + 1 + lane; r < m; r += 32) A[r * ld + j] = qr_mtau(t, A[r * ld + j]);
    if (lane == 0) A[j * ld + j] = make_float2(1.f - t.x, -t.y);
    for (int r = lane; r < j; r += 32) A[r * ld + j] = make_float2(0.f, 0.f);
    __syncwarp();
  }
  for (int i = lane; i < m * k; i += 32) {
    const int r = i / k;
    W[i] = A[r * ld + (i - r * k)];
  }
}

// Slabs of more than 32 columns, or too long for four to share an SM: one CTA per (walker, slab).
AFQ_D float warp_sumf(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256) k_qr_householder(const afq_ctx_dev c, int s0, float2* __restrict__ w_up,
                                                        float2* __restrict__ w_dn) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wlk = blockIdx.x, s = s0;
  const int m = c.norb, k = c.kslab[s];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5,
            nwarp = nt >> 5;
  float2* A = reinterpret_cast<float2*>(smem_raw);  // [m][k]
  float2* y = A + (size_t)m * k;                // [k]
  float2* tau = y + k;                          // [k]
  __shared__ double red[32];
  __shared__ float2 sc_sh, beta_sh;
  float2* W = (s == 0 ? w_up : w_dn) + (size_t)wlk * m * k;
  for (int i = tid; i < m * k; i += nt) A[i] = W[i];
  __syncthreads();
  // ---- factorisation
  for (int j = 0; j < k; ++j) {
    double xnd = 0.0;
    for (int r = j + 1 + tid; r < m; r += nt) xnd += (double)abs2_rn(A[r * k + j]);
    xnd = block_sum(xnd, red);
    if (tid == 0) {
      const float2 alpha = A[j * k + j];
      qr_reflector<false>(alpha, (float)xnd, tau[j], sc_sh, beta_sh);
    }
    __syncthreads();
    const float2 scl = sc_sh;
    for (int r = j + 1 + tid; r < m; r += nt) A[r * k + j] = mul_rn(A[r * k + j], scl);
    if (tid == 0) A[j * k + j] = make_float2(1, 0);
    __syncthreads();
    // y[col] = sum_r conj(v[r]) A[r][col], col > j ; then A -= conj(tau) v y
    for (int col = j + 1 + wid; col < k; col += nwarp) {
      float yx = 0, yy = 0;
      for (int r = j + lane; r < m; r += 32) {
        const float2 pr = mulc_rn(A[r * k + col], A[r * k + j]);
        yx = __fadd_rn(yx, pr.x);
        yy = __fadd_rn(yy, pr.y);
      }
      yx = warp_sumf(yx);
      yy = warp_sumf(yy);
      if (lane == 0) y[col] = make_float2(yx, yy);
    }
    __syncthreads();
    const float2 ct = cconj(tau[j]);
    const int ncol = k - j - 1;
    if (ncol > 0) {
      for (int e = tid; e < (m - j) * ncol; e += nt) {
        const int r = j + e / ncol, col = j + 1 + e % ncol;
        A[r * k + col] = qr_update(A[r * k + col], ct, A[r * k + j], y[col]);
      }
    }
    __syncthreads();
    if (tid == 0) A[j * k + j] = beta_sh;
    __syncthreads();
  }
  // ---- form Q (zung2r): columns from last to first
  for (int j = k - 1; j >= 0; --j) {
    if (j < k - 1) {
      if (tid == 0) A[j * k + j] = make_float2(1, 0);
      __syncthreads();
      for (int col = j + 1 + wid; col < k; col += nwarp) {
        float yx = 0, yy = 0;
        for (int r = j + lane; r < m; r += 32) {
          const float2 pr = mulc_rn(A[r * k + col], A[r * k + j]);
          yx = __fadd_rn(yx, pr.x);
          yy = __fadd_rn(yy, pr.y);
        }
        yx = warp_sumf(yx);
        yy = warp_sumf(yy);
        if (lane == 0) y[col] = make_float2(yx, yy);
      }
      __syncthreads();
      const float2 t = tau[j];
      const int ncol = k - j - 1;
      for (int e = tid; e < (m - j) * ncol; e += nt) {
        const int r = j + e / ncol, col = j + 1 + e % ncol;
        A[r * k + col] = qr_update(A[r * k + col], t, A[r * k + j], y[col]);
      }
      __syncthreads();
    }
    const float2 t = tau[j];
    for (int r = j + 1 + tid; r < m; r += nt) A[r * k + j] = qr_mtau(t, A[r * k + j]);
    if (tid == 0) A[j * k + j] = make_float2(1 - t.x, -t.y);
    for (int r = tid; r < j; r += nt) A[r * k + j] = make_float2(0, 0);
    __syncthreads();
  }
  for (int i = tid; i < m * k; i += nt) W[i] = A[i];
}

int launch_qr_f32(const afq_ctx_dev& c, void* wu, void* wd, cudaStream_t st) {
  float2 *u = static_cast<float2*>(wu), *d = static_cast<float2*>(wd);
  auto warp_smem = [&](int s) {
    return kQrWarps * ((size_t)c.norb * qr_ld(c.kslab[s]) + 64) * sizeof(float2);
  };
  // longer slabs would leave an SM fewer than four warps; the second slab follows the first into the block form (the two
  // forms sum a column in different orders)
  auto fits = [&](int s) { return c.kslab[s] <= 32 && 4 / kQrWarps * warp_smem(s) <= 227 * 1024; };
  auto by_warp = [&](int s) { return fits(0) && fits(s); };
  const bool both = c.nslab == 2 && by_warp(0) && by_warp(1);  // one launch for both slabs
  ProfScope _ps(K_QR, st);
  for (int s = 0; s < (both ? 1 : c.nslab); ++s) {
    if (by_warp(s)) {
      const size_t smem = both && warp_smem(1) > warp_smem(0) ? warp_smem(1) : warp_smem(s);
      raise_smem_limit((const void*)k_qr_warp, smem);
      launch_pdl(k_qr_warp, dim3((c.nw + kQrWarps - 1) / kQrWarps, both ? 2 : 1), 32 * kQrWarps, smem, st, c, s, u, d);
    } else {
      const size_t smem = ((size_t)c.norb + 2) * c.kslab[s] * sizeof(float2);
      raise_smem_limit((const void*)k_qr_householder, smem);
      launch_pdl(k_qr_householder, c.nw, 256, smem, st, c, s, u, d);
    }
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    afq_set_error("qr_f32: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

}  // namespace afq
