// Green's function and overlap of FP64 walkers, one CTA per walker, up to 32 electrons per spin
// (wavefunctions.py:478-501 rhf, 658-692 uhf).

#include "afq_common.cuh"
#include "afq_kernels.cuh"
#include "afq_launch.cuh"
#include "afq_prof.cuh"

namespace afq {

constexpr int kG64Threads = 128;

// 1 / d for d in [0.5, 16): the FP32 reciprocal and two Newton steps r <- r + r (1 - d r), the
// relative error squared by each (2^-23, 2^-46, then rounding)
AFQ_D double rcp_scaled(double d) {
  double r = (double)__frcp_rn((float)d);
#pragma unroll
  for (int i = 0; i < 2; ++i) r = fma(r, fma(-d, r, 1.0), r);
  return r;
}

// What bounds it: the FP64 units (1.8 FMAs per cycle and SM): per walker and slab 2 n o^2 FMAs for
// S = C^T W, 4 OM^3 for the inverse, 4 n o^2 for G = W S^-1, that is 188 k cycles at norb 120 with
// 20 electrons. The phases therefore only have to keep a few warps of FP64 work ready at any time:
//  * S in 2 x 2 register blocks, the orbitals dealt to the threads that the blocks leave over;
//  * Gauss-Jordan in registers, a matrix row per lane, OM <= 16 with both slabs in the two
//    halves of one warp (a half-empty FP64 instruction costs as much as a full one), otherwise a
//    warp per slab; implicit partial pivoting and columns that rotate by one register a step, as
//    in the mixed-precision kernel (afq_green.cu);
//  * G with one walker row per thread in registers, stored straight to its [i][p] layout.
template <int OM>
__global__ void __launch_bounds__(kG64Threads, OM <= 20 ? 3 : 2)
    k_green_f64(const afq_ctx_dev c, const double2* __restrict__ w_up, const double2* __restrict__ w_dn,
                double2* __restrict__ green, double2* __restrict__ overlap, int write_green) {
  pdl_enter();
  constexpr int NT = kG64Threads, NW = NT / 32;
  constexpr bool HALF = OM <= 16;
  __shared__ double2 Pt[4 * NT];
  __shared__ __align__(16) double2 Sm[2][OM * (OM + 1)];  // S, then S^-1 [k][i] with row stride OM
  __shared__ __align__(16) double2 prow[2][2][OM];
  __shared__ double2 pivv[2][OM];
  __shared__ int piv_s[2][OM], odd_s[2];
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = c.norb;
  const double2* Wg[2] = {w_up + (size_t)w * n * c.kslab[0], c.nslab == 2 ? w_dn + (size_t)w * n * c.kslab[1] : nullptr};

  for (int s = 0; s < c.nslab; ++s) {
    const int o = c.nocc_slab[s], nb = (o + 1) >> 1, nbb = nb * nb;
    const double* __restrict__ C = c.trial[s];
    const double2* __restrict__ W = Wg[s];
    for (int b0 = 0; b0 < nbb; b0 += NT) {  // one pass up to 22 electrons
      const int nbp = min(nbb - b0, NT), ps_n = NT / nbp, ps = tid / nbp, b = b0 + tid - ps * nbp;
      const int i0 = 2 * (b / nb), k0 = 2 * (b % nb);
      const bool i1 = i0 + 1 < o, k1 = k0 + 1 < o;
      if (ps < ps_n) {
        double2 a00 = c2(0, 0), a01 = a00, a10 = a00, a11 = a00;
#pragma unroll 4
        for (int p = ps; p < n; p += ps_n) {
          const double c0 = __ldg(C + p * o + i0), c1 = i1 ? __ldg(C + p * o + i0 + 1) : 0.0;
          const double2 x = __ldg(W + (size_t)p * o + k0), y = k1 ? __ldg(W + (size_t)p * o + k0 + 1) : c2(0.0, 0.0);
          a00 = c2(fma(c0, x.x, a00.x), fma(c0, x.y, a00.y));
          a01 = c2(fma(c0, y.x, a01.x), fma(c0, y.y, a01.y));
          a10 = c2(fma(c1, x.x, a10.x), fma(c1, x.y, a10.y));
          a11 = c2(fma(c1, y.x, a11.x), fma(c1, y.y, a11.y));
        }
        Pt[tid] = a00;
        Pt[NT + tid] = a01;
        Pt[2 * NT + tid] = a10;
        Pt[3 * NT + tid] = a11;
      }
      __syncthreads();
      for (int e = tid; e < 4 * nbp; e += NT) {
        const int q = e / nbp, bb = e - q * nbp;
        double2 v = Pt[q * NT + bb];
        for (int r = 1; r < ps_n; ++r) v = cadd(v, Pt[q * NT + r * nbp + bb]);
        const int i = 2 * ((b0 + bb) / nb) + (q >> 1), k = 2 * ((b0 + bb) % nb) + (q & 1);
        if (i < o && k < o) Sm[s][i * (OM + 1) + k] = v;
      }
      __syncthreads();
    }
    for (int e = tid; e < OM * OM; e += NT) {  // identity beyond the electrons
      const int i = e / OM, k = e - i * OM;
      if (i >= o || k >= o) Sm[s][i * (OM + 1) + k] = c2(i == k ? 1.0 : 0.0, 0.0);
    }
  }
  __syncthreads();

  const bool one_warp = HALF && c.nslab == 2;
  if (warp < (one_warp ? 1 : c.nslab)) {
    const int s = one_warp ? lane >> 4 : warp, row = one_warp ? lane & 15 : lane;
    const unsigned mask = one_warp ? (lane < 16 ? 0xffffu : 0xffff0000u) : 0xffffffffu;
    // pivots: the electrons (with two slabs in the warp, the larger count; the identity fills up)
    const int steps = one_warp ? max(c.nocc_slab[0], c.nocc_slab[1]) : c.nocc_slab[s];
    double2 a[OM];
    bool used = row >= steps;
    int step = 0;
#pragma unroll
    for (int k = 0; k < OM; ++k) a[k] = row < OM ? Sm[s][row * (OM + 1) + k] : c2(0.0, 0.0);
    unsigned open = steps == 32 ? 0xffffffffu : (1u << steps) - 1u;  // rows without a pivot
    int odd = 0;
#pragma unroll 1
    for (int j = 0; j < steps; ++j) {  // column c ends in register OM - steps + c
      double2* pw = prow[s][j & 1];
      // |re| + |im| of the candidates by the high word, the row index in its low bits
      const unsigned mag = (unsigned)__double2hiint(fabs(a[0].x) + fabs(a[0].y));
      const unsigned key = used ? 0u : ((mag & ~31u) | (unsigned)(31 - row));
      const int pr = 31 - (int)(__reduce_max_sync(mask, key) & 31u);
      const bool own = row == pr;
      if (own) {
        used = true;
        step = j;
        pivv[s][j] = a[0];
        piv_s[s][j] = pr;
#pragma unroll
        for (int k = 0; k < OM; ++k) pw[k] = a[k];
#pragma unroll
        for (int k = 1; k < OM; ++k) a[k] = c2(0.0, 0.0);
      }
      __syncwarp();
      const double2 pv = pw[0];
      // 1 / pv = conj(pv) / |pv|^2 with pv scaled by a power of two first
      const int ef = min(max((int)((unsigned)__double2hiint(fmax(fabs(pv.x), fabs(pv.y))) >> 20), 1), 2045);
      const double sc = __hiloint2double((2046 - ef) << 20, 0);
      const double px = pv.x * sc, py = pv.y * sc, d2 = fma(px, px, py * py);
      const double dd = (d2 >= 0.5 && d2 < 16.0 ? rcp_scaled(d2) : 1.0 / d2) * sc;  // else: zero, denormal or not finite
      const double2 inv = c2(px * dd, -py * dd);
      const double2 t = cmul(a[0], inv);
      const double2 f = own ? inv : c2(-t.x, -t.y);
#pragma unroll
      for (int k = 1; k < OM; ++k) {
        const double2 v = pw[k];
        a[k - 1].x = fma(f.x, v.x, fma(-f.y, v.y, a[k].x));
        a[k - 1].y = fma(f.x, v.y, fma(f.y, v.x, a[k].y));
      }
      a[OM - 1] = f;
      odd += __popc(open & ((1u << pr) - 1u));
      open &= ~(1u << pr);
    }
    __syncwarp();
    if (row == 0) odd_s[s] = odd;
    if (write_green && row < OM) {
#pragma unroll
      for (int k = 0; k < OM; ++k) {
        if (row >= steps) Sm[s][row * OM + k] = c2(0.0, 0.0);
        else if (k >= OM - steps) Sm[s][step * OM + piv_s[s][k - (OM - steps)]] = a[k];
      }
    }
  }
  __syncthreads();
  if (warp == NW - 1) {  // the product of the pivots, while the others form G
    double2 det = c2(1.0, 0.0);
    for (int s = 0; s < c.nslab; ++s) {
      double2 pd = lane < c.nocc_slab[s] ? pivv[s][lane] : c2(1.0, 0.0);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        pd = cmul(pd, c2(__shfl_xor_sync(0xffffffffu, pd.x, off), __shfl_xor_sync(0xffffffffu, pd.y, off)));
      det = cmul(det, (odd_s[s] & 1) ? c2(-pd.x, -pd.y) : pd);
    }
    if (lane == 0 && overlap) overlap[w] = c.nslab == 1 && c.restricted_square ? cmul(det, det) : det;
  }
  if (!write_green) return;
  double2* Gw = green + (size_t)w * c.ktot;
  for (int s = 0; s < c.nslab; ++s) {
    const int o = c.nocc_slab[s];
    double2* G = Gw + (c.nspin_g == 2 && s == 1 ? (size_t)c.nocc_slab[0] * n : 0);
    const bool sum = c.nspin_g == 1 && s == 1;  // RHF two slabs: G_up + G_dn
    for (int p = tid; p < n; p += NT) {
      double2 wr[OM];
#pragma unroll
      for (int k = 0; k < OM; ++k) wr[k] = k < o ? __ldg(Wg[s] + (size_t)p * o + k) : c2(0.0, 0.0);
#pragma unroll 1
      for (int i = 0; i < o; ++i) {
        double2 g0 = c2(0, 0), g1 = g0;
#pragma unroll
        for (int k = 0; k < OM; k += 2)
          if (k < o) {
            const double2 s0 = Sm[s][k * OM + i], s1 = Sm[s][(k + 1) * OM + i];
            g0 = c2(fma(wr[k].x, s0.x, fma(-wr[k].y, s0.y, g0.x)), fma(wr[k].x, s0.y, fma(wr[k].y, s0.x, g0.y)));
            g1 = c2(fma(wr[k + 1].x, s1.x, fma(-wr[k + 1].y, s1.y, g1.x)),
                    fma(wr[k + 1].x, s1.y, fma(wr[k + 1].y, s1.x, g1.y)));
          }
        double2 g = cadd(g0, g1);
        if (sum) g = cadd(g, G[(size_t)i * n + p]);
        G[(size_t)i * n + p] = g;
      }
    }
  }
}

int launch_green_f64(const afq_ctx_dev& c, const void* wu, const void* wd, double2* green, double2* ovl,
                     bool write_green, cudaStream_t st) {
  ProfScope _ps(K_GREEN, st);
  const double2 *u = (const double2*)wu, *d = (const double2*)wd;
  const int wg = write_green ? 1 : 0;
  switch ((c.kmax + 3) / 4) {
    case 1: launch_pdl(k_green_f64<4>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 2: launch_pdl(k_green_f64<8>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 3: launch_pdl(k_green_f64<12>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 4: launch_pdl(k_green_f64<16>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 5: launch_pdl(k_green_f64<20>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 6: launch_pdl(k_green_f64<24>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    case 7: launch_pdl(k_green_f64<28>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
    default: launch_pdl(k_green_f64<32>, c.nw, kG64Threads, 0, st, c, u, d, green, ovl, wg); break;
  }
  return 0;
}

}  // namespace afq
