// QR of FP32 walker slabs with the slab in registers (propagation.py:251-253 -> linalg_utils.py:51-65):
// the LAPACK Householder factorisation (zgeqr2) and explicit Q (zung2r), up to 40 electrons per slab.

#include <type_traits>
#include <utility>

#include "afq_common.cuh"
#include "afq_kernels.cuh"
#include "afq_launch.cuh"
#include "afq_prof.cuh"

namespace afq {

// A warp's lanes are eight row groups by four column groups: lane (g, cg) holds rows base + 8 r + g and
// columns 4 i + cg of the slab. Step j broadcasts column j from its column group with shuffles, sums its
// norm over the row groups, scales it into the reflector v, forms v^H a_c for every trailing column in
// the same way and updates. Slabs of more than 64 rows are split between the warps of the CTA, which
// exchange their sums through shared memory with two barriers a step. Nothing else leaves the
// registers: the reflectors stay in place as in zgeqr2, and zung2r runs backwards over them.
//
// What bounds it: the chain of a step (norm, square root, divisions, shuffles: some 2000 cycles) over the
// two to four slabs that an SM's scheduler has registers for. Fewer registers, more slabs: lost to the
// spills (28 columns: 125 us at 184 registers and 160 at 144, 118 without a limit, in a form that fused the
// update into two roundings an element; the product is rounded first now, which keeps the error of Q at
// what it was: 7.1e-7 at 120 x 20, 1.04e-6 at 198 x 33 against quadruple precision, and costs 8%).
// Measured against a slab per warp, or per CTA above 32 columns, in shared memory: 64 x 28 electrons, 2048
// slabs 305 -> 131 us; 120 x 20, 1024 slabs 159 -> 114 us; 198 x 33, 256 slabs 219 -> 161 us; 60 x 10 and
// 60 x 8, 512 walkers 45 us for one spin -> 16 us for both; 53 x 8, 64 slabs 26 -> 10 us.
//
// FP64 walkers keep the slab in shared memory (k_qr_f64): their units take some 18 cycles for a warp
// instruction whatever its lanes do, and with eight lanes along the rows instead of 32 there are more of
// them. Measured in this form at 256 walkers of two slabs, against a warp per slab in shared memory: 100 x 20 electrons
// 559 -> 919 us, 60 x 36 959 -> 1835 us.
constexpr int kQrRows = 8;   // rows per lane: 64 a warp
constexpr int kQrWarps = 8;  // warps per CTA at most: 255 registers a thread

struct QrArgs {
  float2* w[2];
  int k[2];
  int m;
};

// sum of squares as an unevaluated pair (TwoSum per term): FP64-class accuracy without the FP64 units
struct QrNorm {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(float o, float ol) {
    const float s = h + o, b = s - h;
    l += ol + ((h - (s - b)) + (o - b));
    h = s;
  }
};

__device__ __forceinline__ float qr_shfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }

template <class F, class G, int... I>
__device__ __forceinline__ void qr_blocks(F& factor, G& form, std::integer_sequence<int, I...>) {
  (factor(std::integral_constant<int, I>{}), ...);
  (form(std::integral_constant<int, (int)sizeof...(I) - 1 - I>{}), ...);
}

template <int NCL, bool MULTI>
__global__ void __launch_bounds__(MULTI ? 32 * kQrWarps : 32) k_qr_regs(const QrArgs q) {
  constexpr int RL = kQrRows, NW = MULTI ? kQrWarps : 1;
  __shared__ float2 part[2][NW][MULTI ? 4 * NCL : 1];  // column sums of each warp
  __shared__ float4 pnorm[NW];                         // its share of the norm, and the diagonal element
  pdl_enter();
  const int s = blockIdx.y, m = q.m, k = q.k[s], lane = threadIdx.x & 31, warp = MULTI ? threadIdx.x >> 5 : 0;
  const int g = lane >> 2, cg = lane & 3, row0 = warp * 8 * RL + g, nwarp = MULTI ? blockDim.x >> 5 : 1;
  float2* W = q.w[s] + (size_t)blockIdx.x * m * k;
  float ax[RL][NCL], ay[RL][NCL], tx[NCL], ty[NCL];
#pragma unroll
  for (int r = 0; r < RL; ++r)
#pragma unroll
    for (int c = 0; c < NCL; ++c) {
      const int row = row0 + 8 * r, col = 4 * c + cg;
      const float2 v = row < m && col < k ? W[(size_t)row * k + col] : make_float2(0.f, 0.f);
      ax[r][c] = v.x;
      ay[r][c] = v.y;
    }
  int par = 0;

  // sums over all rows of y[c], c >= B
  auto reduce = [&](auto bc, float* yx, float* yy) {
    constexpr int B = decltype(bc)::value;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
#pragma unroll
      for (int c = B; c < NCL; ++c) {
        yx[c] += __shfl_xor_sync(0xffffffffu, yx[c], o);
        yy[c] += __shfl_xor_sync(0xffffffffu, yy[c], o);
      }
    if constexpr (MULTI) {
      if (g == 0) {
#pragma unroll
        for (int c = B; c < NCL; ++c) part[par][warp][4 * c + cg] = make_float2(yx[c], yy[c]);
      }
      __syncthreads();
#pragma unroll
      for (int c = B; c < NCL; ++c) yx[c] = yy[c] = 0.f;
      for (int w = 0; w < nwarp; ++w)
#pragma unroll
        for (int c = B; c < NCL; ++c) {
          const float2 p = part[par][w][4 * c + cg];
          yx[c] += p.x;
          yy[c] += p.y;
        }
      par ^= 1;  // a warp that is still reading is at most one reduction behind
    }
  };

  // ---- factorisation: steps j = 4 b + ii
  auto factor = [&](auto bc) {
    constexpr int B = decltype(bc)::value, WJ = (B / 2) / RL, RJ = (B / 2) % RL, R0 = MULTI ? 0 : RJ;
#pragma unroll 1
    for (int ii = 0; ii < 4; ++ii) {
      const int j = 4 * B + ii;
      if (j >= k) break;
      const int src = (lane & ~3) | ii, gj = (4 * B) % 8 + ii;
      float vx[RL], vy[RL], yx[NCL], yy[NCL];
      QrNorm nrm;
      float2 al = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = R0; r < RL; ++r) {
        const float bx = qr_shfl(ax[r][B], src), by = qr_shfl(ay[r][B], src);
        if (r == RJ) al = make_float2(qr_shfl(bx, 4 * gj), qr_shfl(by, 4 * gj));
        const bool below = row0 + 8 * r > j;
        vx[r] = below ? bx : 0.f;
        vy[r] = below ? by : 0.f;
        nrm.add(vx[r] * vx[r] + vy[r] * vy[r], 0.f);
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1)
        nrm.add(__shfl_xor_sync(0xffffffffu, nrm.h, o), __shfl_xor_sync(0xffffffffu, nrm.l, o));
      if constexpr (MULTI) {
        // the column sums' barrier below stands between these reads and the next step's writes
        if (lane == 0) pnorm[warp] = make_float4(nrm.h, nrm.l, al.x, al.y);
        __syncthreads();
        al = make_float2(pnorm[WJ].z, pnorm[WJ].w);
        nrm.h = nrm.l = 0.f;
        for (int w = 0; w < nwarp; ++w) nrm.add(pnorm[w].x, pnorm[w].y);
      }
      const float xn = nrm.h + nrm.l;
      float2 t = make_float2(0.f, 0.f), scl = make_float2(1.f, 0.f);
      if (!(xn == 0.f && al.y == 0.f)) {
        const float n2 = sqrtf(al.x * al.x + al.y * al.y + xn), b = al.x >= 0.f ? -n2 : n2;
        t = make_float2((b - al.x) / b, -al.y / b);
        scl = cdiv(make_float2(1.f, 0.f), make_float2(al.x - b, al.y));
      }
      if (cg == ii) {
        tx[B] = t.x;
        ty[B] = t.y;
      }
#pragma unroll
      for (int c = B; c < NCL; ++c) yx[c] = yy[c] = 0.f;
#pragma unroll
      for (int r = R0; r < RL; ++r) {
        const float2 v = row0 + 8 * r == j ? make_float2(1.f, 0.f) : cmul(make_float2(vx[r], vy[r]), scl);
        vx[r] = v.x;
        vy[r] = v.y;
#pragma unroll
        for (int c = B; c < NCL; ++c) {
          yx[c] = fmaf(v.x, ax[r][c], fmaf(v.y, ay[r][c], yx[c]));
          yy[c] = fmaf(v.x, ay[r][c], fmaf(-v.y, ax[r][c], yy[c]));
        }
      }
      reduce(bc, yx, yy);
      // a_c -= conj(tau) v (v^H a_c), columns behind j only
#pragma unroll
      for (int c = B; c < NCL; ++c) {
        const float2 p = cmul(make_float2(t.x, -t.y), make_float2(yx[c], yy[c]));
        yx[c] = p.x;
        yy[c] = p.y;
      }
#pragma unroll
      for (int r = R0; r < RL; ++r) {
        if (cg == ii && row0 + 8 * r > j) {
          ax[r][B] = vx[r];
          ay[r][B] = vy[r];
        }
        if (cg > ii) {
          ax[r][B] -= fmaf(vx[r], yx[B], -vy[r] * yy[B]);
          ay[r][B] -= fmaf(vx[r], yy[B], vy[r] * yx[B]);
        }
#pragma unroll
        for (int c = B + 1; c < NCL; ++c) {
          ax[r][c] -= fmaf(vx[r], yx[c], -vy[r] * yy[c]);
          ay[r][c] -= fmaf(vx[r], yy[c], vy[r] * yx[c]);
        }
      }
    }
  };

  // ---- Q = H_0 .. H_{k-1} I: column j becomes e_j - tau v, after H_j acts on the columns behind it
  auto form = [&](auto bc) {
    constexpr int B = decltype(bc)::value, RJ = (B / 2) % RL, R0 = MULTI ? 0 : RJ;
#pragma unroll 1
    for (int ii = 3; ii >= 0; --ii) {
      const int j = 4 * B + ii;
      if (j >= k) continue;
      const int src = (lane & ~3) | ii;
      float vx[RL], vy[RL], yx[NCL], yy[NCL];
#pragma unroll
      for (int c = B; c < NCL; ++c) yx[c] = yy[c] = 0.f;
#pragma unroll
      for (int r = R0; r < RL; ++r) {
        const float bx = qr_shfl(ax[r][B], src), by = qr_shfl(ay[r][B], src);
        const int row = row0 + 8 * r;
        vx[r] = row > j ? bx : row == j ? 1.f : 0.f;
        vy[r] = row > j ? by : 0.f;
#pragma unroll
        for (int c = B; c < NCL; ++c) {
          yx[c] = fmaf(vx[r], ax[r][c], fmaf(vy[r], ay[r][c], yx[c]));
          yy[c] = fmaf(vx[r], ay[r][c], fmaf(-vy[r], ax[r][c], yy[c]));
        }
      }
      reduce(bc, yx, yy);
      const float2 t = make_float2(qr_shfl(tx[B], ii), qr_shfl(ty[B], ii));
#pragma unroll
      for (int c = B; c < NCL; ++c) {
        const float2 p = cmul(t, make_float2(yx[c], yy[c]));
        yx[c] = p.x;
        yy[c] = p.y;
      }
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        if (r < R0) {
          if (cg == ii) ax[r][B] = ay[r][B] = 0.f;
          continue;
        }
        if (cg == ii) {
          const float2 p = cmul(t, make_float2(vx[r], vy[r]));
          ax[r][B] = (row0 + 8 * r == j ? 1.f : 0.f) - p.x;
          ay[r][B] = -p.y;
        }
        if (cg > ii) {
          ax[r][B] -= fmaf(vx[r], yx[B], -vy[r] * yy[B]);
          ay[r][B] -= fmaf(vx[r], yy[B], vy[r] * yx[B]);
        }
#pragma unroll
        for (int c = B + 1; c < NCL; ++c) {
          ax[r][c] -= fmaf(vx[r], yx[c], -vy[r] * yy[c]);
          ay[r][c] -= fmaf(vx[r], yy[c], vy[r] * yx[c]);
        }
      }
    }
  };

  qr_blocks(factor, form, std::make_integer_sequence<int, NCL>{});

#pragma unroll
  for (int r = 0; r < RL; ++r)
#pragma unroll
    for (int c = 0; c < NCL; ++c) {
      const int row = row0 + 8 * r, col = 4 * c + cg;
      if (row < m && col < k) W[(size_t)row * k + col] = make_float2(ax[r][c], ay[r][c]);
    }
}

template <int NCL>
static void launch_regs(const QrArgs& q, int nw, int nslab, cudaStream_t st) {
  const int nwarp = (q.m + 8 * kQrRows - 1) / (8 * kQrRows);
  ProfScope _ps(K_QR, st);
  if (nwarp == 1)
    launch_pdl(k_qr_regs<NCL, false>, dim3(nw, nslab), 32, 0, st, q);
  else
    launch_pdl(k_qr_regs<NCL, true>, dim3(nw, nslab), 32 * nwarp, 0, st, q);
}

int launch_qr_f32(const afq_ctx_dev& c, void* wu, void* wd, cudaStream_t st) {
  const QrArgs q = {{static_cast<float2*>(wu), static_cast<float2*>(wd)}, {c.kslab[0], c.nslab > 1 ? c.kslab[1] : 0}, c.norb};
  const int ncl = ((q.k[0] > q.k[1] ? q.k[0] : q.k[1]) + 3) / 4;
  if (q.m > 8 * kQrRows * kQrWarps || ncl > 10) {
    afq_set_error("FP32 QR: at most %d orbitals and 40 electrons per spin", 8 * kQrRows * kQrWarps);
    return -1;
  }
  switch (ncl) {
    case 0:
    case 1: launch_regs<1>(q, c.nw, c.nslab, st); break;
    case 2: launch_regs<2>(q, c.nw, c.nslab, st); break;
    case 3: launch_regs<3>(q, c.nw, c.nslab, st); break;
    case 4: launch_regs<4>(q, c.nw, c.nslab, st); break;
    case 5: launch_regs<5>(q, c.nw, c.nslab, st); break;
    case 6: launch_regs<6>(q, c.nw, c.nslab, st); break;
    case 7: launch_regs<7>(q, c.nw, c.nslab, st); break;
    case 8: launch_regs<8>(q, c.nw, c.nslab, st); break;
    case 9: launch_regs<9>(q, c.nw, c.nslab, st); break;
    default: launch_regs<10>(q, c.nw, c.nslab, st); break;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    afq_set_error("qr_f32: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

}  // namespace afq
