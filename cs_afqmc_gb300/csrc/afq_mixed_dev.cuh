// What the mixed-precision kernels share: 16-bit splitting helpers and the plain-data view of the
// mixed state that is passed to them.
#pragma once
#include <cuda_fp16.h>

#include "afq_launch.cuh"
#include "afq_tc.cuh"

namespace afq {

// ---- 16-bit helpers -------------------------------------------------------------------

__device__ __forceinline__ uint16_t f2h(float x, bool bf) {
  return bf ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
}
__device__ __forceinline__ float h2f(uint16_t h, bool bf) {
  return bf ? __bfloat162float(__ushort_as_bfloat16(h)) : __half2float(__ushort_as_half(h));
}
// x ~ hi + lo with both parts 16-bit
__device__ __forceinline__ void split16(float x, bool bf, uint16_t& hi, uint16_t& lo) {
  hi = f2h(x, bf);
  lo = f2h(x - h2f(hi, bf), bf);
}
// byte offset of (row r, column k < 64) inside a [rows x 64] 16-bit tile, 128-byte swizzle
__device__ __forceinline__ uint32_t sw128(int r, int k) {
  return (uint32_t)(r * 128 + ((((k >> 3) ^ (r & 7)) << 4) | ((k & 7) << 1)));
}
// exact power of two 2^-e with 2^-e * amax in (0.5, 1]; 1 for amax == 0
__device__ __forceinline__ float pow2_scale(float amax) {
  if (!(amax > 0.0f) || !isfinite(amax)) return 1.0f;
  int e;
  frexpf(amax, &e);  // amax = m * 2^e, m in [0.5, 1)
  return ldexpf(1.0f, -e);
}

// Plain-data view of the mixed state passed to kernels.
struct MixedDev {
  int n, nq, nk, ldfb, ldg, nw, nchol, nslab, nblk, kfb, restricted_square, energy_mode;
  int o_slab[2], R[2], o_blk[2], ldkb[2];
  int bf16;
  double h0;
  const float* trial32[2];
  const float* rh1_32[2];
  uint16_t* g_fb[2];
  uint16_t* g_blk[2][2];  // per-block Green operand (two Green blocks only)
  uint16_t* wt[2][2];
  float* g_inv;
  double2* ene1;
};

// Green's function, overlap and operands (afq_green.cu). flags: kGreenG forms G, its 16-bit operands
// and the one-body energy, kGreenWT also the walker operand of the exp_h1 products.
constexpr int kGreenWT = 1, kGreenG = 2;
int launch_green_mixed(const MixedDev& md, const float2* wu, const float2* wd, double2* ovl, int flags,
                       cudaStream_t st);

}  // namespace afq
