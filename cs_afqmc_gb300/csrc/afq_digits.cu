// Sliced FP64 contractions: slicing kernels, the digit GEMM and its launchers (afq_digits.cuh).

#include <math.h>

#include <algorithm>

#include "afq_common.cuh"
#include "afq_digits.cuh"
#include "afq_launch.cuh"
#include "afq_prof.cuh"
#include "afq_ptx.cuh"

namespace afq {

// ======================================================================================
// digits
// ======================================================================================

// Position of the leading bit of |x| above 2^-1074 (0 for zero); 2098 for NaN and infinities
AFQ_D unsigned dig_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  const unsigned ef = (unsigned)(b >> 52);
  return ef ? ef + 51u : 63u - (unsigned)__clzll((long long)(b | 1ull));
}

// exponent e with |x| < 2^e for every x of a row whose largest key is `key`
AFQ_D int dig_row_exp(unsigned key) { return key >= 2098u ? kDigBad : (int)key - 1073; }

// x 2^(56 - e) rounded to an integer (|x| < 2^e); e = kDigBad gives 0
AFQ_D long long dig_fixed(double x, int e) {
  const long long b = __double_as_longlong(x);
  const int ef = (int)((b >> 52) & 0x7ff);
  long long m = b & 0xfffffffffffffll;
  if (ef) m |= 1ll << 52;
  const int sh = 4 + (ef ? ef : 1) - 1023 - e;  // m << sh < 2^56
  long long q;
  if (e == kDigBad || sh < -58) q = 0;
  else if (sh >= 0) q = m << sh;
  else q = (m + (1ll << (-sh - 1))) >> -sh;
  return b < 0 ? -q : q;
}

// sum_{k<7} 64 * 128^k: makes the seven lower digits of q + offset non-negative
constexpr long long kDigOffset = 64ll * (((1ll << 49) - 1) / 127);

// Digit j of q times its weight as an FP32 value (exact; its upper 16 bits are the BF16 value).
template <int J>
AFQ_D unsigned dig_f32(long long qo) {
  constexpr float s = 1.0f / (float)(1ll << (7 + 7 * J));
  if (J == 0) {
    const int u = (int)(qo >> 49) + 128;
    return __float_as_uint(fmaf(__uint_as_float(0x4B000000u | (unsigned)u), s, -(8388608.0f + 128.0f) * s));
  }
  const unsigned u = (unsigned)(qo >> (49 - 7 * J)) & 127u;
  return __float_as_uint(fmaf(__uint_as_float(0x4B000000u | u), s, -(8388608.0f + 64.0f) * s));
}

template <int J>
AFQ_D uint4 dig_chunk(const long long (&qo)[8], unsigned flip) {
  uint4 w;
  w.x = __byte_perm(dig_f32<J>(qo[0]), dig_f32<J>(qo[1]), 0x7632) ^ flip;
  w.y = __byte_perm(dig_f32<J>(qo[2]), dig_f32<J>(qo[3]), 0x7632) ^ flip;
  w.z = __byte_perm(dig_f32<J>(qo[4]), dig_f32<J>(qo[5]), 0x7632) ^ flip;
  w.w = __byte_perm(dig_f32<J>(qo[6]), dig_f32<J>(qo[7]), 0x7632) ^ flip;
  return w;
}

// Writes the eight digits of eight consecutive k of one row. base: the row tile's K block,
// row: within the tile, half: k & 8. flip = 0x80008000 stores the negated values as well or
// instead.
AFQ_D void dig_store(const long long (&q)[8], unsigned char* base, int tr, int row, int half, unsigned flip = 0) {
  long long qo[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) qo[i] = q[i] + kDigOffset;
  unsigned char* r = base + row * 128;
  const int x = row & 7;
  auto at = [&](int j) -> uint4* {
    return reinterpret_cast<uint4*>(r + (j >> 2) * (tr * 128) + (((((j & 3) << 1) | half) ^ x) << 4));
  };
  *at(0) = dig_chunk<0>(qo, flip);
  *at(1) = dig_chunk<1>(qo, flip);
  *at(2) = dig_chunk<2>(qo, flip);
  *at(3) = dig_chunk<3>(qo, flip);
  *at(4) = dig_chunk<4>(qo, flip);
  *at(5) = dig_chunk<5>(qo, flip);
  *at(6) = dig_chunk<6>(qo, flip);
  *at(7) = dig_chunk<7>(qo, flip);
}

AFQ_D unsigned char* dig_block(unsigned char* d, int row, int kblk, int kb, int tr) {
  return d + ((size_t)(row / tr) * kb + kblk) * ((size_t)tr * 256);
}

AFQ_D unsigned block_max_u(unsigned v, unsigned* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[wid] = v;
  __syncthreads();
  unsigned m = red[0];
  for (int i = 1; i < nw; ++i) m = max(m, red[i]);
  return m;
}

// One CTA per complex row: lane pairs hold the two halves of a K block, so each 32-byte
// sector of the digit tile is written by one instruction.
__global__ void __launch_bounds__(128) k_dig_cplx_rows(const double2* __restrict__ src, long ld, int K, int kb,
                                                       double mul, unsigned char* __restrict__ d,
                                                       int* __restrict__ e) {
  pdl_enter();
  __shared__ unsigned red[2][4];
  const int m = blockIdx.x;
  const double2* s = src + (size_t)m * ld;
  unsigned er = 0, ei = 0;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const double2 v = s[k];
    er = max(er, dig_key(v.x * mul));
    ei = max(ei, dig_key(v.y * mul));
  }
  const int xr = dig_row_exp(block_max_u(er, red[0])), xi = dig_row_exp(block_max_u(ei, red[1]));
  if (threadIdx.x == 0) {
    e[2 * m] = xr;
    e[2 * m + 1] = xi;
  }
  const int row = (2 * m) & (kDigTile - 1);
  for (int t = threadIdx.x; t < 2 * kb; t += blockDim.x) {
    long long qr[8], qi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = 8 * t + i;
      const double2 v = k < K ? s[k] : c2(0.0, 0.0);
      qr[i] = dig_fixed(v.x * mul, xr);
      qi[i] = dig_fixed(v.y * mul, xi);
    }
    unsigned char* b = dig_block(d, 2 * m, t >> 1, kb, kDigTile);
    dig_store(qr, b, kDigTile, row, t & 1);
    dig_store(qi, b, kDigTile, row + 1, t & 1);
  }
}

__global__ void __launch_bounds__(128) k_dig_real_rows(const double* __restrict__ src, long ld, int K, int kb, int tr,
                                                       int row0, unsigned char* __restrict__ d,
                                                       int* __restrict__ e) {
  __shared__ unsigned red[4];
  const int m = row0 + blockIdx.x;
  const double* s = src + (size_t)blockIdx.x * ld;
  unsigned er = 0;
  for (int k = threadIdx.x; k < K; k += blockDim.x) er = max(er, dig_key(s[k]));
  const int xr = dig_row_exp(block_max_u(er, red));
  if (threadIdx.x == 0) e[m] = xr;
  for (int t = threadIdx.x; t < 2 * kb; t += blockDim.x) {
    long long q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = 8 * t + i;
      q[i] = dig_fixed(k < K ? s[k] : 0.0, xr);
    }
    dig_store(q, dig_block(d, m, t >> 1, kb, tr), tr, m % tr, t & 1);
  }
}

// src [K][ld]: lanes along the rows (contiguous), the eight warps split K.
__global__ void __launch_bounds__(256) k_dig_real_cols(const double* __restrict__ src, long ld, int rows, int K,
                                                       int kb, int tr, int row0, unsigned char* __restrict__ d,
                                                       int* __restrict__ e) {
  __shared__ unsigned red[8][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, col = blockIdx.x * 32 + lane, row = row0 + col;
  const bool in = col < rows;
  unsigned er = 0;
  if (in)
    for (int k = wid; k < K; k += 8) er = max(er, dig_key(src[(size_t)k * ld + col]));
  red[wid][lane] = er;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) er = max(er, red[i][lane]);
  const int x = dig_row_exp(er);
  if (!in) return;
  if (wid == 0) e[row] = x;
  for (int t = wid; t < 2 * kb; t += 8) {
    long long q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = 8 * t + i;
      q[i] = dig_fixed(k < K ? src[(size_t)k * ld + col] : 0.0, x);
    }
    dig_store(q, dig_block(d, row, t >> 1, kb, tr), tr, row % tr, t & 1);
  }
}

// y -> B digits of DigWalk. One CTA per walker; a work item is eight orbitals of one column.
__global__ void __launch_bounds__(256) k_dig_walk_y(const double2* __restrict__ y0, const double2* __restrict__ y1,
                                                    size_t ws0, size_t ws1, int o0, int ncol, int n, int np, int nt,
                                                    int tr, int stack, unsigned char* __restrict__ d,
                                                    int* __restrict__ e) {
  pdl_enter();
  __shared__ unsigned key[128];
  const int w = blockIdx.x, kb = stack ? np >> 4 : np >> 3, nchunk = np >> 3;
  const int o1 = ncol - o0, items = ncol * nchunk;
  for (int i = threadIdx.x; i < ncol; i += blockDim.x) key[i] = 0;
  __syncthreads();
  auto load = [&](int it, int& c, int& ch, double2 (&v)[8]) {
    c = it % ncol;
    ch = it / ncol;
    const double2* src = c < o0 ? y0 + w * ws0 + c : y1 + w * ws1 + (c - o0);
    const int o = c < o0 ? o0 : o1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = 8 * ch + i;
      v[i] = p < n ? src[(size_t)p * o] : c2(0.0, 0.0);
    }
  };
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int c, ch;
    double2 v[8];
    load(it, c, ch, v);
    unsigned k = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) k = max(k, max(dig_key(v[i].x), dig_key(v[i].y)));
    atomicMax(&key[c], k);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ncol; i += blockDim.x) {
    const int x = dig_row_exp(key[i]);
    e[(size_t)w * nt * tr + 2 * i] = x;
    e[(size_t)w * nt * tr + 2 * i + 1] = x;
  }
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int c, ch;
    double2 v[8];
    load(it, c, ch, v);
    const int x = dig_row_exp(key[c]), row = 2 * c, tile = row / tr, r = row % tr;
    unsigned char* b = d + ((size_t)(w * nt + tile) * kb + (ch >> 1)) * ((size_t)tr * 256);
    unsigned char* b2 = b + (size_t)(np >> 4) * ((size_t)tr * 256);
    long long q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = dig_fixed(v[i].x, x);
    dig_store(q, b, tr, r, ch & 1);
    if (!stack) dig_store(q, b2, tr, r + 1, ch & 1);
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = dig_fixed(v[i].y, x);
    dig_store(q, b, tr, r + 1, ch & 1);
    if (!stack) dig_store(q, b2, tr, r, ch & 1, 0x80008000u);
  }
}

// V [w][n][n] -> A digits, rows p, K = [Re V[p][q] | Im V[p][q]], or stacked, rows p = Re V[p][q] and
// 64 + p = Im V[p][q]. LPR lanes per row, eight q each
// (LPR * 8 >= np).
template <int LPR>
__global__ void __launch_bounds__(256) k_dig_walk_v(const double2* __restrict__ V, int nrows, int n, int np, int mt,
                                                    int stack, unsigned char* __restrict__ d,
                                                    int* __restrict__ e) {
  pdl_enter();
  const int g = (blockIdx.x * 256 + threadIdx.x) / LPR, ch = threadIdx.x % LPR, kb = stack ? np >> 4 : np >> 3;
  const bool in = g < nrows;
  const int w = in ? g / n : 0, p = in ? g % n : 0;
  const double2* src = V + ((size_t)w * n + p) * n;
  double2 v[8];
  unsigned k = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = 8 * ch + i;
    v[i] = in && q < n ? src[q] : c2(0.0, 0.0);
    k = max(k, max(dig_key(v[i].x), dig_key(v[i].y)));
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
  if (!in) return;
  const int x = dig_row_exp(k);
  if (ch == 0) {
    e[(size_t)w * mt * kDigTile + p] = x;
    if (stack) e[(size_t)w * mt * kDigTile + 64 + p] = x;
  }
  if (8 * ch >= np) return;
  unsigned char* b = dig_block(d + (size_t)w * mt * kb * (kDigTile * 256), p, ch >> 1, kb, kDigTile);
  long long q8[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) q8[i] = dig_fixed(v[i].x, x);
  dig_store(q8, b, kDigTile, p & (kDigTile - 1), ch & 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) q8[i] = dig_fixed(v[i].y, x);
  if (stack) dig_store(q8, b, kDigTile, 64 + p, ch & 1);
  else dig_store(q8, b + (size_t)(np >> 4) * (kDigTile * 256), kDigTile, p & (kDigTile - 1), ch & 1);
}

// V^H: rows q, K = [Re V[p][q] | -Im V[p][q]] over p, or stacked the same way. CTA per (walker, 32 rows), lanes along q.
__global__ void __launch_bounds__(256) k_dig_walk_vh(const double2* __restrict__ V, int n, int np, int mt, int stack,
                                                     unsigned char* __restrict__ d, int* __restrict__ e) {
  pdl_enter();
  __shared__ unsigned red[8][32];
  const int w = blockIdx.y, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = blockIdx.x * 32 + lane,
            kb = stack ? np >> 4 : np >> 3;
  const bool in = q < n;
  const double2* src = V + (size_t)w * n * n + q;
  unsigned k = 0;
  if (in)
    for (int p = wid; p < n; p += 8) {
      const double2 v = src[(size_t)p * n];
      k = max(k, max(dig_key(v.x), dig_key(v.y)));
    }
  red[wid][lane] = k;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) k = max(k, red[i][lane]);
  const int x = dig_row_exp(k);
  if (!in) return;
  if (wid == 0) {
    e[(size_t)w * mt * kDigTile + q] = x;
    if (stack) e[(size_t)w * mt * kDigTile + 64 + q] = x;
  }
  for (int t = wid; t < (np >> 3); t += 8) {
    long long a[8], b8[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = 8 * t + i;
      const double2 v = p < n ? src[(size_t)p * n] : c2(0.0, 0.0);
      a[i] = dig_fixed(v.x, x);
      b8[i] = dig_fixed(v.y, x);
    }
    unsigned char* b = dig_block(d + (size_t)w * mt * kb * (kDigTile * 256), q, t >> 1, kb, kDigTile);
    dig_store(a, b, kDigTile, q & (kDigTile - 1), t & 1);
    if (stack) dig_store(b8, b, kDigTile, 64 + q, t & 1, 0x80008000u);
    else dig_store(b8, b + (size_t)(np >> 4) * (kDigTile * 256), kDigTile, q & (kDigTile - 1), t & 1, 0x80008000u);
  }
}

// Operands of the V cotangents: rows r (an orbital) of a walker, K index m ncol + c over the terms
// t0.. of tay. A (b = 0): rows p, [Re | Im]; B (b = 1): rows 2q = [Re | Im], 2q + 1 = [-Im | Re],
// so that A B^T holds the parts of sum Q conj(P). CTA per walker.
__global__ void __launch_bounds__(256) k_dig_vbar(const double2* __restrict__ tay, int terms, int t0, int M, int n,
                                                  int o0, int ncol, int K, int b, int rt, int tr,
                                                  unsigned char* __restrict__ d, int* __restrict__ e) {
  pdl_enter();
  __shared__ unsigned key[256];
  const int w = blockIdx.x, kc = K >> 1, kb = K >> 4, nchunk = kc >> 3, items = n * nchunk, o1 = ncol - o0;
  const size_t nk = (size_t)n * ncol;
  const double2* src = tay + ((size_t)w * terms + t0) * nk;
  for (int i = threadIdx.x; i < n; i += blockDim.x) key[i] = 0;
  __syncthreads();
  auto load = [&](int it, int& r, int& ch, double2 (&v)[8]) {
    ch = it % nchunk;
    r = it / nchunk;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = 8 * ch + i, m = k / ncol, c = k % ncol;
      v[i] = m < M ? src[(size_t)m * nk + (c < o0 ? (size_t)r * o0 + c : (size_t)n * o0 + (size_t)r * o1 + (c - o0))]
                   : c2(0.0, 0.0);
    }
  };
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int r, ch;
    double2 v[8];
    load(it, r, ch, v);
    unsigned k = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) k = max(k, max(dig_key(v[i].x), dig_key(v[i].y)));
    atomicMax(&key[r], k);
  }
  __syncthreads();
  const size_t erow = (size_t)w * rt * tr;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int x = dig_row_exp(key[i]);
    if (b) {
      e[erow + 2 * i] = x;
      e[erow + 2 * i + 1] = x;
    } else {
      e[erow + i] = x;
    }
  }
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int r, ch;
    double2 v[8];
    load(it, r, ch, v);
    const int x = dig_row_exp(key[r]), row = b ? 2 * r : r, tile = row / tr, rr = row % tr;
    unsigned char* p = d + ((size_t)(w * rt + tile) * kb + (ch >> 1)) * ((size_t)tr * 256);
    unsigned char* p2 = p + (size_t)(kc >> 4) * ((size_t)tr * 256);
    long long q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = dig_fixed(v[i].x, x);
    dig_store(q, p, tr, rr, ch & 1);
    if (b) dig_store(q, p2, tr, rr + 1, ch & 1);
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = dig_fixed(v[i].y, x);
    dig_store(q, p2, tr, rr, ch & 1);
    if (b) dig_store(q, p, tr, rr + 1, ch & 1, 0x80008000u);
  }
}

// ======================================================================================
// the digit GEMM
// ======================================================================================

// The sum hi 2^28 + lo in units of 2^-63 (lo < 2^28), times 2^e, rounded to FP64.
AFQ_D double dig_combine(long long hi, unsigned lo, int e) {
  const int sgn = (int)(hi >> 63);  // sign of the whole sum: lo is non-negative
  unsigned long long a = (unsigned long long)(hi ^ sgn);  // |sum| = a 2^28 + lo, sum < 0: complement + 1
  lo = ((lo ^ (unsigned)sgn) & 0xfffffffu) - (unsigned)sgn;
  a += lo >> 28;
  lo &= 0xfffffffu;
  if (a == 0) {  // below 2^28 units: shift up (exact)
    if (lo == 0) return e > kDigBad / 2 ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
    a = lo;
    lo = 0;
    e -= 28;
  }
  const int lz = __clzll((long long)a);  // a has at most 46 bits: lz >= 18
  const unsigned long long m = (a << lz) | (((unsigned long long)lo << 36) >> (64 - lz));
  const unsigned long long r = (m >> 11) + ((m >> 10) & 1ull);
  const int be = 28 - lz + e + 1022;  // biased exponent - 1: r carries the hidden bit
  if (be < 0 || be > 2044) {          // outside the normal range, or a bad row
    if (e > kDigBad / 2) return __longlong_as_double(0x7ff8000000000000ll);
    const double v = scalbn((double)r, be - 1022 - 52);
    return sgn ? -v : v;
  }
  return __hiloint2double((int)((unsigned)(r >> 32) + ((unsigned)be << 20)) | (sgn & (int)0x80000000), (int)(unsigned)r);
}

// Integer sums of groups C..C+3 of one element, i_C 2^21 + i_(C+1) 2^14 + i_(C+2) 2^7 + i_(C+3).
// Fast form: v 2^(14+7c) + 1.5 2^23 holds the integer in its low mantissa bits while it is
// below 2^22 in size (one FFMA instead of a conversion at a quarter of the rate); `over`
// collects a nonzero value above bit 22 when one is not.
template <int C>
AFQ_D unsigned dig_magic(float v, unsigned& over) {
  constexpr float s = (float)(1ll << (14 + 7 * (C < 7 ? C : 6)));
  const unsigned b = __float_as_uint(fmaf(C < 7 ? v : v * 128.0f, s, 12582912.0f));
  over |= b ^ 0x4B000000u;
  return b;
}
constexpr long long kDigMagic = 0x4B400000ll * ((1ll << 21) + (1ll << 14) + (1ll << 7) + 1ll);
template <int C>
AFQ_D long long dig_quad_fast(float a, float b, float c, float d, unsigned& over) {
  const unsigned i0 = dig_magic<C>(a, over), i1 = dig_magic<C + 1>(b, over), i2 = dig_magic<C + 2>(c, over),
                 i3 = dig_magic<C + 3>(d, over);
  const unsigned long long x = (unsigned long long)i0 * (1u << 21) + (unsigned long long)i1 * (1u << 14) +
                               (unsigned long long)i2 * (1u << 7) + i3;
  return (long long)(x - (unsigned long long)kDigMagic);
}
template <int C>
AFQ_D int dig_int(float v) {
  constexpr float s = (float)(1ll << (14 + 7 * (C < 7 ? C : 6)));
  return __float2int_rn(C < 7 ? v * s : v * s * 128.0f);
}
template <int C>
__device__ __noinline__ long long dig_quad_slow(float a, float b, float c, float d) {
  return ((long long)dig_int<C>(a) << 21) + ((long long)dig_int<C + 1>(b) << 14) +
         ((long long)dig_int<C + 2>(c) << 7) + (long long)dig_int<C + 3>(d);
}
template <int C>
AFQ_D long long dig_quad(float a, float b, float c, float d) {
  unsigned over = 0;
  const long long x = dig_quad_fast<C>(a, b, c, d, over);
  return (over >> 23) ? dig_quad_slow<C>(a, b, c, d) : x;
}

struct DigGemm {
  const unsigned char *a, *b;
  const int *ea, *eb;
  int kba, kbb;    // K blocks per row tile in the layouts
  int kb;          // K blocks contracted
  int mt, nt, nb;  // row tiles, column tiles, batch entries
  int a_bt, b_bt;  // row tiles per batch entry (0: one operand for all entries)
  int tr;          // B rows per tile
  int splits, kps; // K ranges, K blocks per range
  int stages, ring;  // operand K blocks in flight and the bytes they take
  uint32_t idesc;
};

struct DigWhere {
  int batch, m, n, split;
  bool add;   // a later K segment of the same range: add to what is there
  bool more;  // not the last one
};

constexpr int kDigEpiWarps = 16;
constexpr int kDigThreads = 64 + 32 * kDigEpiWarps;
constexpr int kDigABlock = kDigTile * 256;  // bytes of an A K block
// Walker products stage a tile's sums in shared memory: per column 128 rows (+ 1: conflict-free
// reads along the columns) of the 8-byte and the 4-byte part.
constexpr int kDigStageRows = kDigTile + 1;
constexpr int kDigStageCol = kDigStageRows * 12;
constexpr int kDigSmemMax = 227 * 1024;
constexpr int kDigMaxStages = 5;

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   ptx::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(ptx::smem_u32(bar))
               : "memory");
}

// Persistent over (K range, batch entry, column tile, row tile). Warp 0 loads K blocks
// (A 32 KB + B) with bulk copies, warp 1 issues the MMAs, warps 2..17 combine and store: warp w
// reads TMEM lanes 32 (w % 4).. and a quarter of the columns.
//
// What bounds it: the tensor core. A tcgen05.mma of M 128, K 16 takes 58 cycles at N 16 and 32, 72
// at N 64 and 130 at N 128 here (shared-memory operand reads), so tiles are up to 64 columns
// wide and all eight accumulators fit the tensor memory (8 x 64 columns; two sets at 32). With one set
// the MMAs of the next tile wait for the accumulators to be read: sixteen warps turn them into
// the two 64-bit sums (14 integer instructions a group of four) and free them before the longer
// part, the normalisation and the stores. 512 x 14400 x 512: 247 us, 31 TFLOP/s of FP64 products
// (1.1 PFLOP/s of MMAs; 291 us with eight warps that stored before they freed the accumulators);
// the FP64 units do 1.04 TFLOP/s.
template <class Epi>
__global__ void __launch_bounds__(kDigThreads, 1)
    k_gemm_digits(const DigGemm g, const __grid_constant__ typename Epi::Params ep, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + g.ring);
  uint64_t* empty = full + kDigMaxStages;
  uint64_t* accfull = empty + kDigMaxStages;  // [2]
  uint64_t* accempty = accfull + 2;           // [2]
  uint64_t* done = accempty + 2;
  uint64_t* staged = done + 1;  // walker products: the epilogue warps meet
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(staged + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tr = g.tr, bblock = tr * 256, unit = kDigABlock + bblock;
  const int acols = tr <= 32 ? 32 : 64;  // columns between accumulators
  const int nbuf = tr <= 32 ? 2 : 1;
  const int mn = g.mt * g.nt * g.nb, ntiles = mn * g.splits;
  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&accfull[i], 1);
      ptx::mbar_init(&accempty[i], kDigEpiWarps);
    }
    ptx::mbar_init(done, 1);
    ptx::mbar_init(staged, kDigEpiWarps);
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_holder, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  pdl_enter();
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int ks = tile / mn, x = tile % mn;
        const int m = x % g.mt, n = (x / g.mt) % g.nt, b = x / (g.mt * g.nt);
        const int ka = ks * g.kps, kz = min(g.kb, ka + g.kps);
        const unsigned char* pa = g.a + (size_t)(b * g.a_bt + m) * g.kba * kDigABlock;
        const unsigned char* pb = g.b + (size_t)(b * g.b_bt + n) * g.kbb * bblock;
        for (int k0 = ka; k0 < kz && ok; k0 += kDigSegBlocks) {
          const int k1 = min(kz, k0 + kDigSegBlocks);
          for (int k = k0; k < k1; ++k, ++it) {
            const int s = it % g.stages, r = it / g.stages;
            if (r > 0 && !ptx::mbar_wait(&empty[s], (r - 1) & 1)) {
              ok = false;
              break;
            }
            unsigned char* u = smem + s * unit;
            ptx::mbar_expect_tx(&full[s], (uint32_t)unit);
            bulk_load(u, pa + (size_t)k * kDigABlock, kDigABlock, &full[s]);
            bulk_load(u + kDigABlock, pb + (size_t)k * bblock, (uint32_t)bblock, &full[s]);
          }
        }
      }
      // never leave a copy in flight
      for (int j = it - 1; j >= 0 && j >= it - g.stages; --j)
        if (!ptx::mbar_wait(&full[j % g.stages], (j / g.stages) & 1)) ok = false;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int it = 0, run = 0;
      for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int ka = (tile / mn) * g.kps, kz = min(g.kb, ka + g.kps);
        for (int k0 = ka; k0 < kz && ok; k0 += kDigSegBlocks) {
          const int k1 = min(kz, k0 + kDigSegBlocks);
          const int buf = run % nbuf, use = run / nbuf;
          ++run;
          if (use > 0 && !ptx::mbar_wait(&accempty[buf], (use - 1) & 1)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t acc = tmem + (uint32_t)(buf * 256);
          for (int k = k0; k < k1; ++k, ++it) {
            const int s = it % g.stages, r = it / g.stages;
            if (!ptx::mbar_wait(&full[s], r & 1)) {
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t ua = ptx::smem_u32(smem + s * unit), ub = ua + kDigABlock;
            const uint64_t da = ptx::desc_kmajor_sw128(ua), db = ptx::desc_kmajor_sw128(ub);
            const uint64_t qa = (kDigABlock / 2) >> 4, qb = (uint64_t)(bblock / 2) >> 4;
            auto mma = [&](int c, int i, int j, uint32_t accumulate) {
              ptx::mma_f16(acc + (uint32_t)(c * acols), da + (i >> 2) * qa + (i & 3) * 2,
                           db + (j >> 2) * qb + (j & 3) * 2, g.idesc, accumulate);
            };
#pragma unroll
            for (int c = 0; c < 8; ++c)
#pragma unroll
              for (int i = 0; i <= c; ++i) mma(c, i, c - i, (k > k0 || i > 0) ? 1u : 0u);
            if constexpr (Epi::kNine) {
#pragma unroll
              for (int i = 1; i < 8; ++i) mma(7, i, 8 - i, 1u);
            }
            ptx::mma_commit(&empty[s]);
          }
          ptx::mma_commit(&accfull[buf]);
        }
      }
      ptx::mma_commit(done);
      if (!ptx::mbar_wait(done, 0)) ok = false;
    }
  } else {
    const int q = warp & 3, r = q * 32 + lane;
    const int nc = tr >> 2, col0 = ((warp - 2) >> 2) * nc;  // this warp's columns (4..16)
    const uint32_t src0 = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
    int run = 0, meets = 0;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
      DigWhere w;
      w.split = tile / mn;
      const int x = tile % mn;
      w.m = x % g.mt;
      w.n = (x / g.mt) % g.nt;
      w.batch = x / (g.mt * g.nt);
      const int ka = w.split * g.kps, kz = min(g.kb, ka + g.kps);
      for (int k0 = ka; k0 < kz; k0 += kDigSegBlocks, ++run) {
        w.add = k0 > ka;
        w.more = k0 + kDigSegBlocks < kz;
        const int buf = run % nbuf, use = run / nbuf;
        // warp-uniform outcome: the TMEM loads below are .sync.aligned
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&accfull[buf], use & 1))) {
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const uint32_t src = src0 + (uint32_t)(buf * 256);
        if constexpr (Epi::kWalk) {
          // The sums of the tile to shared memory (free the accumulators), then one element of the result
          // per thread and turn, neighbours along the columns.
          long long* sh = reinterpret_cast<long long*>(smem + g.ring + 256);
          unsigned* sl = reinterpret_cast<unsigned*>(sh + tr * kDigStageRows);
#pragma unroll 1
          for (int c0 = 0; c0 < nc; c0 += 4) {
            float v[8][4];
#pragma unroll
            for (int c = 0; c < 8; ++c) ptx::tmem_ld4p(src + (uint32_t)(c * acols + c0), v[c]);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const long long l = dig_quad<4>(v[4][j], v[5][j], v[6][j], v[7][j]);
              // column 2c goes to plane c, column 2c + 1 to plane tr / 2 + c
              const int at = (((col0 + c0 + j) >> 1) + (j & 1) * (tr >> 1)) * kDigStageRows + r;
              sh[at] = dig_quad<0>(v[0][j], v[1][j], v[2][j], v[3][j]) + (l >> 28);
              sl[at] = (unsigned)l & 0xfffffffu;
            }
          }
          ptx::tc_fence_before();
          auto meet = [&]() {  // bounded, as every wait here
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(staged);
            const bool got = ptx::mbar_wait(staged, meets & 1);
            ++meets;
            return __all_sync(0xffffffffu, got) != 0;
          };
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&accempty[buf]);
          if (!meet()) {
            ok = false;
            break;
          }
          Epi::finish(ep, g, w, sh, sl, threadIdx.x - 64);
          if (!meet()) {  // read before the next tile's sums go there
            ok = false;
            break;
          }
        } else {
          long long hi[16];  // the sum in units of 2^-35 and its remainder in units of 2^-63
          unsigned lo[16];
#pragma unroll
          for (int c0 = 0; c0 < 16; c0 += 4)
            if (c0 < nc) {
              float v[8][4];
#pragma unroll
              for (int c = 0; c < 8; ++c) ptx::tmem_ld4p(src + (uint32_t)(c * acols + c0), v[c]);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const long long l = dig_quad<4>(v[4][j], v[5][j], v[6][j], v[7][j]);
                hi[c0 + j] = dig_quad<0>(v[0][j], v[1][j], v[2][j], v[3][j]) + (l >> 28);
                lo[c0 + j] = (unsigned)l & 0xfffffffu;
              }
            }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&accempty[buf]);
          const int er = g.ea[(size_t)(w.batch * g.a_bt + w.m) * kDigTile + r] + Epi::shift(ep);
          const int* eb = g.eb + (size_t)(w.batch * g.b_bt + w.n) * tr + col0;
#pragma unroll
          for (int c0 = 0; c0 < 16; c0 += 4)
            if (c0 < nc) {
              double o[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) o[j] = dig_combine(hi[c0 + j], lo[c0 + j], er + eb[c0 + j]);
              Epi::store(ep, w, r, col0 + c0, o);
            }
        }
      }
    }
  }
  if (!ok) atomicOr(status, kDigTimeout);
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// Complex results: rows 2m / 2m + 1 of D are the real and imaginary parts of row m of C.
// Neighbouring lanes exchange halves so that each stores whole complex numbers.
struct EpiDigC {
  static constexpr bool kNine = false, kWalk = false;
  struct Params {
    double2* c;
    int M, N, tr;
    long ldc, split_stride;
    int rot, shift;  // C = i^rot 2^shift D
  };
  AFQ_D static int shift(const Params& p) { return p.shift; }
  AFQ_D static void store(const Params& p, const DigWhere& w, int r, int col0, const double (&v)[4]) {
    const int m = (w.m * kDigTile + r) >> 1, odd = r & 1, n0 = w.n * p.tr + col0;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const double x = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
      const double re = odd ? x : v[j], im = odd ? v[j + 1] : x;
      const int n = n0 + j + odd;
      double2 o = c2(re, im);
      if (p.rot == 1) o = c2(-im, re);
      if (p.rot == 3) o = c2(im, -re);
      if (m < p.M && n < p.N) {
        double2* dst = p.c + (size_t)w.split * p.split_stride + (size_t)m * p.ldc + n;
        if (w.add) o = cadd(o, *dst);
        *dst = o;
      }
    }
  }
};

struct EpiDigR {
  static constexpr bool kNine = false, kWalk = false;
  struct Params {
    double* d;
    int M, N, tr;
    long ldd;
    int swap;
  };
  AFQ_D static int shift(const Params&) { return 0; }
  AFQ_D static void store(const Params& p, const DigWhere& w, int r, int col0, const double (&v)[4]) {
    const int m = w.m * kDigTile + r, n0 = w.n * p.tr + col0;
    if (m >= p.M) return;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n0 + j < p.N) {
        int rr = m, cc = n0 + j;
        if (p.swap) {
          rr = m - m % p.swap + cc % p.swap;
          cc = cc - cc % p.swap + m % p.swap;
        }
        double* dst = p.d + (size_t)rr * p.ldd + cc;
        *dst = w.add ? *dst + v[j] : v[j];
      }
  }
};

// Products of DigWalk: row p of tile m, columns 2c and 2c + 1 of one walker.
// These also take the digit products with i + j = 8 (into the last accumulator, which then holds two weights and may
// round): exp_h1 is nearly diagonal and a column of a walker has a few large entries,
// so the scale of a dot product can be far above its value. Walkers after a step, against
// extended precision: 1.7e-16 at norb 33, 2.1e-16 at norb 120; the FP64 units: 3.5e-16, 6.2e-16.
struct WalkParams {
  WalkOut o;
  int n, o0, ncol, tr, only;  // only: the slab to store (-1: both)
  int stack, pair;            // stacked rows; V (the two row halves make one result) or E (a slab each)
};

struct EpiWalk {
  static constexpr bool kNine = true, kWalk = true;
  using Params = WalkParams;
  AFQ_D static void finish(const Params& p, const DigGemm& g, const DigWhere& w, const long long* sh, const unsigned* sl,
                           int t) {
    constexpr int NT = 32 * kDigEpiWarps, U = 2;  // results in flight per thread (their loads are from L2)
    const int half = p.tr >> 1, c_lo = w.n * half, cc = min(half, p.ncol - c_lo), rows = min(p.n - w.m * kDigTile, kDigTile);
    const int* ea = g.ea + (size_t)(w.batch * g.a_bt + w.m) * kDigTile;
    const int* eb = g.eb + (size_t)(w.batch * g.b_bt + w.n) * p.tr;
    const int dp = NT / cc, dc = NT - dp * cc, items = rows * cc;
    int pr = t / cc, c = t - pr * cc;
    const bool last = !w.more;
    for (int it = t; it < items; it += U * NT) {
      double2 z[U], in[U], ac[U];
      size_t at[U];
      int sl_[U];
      bool on[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int s = c_lo + c >= p.o0 ? 1 : 0;
        on[u] = it + u * NT < items && (p.only < 0 || s == p.only);
        sl_[u] = s;
        const int k = s ? p.ncol - p.o0 : p.o0;
        at[u] = (size_t)(w.m * kDigTile + pr) * k + (c_lo + c - (s ? p.o0 : 0));
        if (on[u]) {
          if (last && p.o.in.p[s]) in[u] = p.o.in.p[s][(size_t)w.batch * p.o.in.stride(s) + at[u]];
          if (last && p.o.acc.p[s] && !p.o.init) ac[u] = p.o.acc.p[s][(size_t)w.batch * p.o.acc.stride(s) + at[u]];
          const int row = p.stack && !p.pair ? pr + 64 * s : pr, e = ea[row] + eb[2 * c];
          const int a = c * kDigStageRows + row, b = a + half * kDigStageRows;
          long long rh = sh[a], ih = sh[b];
          int rl = (int)sl[a], il = (int)sl[b];
          if (p.pair) {  // Re = Re V Re y - Im V Im y, Im = Re V Im y + Im V Re y
            rh -= sh[b + 64];
            rl -= (int)sl[b + 64];
            ih += sh[a + 64];
            il += (int)sl[a + 64];
          }
          z[u] = c2(dig_combine(rh + (rl >> 28), (unsigned)rl & 0xfffffffu, e),
                    dig_combine(ih + (il >> 28), (unsigned)il & 0xfffffffu, e));
        }
        pr += dp;
        c += dc;
        if (c >= cc) {
          c -= cc;
          ++pr;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (on[u]) {
          const int s = sl_[u];
          double2* out = p.o.out.p[s] ? p.o.out.p[s] + (size_t)w.batch * p.o.out.stride(s) + at[u] : nullptr;
          double2 x = z[u];
          if (w.add) x = cadd(x, *out);
          if (last && p.o.in.p[s]) x = c2(fma(in[u].x, p.o.fin, x.x), fma(in[u].y, p.o.fin, x.y));
          if (out) *out = last && p.o.fout != 1.0 ? cscale(x, p.o.fout) : x;
          if (last && p.o.acc.p[s])
            p.o.acc.p[s][(size_t)w.batch * p.o.acc.stride(s) + at[u]] =
                p.o.init ? x : c2(fma(x.x, p.o.facc, ac[u].x), fma(x.y, p.o.facc, ac[u].y));
        }
    }
  }
};

// C = sum of the partial results of a split contraction
__global__ void k_dig_sum(long M, long N, int splits, long sst, const double2* __restrict__ part,
                          double2* __restrict__ c, long ldc) {
  pdl_enter();
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < M * N; i += (long)gridDim.x * blockDim.x) {
    double2 a = part[i];
    for (int s = 1; s < splits; ++s) a = cadd(a, part[i + s * sst]);
    c[(i / N) * ldc + i % N] = a;
  }
}

// ======================================================================================
// Local energy (wavefunctions.py:529-561, 711-743) from Z = U G and the Coulomb sums
//   exc = sum_g sum_ik f_g[i,k] f_g[k,i] = sum_(i,q) Z[i,q] G[i,q],
//   U[(i,q),(k,p)] = sum_g rc_g[i,p] rc_g[k,q],   coul_g = tr f_g (both spins together),
// which is 4 (nocc norb)^2 flops per walker instead of 4 nchol norb nocc^2, and a contraction
// with one operand for all walkers. U is symmetric: d exc = 2 sum Z dG and d exc / dG = 2 Z.
// ======================================================================================

AFQ_D double2 block_sum2(double2 v, double* red) { return c2(block_sum(v.x, red), block_sum(v.y, red)); }

__global__ void __launch_bounds__(128) k_dig_energy(const afq_ctx_dev c, const double2* __restrict__ green,
                                                    const double2* __restrict__ z, const double2* __restrict__ coul,
                                                    double2* __restrict__ energy, const int* __restrict__ status) {
  pdl_enter();
  __shared__ double red[32];
  const size_t w = blockIdx.x;
  double2 e1 = c2(0, 0), ex = c2(0, 0), co = c2(0, 0);
  for (int i = threadIdx.x; i < c.ktot; i += blockDim.x) {
    const int s = (c.nspin_g == 2 && i >= c.gocc[0] * c.norb) ? 1 : 0;
    const double2 g = green[w * c.ktot + i];
    e1 = cadd(e1, cscale(g, c.rot_h1[s][i - s * c.gocc[0] * c.norb]));
    ex = cadd(ex, cmul(z[w * c.ktot + i], g));
  }
  for (int g = threadIdx.x; g < c.nchol; g += blockDim.x) {
    const double2 x = coul[w * c.nchol + g];
    co = cadd(co, cmul(x, x));
  }
  e1 = block_sum2(e1, red);
  ex = block_sum2(ex, red);
  co = block_sum2(co, red);
  if (threadIdx.x) return;
  double2 e2;
  if (c.energy_mode == 0) {  // RHF restricted
    e1 = cscale(e1, 2.0);
    e2 = csub(cscale(co, 2.0), ex);
  } else if (c.energy_mode == 1) {  // RHF two-slab (G = G_up + G_dn)
    e2 = csub(co, ex);
  } else {  // UHF
    e2 = cscale(csub(co, ex), 0.5);
  }
  energy[w] = *status == 0 ? cadd(cadd(e2, e1), c2(c.h0, 0.0)) : c2(nan(""), nan(""));
}

__global__ void __launch_bounds__(128) k_dig_energy_tangent(const afq_ctx_dev c, const double2* __restrict__ green,
                                                            const double2* __restrict__ dgreen,
                                                            const double2* __restrict__ z,
                                                            const double2* __restrict__ coul,
                                                            const double2* __restrict__ dcoul, const double* drot_up,
                                                            const double* drot_dn, double2* __restrict__ denergy) {
  pdl_enter();
  __shared__ double red[32];
  const size_t w = blockIdx.x;
  double2 e1 = c2(0, 0), ex = c2(0, 0), co = c2(0, 0);
  for (int i = threadIdx.x; i < c.ktot; i += blockDim.x) {
    const int s = (c.nspin_g == 2 && i >= c.gocc[0] * c.norb) ? 1 : 0, j = i - s * c.gocc[0] * c.norb;
    const double2 g = green[w * c.ktot + i], dg = dgreen[w * c.ktot + i];
    const double dr = (s == 0 ? drot_up : drot_dn)[j];
    e1 = cadd(e1, cadd(cscale(dg, c.rot_h1[s][j]), cscale(g, dr)));
    ex = cadd(ex, cmul(z[w * c.ktot + i], dg));
  }
  for (int g = threadIdx.x; g < c.nchol; g += blockDim.x)
    co = cadd(co, cmul(coul[w * c.nchol + g], dcoul[w * c.nchol + g]));
  e1 = block_sum2(e1, red);
  ex = cscale(block_sum2(ex, red), 2.0);
  co = cscale(block_sum2(co, red), 2.0);
  if (threadIdx.x) return;
  if (c.energy_mode == 0)
    denergy[w] = cadd(csub(cscale(co, 2.0), ex), cscale(e1, 2.0));
  else if (c.energy_mode == 1)
    denergy[w] = cadd(csub(co, ex), e1);
  else
    denergy[w] = cadd(cscale(csub(co, ex), 0.5), e1);
}

// Convention of afq_adjoint.cu: G-bar = e-bar (kappa conj(Z) + gamma conj(sum_g c_g rc_g) + mult1
// rot_h1); zero for a walker without an energy cotangent, whatever its G holds.
__global__ void k_dig_energy_adjoint(const afq_ctx_dev c, const double2* __restrict__ z,
                                     const double* __restrict__ ebar, double2* __restrict__ gene) {
  pdl_enter();
  const double kappa = c.energy_mode == 2 ? -1.0 : -2.0;
  const double gamma = c.energy_mode == 0 ? 4.0 : (c.energy_mode == 1 ? 2.0 : 1.0);
  const double mult1 = c.energy_mode == 0 ? 2.0 : 1.0;
  const size_t w = blockIdx.x;
  const double eb = ebar[w];
  for (int i = threadIdx.x; i < c.ktot; i += blockDim.x) {
    const int s = (c.nspin_g == 2 && i >= c.gocc[0] * c.norb) ? 1 : 0;
    const double2 a = z[w * c.ktot + i], b = gene[w * c.ktot + i];
    const double r = c.rot_h1[s][i - s * c.gocc[0] * c.norb];
    gene[w * c.ktot + i] = eb == 0.0 ? c2(0, 0)
                                     : c2(eb * (kappa * a.x + gamma * b.x + mult1 * r),
                                          -eb * (kappa * a.y + gamma * b.y));
  }
}

// ======================================================================================
// host launchers
// ======================================================================================

static int dig_err(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    afq_set_error("%s: %s", what, cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

int dig_sms() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    cudaGetLastError();
    sms = 148;
  }
  return sms;
}

int dig_slice_cplx_rows(const DigOp& op, const double2* src, long ld, double mul, cudaStream_t st) {
  {
    ProfScope _ps(K_PREP, st);
    launch_pdl(k_dig_cplx_rows, op.rows / 2, 128, 0, st, src, ld, op.K, op.kb(), mul, op.d, op.e);
  }
  return dig_err("slice rows");
}

int dig_slice_real_rows(const DigOp& op, const double* src, long ld, cudaStream_t st, int rows, int row0) {
  {
    ProfScope _ps(K_PREP, st);
    k_dig_real_rows<<<rows < 0 ? op.rows : rows, 128, 0, st>>>(src, ld, op.K, op.kb(), op.tr, row0, op.d, op.e);
  }
  return dig_err("slice rows");
}

int dig_slice_real_cols(const DigOp& op, const double* src, long ld, cudaStream_t st, int rows, int row0) {
  {
    ProfScope _ps(K_PREP, st);
    const int r = rows < 0 ? op.rows : rows;
    k_dig_real_cols<<<(r + 31) / 32, 256, 0, st>>>(src, ld, r, op.K, op.kb(), op.tr, row0, op.d, op.e);
  }
  return dig_err("slice columns");
}

template <class Epi>
static int launch_digits(int cls, DigGemm g, const typename Epi::Params& ep, int* status, cudaStream_t st) {
  const int unit = kDigABlock + g.tr * 256, stage = Epi::kWalk ? g.tr * kDigStageCol : 0;
  g.stages = std::min((kDigSmemMax - 1024 - 256 - stage) / unit, kDigMaxStages);
  g.ring = g.stages * unit;
  const int smem = 1024 + g.ring + 256 + stage;
  g.idesc = ptx::idesc_f16(128, g.tr, 1);
  const long tiles = (long)g.mt * g.nt * g.nb * g.splits;
  const int sms = dig_sms();
  auto kfn = k_gemm_digits<Epi>;
  cudaError_t e = raise_smem_limit((const void*)kfn, smem);
  if (e != cudaSuccess) {
    afq_set_error("digit GEMM: shared-memory attribute: %s", cudaGetErrorString(e));
    return (int)e;
  }
  {
    ProfScope _ps(cls, st);
    launch_pdl(kfn, (unsigned)(tiles < sms ? tiles : sms), kDigThreads, smem, st, g, ep, status);
  }
  return dig_err("digit GEMM");
}

static DigGemm dig_args(const DigOp& A, const DigOp& B) {
  DigGemm g;
  g.a = A.d;
  g.b = B.d;
  g.ea = A.e;
  g.eb = B.e;
  g.kba = A.kb();
  g.kbb = B.kb();
  g.kb = g.kba < g.kbb ? g.kba : g.kbb;
  g.mt = (A.rows + kDigTile - 1) / kDigTile;
  g.nt = (B.rows + B.tr - 1) / B.tr;
  g.nb = 1;
  g.a_bt = g.b_bt = 0;
  g.tr = B.tr;
  g.splits = 1;
  g.kps = g.kb;
  g.stages = 0;
  g.idesc = 0;
  return g;
}

int dig_tr(int M, int N, int kb, int sms) {
  const int mt = (2 * M + kDigTile - 1) / kDigTile, need = (N + 15) / 16 * 16;
  const int tr = mt * ((N + 63) / 64) * (kb < 8 ? kb : 8) * 2 >= sms ? 64 : 32;
  return need < tr ? need : tr;
}

// The count of K ranges that gives the fewest (rounds of tiles over the SMs) x (K blocks per
// range + 2 for a segment's epilogue; the contractions of a two-step block of 512 walkers in 60 orbitals take 315 us with 2
// or 6 and 335 with none, other sizes the same with all three).
DigPlan dig_plan(int tiles, int kb, int sms, int max_splits) {
  DigPlan best{1, kb};
  long cost = -1;
  for (int s = 1; s <= max_splits && s <= kb; ++s) {
    const int kps = (kb + s - 1) / s, used = (kb + kps - 1) / kps;
    const long c = (long)((tiles * (long)used + sms - 1) / sms) * (kps + 2 * ((kps + kDigSegBlocks - 1) / kDigSegBlocks));
    if (cost < 0 || c < cost) {
      cost = c;
      best = DigPlan{used, kps};
    }
  }
  return best;
}

size_t dig_partial_bytes(int M, int N, int splits) {
  return splits > 1 ? (size_t)splits * M * N * sizeof(double2) : 256;
}

int dig_gemm_c(int cls, const DigOp& A, const DigOp& B, int M, int N, double2* C, long ldc, int rot, int shift,
               const DigPlan& plan, double2* part, int* status, cudaStream_t st) {
  DigGemm g = dig_args(A, B);
  g.mt = (2 * M + kDigTile - 1) / kDigTile;
  g.nt = (N + B.tr - 1) / B.tr;
  g.splits = plan.splits;
  g.kps = plan.kps;
  const bool split = plan.splits > 1;
  EpiDigC::Params ep{split ? part : C, M, N, B.tr, split ? (long)N : ldc, (long)M * N, rot, shift};
  int rc = launch_digits<EpiDigC>(cls, g, ep, status, st);
  if (rc || !split) return rc;
  {
    ProfScope _ps(cls, st);
    const long n = (long)M * N;
    launch_pdl(k_dig_sum, (unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096), 256, 0, st, M, N, plan.splits, n, part,
                                                                                          C, ldc);
  }
  return dig_err("digit GEMM sum");
}

int dig_gemm_r(int cls, const DigOp& A, const DigOp& B, int M, int N, double* D, long ldd, int swap,
               int* status, cudaStream_t st) {
  DigGemm g = dig_args(A, B);
  EpiDigR::Params ep{D, M, N, B.tr, ldd, swap};
  return launch_digits<EpiDigR>(cls, g, ep, status, st);
}

void dig_walk_dims(int norb, const int* k, int nslab, int nw, DigWalk* d) {
  d->stack = norb <= 64 ? 1 : 0;
  d->n = norb;
  d->np = (norb + 15) / 16 * 16;
  d->o[0] = k[0];
  d->o[1] = nslab == 2 ? k[1] : 0;
  d->ncol = d->o[0] + d->o[1];
  d->mt = (norb + kDigTile - 1) / kDigTile;
  d->nt = (2 * d->ncol + 63) / 64;
  d->tr = ((2 * d->ncol + d->nt - 1) / d->nt + 15) / 16 * 16;
  // V digits of a chunk: at most 160 MB or 152 walkers, whichever is more (171 MB at 129 orbitals, 304 at 256), in whole
  // rounds of the full part's 152 SMs. Two steps with chunks of 40, 160 and 640 MB: 2000 walkers in 60 orbitals 2.81, 2.28
  // and 2.12 ms; 1216 in 120 5.77, 4.83 and 4.26; 304 in 200 5.63, 5.65 and 5.61.
  const size_t per = (size_t)d->mt * kDigTile * d->kbv() * 256;
  const long most = std::max<long>((long)((160u << 20) / per) / 152 * 152, 152);
  d->chunk = nw < most ? nw : (int)most;
  for (int s = 0; s < 2; ++s) {
    d->e[s].rows = d->stack ? kDigTile : norb;
    d->e[s].K = norb;
    d->e[s].tr = kDigTile;
  }
}
size_t dig_walk_v_bytes(const DigWalk& d) { return (size_t)d.chunk * d.mt * kDigTile * d.kbv() * 256; }
size_t dig_walk_x_bytes(const DigWalk& d) { return (size_t)d.chunk * d.nt * d.tr * d.kbv() * 256; }
size_t dig_walk_ve_bytes(const DigWalk& d) { return (size_t)d.chunk * d.mt * kDigTile * sizeof(int); }
size_t dig_walk_xe_bytes(const DigWalk& d) { return (size_t)d.chunk * d.nt * d.tr * sizeof(int); }

int dig_walk_slice_v(const DigWalk& d, const double2* V, int nw, bool adjoint, cudaStream_t st) {
  {
    ProfScope _ps(K_TAYLOR, st);
    const int rows = nw * d.n;
    if (adjoint) {
      launch_pdl(k_dig_walk_vh, dim3((d.n + 31) / 32, nw), 256, 0, st, V, d.n, d.np, d.mt, d.stack, d.vd, d.ve);
    } else if (d.np <= 64) {
      launch_pdl(k_dig_walk_v<8>, (rows + 31) / 32, 256, 0, st, V, rows, d.n, d.np, d.mt, d.stack, d.vd, d.ve);
    } else if (d.np <= 128) {
      launch_pdl(k_dig_walk_v<16>, (rows + 15) / 16, 256, 0, st, V, rows, d.n, d.np, d.mt, d.stack, d.vd, d.ve);
    } else {
      launch_pdl(k_dig_walk_v<32>, (rows + 7) / 8, 256, 0, st, V, rows, d.n, d.np, d.mt, d.stack, d.vd, d.ve);
    }
  }
  return dig_err("slice V");
}

int dig_walk_slice_y(const DigWalk& d, const WalkVec& y, int nw, cudaStream_t st) {
  {
    ProfScope _ps(K_TAYLOR, st);
    launch_pdl(k_dig_walk_y, nw, 256, 0, st, y.p[0], y.p[1], y.stride(0), y.stride(1), d.o[0], d.ncol, d.n, d.np, d.nt, d.tr,
                                     d.stack, d.xd, d.xe);
  }
  return dig_err("slice y");
}

int dig_walk_mul(int cls, const DigWalk& d, int e, const DigOp* E, const WalkOut& o, int nw, cudaStream_t st) {
  DigGemm g;
  g.a = e < 0 ? d.vd : E[e].d;
  g.ea = e < 0 ? d.ve : E[e].e;
  g.b = d.xd;
  g.eb = d.xe;
  g.kbb = d.kbv();
  g.kb = g.kba = e < 0 ? d.kbv() : d.np / 16;
  g.mt = d.mt;
  g.nt = d.nt;
  g.nb = nw;
  g.a_bt = e < 0 ? d.mt : 0;
  g.b_bt = d.nt;
  g.tr = d.tr;
  g.splits = 1;
  g.kps = g.kb;
  WalkParams ep{o, d.n, d.o[0], d.ncol, d.tr, d.stack || e < 0 || d.o[1] == 0 ? -1 : e, d.stack, d.stack && e < 0};
  return launch_digits<EpiWalk>(cls, g, ep, d.status, st);
}

int dig_walk_slice_e(const DigWalk& d, const DigOp* e, const double* const* exp_h1, int nslab, bool transpose,
                     cudaStream_t st) {
  for (int s = 0; s < nslab; ++s) {
    const DigOp& op = d.stack ? e[0] : e[s];
    const int row0 = d.stack ? 64 * s : 0;
    if (int rc = transpose ? dig_slice_real_cols(op, exp_h1[s], d.n, st, d.n, row0)
                           : dig_slice_real_rows(op, exp_h1[s], d.n, st, d.n, row0))
      return rc;
  }
  return 0;
}

void dig_walk_vbar_dims(const DigWalk& d, int M, DigVbar* v) {
  v->K = 2 * ((M * d.ncol + 15) / 16 * 16);
  v->mt = d.mt;
  v->nt = (2 * d.n + 63) / 64;
  v->tr = ((2 * d.n + v->nt - 1) / v->nt + 15) / 16 * 16;
}
size_t dig_walk_vbar_a_bytes(const DigWalk& d, const DigVbar& v) {
  return (size_t)d.chunk * v.mt * kDigTile * v.K * 16;
}
size_t dig_walk_vbar_b_bytes(const DigWalk& d, const DigVbar& v) { return (size_t)d.chunk * v.nt * v.tr * v.K * 16; }
size_t dig_walk_vbar_ae_bytes(const DigWalk& d, const DigVbar& v) {
  return (size_t)d.chunk * v.mt * kDigTile * sizeof(int);
}
size_t dig_walk_vbar_be_bytes(const DigWalk& d, const DigVbar& v) {
  return (size_t)d.chunk * v.nt * v.tr * sizeof(int);
}

int dig_walk_vbar(const DigWalk& d, const DigVbar& v, const double2* tay, int terms, int qt, int pt, int M,
                  double2* vbar, int nw, cudaStream_t st) {
  {
    ProfScope _ps(K_TAYLOR, st);
    launch_pdl(k_dig_vbar, nw, 256, 0, st, tay, terms, qt, M, d.n, d.o[0], d.ncol, v.K, 0, v.mt, kDigTile, v.ad, v.ae);
    launch_pdl(k_dig_vbar, nw, 256, 0, st, tay, terms, pt, M, d.n, d.o[0], d.ncol, v.K, 1, v.nt, v.tr, v.bd, v.be);
  }
  if (int e = dig_err("slice V cotangents")) return e;
  DigGemm g;
  g.a = v.ad;
  g.ea = v.ae;
  g.b = v.bd;
  g.eb = v.be;
  g.kba = g.kbb = g.kb = v.K / 16;
  g.mt = g.a_bt = v.mt;
  g.nt = g.b_bt = v.nt;
  g.nb = nw;
  g.tr = v.tr;
  g.splits = 1;
  g.kps = g.kb;
  WalkOut o;  // [norb][norb] per walker: one slab of norb columns
  o.out = WalkVec{{vbar, nullptr}, (size_t)d.n * d.n};
  WalkParams ep{o, d.n, d.n, d.n, v.tr, -1, 0, 0};
  return launch_digits<EpiWalk>(K_TAYLOR, g, ep, d.status, st);
}

int dig_launch_energy(const afq_ctx_dev& c, const double2* green, const double2* z, const double2* coul,
                      double2* energy, const int* status, cudaStream_t st) {
  {
    ProfScope _ps(K_ENERGY_FIN, st);
    launch_pdl(k_dig_energy, c.nw, 128, 0, st, c, green, z, coul, energy, status);
  }
  return dig_err("energy");
}

int dig_launch_energy_tangent(const afq_ctx_dev& c, const double2* green, const double2* dgreen, const double2* z,
                              const double2* coul, const double2* dcoul, const double* drot_up,
                              const double* drot_dn, double2* denergy, cudaStream_t st) {
  {
    ProfScope _ps(K_ENERGY_FIN, st);
    launch_pdl(k_dig_energy_tangent, c.nw, 128, 0, st, c, green, dgreen, z, coul, dcoul, drot_up, drot_dn, denergy);
  }
  return dig_err("energy tangent");
}

int dig_launch_energy_adjoint(const afq_ctx_dev& c, const double2* z, const double* ebar, double2* gene,
                              cudaStream_t st) {
  {
    ProfScope _ps(K_ENERGY_FIN, st);
    launch_pdl(k_dig_energy_adjoint, c.nw, 128, 0, st, c, z, ebar, gene);
  }
  return dig_err("energy adjoint");
}

}  // namespace afq

extern "C" long afq_test_digits_smem_limit(void) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, (const void*)afq::k_gemm_digits<afq::EpiDigC>);
  if (e != cudaSuccess) {
    afq_set_error("afq_test_digits_smem_limit: %s", cudaGetErrorString(e));
    return -(long)e;
  }
  return a.maxDynamicSharedSizeBytes;
}

extern "C" size_t afq_test_gemm_digits_bytes(int M, int N, int K, int tr) {
  return afq::dig_bytes(M, K) + afq::dig_bytes(N, K, tr) + afq::dig_exps(M) + afq::dig_exps(N, tr) + 1024;
}

extern "C" int afq_test_gemm_digits(const double* a, const double* b, double* d, int M, int N, int K, int tr,
                                    void* scratch, int* status, void* stream) {
  using namespace afq;
  if (!a || !b || !d || !scratch || !status || M < 1 || N < 1 || K < 1 || tr % 16 || tr < 16 || tr > 64) {
    afq_set_error("afq_test_gemm_digits: bad arguments");
    return -1;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  unsigned char* p = static_cast<unsigned char*>(scratch);
  p += (256 - (reinterpret_cast<uintptr_t>(p) & 255)) & 255;
  DigOp A, B;
  A.d = p;
  B.d = A.d + dig_bytes(M, K);
  A.e = reinterpret_cast<int*>(B.d + dig_bytes(N, K, tr));
  B.e = A.e + dig_exps(M) / sizeof(int);
  A.rows = M;
  B.rows = N;
  A.K = B.K = K;
  B.tr = tr;
  cudaError_t e = cudaMemsetAsync(p, 0, afq_test_gemm_digits_bytes(M, N, K, tr) - 512, st);
  if (e != cudaSuccess) {
    afq_set_error("afq_test_gemm_digits: %s", cudaGetErrorString(e));
    return (int)e;
  }
  if (int rc = dig_slice_real_rows(A, a, K, st)) return rc;
  if (int rc = dig_slice_real_rows(B, b, K, st)) return rc;
  return dig_gemm_r(K_PREP, A, B, M, N, d, N, 0, status, st);
}
