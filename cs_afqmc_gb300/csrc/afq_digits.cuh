// FP64 contractions on the BF16 tensor cores, by exact digit slicing.
//
// Every FP64 operand row is scaled by a power of two 2^e >= max|row| and cut into eight
// balanced digits, x 2^-e = sum_j d_j 2^(-7-7j) with |d_0| <= 128, |d_j| <= 64 and a remainder
// of at most 2^-57 (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms
// 59, 2012, with digits of a fixed weight). A digit times its weight is exact in BF16, a
// product of two is exact in FP32, and the sum of all products with i + j = c over up to 512
// terms of K is an integer below 2^24 in units of 2^(-14-7c) for c <= 5: the tensor core's FP32
// accumulator never rounds it. There is one accumulator per c = 0..7, 36 of the 64 digit products; those of
// c = 6 and 7 can pass 2^24 (35847 x 512 and 38038 x 512 at most) and then round to a few units of 2^-56
// and 2^-63. The eight are combined in 64-bit integer arithmetic and rounded to FP64.
//
// Error of a dot product of up to 512 terms, with 2^ea, 2^eb the scales of its two rows (at most twice
// their largest elements): the rounding of the result; per term the two remainders, 2^-57 2^(ea + eb) each at most, and
// the seven products with i + j = 8 (plus less from the others), 2^-58 each at most: altogether below K 2^(ea + eb - 54), for
// terms of no common sign about sqrt(K) 2^(ea + eb - 58). More terms come in segments of 512, and
// contractions cut into K ranges in ranges, whose results are added in FP64.
// A plain FP64 sum rounds K times at the size of its partial sums: for rows of similar elements (Gaussian: 3.2e-16 of the
// result against 0.9e-16) and for Cholesky vectors that fall by 1e5 against flat fields (4.5e-16, 1.5e-16) it is further
// off. But the digits' error is relative to the rows' largest elements, not to the terms: one large element that meets a zero
// with the others 1e-4 leaves 2e-13, rows that fall and rise against each other by 1e6 1e-11. Contexts can ask for the
// FP64 units instead (AFQ_FP64_UNITS).
//
// Why: this part does FP64 at 1.04 TFLOP/s (DGEMM) and BF16 at 1.9 PFLOP/s, so 36 tensor-core
// products cost about 2 % of the FP64 ones; integer instructions combine the accumulators
// because FP64 adds and conversions (two per cycle and SM) would cost as much as the products.
//
// Layout of a sliced operand ("digit tiles"): rows in tiles of TR (128 for A; 16..64 for B),
// K in blocks of 16. One (row tile, K block) is contiguous: two quads (digits 0-3, 4-7) of
// [TR rows][128 bytes], a row's 128 bytes = 4 digits x 16 k in the 128-byte swizzle the
// tensor core reads, so that a K block of an operand is one plain bulk copy (A 32 KB) and no
// tensor map is needed. Padding rows and columns are zero.
#pragma once
#include "afq_kernels.cuh"

namespace afq {

constexpr int kDigTile = 128;     // A rows per tile
constexpr int kDigSegBlocks = 32; // K blocks (of 16) an accumulator may sum exactly
constexpr int kDigTimeout = 8;    // status bit: a wait of the digit GEMM ran out
constexpr int kDigBad = 1 << 20;  // row exponent of a row with a NaN or an infinity

inline size_t dig_bytes(long rows, long K, int tr = kDigTile) {
  return (size_t)((rows + tr - 1) / tr) * ((K + 15) / 16) * tr * 256;
}
inline size_t dig_exps(long rows, int tr = kDigTile) { return (size_t)((rows + tr - 1) / tr) * tr * sizeof(int); }

// One sliced operand: digit tiles and row exponents.
struct DigOp {
  unsigned char* d = nullptr;
  int* e = nullptr;
  int rows = 0, K = 0, tr = kDigTile;
  int kb() const { return (K + 15) / 16; }
};

// ---- slicing --------------------------------------------------------------------------
// complex [M][ld] (M walkers x K): rows 2m (real parts) and 2m + 1 (imaginary parts), times mul
int dig_slice_cplx_rows(const DigOp& op, const double2* src, long ld, double mul, cudaStream_t st);
// real [rows][ld] (to rows row0.. of the operand)
int dig_slice_real_rows(const DigOp& op, const double* src, long ld, cudaStream_t st, int rows = -1, int row0 = 0);
// real [K][ld], rows along the contiguous index
int dig_slice_real_cols(const DigOp& op, const double* src, long ld, cudaStream_t st, int rows = -1, int row0 = 0);

// ---- contractions ---------------------------------------------------------------------
// C[m][n] (complex, ldc) = i^rot 2^shift sum_k A[m][k] B[n][k]: A sliced by
// dig_slice_cplx_rows, B real. part: split partials when the K range is cut (see
// dig_plan); may be NULL when the plan has one split.
struct DigPlan {
  int splits, kps;  // K ranges computed independently, K blocks per range
};
// K ranges of a contraction with `tiles` output tiles on `sms` SMs
DigPlan dig_plan(int tiles, int kb, int sms, int max_splits);
// bytes of the partial results of dig_gemm_c
size_t dig_partial_bytes(int M, int N, int splits);
int dig_gemm_c(int cls, const DigOp& A, const DigOp& B, int M, int N, double2* C, long ldc, int rot, int shift,
               const DigPlan& plan, double2* part, int* status, cudaStream_t st);
// D[m][n] (real, ldd) = sum_k A[m][k] B[n][k], both real. swap > 0: rows m = (i, p) and columns
// n = (k, q) with p, q < swap; the result goes to row (i, q), column (k, p)
int dig_gemm_r(int cls, const DigOp& A, const DigOp& B, int M, int N, double* D, long ldd, int swap, int* status,
               cudaStream_t st);

// ---- local energy from the sliced contractions -----------------------------------------
// z [nw][ktot] = U G per spin, coul [nw][nchol] = rc . G; final sums per walker (NaN if *status != 0)
int dig_launch_energy(const afq_ctx_dev& c, const double2* green, const double2* z, const double2* coul,
                      double2* energy, const int* status, cudaStream_t st);
// its tangent: dcoul [nw][nchol], the tangents of G and rot_h1
int dig_launch_energy_tangent(const afq_ctx_dev& c, const double2* green, const double2* dgreen, const double2* z,
                              const double2* coul, const double2* dcoul, const double* drot_up,
                              const double* drot_dn, double2* denergy, cudaStream_t st);
// its adjoint: gene [nw][ktot] holds sum_g c_g rc_g on entry and the G cotangent on return
int dig_launch_energy_adjoint(const afq_ctx_dev& c, const double2* z, const double* ebar, double2* gene,
                              cudaStream_t st);
int dig_sms();

// ---- products with one walker's matrices (Taylor series) -------------------------------
// For every walker w of a chunk: out_w = X y_w, X = E (real, shared, per spin), V_w or V_w^H
// (complex), y_w [norb][nocc_s] complex per slab. V is sliced as [Re | Im] along K, y as
// columns 2c = [Re y_c | -Im y_c] and 2c + 1 = [Im y_c | Re y_c], so that one real contraction
// over K = 2 np (np: norb padded to 16) gives both parts; E uses the first half of K.
// Up to 64 orbitals (stack) Re V has rows 0..63 of the 128-row tile and Im V rows 64..127, the
// columns are plain [Re y_c], [Im y_c] and K = np: half the products, half the digits, and the four
// partial sums of an element are added in the epilogue. E has up in rows 0..63 and down in
// 64..127, so that both slabs are one product.
struct DigWalk {
  int stack;
  int n, np, o[2], ncol;  // orbitals, padded; columns per slab and together
  int mt, nt, tr;         // row tiles of V; column tiles per walker and columns (2 per c) per tile
  int chunk;              // walkers sliced at a time
  DigOp e[2];             // exp_h1 per slab (stack: both in e[0])
  unsigned char *vd, *xd; // V digits, y digits
  int *ve, *xe;
  int* status;
  int kbv() const { return stack ? np / 16 : np / 8; }
  int n_e(int nslab) const { return stack ? 1 : nslab; }  // operands in e
};
// complex [walker][norb][nocc_s] per slab, walker stride in elements
struct WalkVec {
  double2* p[2];
  size_t ws;       // walker stride of slab 0 (and of slab 1 unless ws1 is set)
  size_t ws1 = 0;
  AFQ_HD size_t stride(int s) const { return s == 1 && ws1 ? ws1 : ws; }
};
void dig_walk_dims(int norb, const int* k, int nslab, int nw, DigWalk* d);
size_t dig_walk_v_bytes(const DigWalk& d);  // digits, then row exponents
size_t dig_walk_x_bytes(const DigWalk& d);
size_t dig_walk_ve_bytes(const DigWalk& d);
size_t dig_walk_xe_bytes(const DigWalk& d);
// V [nw][norb][norb]; adjoint: V^H
int dig_walk_slice_v(const DigWalk& d, const double2* V, int nw, bool adjoint, cudaStream_t st);
int dig_walk_slice_y(const DigWalk& d, const WalkVec& y, int nw, cudaStream_t st);
// What a product leaves: r = X y + fin in (in may be NULL), out = fout r, acc = r (init) or
// acc + facc r (out, acc may be NULL; in, out and acc may be the same array).
struct WalkOut {
  WalkVec out{{nullptr, nullptr}, 0}, in{{nullptr, nullptr}, 0}, acc{{nullptr, nullptr}, 0};
  double fin = 1.0, fout = 1.0, facc = 0.0;
  int init = 0;
};
// V cotangents of the Taylor adjoint: vbar[w][p][q] = sum_{m=1..M} sum_c Q_m[p,c] conj(P_m[q,c])
// over the columns of both slabs, Q_m = term qt + m - 1 and P_m = term pt + m - 1 of tay
// [w][terms][norb (k0 + k1)]. ad / bd (+ exponents): digits, dig_walk_vbar_bytes each.
struct DigVbar {
  int K, mt, nt, tr;
  unsigned char *ad, *bd;
  int *ae, *be;
};
void dig_walk_vbar_dims(const DigWalk& d, int M, DigVbar* v);
size_t dig_walk_vbar_a_bytes(const DigWalk& d, const DigVbar& v);
size_t dig_walk_vbar_b_bytes(const DigWalk& d, const DigVbar& v);
size_t dig_walk_vbar_ae_bytes(const DigWalk& d, const DigVbar& v);
size_t dig_walk_vbar_be_bytes(const DigWalk& d, const DigVbar& v);
int dig_walk_vbar(const DigWalk& d, const DigVbar& v, const double2* tay, int terms, int qt, int pt, int M,
                  double2* vbar, int nw, cudaStream_t st);
// E (or its transpose) of both slabs into the operands e
int dig_walk_slice_e(const DigWalk& d, const DigOp* e, const double* const* exp_h1, int nslab, bool transpose,
                     cudaStream_t st);
// X = the sliced V (e < 0) or E[e]: that slab's columns (stack: e = 0, every column)
int dig_walk_mul(int cls, const DigWalk& d, int e, const DigOp* E, const WalkOut& o, int nw, cudaStream_t st);
// B columns per tile for an output of 2 M x N with kb K blocks: 64 where the tiles (times up to
// eight K ranges) reach half of the SMs, else 32, so that small problems still spread out; never
// more than N needs. The contractions of a two-step block in us, with 32 / with 64 / by the rule: 20 orbitals, 50 and 500
// walkers 87 / 109 / 87, 90 / 114 / 102; 60 orbitals, 64 and 512 walkers 135 / 158 / 134, 464 / 315 / 315; 80 orbitals, 256
// walkers 576 / 367 / 391; 120 orbitals, 16 and 256 walkers 476 / 391 / 424, 1716 / 1036 / 1035.
int dig_tr(int M, int N, int kb, int sms);

}  // namespace afq
