// C ABI of the AFQMC hot path: context creation, workspace layout and the stream-ordered
// orchestration of the kernels (one propagation step, QR, SR, measurements, and the
// sampler's block loop). See include/afqmc_gb300.h for the contract of each entry point.

#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <new>

#include "afq_common.cuh"
#include "afq_adjoint.cuh"
#include "afq_digits.cuh"
#include "afq_kernels.cuh"
#include "afq_prof.cuh"
#include "afq_tangent.cuh"
#include "afq_tc.cuh"

static thread_local char g_err[512] = "";

void afq_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

// FP64 contractions of a context (afq_digits.cuh): operands sliced once (chol, rc) and the
// scratch of the walker-dependent ones.
struct DigCtx {
  afq::DigOp chol;  // vhs: rows (p, q), K = g
  afq::DigOp rc;    // force bias: rows g, K = (i, p)
  afq::DigOp xa;    // [2 nw] x nchol
  afq::DigOp ga;    // [2 nw] x ktot
  afq::DigPlan fb;  // K ranges of the force bias
  // exchange energy: U per spin of G (rows (i, q), K = (k, p)); has_u 0: too few vectors for it
  int has_u;
  afq::DigOp u[2], ua[2], ub[2];  // ua, ub: rot_chol^T, at set-up only; ua for u_strip of the i at a time
  int u_strip;
  afq::DigPlan uplan[2];
  double2* z;     // [nw][ktot]
  double2* part;  // partial results of split K ranges
  // operands of the Taylor products on the digit GEMM (walk) are there; used by the steps, by forward mode (by
  // reverse mode wherever they are there); else the FP64 units
  int use_walk, walk_fwd, walk_jvp;
  afq::DigWalk walk;
  double2 *walk_t, *walk_acc;  // [chunk][norb * (k0 + k1)]
  int* status;
};

struct afq_ctx {
  afq_dims d;
  afq_hamiltonian h;
  afq_ctx_dev dev;
  int nw_chunk;
  int e_chunks, e_gchunk;
  size_t welem;  // bytes per walker element (16 complex128, 8 complex64)
  // workspace views
  char* ws;
  size_t ws_bytes;
  double2* green;
  double2* fb;
  double2* xt;
  double2* shift;
  double2* fbt;
  double2* vhs;
  double2* ovl_new;
  double2* ene;
  double2* epart;
  double* rccat;
  void* wcopy;
  int32_t* sr_idx;
  double* cum;
  double2* free_scr;  // free projection: spin constants and QR norm factors [4][nw]
  afq::TcState tc;  // tensor-core (mixed precision) operands and plans
  DigCtx dg;        // digit-sliced FP64 operands and plans
  // Inside a block only: 1 when c->green (mixed path: the operand buffers, with G, its operands
  // and the walker operand) already belongs to the current walkers, else 0.
  int gstate;
};

namespace {

struct Layout {
  size_t off = 0;
  size_t take(size_t bytes) {
    size_t o = off;
    off += (bytes + 255) & ~(size_t)255;
    return o;
  }
};

struct Sizes {
  // digits: [tiles, row exponents]; dg .. dg_end the operands sliced once, dgw .. dgw_end the walkers'
  size_t dg, dg_chol[2], dg_rc[2], dg_u[2][2], dg_e[2][2], dg_status, dg_end;
  size_t dgw, dg_xa[2], dg_ga[2], dg_v[2], dg_x[2], dgw_end, dg_part, dg_z, dg_wt, dg_wa;
  size_t dg_ua[2], dg_ub[2], dg_utmp;  // set-up of U, in the place of the walkers' scratch
  size_t green, fb, xt, shift, fbt, vhs, ovl_new, ene, epart, rccat, wcopy, sr_idx, cum, free_scr, tc, total;
};

int derive(const afq_dims* d, afq_ctx_dev* c, int* nw_chunk, int* e_chunks, int* e_gchunk,
           size_t* welem) {
  if (!d) { afq_set_error("dims is NULL"); return -1; }
  if (d->norb < 1 || d->n_up < 1 || d->n_dn < 0 || d->nchol < 1 || d->n_walkers < 1) {
    afq_set_error("bad sizes norb=%d n_up=%d n_dn=%d nchol=%d n_walkers=%d", d->norb, d->n_up,
                  d->n_dn, d->nchol, d->n_walkers);
    return -1;
  }
  if (d->n_up > d->norb || d->n_dn > d->norb) { afq_set_error("more electrons than orbitals"); return -1; }
  if (d->precision != AFQ_PREC_FP64 && d->precision != AFQ_PREC_MIXED) {
    afq_set_error("unknown precision %d", d->precision); return -1;
  }
  if (d->walker_type != AFQ_WALKERS_RESTRICTED && d->walker_type != AFQ_WALKERS_UNRESTRICTED) {
    afq_set_error("unknown walker_type %d", d->walker_type); return -1;
  }
  if (d->trial_type != AFQ_TRIAL_RHF && d->trial_type != AFQ_TRIAL_UHF) {
    afq_set_error("unknown trial_type %d", d->trial_type); return -1;
  }
  if (d->trial_type == AFQ_TRIAL_RHF && d->n_up != d->n_dn) {
    afq_set_error("RHF requires equal number of up and down electrons"); return -1;
  }
  if (d->walker_type == AFQ_WALKERS_RESTRICTED && d->trial_type != AFQ_TRIAL_RHF) {
    afq_set_error("restricted walkers are supported with the RHF trial only"); return -1;
  }
  if (d->walker_type == AFQ_WALKERS_UNRESTRICTED && d->n_dn < 1) {
    afq_set_error("unrestricted walkers need n_dn >= 1"); return -1;
  }
  if (d->n_exp_terms < 1 || d->n_exp_terms > 32) { afq_set_error("n_exp_terms out of range"); return -1; }
  if (!(d->dt > 0.0)) { afq_set_error("dt must be positive"); return -1; }
  int nb = d->n_batch < 1 ? 1 : d->n_batch;
  if (d->n_walkers % nb != 0) { afq_set_error("n_batch must divide n_walkers"); return -1; }
  memset(c, 0, sizeof(*c));
  c->norb = d->norb;
  c->nchol = d->nchol;
  c->nw = d->n_walkers;
  c->n_exp_terms = d->n_exp_terms;
  c->dt = d->dt;
  if (d->walker_type == AFQ_WALKERS_RESTRICTED) {
    c->nslab = 1;
    c->kslab[0] = c->nocc_slab[0] = d->n_up;
    c->restricted_square = 1;
  } else {
    c->nslab = 2;
    c->kslab[0] = c->nocc_slab[0] = d->n_up;
    c->kslab[1] = c->nocc_slab[1] = d->n_dn;
  }
  c->kmax = c->kslab[0] > c->kslab[1] ? c->kslab[0] : c->kslab[1];
  c->digits = d->precision == AFQ_PREC_FP64 && !(d->mixed_config & AFQ_FP64_UNITS) ? 1 : 0;
  c->measure = c->digits && (d->mixed_config & AFQ_FP64_MEASURE) ? 1 : 0;
  if (d->trial_type == AFQ_TRIAL_RHF) {
    c->nspin_g = 1;
    c->gocc[0] = d->n_up;
    c->ktot = d->n_up * d->norb;
    c->energy_mode = (c->nslab == 1) ? 0 : 1;
  } else {
    c->nspin_g = 2;
    c->gocc[0] = d->n_up;
    c->gocc[1] = d->n_dn;
    c->ktot = (d->n_up + d->n_dn) * d->norb;
    c->energy_mode = 2;
  }
  // kernel resource limits
  if (c->kmax > 64) { afq_set_error("at most 64 electrons per spin are supported"); return -1; }
  if ((size_t)d->norb * c->kmax > 7000) { afq_set_error("norb * nocc too large (<= 7000)"); return -1; }
  *nw_chunk = d->n_walkers / nb;
  *e_gchunk = 16;
  *e_chunks = (d->nchol + *e_gchunk - 1) / *e_gchunk;
  *welem = d->precision == AFQ_PREC_FP64 ? 16 : 8;
  return 0;
}

// Shapes of the sliced FP64 operands (no pointers). The plan assumes the full part's 152 SMs, so
// that workspace sizes do not depend on where they are asked for.
constexpr int kPlanSms = 152;
constexpr int kUWalkers = 4;
constexpr size_t kUBytes = (size_t)32 << 20;
void dig_dims(const afq_ctx_dev& c, int nw_chunk, DigCtx* g) {
  const int nn = c.norb * c.norb;
  auto op = [](afq::DigOp& o, int rows, int K, int tr) {
    o.rows = rows;
    o.K = K;
    o.tr = tr;
  };
  op(g->chol, nn, c.nchol, afq::dig_tr(c.nw, nn, 1, kPlanSms));
  op(g->rc, c.nchol, c.ktot, afq::dig_tr(c.nw, c.nchol, (c.ktot + 15) / 16, kPlanSms));
  op(g->xa, 2 * c.nw, c.nchol, afq::kDigTile);
  op(g->ga, 2 * c.nw, c.ktot, afq::kDigTile);
  const int tiles = ((2 * c.nw + afq::kDigTile - 1) / afq::kDigTile) * ((c.nchol + g->rc.tr - 1) / g->rc.tr);
  g->fb = afq::dig_plan(tiles, g->rc.kb(), kPlanSms, 8);
  // Z = U G costs 4 (nocc norb)^2 per walker on the tensor cores, about 1/28 of the time of the
  // same flops on the FP64 units, where the sums over f_g cost 4 nchol norb nocc^2: even at
  // norb = 28 nchol, and U takes memory, so a quarter of that. U has 16 (nocc norb)^2 bytes whatever the
  // population: above kUBytes it takes kUWalkers. An energy with it and without, 198 orbitals and 33 electrons
  // (683 MB, 2.7 ms to form): 1 or 2 walkers 1.29 / 2.75 ms, 4 walkers 1.29 / 4.73, 64 walkers 1.3 / 54; 120 and 20
  // (92 MB): 1 to 4 walkers 0.34 / 0.75 ms; 40 and 7 (1.3 MB): 0.07 / 0.17.
  size_t u_bytes = 0;
  for (int s = 0; s < c.nspin_g; ++s) u_bytes += afq::dig_bytes((long)c.gocc[s] * c.norb, (long)c.gocc[s] * c.norb, 64);
  g->has_u = c.digits && c.norb <= 7 * c.nchol && (c.nw >= kUWalkers || u_bytes <= kUBytes) ? 1 : 0;
  // U is formed by strips of about 1024 rows: their FP64 values would otherwise take half of what U does
  g->u_strip = std::max(1, 1024 / c.norb);
  for (int s = 0; s < 2; ++s) {
    const int on = g->has_u && s < c.nspin_g ? c.gocc[s] * c.norb : 0;
    op(g->u[s], on, on, on ? afq::dig_tr(c.nw, on, 1, kPlanSms) : 16);
    op(g->ua[s], std::min(on, g->u_strip * c.norb), c.nchol, afq::kDigTile);
    op(g->ub[s], on, c.nchol, 64);
    const int t = ((2 * c.nw + afq::kDigTile - 1) / afq::kDigTile) * ((on + g->u[s].tr - 1) / g->u[s].tr);
    g->uplan[s] = afq::dig_plan(t, g->u[s].kb(), kPlanSms, 4);
  }
  afq::dig_walk_dims(c.norb, c.kslab, c.nslab, nw_chunk, &g->walk);
  // Taylor products on digits or on the FP64 units. Digits take 0.1 ms a step (14 launches) and then 0.3 to 1 us a
  // walker; the units up to kTaylorSmall a time that grows with q = norb^2 electrons, 0.3 us a walker at 20 x 5 and 2.2
  // at 40 x 12, above it several times that. Two steps in us, digits / units: 20 x 5 (q 2000), 50, 400 and 2000 walkers
  // 206 / 53, 372 / 135, 1296 / 610; 28 x 7 (5488) 203 / 121, 369 / 304, 1283 / 1380; 32 x 8 (8192) 196 / 144, 362 / 395,
  // 1283 / 1811; 40 x 7 (11200) 227 / 212, 447 / 580; 64 x 4 (16384) 236 / 240, 502 / 684; 60 x 10 (36000), 8 walkers
  // 263 / 753.
  const long q = (long)nn * c.kmax;
  const bool can = c.digits && !c.measure && c.norb <= 256;
  g->walk_fwd = can && (c.norb * c.kmax > afq::kTaylorSmall || q >= 14000 || (q >= 7500 && nw_chunk * c.nslab >= 200));
  // Forward mode, the whole call of three steps, 50 and 1000 walkers: 24 x 6 (3456) 2.37 / 2.02, 5.52 / 5.34 ms; 28 x 7
  // 2.46 / 2.29, 5.87 / 6.86; 24 x 12 (6912) 2.71 / 2.72, 7.54 / 9.81.
  g->walk_jvp = can && q >= 5000;
  // Reverse mode, 50, 200 and 1000 walkers: 20 x 5 3.18 / 2.95, 3.63 / 3.73, 7.21 / 8.26 ms; 28 x 7 3.41 / 3.45, 4.02 /
  // 4.55, 8.03 / 10.84.
  g->use_walk = can && (q >= 5000 || (long)nw_chunk * g->walk.ncol * nn >= 1000000);
}

Sizes sizes_for(const afq_dims* d, const afq_ctx_dev& c, int nw_chunk, int e_chunks, size_t welem,
                Layout* L) {
  Sizes s;
  const size_t nw = c.nw, C16 = sizeof(double2);
  s.rccat = L->take(c.nspin_g == 2 ? (size_t)c.nchol * c.ktot * sizeof(double) : 256);
  s.tc = L->take(d->precision == AFQ_PREC_MIXED ? afq::tc_workspace_bytes(c, nw_chunk, d->mixed_config)
                                                : 256);
  DigCtx g;
  if (c.digits) dig_dims(c, nw_chunk, &g);
  auto take = [&](size_t (&o)[2], const afq::DigOp& op) {
    o[0] = L->take(afq::dig_bytes(op.rows, op.K, op.tr));
    o[1] = L->take(afq::dig_exps(op.rows, op.tr));
  };
  if (c.digits) {
    s.dg = L->off;
    if (!c.measure) take(s.dg_chol, g.chol);
    take(s.dg_rc, g.rc);
    for (int i = 0; i < 2; ++i) take(s.dg_u[i], g.u[i]);
    for (int i = 0; g.use_walk && i < g.walk.n_e(c.nslab); ++i) take(s.dg_e[i], g.walk.e[i]);
    s.dg_status = L->take(256);
    s.dg_end = L->off;
  }
  const size_t scratch = L->off;
  s.green = L->take(nw * c.ktot * C16);
  s.fb = L->take(nw * c.nchol * C16);
  s.xt = L->take(nw * c.nchol * C16);
  s.shift = L->take(nw * C16);
  s.fbt = L->take(nw * C16);
  s.vhs = L->take(d->precision == AFQ_PREC_FP64 && !c.measure ? (size_t)nw_chunk * c.norb * c.norb * C16 : 256);
  s.ovl_new = L->take(nw * C16);
  s.ene = L->take(nw * C16);
  s.epart = L->take(nw * e_chunks * 5 * C16);
  s.wcopy = L->take(c.measure ? 256 : nw * c.norb * (c.kslab[0] + c.kslab[1]) * welem);
  s.sr_idx = L->take(nw * sizeof(int32_t));
  s.cum = L->take(nw * sizeof(double));
  s.free_scr = L->take(4 * nw * C16);
  if (c.digits) {
    s.dgw = L->off;
    if (!c.measure) take(s.dg_xa, g.xa);
    take(s.dg_ga, g.ga);
    if (g.use_walk) {
      s.dg_v[0] = L->take(afq::dig_walk_v_bytes(g.walk));
      s.dg_v[1] = L->take(afq::dig_walk_ve_bytes(g.walk));
      s.dg_x[0] = L->take(afq::dig_walk_x_bytes(g.walk));
      s.dg_x[1] = L->take(afq::dig_walk_xe_bytes(g.walk));
    }
    s.dgw_end = L->off;
    if (g.use_walk) {
      const size_t wt = (size_t)g.walk.chunk * c.norb * g.walk.ncol * C16;
      s.dg_wt = L->take(wt);
      s.dg_wa = L->take(wt);
    }
    size_t part = afq::dig_partial_bytes(c.nw, c.nchol, g.fb.splits);
    for (int i = 0; i < 2; ++i) part = std::max(part, afq::dig_partial_bytes(c.nw, g.u[i].rows, g.uplan[i].splits));
    s.dg_part = L->take(part);
    s.dg_z = L->take(g.has_u ? nw * c.ktot * C16 : 256);
    const size_t end = L->off;
    L->off = scratch;  // used before the walkers' scratch is
    const int big = g.ub[1].rows > g.ub[0].rows ? 1 : 0;
    take(s.dg_ua, g.ua[big]);
    take(s.dg_ub, g.ub[big]);
    s.dg_utmp = L->take((size_t)g.ua[big].rows * g.ub[big].rows * sizeof(double));
    L->off = std::max(L->off, end);
  }
  s.total = L->off;
  return s;
}

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

#define CHECK(x)            \
  do {                      \
    int _e = (x);           \
    if (_e) return _e;      \
  } while (0)

bool is_fp64(const afq_ctx* c) { return c->d.precision == AFQ_PREC_FP64; }

// The guard word of the context's tensor-core kernels (NULL without any)
const int* status_word(const afq_ctx* c) { return is_fp64(c) ? c->dg.status : c->tc.status; }

// rot_chol with rows g, both spins of a UHF trial together
const double* rc_all(const afq_ctx* c) { return c->dev.nspin_g == 2 ? c->rccat : c->dev.rot_chol[0]; }

// Green's function + overlap. FP64: G into c->green. Mixed: the 16-bit operands of the
// force-bias, energy and exp_h1 contractions (wg) and/or the overlap.
// chain (inside a block): the walkers are propagated next, so the same launch also forms G (mixed
// path: and the operands); c->gstate records that for the next step.
int green(afq_ctx* c, const void* wu, const void* wd, double2* g, double2* ovl, bool wg, cudaStream_t st,
          bool chain = false) {
  if (is_fp64(c))
    CHECK(afq::launch_green<double>(c->dev, wu, wd, chain ? c->green : g, ovl, wg || chain, st));
  else
    CHECK(afq::tc_green(c->tc, c->dev, wu, wd, ovl, wg, st, chain));
  c->gstate = chain ? 1 : 0;
  return 0;
}

// out [nw][nchol] = alpha g . rc^T (FP64), alpha = 2 (RHF, one slab) or 1; rc and its digits
int fb_gemm(afq_ctx* c, const double2* g, const double* rcd, const afq::DigOp& rc, double2* out, cudaStream_t st,
            bool coulomb = false) {
  const afq_ctx_dev& d = c->dev;
  if (!d.digits)
    return afq::launch_gemm_cr(false, d.nw, d.nchol, d.ktot, g, d.ktot, rcd, d.ktot, out, d.nchol,
                               c2(d.energy_mode == 0 && !coulomb ? 2.0 : 1.0, 0.0), st);
  CHECK(afq::dig_slice_cplx_rows(c->dg.ga, g, d.ktot, 1.0, st));
  return afq::dig_gemm_c(coulomb ? afq::K_ENERGY : afq::K_FB, c->dg.ga, rc, d.nw, d.nchol, out, d.nchol, 0,
                         d.energy_mode == 0 && !coulomb ? 1 : 0, c->dg.fb, c->dg.part, c->dg.status, st);
}

// The local energy's contractions of c->green: c->fb = Coulomb sums, dg.z = U G (FP64)
int energy_gemms(afq_ctx* c, cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  CHECK(fb_gemm(c, c->green, rc_all(c), c->dg.rc, c->fb, st, true));
  for (int s = 0, off = 0; s < d.nspin_g; ++s) {
    afq::DigOp a = c->dg.ga;
    a.K = c->dg.u[s].K;
    if (d.nspin_g == 2) CHECK(afq::dig_slice_cplx_rows(a, c->green + off, d.ktot, 1.0, st));  // else as sliced above
    CHECK(afq::dig_gemm_c(afq::K_ENERGY, a, c->dg.u[s], d.nw, a.K, c->dg.z + off, d.ktot, 0, 0, c->dg.uplan[s],
                          c->dg.part, c->dg.status, st));
    off += a.K;
  }
  return 0;
}

// vhs [nwc][norb^2] = i sqrt(dt) x . chol (FP64)
int vhs_gemm(afq_ctx* c, const double2* x, int nwc, double2* vhs, cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  const int nn = d.norb * d.norb;
  if (!d.digits)
    return afq::launch_gemm_cr(true, nwc, nn, d.nchol, x, d.nchol, c->h.chol, nn, vhs, nn, c2(0.0, sqrt(d.dt)), st);
  afq::DigOp a = c->dg.xa;
  a.rows = 2 * nwc;
  CHECK(afq::dig_slice_cplx_rows(a, x, d.nchol, sqrt(d.dt), st));
  return afq::dig_gemm_c(afq::K_VHS, a, c->dg.chol, nwc, nn, vhs, nn, 1, 0, afq::DigPlan{1, a.kb()}, nullptr,
                         c->dg.status, st);
}

int force_bias_from_green(afq_ctx* c, double2* out, cudaStream_t st) {
  if (!is_fp64(c)) return afq::tc_force_bias(c->tc, c->dev, out, st);
  return fb_gemm(c, c->green, rc_all(c), c->dg.rc, out, st);
}

int energy_from_green(afq_ctx* c, double2* out, cudaStream_t st) {
  if (!is_fp64(c)) return afq::tc_energy(c->tc, c->dev, out, st);
  if (c->dg.has_u) {
    CHECK(energy_gemms(c, st));
    return afq::dig_launch_energy(c->dev, c->green, c->dg.z, c->fb, out, c->dg.status, st);
  }
  return afq::launch_energy_f64(c->dev, c->e_chunks, c->e_gchunk, c->green, c->epart, out, st);
}

int check_walkers(const afq_ctx* c, const void* wu, const void* wd) {
  if (!wu) { afq_set_error("walkers_up is NULL"); return -1; }
  if (c->dev.nslab == 2 && !wd) { afq_set_error("unrestricted walkers need walkers_dn"); return -1; }
  return 0;
}

int check_state(const afq_ctx* c, const afq_walker_state* s) {
  if (!s) { afq_set_error("state is NULL"); return -1; }
  if (c->dev.measure) { afq_set_error("the context was created for measurements only"); return -1; }
  CHECK(check_walkers(c, s->walkers_up, s->walkers_dn));
  if (!s->weights || !s->overlaps || !s->scalars) { afq_set_error("state has NULL arrays"); return -1; }
  return 0;
}

// The walker slabs from walker w0 on, and a [walker][norb * (k0 + k1)] buffer.
afq::WalkVec walk_slabs(const afq_ctx_dev& d, void* wu, void* wd, size_t w0) {
  const size_t a = (size_t)d.norb * d.kslab[0], b = (size_t)d.norb * d.kslab[1];
  return {{static_cast<double2*>(wu) + w0 * a, d.nslab == 2 ? static_cast<double2*>(wd) + w0 * b : nullptr}, a, b};
}
afq::WalkVec walk_buf(const afq_ctx_dev& d, double2* p, size_t nterm = 1) {
  const size_t a = (size_t)d.norb * d.kslab[0], b = (size_t)d.norb * d.kslab[1];
  return {{p, d.nslab == 2 ? p + a : nullptr}, nterm * (a + b), nterm * (a + b)};
}

// out = E_s y_s for every slab (y sliced); acc (optional) = out
int walk_exp(const afq::DigWalk& w, const afq_ctx_dev& d, const afq::DigOp* E, const afq::WalkOut& o, int nw,
             cudaStream_t st) {
  for (int s = 0; s < w.n_e(d.nslab); ++s) CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w, s, E, o, nw, st));
  return 0;
}

// W <- E exp(V) E W (propagation.py:67-92) of nwc walkers from w0 on, FP64
int taylor_fp64(afq_ctx* c, int w0, int nwc, const double2* vhs, void* wu, void* wd, cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  if (!c->dg.walk_fwd) return afq::launch_taylor_f64<double>(d, w0, nwc, vhs, wu, wd, st);
  const afq::DigWalk& w = c->dg.walk;
  const afq::WalkVec T = walk_buf(d, c->dg.walk_t), A = walk_buf(d, c->dg.walk_acc);
  for (int k = 0; k < nwc; k += w.chunk) {
    const int nw = std::min(w.chunk, nwc - k);
    const afq::WalkVec W = walk_slabs(d, wu, wd, (size_t)w0 + k);
    CHECK(afq::dig_walk_slice_v(w, vhs + (size_t)k * d.norb * d.norb, nw, false, st));
    CHECK(afq::dig_walk_slice_y(w, W, nw, st));
    afq::WalkOut o;
    o.out = T;
    o.acc = A;
    o.init = 1;
    CHECK(walk_exp(w, d, w.e, o, nw, st));
    o.init = 0;
    double fact = 1.0;
    for (int m = 1; m < d.n_exp_terms; ++m) {
      fact *= (double)m;
      o.facc = 1.0 / fact;
      CHECK(afq::dig_walk_slice_y(w, T, nw, st));
      CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w, -1, nullptr, o, nw, st));
    }
    CHECK(afq::dig_walk_slice_y(w, A, nw, st));
    afq::WalkOut last;
    last.out = W;
    CHECK(walk_exp(w, d, w.e, last, nw, st));
  }
  return 0;
}

// The same with tangents (t_launch_taylor's products): V and the walkers in w's digits, their
// tangents in dw's.
int taylor_jvp(afq_ctx* c, const afq::TangentBufs& t, const afq::DigWalk& dw, double2* dt_buf, double2* da_buf, int w0,
               int nwc, const double2* vhs, void* wu, void* wd, cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  const afq::DigWalk& w = c->dg.walk;
  const afq::WalkVec T = walk_buf(d, c->dg.walk_t), A = walk_buf(d, c->dg.walk_acc), dT = walk_buf(d, dt_buf),
                     dA = walk_buf(d, da_buf);
  afq::DigWalk w_dy = w, dw_y = dw;  // V with the tangent columns, dV with the value columns
  w_dy.xd = dw.xd;
  w_dy.xe = dw.xe;
  dw_y.xd = w.xd;
  dw_y.xe = w.xe;
  for (int k = 0; k < nwc; k += w.chunk) {
    const int nw = std::min(w.chunk, nwc - k);
    const size_t vo = (size_t)k * d.norb * d.norb;
    const afq::WalkVec W = walk_slabs(d, wu, wd, (size_t)w0 + k), dW = walk_slabs(d, t.dw[0], t.dw[1], (size_t)w0 + k);
    CHECK(afq::dig_walk_slice_v(w, vhs + vo, nw, false, st));
    CHECK(afq::dig_walk_slice_v(dw, t.dvhs + vo, nw, false, st));
    // (out, acc) = (r, acc + f r) of r = X y, and of its tangent X dy + dX y
    auto both = [&](const afq::WalkVec& y, const afq::WalkVec& dy, int e, afq::WalkOut o, afq::WalkOut od) -> int {
      CHECK(afq::dig_walk_slice_y(w, y, nw, st));
      CHECK(afq::dig_walk_slice_y(dw, dy, nw, st));
      afq::WalkOut part;
      part.out = od.out;
      od.in = od.out;
      if (e < 0) {
        CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w, -1, nullptr, o, nw, st));
        CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w_dy, -1, nullptr, part, nw, st));
        return afq::dig_walk_mul(afq::K_TAYLOR, dw_y, -1, nullptr, od, nw, st);
      }
      CHECK(walk_exp(w, d, w.e, o, nw, st));
      CHECK(walk_exp(w_dy, d, w.e, part, nw, st));
      return walk_exp(dw_y, d, dw.e, od, nw, st);
    };
    afq::WalkOut o, od;
    o.out = T;
    o.acc = A;
    od.out = dT;
    od.acc = dA;
    o.init = od.init = 1;
    CHECK(both(W, dW, 0, o, od));
    o.init = od.init = 0;
    double fact = 1.0;
    for (int m = 1; m < d.n_exp_terms; ++m) {
      fact *= (double)m;
      o.facc = od.facc = 1.0 / fact;
      CHECK(both(T, dT, -1, o, od));
    }
    afq::WalkOut last, dlast;
    last.out = W;
    dlast.out = dW;
    CHECK(both(A, dA, 0, last, dlast));
  }
  return 0;
}

// chain: a step inside afq_propagate_phaseless, where the Green's-function work of the
// previous overlap evaluation on the same walkers (c->gstate) is reused.
// next_g (with chain): the next operation propagates the same walkers again, so the overlap
// evaluation after the step also forms G and the operands (not before a QR).
int propagate_impl(afq_ctx* c, afq_walker_state* s, const double* fields, cudaStream_t st,
                   bool chain = false, bool next_g = true) {
  const afq_ctx_dev& d = c->dev;
  if (!is_fp64(c)) {
    // mixed: operands -> fused force bias / field shifts -> exp_h1, vhs + Taylor, exp_h1
    if (!(chain && c->gstate == 1)) CHECK(afq::tc_green(c->tc, d, s->walkers_up, s->walkers_dn, nullptr, true, st));
    CHECK(afq::tc_field_shifts(c->tc, d, fields, st));
    CHECK(afq::tc_propagate_walkers(c->tc, d, s->walkers_up, s->walkers_dn, st));
    CHECK(green(c, s->walkers_up, s->walkers_dn, nullptr, c->ovl_new, false, st, chain && next_g));
    return afq::tc_weights(c->tc, d, c->ovl_new, reinterpret_cast<double2*>(s->overlaps), s->weights,
                           s->scalars, st);
  }
  if (!(chain && c->gstate == 1)) CHECK(green(c, s->walkers_up, s->walkers_dn, c->green, nullptr, true, st));
  CHECK(force_bias_from_green(c, c->fb, st));
  CHECK(afq::launch_field_shifts(d, fields, c->fb, c->xt, c->shift, c->fbt, st));
  const int nb = d.nw / c->nw_chunk;
  for (int b = 0; b < nb; ++b) {
    const int w0 = b * c->nw_chunk;
    CHECK(vhs_gemm(c, c->xt + (size_t)w0 * d.nchol, c->nw_chunk, c->vhs, st));
    CHECK(taylor_fp64(c, w0, c->nw_chunk, c->vhs, s->walkers_up, s->walkers_dn, st));
  }
  CHECK(green(c, s->walkers_up, s->walkers_dn, nullptr, c->ovl_new, false, st, chain && next_g));
  return afq::launch_weights(d, c->shift, c->fbt, 1, c->ovl_new, reinterpret_cast<double2*>(s->overlaps),
                             s->weights, s->scalars, st, c->dg.status);
}

int qr_impl(afq_ctx* c, afq_walker_state* s, cudaStream_t st) {
  if (is_fp64(c)) return afq::launch_qr_f64(c->dev, s->walkers_up, s->walkers_dn, st);
  return afq::launch_qr_f32(c->dev, s->walkers_up, s->walkers_dn, st);
}

int sr_impl(afq_ctx* c, afq_walker_state* s, const double* zeta, int32_t* indices, cudaStream_t st) {
  if (is_fp64(c))
    CHECK(afq::launch_sr<double>(c->dev, zeta, s->weights, c->cum, c->sr_idx, s->walkers_up,
                                 s->walkers_dn, c->wcopy, st));
  else
    CHECK(afq::launch_sr<float>(c->dev, zeta, s->weights, c->cum, c->sr_idx, s->walkers_up,
                                s->walkers_dn, c->wcopy, st));
  if (indices) {
    cudaError_t e = cudaMemcpyAsync(indices, c->sr_idx, sizeof(int32_t) * c->dev.nw,
                                    cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) { afq_set_error("sr index copy: %s", cudaGetErrorString(e)); return (int)e; }
  }
  return 0;
}

// One free-projection step (propagation.py:436-462), FP64 unrestricted walkers.
int free_step(afq_ctx* c, afq_walker_state* s, const double* fields, double ene0, double2* norms, double2* normed,
              cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  double2* consts = c->free_scr;
  double2* rdiag = c->free_scr + 2 * (size_t)d.nw;
  double2* ovl = reinterpret_cast<double2*>(s->overlaps);
  CHECK(afq::launch_free_prep(d, fields, ene0, c->xt, consts, st));
  const int nb = d.nw / c->nw_chunk;
  for (int b = 0; b < nb; ++b) {
    const int w0 = b * c->nw_chunk;
    CHECK(vhs_gemm(c, c->xt + (size_t)w0 * d.nchol, c->nw_chunk, c->vhs, st));
    CHECK(taylor_fp64(c, w0, c->nw_chunk, c->vhs, s->walkers_up, s->walkers_dn, st));
  }
  CHECK(afq::launch_free_scale(d, consts, s->walkers_up, s->walkers_dn, st));
  CHECK(afq::launch_qr_f64(d, s->walkers_up, s->walkers_dn, st, rdiag));
  CHECK(green(c, s->walkers_up, s->walkers_dn, nullptr, ovl, false, st));
  CHECK(afq::launch_free_finish(d.nw, rdiag, norms, ovl, st));
  // normed overlaps: the walkers through the QR once more, on a copy
  const size_t e0 = (size_t)d.nw * d.norb * d.kslab[0], e1 = (size_t)d.nw * d.norb * d.kslab[1];
  double2* cu = static_cast<double2*>(c->wcopy);
  double2* cd = cu + e0;
  cudaError_t e = cudaMemcpyAsync(cu, s->walkers_up, e0 * sizeof(double2), cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(cd, s->walkers_dn, e1 * sizeof(double2), cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) { afq_set_error("walker copy: %s", cudaGetErrorString(e)); return (int)e; }
  CHECK(afq::launch_qr_f64(d, cu, cd, st));
  return green(c, cu, cd, nullptr, normed, false, st);
}

int check_free(const afq_ctx* c) {
  if (!is_fp64(c) || c->dev.nslab != 2) {
    afq_set_error("free projection needs an FP64 context with unrestricted walkers");
    return -1;
  }
  return 0;
}

// Tangent workspace of afq_propagate_phaseless_jvp, carved like the main workspace.
struct TSizes {
  size_t dw[2], wold[2], dgreen, dfb, dxt, dshift, dfbt, dvhs, dlo, dlo_new, dweights, dscalars, dene, dpart,
      dsum, drccat, drc_d, drc_e, total;  // drc_*: sliced drccat
  size_t wk, de[2][2], v[2], x[2], wt, wa;  // digits of the tangent Taylor products
};

TSizes tangent_sizes(const afq_ctx_dev& c, int nw_chunk, int e_chunks, Layout* L) {
  TSizes s;
  const size_t nw = c.nw, C16 = sizeof(double2);
  for (int k = 0; k < 2; ++k) {  // kslab[1] is 0 for restricted walkers
    s.dw[k] = L->take(nw * c.norb * c.kslab[k] * C16);
    s.wold[k] = L->take(nw * c.norb * c.kslab[k] * C16);
  }
  s.dgreen = L->take(nw * c.ktot * C16);
  s.dfb = L->take(nw * c.nchol * C16);
  s.dxt = L->take(nw * c.nchol * C16);
  s.dshift = L->take(nw * C16);
  s.dfbt = L->take(nw * C16);
  s.dvhs = L->take((size_t)nw_chunk * c.norb * c.norb * C16);
  s.dlo = L->take(nw * C16);
  s.dlo_new = L->take(nw * C16);
  s.dweights = L->take(nw * sizeof(double));
  s.dscalars = L->take(AFQ_NSCALARS * sizeof(double));
  s.dene = L->take(nw * C16);
  s.dpart = L->take(nw * e_chunks * 5 * C16);
  s.dsum = L->take(sizeof(double));
  s.drccat = L->take(c.nspin_g == 2 ? (size_t)c.nchol * c.ktot * sizeof(double) : 256);
  DigCtx g;
  dig_dims(c, nw_chunk, &g);
  if (c.digits) {
    s.drc_d = L->take(afq::dig_bytes(g.rc.rows, g.rc.K, g.rc.tr));
    s.drc_e = L->take(afq::dig_exps(g.rc.rows, g.rc.tr));
  }
  s.wk = L->off;
  if (g.walk_jvp) {
    for (int i = 0; i < g.walk.n_e(c.nslab); ++i) {
      s.de[i][0] = L->take(afq::dig_bytes(g.walk.e[i].rows, c.norb));
      s.de[i][1] = L->take(afq::dig_exps(g.walk.e[i].rows));
    }
    s.v[0] = L->take(afq::dig_walk_v_bytes(g.walk));
    s.v[1] = L->take(afq::dig_walk_ve_bytes(g.walk));
    s.x[0] = L->take(afq::dig_walk_x_bytes(g.walk));
    s.x[1] = L->take(afq::dig_walk_xe_bytes(g.walk));
    s.wt = L->take((size_t)g.walk.chunk * c.norb * g.walk.ncol * C16);
    s.wa = L->take((size_t)g.walk.chunk * c.norb * g.walk.ncol * C16);
  }
  s.total = L->off;
  return s;
}

// The Taylor products' tangent operands: dV, the tangent columns and d exp_h1; term and sum.
struct JvpWalk {
  afq::DigWalk w;
  double2 *t, *a;
};

// One phaseless step with tangents (propagate_impl's FP64 branch, each stage followed by
// its tangent). c->green and t.dgreen belong to the walkers; next_g: also after the step.
int propagate_jvp(afq_ctx* c, afq_walker_state* s, const afq::TangentBufs& t, const afq::DigOp& drc,
                  const JvpWalk& jw, const double* fields, cudaStream_t st, bool next_g) {
  const afq_ctx_dev& d = c->dev;
  CHECK(force_bias_from_green(c, c->fb, st));
  CHECK(fb_gemm(c, t.dgreen, rc_all(c), c->dg.rc, t.dfb, st));
  if (t.drccat) {  // orbital rotation: + alpha G dRC^T (t.dxt as scratch, rewritten below)
    CHECK(fb_gemm(c, c->green, t.drccat, drc, t.dxt, st));
    CHECK(afq::t_launch_add((long)d.nw * d.nchol, t.dxt, t.dfb, st));
  }
  CHECK(afq::t_launch_field_shifts(d, fields, c->fb, t.dfb, c->xt, t.dxt, c->shift, t.dshift, c->fbt, t.dfbt, st));
  const int nb = d.nw / c->nw_chunk;
  for (int b = 0; b < nb; ++b) {
    const int w0 = b * c->nw_chunk;
    CHECK(vhs_gemm(c, c->xt + (size_t)w0 * d.nchol, c->nw_chunk, c->vhs, st));
    CHECK(vhs_gemm(c, t.dxt + (size_t)w0 * d.nchol, c->nw_chunk, t.dvhs, st));
    if (c->dg.walk_jvp)
      CHECK(taylor_jvp(c, t, jw.w, jw.t, jw.a, w0, c->nw_chunk, c->vhs, s->walkers_up, s->walkers_dn, st));
    else
      CHECK(afq::t_launch_taylor(d, t, w0, c->nw_chunk, c->vhs, t.dvhs, s->walkers_up, s->walkers_dn, st));
  }
  CHECK(afq::t_launch_green(d, t, s->walkers_up, s->walkers_dn, next_g ? c->green : nullptr,
                            next_g ? t.dgreen : nullptr, c->ovl_new, t.dlo_new, st));
  return afq::t_launch_weights(d, t, c->shift, c->fbt, c->ovl_new, reinterpret_cast<double2*>(s->overlaps),
                               s->weights, s->scalars, st);
}

int copy_d2d(void* dst, const void* src, size_t bytes, cudaStream_t st, const char* what) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) { afq_set_error("%s: %s", what, cudaGetErrorString(e)); return (int)e; }
  return 0;
}

// Sliced operands of the backward sweep: Cholesky vectors with rows g (field cotangents from V
// cotangents), rot_chol with rows (i, p) (G cotangents), the V cotangents, and the K ranges of
// the field cotangents (K = norb^2).
struct AdjOps {
  afq::DigOp cn, rt, va;
  afq::DigPlan xtb;
};
// The Taylor adjoint on the digit GEMM (at least one V product)
bool adj_walk(const afq_ctx_dev& c, const DigCtx& g) { return g.use_walk && c.n_exp_terms >= 2; }

AdjOps adj_ops(const afq_ctx_dev& c, int nwc) {
  AdjOps o;
  const int nn = c.norb * c.norb, kb = (nn + 15) / 16;
  o.cn.rows = c.nchol;
  o.cn.K = nn;
  o.cn.tr = afq::dig_tr(nwc, c.nchol, kb, kPlanSms);
  o.rt.rows = c.ktot;
  o.rt.K = c.nchol;
  o.rt.tr = afq::dig_tr(c.nw, c.ktot, 1, kPlanSms);
  o.va.rows = 2 * nwc;
  o.va.K = nn;
  o.xtb = afq::dig_plan(((2 * nwc + afq::kDigTile - 1) / afq::kDigTile) * ((c.nchol + o.cn.tr - 1) / o.cn.tr), kb,
                        kPlanSms, 16);
  return o;
}

// Workspace of afq_propagate_phaseless_vjp: the recorded forward sweep (snapshots of the
// walker state before every step, after the last step of an energy block and after its QR;
// shifted fields and shift terms of every step; local energies of every block; SR indices)
// followed by the backward sweep's cotangents.
struct AdjSizes {
  size_t snap_w, snap_wt, snap_ov, snap_sc, t_xt, t_sh, t_fbt, t_ene, t_idx;
  size_t wb, wb2, wbar, lbar, lbar2, gpend, gene, fbb, xtb, shb, fbtb, vbar, tay, exp_part, ebar, scal, beb, bwb, total;
  size_t dg_end, part, et[2][2], vb_ad, vb_ae, vb_bd, vb_be;  // exp_h1^T; operands of the V cotangents
  size_t dg, cn_d, cn_e, rt_d, rt_e, va_d, va_e;  // digits: chol (rows g), rot_chol^T, V cotangents
  size_t wslab;  // walker elements of one snapshot, both slabs
  int nblk, nsteps, nsnap;
};

AdjSizes adjoint_sizes(const afq_ctx_dev& c, int nw_chunk, int n_prop, int n_ene, int n_sr, Layout* L) {
  AdjSizes s;
  const size_t nw = c.nw, C16 = sizeof(double2), nk = (size_t)c.norb * (c.kslab[0] + c.kslab[1]);
  s.nblk = n_ene * n_sr;
  s.nsteps = s.nblk * n_prop;
  s.nsnap = s.nblk * (n_prop + 2);
  s.wslab = nw * nk;
  s.snap_w = L->take((size_t)s.nsnap * s.wslab * C16);
  s.snap_wt = L->take((size_t)s.nsnap * nw * sizeof(double));
  s.snap_ov = L->take((size_t)s.nsnap * nw * C16);
  s.snap_sc = L->take((size_t)s.nsnap * AFQ_NSCALARS * sizeof(double));
  s.t_xt = L->take((size_t)s.nsteps * nw * c.nchol * C16);
  s.t_sh = L->take((size_t)s.nsteps * nw * C16);
  s.t_fbt = L->take((size_t)s.nsteps * nw * C16);
  s.t_ene = L->take((size_t)s.nblk * nw * C16);
  s.t_idx = L->take((size_t)n_sr * nw * sizeof(int32_t));
  s.wb = L->take(s.wslab * C16);
  s.wb2 = L->take(s.wslab * C16);
  s.wbar = L->take(nw * sizeof(double));
  s.lbar = L->take(nw * C16);
  s.lbar2 = L->take(nw * C16);
  s.gpend = L->take(nw * c.ktot * C16);
  s.gene = L->take(nw * c.ktot * C16);
  s.fbb = L->take(nw * c.nchol * C16);
  s.xtb = L->take(nw * c.nchol * C16);
  s.shb = L->take(nw * C16);
  s.fbtb = L->take(nw * C16);
  s.vbar = L->take((size_t)nw_chunk * c.norb * c.norb * C16);
  s.tay = L->take((size_t)nw_chunk * (2 * (c.n_exp_terms - 1) + 2) * nk * C16);
  s.exp_part = L->take((size_t)afq::kExpSplits * c.nslab * c.norb * c.norb * sizeof(double));
  s.ebar = L->take(nw * sizeof(double));
  s.scal = L->take(8 * sizeof(double));
  s.beb = L->take((size_t)s.nblk * sizeof(double));
  s.bwb = L->take((size_t)s.nblk * sizeof(double));
  s.dg = s.dg_end = s.part = L->off;
  if (!c.digits) {
    s.total = L->off;
    return s;
  }
  const AdjOps o = adj_ops(c, nw_chunk);
  s.cn_d = L->take(afq::dig_bytes(o.cn.rows, o.cn.K, o.cn.tr));
  s.cn_e = L->take(afq::dig_exps(o.cn.rows, o.cn.tr));
  s.rt_d = L->take(afq::dig_bytes(o.rt.rows, o.rt.K, o.rt.tr));
  s.rt_e = L->take(afq::dig_exps(o.rt.rows, o.rt.tr));
  s.va_d = L->take(afq::dig_bytes(o.va.rows, o.va.K));
  s.va_e = L->take(afq::dig_exps(o.va.rows));
  DigCtx g;
  dig_dims(c, nw_chunk, &g);
  if (adj_walk(c, g)) {
    afq::DigVbar v;
    afq::dig_walk_vbar_dims(g.walk, c.n_exp_terms - 1, &v);
    for (int i = 0; i < g.walk.n_e(c.nslab); ++i) {
      s.et[i][0] = L->take(afq::dig_bytes(g.walk.e[i].rows, c.norb));
      s.et[i][1] = L->take(afq::dig_exps(g.walk.e[i].rows));
    }
    s.vb_ad = L->take(afq::dig_walk_vbar_a_bytes(g.walk, v));
    s.vb_ae = L->take(afq::dig_walk_vbar_ae_bytes(g.walk, v));
    s.vb_bd = L->take(afq::dig_walk_vbar_b_bytes(g.walk, v));
    s.vb_be = L->take(afq::dig_walk_vbar_be_bytes(g.walk, v));
  }
  s.dg_end = L->off;
  s.part = L->take(afq::dig_partial_bytes(nw_chunk, c.nchol, o.xtb.splits));
  s.total = L->off;
  return s;
}

// Views of the recorded forward sweep. Snapshot i = blk * (n_prop + 2) + j: j < n_prop
// before step j, j == n_prop after the last step (before the QR), j == n_prop + 1 after
// the QR and the overlap evaluation.
struct Tape {
  char* base;
  AdjSizes s;
  const afq_ctx_dev* d;
  double2* w(int i, int slab) const {
    return reinterpret_cast<double2*>(base + s.snap_w) + (size_t)i * s.wslab +
           (slab ? (size_t)d->nw * d->norb * d->kslab[0] : 0);
  }
  double* wt(int i) const { return reinterpret_cast<double*>(base + s.snap_wt) + (size_t)i * d->nw; }
  double2* ov(int i) const { return reinterpret_cast<double2*>(base + s.snap_ov) + (size_t)i * d->nw; }
  double* sc(int i) const { return reinterpret_cast<double*>(base + s.snap_sc) + (size_t)i * AFQ_NSCALARS; }
  double2* xt(int step) const {
    return reinterpret_cast<double2*>(base + s.t_xt) + (size_t)step * d->nw * d->nchol;
  }
  double2* sh(int step) const { return reinterpret_cast<double2*>(base + s.t_sh) + (size_t)step * d->nw; }
  double2* fbt(int step) const { return reinterpret_cast<double2*>(base + s.t_fbt) + (size_t)step * d->nw; }
  double2* ene(int blk) const { return reinterpret_cast<double2*>(base + s.t_ene) + (size_t)blk * d->nw; }
  int32_t* idx(int sr) const { return reinterpret_cast<int32_t*>(base + s.t_idx) + (size_t)sr * d->nw; }
};

// The Taylor adjoint (a_launch_taylor's chain and layout of a.tay) on the digit GEMM: products
// with V, then with V^H, then the V cotangents; et: exp_h1^T per slab.
int taylor_vjp(afq_ctx* c, const afq::AdjointBufs& a, const afq::DigOp* et, const afq::DigVbar& vb, int w0, int nwc,
               const double2* vhs, double2* wu, double2* wd, cudaStream_t st) {
  const afq_ctx_dev& d = c->dev;
  const afq::DigWalk& w = c->dg.walk;
  const int M = d.n_exp_terms - 1, T = 2 * M + 2;
  const size_t nk = (size_t)d.norb * w.ncol, nn = (size_t)d.norb * d.norb;
  const afq::WalkVec B = walk_buf(d, c->dg.walk_acc);  // W'-bar through exp_h1^T
  for (int k = 0; k < nwc; k += w.chunk) {
    const int nw = std::min(w.chunk, nwc - k);
    double2* tay = a.tay + (size_t)k * T * nk;
    auto term = [&](int i) { return walk_buf(d, tay + (size_t)i * nk, T); };
    CHECK(afq::dig_walk_slice_v(w, vhs + k * nn, nw, false, st));
    CHECK(afq::dig_walk_slice_y(w, walk_slabs(d, wu, wd, (size_t)w0 + k), nw, st));
    afq::WalkOut f;
    f.out = term(0);
    f.acc = term(2 * M);
    f.init = 1;
    CHECK(walk_exp(w, d, w.e, f, nw, st));
    f.init = 0;
    double fact = 1.0;
    for (int m = 1; m <= M; ++m) {
      fact *= (double)m;
      f.facc = 1.0 / fact;
      f.out = m < M ? term(m) : afq::WalkVec{{nullptr, nullptr}, 0};
      CHECK(afq::dig_walk_slice_y(w, term(m - 1), nw, st));
      CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w, -1, nullptr, f, nw, st));
    }
    CHECK(afq::dig_walk_slice_v(w, vhs + k * nn, nw, true, st));
    CHECK(afq::dig_walk_slice_y(w, walk_slabs(d, a.wb[0], a.wb[1], (size_t)w0 + k), nw, st));
    afq::WalkOut top;
    top.out = term(2 * M - 1);
    top.fout = 1.0 / fact;
    top.acc = B;
    top.init = 1;
    CHECK(walk_exp(w, d, et, top, nw, st));
    double invf = 1.0 / fact;
    for (int m = M - 1; m >= 0; --m) {
      invf *= (double)(m + 1);  // 1 / m!
      CHECK(afq::dig_walk_slice_y(w, term(M + m), nw, st));
      afq::WalkOut o;
      o.out = term(m >= 1 ? M + m - 1 : 2 * M + 1);
      o.in = B;
      o.fin = invf;
      CHECK(afq::dig_walk_mul(afq::K_TAYLOR, w, -1, nullptr, o, nw, st));
    }
    CHECK(afq::dig_walk_slice_y(w, term(2 * M + 1), nw, st));
    afq::WalkOut out;
    out.out = walk_slabs(d, a.wb2[0], a.wb2[1], (size_t)w0 + k);
    CHECK(walk_exp(w, d, et, out, nw, st));
    CHECK(afq::dig_walk_vbar(w, vb, tay, T, M, 0, M, a.vbar + k * nn, nw, st));
  }
  return afq::a_launch_exp_grad(d, a, w0, nwc, wu, wd, st);
}

int snapshot(const Tape& t, int i, const afq_walker_state* st_, cudaStream_t st) {
  const afq_ctx_dev& d = *t.d;
  const size_t e0 = (size_t)d.nw * d.norb * d.kslab[0], e1 = (size_t)d.nw * d.norb * d.kslab[1];
  CHECK(copy_d2d(t.w(i, 0), st_->walkers_up, e0 * sizeof(double2), st, "walker snapshot"));
  if (d.nslab == 2) CHECK(copy_d2d(t.w(i, 1), st_->walkers_dn, e1 * sizeof(double2), st, "walker snapshot"));
  CHECK(copy_d2d(t.wt(i), st_->weights, d.nw * sizeof(double), st, "weight snapshot"));
  CHECK(copy_d2d(t.ov(i), st_->overlaps, d.nw * sizeof(double2), st, "overlap snapshot"));
  return copy_d2d(t.sc(i), st_->scalars, AFQ_NSCALARS * sizeof(double), st, "scalar snapshot");
}

int zero(void* p, size_t bytes, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(p, 0, bytes, st);
  if (e != cudaSuccess) { afq_set_error("memset: %s", cudaGetErrorString(e)); return (int)e; }
  return 0;
}

void swap_slabs(double2* a[2], double2* b[2]) {
  for (int k = 0; k < 2; ++k) {
    double2* t = a[k];
    a[k] = b[k];
    b[k] = t;
  }
}

}  // namespace

extern "C" {

int afq_abi_version(void) { return AFQ_ABI_VERSION; }

int afq_test_preset_status(afq_ctx* ctx, int bits, void* stream) {
  if (!ctx || bits < 0 || bits > 255 || !status_word(ctx)) { afq_set_error("bad argument"); return -1; }
  // the word's low byte (little endian); the rest stays zero
  const cudaError_t e = cudaMemsetAsync(const_cast<int*>(status_word(ctx)), bits, 1, S(stream));
  if (e != cudaSuccess) { afq_set_error("preset status: %s", cudaGetErrorString(e)); return (int)e; }
  return 0;
}

const char* afq_last_error(void) { return g_err; }

size_t afq_workspace_size(const afq_dims* dims) {
  afq_ctx_dev c;
  int nwc, ec, eg;
  size_t we;
  if (derive(dims, &c, &nwc, &ec, &eg, &we)) return 0;
  Layout L;
  return sizes_for(dims, c, nwc, ec, we, &L).total;
}

int afq_ctx_create(const afq_dims* dims, const afq_hamiltonian* ham, void* workspace,
                   size_t workspace_bytes, void* stream, afq_ctx** out) {
  if (!out) { afq_set_error("out is NULL"); return -1; }
  *out = nullptr;
  afq_ctx_dev dev;
  int nwc, ec, eg;
  size_t we;
  CHECK(derive(dims, &dev, &nwc, &ec, &eg, &we));
  if (!ham) { afq_set_error("hamiltonian is NULL"); return -1; }
  const bool uhf = dims->trial_type == AFQ_TRIAL_UHF;
  const bool unres = dims->walker_type == AFQ_WALKERS_UNRESTRICTED;
  if (!ham->trial_up || !ham->chol || !ham->rot_chol_up || !ham->rot_h1_up || !ham->exp_h1_up ||
      !ham->mf_shifts || (uhf && (!ham->trial_dn || !ham->rot_chol_dn || !ham->rot_h1_dn)) ||
      (unres && !ham->exp_h1_dn)) {
    afq_set_error("hamiltonian has NULL arrays");
    return -1;
  }
  Layout L;
  Sizes sz = sizes_for(dims, dev, nwc, ec, we, &L);
  if (!workspace || workspace_bytes < sz.total) {
    afq_set_error("workspace too small: need %zu bytes, got %zu", sz.total, workspace_bytes);
    return -1;
  }
  if (reinterpret_cast<uintptr_t>(workspace) & 255) { afq_set_error("workspace must be 256-byte aligned"); return -1; }
  afq_ctx* c = new (std::nothrow) afq_ctx();
  if (!c) { afq_set_error("out of host memory"); return -1; }
  c->d = *dims;
  if (c->d.n_batch < 1) c->d.n_batch = 1;
  c->h = *ham;
  c->nw_chunk = nwc;
  c->e_chunks = ec;
  c->e_gchunk = eg;
  c->welem = we;
  dev.h0 = ham->h0;
  dev.h0_prop_re = ham->h0_prop_re;
  dev.h0_prop_im = ham->h0_prop_im;
  dev.trial[0] = ham->trial_up;
  dev.trial[1] = uhf ? ham->trial_dn : ham->trial_up;
  dev.exp_h1[0] = ham->exp_h1_up;
  dev.exp_h1[1] = unres ? ham->exp_h1_dn : ham->exp_h1_up;
  dev.rot_chol[0] = ham->rot_chol_up;
  dev.rot_chol[1] = uhf ? ham->rot_chol_dn : ham->rot_chol_up;
  dev.rot_h1[0] = ham->rot_h1_up;
  dev.rot_h1[1] = uhf ? ham->rot_h1_dn : ham->rot_h1_up;
  dev.mf = reinterpret_cast<const double2*>(ham->mf_shifts);
  c->dev = dev;
  char* ws = static_cast<char*>(workspace);
  c->ws = ws;
  c->ws_bytes = workspace_bytes;
  c->green = reinterpret_cast<double2*>(ws + sz.green);
  c->fb = reinterpret_cast<double2*>(ws + sz.fb);
  c->xt = reinterpret_cast<double2*>(ws + sz.xt);
  c->shift = reinterpret_cast<double2*>(ws + sz.shift);
  c->fbt = reinterpret_cast<double2*>(ws + sz.fbt);
  c->vhs = reinterpret_cast<double2*>(ws + sz.vhs);
  c->ovl_new = reinterpret_cast<double2*>(ws + sz.ovl_new);
  c->ene = reinterpret_cast<double2*>(ws + sz.ene);
  c->epart = reinterpret_cast<double2*>(ws + sz.epart);
  c->rccat = reinterpret_cast<double*>(ws + sz.rccat);
  c->wcopy = ws + sz.wcopy;
  c->sr_idx = reinterpret_cast<int32_t*>(ws + sz.sr_idx);
  c->cum = reinterpret_cast<double*>(ws + sz.cum);
  c->free_scr = reinterpret_cast<double2*>(ws + sz.free_scr);
  cudaStream_t st = S(stream);
  if (uhf) {
    // rccat[g] = [rot_chol_up[g] | rot_chol_dn[g]]
    const size_t a = (size_t)dims->n_up * dims->norb, b = (size_t)dims->n_dn * dims->norb;
    cudaError_t e = cudaMemcpy2DAsync(c->rccat, dev.ktot * sizeof(double), ham->rot_chol_up, a * sizeof(double),
                                      a * sizeof(double), dims->nchol, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess)
      e = cudaMemcpy2DAsync(c->rccat + a, dev.ktot * sizeof(double), ham->rot_chol_dn, b * sizeof(double),
                            b * sizeof(double), dims->nchol, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) {
      afq_set_error("rot_chol concat: %s", cudaGetErrorString(e));
      delete c;
      return (int)e;
    }
  }
  if (dims->precision == AFQ_PREC_FP64) dig_dims(c->dev, nwc, &c->dg);
  if (dev.digits) {
    auto at = [&](afq::DigOp& o, const size_t (&off)[2]) {
      o.d = reinterpret_cast<unsigned char*>(ws + off[0]);
      o.e = reinterpret_cast<int*>(ws + off[1]);
    };
    at(c->dg.rc, sz.dg_rc);
    at(c->dg.ga, sz.dg_ga);
    c->dg.status = reinterpret_cast<int*>(ws + sz.dg_status);
    c->dg.part = reinterpret_cast<double2*>(ws + sz.dg_part);
    c->dg.z = reinterpret_cast<double2*>(ws + sz.dg_z);
    c->dg.walk.status = c->dg.status;
    int e = zero(ws + sz.dg, sz.dg_end - sz.dg, st);  // padding stays zero
    for (int s = 0; s < dev.nspin_g && c->dg.has_u && !e; ++s) {
      // U[(i,q),(k,p)] = (X X^T)[(i,p),(k,q)], X = rot_chol^T; u_strip of the i at a time
      at(c->dg.u[s], sz.dg_u[s]);
      at(c->dg.ua[s], sz.dg_ua);
      at(c->dg.ub[s], sz.dg_ub);
      const int on = c->dg.u[s].rows;
      double* tmp = reinterpret_cast<double*>(ws + sz.dg_utmp);
      e = afq::dig_slice_real_cols(c->dg.ub[s], dev.rot_chol[s], on, st);
      for (int r0 = 0; r0 < on && !e; r0 += c->dg.ua[s].rows) {
        afq::DigOp a = c->dg.ua[s];
        a.rows = std::min(a.rows, on - r0);
        e = afq::dig_slice_real_cols(a, dev.rot_chol[s] + r0, on, st);
        if (!e) e = afq::dig_gemm_r(afq::K_PREP, a, c->dg.ub[s], a.rows, on, tmp, on, dev.norb, c->dg.status, st);
        if (!e) e = afq::dig_slice_real_rows(c->dg.u[s], tmp, on, st, a.rows, r0);
      }
    }
    if (!e) e = afq::dig_slice_real_rows(c->dg.rc, rc_all(c), dev.ktot, st);
    if (!dev.measure) {
      at(c->dg.chol, sz.dg_chol);
      at(c->dg.xa, sz.dg_xa);
      if (!e) e = afq::dig_slice_real_cols(c->dg.chol, ham->chol, (long)dims->norb * dims->norb, st);
    }
    if (c->dg.use_walk) {
      c->dg.walk.vd = reinterpret_cast<unsigned char*>(ws + sz.dg_v[0]);
      c->dg.walk.ve = reinterpret_cast<int*>(ws + sz.dg_v[1]);
      c->dg.walk.xd = reinterpret_cast<unsigned char*>(ws + sz.dg_x[0]);
      c->dg.walk.xe = reinterpret_cast<int*>(ws + sz.dg_x[1]);
      c->dg.walk_t = reinterpret_cast<double2*>(ws + sz.dg_wt);
      c->dg.walk_acc = reinterpret_cast<double2*>(ws + sz.dg_wa);
      for (int s = 0; s < c->dg.walk.n_e(dev.nslab); ++s) at(c->dg.walk.e[s], sz.dg_e[s]);
      if (!e) e = afq::dig_walk_slice_e(c->dg.walk, c->dg.walk.e, dev.exp_h1, dev.nslab, false, st);
    }
    if (!e) e = zero(ws + sz.dgw, sz.dgw_end - sz.dgw, st);  // the walkers' padding, after the set-up in its place
    if (e) {
      delete c;
      return e;
    }
  }
  if (dims->precision == AFQ_PREC_MIXED) {
    int e = afq::tc_init(&c->tc, c->dev, *ham, c->rccat, nwc, dims->mixed_config, ws + sz.tc, st);
    if (e) {
      delete c;
      return e;
    }
  }
  *out = c;
  return 0;
}

void afq_ctx_destroy(afq_ctx* ctx) { delete ctx; }

int afq_calc_overlap(afq_ctx* ctx, const void* walkers_up, const void* walkers_dn, double* overlaps,
                     void* stream) {
  if (!ctx || !overlaps) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_walkers(ctx, walkers_up, walkers_dn));
  return green(ctx, walkers_up, walkers_dn, nullptr, reinterpret_cast<double2*>(overlaps), false, S(stream));
}

int afq_calc_force_bias(afq_ctx* ctx, const void* walkers_up, const void* walkers_dn,
                        double* force_bias, void* stream) {
  if (!ctx || !force_bias) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_walkers(ctx, walkers_up, walkers_dn));
  CHECK(green(ctx, walkers_up, walkers_dn, ctx->green, nullptr, true, S(stream)));
  CHECK(force_bias_from_green(ctx, reinterpret_cast<double2*>(force_bias), S(stream)));
  if (!ctx->dev.digits) return 0;
  return afq::launch_poison((long)ctx->dev.nw * ctx->dev.nchol, reinterpret_cast<double2*>(force_bias),
                            ctx->dg.status, S(stream));
}

int afq_calc_energy(afq_ctx* ctx, const void* walkers_up, const void* walkers_dn, double* energies,
                    void* stream) {
  if (!ctx || !energies) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_walkers(ctx, walkers_up, walkers_dn));
  CHECK(green(ctx, walkers_up, walkers_dn, ctx->green, nullptr, true, S(stream)));
  return energy_from_green(ctx, reinterpret_cast<double2*>(energies), S(stream));
}

int afq_propagate(afq_ctx* ctx, afq_walker_state* state, const double* fields, void* stream) {
  if (!ctx || !fields) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_state(ctx, state));
  return propagate_impl(ctx, state, fields, S(stream));
}

int afq_orthonormalize_walkers(afq_ctx* ctx, afq_walker_state* state, void* stream) {
  if (!ctx) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_state(ctx, state));
  return qr_impl(ctx, state, S(stream));
}

int afq_stochastic_reconfiguration(afq_ctx* ctx, afq_walker_state* state, const double* zeta,
                                   int32_t* indices, void* stream) {
  if (!ctx || !zeta) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_state(ctx, state));
  return sr_impl(ctx, state, zeta, indices, S(stream));
}

int afq_propagate_phaseless(afq_ctx* ctx, afq_walker_state* state, const double* fields,
                            const double* zetas, int32_t n_prop_steps, int32_t n_ene_blocks,
                            int32_t n_sr_blocks, double* block_energy, double* block_weight,
                            double* energy, void* stream) {
  if (!ctx || !fields || !zetas || !block_energy || !block_weight || !energy) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (n_prop_steps < 1 || n_ene_blocks < 1 || n_sr_blocks < 1) {
    afq_set_error("block counts must be >= 1");
    return -1;
  }
  CHECK(check_state(ctx, state));
  cudaStream_t st = S(stream);
  const afq_ctx_dev& d = ctx->dev;
  double2* ovl = reinterpret_cast<double2*>(state->overlaps);
  ctx->gstate = 0;
  CHECK(green(ctx, state->walkers_up, state->walkers_dn, nullptr, ovl, false, st, true));
  CHECK(afq::launch_phaseless_begin(state->scalars, st));
  const size_t step_elems = (size_t)d.nw * d.nchol;
  int blk = 0;
  for (int sr = 0; sr < n_sr_blocks; ++sr) {
    for (int eb = 0; eb < n_ene_blocks; ++eb, ++blk) {
      for (int p = 0; p < n_prop_steps; ++p) {
        const double* f = fields + ((size_t)blk * n_prop_steps + p) * step_elems;
        CHECK(propagate_impl(ctx, state, f, st, true, p + 1 < n_prop_steps));
      }
      ctx->gstate = 0;
      CHECK(qr_impl(ctx, state, st));
      CHECK(green(ctx, state->walkers_up, state->walkers_dn, ctx->green, ovl, true, st, true));
      CHECK(energy_from_green(ctx, ctx->ene, st));
      CHECK(afq::launch_block_stats(d, ctx->ene, state->weights, state->scalars, block_energy + blk,
                                    block_weight + blk, st, status_word(ctx)));
    }
    ctx->gstate = 0;
    CHECK(sr_impl(ctx, state, zetas + sr, nullptr, st));
    CHECK(green(ctx, state->walkers_up, state->walkers_dn, nullptr, ovl, false, st, sr + 1 < n_sr_blocks));
  }
  ctx->gstate = 0;
  return afq::launch_phaseless_end(blk, (double)n_sr_blocks * n_ene_blocks * d.nw, block_energy,
                                   block_weight, state->scalars, energy, st);
}

size_t afq_tangent_workspace_size(const afq_dims* dims) {
  afq_ctx_dev c;
  int nwc, ec, eg;
  size_t we;
  if (derive(dims, &c, &nwc, &ec, &eg, &we)) return 0;
  Layout L;
  return tangent_sizes(c, nwc, ec, &L).total;
}

int afq_propagate_phaseless_jvp(afq_ctx* ctx, afq_walker_state* state, const double* dexp_h1_up,
                                const double* dexp_h1_dn, const double* drot_h1_up, const double* drot_h1_dn,
                                void* tangent_workspace, size_t tangent_workspace_bytes, const double* fields,
                                const double* zetas, int32_t n_prop_steps, int32_t n_ene_blocks,
                                int32_t n_sr_blocks, int32_t flags, double* block_energy, double* block_weight,
                                double* dblock_energy, double* dblock_weight, double* energy, double* denergy,
                                void* stream) {
  afq_jvp_inputs in;
  memset(&in, 0, sizeof(in));
  in.dexp_h1_up = dexp_h1_up;
  in.dexp_h1_dn = dexp_h1_dn;
  in.drot_h1_up = drot_h1_up;
  in.drot_h1_dn = drot_h1_dn;
  return afq_propagate_phaseless_jvp_ex(ctx, state, &in, tangent_workspace, tangent_workspace_bytes, fields, zetas,
                                        n_prop_steps, n_ene_blocks, n_sr_blocks, flags, block_energy, block_weight,
                                        dblock_energy, dblock_weight, energy, denergy, stream);
}

int afq_propagate_phaseless_jvp_ex(afq_ctx* ctx, afq_walker_state* state, const afq_jvp_inputs* in,
                                   void* tangent_workspace, size_t tangent_workspace_bytes, const double* fields,
                                   const double* zetas, int32_t n_prop_steps, int32_t n_ene_blocks,
                                   int32_t n_sr_blocks, int32_t flags, double* block_energy, double* block_weight,
                                   double* dblock_energy, double* dblock_weight, double* energy, double* denergy,
                                   void* stream) {
  if (!in) { afq_set_error("NULL argument"); return -1; }
  const double *dexp_h1_up = in->dexp_h1_up, *dexp_h1_dn = in->dexp_h1_dn, *drot_h1_up = in->drot_h1_up,
               *drot_h1_dn = in->drot_h1_dn;
  const bool do_sr = !(flags & AFQ_JVP_NO_SR);
  if (!ctx || !fields || (do_sr && !zetas) || !block_energy || !block_weight || !dblock_energy || !dblock_weight || !energy ||
      !denergy || !dexp_h1_up || !drot_h1_up) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (!is_fp64(ctx)) { afq_set_error("the derivative path needs an FP64 context"); return -1; }
  if (n_prop_steps < 1 || n_ene_blocks < 1 || n_sr_blocks < 1 || (!do_sr && n_sr_blocks != 1)) {
    afq_set_error("block counts must be >= 1 (n_sr_blocks == 1 without SR)");
    return -1;
  }
  if (flags & ~AFQ_JVP_NO_SR) { afq_set_error("unknown flags 0x%x", (unsigned)flags); return -1; }
  CHECK(check_state(ctx, state));
  const afq_ctx_dev& d = ctx->dev;
  if (d.nslab == 2 && !dexp_h1_dn) { afq_set_error("unrestricted walkers need dexp_h1_dn"); return -1; }
  if (d.nspin_g == 2 && !drot_h1_dn) { afq_set_error("the UHF trial needs drot_h1_dn"); return -1; }
  const bool rot = in->dtrial_up || in->drot_chol_up;
  if (rot && (!in->dtrial_up || !in->drot_chol_up ||
              (d.nspin_g == 2 && (!in->dtrial_dn || !in->drot_chol_dn)))) {
    afq_set_error("orbital rotation needs dtrial and drot_chol for every spin of the trial");
    return -1;
  }
  Layout L;
  const TSizes ts = tangent_sizes(d, ctx->nw_chunk, ctx->e_chunks, &L);
  if (!tangent_workspace || tangent_workspace_bytes < ts.total) {
    afq_set_error("tangent workspace too small: need %zu bytes, got %zu", ts.total, tangent_workspace_bytes);
    return -1;
  }
  if (reinterpret_cast<uintptr_t>(tangent_workspace) & 255) {
    afq_set_error("tangent workspace must be 256-byte aligned");
    return -1;
  }
  char* tw = static_cast<char*>(tangent_workspace);
  afq::TangentBufs t;
  for (int k = 0; k < 2; ++k) {
    t.dw[k] = reinterpret_cast<double2*>(tw + ts.dw[k]);
    t.wold[k] = reinterpret_cast<double2*>(tw + ts.wold[k]);
  }
  t.dgreen = reinterpret_cast<double2*>(tw + ts.dgreen);
  t.dfb = reinterpret_cast<double2*>(tw + ts.dfb);
  t.dxt = reinterpret_cast<double2*>(tw + ts.dxt);
  t.dshift = reinterpret_cast<double2*>(tw + ts.dshift);
  t.dfbt = reinterpret_cast<double2*>(tw + ts.dfbt);
  t.dvhs = reinterpret_cast<double2*>(tw + ts.dvhs);
  t.dlo = reinterpret_cast<double2*>(tw + ts.dlo);
  t.dlo_new = reinterpret_cast<double2*>(tw + ts.dlo_new);
  t.dweights = reinterpret_cast<double*>(tw + ts.dweights);
  t.dscalars = reinterpret_cast<double*>(tw + ts.dscalars);
  t.dene = reinterpret_cast<double2*>(tw + ts.dene);
  t.dpart = reinterpret_cast<double2*>(tw + ts.dpart);
  t.dsum = reinterpret_cast<double*>(tw + ts.dsum);
  t.dbe = dblock_energy;
  t.dbw = dblock_weight;
  t.dexp[0] = dexp_h1_up;
  t.dexp[1] = d.nslab == 2 ? dexp_h1_dn : dexp_h1_up;
  t.drot[0] = drot_h1_up;
  t.drot[1] = d.nspin_g == 2 ? drot_h1_dn : drot_h1_up;
  // the RHF trial serves both walker slabs: one trial tangent for both
  t.dtrial[0] = rot ? in->dtrial_up : nullptr;
  t.dtrial[1] = rot ? (d.nspin_g == 2 ? in->dtrial_dn : in->dtrial_up) : nullptr;
  t.drc[0] = rot ? in->drot_chol_up : nullptr;
  t.drc[1] = rot && d.nspin_g == 2 ? in->drot_chol_dn : nullptr;
  t.drccat = nullptr;
  cudaStream_t st = S(stream);
  // walker, weight, overlap and shift tangents start at zero (driver.py:190-200)
  {
    cudaError_t e = cudaMemsetAsync(tangent_workspace, 0, ts.total, st);
    if (e != cudaSuccess) { afq_set_error("tangent workspace clear: %s", cudaGetErrorString(e)); return (int)e; }
  }
  if (rot && d.nspin_g == 2) {  // [drot_chol_up[g] | drot_chol_dn[g]], the layout of rccat
    double* cat = reinterpret_cast<double*>(tw + ts.drccat);
    const size_t a = (size_t)d.gocc[0] * d.norb, b = (size_t)d.gocc[1] * d.norb;
    cudaError_t e = cudaMemcpy2DAsync(cat, d.ktot * sizeof(double), in->drot_chol_up, a * sizeof(double),
                                      a * sizeof(double), d.nchol, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess)
      e = cudaMemcpy2DAsync(cat + a, d.ktot * sizeof(double), in->drot_chol_dn, b * sizeof(double),
                            b * sizeof(double), d.nchol, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) { afq_set_error("drot_chol concat: %s", cudaGetErrorString(e)); return (int)e; }
    t.drccat = cat;
  } else if (rot) {
    t.drccat = in->drot_chol_up;
  }
  afq::DigOp drc = ctx->dg.rc;
  drc.d = reinterpret_cast<unsigned char*>(tw + ts.drc_d);
  drc.e = reinterpret_cast<int*>(tw + ts.drc_e);
  if (t.drccat && d.digits) CHECK(afq::dig_slice_real_rows(drc, t.drccat, d.ktot, st));
  JvpWalk jw{ctx->dg.walk, nullptr, nullptr};
  if (ctx->dg.walk_jvp) {  // (the workspace was cleared above: padding is zero)
    jw.w.vd = reinterpret_cast<unsigned char*>(tw + ts.v[0]);
    jw.w.ve = reinterpret_cast<int*>(tw + ts.v[1]);
    jw.w.xd = reinterpret_cast<unsigned char*>(tw + ts.x[0]);
    jw.w.xe = reinterpret_cast<int*>(tw + ts.x[1]);
    jw.t = reinterpret_cast<double2*>(tw + ts.wt);
    jw.a = reinterpret_cast<double2*>(tw + ts.wa);
    for (int k = 0; k < jw.w.n_e(d.nslab); ++k) {
      jw.w.e[k].d = reinterpret_cast<unsigned char*>(tw + ts.de[k][0]);
      jw.w.e[k].e = reinterpret_cast<int*>(tw + ts.de[k][1]);
    }
    CHECK(afq::dig_walk_slice_e(jw.w, jw.w.e, t.dexp, d.nslab, false, st));
  }
  double2* ovl = reinterpret_cast<double2*>(state->overlaps);
  const size_t welems[2] = {(size_t)d.nw * d.norb * d.kslab[0], (size_t)d.nw * d.norb * d.kslab[1]};
  void* wslab[2] = {state->walkers_up, state->walkers_dn};
  ctx->gstate = 0;
  CHECK(afq::t_launch_green(d, t, state->walkers_up, state->walkers_dn, ctx->green, t.dgreen, ovl, t.dlo, st));
  CHECK(afq::launch_phaseless_begin(state->scalars, st));
  const size_t step_elems = (size_t)d.nw * d.nchol;
  int blk = 0;
  for (int sr = 0; sr < n_sr_blocks; ++sr) {
    for (int eb = 0; eb < n_ene_blocks; ++eb, ++blk) {
      for (int p = 0; p < n_prop_steps; ++p) {
        const double* f = fields + ((size_t)blk * n_prop_steps + p) * step_elems;
        CHECK(propagate_jvp(ctx, state, t, drc, jw, f, st, p + 1 < n_prop_steps));
      }
      for (int k = 0; k < d.nslab; ++k)
        CHECK(copy_d2d(t.wold[k], wslab[k], welems[k] * sizeof(double2), st, "walker copy before QR"));
      CHECK(qr_impl(ctx, state, st));
      CHECK(afq::t_launch_qr(d, t, state->walkers_up, state->walkers_dn, st));
      CHECK(afq::t_launch_green(d, t, state->walkers_up, state->walkers_dn, ctx->green, t.dgreen, ovl, t.dlo, st));
      CHECK(energy_from_green(ctx, ctx->ene, st));
      if (ctx->dg.has_u && !rot) {  // ctx->fb and dg.z are those of the energy just evaluated
        CHECK(fb_gemm(ctx, t.dgreen, rc_all(ctx), ctx->dg.rc, t.dfb, st, true));
        CHECK(afq::dig_launch_energy_tangent(d, ctx->green, t.dgreen, ctx->dg.z, ctx->fb, t.dfb, t.drot[0], t.drot[1],
                                             t.dene, st));
      } else {
        CHECK(afq::t_launch_energy(d, t, ctx->e_chunks, ctx->e_gchunk, ctx->green, st));
      }
      CHECK(afq::launch_block_stats(d, ctx->ene, state->weights, state->scalars, block_energy + blk,
                                    block_weight + blk, st, status_word(ctx)));
      CHECK(afq::t_launch_block_stats(d, t, ctx->ene, state->weights, state->scalars, block_energy + blk,
                                      dblock_energy + blk, dblock_weight + blk, st));
    }
    if (!do_sr) continue;
    CHECK(afq::t_launch_sr_pre(d, t, st));
    CHECK(sr_impl(ctx, state, zetas + sr, nullptr, st));
    CHECK(afq::t_launch_sr_post(d, t, ctx->sr_idx, st));
    const bool more = sr + 1 < n_sr_blocks;
    CHECK(afq::t_launch_green(d, t, state->walkers_up, state->walkers_dn, more ? ctx->green : nullptr,
                              more ? t.dgreen : nullptr, ovl, t.dlo, st));
  }
  CHECK(afq::launch_phaseless_end(blk, (double)n_sr_blocks * n_ene_blocks * d.nw, block_energy, block_weight,
                                  state->scalars, energy, st));
  return afq::t_launch_end(blk, block_energy, block_weight, t, nullptr, denergy, st);
}

size_t afq_vjp_workspace_size(const afq_dims* dims, int32_t n_prop_steps, int32_t n_ene_blocks,
                              int32_t n_sr_blocks) {
  afq_ctx_dev c;
  int nwc, ec, eg;
  size_t we;
  if (n_prop_steps < 1 || n_ene_blocks < 1 || n_sr_blocks < 1) return 0;
  if (derive(dims, &c, &nwc, &ec, &eg, &we)) return 0;
  Layout L;
  return adjoint_sizes(c, nwc, n_prop_steps, n_ene_blocks, n_sr_blocks, &L).total;
}

int afq_propagate_phaseless_vjp(afq_ctx* ctx, afq_walker_state* state, void* vjp_workspace,
                                size_t vjp_workspace_bytes, const double* fields, const double* zetas,
                                int32_t n_prop_steps, int32_t n_ene_blocks, int32_t n_sr_blocks,
                                int32_t flags, double* block_energy, double* block_weight,
                                double* energy, double* gexp_h1_up, double* gexp_h1_dn,
                                double* grot_h1_up, double* grot_h1_dn, void* stream) {
  afq_vjp_outputs out;
  memset(&out, 0, sizeof(out));
  out.gexp_h1_up = gexp_h1_up;
  out.gexp_h1_dn = gexp_h1_dn;
  out.grot_h1_up = grot_h1_up;
  out.grot_h1_dn = grot_h1_dn;
  return afq_propagate_phaseless_vjp_ex(ctx, state, vjp_workspace, vjp_workspace_bytes, fields, zetas, n_prop_steps,
                                        n_ene_blocks, n_sr_blocks, flags, block_energy, block_weight, energy, &out,
                                        stream);
}

int afq_propagate_phaseless_vjp_ex(afq_ctx* ctx, afq_walker_state* state, void* vjp_workspace,
                                   size_t vjp_workspace_bytes, const double* fields, const double* zetas,
                                   int32_t n_prop_steps, int32_t n_ene_blocks, int32_t n_sr_blocks, int32_t flags,
                                   double* block_energy, double* block_weight, double* energy,
                                   const afq_vjp_outputs* out, void* stream) {
  if (!out) { afq_set_error("NULL argument"); return -1; }
  double *gexp_h1_up = out->gexp_h1_up, *gexp_h1_dn = out->gexp_h1_dn, *grot_h1_up = out->grot_h1_up,
         *grot_h1_dn = out->grot_h1_dn;
  const bool do_sr = !(flags & AFQ_JVP_NO_SR);
  if (!ctx || !fields || (do_sr && !zetas) || !block_energy || !block_weight || !energy || !gexp_h1_up ||
      !grot_h1_up) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (!is_fp64(ctx)) { afq_set_error("the derivative path needs an FP64 context"); return -1; }
  if (n_prop_steps < 1 || n_ene_blocks < 1 || n_sr_blocks < 1 || (!do_sr && n_sr_blocks != 1)) {
    afq_set_error("block counts must be >= 1 (n_sr_blocks == 1 without SR)");
    return -1;
  }
  if (flags & ~AFQ_JVP_NO_SR) { afq_set_error("unknown flags 0x%x", (unsigned)flags); return -1; }
  CHECK(check_state(ctx, state));
  const afq_ctx_dev& d = ctx->dev;
  if (d.nslab == 2 && !gexp_h1_dn) { afq_set_error("unrestricted walkers need gexp_h1_dn"); return -1; }
  if (d.nspin_g == 2 && !grot_h1_dn) { afq_set_error("the UHF trial needs grot_h1_dn"); return -1; }
  const bool rot = out->gtrial_up || out->grot_chol;
  if (rot && (!out->gtrial_up || !out->grot_chol || (d.nspin_g == 2 && !out->gtrial_dn))) {
    afq_set_error("orbital-rotation gradients need gtrial for every spin of the trial and grot_chol");
    return -1;
  }
  const int P = n_prop_steps, NE = n_ene_blocks;
  Layout L;
  const AdjSizes as = adjoint_sizes(d, ctx->nw_chunk, P, NE, n_sr_blocks, &L);
  if (!vjp_workspace || vjp_workspace_bytes < as.total) {
    afq_set_error("vjp workspace too small: need %zu bytes, got %zu", as.total, vjp_workspace_bytes);
    return -1;
  }
  if (reinterpret_cast<uintptr_t>(vjp_workspace) & 255) {
    afq_set_error("vjp workspace must be 256-byte aligned");
    return -1;
  }
  char* base = static_cast<char*>(vjp_workspace);
  const Tape tp{base, as, &d};
  afq::AdjointBufs a;
  const size_t e0 = (size_t)d.nw * d.norb * d.kslab[0];
  a.wb[0] = reinterpret_cast<double2*>(base + as.wb);
  a.wb[1] = a.wb[0] + e0;
  a.wb2[0] = reinterpret_cast<double2*>(base + as.wb2);
  a.wb2[1] = a.wb2[0] + e0;
  a.wbar = reinterpret_cast<double*>(base + as.wbar);
  a.lbar = reinterpret_cast<double2*>(base + as.lbar);
  a.lbar2 = reinterpret_cast<double2*>(base + as.lbar2);
  a.gpend = reinterpret_cast<double2*>(base + as.gpend);
  a.gene = reinterpret_cast<double2*>(base + as.gene);
  a.fbb = reinterpret_cast<double2*>(base + as.fbb);
  a.xtb = reinterpret_cast<double2*>(base + as.xtb);
  a.shb = reinterpret_cast<double2*>(base + as.shb);
  a.fbtb = reinterpret_cast<double2*>(base + as.fbtb);
  a.vbar = reinterpret_cast<double2*>(base + as.vbar);
  a.tay = reinterpret_cast<double2*>(base + as.tay);
  a.exp_part = reinterpret_cast<double*>(base + as.exp_part);
  a.ebar = reinterpret_cast<double*>(base + as.ebar);
  a.scal = reinterpret_cast<double*>(base + as.scal);
  a.beb = reinterpret_cast<double*>(base + as.beb);
  a.bwb = reinterpret_cast<double*>(base + as.bwb);
  a.gexp[0] = gexp_h1_up;
  a.gexp[1] = d.nslab == 2 ? gexp_h1_dn : nullptr;
  a.grot[0] = grot_h1_up;
  a.grot[1] = d.nspin_g == 2 ? grot_h1_dn : nullptr;
  a.gtrial[0] = rot ? out->gtrial_up : nullptr;
  a.gtrial[1] = rot && d.nspin_g == 2 ? out->gtrial_dn : nullptr;
  a.grc = rot ? out->grot_chol : nullptr;
  double* const* gt = rot ? a.gtrial : nullptr;
  const bool cg = out->gchol != nullptr;
  if (cg && (!out->gmf_shifts || !out->gh0_prop)) {
    afq_set_error("Cholesky-vector gradients need gchol, gmf_shifts and gh0_prop");
    return -1;
  }
  a.gchol = cg ? out->gchol : nullptr;
  a.gmf = cg ? reinterpret_cast<double2*>(out->gmf_shifts) : nullptr;
  cudaStream_t st = S(stream);
  double2* ovl = reinterpret_cast<double2*>(state->overlaps);
  const size_t step_elems = (size_t)d.nw * d.nchol;

  // forward sweep: afq_propagate_phaseless's FP64 path, recording the state
  ctx->gstate = 0;
  CHECK(green(ctx, state->walkers_up, state->walkers_dn, nullptr, ovl, false, st, true));
  CHECK(afq::launch_phaseless_begin(state->scalars, st));
  int blk = 0;
  for (int sr = 0; sr < n_sr_blocks; ++sr) {
    for (int eb = 0; eb < NE; ++eb, ++blk) {
      for (int p = 0; p < P; ++p) {
        const int step = blk * P + p;
        CHECK(snapshot(tp, blk * (P + 2) + p, state, st));
        CHECK(propagate_impl(ctx, state, fields + (size_t)step * step_elems, st, true, p + 1 < P));
        CHECK(copy_d2d(tp.xt(step), ctx->xt, step_elems * sizeof(double2), st, "shifted-field record"));
        CHECK(copy_d2d(tp.sh(step), ctx->shift, d.nw * sizeof(double2), st, "shift record"));
        CHECK(copy_d2d(tp.fbt(step), ctx->fbt, d.nw * sizeof(double2), st, "fbt record"));
      }
      CHECK(snapshot(tp, blk * (P + 2) + P, state, st));
      ctx->gstate = 0;
      CHECK(qr_impl(ctx, state, st));
      CHECK(green(ctx, state->walkers_up, state->walkers_dn, ctx->green, ovl, true, st, true));
      CHECK(snapshot(tp, blk * (P + 2) + P + 1, state, st));
      CHECK(energy_from_green(ctx, ctx->ene, st));
      CHECK(copy_d2d(tp.ene(blk), ctx->ene, d.nw * sizeof(double2), st, "local-energy record"));
      CHECK(afq::launch_block_stats(d, ctx->ene, state->weights, state->scalars, block_energy + blk,
                                    block_weight + blk, st, status_word(ctx)));
    }
    if (!do_sr) continue;
    ctx->gstate = 0;
    CHECK(sr_impl(ctx, state, zetas + sr, tp.idx(sr), st));
    CHECK(green(ctx, state->walkers_up, state->walkers_dn, nullptr, ovl, false, st, sr + 1 < n_sr_blocks));
  }
  ctx->gstate = 0;
  CHECK(afq::launch_phaseless_end(blk, (double)n_sr_blocks * NE * d.nw, block_energy, block_weight,
                                  state->scalars, energy, st));

  // backward sweep, from the sampler total to the start of the first block
  CHECK(zero(base + as.wb, as.wslab * sizeof(double2), st));
  CHECK(zero(a.wbar, d.nw * sizeof(double), st));
  CHECK(zero(a.lbar, d.nw * sizeof(double2), st));
  CHECK(zero(a.scal, 8 * sizeof(double), st));
  CHECK(zero(gexp_h1_up, (size_t)d.norb * d.norb * sizeof(double), st));
  if (d.nslab == 2) CHECK(zero(gexp_h1_dn, (size_t)d.norb * d.norb * sizeof(double), st));
  CHECK(zero(grot_h1_up, (size_t)d.gocc[0] * d.norb * sizeof(double), st));
  if (d.nspin_g == 2) CHECK(zero(grot_h1_dn, (size_t)d.gocc[1] * d.norb * sizeof(double), st));
  if (rot) {
    for (int b = 0; b < d.nspin_g; ++b)
      CHECK(zero(a.gtrial[b], (size_t)d.norb * d.gocc[b] * sizeof(double), st));
    CHECK(zero(a.grc, (size_t)d.nchol * d.ktot * sizeof(double), st));
  }
  if (cg) {
    CHECK(zero(a.gchol, (size_t)d.nchol * d.norb * d.norb * sizeof(double), st));
    CHECK(zero(a.gmf, (size_t)d.nchol * sizeof(double2), st));
  }
  CHECK(afq::a_launch_end(blk, block_energy, block_weight, a, st));
  const int nwc = ctx->nw_chunk, nb = d.nw / nwc;
  const long nn = (long)d.norb * d.norb;
  const double* brc = rc_all(ctx);
  AdjOps ao = adj_ops(d, nwc);
  ao.cn.d = reinterpret_cast<unsigned char*>(base + as.cn_d);
  ao.cn.e = reinterpret_cast<int*>(base + as.cn_e);
  ao.rt.d = reinterpret_cast<unsigned char*>(base + as.rt_d);
  ao.rt.e = reinterpret_cast<int*>(base + as.rt_e);
  ao.va.d = reinterpret_cast<unsigned char*>(base + as.va_d);
  ao.va.e = reinterpret_cast<int*>(base + as.va_e);
  if (d.digits) {
    CHECK(zero(base + as.dg, as.dg_end - as.dg, st));
    CHECK(afq::dig_slice_real_rows(ao.cn, ctx->h.chol, nn, st));
    CHECK(afq::dig_slice_real_cols(ao.rt, brc, d.ktot, st));
  }
  const bool walk = adj_walk(d, ctx->dg);
  afq::DigOp et[2] = {ctx->dg.walk.e[0], ctx->dg.walk.e[1]};
  afq::DigVbar vb;
  if (walk) {
    afq::dig_walk_vbar_dims(ctx->dg.walk, d.n_exp_terms - 1, &vb);
    vb.ad = reinterpret_cast<unsigned char*>(base + as.vb_ad);
    vb.ae = reinterpret_cast<int*>(base + as.vb_ae);
    vb.bd = reinterpret_cast<unsigned char*>(base + as.vb_bd);
    vb.be = reinterpret_cast<int*>(base + as.vb_be);
    for (int k = 0; k < ctx->dg.walk.n_e(d.nslab); ++k) {
      et[k].d = reinterpret_cast<unsigned char*>(base + as.et[k][0]);
      et[k].e = reinterpret_cast<int*>(base + as.et[k][1]);
    }
    CHECK(afq::dig_walk_slice_e(ctx->dg.walk, et, d.exp_h1, d.nslab, true, st));
  }
  const double alpha = d.energy_mode == 0 ? 2.0 : 1.0;
  bool gp = false;  // a.gpend holds the pending G cotangent of the current point
  for (int b = blk - 1; b >= 0; --b) {
    if (do_sr && b + 1 < blk && b % NE == NE - 1) {
      // the SR between blocks b and b + 1: finish the cotangent of its output walkers,
      // then send it back through the gather
      const int s0 = (b + 1) * (P + 2);
      CHECK(afq::a_launch_green(d, tp.w(s0, 0), tp.w(s0, 1), gp ? a.gpend : nullptr, nullptr, a.lbar, a.wb[0],
                                a.wb[1], st, gt));
      CHECK(afq::a_launch_sr(d, a, tp.idx(b / NE), st));
      swap_slabs(a.wb, a.wb2);
      CHECK(zero(a.lbar, d.nw * sizeof(double2), st));
      gp = false;
    }
    const int sq_i = b * (P + 2) + P + 1, sw_i = b * (P + 2) + P;
    CHECK(afq::a_launch_block_stats(d, a, b, tp.ene(b), tp.wt(sq_i), tp.sc(sq_i), block_energy, st));
    CHECK(afq::launch_green<double>(d, tp.w(sq_i, 0), tp.w(sq_i, 1), ctx->green, nullptr, true, st));
    if (ctx->dg.has_u) {
      CHECK(energy_gemms(ctx, st));
      CHECK(afq::dig_slice_cplx_rows(ctx->dg.xa, ctx->fb, d.nchol, 1.0, st));
      CHECK(afq::dig_gemm_c(afq::K_ENERGY, ctx->dg.xa, ao.rt, d.nw, d.ktot, a.gene, d.ktot, 0, 0,
                            afq::DigPlan{1, ctx->dg.xa.kb()}, nullptr, ctx->dg.status, st));
      CHECK(afq::dig_launch_energy_adjoint(d, ctx->dg.z, a.ebar, a.gene, st));
      CHECK(afq::a_launch_rot(d, a, ctx->green, st));
    } else {
      CHECK(afq::a_launch_energy(d, a, ctx->green, st));
    }
    if (rot) CHECK(afq::a_launch_rc_energy(d, a, ctx->green, st));
    CHECK(afq::a_launch_green(d, tp.w(sq_i, 0), tp.w(sq_i, 1), a.gene, gp ? a.gpend : nullptr, a.lbar, a.wb[0],
                              a.wb[1], st, gt));
    CHECK(zero(a.lbar, d.nw * sizeof(double2), st));
    gp = false;
    CHECK(afq::a_launch_qr(d, tp.w(sw_i, 0), tp.w(sw_i, 1), tp.w(sq_i, 0), tp.w(sq_i, 1), a.wb[0], a.wb[1],
                           a.wb2[0], a.wb2[1], st));
    swap_slabs(a.wb, a.wb2);
    for (int p = P - 1; p >= 0; --p) {
      const int post = b * (P + 2) + p + 1, start = b * (P + 2) + p, step = b * P + p;
      CHECK(afq::a_launch_weights(d, a, tp.sh(step), tp.fbt(step), tp.ov(post), tp.ov(start), tp.wt(start),
                                  tp.wt(post), tp.sc(start), st));
      CHECK(afq::a_launch_green(d, tp.w(post, 0), tp.w(post, 1), gp ? a.gpend : nullptr, nullptr, a.lbar, a.wb[0],
                                a.wb[1], st, gt));
      for (int k = 0; k < nb; ++k) {
        const int w0 = k * nwc;
        CHECK(vhs_gemm(ctx, tp.xt(step) + (size_t)w0 * d.nchol, nwc, ctx->vhs, st));
        if (walk)
          CHECK(taylor_vjp(ctx, a, et, vb, w0, nwc, ctx->vhs, tp.w(start, 0), tp.w(start, 1), st));
        else
          CHECK(afq::a_launch_taylor(d, a, w0, nwc, ctx->vhs, tp.w(start, 0), tp.w(start, 1), st));
        if (cg) CHECK(afq::a_launch_chol_grad(d, a, nwc, tp.xt(step) + (size_t)w0 * d.nchol, st));
        double2* xtb = a.xtb + (size_t)w0 * d.nchol;
        if (d.digits) {
          CHECK(afq::dig_slice_cplx_rows(ao.va, a.vbar, nn, sqrt(d.dt), st));
          CHECK(afq::dig_gemm_c(afq::K_FB, ao.va, ao.cn, nwc, d.nchol, xtb, d.nchol, 3, 0, ao.xtb,
                                reinterpret_cast<double2*>(base + as.part), ctx->dg.status, st));
        } else {
          CHECK(afq::launch_gemm_cr(false, nwc, d.nchol, (int)nn, a.vbar, nn, ctx->h.chol, nn, xtb, d.nchol,
                                    c2(0.0, -sqrt(d.dt)), st));
        }
      }
      CHECK(afq::a_launch_field(d, a, tp.xt(step), st));
      if (rot) {  // fb = alpha rot_chol G(W_start): rot_chol-bar += alpha Re(fb-bar^H G)
        CHECK(afq::launch_green<double>(d, tp.w(start, 0), tp.w(start, 1), ctx->green, nullptr, true, st));
        CHECK(afq::a_launch_rc_fb(d, a, ctx->green, alpha, st));
      }
      if (d.digits) {
        CHECK(afq::dig_slice_cplx_rows(ctx->dg.xa, a.fbb, d.nchol, 1.0, st));
        CHECK(afq::dig_gemm_c(afq::K_VHS, ctx->dg.xa, ao.rt, d.nw, d.ktot, a.gpend, d.ktot, 0,
                              d.energy_mode == 0 ? 1 : 0, afq::DigPlan{1, ctx->dg.xa.kb()}, nullptr, ctx->dg.status, st));
      } else {
        CHECK(afq::launch_gemm_cr(true, d.nw, d.ktot, d.nchol, a.fbb, d.nchol, brc, d.ktot, a.gpend, d.ktot,
                                  c2(alpha, 0.0), st));
      }
      gp = true;
      swap_slabs(a.wb, a.wb2);
      double2* t = a.lbar;
      a.lbar = a.lbar2;
      a.lbar2 = t;
    }
  }
  // the first step's G and the block's initial overlap were evaluated with the trial too
  if (rot)
    CHECK(afq::a_launch_green(d, tp.w(0, 0), tp.w(0, 1), gp ? a.gpend : nullptr, nullptr, a.lbar, a.wb[0], a.wb[1], st,
                              gt));
  if (cg) {  // h0_prop-bar = (scal[1], 0): only its real part enters the weights
    CHECK(zero(out->gh0_prop, 2 * sizeof(double), st));
    CHECK(copy_d2d(out->gh0_prop, a.scal + 1, sizeof(double), st, "h0_prop cotangent"));
  }
  return afq::launch_fold_status(state->scalars, status_word(ctx), st);
}

int afq_propagate_free(afq_ctx* ctx, afq_walker_state* state, const double* fields, double ene0, double* norms,
                       double* normed_overlaps, void* stream) {
  if (!ctx || !fields || !norms || !normed_overlaps) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_state(ctx, state));
  CHECK(check_free(ctx));
  CHECK(free_step(ctx, state, fields, ene0, reinterpret_cast<double2*>(norms),
                  reinterpret_cast<double2*>(normed_overlaps), S(stream)));
  return afq::launch_fold_status(state->scalars, status_word(ctx), S(stream));
}

int afq_propagate_free_blocks(afq_ctx* ctx, afq_walker_state* state, const double* fields, int32_t n_prop_steps,
                              int32_t n_blocks, double ene0, double* norms, double* normed_overlaps,
                              double* block_energy, double* block_weight, void* stream) {
  if (!ctx || !fields || !norms || !normed_overlaps || !block_energy || !block_weight) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (n_prop_steps < 1 || n_blocks < 1) { afq_set_error("block counts must be >= 1"); return -1; }
  CHECK(check_state(ctx, state));
  CHECK(check_free(ctx));
  cudaStream_t st = S(stream);
  const afq_ctx_dev& d = ctx->dev;
  double2* ovl = reinterpret_cast<double2*>(state->overlaps);
  CHECK(green(ctx, state->walkers_up, state->walkers_dn, nullptr, ovl, false, st));
  const size_t step_elems = (size_t)d.nw * d.nchol;
  for (int b = 0; b < n_blocks; ++b) {
    for (int p = 0; p < n_prop_steps; ++p)
      CHECK(free_step(ctx, state, fields + ((size_t)b * n_prop_steps + p) * step_elems, ene0,
                      reinterpret_cast<double2*>(norms), reinterpret_cast<double2*>(normed_overlaps), st));
    CHECK(green(ctx, state->walkers_up, state->walkers_dn, ctx->green, nullptr, true, st));
    CHECK(energy_from_green(ctx, ctx->ene, st));
    CHECK(afq::launch_free_block_stats(d.nw, ctx->ene, ovl, reinterpret_cast<double2*>(block_energy) + b,
                                       reinterpret_cast<double2*>(block_weight) + b, st));
  }
  return afq::launch_fold_status(state->scalars, status_word(ctx), st);
}

int afq_field_block(afq_ctx* ctx, afq_walker_state* state, const double* fields, int32_t n_prop_steps,
                    double* local_energies, double* block_energy, double* block_weight, void* stream) {
  if (!ctx || !fields || !block_energy || !block_weight) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (n_prop_steps < 1) {
    afq_set_error("n_prop_steps must be >= 1");
    return -1;
  }
  CHECK(check_state(ctx, state));
  cudaStream_t st = S(stream);
  const afq_ctx_dev& d = ctx->dev;
  const size_t step_elems = (size_t)d.nw * d.nchol;
  for (int p = 0; p < n_prop_steps; ++p) CHECK(propagate_impl(ctx, state, fields + p * step_elems, st));
  CHECK(qr_impl(ctx, state, st));
  CHECK(green(ctx, state->walkers_up, state->walkers_dn, ctx->green, reinterpret_cast<double2*>(state->overlaps),
              true, st));
  CHECK(energy_from_green(ctx, ctx->ene, st));
  CHECK(afq::launch_block_stats(d, ctx->ene, state->weights, state->scalars, block_energy, block_weight, st,
                                status_word(ctx)));
  if (local_energies) CHECK(afq::launch_clamped_energies(d, ctx->ene, state->scalars, local_energies, st));
  return 0;
}

int afq_cs_outlier_removal(double* weights1, double* weights2, const double* local_energies1,
                           const double* local_energies2, int32_t n_walkers, double z_thresh, double* sums,
                           void* stream) {
  if (!weights1 || !weights2 || !local_energies1 || !local_energies2 || !sums || n_walkers < 1) {
    afq_set_error("afq_cs_outlier_removal: bad arguments");
    return -1;
  }
  return afq::launch_cs_outlier(weights1, weights2, local_energies1, local_energies2, n_walkers, z_thresh, sums,
                                S(stream));
}

int afq_block_end(afq_ctx* ctx, afq_walker_state* state, const double* energy, const double* zeta,
                  double* block_weight, void* stream) {
  if (!ctx || !energy || !zeta || !block_weight) { afq_set_error("NULL argument"); return -1; }
  CHECK(check_state(ctx, state));
  cudaStream_t st = S(stream);
  CHECK(afq::launch_driver_update(ctx->dev, state->weights, energy, state->scalars, block_weight, st));
  CHECK(qr_impl(ctx, state, st));
  return sr_impl(ctx, state, zeta, nullptr, st);
}

int afq_cpmc_init(int32_t norb, int32_t n_up, int32_t n_dn, int32_t n_walkers, const double* trial_up,
                  const double* trial_dn, double* walkers_up, double* walkers_dn, double* overlaps, double* greens,
                  void* stream) {
  if (!trial_up || !trial_dn || !walkers_up || !walkers_dn || !overlaps || !greens) {
    afq_set_error("NULL argument");
    return -1;
  }
  return afq::launch_cpmc(norb, n_up, n_dn, n_walkers, 1.0, 0.0, nullptr, nullptr, trial_up, trial_dn, walkers_up,
                          walkers_dn, nullptr, overlaps, greens, nullptr, nullptr, 0, S(stream));
}

int afq_cpmc_propagate(int32_t norb, int32_t n_up, int32_t n_dn, int32_t n_walkers, double dt, double u,
                       const double* exp_h1_up, const double* exp_h1_dn, const double* trial_up,
                       const double* trial_dn, double* walkers_up, double* walkers_dn, double* weights,
                       double* overlaps, double* greens, double* scalars, const double* gaussian, void* stream) {
  if (!exp_h1_up || !exp_h1_dn || !trial_up || !trial_dn || !walkers_up || !walkers_dn || !weights || !overlaps ||
      !greens || !scalars || !gaussian) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (!(dt > 0.0)) { afq_set_error("dt must be positive"); return -1; }
  return afq::launch_cpmc(norb, n_up, n_dn, n_walkers, dt, u, exp_h1_up, exp_h1_dn, trial_up, trial_dn, walkers_up,
                          walkers_dn, weights, overlaps, greens, scalars, gaussian, 1, S(stream));
}

int afq_cpmc_nn_propagate(int32_t norb, int32_t n_up, int32_t n_dn, int32_t n_walkers, double dt, double u,
                          double u_1, const int32_t* neighbors, int32_t n_pairs, const double* exp_h1_up,
                          const double* exp_h1_dn, const double* trial_up, const double* trial_dn,
                          double* walkers_up, double* walkers_dn, double* weights, double* overlaps,
                          double* greens, double* scalars, const double* uniforms, void* stream) {
  if (!exp_h1_up || !exp_h1_dn || !trial_up || !trial_dn || !walkers_up || !walkers_dn || !weights || !overlaps ||
      !greens || !scalars || !uniforms || (n_pairs > 0 && !neighbors) || n_pairs < 0) {
    afq_set_error("NULL argument or negative n_pairs");
    return -1;
  }
  if (!(dt > 0.0)) { afq_set_error("dt must be positive"); return -1; }
  return afq::launch_cpmc(norb, n_up, n_dn, n_walkers, dt, u, exp_h1_up, exp_h1_dn, trial_up, trial_dn, walkers_up,
                          walkers_dn, weights, overlaps, greens, scalars, nullptr, 3, S(stream), u_1, neighbors,
                          n_pairs, uniforms);
}

int afq_cpmc_continuous_propagate(int32_t norb, int32_t n_up, int32_t n_dn, int32_t n_walkers, double dt,
                                  double hs_constant, const double* exp_h1_up, const double* exp_h1_dn,
                                  const double* trial_up, const double* trial_dn, double* walkers_up,
                                  double* walkers_dn, double* weights, double* overlaps, double* scalars,
                                  const double* gaussian, void* stream) {
  if (!exp_h1_up || !exp_h1_dn || !trial_up || !trial_dn || !walkers_up || !walkers_dn || !weights || !overlaps ||
      !scalars || !gaussian) {
    afq_set_error("NULL argument");
    return -1;
  }
  if (!(dt > 0.0)) { afq_set_error("dt must be positive"); return -1; }
  return afq::launch_cpmc(norb, n_up, n_dn, n_walkers, dt, hs_constant, exp_h1_up, exp_h1_dn, trial_up, trial_dn,
                          walkers_up, walkers_dn, weights, overlaps, nullptr, scalars, gaussian, 2, S(stream));
}

int afq_fill_normal(double* out, int64_t n, uint64_t seed, uint64_t offset, void* stream) {
  if (!out && n > 0) { afq_set_error("NULL argument"); return -1; }
  return afq::launch_fill_normal(out, n, seed, offset, S(stream));
}

int afq_fill_uniform(double* out, int64_t n, uint64_t seed, uint64_t offset, void* stream) {
  if (!out && n > 0) { afq_set_error("NULL argument"); return -1; }
  return afq::launch_fill_uniform(out, n, seed, offset, S(stream));
}

}  // extern "C"
