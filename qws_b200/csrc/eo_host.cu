// Host side of the even-odd (site parity) operator family and its solver
// (deo_*/dee_*/one_minus_*, clvd_vm_/clv_s_, mtilde_vm_, mtilde_dag_vm_,
// mtilde_s_ of qws.cc:390-605 and bicgstab_vm_ of bicgstab.cc:68-333).
// At the API a parity-p vector is the parity-p sites of full DD-order planes.
// Single operators run on those; the Schur operators and solvers run on compact
// one-parity vectors, and on a compact copy of the fields where there can be one
// (eo.cu).
#include <cmath>
#include <complex>
#include <string>
#include <type_traits>
#include <vector>

#include "ctx.h"

namespace qwsg {

[[noreturn]] void throw_unsupported_eo() {
  throw Error(2, "even-odd operator: unsupported combination of hop set / adjoint / clover / mode");
}

// n doubles of work vectors, cleared
static double* eo_alloc(Ctx& c, size_t n) {
  void* q = c.device_alloc(sizeof(double) * n);
  const cudaError_t e = cudaMemsetAsync(q, 0, sizeof(double) * n, c.st);
  if (e != cudaSuccess) cudaFree(q);
  QWSG_CUDA(e);
  return static_cast<double*>(q);
}
// The first n FP64 work vectors.  Those of the operators (four, and two in
// FP32) come in one allocation on the first use of any of them: neighbouring
// pairs also serve as one vector on the full planes (2 eo_pad() >= G.pad), and
// a capture after that needs no more.
static double** eo_work(Ctx& c, int n) {
  const size_t ne = (size_t)24 * c.eo_pad();
  if (!c.eo_d[0]) {
    c.eo_d[0] = eo_alloc(c, (Ctx::kEoOpVecs + 1) * ne);
    c.owned.push_back(c.eo_d[0]);
    for (int i = 1; i < Ctx::kEoOpVecs; i++) c.eo_d[i] = c.eo_d[0] + i * ne;
    c.eo_s[0] = reinterpret_cast<float*>(c.eo_d[0] + Ctx::kEoOpVecs * ne);
    c.eo_s[1] = c.eo_s[0] + ne;
  }
  if (n > Ctx::kEoOpVecs && !c.eo_d[Ctx::kEoOpVecs]) {  // the solvers'
    c.eo_d[Ctx::kEoOpVecs] = eo_alloc(c, (Ctx::kEoVecs - Ctx::kEoOpVecs) * ne);
    c.owned.push_back(c.eo_d[Ctx::kEoOpVecs]);
    for (int i = Ctx::kEoOpVecs + 1; i < Ctx::kEoVecs; i++)
      c.eo_d[i] = c.eo_d[Ctx::kEoOpVecs] + (i - Ctx::kEoOpVecs) * ne;
  }
  return c.eo_d;
}

// The compact copy of the fields, made to follow them.  Null, and the fields
// are then read on the full planes (normal operator in FP64 at 24^3x48:
// 0.95 ms instead of 0.67),
//  - where device memory does not hold the copy (tried again by the next call);
//  - while the handle's stream is being captured: a graph that held launches on
//    the copy would read it as it was at the capture, whatever the fields have
//    become by its replay.
// One copy serves a lattice and the handles that borrow its fields, each on a
// stream of its own and perhaps in a thread of its own: it is made under the
// lock and complete when the lock is given back, and a call keeps the one it
// was given.
template <typename R>
using EoFields = std::shared_ptr<const EoCopy<R>>;
template <typename R>
static EoFields<R> eo_compact(Ctx& c) {
  constexpr bool d = std::is_same<R, double>::value;
  const R *U, *C;
  if constexpr (d) {
    U = c.eoUd ? c.eoUd : c.Ud;
    C = c.eoCd ? c.eoCd : c.Cd;
  } else {
    U = c.eoUs ? c.eoUs : c.Us;
    C = c.eoCs ? c.eoCs : c.Cs;
  }
  if (!U || !C) throw Error(4, "gauge/clover fields not loaded");
  if (c.st != nullptr && c.st != cudaStreamLegacy) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    QWSG_CUDA(cudaStreamIsCapturing(c.st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return nullptr;
  }
  Ctx& owner = c.parent ? *c.parent : c;
  std::lock_guard<std::mutex> lk(owner.eo_mu);
  const long gen = d ? owner.fields_gen_d : owner.fields_gen_s;
  const size_t pad = c.eo_pad();
  auto& copy = [&]() -> std::shared_ptr<EoCopy<R>>& {
    if constexpr (d)
      return owner.eoc_d;
    else
      return owner.eoc_s;
  }();
  if (!copy) {
    void* q = nullptr;
    const cudaError_t e = cudaMalloc(&q, sizeof(R) * 288 * pad);
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      return nullptr;
    }
    if (e != cudaSuccess)
      throw Error(3, std::string("even-odd copy of the fields: ") + cudaGetErrorString(e));
    copy = std::make_shared<EoCopy<R>>(static_cast<R*>(q));
  }
  if (copy->gen != gen) {
    eo_fields<R>(c.G, copy->p, copy->p + 144 * pad, (int)pad, U, C, c.st);
    c.check_launch("eo_fields");
    QWSG_CUDA(cudaStreamSynchronize(c.st));
    copy->gen = gen;
  }
  return copy;
}

// the compact vectors as the BLAS kernels see them: one RHS of Vh sites
static Geom eo_geom(const Ctx& c) {
  Geom G = c.G;
  G.V = c.G.Vh;
  G.pad = c.eo_pad();
  return G;
}

template <typename R>
static EoArgs<R> eo_args(const Ctx& c, int pe) {
  EoArgs<R> a{};
  a.G = c.G;
  a.pad = c.eo_pad();
  a.pe = pe;
  // the reference's rank box: each rank holds two x-halves (NB = 2*npe0, ...)
  a.box[0] = c.G.L[0] / (c.G.NB[0] / 2);
  for (int mu = 1; mu < 4; mu++) a.box[mu] = c.G.L[mu] / c.G.NB[mu];
  a.dxh = make_fastdiv(c.G.L[0] / 2);
  a.dy = make_fastdiv(c.G.L[1]);
  a.dz = make_fastdiv(c.G.L[2]);
  return a;
}
// on a compact copy F of the fields
template <typename R>
static EoArgs<R> eo_args_compact(const Ctx& c, const R* F, int pe) {
  EoArgs<R> a = eo_args<R>(c, pe);
  const size_t par = (size_t)72 * a.pad;
  a.U[0] = F + pe * par;
  a.U[1] = F + (1 - pe) * par;
  a.C = F + (2 + pe) * par;
  return a;
}

// one application of all hops on compact vectors (out: parity pe, in: the
// other; mode 0, or 2: out = in0 + factor * hops)
template <typename R>
static void eo_apply(Ctx& c, const R* F, R* out, const R* in, int pe, int dag, int clov, int mode,
                     double factor, const R* in0) {
  auto a = eo_args_compact<R>(c, F, pe);
  a.src = in;
  a.out = out;
  a.in0 = in0;
  a.coef = (R)factor;
  launch_eo<R>(dag, clov, mode, a, c.st);
}

// One operator of the API on the full planes as they are: no copy of the
// fields and no work vector, so that a call on new fields, the first call on a
// handle and one inside a stream capture cost what every call costs.
template <typename R>
void deo(Ctx& c, R* out, const R* in, int pe, int which, int dag, int clov, int mode,
         double factor, const R* in0) {
  if (pe != 0 && pe != 1) throw Error(1, "parity must be 0 or 1");
  if (mode == 2 && !in0) throw Error(1, "mode 2 needs in0");
  auto a = eo_args<R>(c, pe);
  if constexpr (std::is_same<R, double>::value) {
    a.U[0] = a.U[1] = c.eoUd ? c.eoUd : c.Ud;
    a.C = c.eoCd ? c.eoCd : c.Cd;
  } else {
    a.U[0] = a.U[1] = c.eoUs ? c.eoUs : c.Us;
    a.C = c.eoCs ? c.eoCs : c.Cs;
  }
  if (!a.U[0] || !a.C) throw Error(4, "gauge/clover fields not loaded");
  a.src = in;
  a.out = out;
  a.in0 = in0;
  a.coef = (R)factor;
  launch_eo_planes<R>(which, dag, clov, mode, a, c.st);
  c.check_launch("deo");
}
template void deo<float>(Ctx&, float*, const float*, int, int, int, int, int, double, const float*);
template void deo<double>(Ctx&, double*, const double*, int, int, int, int, int, double,
                          const double*);

template <typename R>
void clv(Ctx& c, R* out, const R* in, int pe) {
  const R* C;
  if constexpr (std::is_same<R, double>::value)
    C = c.eoCd ? c.eoCd : c.Cd;
  else
    C = c.eoCs ? c.eoCs : c.Cs;
  if (!C) throw Error(4, "clover field not loaded");
  launch_clv<R>(c.G, out, in, C, pe, c.st);
  c.check_launch("clv");
}
template void clv<float>(Ctx&, float*, const float*, int);
template void clv<double>(Ctx&, double*, const double*, int);

// mtilde_vm_: out_e = in_e - kappa^2 A_ee^-1 H_eo A_oo^-1 H_oe in_e
// (dee_deo_vm_(pco, pce) then one_minus_dee_deo_vm_(pce, pco)); compact, on the
// copy F of the fields, tmp of the other parity; out may be in
static void mtilde_c(Ctx& c, const double* F, double* out, const double* in, double* tmp) {
  eo_apply<double>(c, F, tmp, in, c.pco, 0, 1, 0, 0.0, nullptr);
  eo_apply<double>(c, F, out, tmp, c.pce, 0, 1, 2, -c.kappa * c.kappa, in);
}
// mtilde_dag_vm_: clvd_vm2_(pce), dee_deo_dag_vm_(pco, pce), one_minus_deo_dag_vm_(pce, pco)
static void mtilde_dag_c(Ctx& c, const double* F, double* out, const double* in, double* t0,
                         double* t1) {
  auto a = eo_args_compact<double>(c, F, c.pce);
  a.src = in;
  a.out = t0;
  launch_eo_clv<double>(a, c.st);
  eo_apply<double>(c, F, t1, t0, c.pco, 1, 1, 0, 0.0, nullptr);
  eo_apply<double>(c, F, out, t1, c.pce, 1, 0, 2, -c.kappa * c.kappa, in);
}
// mtdagmt_vm_ (qws.cc:566-571): mtilde_dag(mtilde(in)); work: eo_d[0 .. 2]
static void mtdagmt_c(Ctx& c, const double* F, double* out, const double* in) {
  mtilde_c(c, F, c.eo_d[2], in, c.eo_d[0]);
  mtilde_dag_c(c, F, out, c.eo_d[2], c.eo_d[0], c.eo_d[1]);
}

// the same on full planes; a work vector holds both parities' intermediates
// (mtilde_p: out may be in, or w; mtdagmt_p: in may be w0, out w1 or in)
template <typename R>
static void mtilde_p(Ctx& c, R* out, const R* in, R* w, double coef) {
  deo<R>(c, w, in, c.pco, 3, 0, 1, 0, 0.0, nullptr);
  deo<R>(c, out, w, c.pce, 3, 0, 1, 2, coef, in);
}
static void mtilde_dag_p(Ctx& c, double* out, const double* in, double* w) {
  clv<double>(c, w, in, c.pce);
  deo<double>(c, w, w, c.pco, 3, 1, 1, 0, 0.0, nullptr);
  deo<double>(c, out, w, c.pce, 3, 1, 0, 2, -c.kappa * c.kappa, in);
}
static void mtdagmt_p(Ctx& c, double* out, const double* in, double* w0, double* w1) {
  deo<double>(c, w0, in, c.pco, 3, 0, 1, 0, 0.0, nullptr);
  deo<double>(c, w1, w0, c.pce, 3, 0, 1, 2, -c.kappa * c.kappa, in);
  mtilde_dag_p(c, out, w1, w0);
}

// the solvers' operators: compact vectors in and out, on a compact copy F of
// the fields or (null) on the full planes; work: eo_d[0, 1] and eo_d[0 .. 3]
static void solve_mtilde(Ctx& c, const double* F, double* out, const double* in) {
  double* w = c.eo_d[0];
  if (F) return mtilde_c(c, F, out, in, w);
  eo_scatter<double>(c.G, w, in, c.eo_pad(), c.pce, false, c.st);
  mtilde_p<double>(c, w, w, w, -c.kappa * c.kappa);
  eo_gather<double>(c.G, out, c.eo_pad(), w, c.pce, c.st);
}
static void solve_mtdagmt(Ctx& c, const double* F, double* out, const double* in) {
  if (F) return mtdagmt_c(c, F, out, in);
  double *w0 = c.eo_d[0], *w1 = c.eo_d[2];
  eo_scatter<double>(c.G, w0, in, c.eo_pad(), c.pce, false, c.st);
  mtdagmt_p(c, w1, w0, w0, w1);
  eo_gather<double>(c.G, out, c.eo_pad(), w1, c.pce, c.st);
}

void mtilde_d(Ctx& c, double* out, const double* in) {
  double** v = eo_work(c, 2);
  if (const auto F = eo_compact<double>(c)) {
    eo_gather<double>(c.G, v[1], c.eo_pad(), in, c.pce, c.st);
    mtilde_c(c, F->p, v[1], v[1], v[0]);
    eo_scatter<double>(c.G, out, v[1], c.eo_pad(), c.pce, false, c.st);
  } else {
    mtilde_p<double>(c, out, in, v[0], -c.kappa * c.kappa);
  }
  c.n_mtilde++;
  c.check_launch("mtilde_d");
}

void mtilde_dag_d(Ctx& c, double* out, const double* in) {
  double** v = eo_work(c, 3);
  if (const auto F = eo_compact<double>(c)) {
    eo_gather<double>(c.G, v[2], c.eo_pad(), in, c.pce, c.st);
    mtilde_dag_c(c, F->p, v[2], v[2], v[0], v[1]);
    eo_scatter<double>(c.G, out, v[2], c.eo_pad(), c.pce, false, c.st);
  } else {
    mtilde_dag_p(c, out, in, v[0]);
  }
  c.check_launch("mtilde_dag_d");
}

void mtilde_s(Ctx& c, float* out, const float* in) {
  eo_work(c, 0);
  float** v = c.eo_s;
  const double coef = -(double)(float)(c.kappa * c.kappa);
  if (const auto F = eo_compact<float>(c)) {
    eo_gather<float>(c.G, v[1], c.eo_pad(), in, c.pce, c.st);
    eo_apply<float>(c, F->p, v[0], v[1], c.pco, 0, 1, 0, 0.0, nullptr);
    eo_apply<float>(c, F->p, v[1], v[0], c.pce, 0, 1, 2, coef, v[1]);
    eo_scatter<float>(c.G, out, v[1], c.eo_pad(), c.pce, false, c.st);
  } else {
    mtilde_p<float>(c, out, in, v[0], coef);
  }
  c.check_launch("mtilde_s");
}

void mtdagmt_d(Ctx& c, double* out, const double* in) {
  double** v = eo_work(c, 4);
  if (const auto F = eo_compact<double>(c)) {
    eo_gather<double>(c.G, v[3], c.eo_pad(), in, c.pce, c.st);
    mtdagmt_c(c, F->p, v[3], v[3]);
    eo_scatter<double>(c.G, out, v[3], c.eo_pad(), c.pce, false, c.st);
  } else {
    mtdagmt_p(c, out, in, v[0], v[2]);
  }
  c.check_launch("mtdagmt_d");
}

// bicgstab_vm_ (bicgstab.cc:68-333): BiCGStab on mtilde for the pce parity,
// iter = 1..maxiter-1, converged when sqrt(|r|^2/|b|^2) < 1e-14 after the
// omega step.  x: initial guess in, solution out.  Returns conviter.
int bicgstab_vm(Ctx& c, double* x, const double* b, int maxiter) {
  double** v = eo_work(c, 9);
  const auto fields = eo_compact<double>(c);
  const double* F = fields ? fields->p : nullptr;
  const Geom G = eo_geom(c);
  double *bb = v[2], *q = v[3], *r = v[4], *p = v[5], *t = v[6], *r0 = v[7], *xx = v[8];
  eo_gather<double>(c.G, bb, G.pad, b, c.pce, c.st);
  eo_gather<double>(c.G, xx, G.pad, x, c.pce, c.st);
  solve_mtilde(c, F, q, xx);
  blas_bicg_init<double>(G, bb, q, r, p, r0, c.d_res, c.rb, c.st);
  const double* h = c.fetch(2);
  const double bnorm = h[0];
  std::complex<double> rho0(h[1], 0), rho, beta, omega, alpha, ctmp;
  int iter;
  for (iter = 1; iter < maxiter; iter++) {
    solve_mtilde(c, F, q, p);
    blas_cdot<double>(G, r0, q, c.d_res, c.rb, c.st);
    h = c.fetch(2);
    ctmp = std::complex<double>(h[0], h[1]);
    alpha = rho0 / ctmp;
    blas_bicg_update<double>(G, xx, r, p, q, alpha.real(), alpha.imag(), nullptr, c.d_res, c.rb,
                             c.st);
    solve_mtilde(c, F, t, r);
    blas_norm_cdot<double>(G, t, r, c.d_res, c.rb, c.st);
    h = c.fetch(3);
    omega = std::complex<double>(h[1] / h[0], h[2] / h[0]);
    blas_bicg_update<double>(G, xx, r, r, t, omega.real(), omega.imag(), r0, c.d_res, c.rb, c.st);
    h = c.fetch(3);
    const double rnorm = h[0];
    rho = std::complex<double>(h[1], h[2]);
    if (std::sqrt(rnorm / bnorm) < 1e-14) break;
    beta = alpha * rho / (rho0 * omega);
    rho0 = rho;
    blas_bicg_p<double>(G, p, r, q, beta.real(), beta.imag(), omega.real(), omega.imag(), c.st);
  }
  eo_scatter<double>(c.G, x, xx, G.pad, c.pce, true, c.st);
  c.check_launch("bicgstab_vm");
  return iter;
}

static void check_finite(double v, const char* what) {
  if (!std::isfinite(v)) throw Error(3, std::string(what) + ": non-finite residual norm");
}

// cg_vm_ (cg.cc:65-172): CG on mtdagmt for the pce parity; x: initial guess
// in, solution out.  iter = 1..maxiter-1; converged when
// sqrt(|r|^2/|b|^2) < 1e-14 after the x/r update.  Returns the last iter
// (the reference does not report it).  A zero source returns x = 0 at
// iteration 0 (the reference divides 0 by 0 there).
int cg_vm(Ctx& c, double* x, const double* b, int maxiter) {
  double** v = eo_work(c, 10);
  const auto fields = eo_compact<double>(c);
  const double* F = fields ? fields->p : nullptr;
  const Geom G = eo_geom(c);
  double *q = v[4], *r = v[5], *p = v[6], *r0 = v[7], *bb = v[8], *xx = v[9];
  eo_gather<double>(c.G, bb, G.pad, b, c.pce, c.st);
  eo_gather<double>(c.G, xx, G.pad, x, c.pce, c.st);
  solve_mtdagmt(c, F, q, xx);
  blas_bicg_init<double>(G, bb, q, r, p, r0, c.d_res, c.rb, c.st);
  const double* h = c.fetch(2);
  const double bnorm = h[0];
  double rho0 = h[1];
  if (bnorm == 0) {
    blas_zero<double>(c.G, x, 0, c.G.V, c.st);
    return 0;
  }
  int iter;
  for (iter = 1; iter < maxiter; iter++) {
    solve_mtdagmt(c, F, q, p);
    blas_cdot<double>(G, p, q, c.d_res, c.rb, c.st);
    h = c.fetch(1);
    const double alpha = rho0 / h[0];
    blas_bicg_update<double>(G, xx, r, p, q, alpha, 0.0, nullptr, c.d_res, c.rb, c.st);
    h = c.fetch(1);
    const double rnorm = h[0];
    check_finite(rnorm, "cg_vm");
    if (std::sqrt(rnorm / bnorm) < 1e-14) break;
    const double beta = rnorm / rho0;
    rho0 = rnorm;
    blas_bicg_p<double>(G, p, r, q, beta, 0.0, 0.0, 0.0, c.st);
  }
  eo_scatter<double>(c.G, x, xx, G.pad, c.pce, true, c.st);
  c.check_launch("cg_vm");
  return iter;
}

// mcg_vm_ (mcg.cc:65-219): multi-shift CG for (mtdagmt + sigma_k) x_k = b,
// k < n, all x_k from zero, sharing the Krylov space of the unshifted
// system; the shifted coefficients follow the recurrence of mcg.cc:141-147
// (zeta ratios z_k) and every iteration's shift updates run in one kernel.
// Same stopping rule as cg_vm on the unshifted residual.  Returns the last
// iter.  A shift whose residual |z_k| |r| / |b| fell below 1e-14 is no
// longer updated (the reference keeps updating it until z_k underflows and
// 0/0 turns its solution into NaN; up to that point the two agree).
int mcg_vm(Ctx& c, double* X, const double* b, int n, const double* sigma, int maxiter) {
  if (n < 1 || n > Ctx::kMaxRhs) throw Error(1, "mcg_vm: number of shifts must be 1..32");
  if (c.G.nr != 1) throw Error(1, "mcg_vm: single right-hand side only");
  double** v = eo_work(c, 9);
  const Geom G = eo_geom(c);
  const size_t ne = (size_t)24 * G.pad;
  if (c.ms_n < n) {
    QWSG_CUDA(cudaStreamSynchronize(c.st));
    cudaFree(c.ms);
    c.ms = nullptr;
    c.ms_n = 0;
    c.ms = eo_alloc(c, 2 * ne * n);
    c.ms_n = n;
  }
  double *ms_p = c.ms, *ms_x = c.ms + ne * n;
  const auto fields = eo_compact<double>(c);
  const double* F = fields ? fields->p : nullptr;
  double *q = v[4], *r = v[5], *p = v[6], *r0 = v[7], *bb = v[8];
  eo_gather<double>(c.G, bb, G.pad, b, c.pce, c.st);
  blas_bicg_init<double>(G, bb, nullptr, r, p, r0, c.d_res, c.rb, c.st);
  const double* h = c.fetch(1);
  const double bnorm = h[0];
  double rho0 = bnorm;
  for (int k = 0; k < n; k++) {
    blas_zero<double>(G, ms_x + k * ne, 0, G.V, c.st);
    blas_copy<double>(G, ms_p + k * ne, r, 0, G.V, c.st);
  }
  if (bnorm == 0) {
    for (int k = 0; k < n; k++)
      blas_zero<double>(c.G, X + k * c.spinor_elems(), 0, c.G.V, c.st);
    return 0;
  }
  std::vector<double> z0(n, 1.0), z1(n, 1.0), z2(n, 0.0), cf(4 * n, 0.0);
  std::vector<char> active(n, 1);
  double alpha0 = 1.0, beta = 0.0;
  int iter;
  for (iter = 1; iter < maxiter; iter++) {
    solve_mtdagmt(c, F, q, p);
    blas_cdot<double>(G, p, q, c.d_res, c.rb, c.st);
    h = c.fetch(1);
    const double alpha = -rho0 / h[0];
    blas_axpy_norm<double>(G, r, q, alpha, c.d_res, c.rb, c.st);
    h = c.fetch(1);
    const double rnorm = h[0];
    check_finite(rnorm, "mcg_vm");
    const bool done = std::sqrt(rnorm / bnorm) < 1e-14;
    const double beta_new = rnorm / rho0;
    for (int k = 0; k < n; k++) {
      cf[4 * k + 3] = active[k];
      if (!active[k]) continue;
      z2[k] = z1[k] * z0[k] * alpha0 /
              (alpha * beta * (z0[k] - z1[k]) + z0[k] * alpha0 * (1.0 - sigma[k] * alpha));
      const double ratio = z2[k] / z1[k];
      cf[4 * k + 0] = alpha * ratio;           // x_k -= alpha z2/z1 pp_k
      cf[4 * k + 1] = z2[k];                   // pp_k = z2 r + ...
      cf[4 * k + 2] = beta_new * ratio * ratio;  // ... + beta (z2/z1)^2 pp_k
    }
    blas_mshift(G, ms_x, ms_p, n, r, p, beta_new, c.put_coefs(cf.data(), 4 * n), !done, c.st);
    if (done) break;
    beta = beta_new;
    rho0 = rnorm;
    for (int k = 0; k < n; k++) {
      if (!active[k]) continue;
      // converged shifts: their x_k is final after this iteration's update
      if (std::fabs(z2[k]) * std::sqrt(rnorm / bnorm) < 1e-14) active[k] = 0;
      z0[k] = z1[k];
      z1[k] = z2[k];
    }
    alpha0 = alpha;
  }
  for (int k = 0; k < n; k++)
    eo_scatter<double>(c.G, X + k * c.spinor_elems(), ms_x + k * ne, G.pad, c.pce, true, c.st);
  c.check_launch("mcg_vm");
  return iter;
}

}  // namespace qwsg
