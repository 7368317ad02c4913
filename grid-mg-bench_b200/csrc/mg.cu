// mg.cu -- multigrid-preconditioned Wilson-clover solve on the GPU.
//
// Restates the reference's multigrid driver:
//   MultiGridPreconditioner::operator() (include/MultigridPreconditioner.h:253-309):
//       restrict -> K-cycle wrapper solve on the next level, preconditioned by
//       the next level's cycle -> prolong -> post-smooth (no pre-smoothing)
//   coarsest level: a GMRES solve (:622-641)
//   test-vector setup (include/BasisVectors.h:74-149, NullVectorSetupRework.h):
//       random vectors, an approximate solve A psi = v, chiral doubling,
//       block orthonormalisation, then CoarsenOperator on every level
//   outer solve: FGMRES with the MG preconditioner (src/Test_wilsonclover_mg.cc:140,
//       mixed precision as src/Test_wilsonclover_mg_mp.cc:149-155)
// with the smoother of the multi-RHS configuration (MR, a fixed number of
// iterations) and every right-hand side of a batch solved together: vectors
// are [site][rhs][dof], each RHS keeps its own Krylov coefficients, and the
// outer solver compacts the batch at every restart so converged RHS drop out.
// The small per-RHS Krylov algebra (Hessenberg columns, Givens rotations,
// triangular solves) runs on the host.
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include <map>

#include "mg_internal.cuh"

typedef std::complex<double> zc;

namespace gmg {

struct MGLevel {
  int l = 0;
  Dims dims;
  int64_t V = 0;
  int dof = 0;
  int vprec = GMG_F64;    // vector precision inside the preconditioner
  int compute = GMG_F64;  // coarse-operator compute form (F64, F32, BF16)
  bool bf16_smoother = false;  // level 0: the MR smoother's residual fields in BF16
  gmg_wilson* w = nullptr;  // level 0 (not owned)
  gmg_coarse* c = nullptr;  // level > 0 (owned)
  gmg_agg* agg = nullptr;   // aggregation to level l+1 (owned)
  int m = 0;                // Krylov restart of the solver that runs on this level
  VecBuf V0, Z0, kw, kt;    // Krylov basis (m+1), flexible directions (m), temporaries
  VecBuf mr_r;              // MR smoother: the residual r and A r, two fields of one buffer
  VecBuf mr_r16, mr_Ar16;    // the fine smoother's residual fields in BF16 (params.smoother_bf16)
  int mr_keep = 1;           // residual fields in mr_r16: every step's (smoother_iters) or one
  VecBuf bc, xc;            // right-hand side / solution of this level inside the cycle above
  VecBuf tv;                // test vectors (nvec[l]) the basis to level l+1 is built from
  // device state of this level's solver inside a captured K-cycle: Hessenberg
  // [R][m+1][m], rhs g [R][m+1], Givens cs / sn [R][m], residual estimates [R],
  // solution coefficients y [m][R], counters {iterations, steps of the cycle},
  // |b|^2 and |r0|^2 per RHS
  DevBuf gH, gG, gCs, gSn, gRes, gY, gCtr, gBn, gBeta;
  ~MGLevel() {
    if (c) gmg_coarse_destroy(c);
    if (agg) gmg_agg_destroy(agg);
  }
};

}  // namespace gmg

struct gmg_mg {
  gmg_mg_params P;
  gmg_wilson* fine = nullptr;
  int Rmax = 0;
  std::vector<gmg::MGLevel*> L;
  gmg::DevBuf coef;        // device coefficients uploaded from the host (double2)
  gmg::DevBuf dscr;        // device-only per-RHS scalars: dots, norms (double2)
  double2* hpin = nullptr; // pinned host staging for coefficient transfers
  bool setup_done = false;
  // outer FGMRES workspace for max_rhs right-hand sides, allocated once.  The
  // Arnoldi fields (oV0, ow, otv, owc) are FP32 with params.arnoldi_f32, else
  // FP64; the residuals (orr: all RHS, orA: the batch) and ot64 are FP64.
  bool arn32 = false;
  gmg::VecBuf oV0, oZ0, ow, ot64, otz, obb, oxx, otv, orr, orA;
  gmg::VecBuf ozc, owc;   // compacted preconditioner output / operator output (in-cycle drop)
  gmg::DevBuf oidx, oidx2;
  bool outer_ready = false;
  // captured coarse-level solves of the K-cycle per active-batch size
  // (params.graph) and the capture streams of the nested conditional bodies
  std::map<int, cudaGraphExec_t> kgraph;
  cudaStream_t cap_st[8] = {};
  bool graph_broken = false;
  // per-RHS outcome of the last solve: the outer iteration count at which the
  // RHS left the active batch (its true residual below tol), and that residual
  std::vector<int> last_iters;
  std::vector<double> last_relres;
  std::vector<int> last_batches;  // active batch size of every outer Arnoldi step of the last solve
  ~gmg_mg() {
    for (auto& g : kgraph) cudaGraphExecDestroy(g.second);
    for (auto& st : cap_st)
      if (st) cudaStreamDestroy(st);
    for (auto* l : L) delete l;
    if (hpin) cudaFreeHost(hpin);
  }
};

namespace gmg {
namespace {

// ------------------------------------------------------------- small helpers
gmg_status apply_op(gmg_mg* h, int l, const Vec& in, Vec& out, cudaStream_t s);

// out = A in with in in the preconditioner precision and out in FP64: on the
// fine level the FP64 operator reads the FP32 field directly; elsewhere `in`
// is converted into t (FP64) first
gmg_status apply_op_mixed(gmg_mg* h, int l, const Vec& in, Vec& t, Vec& out, cudaStream_t s) {
  if (l == 0 && in.prec == GMG_F32 && out.prec == GMG_F64)
    return gmg_wilson_apply_f32_in(h->L[0]->w, GMG_OP_M, in.R, static_cast<const float*>(in.p),
                                   static_cast<double*>(out.p), (gmg_stream)s);
  GMG_TRY(vec_convert(in, t, s));
  return apply_op(h, l, t, out, s);
}

gmg_status apply_op(gmg_mg* h, int l, const Vec& in, Vec& out, cudaStream_t s) {
  MGLevel& L = *h->L[l];
  if (l == 0) return gmg_wilson_apply(L.w, GMG_OP_M, 0, 0, (gmg_prec)in.prec, in.R, in.p, out.p, (gmg_stream)s);
  const int compute = in.prec == GMG_F64 ? GMG_F64 : L.compute;
  return gmg_coarse_apply(L.c, GMG_OP_M, 8, (gmg_prec)compute, (gmg_prec)in.prec, in.R, in.p, out.p, nullptr, 0,
                          (gmg_stream)s);
}

// r = b - A x on the fine level in FP64: one fused operator pass where the
// tile kernel applies (4+ RHS, 32-byte aligned fields), else the operator and
// a subtraction sweep
gmg_status fine_residual(gmg_mg* h, const Vec& b, const Vec& x, Vec& r, cudaStream_t s) {
  if (x.R >= 4 && x.prec == GMG_F64 && (((uintptr_t)b.p | (uintptr_t)x.p | (uintptr_t)r.p) & 31) == 0)
    return wilson_residual_f64(h->L[0]->w, x.R, static_cast<const double*>(b.p), static_cast<const double*>(x.p),
                               static_cast<double*>(r.p), s);
  GMG_TRY(apply_op(h, 0, x, r, s));
  return vec_xmy(b, r, s);
}

constexpr int kScalars = 8192;  // double2 slots of h->coef, h->dscr and h->hpin

// host <- n device scalars (one stream synchronisation)
gmg_status download(gmg_mg* h, const double2* d, int n, std::vector<zc>& out, cudaStream_t s) {
  GMG_CHECK(n <= kScalars, GMG_ERR_UNSUPPORTED, "mg: too many per-RHS scalars");
  GMG_CUDA(cudaMemcpyAsync(h->hpin, d, sizeof(double2) * n, cudaMemcpyDeviceToHost, s));
  GMG_CUDA(cudaStreamSynchronize(s));
  out.resize(n);
  for (int k = 0; k < n; ++k) out[k] = zc(h->hpin[k].x, h->hpin[k].y);
  return GMG_OK;
}

// host <- per-RHS <X_j, Y> for j < nx
gmg_status dots(gmg_mg* h, const Vec& X0, int nx, int64_t xstride, const Vec& Y, std::vector<zc>& out,
                cudaStream_t s) {
  double2* d = h->dscr.as<double2>();
  GMG_TRY(vec_multidot(X0, nx, xstride, Y, d, nullptr, s));
  return download(h, d, nx * Y.R, out, s);
}

// device coef[offset...] <- a, through the pinned staging buffer.  The copy is
// asynchronous: every caller reaches a download() (a stream synchronisation)
// before the staging buffer is written again.
gmg_status upload(gmg_mg* h, const std::vector<zc>& a, size_t offset_elems, cudaStream_t s) {
  GMG_CHECK(a.size() <= (size_t)kScalars, GMG_ERR_UNSUPPORTED, "mg: too many coefficients");
  for (size_t k = 0; k < a.size(); ++k) h->hpin[k] = make_double2(a[k].real(), a[k].imag());
  GMG_CUDA(cudaMemcpyAsync(h->coef.as<double2>() + offset_elems, h->hpin, sizeof(double2) * a.size(),
                           cudaMemcpyHostToDevice, s));
  return GMG_OK;
}

// Y += sum_j c[j*R + r] X_j
gmg_status multiaxpy_h(gmg_mg* h, const std::vector<zc>& c, const Vec& X0, int nx, int64_t xstride, Vec& Y,
                       cudaStream_t s) {
  GMG_TRY(upload(h, c, 0, s));
  return vec_multiaxpy(h->coef.as<double2>(), X0, nx, xstride, Y, s);
}

Vec nth(const Vec& base, int j) {
  Vec v = base;
  v.p = static_cast<char*>(base.p) + (size_t)j * base.bytes();
  return v;
}

gmg_status zero(Vec& v, cudaStream_t s) {
  GMG_CUDA(cudaMemsetAsync(v.p, 0, v.bytes(), s));
  return GMG_OK;
}


// ------------------------------------------------------------- global orthonormalisation
// Orthonormalise the R columns of X over the whole lattice, as the reference's
// test-vector setup does before and after the solves (BasisVectors.h:86-147,
// setupPre/PostOrthonormalise, MultigridParams.h:103-104): Cholesky QR on the
// R x R Gram matrix (formed on the device, factored on the host), two passes;
// a pass whose factorisation breaks down is redone with the shifted-Cholesky
// diagonal shift and followed by extra plain passes.
gmg_status global_orthonormalise(gmg_mg* h, Vec& X, cudaStream_t s) {
  const int R = X.R;
  double2* G = h->dscr.as<double2>();
  const double K = (double)X.V * X.dof;
  int passes = 2;
  for (int pass = 0; pass < passes; ++pass) {
    GMG_TRY(vec_gram(X, G, s));
    std::vector<zc> g;
    GMG_TRY(download(h, G, R * R, g, s));
    std::vector<zc> L;
    auto chol = [&](double shift) -> bool {
      L.assign((size_t)R * R, zc(0));
      for (int j = 0; j < R; ++j) {
        double d = g[(size_t)j * R + j].real() + shift;
        for (int k = 0; k < j; ++k) d -= std::norm(L[(size_t)j * R + k]);
        if (!(d > 0.0)) return false;
        const double dj = std::sqrt(d);
        L[(size_t)j * R + j] = dj;
        for (int i = j + 1; i < R; ++i) {  // L[i][j] = (G[i][j] - sum_k L[i][k] conj(L[j][k])) / L[j][j]
          zc v = g[(size_t)i * R + j];
          for (int k = 0; k < j; ++k) v -= L[(size_t)i * R + k] * std::conj(L[(size_t)j * R + k]);
          L[(size_t)i * R + j] = v / dj;
        }
      }
      return true;
    };
    if (!chol(0.0)) {
      double tr = 0.0;
      for (int i = 0; i < R; ++i) tr += g[(size_t)i * R + i].real();
      const double shift = 11.0 * (K * R + (double)R * (R + 1)) * 1.1102230246251565e-16 * tr;
      if (!chol(shift)) return fail(GMG_ERR_NONFINITE, "mg setup: test vectors are linearly dependent");
      passes = std::min(pass + 3, 5);
    }
    // T = conj(L^{-1}) (lower triangular): X(a) <- sum_{b <= a} T[a][b] X(b)
    std::vector<zc> Li((size_t)R * R, zc(0));
    for (int j = 0; j < R; ++j) {
      Li[(size_t)j * R + j] = 1.0 / L[(size_t)j * R + j];
      for (int i = j + 1; i < R; ++i) {
        zc acc = 0.0;
        for (int k = j; k < i; ++k) acc += L[(size_t)i * R + k] * Li[(size_t)k * R + j];
        Li[(size_t)i * R + j] = -acc / L[(size_t)i * R + i];
      }
    }
    for (auto& v : Li) v = std::conj(v);
    GMG_TRY(upload(h, Li, 0, s));
    GMG_TRY(vec_tri_apply(h->coef.as<double2>(), X, s));
  }
  return GMG_OK;
}

// ------------------------------------------------------------- BiCGStab (setup solver)
// Multi-RHS BiCGStab on A x = b at level l, the reference's setup solver
// (setupSolverType BiCGSTAB, tolerance 1e-3, 100 iterations,
// MultigridParams.h:105-107).  The per-RHS scalars rho, alpha, omega, beta stay
// on the device (h->coef + 4096); residual norms come back every 8 iterations.
// ws: 6 fields shaped like b (r, r0, p, v, s, t).
gmg_status bicgstab(gmg_mg* h, int l, const Vec& b, Vec& x, int maxit, double tol, VecBuf* ws, cudaStream_t s) {
  const int R = b.R;
  GMG_CHECK(R <= 32, GMG_ERR_UNSUPPORTED, "bicgstab: at most 32 right-hand sides");
  Vec r = ws[0].with_rhs(R), r0 = ws[1].with_rhs(R), p = ws[2].with_rhs(R), v = ws[3].with_rhs(R),
      sv = ws[4].with_rhs(R), t = ws[5].with_rhs(R);
  double2* sc = h->coef.as<double2>() + 4096;  // [4R]: rho, alpha, omega, beta
  double2* d = h->dscr.as<double2>() + 2048;   // dot products [5R]
  std::vector<zc> bn;
  GMG_TRY(dots(h, b, 1, 0, b, bn, s));
  GMG_TRY(apply_op(h, l, x, r, s));
  GMG_TRY(vec_xmy(b, r, s));  // r = b - A x
  GMG_CUDA(cudaMemcpyAsync(r0.p, r.p, r.bytes(), cudaMemcpyDeviceToDevice, s));
  GMG_TRY(zero(p, s));
  GMG_TRY(zero(v, s));
  std::vector<zc> init(4 * (size_t)R, zc(1.0));
  GMG_TRY(upload(h, init, 4096, s));
  for (int it = 0; it < maxit; ++it) {
    GMG_TRY(vec_multidot(r0, 1, 0, r, d, nullptr, s));  // rho_new = <r0, r>
    GMG_TRY(bicg_scalar(0, d, nullptr, sc, R, s));       // beta, rho
    GMG_TRY(bicg_vec(0, p, r, v, v, v, sc, s));          // p = r + beta (p - omega v)
    GMG_TRY(apply_op(h, l, p, v, s));                    // v = A p
    GMG_TRY(vec_multidot(r0, 1, 0, v, d + R, nullptr, s));
    GMG_TRY(bicg_scalar(1, d + R, nullptr, sc, R, s));   // alpha = rho / <r0, v>
    GMG_TRY(bicg_vec(1, sv, r, v, v, v, sc, s));         // s = r - alpha v
    GMG_TRY(apply_op(h, l, sv, t, s));                   // t = A s
    GMG_TRY(vec_multidot(t, 1, 0, sv, d + 2 * R, nullptr, s));
    GMG_TRY(vec_multidot(t, 1, 0, t, d + 3 * R, nullptr, s));
    GMG_TRY(bicg_scalar(2, d + 2 * R, d + 3 * R, sc, R, s));  // omega = <t, s> / <t, t>
    GMG_TRY(bicg_vec(2, x, r, p, sv, t, sc, s));         // x += alpha p + omega s; r = s - omega t
    if ((it + 1) % 8 == 0 || it + 1 == maxit) {
      std::vector<zc> rn;
      GMG_TRY(dots(h, r, 1, 0, r, rn, s));
      bool conv = true;
      for (int k = 0; k < R; ++k)
        if (rn[k].real() > tol * tol * bn[k].real()) conv = false;
      if (conv) break;
    }
  }
  return GMG_OK;
}

// ------------------------------------------------------------- MR smoother
// x <- x + iters steps of minimal residual for A x = b on level l
// The step lengths stay on the device: no host synchronisation.
gmg_status mr_smooth(gmg_mg* h, int l, const Vec& b, Vec& x, int iters, cudaStream_t s) {
  MGLevel& L = *h->L[l];
  const int R = b.R;
  Vec r = L.mr_r.with_rhs(R), Ar = r;
  Ar.p = static_cast<char*>(r.p) + r.bytes();
  double2* d1 = h->dscr.as<double2>() + kScalars / 2;  // above the Krylov scalars
  double2* d2 = d1 + R;
  if (l == 0 && L.bf16_smoother && x.prec == GMG_F32) {
    // the residual and the operator product kept in BF16 (FP32 arithmetic,
    // FP32 solution): the smoother's sweeps move half the bytes
    Vec r16 = L.mr_r16.with_rhs(R), Ar16 = L.mr_Ar16.with_rhs(R);
    if (iters <= L.mr_keep) {
      // every step's residual kept (r_j at j * fs words, its step length at
      // d1 + 2 R j): x += sum_j a_j r_j in one sweep at the end, so a step
      // moves r, Ar and the next r, and x is read and written once.  The
      // residual fields are site-blocked (the quarters of one site's records
      // back to back), so the operator's record gathers read contiguous runs.
      if ((((uintptr_t)b.p | (uintptr_t)x.p) & 31) == 0) {
        // r = b - A x, formed by the operator's epilogue
        GMG_TRY(wilson_residual_bf16(L.w, R, static_cast<const float*>(b.p), static_cast<const float*>(x.p),
                                     static_cast<uint32_t*>(r16.p), s));
      } else {
        GMG_TRY(apply_op(h, l, x, r, s));
        GMG_TRY(vec_xmy_bf16_blocked(b, r, r16, s));  // r = b - A x
      }
      const int64_t fs = r16.elems();
      for (int it = 0; it < iters; ++it) {
        Vec rj = r16;
        rj.p = static_cast<uint32_t*>(r16.p) + it * fs;
        double2* a1 = d1 + 2 * (size_t)R * it;
        GMG_TRY(wilson_apply_mr_bf16(L.w, R, static_cast<const uint32_t*>(rj.p), static_cast<uint32_t*>(Ar16.p), a1,
                                     a1 + R, s, true));
        if (it + 1 < iters) {
          Vec rn = rj;
          rn.p = static_cast<uint32_t*>(rj.p) + fs;
          GMG_TRY(vec_mr_resid_bf16(a1, a1 + R, rj, Ar16, rn, s, true));
        }
      }
      return vec_mr_xsum_bf16(d1, 2 * R, iters, r16, fs, x, s, true);
    }
    GMG_TRY(apply_op(h, l, x, r, s));
    GMG_TRY(vec_xmy_bf16(b, r, r16, s));  // r = b - A x
    for (int it = 0; it < iters; ++it) {
      GMG_TRY(wilson_apply_mr_bf16(L.w, R, static_cast<const uint32_t*>(r16.p), static_cast<uint32_t*>(Ar16.p), d1,
                                   d2, s));
      GMG_TRY(vec_mr_update(d1, d2, x, r16, Ar16, s, it + 1 < iters));
    }
    return GMG_OK;
  }
  GMG_TRY(apply_op(h, l, x, r, s));
  GMG_TRY(vec_xmy(b, r, s));  // r = b - A x
  for (int it = 0; it < iters; ++it) {
    if (l == 0) {
      // the fine operator forms both inner products in its epilogue
      GMG_TRY(wilson_apply_mr(L.w, r.prec, R, r.p, Ar.p, d1, d2, s));
      // the residual of the last step is never read
      GMG_TRY(vec_mr_update(d1, d2, x, r, Ar, s, it + 1 < iters));
    } else {
      GMG_TRY(apply_op(h, l, r, Ar, s));
      if (rhs_fused(x, 1)) {
        GMG_TRY(rhs_mr_step(x, r, Ar, it + 1 < iters, s));
        continue;
      }
      // one sweep for both products: d1 = <r, Ar> (the conjugate of <Ar, r>), d2 = <Ar, Ar>
      GMG_TRY(vec_multidot(r, 2, r.elems(), Ar, d1, nullptr, s));
      GMG_TRY(vec_mr_update(d1, d2, x, r, Ar, s, it + 1 < iters, true));
    }
  }
  return GMG_OK;
}

// ------------------------------------------------------------- (F)GMRES
// Solve A x = b on level l from the initial guess in x; per-RHS relative
// tolerance tol; at most maxit iterations in cycles of m.  `prec(in, out)`
// (flexible) is applied when given.  Krylov vectors live on level l's
// workspace; for level 0 with FP64 vectors the caller supplies them (outer).
struct Krylov {
  Vec V0, Z0;   // V: m+1 vectors, Z: m vectors (Z0.p == nullptr -> not flexible)
  Vec w, t;     // temporaries, precision of V (t: precision of Z)
  Vec tz;       // Z-precision temporary for the preconditioner input (may equal V precision)
};

// In-cycle drop of converged right-hand sides (outer solve, flexible).  The
// Arnoldi processes of the RHS are independent (one Hessenberg matrix each),
// so an RHS whose residual estimate meets the tolerance at step j keeps its
// j + 1 directions and takes no further part: the preconditioner and the
// operator of the later steps run on the still-active columns only, gathered
// into a compact batch (zc, wc; idx on the device) and scattered back into
// the full-width Krylov vectors, whose other columns are zero.
struct DropCtx {
  Vec zc, wc;                  // compact scratch: preconditioner precision, FP64
  int* idx = nullptr;          // device, active columns of the compact batch
  bool enabled = false;        // drop (true) or only record the steps
  bool dcgs = false;           // Gram-Schmidt with delayed reorthogonalisation (params.outer_dcgs)
  std::vector<int> conv_step;  // out: per column, the step (1-based) its estimate met tol; 0: never
  std::vector<int>* batches = nullptr;  // out: appended active-batch size of every step
  // FP64 residual b - A x of the batch, formed by the caller: one restart
  // cycle starts from it (the first Krylov vector in the basis precision)
  // and the solve returns after that cycle, the caller forming the next one
  const Vec* r0 = nullptr;
};

// min |beta0 e1 - H y| over y for the (n + 1) x n upper Hessenberg H (row
// stride m), by Givens rotations on a copy; returns the residual norm and, when
// y is given, the solution y[0 .. n-1] (entries at stride ys)
double hess_lsq(const zc* H, int m, int n, double beta0, zc* y, int ys) {
  std::vector<zc> A((size_t)(n + 1) * n), gg(n + 1, zc(0));
  for (int i = 0; i <= n; ++i)
    for (int k = 0; k < n; ++k) A[(size_t)i * n + k] = H[i * m + k];
  gg[0] = beta0;
  for (int k = 0; k < n; ++k) {
    const zc a = A[(size_t)k * n + k], bq = A[(size_t)(k + 1) * n + k];
    const double den = std::sqrt(std::norm(a) + std::norm(bq));
    zc c = 1.0, sg = 0.0;
    if (den > 0) {
      c = a / den;
      sg = bq / den;
    }
    for (int q = k; q < n; ++q) {
      const zc u = A[(size_t)k * n + q], v = A[(size_t)(k + 1) * n + q];
      A[(size_t)k * n + q] = std::conj(c) * u + std::conj(sg) * v;
      A[(size_t)(k + 1) * n + q] = -sg * u + c * v;
    }
    const zc gk = gg[k];
    gg[k] = std::conj(c) * gk;
    gg[k + 1] = -sg * gk;
  }
  if (y) {
    for (int i = n - 1; i >= 0; --i) {
      zc acc = gg[i];
      for (int k = i + 1; k < n; ++k) acc -= A[(size_t)i * n + k] * y[(size_t)k * ys];
      y[(size_t)i * ys] = A[(size_t)i * n + i] != zc(0) ? acc / A[(size_t)i * n + i] : zc(0);
    }
  }
  return std::abs(gg[n]);
}

template <class Prec>
gmg_status fgmres(gmg_mg* h, int l, const Vec& b, Vec& x, const Krylov& K, int m, int maxit, double tol, Prec prec,
                  bool flexible, int* iters_out, std::vector<double>* relres, cudaStream_t s,
                  DropCtx* drop = nullptr) {
  const int R = b.R;
  // per column: still iterating, and the Arnoldi steps it keeps
  std::vector<char> live(R, 1);
  std::vector<int> keep(R, 0), act;
  if (drop) drop->conv_step.assign(R, 0);
  Vec V0 = K.V0.with_rhs(R), Z0 = K.Z0.with_rhs(R), w = K.w.with_rhs(R), t = K.t.with_rhs(R), tz = K.tz.with_rhs(R);
  const int64_t vstride = V0.elems(), zstride = Z0.elems();
  std::vector<zc> bn;
  GMG_TRY(dots(h, b, 1, 0, b, bn, s));
  std::vector<double> bnorm(R);
  for (int r = 0; r < R; ++r) bnorm[r] = std::sqrt(std::max(bn[r].real(), 1e-300));
  std::vector<double> res(R, 1.0);
  int iters = 0;
  std::vector<zc> H((size_t)(m + 1) * m * R), g((size_t)(m + 1) * R), cs((size_t)m * R), sn((size_t)m * R);
  // DCGS2 (outer solve): H kept unrotated, with each column corrected one step
  // later for the delayed second projection of its last basis vector
  const bool dcgs = drop && drop->dcgs && flexible && vec_dcgs_supported(K.w.with_rhs(R), m - 1);
  std::vector<double> beta0(R, 0.0), betaT(R, 0.0), ctol(R, tol);
  const Vec* r0 = drop ? drop->r0 : nullptr;
  for (int cycle = 0;; ++cycle) {
    // r0 = b - A x -> V_0 (given by the caller for one cycle, or formed here)
    Vec v0 = nth(V0, 0);
    if (r0 && cycle > 0) break;
    if (!r0) {
      GMG_TRY(apply_op(h, l, x, w, s));
      GMG_TRY(vec_xmy(b, w, s));  // w = b - A x
    }
    const Vec& rv = r0 ? *r0 : w;
    std::vector<zc> bb;
    double2* dn = h->dscr.as<double2>();
    GMG_TRY(vec_multidot(rv, 1, 0, rv, dn, nullptr, s));
    GMG_TRY(download(h, dn, R, bb, s));
    bool all = true;
    std::vector<double> beta(R);
    for (int r = 0; r < R; ++r) {
      beta[r] = std::sqrt(std::max(bb[r].real(), 0.0));
      res[r] = beta[r] / bnorm[r];
      if (res[r] > tol) all = false;
    }
    if (all || iters >= maxit) break;
    // a cycle in FP32 (the basis precision) cannot reduce a residual by much
    // more than FP32 resolves: a column whose estimate falls to 1e-6 of the
    // cycle's starting residual has done what the cycle can do, and is treated
    // as converged for this cycle (the caller's FP64 residual decides)
    const double floor = V0.prec == GMG_F32 ? 1e-6 : 0.0;
    for (int r = 0; r < R; ++r) ctol[r] = std::max(tol, floor * res[r]);
    // a new cycle: every column takes part again (dropped ones have been folded into x)
    std::fill(live.begin(), live.end(), 1);
    act.resize(R);
    for (int r = 0; r < R; ++r) act[r] = r;
    GMG_TRY(vec_scale_inv_norm(dn, rv, v0, s));
    std::fill(H.begin(), H.end(), zc(0));
    std::fill(g.begin(), g.end(), zc(0));
    for (int r = 0; r < R; ++r) g[(size_t)r * (m + 1)] = beta[r];  // per-RHS residual vector, [R][m+1]
    beta0 = beta;
    int jl = -1;
    for (int j = 0; j < m && iters < maxit; ++j) {
      Vec vj = nth(V0, j);
      Vec zj = flexible ? nth(Z0, j) : vj;
      const int Ra = (int)act.size();
      if (drop && drop->batches) drop->batches->push_back(Ra);
      if (drop && drop->enabled && flexible && Ra < R) {
        // compact: v_j's active columns -> preconditioner -> operator, scattered back
        Vec vc = t.with_rhs(Ra), zc = drop->zc.with_rhs(Ra), wc = drop->wc.with_rhs(Ra);
        GMG_TRY(vec_gather(vj, drop->idx, vc, s));
        GMG_TRY(prec(vc, zc, tz));
        GMG_CUDA(cudaMemsetAsync(zj.p, 0, zj.bytes(), s));
        GMG_TRY(vec_scatter(zc, drop->idx, zj, s));
        if (zc.prec != wc.prec) {
          GMG_TRY(apply_op_mixed(h, l, zc, vc, wc, s));
        } else {
          GMG_TRY(apply_op(h, l, zc, wc, s));
        }
        GMG_CUDA(cudaMemsetAsync(w.p, 0, w.bytes(), s));
        GMG_TRY(vec_scatter(wc, drop->idx, w, s));
      } else {
        if (flexible) GMG_TRY(prec(vj, zj, tz));
        if (zj.prec != w.prec) {
          GMG_TRY(apply_op_mixed(h, l, zj, t, w, s));
        } else {
          GMG_TRY(apply_op(h, l, zj, w, s));
        }
      }
      if (dcgs) {
        // Gram-Schmidt with delayed reorthogonalisation: V_0 .. V_{j-1} are
        // final, V_j has had one projection.  One sweep forms V_j's second
        // projection coefficients c, w's projections g and three norms; the host
        // forms alpha = |V_j - V c| and the new vector's coefficient d and norm
        // beta by Pythagoras; a second sweep finishes V_j and writes V_{j+1}
        // after one projection.  Two sweeps over the basis per step instead of
        // three and a scaling sweep.
        const int nv = j;
        double2* dd = h->dscr.as<double2>();
        GMG_TRY(vec_dcgs_dots(V0, vstride, nv, w, dd, s));
        std::vector<zc> col;
        GMG_TRY(download(h, dd, (2 * nv + 3) * R, col, s));
        std::vector<zc> cf((size_t)(2 * nv + 3) * R, zc(0));
        for (int r = 0; r < R; ++r) {
          cf[(size_t)(2 * nv) * R + r] = 1.0;  // dropped columns: V_j unchanged, V_{j+1} = 0
          if (!live[r]) continue;
          const double t1 = col[(size_t)(2 * nv) * R + r].real(), t3 = col[(size_t)(2 * nv + 2) * R + r].real();
          double a2 = t1;
          zc d = col[(size_t)(2 * nv + 1) * R + r];
          for (int k = 0; k < nv; ++k) a2 -= std::norm(col[(size_t)k * R + r]);
          const double alpha = nv == 0 ? 1.0 : std::sqrt(std::max(a2, 1e-30 * std::max(t1, 1e-300)));
          for (int k = 0; k < nv; ++k) d -= std::conj(col[(size_t)k * R + r]) * col[(size_t)(nv + k) * R + r];
          d /= alpha;
          double b2 = t3 - std::norm(d);
          for (int k = 0; k < nv; ++k) b2 -= std::norm(col[(size_t)(nv + k) * R + r]);
          const double bt = std::sqrt(std::max(b2, 0.0));
          for (int k = 0; k < nv; ++k) {
            cf[(size_t)k * R + r] = col[(size_t)k * R + r];
            cf[(size_t)(nv + k) * R + r] = col[(size_t)(nv + k) * R + r];
          }
          cf[(size_t)(2 * nv) * R + r] = 1.0 / alpha;
          cf[(size_t)(2 * nv + 1) * R + r] = d;
          cf[(size_t)(2 * nv + 2) * R + r] = bt > 0 ? 1.0 / bt : 0.0;
          zc* Hr = &H[(size_t)r * (m + 1) * m];
          if (nv > 0) {  // column j - 1 with V_j's second projection
            for (int k = 0; k < nv; ++k) Hr[k * m + (j - 1)] += betaT[r] * col[(size_t)k * R + r];
            Hr[j * m + (j - 1)] = betaT[r] * alpha;
          }
          for (int k = 0; k < nv; ++k) Hr[k * m + j] = col[(size_t)(nv + k) * R + r];
          Hr[j * m + j] = d;
          Hr[(j + 1) * m + j] = bt;
          betaT[r] = bt;
          res[r] = hess_lsq(Hr, m, j + 1, beta0[r], nullptr, 0) / bnorm[r];
        }
        GMG_TRY(upload(h, cf, 0, s));
        GMG_TRY(vec_dcgs_update(h->coef.as<double2>(), V0, vstride, nv, w, s));
      } else {
      // classical Gram-Schmidt, twice, with the coefficients kept on the device;
      // the Hessenberg column comes back to the host in one transfer.  (With a
      // good preconditioner w = A z_j is close to v_j, the first pass cancels
      // most of w, and a selective second pass would run on every step.)
      const size_t nc = (size_t)(j + 1) * R;
      double2* dh = h->dscr.as<double2>();
      double2* dh2 = dh + nc;
      double2* dw = dh2 + nc;
      // pass 1: dh = V^H w; then w -= V dh fused with pass 2's dh2 = V^H w;
      // then w -= V dh2 fused with dw = |w|^2
      Vec vn = nth(V0, j + 1);
      if (l > 0 && V0.prec == w.prec && rhs_fused(w, m)) {
        GMG_TRY(rhs_gs_step(V0, vstride, j + 1, w, vn, dh, dh2, dw, RhsGivens{}, s));
      } else {
        GMG_TRY(vec_multidot(V0, j + 1, vstride, w, dh, nullptr, s));
        GMG_TRY(vec_multiaxpy_dot(dh, V0, j + 1, vstride, w, s, -1.0, dh2, 1));
        GMG_TRY(vec_multiaxpy_dot(dh2, V0, j + 1, vstride, w, s, -1.0, dw, 2));
        GMG_TRY(vec_scale_inv_norm(dw, w, vn, s));
      }
      std::vector<zc> col;
      GMG_TRY(download(h, dh, (int)(2 * nc + R), col, s));
      std::vector<zc> hc(nc);
      for (size_t k = 0; k < nc; ++k) hc[k] = col[k] + col[nc + k];
      for (int r = 0; r < R; ++r) {
        if (!live[r]) continue;  // dropped: its Hessenberg matrix is complete
        const double hn = std::sqrt(std::max(col[2 * nc + r].real(), 0.0));
        // Hessenberg column j of RHS r, Givens rotations
        zc* Hr = &H[(size_t)r * (m + 1) * m];
        for (int i = 0; i <= j; ++i) Hr[i * m + j] = hc[(size_t)i * R + r];
        Hr[(j + 1) * m + j] = hn;
        for (int i = 0; i < j; ++i) {
          const zc c = cs[(size_t)r * m + i], sgn = sn[(size_t)r * m + i];
          const zc a = Hr[i * m + j], bq = Hr[(i + 1) * m + j];
          Hr[i * m + j] = std::conj(c) * a + std::conj(sgn) * bq;
          Hr[(i + 1) * m + j] = -sgn * a + c * bq;
        }
        const zc a = Hr[j * m + j];
        const double bq = std::abs(Hr[(j + 1) * m + j]);
        const double den = std::sqrt(std::norm(a) + bq * bq);
        zc c = 1.0, sgn = 0.0;
        if (den > 0) {
          c = a / den;
          sgn = Hr[(j + 1) * m + j] / den;
        }
        cs[(size_t)r * m + j] = c;
        sn[(size_t)r * m + j] = sgn;
        Hr[j * m + j] = std::conj(c) * a + std::conj(sgn) * Hr[(j + 1) * m + j];
        Hr[(j + 1) * m + j] = 0.0;
        zc* gr = &g[(size_t)r * (m + 1)];
        const zc gj = gr[j];
        gr[j] = std::conj(c) * gj;
        gr[j + 1] = -sgn * gj;
        res[r] = std::abs(gr[j + 1]) / bnorm[r];
      }
      }
      ++iters;
      jl = j;
      bool conv = true, dropped = false;
      for (int r = 0; r < R; ++r) {
        if (!live[r]) continue;
        if (res[r] > ctol[r]) {
          conv = false;
        } else if (drop) {
          if (!drop->conv_step[r] && res[r] <= tol) drop->conv_step[r] = iters;
          if (drop->enabled && flexible) {
            live[r] = 0;
            keep[r] = j + 1;
            dropped = true;
          }
        }
      }
      if (conv) break;
      if (dropped) {
        act.clear();
        for (int r = 0; r < R; ++r)
          if (live[r]) act.push_back(r);
        GMG_CUDA(cudaMemcpyAsync(drop->idx, act.data(), sizeof(int) * act.size(), cudaMemcpyHostToDevice, s));
      }
    }
    if (jl < 0) break;
    // y = H^{-1} g per RHS, x += sum_j y_j Z_j
    const int n = jl + 1;
    std::vector<zc> y((size_t)n * R);
    for (int r = 0; r < R; ++r) {
      const zc* Hr = &H[(size_t)r * (m + 1) * m];
      const zc* gr = &g[(size_t)r * (m + 1)];
      // a dropped column uses the steps it kept; its later coefficients are zero
      const int nr = live[r] ? n : keep[r];
      for (int i = n - 1; i >= nr; --i) y[(size_t)i * R + r] = zc(0);
      if (dcgs) {
        if (nr > 0) hess_lsq(Hr, m, nr, beta0[r], &y[r], R);
        continue;
      }
      for (int i = nr - 1; i >= 0; --i) {
        zc acc = gr[i];
        for (int k = i + 1; k < nr; ++k) acc -= Hr[i * m + k] * y[(size_t)k * R + r];
        y[(size_t)i * R + r] = Hr[i * m + i] != zc(0) ? acc / Hr[i * m + i] : zc(0);
      }
    }
    GMG_TRY(multiaxpy_h(h, y, flexible ? Z0 : V0, n, flexible ? zstride : vstride, x, s));
  }
  if (iters_out) *iters_out = iters;
  if (relres) *relres = res;
  return GMG_OK;
}

Krylov level_krylov(MGLevel& L) {
  Krylov K;
  K.V0 = L.V0;
  K.Z0 = L.Z0;
  K.w = L.kw;
  K.t = L.kt;
  K.tz = L.kt;
  return K;
}

// ------------------------------------------------------------- K-cycle
gmg_status kcycle(gmg_mg* h, int l, const Vec& in, Vec& out, cudaStream_t s, cudaGraphExec_t graph = nullptr);

gmg_status coarse_solve(gmg_mg* h, int lc, const Vec& b, Vec& x, cudaStream_t s) {
  MGLevel& C = *h->L[lc];
  const bool coarsest = lc == (int)h->L.size() - 1;
  const gmg_mg_params& P = h->P;
  GMG_TRY(zero(x, s));
  Krylov K = level_krylov(C);
  if (coarsest) {
    auto none = [](const Vec&, Vec&, const Vec&) { return GMG_OK; };
    return fgmres(h, lc, b, x, K, C.m, P.coarsest_iters, P.coarsest_tol, none, false, nullptr, nullptr, s);
  }
  auto pc = [h, lc, s](const Vec& in, Vec& out, const Vec&) { return kcycle(h, lc, in, out, s); };
  return fgmres(h, lc, b, x, K, C.m, P.wrapper_iters, P.wrapper_tol, pc, true, nullptr, nullptr, s);
}

// graph: the captured coarse-level solve of level l + 1 for in.R RHS (l = 0
// only), launched in place of the host-driven one
gmg_status kcycle(gmg_mg* h, int l, const Vec& in, Vec& out, cudaStream_t s, cudaGraphExec_t graph) {
  MGLevel& L = *h->L[l];
  MGLevel& C = *h->L[l + 1];
  const int R = in.R;
  Vec bc = C.bc.with_rhs(R), xc = C.xc.with_rhs(R);
  // the BF16 form restricts and prolongs on the tensor cores (BF16 hi + lo
  // operands, FP32 accumulation: about FP32 accuracy)
  const gmg_prec tc = (h->P.prec == GMG_BF16 && in.prec == GMG_F32 && L.dof % 2 == 0 && C.dof <= 64)
                          ? GMG_BF16
                          : (gmg_prec)in.prec;
  GMG_TRY(gmg_agg_project(L.agg, tc, (gmg_prec)in.prec, R, in.p, bc.p, (gmg_stream)s));
  if (graph)
    GMG_CUDA(cudaGraphLaunch(graph, s));
  else
    GMG_TRY(coarse_solve(h, l + 1, bc, xc, s));
  GMG_TRY(gmg_agg_promote(L.agg, tc, (gmg_prec)in.prec, R, xc.p, out.p, (gmg_stream)s));
  return mr_smooth(h, l, in, out, h->P.smoother_iters, s);
}

// ------------------------------------------------------------- captured K-cycle
// The coarse-level solvers of a K-cycle captured as a CUDA graph.  The
// Hessenberg column, the Givens rotations and the convergence test of every
// RHS run in small device kernels (one thread per RHS) instead of on the host;
// every Arnoldi step and every restart cycle is a conditional IF node, switched
// on by the kernel that ends the step before it (or starts the cycle) while the
// tolerance and the iteration limit are not met, so a replay takes the same
// early exits as the host-driven solver.  The step index is fixed in each
// captured body, so the existing vector kernels are captured unchanged.

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double zabs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double2 zdiv(double2 a, double2 b) {
  const double d = zabs2(b);
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}

// start of a restart cycle: g = |r0| e_0, residual estimates, step counter 0;
// the first step runs while some RHS is above tol and iterations remain
__global__ void cycle_init_kernel(const double2* __restrict__ beta2, const double2* __restrict__ bn2, int R, int m,
                                  double2* __restrict__ g, double* __restrict__ res, double tol, int* __restrict__ ctr,
                                  int maxit, cudaGraphConditionalHandle first_step) {
  const int r = threadIdx.x;
  int ok = 1;
  if (r < R) {
    const double beta = sqrt(fmax(beta2[r].x, 0.0)), bn = sqrt(fmax(bn2[r].x, 1e-300));
    double2* gr = g + (size_t)r * (m + 1);
    gr[0] = make_double2(beta, 0.0);
    for (int k = 1; k <= m; ++k) gr[k] = make_double2(0.0, 0.0);
    res[r] = beta / bn;
    ok = res[r] <= tol;
  }
  const int conv = __syncthreads_and(ok);
  if (r == 0) {
    ctr[1] = 0;
    cudaGraphSetConditional(first_step, (!conv && ctr[0] < maxit) ? 1u : 0u);
  }
}

// end of Arnoldi step j: Hessenberg column j = the two Gram-Schmidt passes'
// coefficients and |w|, previous rotations, a new rotation, the residual
// estimate; the next step runs while some RHS is above tol and iterations remain
__global__ void arnoldi_step_kernel(const double2* __restrict__ dh, const double2* __restrict__ dh2,
                                    const double2* __restrict__ dw, int j, int m, int R, double2* __restrict__ H,
                                    double2* __restrict__ g, double2* __restrict__ cs, double2* __restrict__ sn,
                                    double* __restrict__ res, const double2* __restrict__ bn2, double tol,
                                    int* __restrict__ ctr, int maxit, cudaGraphConditionalHandle next_step,
                                    int has_next) {
  const int r = threadIdx.x;
  int ok = 1;
  if (r < R) {
    double2* Hr = H + (size_t)r * (m + 1) * m;
    for (int i = 0; i <= j; ++i) Hr[i * m + j] = zadd(dh[(size_t)i * R + r], dh2[(size_t)i * R + r]);
    Hr[(j + 1) * m + j] = make_double2(sqrt(fmax(dw[r].x, 0.0)), 0.0);
    for (int i = 0; i < j; ++i) {
      const double2 c = cs[r * m + i], sg = sn[r * m + i];
      const double2 a = Hr[i * m + j], bq = Hr[(i + 1) * m + j];
      Hr[i * m + j] = zadd(zmul(zconj(c), a), zmul(zconj(sg), bq));
      Hr[(i + 1) * m + j] = zsub(zmul(c, bq), zmul(sg, a));
    }
    const double2 a = Hr[j * m + j], hn = Hr[(j + 1) * m + j];
    const double den = sqrt(zabs2(a) + zabs2(hn));
    double2 c = make_double2(1.0, 0.0), sg = make_double2(0.0, 0.0);
    if (den > 0.0) {
      c = make_double2(a.x / den, a.y / den);
      sg = make_double2(hn.x / den, hn.y / den);
    }
    cs[r * m + j] = c;
    sn[r * m + j] = sg;
    Hr[j * m + j] = zadd(zmul(zconj(c), a), zmul(zconj(sg), hn));
    Hr[(j + 1) * m + j] = make_double2(0.0, 0.0);
    double2* gr = g + (size_t)r * (m + 1);
    const double2 gj = gr[j];
    gr[j] = zmul(zconj(c), gj);
    gr[j + 1] = make_double2(-(sg.x * gj.x - sg.y * gj.y), -(sg.x * gj.y + sg.y * gj.x));
    res[r] = sqrt(zabs2(gr[j + 1])) / sqrt(fmax(bn2[r].x, 1e-300));
    ok = res[r] <= tol;
  }
  const int conv = __syncthreads_and(ok);
  if (r == 0) {
    ctr[0] += 1;
    ctr[1] = j + 1;
    if (has_next) cudaGraphSetConditional(next_step, (!conv && ctr[0] < maxit) ? 1u : 0u);
  }
}

// end of a restart cycle: y = H^-1 g over the steps taken (zero beyond), and
// the next cycle runs when this one took a step and iterations remain (it
// starts from the true residual, as the host-driven solver does)
__global__ void cycle_finish_kernel(const double2* __restrict__ H, const double2* __restrict__ g, int R, int m,
                                    const int* __restrict__ ctr, int maxit, double2* __restrict__ y,
                                    cudaGraphConditionalHandle next_cycle, int has_next) {
  const int r = threadIdx.x;
  const int n = ctr[1];
  if (r < R) {
    const double2* Hr = H + (size_t)r * (m + 1) * m;
    const double2* gr = g + (size_t)r * (m + 1);
    for (int i = n - 1; i >= 0; --i) {
      double2 acc = gr[i];
      for (int k = i + 1; k < n; ++k) acc = zsub(acc, zmul(Hr[i * m + k], y[(size_t)k * R + r]));
      const double2 d = Hr[i * m + i];
      y[(size_t)i * R + r] = (d.x != 0.0 || d.y != 0.0) ? zdiv(acc, d) : make_double2(0.0, 0.0);
    }
    for (int i = n; i < m; ++i) y[(size_t)i * R + r] = make_double2(0.0, 0.0);
  }
  if (r == 0 && has_next) cudaGraphSetConditional(next_cycle, (n > 0 && ctr[0] < maxit) ? 1u : 0u);
}

// a conditional handle of the graph that stream s is capturing
gmg_status cap_handle(cudaStream_t s, cudaGraphConditionalHandle* hnd) {
  cudaStreamCaptureStatus st;
  cudaGraph_t g = nullptr;
  GMG_CUDA(cudaStreamGetCaptureInfo(s, &st, nullptr, &g, nullptr, nullptr));
  GMG_CHECK(st == cudaStreamCaptureStatusActive, GMG_ERR_STATE, "mg graph: stream is not capturing");
  GMG_CUDA(cudaGraphConditionalHandleCreate(hnd, g, 0, cudaGraphCondAssignDefault));
  return GMG_OK;
}

// an IF node on hnd at the capture point of s; its body is captured on body_s
gmg_status cap_if_begin(cudaStream_t s, cudaGraphConditionalHandle hnd, cudaStream_t body_s) {
  cudaStreamCaptureStatus st;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  GMG_CUDA(cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, &nd));
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = hnd;
  p.conditional.type = cudaGraphCondTypeIf;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  GMG_CUDA(cudaGraphAddNode(&node, g, deps, nd, &p));
  GMG_CUDA(cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies));
  GMG_CUDA(cudaStreamBeginCaptureToGraph(body_s, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal));
  return GMG_OK;
}

gmg_status cap_if_end(cudaStream_t body_s) {
  cudaGraph_t g = nullptr;
  GMG_CUDA(cudaStreamEndCapture(body_s, &g));
  return GMG_OK;
}

// the restarted (F)GMRES of level l inside a captured K-cycle, on the capture
// stream of nesting depth d; prec(in, out, tz, depth) captures the preconditioner
template <class Prec>
gmg_status fgmres_cap(gmg_mg* h, int l, const Vec& b, Vec& x, const Krylov& K, int m, int maxit, double tol,
                      Prec prec, bool flexible, int d) {
  MGLevel& L = *h->L[l];
  GMG_CHECK(d + 2 < 8, GMG_ERR_UNSUPPORTED, "mg graph: solvers nested too deep");
  cudaStream_t s = h->cap_st[d];
  const int R = b.R;
  Vec V0 = K.V0.with_rhs(R), Z0 = K.Z0.with_rhs(R), w = K.w.with_rhs(R), t = K.t.with_rhs(R), tz = K.tz.with_rhs(R);
  const int64_t vstride = V0.elems(), zstride = Z0.elems();
  double2* bn2 = L.gBn.as<double2>();
  double2* beta2 = L.gBeta.as<double2>();
  int* ctr = L.gCtr.as<int>();
  double2 *H = L.gH.as<double2>(), *G = L.gG.as<double2>(), *CS = L.gCs.as<double2>(), *SN = L.gSn.as<double2>();
  double2* Y = L.gY.as<double2>();
  double* RES = L.gRes.as<double>();
  const int threads = (R + 31) / 32 * 32;
  // every step's vector work in one kernel per step where the level's vectors allow
  const bool fused = V0.prec == w.prec && b.prec == w.prec && x.prec == w.prec && rhs_fused(w, m) && rhs_fused(b, m);
  RhsGivens gv{H, G, CS, SN, RES, bn2, ctr, tol, m, maxit, 0, 0};
  if (!fused) {
    GMG_TRY(vec_multidot(b, 1, 0, b, bn2, nullptr, s));
    GMG_CUDA(cudaMemsetAsync(ctr, 0, 2 * sizeof(int), s));
  }
  const int ncyc = std::max(1, (maxit + m - 1) / m);
  std::vector<cudaGraphConditionalHandle> hcyc(ncyc, 0);
  for (int c = 1; c < ncyc; ++c) GMG_TRY(cap_handle(s, &hcyc[c]));
  for (int c = 0; c < ncyc; ++c) {
    cudaStream_t sc = s;
    int dc = d;
    if (c > 0) {
      GMG_TRY(cap_if_begin(s, hcyc[c], h->cap_st[d + 1]));
      sc = h->cap_st[d + 1];
      dc = d + 1;
    }
    // r0 = b - A x, |r0|, v_0
    Vec v0 = nth(V0, 0);
    GMG_TRY(apply_op(h, l, x, w, sc));
    std::vector<cudaGraphConditionalHandle> hit(m, 0);
    for (int j = 0; j < m; ++j) GMG_TRY(cap_handle(sc, &hit[j]));
    gv.next = hit[0];
    if (fused) {
      GMG_TRY(rhs_cycle_start(b, w, v0, c == 0, bn2, gv, sc));
    } else {
      GMG_TRY(vec_xmy(b, w, sc));
      GMG_TRY(vec_multidot(w, 1, 0, w, beta2, nullptr, sc));
      cycle_init_kernel<<<1, threads, 0, sc>>>(beta2, bn2, R, m, G, RES, tol, ctr, maxit, hit[0]);
      GMG_CUDA(cudaGetLastError());
      GMG_TRY(vec_scale_inv_norm(beta2, w, v0, sc));
    }
    for (int j = 0; j < m; ++j) {
      cudaStream_t si = h->cap_st[dc + 1];
      GMG_TRY(cap_if_begin(sc, hit[j], si));
      Vec vj = nth(V0, j);
      Vec zj = flexible ? nth(Z0, j) : vj;
      if (flexible) GMG_TRY(prec(vj, zj, tz, dc + 1));
      if (zj.prec != w.prec) {
        GMG_TRY(vec_convert(zj, t, si));
        GMG_TRY(apply_op(h, l, t, w, si));
      } else {
        GMG_TRY(apply_op(h, l, zj, w, si));
      }
      const size_t nc = (size_t)(j + 1) * R;
      double2* dh = h->dscr.as<double2>();
      double2* dh2 = dh + nc;
      double2* dw = dh2 + nc;
      Vec vn = nth(V0, j + 1);
      if (fused) {
        gv.has_next = j + 1 < m;
        gv.next = j + 1 < m ? hit[j + 1] : hit[j];
        GMG_TRY(rhs_gs_step(V0, vstride, j + 1, w, vn, dh, dh2, dw, gv, si));
        GMG_TRY(cap_if_end(si));
        continue;
      }
      GMG_TRY(vec_multidot(V0, j + 1, vstride, w, dh, nullptr, si));
      GMG_TRY(vec_multiaxpy_dot(dh, V0, j + 1, vstride, w, si, -1.0, dh2, 1));
      GMG_TRY(vec_multiaxpy_dot(dh2, V0, j + 1, vstride, w, si, -1.0, dw, 2));
      GMG_TRY(vec_scale_inv_norm(dw, w, vn, si));
      arnoldi_step_kernel<<<1, threads, 0, si>>>(dh, dh2, dw, j, m, R, H, G, CS, SN, RES, bn2, tol, ctr, maxit,
                                                 j + 1 < m ? hit[j + 1] : hit[j], j + 1 < m ? 1 : 0);
      GMG_CUDA(cudaGetLastError());
      GMG_TRY(cap_if_end(si));
    }
    gv.has_next = c + 1 < ncyc;
    gv.next = c + 1 < ncyc ? hcyc[c + 1] : hit[0];
    if (fused && (!flexible || Z0.prec == x.prec)) {
      GMG_TRY(rhs_cycle_finish(flexible ? Z0 : V0, flexible ? zstride : vstride, x, gv, sc));
    } else {
      cycle_finish_kernel<<<1, threads, 0, sc>>>(H, G, R, m, ctr, maxit, Y, gv.next, gv.has_next);
      GMG_CUDA(cudaGetLastError());
      GMG_TRY(vec_multiaxpy(Y, flexible ? Z0 : V0, m, flexible ? zstride : vstride, x, sc, 1.0));
    }
    if (c > 0) GMG_TRY(cap_if_end(sc));
  }
  return GMG_OK;
}

gmg_status kcycle_cap(gmg_mg* h, int l, const Vec& in, Vec& out, int d);

gmg_status coarse_solve_cap(gmg_mg* h, int lc, const Vec& b, Vec& x, int d) {
  MGLevel& C = *h->L[lc];
  const bool coarsest = lc == (int)h->L.size() - 1;
  const gmg_mg_params& P = h->P;
  GMG_TRY(zero(x, h->cap_st[d]));
  Krylov K = level_krylov(C);
  if (coarsest) {
    auto none = [](const Vec&, Vec&, const Vec&, int) { return GMG_OK; };
    return fgmres_cap(h, lc, b, x, K, C.m, P.coarsest_iters, P.coarsest_tol, none, false, d);
  }
  auto pc = [h, lc](const Vec& in, Vec& out, const Vec&, int dd) { return kcycle_cap(h, lc, in, out, dd); };
  return fgmres_cap(h, lc, b, x, K, C.m, P.wrapper_iters, P.wrapper_tol, pc, true, d);
}

// kcycle() on the capture stream of depth d
gmg_status kcycle_cap(gmg_mg* h, int l, const Vec& in, Vec& out, int d) {
  MGLevel& L = *h->L[l];
  MGLevel& C = *h->L[l + 1];
  cudaStream_t s = h->cap_st[d];
  const int R = in.R;
  Vec bc = C.bc.with_rhs(R), xc = C.xc.with_rhs(R);
  const gmg_prec tc = (h->P.prec == GMG_BF16 && in.prec == GMG_F32 && L.dof % 2 == 0 && C.dof <= 64)
                          ? GMG_BF16
                          : (gmg_prec)in.prec;
  GMG_TRY(gmg_agg_project(L.agg, tc, (gmg_prec)in.prec, R, in.p, bc.p, (gmg_stream)s));
  GMG_TRY(coarse_solve_cap(h, l + 1, bc, xc, d));
  GMG_TRY(gmg_agg_promote(L.agg, tc, (gmg_prec)in.prec, R, xc.p, out.p, (gmg_stream)s));
  return mr_smooth(h, l, in, out, h->P.smoother_iters, s);
}

// device state of the coarse-level solvers for max_rhs RHS (allocated before any capture),
// cleared on the solve's stream: the legacy default stream, which other streams need not
// wait for, could clear it in the middle of a captured cycle
gmg_status graph_state(gmg_mg* h, cudaStream_t s) {
  const int R = h->Rmax;
  for (size_t l = 1; l < h->L.size(); ++l) {
    MGLevel& L = *h->L[l];
    const int m = L.m;
    if (L.gH.p) continue;
    GMG_TRY(L.gH.alloc(sizeof(double2) * (size_t)R * (m + 1) * m));
    GMG_TRY(L.gG.alloc(sizeof(double2) * (size_t)R * (m + 1)));
    GMG_TRY(L.gCs.alloc(sizeof(double2) * (size_t)R * m));
    GMG_TRY(L.gSn.alloc(sizeof(double2) * (size_t)R * m));
    GMG_TRY(L.gRes.alloc(sizeof(double) * (size_t)R));
    GMG_TRY(L.gY.alloc(sizeof(double2) * (size_t)R * m));
    GMG_TRY(L.gCtr.alloc(sizeof(int) * 4));
    GMG_CUDA(cudaMemsetAsync(L.gCtr.p, 0, sizeof(int) * 4, s));
    GMG_TRY(L.gBn.alloc(sizeof(double2) * (size_t)R));
    GMG_TRY(L.gBeta.alloc(sizeof(double2) * (size_t)R));
    // the captured cycle combines all m Krylov / flexible directions with
    // zero coefficients beyond the steps taken: keep them finite
    GMG_CUDA(cudaMemsetAsync(L.V0.p, 0, L.V0.buf.bytes, s));
    if (L.Z0.p) GMG_CUDA(cudaMemsetAsync(L.Z0.p, 0, L.Z0.buf.bytes, s));
  }
  for (auto& st : h->cap_st)
    if (!st) GMG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  return GMG_OK;
}

// capture the coarse-level solve of kcycle(0) for R RHS: level 1's K-cycle
// FGMRES and everything below it, on level 1's fixed right-hand-side and
// solution buffers.  The fine-level steps (restriction, prolongation, MR
// smoothing: a few large kernels) stay plain launches on the caller's vectors,
// so the Krylov vectors need no copies in and out of fixed buffers.
gmg_status build_kcycle_graph(gmg_mg* h, int R, cudaGraphExec_t* exec, cudaStream_t s) {
  *exec = nullptr;
  GMG_TRY(graph_state(h, s));
  cudaStream_t s0 = h->cap_st[0];
  MGLevel& C = *h->L[1];
  Vec bc = C.bc.with_rhs(R), xc = C.xc.with_rhs(R);
  GMG_CUDA(cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal));
  gmg_status st = coarse_solve_cap(h, 1, bc, xc, 0);
  cudaGraph_t g = nullptr;
  // end every capture still open (an error inside a body leaves it open)
  for (int d = 7; d >= 1; --d) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (h->cap_st[d] && cudaStreamIsCapturing(h->cap_st[d], &cs) == cudaSuccess &&
        cs != cudaStreamCaptureStatusNone) {
      cudaGraph_t gb = nullptr;
      cudaStreamEndCapture(h->cap_st[d], &gb);
    }
  }
  const cudaError_t e = cudaStreamEndCapture(s0, &g);
  if (st != GMG_OK) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    return st;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(GMG_ERR_CUDA, std::string("mg graph: capture failed: ") + cudaGetErrorString(e));
  }
  const cudaError_t ei = cudaGraphInstantiate(exec, g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess) {
    cudaGetLastError();
    *exec = nullptr;
    return fail(GMG_ERR_CUDA, std::string("mg graph: instantiation failed: ") + cudaGetErrorString(ei));
  }
  return GMG_OK;
}

// ------------------------------------------------------------- setup
// `count` consecutive fields of [V][R][dof] in one buffer; the Vec describes the first
gmg_status alloc_fields(VecBuf& b, int64_t V, int R, int dof, int prec, int count) {
  b.V = V;
  b.R = R;
  b.dof = dof;
  b.prec = prec;
  GMG_TRY(b.buf.alloc((size_t)count * b.bytes()));
  b.p = b.buf.p;
  return GMG_OK;
}

// Level workspaces: MR smoother on every level; Krylov basis for the solver
// that runs on a coarse level (flexible directions only where a K-cycle
// preconditions it); right-hand side / solution of the cycle above.
gmg_status alloc_level_ws(MGLevel& L, int R, bool krylov, bool flexible) {
  const int p = L.vprec;
  if (krylov) {
    GMG_TRY(alloc_fields(L.V0, L.V, R, L.dof, p, L.m + 1));
    if (flexible) GMG_TRY(alloc_fields(L.Z0, L.V, R, L.dof, p, L.m));
    GMG_TRY(L.kw.alloc(L.V, R, L.dof, p));
    GMG_TRY(L.kt.alloc(L.V, R, L.dof, p));
  }
  GMG_TRY(alloc_fields(L.mr_r, L.V, R, L.dof, p, 2));
  if (L.l == 0 && L.bf16_smoother) {
    GMG_TRY(alloc_fields(L.mr_r16, L.V, R, L.dof, GMG_BF16, L.mr_keep));
    GMG_TRY(L.mr_Ar16.alloc(L.V, R, L.dof, GMG_BF16));
  }
  if (L.l > 0) {
    GMG_TRY(L.bc.alloc(L.V, R, L.dof, p));
    GMG_TRY(L.xc.alloc(L.V, R, L.dof, p));
  }
  return GMG_OK;
}

// Outer FGMRES workspace for max_rhs right-hand sides (m + 1 Krylov vectors
// in the Arnoldi precision, m flexible directions in the preconditioner
// precision, the FP64 residuals, and the conversion / compacted-batch fields),
// allocated on first use and kept: a solve then allocates nothing.
gmg_status outer_workspace(gmg_mg* h) {
  if (h->outer_ready) return GMG_OK;
  MGLevel& F = *h->L[0];
  const int m = std::max(h->P.outer_restart, 2);
  const int zp = F.vprec, R = h->Rmax, vp = h->arn32 ? GMG_F32 : GMG_F64;
  const int64_t V = F.V;
  GMG_TRY(alloc_fields(h->oV0, V, R, 12, vp, m + 1));
  GMG_TRY(alloc_fields(h->oZ0, V, R, 12, zp, m));
  GMG_TRY(h->ow.alloc(V, R, 12, vp));
  GMG_TRY(h->ot64.alloc(V, R, 12, GMG_F64));
  if (vp != GMG_F64) GMG_TRY(h->otv.alloc(V, R, 12, vp));
  GMG_TRY(h->orr.alloc(V, R, 12, GMG_F64));
  GMG_TRY(h->orA.alloc(V, R, 12, GMG_F64));
  GMG_TRY(h->otz.alloc(V, R, 12, zp));
  GMG_TRY(h->obb.alloc(V, R, 12, GMG_F64));
  GMG_TRY(h->oxx.alloc(V, R, 12, GMG_F64));
  GMG_TRY(h->oidx.alloc(sizeof(int) * R));
  if (h->P.drop_in_cycle) {
    GMG_TRY(h->ozc.alloc(V, R, 12, zp));
    GMG_TRY(h->owc.alloc(V, R, 12, vp));
    GMG_TRY(h->oidx2.alloc(sizeof(int) * R));
  }
  h->outer_ready = true;
  return GMG_OK;
}

// Time the fine-operator kernel variants for the full batch once, at setup,
// so the first solve does not pay for it: FP64 M (outer residual and
// Arnoldi), and M with and without the fused MR products in the K-cycle
// precision.
gmg_status pretune_fine(gmg_mg* h, cudaStream_t s) {
  MGLevel& F = *h->L[0];
  const int R = h->Rmax, zp = F.vprec;
  GMG_CUDA(cudaMemsetAsync(h->orr.p, 0, h->orr.bytes(), s));
  GMG_CUDA(cudaMemsetAsync(h->otz.p, 0, h->otz.bytes(), s));
  GMG_TRY(gmg_wilson_apply(F.w, GMG_OP_M, 0, 0, GMG_F64, R, h->orr.p, h->ot64.p, (gmg_stream)s));
  if (zp != GMG_F64) {
    Vec z0 = nth(h->oZ0, 0);
    GMG_TRY(gmg_wilson_apply(F.w, GMG_OP_M, 0, 0, (gmg_prec)zp, R, h->otz.p, z0.p, (gmg_stream)s));
  }
  if (h->P.smoother_iters > 0) {
    Vec z0 = nth(h->oZ0, 0);
    double2* d1 = h->dscr.as<double2>() + kScalars / 2;
    GMG_TRY(wilson_apply_mr(F.w, zp, R, zp == GMG_F64 ? h->orr.p : h->otz.p, zp == GMG_F64 ? h->ot64.p : z0.p, d1,
                            d1 + R, s));
  }
  GMG_CUDA(cudaStreamSynchronize(s));
  return GMG_OK;
}

// recreateOperators of one transition (MultigridPreconditioner.h:458-477):
// chiral doubling of level l's test vectors into the 2 nvec basis, block
// orthonormalisation (Aggregation::Create), Galerkin coarsening into level
// l+1's operator and its reduced-precision copies.  The handles are created on
// first use and refilled afterwards, so their addresses stay valid.
gmg_status recreate_level(gmg_mg* h, int l, cudaStream_t s) {
  MGLevel& L = *h->L[l];
  MGLevel& C = *h->L[l + 1];
  const int nv = h->P.nvec[l];
  const gmg_stream stream = (gmg_stream)s;
  DevBuf basis;
  GMG_TRY(basis.alloc(sizeof(double2) * 2 * (size_t)nv * L.V * L.dof));
  GMG_TRY(vec_chiral_double(L.tv, basis.as<double>(), s));
  if (!L.agg) GMG_TRY(gmg_agg_create(L.dims.d, C.dims.d, L.dof, 2 * nv, &L.agg));
  GMG_TRY(gmg_agg_set_basis(L.agg, basis.as<double>(), 1, stream));
  GMG_TRY(gmg_agg_orthonormalise(L.agg, 2, stream));
  GMG_CUDA(cudaStreamSynchronize(s));
  if (!C.c) GMG_TRY(gmg_coarse_create(C.dims.d, 2 * nv, 0, &C.c));
  if (l == 0) GMG_TRY(gmg_coarsen_wilson(C.c, L.agg, L.w, stream));
  else GMG_TRY(gmg_coarsen_coarse(C.c, L.agg, L.c, stream));
  if (C.vprec == GMG_F32) GMG_TRY(gmg_coarse_prepare(C.c, GMG_F32, stream));
  if (C.compute == GMG_BF16) GMG_TRY(gmg_coarse_prepare(C.c, GMG_BF16, stream));
  GMG_CUDA(cudaStreamSynchronize(s));
  return GMG_OK;
}

// right-hand sides [s0, s0 + n) of src -> [d0, d0 + n) of dst (same sites,
// dof and precision; the RHS index is the middle one of [V][R][dof])
gmg_status copy_rhs(const Vec& src, int s0, const Vec& dst, int d0, int n, cudaStream_t s) {
  const size_t col = (size_t)src.dof * src.esize();
  GMG_CUDA(cudaMemcpy2DAsync(static_cast<char*>(dst.p) + d0 * col, dst.R * col,
                             static_cast<const char*>(src.p) + s0 * col, src.R * col, n * col, (size_t)src.V,
                             cudaMemcpyDeviceToDevice, s));
  return GMG_OK;
}

void drop_graphs(gmg_mg* h) {
  for (auto& g : h->kgraph) cudaGraphExecDestroy(g.second);
  h->kgraph.clear();
  h->graph_broken = false;
}

}  // namespace
}  // namespace gmg

using namespace gmg;

extern "C" gmg_status gmg_mg_params_default(gmg_mg_params* p) {
  GMG_CHECK(p != nullptr, GMG_ERR_ARGUMENT, "gmg_mg_params_default: null");
  memset(p, 0, sizeof(*p));
  p->nlevels = 3;
  for (int d = 0; d < 4; ++d) {
    p->block[0][d] = 4;
    p->block[1][d] = 2;
  }
  p->nvec[0] = 12;
  p->nvec[1] = 16;
  p->setup_iters = 100;
  p->smoother_iters = 8;
  p->wrapper_iters = 10;
  p->wrapper_tol = 0.1;
  p->coarsest_iters = 50;
  p->coarsest_tol = 0.05;
  p->coarsest_restart = 10;
  p->outer_restart = 8;
  p->prec = GMG_F32;
  p->seed = 1234;
  p->setup_solver = 0;
  p->setup_tol = 1e-3;
  // Null-vector setup (setupBasisVectorsType nullVectors) rather than the
  // reference's default single test-vector pass: on 32^4 near the critical mass
  // one pass of A psi = v leaves the test vectors dominated by bulk modes (the
  // coarse operator's lowest eigenvalue stayed near 1.9 against 0.04 for the
  // fine operator, and the K-cycle cut the outer iterations by nothing), while
  // 100 BiCGStab iterations on A psi = 0 keep the slowly decaying low modes
  // (28 outer iterations on that configuration).
  p->setup_passes = 1;
  p->setup_null = 1;
  p->graph = 1;
  p->refine_iters[0] = p->refine_iters[1] = 0;
  p->recursive_updates = 1;
  p->drop_in_cycle = 1;
  p->smoother_bf16 = -1;
  p->outer_dcgs = 1;
  p->arnoldi_f32 = -1;
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_create(gmg_wilson* fine, const gmg_mg_params* p, int max_rhs, gmg_mg** out) {
  GMG_CHECK(fine && p && out, GMG_ERR_ARGUMENT, "gmg_mg_create: null argument");
  *out = nullptr;
  GMG_CHECK(p->nlevels >= 2 && p->nlevels <= 3, GMG_ERR_ARGUMENT, "gmg_mg_create: nlevels must be 2 or 3");
  GMG_CHECK(max_rhs >= 1 && max_rhs <= 64, GMG_ERR_ARGUMENT, "gmg_mg_create: max_rhs must be in [1, 64]");
  GMG_CHECK(p->prec == GMG_F64 || p->prec == GMG_F32 || p->prec == GMG_BF16, GMG_ERR_ARGUMENT,
            "gmg_mg_create: prec must be F64, F32 or BF16");
  gmg_mg* h = new gmg_mg();
  h->P = *p;
  h->fine = fine;
  h->Rmax = max_rhs;
  h->arn32 = p->arnoldi_f32 > 0 || (p->arnoldi_f32 < 0 && p->prec != GMG_F64);
  Dims d = fine->dims;
  int dof = 12;
  for (int l = 0; l < p->nlevels; ++l) {
    MGLevel* L = new MGLevel();
    L->l = l;
    L->dims = d;
    L->V = d.vol();
    L->dof = dof;
    L->vprec = p->prec == GMG_F64 ? GMG_F64 : GMG_F32;
    L->compute = p->prec == GMG_BF16 && l > 0 ? GMG_BF16 : L->vprec;
    L->bf16_smoother = l == 0 && L->vprec == GMG_F32 &&
                       (p->smoother_bf16 > 0 || (p->smoother_bf16 < 0 && p->prec == GMG_BF16));
    // the sweep that keeps every step's residual (site-blocked fields, whose
    // operator indexes them with 32-bit offsets in 16-byte units)
    if (L->bf16_smoother && p->smoother_iters >= 1 && p->smoother_iters <= kMrMaxSteps &&
        2 * (int64_t)max_rhs * p->smoother_iters <= kScalars / 2 && L->V * 3 * max_rhs < ((int64_t)1 << 31))
      L->mr_keep = p->smoother_iters;
    L->w = l == 0 ? fine : nullptr;
    h->L.push_back(L);
    if (l + 1 < p->nlevels) {
      for (int k = 0; k < 4; ++k) {
        const int b = p->block[l][k];
        if (b <= 0 || d.d[k] % b != 0) {
          delete h;
          return fail(GMG_ERR_SHAPE, "gmg_mg_create: block size does not divide the lattice");
        }
        d.d[k] /= b;
      }
      dof = 2 * p->nvec[l];
    }
  }
  gmg_status st = h->coef.alloc(sizeof(double2) * kScalars);
  if (st == GMG_OK) st = h->dscr.alloc(sizeof(double2) * kScalars);
  if (st == GMG_OK && cudaMallocHost(&h->hpin, sizeof(double2) * kScalars) != cudaSuccess)
    st = fail(GMG_ERR_NOMEM, "gmg_mg_create: pinned host buffer");
  if (st != GMG_OK) {
    delete h;
    return st;
  }
  *out = h;
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_destroy(gmg_mg* h) {
  if (h) {
    cudaDeviceSynchronize();
    delete h;
  }
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_setup(gmg_mg* h, gmg_stream stream) {
  GMG_CHECK(h != nullptr, GMG_ERR_ARGUMENT, "gmg_mg_setup: null handle");
  GMG_CHECK(h->fine->gauge_set, GMG_ERR_STATE, "gmg_mg_setup: gauge field not set");
  cudaStream_t s = S(stream);
  const gmg_mg_params& P = h->P;
  const int nl = (int)h->L.size();
  h->setup_done = false;
  // captured cycles refer to the operators and buffers a new setup replaces
  drop_graphs(h);
  for (int l = 0; l < nl; ++l) {
    MGLevel& L = *h->L[l];
    const bool coarsest = l == nl - 1;
    L.m = l == 0 ? 0 : (coarsest ? std::max(P.coarsest_restart, 2) : std::max(P.wrapper_iters, 2));
  }
  GMG_TRY(alloc_level_ws(*h->L[0], h->Rmax, false, false));
  for (int l = 0; l + 1 < nl; ++l) {
    MGLevel& L = *h->L[l];
    MGLevel& C = *h->L[l + 1];
    const int nv = P.nvec[l];
    // test vectors (BasisVectors::Generate, BasisVectors.h:74-147): random start,
    // then setup_passes passes of {orthonormalise, solve, orthonormalise}; the
    // test-vector form solves A psi = v from psi = 0 (inverse iteration), the
    // null-vector form solves A psi = 0 from psi = v (the slowly decaying low
    // modes remain)
    VecBuf v, zsrc;
    VecBuf& psi = L.tv;  // kept for the refinement setup
    GMG_TRY(v.alloc(L.V, nv, L.dof, L.vprec));
    GMG_TRY(psi.alloc(L.V, nv, L.dof, L.vprec));
    GMG_TRY(vec_gaussian(v, P.seed * 7919 + l, s));
    if (P.setup_null) {
      GMG_TRY(zsrc.alloc(L.V, nv, L.dof, L.vprec));
      GMG_TRY(zero(zsrc, s));
    }
    const double stol = P.setup_tol > 0 ? P.setup_tol : 1e-3;
    const int passes = std::max(P.setup_passes, 1);
    VecBuf ws[6], sV, sw, st;
    for (int pass = 0; pass < passes; ++pass) {
      GMG_TRY(global_orthonormalise(h, v, s));  // setupPreOrthonormalise
      if (P.setup_null)
        GMG_CUDA(cudaMemcpyAsync(psi.p, v.p, v.bytes(), cudaMemcpyDeviceToDevice, s));
      else
        GMG_CUDA(cudaMemsetAsync(psi.p, 0, psi.bytes(), s));
      const Vec& src = P.setup_null ? static_cast<const Vec&>(zsrc) : static_cast<const Vec&>(v);
      if (P.setup_solver == 1) {
        const int ms = 10;
        if (!sV.p) {
          GMG_TRY(alloc_fields(sV, L.V, nv, L.dof, L.vprec, ms + 1));
          GMG_TRY(sw.alloc(L.V, nv, L.dof, L.vprec));
          GMG_TRY(st.alloc(L.V, nv, L.dof, L.vprec));
        }
        Krylov K;
        K.V0 = sV;
        K.w = sw;
        K.t = st;
        K.tz = st;
        auto none = [](const Vec&, Vec&, const Vec&) { return GMG_OK; };
        GMG_TRY(fgmres(h, l, src, psi, K, ms, P.setup_iters, stol, none, false, nullptr, nullptr, s));
      } else {
        if (!ws[0].p)
          for (auto& f : ws) GMG_TRY(f.alloc(L.V, nv, L.dof, L.vprec));
        GMG_TRY(bicgstab(h, l, src, psi, P.setup_iters, stol, ws, s));
      }
      GMG_TRY(global_orthonormalise(h, psi, s));  // setupPostOrthonormalise
      if (pass + 1 < passes) GMG_CUDA(cudaMemcpyAsync(v.p, psi.p, psi.bytes(), cudaMemcpyDeviceToDevice, s));
    }
    // chiral doubling -> basis, block orthonormalisation, Galerkin coarsening
    GMG_TRY(recreate_level(h, l, s));
    const bool coarsest = l + 1 == nl - 1;
    GMG_TRY(alloc_level_ws(C, h->Rmax, true, !coarsest));
    GMG_CUDA(cudaStreamSynchronize(s));
  }
  GMG_TRY(outer_workspace(h));
  GMG_TRY(pretune_fine(h, s));
  h->setup_done = true;
  return GMG_OK;
}

// refinementSetup (MultigridPreconditioner.h:213-251) with the test-vector
// form of BasisVectors::Generate (BasisVectors.h:74-147): the solver is the
// level's own preconditioner (OperatorFunctionWrapper over operator(),
// :253-309), applied from psi = 0 to each test vector; updateBasisVector
// (:479-501) and recreateOperators (:458-477) are the callbacks.  The
// reference applies the preconditioner to one vector at a time; the operators
// do not change within a pass, so the vectors go through the K-cycle as one
// multi-RHS batch (max_rhs at a time) with the same result per vector up to
// the batch's shared iteration count on the coarse levels.
extern "C" gmg_status gmg_mg_refine(gmg_mg* h, gmg_stream stream) {
  GMG_CHECK(h != nullptr, GMG_ERR_ARGUMENT, "gmg_mg_refine: null handle");
  GMG_CHECK(h->setup_done, GMG_ERR_STATE, "gmg_mg_refine: call gmg_mg_setup first");
  cudaStream_t s = S(stream);
  const gmg_mg_params& P = h->P;
  const int nl = (int)h->L.size();
  for (int l = 0; l + 1 < nl; ++l) {
    const int iters = P.refine_iters[l];
    // a level without refinement iterations does not recurse (:214, :246)
    if (iters <= 0) break;
    drop_graphs(h);
    MGLevel& L = *h->L[l];
    MGLevel& C = *h->L[l + 1];
    const int nv = P.nvec[l];
    const int Rc = std::min(nv, h->Rmax);
    VecBuf a, b;
    GMG_TRY(a.alloc(L.V, Rc, L.dof, L.vprec));
    GMG_TRY(b.alloc(L.V, Rc, L.dof, L.vprec));
    // updateBasisVector reaches level l+1's test vectors when that level has
    // an aggregation below it (the coarsest level keeps none, :653)
    const bool update_next = P.recursive_updates && l + 2 < nl;
    for (int it = 0; it < iters; ++it) {
      GMG_TRY(global_orthonormalise(h, L.tv, s));  // setupPreOrthonormalise
      for (int k0 = 0; k0 < nv; k0 += Rc) {
        const int n = std::min(Rc, nv - k0);
        Vec in = a.with_rhs(n), out = b.with_rhs(n);
        GMG_TRY(copy_rhs(L.tv, k0, in, 0, n, s));
        GMG_TRY(kcycle(h, l, in, out, s));  // psi = MG(v) from psi = 0
        GMG_TRY(copy_rhs(out, 0, L.tv, k0, n, s));
        // level l+1's vector k <- its solution inside this application (_FineSol)
        const int nu = update_next ? std::min(n, P.nvec[l + 1] - k0) : 0;
        if (nu > 0) GMG_TRY(copy_rhs(C.xc.with_rhs(n), 0, C.tv, k0, nu, s));
      }
      GMG_TRY(global_orthonormalise(h, L.tv, s));  // setupPostOrthonormalise
      // recreateOperators(setupRecursiveUpdates)
      for (int q = l; q + 1 < nl; ++q) {
        GMG_TRY(recreate_level(h, q, s));
        if (!P.recursive_updates) break;
      }
    }
  }
  GMG_CUDA(cudaStreamSynchronize(s));
  return GMG_OK;
}

// Outer FGMRES on the fine operator, preconditioned by the K-cycle in the
// preconditioner precision.  b, x: device FP64 [V][nrhs][12]; x holds the
// initial guess.  Every restart cycle starts from the FP64 residual b - A x
// (formed once per cycle, after the solution update) and runs its Arnoldi
// process in FP64 or, with params.arnoldi_f32, in FP32; the tolerance is
// checked on that FP64 residual.  At every restart the still-unconverged RHS
// are compacted into a contiguous batch, so converged ones drop out of all
// later work.
extern "C" gmg_status gmg_mg_solve(gmg_mg* h, int nrhs, const double* b, double* x, double tol, int maxiter,
                                   int* iters_out, double* max_relres, gmg_stream stream) {
  GMG_CHECK(h && b && x, GMG_ERR_ARGUMENT, "gmg_mg_solve: null argument");
  GMG_CHECK(h->setup_done, GMG_ERR_STATE, "gmg_mg_solve: call gmg_mg_setup first");
  GMG_CHECK(nrhs >= 1 && nrhs <= h->Rmax, GMG_ERR_ARGUMENT, "gmg_mg_solve: nrhs exceeds max_rhs");
  GMG_CHECK(tol > 0 && maxiter >= 1, GMG_ERR_ARGUMENT, "gmg_mg_solve: bad tolerance / iteration limit");
  cudaStream_t s = S(stream);
  MGLevel& F = *h->L[0];
  const int m = std::max(h->P.outer_restart, 2);
  const int zp = F.vprec;
  const int64_t V = F.V;
  GMG_TRY(outer_workspace(h));
  VecBuf &V0 = h->oV0, &Z0 = h->oZ0, &w = h->ow, &tz = h->otz, &bb = h->obb, &xx = h->oxx;
  VecBuf& tv = h->arn32 ? h->otv : h->ot64;  // the batch's Krylov-precision scratch
  DevBuf& idx = h->oidx;
  Vec Bfull, Xfull;
  Bfull.p = const_cast<double*>(b);
  Bfull.V = V;
  Bfull.R = nrhs;
  Bfull.dof = 12;
  Xfull = Bfull;
  Xfull.p = x;
  std::vector<int> active(nrhs);
  for (int r = 0; r < nrhs; ++r) active[r] = r;
  std::vector<double> relres(nrhs, 1.0);
  std::vector<int> conv_it(nrhs, 0);
  std::vector<int> batches;
  int total = 0;
  // per-RHS norms of b for the global convergence criterion
  std::vector<zc> bnz;
  GMG_TRY(dots(h, Bfull, 1, 0, Bfull, bnz, s));
  // FP64 residual of every RHS; each cycle starts from it and refreshes it
  Vec Rfull = h->orr.with_rhs(nrhs);
  GMG_TRY(fine_residual(h, Bfull, Xfull, Rfull, s));
  while (!active.empty() && total < maxiter) {
    const int Ra = (int)active.size();
    // every RHS still active (the active list is ascending): the batch is the
    // caller's fields themselves, with no gather or scatter
    const bool whole = Ra == nrhs;
    Vec bA = Bfull, xA = Xfull, rA = Rfull;
    if (!whole) {
      GMG_CUDA(cudaMemcpyAsync(idx.p, active.data(), sizeof(int) * Ra, cudaMemcpyHostToDevice, s));
      bA = bb.with_rhs(Ra);
      xA = xx.with_rhs(Ra);
      rA = h->orA.with_rhs(Ra);
      GMG_TRY(vec_gather(Bfull, idx.as<int>(), bA, s));
      GMG_TRY(vec_gather(Xfull, idx.as<int>(), xA, s));
      GMG_TRY(vec_gather(Rfull, idx.as<int>(), rA, s));
    }
    Krylov K;
    K.V0 = V0.with_rhs(Ra);
    K.Z0 = Z0.with_rhs(Ra);
    K.w = w.with_rhs(Ra);
    K.t = tv.with_rhs(Ra);
    K.tz = tz.with_rhs(Ra);
    auto pc = [h, s, &tz, zp](const Vec& in, Vec& out, const Vec&) -> gmg_status {
      // in: Krylov vector (FP64, or FP32 in an FP32 Arnoldi cycle); out: Z
      // direction in the preconditioner precision
      const int Rb = in.R;  // the active columns (fewer than the batch after an in-cycle drop)
      if (zp == GMG_F64) return kcycle(h, 0, in, out, s);
      Vec src = in;
      if (in.prec != zp) {  // an FP64 Arnoldi vector, converted for the FP32 cycle
        src = tz.with_rhs(Rb);
        GMG_TRY(vec_convert(in, src, s));
      }
      const bool graph = h->P.graph && !h->graph_broken && Rb <= 1024;
      if (!graph) return kcycle(h, 0, src, out, s);
      auto it = h->kgraph.find(Rb);
      if (it == h->kgraph.end()) {
        // first cycle of this batch size: host-driven (it also builds every
        // buffer and tuning key the cycle needs), then the coarse-level solve
        // is captured for the next ones
        GMG_TRY(kcycle(h, 0, src, out, s));
        GMG_CUDA(cudaStreamSynchronize(s));
        cudaGraphExec_t ex = nullptr;
        if (build_kcycle_graph(h, Rb, &ex, s) == GMG_OK)
          h->kgraph[Rb] = ex;
        else
          h->graph_broken = true;  // keep the host-driven cycle
        return GMG_OK;
      }
      return kcycle(h, 0, src, out, s, it->second);
    };
    int it = 0;
    std::vector<double> rr;
    DropCtx dc;
    dc.enabled = h->P.drop_in_cycle != 0;
    dc.dcgs = h->P.outer_dcgs != 0;
    if (dc.enabled) {
      dc.zc = h->ozc.with_rhs(Ra);
      dc.wc = h->owc.with_rhs(Ra);
      dc.idx = h->oidx2.as<int>();
    }
    dc.batches = &batches;
    dc.r0 = &rA;
    GMG_TRY(fgmres(h, 0, bA, xA, K, m, std::min(m, maxiter - total), tol, pc, true, &it, &rr, s, &dc));
    if (!whole) GMG_TRY(vec_scatter(xA, idx.as<int>(), Xfull, s));
    const int before = total;
    total += std::max(it, 1);
    // true residuals of the batch decide who stays active, and start the next cycle
    GMG_TRY(fine_residual(h, bA, xA, rA, s));
    std::vector<zc> rn;
    if (!whole) GMG_TRY(vec_scatter(rA, idx.as<int>(), Rfull, s));
    GMG_TRY(dots(h, rA, 1, 0, rA, rn, s));
    std::vector<int> still;
    for (int k = 0; k < Ra; ++k) {
      const int r = active[k];
      relres[r] = std::sqrt(std::max(rn[k].real(), 0.0) / std::max(bnz[r].real(), 1e-300));
      // the step at which its residual estimate met tol within this cycle, else the cycle's end
      conv_it[r] = dc.conv_step[k] ? before + dc.conv_step[k] : total;
      if (relres[r] > tol) still.push_back(r);
    }
    if (it == 0 && still.size() == active.size()) break;  // no progress possible
    active.swap(still);
  }
  GMG_CUDA(cudaStreamSynchronize(s));
  double mx = 0;
  for (double v : relres) mx = std::max(mx, v);
  if (iters_out) *iters_out = total;
  if (max_relres) *max_relres = mx;
  h->last_iters = conv_it;
  h->last_relres = relres;
  h->last_batches = batches;
  if (mx > tol) return fail(GMG_ERR_NOT_CONVERGED, "gmg_mg_solve: not converged within maxiter");
  return GMG_OK;
}

// MultiGridPreconditioner::operator() (include/MultigridPreconditioner.h:253):
// one K-cycle on device FP64 fields [V][nrhs][12], run host-driven in the
// preconditioner precision (in converted on entry, out on exit).
extern "C" gmg_status gmg_mg_apply(gmg_mg* h, int nrhs, const double* in, double* out, gmg_stream stream) {
  GMG_CHECK(h && in && out, GMG_ERR_ARGUMENT, "gmg_mg_apply: null argument");
  GMG_CHECK(in != out, GMG_ERR_ARGUMENT, "gmg_mg_apply: in and out must not alias");
  GMG_CHECK(h->setup_done, GMG_ERR_STATE, "gmg_mg_apply: call gmg_mg_setup first");
  GMG_CHECK(nrhs >= 1 && nrhs <= h->Rmax, GMG_ERR_ARGUMENT, "gmg_mg_apply: nrhs exceeds max_rhs");
  cudaStream_t s = S(stream);
  MGLevel& F = *h->L[0];
  GMG_TRY(outer_workspace(h));
  Vec In, Out;
  In.p = const_cast<double*>(in);
  In.V = F.V;
  In.R = nrhs;
  In.dof = 12;
  Out = In;
  Out.p = out;
  if (F.vprec == GMG_F64) {
    GMG_TRY(kcycle(h, 0, In, Out, s));
  } else {
    Vec tin = h->otz.with_rhs(nrhs), z = nth(h->oZ0, 0).with_rhs(nrhs);
    GMG_TRY(vec_convert(In, tin, s));
    GMG_TRY(kcycle(h, 0, tin, z, s));
    GMG_TRY(vec_convert(z, Out, s));
  }
  GMG_CUDA(cudaStreamSynchronize(s));
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_solve_batches(gmg_mg* h, int cap, int* sizes, int* n) {
  GMG_CHECK(h && n, GMG_ERR_ARGUMENT, "gmg_mg_solve_batches: null argument");
  *n = (int)h->last_batches.size();
  GMG_CHECK(cap >= 0 && (cap == 0 || sizes), GMG_ERR_ARGUMENT, "gmg_mg_solve_batches: bad capacity");
  for (int k = 0; k < std::min(cap, *n); ++k) sizes[k] = h->last_batches[k];
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_solve_stats(gmg_mg* h, int nrhs, int* iters, double* relres) {
  GMG_CHECK(h && iters && relres, GMG_ERR_ARGUMENT, "gmg_mg_solve_stats: null argument");
  GMG_CHECK(nrhs == (int)h->last_iters.size(), GMG_ERR_SHAPE,
            "gmg_mg_solve_stats: nrhs differs from the last solve's");
  for (int r = 0; r < nrhs; ++r) {
    iters[r] = h->last_iters[r];
    relres[r] = h->last_relres[r];
  }
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_graphs(gmg_mg* h, int* graphs, int* fell_back) {
  GMG_CHECK(h && graphs && fell_back, GMG_ERR_ARGUMENT, "gmg_mg_graphs: null argument");
  *graphs = (int)h->kgraph.size();
  *fell_back = h->graph_broken ? 1 : 0;
  return GMG_OK;
}

extern "C" gmg_status gmg_mg_level(gmg_mg* h, int level, gmg_coarse** op, gmg_agg** agg) {
  GMG_CHECK(h && level >= 0 && level < (int)h->L.size(), GMG_ERR_ARGUMENT, "gmg_mg_level: bad level");
  if (op) *op = h->L[level]->c;
  if (agg) *agg = h->L[level]->agg;
  return GMG_OK;
}
