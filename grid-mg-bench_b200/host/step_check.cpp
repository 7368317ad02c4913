// step_check.cpp -- the coarse-level solver steps (mg_fused.cu) against FP64 sums on the
// host, over the unit counts at which a thread's share or the cluster's size changes:
//   Gram-Schmidt step   h1, h2, |w''|^2, v and the Givens update of its column
//   MR step             x += a r, r -= a Ar, a = <Ar, r> / <Ar, Ar>
//   cycle start / end   in a captured graph whose IF node holds a Gram-Schmidt step
// Sums of FP32 fields are formed in FP64 (1e-11 of the product of the norms); what is
// rounded to FP32 on the way agrees to 1e-6 of the vector's size per element or sum.
// Prints one line per failed check and exits non-zero if there is one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "mg_internal.cuh"

using namespace gmg;
typedef std::complex<double> zc;
typedef std::complex<float> cf;

static int failures = 0;
static void check(bool ok, const char* what, int64_t units, int R, int nx, double dev) {
  if (ok) return;
  ++failures;
  std::printf("FAILED %s: units %lld, R %d, nx %d: %g\n", what, (long long)units, R, nx, dev);
}
static void cuda(cudaError_t e) {
  if (e != cudaSuccess) {
    std::printf("CUDA: %s\n", cudaGetErrorString(e));
    std::exit(2);
  }
}
static void must(gmg_status s) {
  if (s != GMG_OK) {
    std::printf("status %d: %s\n", (int)s, gmg_last_error());
    std::exit(2);
  }
}

static std::mt19937_64 rng(7);
template <class T> struct Dev {  // a device array with its host copy
  T* p = nullptr;
  std::vector<T> h;
  explicit Dev(size_t n) : h(n) { cuda(cudaMalloc(&p, sizeof(T) * n)); }
  ~Dev() { cudaFree(p); }
  void up() { cuda(cudaMemcpy(p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice)); }
  void down() { cuda(cudaMemcpy(h.data(), p, sizeof(T) * h.size(), cudaMemcpyDeviceToHost)); }
  void random(double scale) {
    std::normal_distribution<double> g;
    for (auto& v : h) v = T(scale * g(rng), scale * g(rng));
    up();
  }
};
typedef Dev<cf> Field;
typedef Dev<zc> Scalars;

static Vec vec(void* p, int64_t V, int R, int dof) {
  Vec v;
  v.p = p;
  v.V = V;
  v.R = R;
  v.dof = dof;
  v.prec = GMG_F32;
  return v;
}
static double2* d2(Scalars& s) { return reinterpret_cast<double2*>(s.p); }

struct Shape {
  int64_t V;
  int R, dof;
  int64_t n() const { return V * R * dof; }
  size_t at(int64_t e, int r) const { return (size_t)(e / dof * R + r) * dof + e % dof; }  // component e of one RHS
  int64_t len() const { return V * dof; }
};
static zc dot(const Shape& s, const cf* a, const cf* b, int r) {
  zc t = 0;
  for (int64_t e = 0; e < s.len(); ++e) t += std::conj(zc(a[s.at(e, r)])) * zc(b[s.at(e, r)]);
  return t;
}

// the captured solve's state for m Krylov vectors
struct State {
  int m;
  Scalars H, g, cs, sn, bn2;
  Dev<double> res;
  Dev<int> ctr;
  State(int m_, int R)
      : m(m_), H((size_t)R * (m_ + 1) * m_), g((size_t)R * (m_ + 1)), cs((size_t)R * m_), sn((size_t)R * m_), bn2(R), res(R), ctr(4) {}
  RhsGivens args(double tol, int maxit) {
    return RhsGivens{d2(H), d2(g), d2(cs), d2(sn), res.p, d2(bn2), ctr.p, tol, m, maxit, 0, 0};
  }
};

static void gram_schmidt(Shape s, int nx, cudaStream_t st) {
  const int64_t units = s.len() / 2, n = s.n();
  const double sz = 1.0 / std::sqrt((double)s.len());
  Field V(n * (nx + 1)), w(n);
  V.random(sz * 0.7 / std::sqrt(std::max(1.0, 2.0 * nx / s.len())));  // V V^H stays below one
  w.random(sz);
  Scalars dh((size_t)nx * s.R), dh2((size_t)nx * s.R), dw(s.R);
  State S(nx, s.R);
  S.H.random(1.0);
  S.g.random(1.0);
  std::uniform_real_distribution<double> u(0.0, 6.28);
  for (size_t k = 0; k < S.cs.h.size(); ++k) {  // rotations: |c|^2 + |s|^2 = 1
    const double t = u(rng);
    S.cs.h[k] = std::polar(std::cos(t), u(rng));
    S.sn.h[k] = std::sin(t);
  }
  S.cs.up();
  S.sn.up();
  for (int r = 0; r < s.R; ++r) S.bn2.h[r] = 4.0 + r;
  S.bn2.up();
  S.ctr.h = {nx - 1, nx - 1, 0, 0};
  S.ctr.up();
  const State before = [&] { State c(nx, s.R); c.H.h = S.H.h; c.g.h = S.g.h; c.cs.h = S.cs.h; c.sn.h = S.sn.h; return c; }();
  Vec vV = vec(V.p, s.V, s.R, s.dof), vw = vec(w.p, s.V, s.R, s.dof), vn = vec(V.p + n * nx, s.V, s.R, s.dof);
  must(rhs_gs_step(vV, n, nx, vw, vn, d2(dh), d2(dh2), d2(dw), S.args(1e-30, 100), st));
  cuda(cudaStreamSynchronize(st));
  const std::vector<cf> w0 = w.h;
  w.down();
  check(w.h == w0, "w unchanged", units, s.R, nx, 0);
  for (auto* x : {&dh, &dh2, &dw, &S.H, &S.g, &S.cs, &S.sn}) x->down();
  V.down();
  S.res.down();
  S.ctr.down();
  for (int r = 0; r < s.R; ++r) {
    std::vector<cf> y(w.h);
    double worst = 0;
    std::vector<zc> h(nx);
    for (int pass = 0; pass < 2; ++pass) {
      for (int j = 0; j < nx; ++j) {
        h[j] = dot(s, &V.h[(size_t)j * n], y.data(), r);
        const double e = std::abs(h[j] - (pass ? dh2 : dh).h[(size_t)j * s.R + r]);
        check(e < (pass ? 1e-6 : 1e-11), pass ? "h2" : "h1", units, s.R, nx, e);
      }
      for (int64_t e = 0; e < s.len(); ++e) {
        zc t = y[s.at(e, r)];
        for (int j = 0; j < nx; ++j) t -= h[j] * zc(V.h[(size_t)j * n + s.at(e, r)]);
        y[s.at(e, r)] = cf(t);
      }
    }
    const double nn = dot(s, y.data(), y.data(), r).real(), gn = dw.h[r].real();
    check(std::abs(nn - gn) < 1e-5 * nn, "|w''|^2", units, s.R, nx, nn - gn);
    for (int64_t e = 0; e < s.len(); ++e)
      worst = std::max(worst, (double)std::abs(y[s.at(e, r)] * (float)(1 / std::sqrt(nn)) - V.h[(size_t)nx * n + s.at(e, r)]));
    check(worst < 2e-5 * sz + 1e-6, "v", units, s.R, nx, worst);
    // the column's rotations, from the device's own sums
    const int j = nx - 1, m = nx;
    zc a = dh.h[r] + dh2.h[r];
    auto hs = [&](int i) { return dh.h[(size_t)i * s.R + r] + dh2.h[(size_t)i * s.R + r]; };
    for (int i = 0; i < j; ++i) {
      const zc c = before.cs.h[(size_t)r * m + i], g = before.sn.h[(size_t)r * m + i], b = hs(i + 1);
      const zc top = std::conj(c) * a + std::conj(g) * b;
      check(std::abs(top - S.H.h[((size_t)r * (m + 1) + i) * m + j]) < 1e-11, "H", units, s.R, nx, i);
      a = c * b - g * a;
    }
    const double hn = std::sqrt(gn), den = std::sqrt(std::norm(a) + hn * hn);
    const zc c = a / den, g = hn / den, gj = before.g.h[(size_t)r * (m + 1) + j];
    check(std::abs(c - S.cs.h[(size_t)r * m + j]) + std::abs(g - S.sn.h[(size_t)r * m + j]) < 1e-11, "rotation", units, s.R, nx, 0);
    check(std::abs(den - S.H.h[((size_t)r * (m + 1) + j) * m + j]) < 1e-11 && S.H.h[((size_t)r * (m + 1) + j + 1) * m + j] == 0.0,
          "H diagonal", units, s.R, nx, den);
    check(std::abs(std::conj(c) * gj - S.g.h[(size_t)r * (m + 1) + j]) < 1e-11 &&
              std::abs(-g * gj - S.g.h[(size_t)r * (m + 1) + j + 1]) < 1e-11, "g", units, s.R, nx, 0);
    check(std::abs(std::abs(g * gj) / std::sqrt(4.0 + r) - S.res.h[r]) < 1e-11, "residual", units, s.R, nx, S.res.h[r]);
  }
  check(S.ctr.h[0] == nx && S.ctr.h[1] == nx && S.ctr.h[2] == 0, "counters", units, s.R, nx, S.ctr.h[0]);
}

static void minimal_residual(Shape s, bool update_r, cudaStream_t st) {
  Field x(s.n()), r(s.n()), A(s.n());
  x.random(1.0);
  r.random(1.0);
  A.random(2.0);
  const std::vector<cf> x0 = x.h, r0 = r.h;
  Vec vx = vec(x.p, s.V, s.R, s.dof), vr = vec(r.p, s.V, s.R, s.dof), vA = vec(A.p, s.V, s.R, s.dof);
  must(rhs_mr_step(vx, vr, vA, update_r, st));
  cuda(cudaStreamSynchronize(st));
  x.down();
  r.down();
  for (int q = 0; q < s.R; ++q) {
    const zc a = dot(s, A.h.data(), r0.data(), q) / dot(s, A.h.data(), A.h.data(), q).real();
    double ex = 0, er = 0;
    for (int64_t e = 0; e < s.len(); ++e) {
      const size_t k = s.at(e, q);
      ex = std::max(ex, std::abs(zc(x0[k]) + a * zc(r0[k]) - zc(x.h[k])));
      er = std::max(er, std::abs(zc(r0[k]) - (update_r ? a * zc(A.h[k]) : 0.0) - zc(r.h[k])));
    }
    check(ex < 1e-5 && er < 1e-5, "MR step", s.len() / 2, s.R, update_r, ex + er);
  }
}

// x += sum y_j z_j, y = H^-1 g over n of m directions
static void finish(Shape s, int m, int n, cudaStream_t st) {
  Field Z(s.n() * m), x(s.n());
  Z.random(1.0);
  x.random(1.0);
  const std::vector<cf> x0 = x.h;
  State S(m, s.R);
  S.H.random(0.3);
  S.g.random(1.0);
  for (int r = 0; r < s.R; ++r)
    for (int i = 0; i < m; ++i) S.H.h[((size_t)r * (m + 1) + i) * m + i] += 3.0;
  S.H.up();
  S.ctr.h = {n, n, 0, 0};
  S.ctr.up();
  Vec vx = vec(x.p, s.V, s.R, s.dof);
  must(rhs_cycle_finish(vec(Z.p, s.V, s.R, s.dof), s.n(), vx, S.args(0, 100), st));
  cuda(cudaStreamSynchronize(st));
  x.down();
  for (int r = 0; r < s.R; ++r) {
    std::vector<zc> y(n);
    for (int i = n - 1; i >= 0; --i) {
      zc t = S.g.h[(size_t)r * (m + 1) + i];
      for (int k = i + 1; k < n; ++k) t -= S.H.h[((size_t)r * (m + 1) + i) * m + k] * y[k];
      y[i] = t / S.H.h[((size_t)r * (m + 1) + i) * m + i];
    }
    double worst = 0;
    for (int64_t e = 0; e < s.len(); ++e) {
      zc t = x0[s.at(e, r)];
      for (int i = 0; i < n; ++i) t += y[i] * zc(Z.h[(size_t)i * s.n() + s.at(e, r)]);
      worst = std::max(worst, std::abs(t - zc(x.h[s.at(e, r)])) / (1.0 + std::abs(t)));
    }
    check(worst < 1e-6, "cycle end", s.len() / 2, s.R, n, worst);
  }
}

// start of a cycle, one step behind its IF node, end of the cycle, as one graph
static void cycle(Shape s, double tol, bool runs, cudaStream_t st, cudaStream_t body) {
  Field b(s.n()), w(s.n()), V(s.n() * 2), q(s.n()), x(s.n());
  b.random(1.0);
  w.random(0.5);
  q.random(1.0);
  x.random(1.0);
  const std::vector<cf> x0 = x.h;
  const int m = 1;
  State S(m, s.R);
  S.ctr.h = {0, 0, 0, 0};
  S.ctr.up();
  Scalars dh(s.R), dh2(s.R), dw(s.R);
  RhsGivens gv = S.args(tol, 10);
  cuda(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  cuda(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr));
  cuda(cudaGraphConditionalHandleCreate(&gv.next, g, 0, cudaGraphCondAssignDefault));
  Vec vb = vec(b.p, s.V, s.R, s.dof), vw = vec(w.p, s.V, s.R, s.dof), v0 = vec(V.p, s.V, s.R, s.dof);
  Vec v1 = vec(V.p + s.n(), s.V, s.R, s.dof), vq = vec(q.p, s.V, s.R, s.dof), vx = vec(x.p, s.V, s.R, s.dof);
  must(rhs_cycle_start(vb, vw, v0, true, d2(S.bn2), gv, st));
  cuda(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &nd));
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = gv.next;
  p.conditional.type = cudaGraphCondTypeIf;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  cuda(cudaGraphAddNode(&node, g, deps, nd, &p));
  cuda(cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
  cuda(cudaStreamBeginCaptureToGraph(body, p.conditional.phGraph_out[0], nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  gv.has_next = 0;
  must(rhs_gs_step(v0, s.n(), 1, vq, v1, d2(dh), d2(dh2), d2(dw), gv, body));
  cudaGraph_t gb = nullptr;
  cuda(cudaStreamEndCapture(body, &gb));
  must(rhs_cycle_finish(v0, s.n(), vx, gv, st));
  cuda(cudaStreamEndCapture(st, &g));
  cudaGraphExec_t ex;
  cuda(cudaGraphInstantiate(&ex, g, 0));
  cuda(cudaGraphLaunch(ex, st));
  cuda(cudaStreamSynchronize(st));
  cudaGraphExecDestroy(ex);
  cudaGraphDestroy(g);
  V.down();
  x.down();
  S.bn2.down();
  S.ctr.down();
  S.H.down();
  S.g.down();
  check(S.ctr.h[0] == (runs ? 1 : 0) && S.ctr.h[1] == (runs ? 1 : 0) && S.ctr.h[2] == 0, "cycle counters", s.len() / 2, s.R, runs, S.ctr.h[0]);
  for (int r = 0; r < s.R; ++r) {
    std::vector<cf> d(b.h);
    for (int64_t e = 0; e < s.len(); ++e) d[s.at(e, r)] -= w.h[s.at(e, r)];
    const double bb = dot(s, b.h.data(), b.h.data(), r).real(), beta = std::sqrt(dot(s, d.data(), d.data(), r).real());
    check(std::abs(S.bn2.h[r].real() - bb) < 1e-11 * bb, "|b|^2", s.len() / 2, s.R, runs, S.bn2.h[r].real() - bb);
    double ev = 0, ex2 = 0;
    // y = g_0 / H_00: conj(c) beta over the rotated h
    const zc y = runs ? S.g.h[(size_t)r * 2] / S.H.h[(size_t)r * 2] : zc(0);
    for (int64_t e = 0; e < s.len(); ++e) {
      const size_t k = s.at(e, r);
      ev = std::max(ev, std::abs(zc(d[k]) / beta - zc(V.h[k])));
      ex2 = std::max(ex2, std::abs(zc(x0[k]) + y * zc(V.h[k]) - zc(x.h[k])));
    }
    check(ev < 1e-6 && ex2 < 1e-5, "cycle", s.len() / 2, s.R, runs, ev + ex2);
    if (runs) {
      const zc h = dot(s, V.h.data(), q.h.data(), r);
      double hn = 0;
      for (int64_t e = 0; e < s.len(); ++e) hn += std::norm(zc(q.h[s.at(e, r)]) - h * zc(V.h[s.at(e, r)]));
      const zc want = std::conj(h) * beta / (std::norm(h) + hn);  // least squares of one column
      check(std::abs(y - want) < 1e-4 * (std::abs(want) + beta / std::sqrt(hn)), "solution", s.len() / 2, s.R, runs, std::abs(y - want));
    }
  }
}

int main() {
  cudaStream_t st, body;
  cuda(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  cuda(cudaStreamCreateWithFlags(&body, cudaStreamNonBlocking));
  const Shape shapes[] = {{1, 1, 2}, {255, 3, 2}, {257, 2, 2}, {256, 2, 16}, {2049, 1, 2}, {4097, 2, 2}, {8193, 1, 2}, {1024, 2, 32}};
  for (const Shape& s : shapes) {
    Vec v = vec(reinterpret_cast<void*>(16), s.V, s.R, s.dof);
    check(rhs_fused(v, 32), "taken", s.len() / 2, s.R, 32, 0);
    for (int nx : {1, 4, 5, 32}) gram_schmidt(s, nx, st);
    minimal_residual(s, true, st);
    minimal_residual(s, false, st);
    finish(s, 5, 5, st);
    finish(s, 8, 3, st);
    finish(s, 4, 0, st);
    cycle(s, 0.0, true, st, body);
    cycle(s, 10.0, false, st, body);
  }
  check(!rhs_fused(vec(reinterpret_cast<void*>(16), 16385, 1, 2), 1), "length refused", 16385, 1, 1, 0);
  check(!rhs_fused(vec(reinterpret_cast<void*>(16), 16, 1, 4), 33), "basis refused", 32, 1, 33, 0);
  check(!rhs_fused(vec(reinterpret_cast<void*>(16), 16, 1, 3), 1), "odd components refused", 24, 1, 1, 0);
  check(!rhs_fused(vec(reinterpret_cast<void*>(8), 16, 1, 4), 1), "alignment refused", 32, 1, 1, 0);
  std::printf("%s (%d)\n", failures ? "failed" : "all steps agree", failures);
  return failures ? 1 : 0;
}
