// mg_fused.cu -- the vector work of one coarse-level solver step in one kernel.
//
// The Krylov and smoother steps of the right-hand sides are independent of one
// another, and on the coarse levels one right-hand side's vectors are small (256
// sites x 24 components: 48 KB): a thread-block cluster takes one right-hand side
// through a whole step, its sums going through shared memory (distributed shared
// memory between the CTAs of the cluster) in a fixed order.  A Gram-Schmidt step
// done with one kernel per product and update is nine launches (three of them
// zeroing the targets of atomic sums), 2 to 6 us each whatever their bytes:
//
//   rhs_gs_step       h1 = V^H w, w -= V h1, h2 = V^H w, w -= V h2, |w|, v = w / |w|,
//                     and in captured solves the Givens update of the Hessenberg column
//   rhs_mr_step       a = <Ar, r> / <Ar, Ar>, x += a r, r -= a Ar
//   rhs_cycle_start   w = b - A x, |w|, v_0 = w / |w|, start of a restart cycle
//   rhs_cycle_finish  y = H^-1 g, x += sum y_j z_j
//
// FP32 vectors, sums and coefficients in FP64, every vector rounded to FP32 where
// the separate kernels store it.  What bounds them: the latency of the cluster's
// exchanges (three per Gram-Schmidt step).  16^4 solve of 24 right-hand sides (level
// 1: 256 sites, nbasis 24; level 2: 16 sites, nbasis 32): 4.54 -> 3.94 ms per outer
// iteration (six setups each); Gram-Schmidt step 36 -> 11 to 16 us, MR step 12 -> 6.
#include <cooperative_groups.h>

#include <type_traits>

#include "mg_internal.cuh"

namespace gmg {
namespace cg = cooperative_groups;

namespace {

constexpr int kNT = 256, kNW = kNT / 32, kMaxCluster = 8, kMaxUnits = 8;

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double zabs2(double2 a) { return a.x * a.x + a.y * a.y; }

// One right-hand side's share of a field [V][R][dof]: 16-byte units (two complex
// numbers), unit u at site u / hd, place u % hd; the cluster's threads take them in
// turn.  off: the thread's units (in 16-byte units of the field), n of them.
template <int UN> struct Share {
  int off[UN];
  int n;
  __device__ __forceinline__ Share(int64_t units, int hd, int R, int r, int rank, int cs) {
    n = 0;
#pragma unroll
    for (int k = 0; k < UN; ++k) {
      const int u = rank * kNT + (int)threadIdx.x + k * cs * kNT;
      off[k] = (u / hd * R + r) * hd + u % hd;
      if (u < units) n = k + 1;
    }
  }
};

// The warp's sums of eight values per lane, halving the values a lane carries with
// every exchange (9 exchanges instead of 40): the first `cnt` go to part[k * kNW + warp].
__device__ __forceinline__ void warp_sums(double (&v)[8], double* part, int cnt) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4; h >= 1; h >>= 1) {
    const bool up = lane & (4 * h);
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * h);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  const int k = (lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1);
  if ((lane & 3) == 0 && k < cnt) part[k * kNW + (threadIdx.x >> 5)] = v[0];
}

// sums over the cluster of cnt values, each thread's contribution to value k
// already folded per warp in part[k * kNW + warp]; the result in tot.  `mine` is a
// region of its own for every call of a kernel (remote CTAs read it).
__device__ __forceinline__ void cluster_sum(cg::cluster_group& cl, const double* part, double* mine, double* tot,
                                            int cnt) {
  __syncthreads();
  for (int k = threadIdx.x; k < cnt; k += kNT) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kNW; ++q) v += part[k * kNW + q];
    mine[k] = v;
  }
  cl.sync();
  const int cs = cl.num_blocks();
  for (int k = threadIdx.x; k < cnt; k += kNT) {
    double v = 0.0;
    for (int c = 0; c < cs; ++c) v += *cl.map_shared_rank(mine + k, c);
    tot[k] = v;
  }
  __syncthreads();
}

// <x, w> of one unit
__device__ __forceinline__ void dot_unit(float4 x, float4 w, double& re, double& im) {
  re += (double)x.x * w.x + (double)x.y * w.y;
  im += (double)x.x * w.y - (double)x.y * w.x;
  re += (double)x.z * w.z + (double)x.w * w.w;
  im += (double)x.z * w.w - (double)x.w * w.z;
}
__device__ __forceinline__ double norm_unit(float4 w) {
  return (double)w.x * w.x + (double)w.y * w.y + (double)w.z * w.z + (double)w.w * w.w;
}
__device__ __forceinline__ float4 scaled(float4 w, double s) {
  return make_float4((float)(s * w.x), (float)(s * w.y), (float)(s * w.z), (float)(s * w.w));
}
// w + sum_j c_j x_j over nx vectors at stride vs (c interleaved re, im), summed in FP64, rounded once
__device__ __forceinline__ float4 combine(float4 w, const double* c, double sgn, const float4* X, int64_t vs, int nx) {
  double a = w.x, b = w.y, d = w.z, e = w.w;
#pragma unroll 5
  for (int j = 0; j < nx; ++j) {
    const float4 x = X[j * vs];
    const double cr = sgn * c[2 * j], ci = sgn * c[2 * j + 1];
    a += cr * x.x - ci * x.y;
    b += cr * x.y + ci * x.x;
    d += cr * x.z - ci * x.w;
    e += cr * x.w + ci * x.z;
  }
  return make_float4((float)a, (float)b, (float)d, (float)e);
}

// true in one CTA of the grid, after every cluster's rank 0 has come here and
// what it wrote before is visible to that CTA; the counter is left at zero
__device__ __forceinline__ bool last_rhs(int* counter, int R) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(counter, 1) == R - 1;
    if (last) {
      *counter = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}

struct Field {
  int64_t units;  // 16-byte units of one right-hand side
  int hd, R;
};

template <int UN>
__global__ void __launch_bounds__(kNT) gs_kernel(Field f, const float4* __restrict__ V0, int64_t vs, int nx,
                                                 const float4* __restrict__ w, float4* __restrict__ vn,
                                                 double2* __restrict__ dh, double2* __restrict__ dh2,
                                                 double2* __restrict__ dw, RhsGivens gv) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int cs = cl.num_blocks(), rank = cl.block_rank(), r = blockIdx.x / cs, t = threadIdx.x;
  double* part = sm;                  // [2 nx][kNW]
  double* mine = part + 2 * nx * kNW;  // two passes of 2 nx, the norm
  double* tot = mine + 4 * nx + 1;    // [2 nx]
  double* hsum = tot + 2 * nx;        // [2 nx]
  const Share<UN> sh(f.units, f.hd, f.R, r, rank, cs);
  float4 y[UN];
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) y[k] = w[sh.off[k]];
  for (int pass = 0; pass < 2; ++pass) {
    for (int j0 = 0; j0 < nx; j0 += 4) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        double re = 0.0, im = 0.0;
        if (j0 + i < nx) {
#pragma unroll
          for (int k = 0; k < UN; ++k)
            if (k < sh.n) dot_unit(V0[(j0 + i) * vs + sh.off[k]], y[k], re, im);
        }
        v[2 * i] = re;
        v[2 * i + 1] = im;
      }
      warp_sums(v, part + 2 * j0 * kNW, 2 * (nx - j0));
    }
    cluster_sum(cl, part, mine + pass * 2 * nx, tot, 2 * nx);
#pragma unroll
    for (int k = 0; k < UN; ++k)
      if (k < sh.n) y[k] = combine(y[k], tot, -1.0, V0 + sh.off[k], vs, nx);
    if (t < 2 * nx) hsum[t] = pass ? hsum[t] + tot[t] : tot[t];
    if (rank == 0 && t < nx) (pass ? dh2 : dh)[(int64_t)t * f.R + r] = make_double2(tot[2 * t], tot[2 * t + 1]);
    __syncthreads();
  }
  double nn = 0.0;
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) nn += norm_unit(y[k]);
  double nv[8] = {nn};
  warp_sums(nv, part, 1);
  cluster_sum(cl, part, mine + 4 * nx, tot, 1);
  nn = tot[0];
  const double sc = nn > 0.0 ? rsqrt(nn) : 0.0;
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) vn[sh.off[k]] = scaled(y[k], sc);
  if (rank == 0) {
    if (t == 0) dw[r] = make_double2(nn, 0.0);
    if (gv.H) {
      // Hessenberg column nx - 1: previous rotations, a new one, the residual estimate
      const int j = nx - 1, m = gv.m;
      if (t == 0) {
        double2* Hr = gv.H + (size_t)r * (m + 1) * m;
        double2 a = make_double2(hsum[0], hsum[1]);
        for (int i = 0; i < j; ++i) {
          const double2 c = gv.cs[r * m + i], sg = gv.sn[r * m + i];
          const double2 b = make_double2(hsum[2 * i + 2], hsum[2 * i + 3]);
          const double2 u = zmul(zconj(c), a), v = zmul(zconj(sg), b);
          const double2 p = zmul(c, b), q = zmul(sg, a);
          Hr[i * m + j] = make_double2(u.x + v.x, u.y + v.y);
          a = make_double2(p.x - q.x, p.y - q.y);
        }
        const double hn = sqrt(fmax(nn, 0.0)), den = sqrt(zabs2(a) + hn * hn);
        double2 c = make_double2(1.0, 0.0), sg = make_double2(0.0, 0.0);
        if (den > 0.0) {
          c = make_double2(a.x / den, a.y / den);
          sg = make_double2(hn / den, 0.0);
        }
        gv.cs[r * m + j] = c;
        gv.sn[r * m + j] = sg;
        const double2 d = zmul(zconj(c), a);
        Hr[j * m + j] = make_double2(d.x + sg.x * hn, d.y);
        Hr[(j + 1) * m + j] = make_double2(0.0, 0.0);
        double2* gr = gv.g + (size_t)r * (m + 1);
        const double2 gj = gr[j];
        gr[j] = zmul(zconj(c), gj);
        gr[j + 1] = make_double2(-sg.x * gj.x, -sg.x * gj.y);
        gv.res[r] = sqrt(zabs2(gr[j + 1])) / sqrt(fmax(gv.bn2[r].x, 1e-300));
      }
      if (last_rhs(gv.ctr + 2, f.R)) {
        int ok = 1;
        for (int q = t; q < f.R; q += kNT) ok &= __ldcg(gv.res + q) <= gv.tol;
        const int conv = __syncthreads_and(ok);
        if (t == 0) {
          const int it = gv.ctr[0] + 1;
          gv.ctr[0] = it;
          gv.ctr[1] = j + 1;
          if (gv.has_next) cudaGraphSetConditional(gv.next, (!conv && it < gv.maxit) ? 1u : 0u);
        }
      }
    }
  }
  cl.sync();  // the other CTAs have read this one's shared memory
}

template <int UN>
__global__ void __launch_bounds__(kNT) mr_kernel(Field f, float4* __restrict__ x, float4* __restrict__ rr,
                                                 const float4* __restrict__ Ar, int update_r) {
  __shared__ double part[3 * kNW], mine[3], tot[3];
  cg::cluster_group cl = cg::this_cluster();
  const int cs = cl.num_blocks(), r = blockIdx.x / cs;
  const Share<UN> sh(f.units, f.hd, f.R, r, cl.block_rank(), cs);
  double re = 0.0, im = 0.0, nn = 0.0;
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) {
      const float4 a = Ar[sh.off[k]];
      dot_unit(a, rr[sh.off[k]], re, im);
      nn += norm_unit(a);
    }
  double v[8] = {re, im, nn};
  warp_sums(v, part, 3);
  cluster_sum(cl, part, mine, tot, 3);
  const double ar = tot[2] > 0.0 ? tot[0] / tot[2] : 0.0, ai = tot[2] > 0.0 ? tot[1] / tot[2] : 0.0;
  const double ap[2] = {ar, ai};
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) {
      const float4 q = rr[sh.off[k]];
      x[sh.off[k]] = combine(x[sh.off[k]], ap, 1.0, &q, 0, 1);
      if (update_r) rr[sh.off[k]] = combine(q, ap, -1.0, Ar + sh.off[k], 0, 1);
    }
  cl.sync();
}

// bn2 (|b|^2 per right-hand side) is formed too with form_bn
template <int UN>
__global__ void __launch_bounds__(kNT) start_kernel(Field f, const float4* __restrict__ b, const float4* __restrict__ w,
                                                    float4* __restrict__ v0, int form_bn, double2* __restrict__ bn2,
                                                    RhsGivens gv) {
  __shared__ double part[2 * kNW], mine[2], tot[2];
  cg::cluster_group cl = cg::this_cluster();
  const int cs = cl.num_blocks(), rank = cl.block_rank(), r = blockIdx.x / cs, t = threadIdx.x, m = gv.m;
  const Share<UN> sh(f.units, f.hd, f.R, r, rank, cs);
  double nn = 0.0, nb = 0.0;
  float4 y[UN];
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) {
      const float4 p = b[sh.off[k]], q = w[sh.off[k]];
      y[k] = make_float4(p.x - q.x, p.y - q.y, p.z - q.z, p.w - q.w);
      nn += norm_unit(y[k]);
      nb += norm_unit(p);
    }
  double v[8] = {nn, nb};
  warp_sums(v, part, 2);
  cluster_sum(cl, part, mine, tot, 2);
  nn = tot[0];
  const double sc = nn > 0.0 ? rsqrt(nn) : 0.0;
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) v0[sh.off[k]] = scaled(y[k], sc);
  if (rank == 0) {
    if (t == 0) {
      nb = form_bn ? tot[1] : bn2[r].x;
      if (form_bn) bn2[r] = make_double2(nb, 0.0);
      const double beta = sqrt(fmax(nn, 0.0));
      double2* gr = gv.g + (size_t)r * (m + 1);
      gr[0] = make_double2(beta, 0.0);
      for (int k = 1; k <= m; ++k) gr[k] = make_double2(0.0, 0.0);
      gv.res[r] = beta / sqrt(fmax(nb, 1e-300));
    }
    if (last_rhs(gv.ctr + 2, f.R)) {
      int ok = 1;
      for (int q = t; q < f.R; q += kNT) ok &= __ldcg(gv.res + q) <= gv.tol;
      const int conv = __syncthreads_and(ok);
      if (t == 0) {
        const int it = form_bn ? 0 : gv.ctr[0];
        gv.ctr[0] = it;
        gv.ctr[1] = 0;
        cudaGraphSetConditional(gv.next, (!conv && it < gv.maxit) ? 1u : 0u);
      }
    }
  }
  cl.sync();
}

template <int UN>
__global__ void __launch_bounds__(kNT) finish_kernel(Field f, const float4* __restrict__ Z0, int64_t zs,
                                                     float4* __restrict__ x, RhsGivens gv) {
  extern __shared__ double sm[];  // [m] y, then H [m][m] and g [m]
  cg::cluster_group cl = cg::this_cluster();
  const int cs = cl.num_blocks(), r = blockIdx.x / cs, t = threadIdx.x, m = gv.m, n = gv.ctr[1];
  double2* y = reinterpret_cast<double2*>(sm);
  double2 *H = y + m, *g = H + m * m;
  for (int k = t; k < m * m; k += kNT) H[k] = gv.H[(size_t)r * (m + 1) * m + k];
  for (int k = t; k < m; k += kNT) g[k] = gv.g[(size_t)r * (m + 1) + k];
  __syncthreads();
  if (t == 0) {
    for (int i = n - 1; i >= 0; --i) {
      double2 acc = g[i];
      for (int k = i + 1; k < n; ++k) {
        const double2 p = zmul(H[i * m + k], y[k]);
        acc = make_double2(acc.x - p.x, acc.y - p.y);
      }
      const double2 d = H[i * m + i];
      const double dd = zabs2(d);
      y[i] = (d.x != 0.0 || d.y != 0.0)
                 ? make_double2((acc.x * d.x + acc.y * d.y) / dd, (acc.y * d.x - acc.x * d.y) / dd)
                 : make_double2(0.0, 0.0);
    }
    if (blockIdx.x == 0 && gv.has_next) cudaGraphSetConditional(gv.next, (n > 0 && gv.ctr[0] < gv.maxit) ? 1u : 0u);
  }
  __syncthreads();
  const Share<UN> sh(f.units, f.hd, f.R, r, cl.block_rank(), cs);
#pragma unroll
  for (int k = 0; k < UN; ++k)
    if (k < sh.n) x[sh.off[k]] = combine(x[sh.off[k]], sm, 1.0, Z0 + sh.off[k], zs, n);
}

// cluster size and units per thread of a field: the smallest cluster that leaves
// a thread one unit, up to kMaxCluster
int cluster_of(int64_t units) {
  int cs = 1;
  while (cs < kMaxCluster && units > (int64_t)cs * kNT) cs *= 2;
  return cs;
}

template <class K, class... A>
gmg_status launch(K kern, int R, int cs, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(R * cs));
  cfg.blockDim = dim3(kNT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  GMG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
  return GMG_OK;
}

Field field_of(const Vec& v) { return Field{v.V * v.dof / 2, v.dof / 2, v.R}; }

// calls go(units per thread as a constant, cluster size)
template <class G> gmg_status by_units(const Field& f, G go) {
  const int cs = cluster_of(f.units);
  const int64_t un = (f.units + (int64_t)cs * kNT - 1) / ((int64_t)cs * kNT);
  if (un <= 1) return go(std::integral_constant<int, 1>(), cs);
  if (un <= 2) return go(std::integral_constant<int, 2>(), cs);
  if (un <= 4) return go(std::integral_constant<int, 4>(), cs);
  return go(std::integral_constant<int, kMaxUnits>(), cs);
}

const float4* q4(const Vec& v) { return static_cast<const float4*>(v.p); }
float4* q4(Vec& v) { return static_cast<float4*>(v.p); }

}  // namespace

// FP32 fields of at most kMaxUnits units per thread of the largest cluster (32,768
// complex numbers per right-hand side: longer ones keep the whole chip busy in the
// separate kernels; 8^4 sites x 24, 24 RHS: MR step 46 us here, 38 there), Krylov
// bases of up to 32 vectors
bool rhs_fused(const Vec& v, int m) {
  return v.prec == GMG_F32 && v.dof % 2 == 0 && v.V * v.dof / 2 <= (int64_t)kMaxCluster * kNT * kMaxUnits &&
         v.elems() / 2 < ((int64_t)1 << 31) && m <= 32 && ((uintptr_t)v.p & 15) == 0;
}

gmg_status rhs_gs_step(const Vec& V0, int64_t vstride, int nx, const Vec& w, Vec& vn, double2* dh, double2* dh2,
                       double2* dw, const RhsGivens& gv, cudaStream_t s) {
  const Field f = field_of(w);
  return by_units(f, [&](auto un, int cs) {
    return launch(gs_kernel<decltype(un)::value>, f.R, cs, sizeof(double) * (size_t)(2 * nx * kNW + 8 * nx + 1), s, f,
                  q4(V0), vstride / 2, nx, q4(w), q4(vn), dh, dh2, dw, gv);
  });
}

gmg_status rhs_mr_step(Vec& x, Vec& r, const Vec& Ar, bool update_r, cudaStream_t s) {
  const Field f = field_of(x);
  return by_units(f, [&](auto un, int cs) {
    return launch(mr_kernel<decltype(un)::value>, f.R, cs, 0, s, f, q4(x), q4(r), q4(Ar), update_r ? 1 : 0);
  });
}

gmg_status rhs_cycle_start(const Vec& b, const Vec& w, Vec& v0, bool form_bn, double2* bn2, const RhsGivens& gv,
                           cudaStream_t s) {
  const Field f = field_of(w);
  return by_units(f, [&](auto un, int cs) {
    return launch(start_kernel<decltype(un)::value>, f.R, cs, 0, s, f, q4(b), q4(w), q4(v0), form_bn ? 1 : 0, bn2, gv);
  });
}

gmg_status rhs_cycle_finish(const Vec& Z0, int64_t zstride, Vec& x, const RhsGivens& gv, cudaStream_t s) {
  const Field f = field_of(x);
  return by_units(f, [&](auto un, int cs) {
    return launch(finish_kernel<decltype(un)::value>, f.R, cs, sizeof(double2) * (size_t)(gv.m * (gv.m + 2)), s, f,
                  q4(Z0), zstride / 2, q4(x), gv);
  });
}

}  // namespace gmg
