// coarse_stencil.cu -- 9-point coarse Dirac stencil in FP64 and FP32.
//
// Restates CoarsenedMatrix::M / Mdag / MdirCalc / Mdiag
// (include/CoarsenedMatrixUpstream.h:546-742) and the multi-RHS form
// (include/CoarsenedMatrixUpstreamImprovedDirsaveLutMRHS.h:736-947):
//
//   out(x, r) = sum_{p in [p0,p1)} A_p(x) in(nbr_p(x), r)        (N x N times N)
//
// with Mdag = G5C M G5C (sign flip of the upper half of the basis index on
// load and store, no temporary).  The reference runs one thread per (site,
// row) and re-reads every link element once per RHS; here a link element is
// read from HBM once for all R right-hand sides.  Three forms:
// coarse_mma_kernel (FP64 tensor cores, most sizes of both precisions),
// coarse_simt_pipe_kernel (FP32 pipe, FP32 fields with many right-hand sides)
// and the single-RHS kernels (small lattices).
//
// Links are kept site-major, [V][9][N][N], so that one site's 9 matrices are
// one contiguous stream.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "f64_mma.cuh"
#include "gmg_internal.cuh"

namespace gmg {

template <class T> struct cplx_t;
template <> struct cplx_t<double> { typedef double2 type; };
template <> struct cplx_t<float> { typedef float2 type; };

template <class C> __device__ __forceinline__ C cmul_add(C acc, C a, C b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
  return acc;
}

// ---------------------------------------------------------------------------
// layout conversion [p][V][N][N] (exchange) -> [V][p][N][N] (site-major)
// ---------------------------------------------------------------------------
template <class To>
__global__ void links_site_major_kernel(const double2* __restrict__ src, To* __restrict__ dst,
                                        int64_t V, int NN) {
  const int64_t total = 9 * V * NN;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = k % NN;
    const int64_t ps = k / NN;
    const int64_t s = ps % V;
    const int64_t p = ps / V;
    const double2 v = src[k];
    To o;
    o.x = v.x;
    o.y = v.y;
    dst[(s * 9 + p) * NN + e] = o;
  }
}

static int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  return (int)std::min<int64_t>(std::max<int64_t>(b, 1), 148 * 32);
}

gmg_status coarse_links_to_site_major(gmg_coarse* h, cudaStream_t s) {
  const int64_t V = h->dims.vol();
  const int NN = h->N * h->N;
  GMG_TRY(h->links_d.alloc(sizeof(double2) * 9 * V * NN));
  links_site_major_kernel<double2><<<grid_for(9 * V * NN, 256), 256, 0, s>>>(
      h->links_ref.as<double2>(), h->links_d.as<double2>(), V, NN);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

gmg_status coarse_prepare_f32(gmg_coarse* h, cudaStream_t s) {
  const int64_t V = h->dims.vol();
  const int NN = h->N * h->N;
  GMG_TRY(h->links_f.alloc(sizeof(float2) * 9 * V * NN));
  links_site_major_kernel<float2><<<grid_for(9 * V * NN, 256), 256, 0, s>>>(
      h->links_ref.as<double2>(), h->links_f.as<float2>(), V, NN);
  GMG_CUDA(cudaGetLastError());
  h->links_f_ok = true;
  return GMG_OK;
}

// ---------------------------------------------------------------------------
// the stencil kernel
// ---------------------------------------------------------------------------
// Link source and site geometry of one apply.  Output index o (V of them: all
// sites, or the sites of one parity) takes its links from link site
// site_map[o] (identity when null): matrix (p - pbase) of the link_pts matrices
// stored per site; its neighbour for point p is input index nbr[p][o] (o
// itself when nbr is null).  dag applies the conjugate transpose of each matrix.
struct LinkSel {
  const void* links;
  int link_pts, pbase;
  const int32_t* site_map;
  const int32_t* nbr;
  int dag;
};

template <class C> __device__ __forceinline__ C cconj(C a) {
  a.y = -a.y;
  return a;
}

// ---------------------------------------------------------------------------
// The stencil on the FP64 tensor cores (f64_mma.cuh), for FP64 fields and for
// FP32 ones widened on load.  A unit is one site, 8 MT rows and 4 RQ right-hand
// sides; a warp forms a unit's sum over its share of the site's (point, basis)
// contraction with the next step's operands requested one step ahead, KS warps
// of the CTA taking the points in turn ranges and adding their tiles through
// shared memory in a fixed order.
// What bounds it: the MMA rate (the links are used once per R right-hand
// sides, 8 N N R flops per 16 N N bytes: above about 10 FP64 right-hand sides
// the arithmetic takes longer than the links).  The register-tiled CUDA-core
// kernels before it were bound by their shared-memory operand reads and one
// barrier pair per point.  At 8^4, nbasis 32, 32 RHS, FP64: 536 -> 356 us
// (27 TFLOP/s of the 37 the MMAs reach; two register sets leave 10 warps per SM,
// which do not always cover the links' DRAM latency); 4096 sites, nbasis 40, 7
// RHS: 1276 -> 197 us; 840 sites, nbasis 40, 5 RHS, FP32: 284 -> 41 us.
// sel (nullable): the output sites (gridDim.x of them) instead of all; skip
// (nullable): per site, bit p leaves point p out.
// ---------------------------------------------------------------------------
template <class C> struct MmaArgs {
  const C* links;
  int link_pts, pbase;
  const int32_t* site_map;
  const int32_t* nbr;
  int dag;
  const C* in;
  C* out;
  int V, N, nrhs;
  const int32_t* active;
  int R, p0, p1, g5;
  const int32_t* sel;
  const uint8_t* skip;
  int units, rchunks, G, KS;  // units per site (rchunks per row chunk), units and point shares per CTA
};

// threads of a CTA: 9 warps (a stencil's points) where the tile leaves the
// registers for three warps on a scheduler, else 8
constexpr int mma_threads(int tiles) { return tiles <= 8 ? 288 : 256; }


template <class T, int MT, int RQ>
__global__ void __launch_bounds__(mma_threads(MT * RQ)) coarse_mma_kernel(const MmaArgs<typename cplx_t<T>::type> a) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int N = a.N, ks = warp % a.KS, g = warp / a.KS, u = blockIdx.y * a.G + g;
  const int site = a.sel ? a.sel[blockIdx.x] : (int)blockIdx.x;
  const int mc = u / a.rchunks, rc = u - mc * a.rchunks;
  const int kk = lane & 3, part = (lane >> 2) & 1, half = N / 2;
  double acc[MT][RQ][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int q = 0; q < RQ; ++q) acc[m][q][0] = acc[m][q][1] = 0.0;

  if (u < a.units) {
    // rows and right-hand sides past the end repeat the last one; their results are not stored
    const int sb = a.dag ? 1 : N, sk = a.dag ? N : 1;
    int rowoff[MT], foff[RQ];
#pragma unroll
    for (int m = 0; m < MT; ++m) rowoff[m] = min((mc * MT + m) * 8 + (lane >> 2), N - 1) * sb;
#pragma unroll
    for (int q = 0; q < RQ; ++q) {
      const int r = min((rc * RQ + q) * 4 + (lane >> 3), a.R - 1);
      foff[q] = (a.active ? a.active[r] : r) * N;
    }
    const uint32_t s1 = f64mma::second_sign(part, a.dag != 0);
    const int64_t lsite = a.site_map ? a.site_map[site] : site;
    const C* lp = a.links + (lsite * a.link_pts - a.pbase) * (int64_t)N * N;
    const int mynb = (a.nbr && lane < 9) ? a.nbr[(int64_t)lane * a.V + site] : site;
    const int npts = a.p1 - a.p0;
    unsigned pts = ((1u << (a.p0 + (ks + 1) * npts / a.KS)) - 1) & ~((1u << (a.p0 + ks * npts / a.KS)) - 1);
    if (a.skip) pts &= ~(unsigned)a.skip[site];
    // Both operands are requested one step ahead of their use, into the other
    // of two register sets.
    if (pts) {
      C av[2][MT], fv[2][RQ];
      int k4 = 0, left = __popc(pts) * ((N + 3) / 4), k0 = 0;
      const C *Ap, *xp;
      auto at_point = [&]() {
        const int p = __ffs(pts) - 1;
        Ap = lp + (int64_t)p * N * N;
        xp = a.in + (int64_t)__shfl_sync(0xffffffffu, mynb, p) * a.nrhs * N;
      };
      auto request = [&](C (&A)[MT], C (&F)[RQ]) {
        const int k = k4 + kk;
        const bool in_k = k < N;
#pragma unroll
        for (int m = 0; m < MT; ++m) A[m] = in_k ? __ldg(Ap + rowoff[m] + k * sk) : C{0, 0};
#pragma unroll
        for (int q = 0; q < RQ; ++q) F[q] = in_k ? __ldg(xp + foff[q] + k) : C{0, 0};
        k4 += 4;
        if (k4 >= N) {
          k4 = 0;
          pts &= pts - 1;
          if (pts) at_point();
        }
      };
      auto multiply = [&](const C (&A)[MT], const C (&F)[RQ]) {
        const uint32_t g5 = (a.g5 && k0 + kk >= half) ? 0x80000000u : 0u;
        double b0[RQ], b1[RQ];
#pragma unroll
        for (int q = 0; q < RQ; ++q) f64mma::expand(F[q], part, g5, s1 ^ g5, b0[q], b1[q]);
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int q = 0; q < RQ; ++q) f64mma::mma(acc[m][q], (double)A[m].x, b0[q]);
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int q = 0; q < RQ; ++q) f64mma::mma(acc[m][q], (double)A[m].y, b1[q]);
        k0 = k0 + 4 >= N ? 0 : k0 + 4;
      };
      at_point();
      request(av[0], fv[0]);
      for (;;) {
        if (left > 1) request(av[1], fv[1]);
        multiply(av[0], fv[0]);
        if (--left == 0) break;
        if (left > 1) request(av[0], fv[0]);
        multiply(av[1], fv[1]);
        if (--left == 0) break;
      }
    }
  }

  auto store = [&](int m, int q, double re, double im) {
    const int b = (mc * MT + m) * 8 + (lane >> 2), r = (rc * RQ + q) * 4 + kk;
    if (b >= N || r >= a.R) return;
    if (a.g5 && b >= half) {
      re = -re;
      im = -im;
    }
    const int slot = a.active ? a.active[r] : r;
    C v;
    v.x = re;
    v.y = im;
    a.out[((int64_t)site * a.nrhs + slot) * N + b] = v;
  };
  if (a.KS == 1) {
    if (u < a.units) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < RQ; ++q) store(m, q, acc[m][q][0], acc[m][q][1]);
    }
    return;
  }
  double2* red = reinterpret_cast<double2*>(smem_raw) + (int64_t)g * a.KS * MT * RQ * 32;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int q = 0; q < RQ; ++q)
      red[(ks * MT * RQ + m * RQ + q) * 32 + lane] = make_double2(acc[m][q][0], acc[m][q][1]);
  __syncthreads();
  if (u < a.units) {
    for (int t = ks; t < MT * RQ; t += a.KS) {
      double re = 0.0, im = 0.0;
      for (int j = 0; j < a.KS; ++j) {
        const double2 v = red[(j * MT * RQ + t) * 32 + lane];
        re += v.x;
        im += v.y;
      }
      store(t / RQ, t % RQ, re, im);
    }
  }
}

template <class T, int MT, int RQ>
static gmg_status launch_mma(const MmaArgs<typename cplx_t<T>::type>& a, int nsites, cudaStream_t s) {
  auto kern = coarse_mma_kernel<T, MT, RQ>;
  const size_t smem = a.KS == 1 ? 0 : sizeof(double2) * 32 * MT * RQ * (size_t)a.G * a.KS;
  if (smem > 48 * 1024)
    GMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  KernelTimer kt("coarse_simt", s);
  kern<<<dim3(nsites, (a.units + a.G - 1) / a.G), 32 * a.G * a.KS, smem, s>>>(a);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

// Registers a thread of coarse_mma_kernel<T, MT, RQ> (allocated in eights; nvcc
// 12.9), which decide how many warps an SM holds.  A wrong entry costs speed only.
static int mma_regs(bool f64, int MT, int w) {
  static const unsigned char tab[2][5][5] = {{
      {56, 72, 72, 88, 96},
      {72, 80, 96, 112, 128},
      {72, 96, 128, 128, 152},
      {88, 112, 128, 160, 176},
      {96, 128, 160, 192, 208}}, {
      {64, 72, 96, 96, 120},
      {72, 96, 112, 128, 152},
      {96, 120, 128, 160, 184},
      {112, 136, 160, 192, 216},
      {128, 160, 192, 224, 248}}};
  return tab[f64 ? 1 : 0][MT - 1][w - 1];
}

// Launch shape: quads of right-hand sides per unit (w, in `chunks` chunks),
// units (G) and point shares (KS) per CTA.
// w gives the fewest padded quads (each chunk reads the links once more, counted
// as half a quad).  FP32 from 7 quads on: where the registers of a tile leave fewer
// than 14 warps per SM its operands' latency shows, and a narrower tile wins (4096
// sites, nbasis 34, 48 RHS: 936 us with w = 4, 714 with 3).  A single point, which
// cannot be split, takes narrower tiles until every scheduler has a warp.
// G: all the units that fit, or half of them or one where that puts a third more
// warps on an SM (FP32, nbasis 50, 64 RHS, 4096 sites: 8 units a CTA 2603 us, 4 2110).
// KS: one warp per unit is fastest where the lattice fills the chip (4096 sites,
// nbasis 32, 32 RHS, FP64: 356 us, 431 with two shares); below that the points are
// split until every SM has about 12 warps, or 24 of the small tiles, whose steps are
// too short to hide the operands' latency (840 sites, nbasis 40, 5 RHS, FP32: 39 us
// with 5 shares, 44 with 2, 48 with 1).  A split of big tiles, or into 5 or 9 shares,
// that would turn one wave of CTAs into one and up to a half is not made (256 sites,
// nbasis 32, 32 RHS, FP64: 5 shares 50 us, 2 31 us).
struct MmaShape {
  int w, chunks, G, KS;
};
static MmaShape mma_shape(bool f64, int64_t nsites, int npts, int MT, int mchunks, int rq) {
  MmaShape sh{1, rq, 1, 1};
  double best = 1e30;
  for (int w = 1; w <= std::min(5, rq); ++w) {
    const int u = (rq + w - 1) / w, warps = 65536 / (32 * mma_regs(f64, MT, w));
    double cost = u * (2 * w + 1);
    if (!f64 && rq >= 7 && warps < 14) cost *= std::pow(14.0 / warps, 0.6);
    if (cost <= best) {
      best = cost;
      sh = MmaShape{w, u, 1, 1};
    }
  }
  while (npts == 1 && sh.w > 1 && nsites * mchunks * sh.chunks < 148 * 4) {
    sh.w = (sh.w + 1) / 2;
    sh.chunks = (rq + sh.w - 1) / sh.w;
  }
  const int units = mchunks * sh.chunks, maxw = mma_threads(MT * sh.w) / 32, regs = mma_regs(f64, MT, sh.w);
  const int64_t want = 148 * (MT * sh.w > 10 ? 12 : 24);
  int64_t wave = 0;  // CTAs of the split before, where those fit the chip at once
  for (const int ks : {1, 2, 3, 5, 9}) {
    const int KS = std::min(ks, std::min(npts, maxw)), gmax = std::min(units, maxw / KS);
    int G = 0;
    int64_t ctas = 0, slots = 0;
    double most = 0.0;
    for (const int g : {gmax, std::max(1, maxw / KS / 2), 1}) {
      if (g > gmax) continue;
      const int per = (units + g - 1) / g;
      const int64_t q = nsites * per, C = std::max(1, std::min(65536 / (32 * regs * g * KS), std::min(64 / (g * KS), 32)));
      const double warps = (double)std::min(C, (q + 147) / 148) * g * KS * units / (per * g);
      if (G == gmax ? warps < 1.3 * most : G && warps <= most) continue;
      G = g;
      most = warps;
      ctas = q;
      slots = 148 * C;
    }
    if ((MT * sh.w > 10 || ks >= 5) && wave && ctas > slots && ctas < slots * 3 / 2) break;
    wave = ctas <= slots ? ctas : 0;
    sh.KS = KS;
    sh.G = G;
    if (nsites * units * KS >= want) break;
  }
  return sh;
}

template <class T>
static gmg_status coarse_mma(const LinkSel& L, const void* in, void* out, int V, int N, int nrhs,
                             const int32_t* active, int R, int p0, int p1, int g5, const int32_t* sel, int nsel,
                             const uint8_t* skip, cudaStream_t s) {
  typedef typename cplx_t<T>::type C;
  const int mt = (N + 7) / 8, mchunks = (mt + 4) / 5, MT = (mt + mchunks - 1) / mchunks;
  const int nsites = sel ? nsel : V, npts = p1 - p0;
  if (nsites == 0) return GMG_OK;
  const MmaShape sh = mma_shape(sizeof(T) == 8, nsites, npts, MT, mchunks, (R + 3) / 4);
  MmaArgs<C> a{reinterpret_cast<const C*>(L.links), L.link_pts, L.pbase, L.site_map, L.nbr, L.dag,
               reinterpret_cast<const C*>(in), reinterpret_cast<C*>(out), V, N, nrhs, active, R, p0, p1, g5,
               sel, skip, mchunks * sh.chunks, sh.chunks, sh.G, sh.KS};
  auto by_rq = [&](auto mtc) -> gmg_status {
    constexpr int M = decltype(mtc)::value;
    switch (sh.w) {
      case 1: return launch_mma<T, M, 1>(a, nsites, s);
      case 2: return launch_mma<T, M, 2>(a, nsites, s);
      case 3: return launch_mma<T, M, 3>(a, nsites, s);
      case 4: return launch_mma<T, M, 4>(a, nsites, s);
      default: return launch_mma<T, M, 5>(a, nsites, s);
    }
  };
  switch (MT) {
    case 1: return by_rq(std::integral_constant<int, 1>());
    case 2: return by_rq(std::integral_constant<int, 2>());
    case 3: return by_rq(std::integral_constant<int, 3>());
    case 4: return by_rq(std::integral_constant<int, 4>());
    default: return by_rq(std::integral_constant<int, 5>());
  }
}

// ---------------------------------------------------------------------------
// The multi-RHS FP32 stencil on the CUDA cores, pipelined: a CTA walks the (site,
// point) items of its sites; while it multiplies item k, the link matrix and
// the neighbour's R vectors of item k + 1 are copied into the other half of
// its shared memory with cp.async.  A thread owns a TR x TB tile of the R x N
// output, its rows and columns interleaved (r = rt + (R / TR) j, b = bt + (N /
// TB) i), so that the lanes of a warp read consecutive rows of the padded
// shared-memory tiles (row stride N + 1 complex numbers: no bank conflicts).
// Needs TB | N and TR | R.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_c(void* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[j][i] += (or -= with NEG) a_i x_j over bb in [bb0, bb1), a_i = A[b_i][bb]
// (DAG: conj(A[bb][b_i])), x_j = X[r_j][bb]; the signs are folded into the FMAs
template <bool DAG, bool NEG, int TR, int TB, class C>
__device__ __forceinline__ void pipe_mac(C (&acc)[TR][TB], const C* __restrict__ A, const C* __restrict__ X, int bb0,
                                         int bb1, int NP, int bt, int NBT, int rt, int NRT) {
  for (int bb = bb0; bb < bb1; ++bb) {
    C a[TB], x[TR];
#pragma unroll
    for (int i = 0; i < TB; ++i) a[i] = DAG ? A[bb * NP + bt + NBT * i] : A[(bt + NBT * i) * NP + bb];
#pragma unroll
    for (int j = 0; j < TR; ++j) x[j] = X[(rt + NRT * j) * NP + bb];
#pragma unroll
    for (int j = 0; j < TR; ++j)
#pragma unroll
      for (int i = 0; i < TB; ++i) {
        // (ar + i s ai)(xr + i xi) with s = -1 for the conjugate, the product negated with NEG
        const auto ar = NEG ? -a[i].x : a[i].x;
        const auto ai = (NEG != DAG) ? -a[i].y : a[i].y;
        acc[j][i].x = fma(ar, x[j].x, acc[j][i].x);
        acc[j][i].x = fma(-ai, x[j].y, acc[j][i].x);
        acc[j][i].y = fma(ar, x[j].y, acc[j][i].y);
        acc[j][i].y = fma(ai, x[j].x, acc[j][i].y);
      }
  }
}

template <class T, int TR, int TB, int NC>  // NC: N as a compile-time constant (0: runtime)
__global__ void __launch_bounds__(256) coarse_simt_pipe_kernel(
    const typename cplx_t<T>::type* __restrict__ links, int link_pts, int pbase, const int32_t* __restrict__ site_map,
    const int32_t* __restrict__ nbr, int dag, const typename cplx_t<T>::type* __restrict__ in,
    typename cplx_t<T>::type* __restrict__ out, int V, int N_, int nrhs, const int32_t* __restrict__ active, int R,
    int p0, int p1, int g5) {
  typedef typename cplx_t<T>::type C;
  const int N = NC ? NC : N_;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NP = N + 1;                     // padded row stride
  const int stage = (N + R) * NP;           // complex numbers per stage: A [N][NP], X [R][NP]
  C* S = reinterpret_cast<C*>(smem_raw);
  const int t = threadIdx.x, nthr = blockDim.x;
  const int NBT = N / TB, NRT = R / TR;
  const int bt = t % NBT, rt = t / NBT;
  const bool comp = t < NBT * NRT;
  const int half = N / 2;
  const int npts = p1 - p0;
  const int nsites = (V - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int nitems = nsites * npts;

  // copies of item k (site blockIdx.x + (k / npts) gridDim.x, point p0 + k % npts) into stage k & 1
  auto issue = [&](int k) {
    const int site = blockIdx.x + (k / npts) * gridDim.x;
    const int p = p0 + k % npts;
    const int64_t lsite = site_map ? site_map[site] : site;
    const C* Ap = links + (lsite * link_pts + (p - pbase)) * (int64_t)N * N;
    const int nb = nbr ? nbr[(int64_t)p * V + site] : site;
    C* A = S + (k & 1) * stage;
    C* X = A + N * NP;
    for (int e = t; e < N * N; e += nthr) cp_async_c(A + (e / N) * NP + e % N, Ap + e);
    const C* xs = in + (int64_t)nb * nrhs * N;
    for (int e = t; e < R * N; e += nthr) {
      const int r = e / N, bb = e - r * N;
      const int slot = active ? active[r] : r;
      cp_async_c(X + r * NP + bb, xs + slot * N + bb);
    }
    cp_async_commit();
  };

  C acc[TR][TB];
  if (nitems > 0) issue(0);
  for (int k = 0; k < nitems; ++k) {
    if (k + 1 < nitems) {
      issue(k + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const int kp = k % npts;
    if (kp == 0) {
#pragma unroll
      for (int j = 0; j < TR; ++j)
#pragma unroll
        for (int i = 0; i < TB; ++i) acc[j][i] = C{0, 0};
    }
    if (comp) {
      const C* A = S + (k & 1) * stage;
      const C* X = A + N * NP;
      // the dagger and the input G5C (the sign of components bb >= N / 2) are
      // uniform per launch and per half of bb: four loop forms, no per-element
      // selects or sign multiplies
      if (!dag) {
        pipe_mac<false, false, TR, TB>(acc, A, X, 0, half, NP, bt, NBT, rt, NRT);
        if (g5) pipe_mac<false, true, TR, TB>(acc, A, X, half, N, NP, bt, NBT, rt, NRT);
        else pipe_mac<false, false, TR, TB>(acc, A, X, half, N, NP, bt, NBT, rt, NRT);
      } else {
        pipe_mac<true, false, TR, TB>(acc, A, X, 0, half, NP, bt, NBT, rt, NRT);
        if (g5) pipe_mac<true, true, TR, TB>(acc, A, X, half, N, NP, bt, NBT, rt, NRT);
        else pipe_mac<true, false, TR, TB>(acc, A, X, half, N, NP, bt, NBT, rt, NRT);
      }
      if (kp == npts - 1) {
        const int site = blockIdx.x + (k / npts) * gridDim.x;
#pragma unroll
        for (int j = 0; j < TR; ++j) {
          const int r = rt + NRT * j;
          const int slot = active ? active[r] : r;
          C* o = out + ((int64_t)site * nrhs + slot) * N;
#pragma unroll
          for (int i = 0; i < TB; ++i) {
            const int b = bt + NBT * i;
            C v = acc[j][i];
            if (g5 && b >= half) {
              v.x = -v.x;
              v.y = -v.y;
            }
            o[b] = v;
          }
        }
      }
    }
    __syncthreads();  // stage k & 1 is refilled by the issue of item k + 2
  }
}

template <class T, int TR, int TB>
static bool launch_simt_pipe(const LinkSel& L, const void* in, void* out, int V, int N, int nrhs,
                             const int32_t* active, int R, int p0, int p1, int g5, cudaStream_t s,
                             gmg_status* st) {
  typedef typename cplx_t<T>::type C;
  if (N % TB || R % TR || (N / TB) * (R / TR) > 256 || p1 <= p0) return false;
  const size_t smem = sizeof(C) * 2 * (size_t)(N + R) * (N + 1);
  // at least 3 CTAs per SM
  if (smem > 72 * 1024) return false;
  const int threads = std::max(32, ((N / TB) * (R / TR) + 31) / 32 * 32);
  auto kern = N == 32 ? coarse_simt_pipe_kernel<T, TR, TB, 32>
             : N == 40 ? coarse_simt_pipe_kernel<T, TR, TB, 40>
                       : coarse_simt_pipe_kernel<T, TR, TB, 0>;
  *st = GMG_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    *st = fail(GMG_ERR_CUDA, "coarse apply: shared-memory attribute");
    return true;
  }
  int dev = 0, nsm = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  const int grid = std::min(V, nsm * std::max(per_sm, 1));
  KernelTimer kt("coarse_simt", s);
  kern<<<grid, threads, smem, s>>>(reinterpret_cast<const C*>(L.links), L.link_pts, L.pbase, L.site_map, L.nbr, L.dag,
                                   reinterpret_cast<const C*>(in), reinterpret_cast<C*>(out), V, N, nrhs, active, R,
                                   p0, p1, g5);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) *st = fail(GMG_ERR_CUDA, std::string("coarse apply: ") + cudaGetErrorString(e));
  return true;
}

// ---------------------------------------------------------------------------
// Single right-hand side (CoarsenedMatrixUpstream.h:572-597 with nrhs = 1).
// The work per site is 9 GEMVs of N x N, too little for register tiling, and
// the 4^4 lattices of the coarse levels have only 256 sites.  One CTA per site,
// one thread per (point, row): the neighbour vectors are staged in shared
// memory, each thread forms one row product from a contiguous link row, and
// the 9 partial rows are summed in shared memory.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(576) coarse_1rhs_kernel(const typename cplx_t<T>::type* __restrict__ links,
                                                          int link_pts, int pbase,
                                                          const int32_t* __restrict__ site_map,
                                                          const int32_t* __restrict__ nbr, int dag,
                                                          const typename cplx_t<T>::type* __restrict__ in,
                                                          typename cplx_t<T>::type* __restrict__ out, int V, int N,
                                                          int nrhs, int slot, int p0, int p1, int g5) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* X = reinterpret_cast<C*>(smem_raw);  // [9][N] neighbour vectors
  C* part = X + 9 * N;                    // [9][N] partial rows
  const int t = threadIdx.x;
  const int p = t / N, b = t % N;  // blockDim = 9 N
  const int half = N / 2;
  for (int site = blockIdx.x; site < V; site += gridDim.x) {
    const int64_t lsite = site_map ? site_map[site] : site;
    if (p >= p0 && p < p1) {
      const int nb = nbr ? nbr[(int64_t)p * V + site] : site;
      C v = in[((int64_t)nb * nrhs + slot) * N + b];
      if (g5 && b >= half) { v.x = -v.x; v.y = -v.y; }
      X[p * N + b] = v;
    }
    __syncthreads();
    C acc{0, 0};
    if (p >= p0 && p < p1) {
      const C* Mp = links + (lsite * link_pts + (p - pbase)) * N * N;
      if (dag) {  // row b of A^dag: conj(A[bb][b])
        for (int bb = 0; bb < N; ++bb) acc = cmul_add(acc, cconj(Mp[(int64_t)bb * N + b]), X[p * N + bb]);
      } else {
        const C* row = Mp + (int64_t)b * N;
        for (int bb = 0; bb < N; ++bb) acc = cmul_add(acc, row[bb], X[p * N + bb]);
      }
    }
    part[p * N + b] = acc;
    __syncthreads();
    if (t < N) {
      C o{0, 0};
      for (int q = p0; q < p1; ++q) {
        o.x += part[q * N + t].x;
        o.y += part[q * N + t].y;
      }
      if (g5 && t >= half) { o.x = -o.x; o.y = -o.y; }
      out[((int64_t)site * nrhs + slot) * N + t] = o;
    }
    __syncthreads();
  }
}

// Single RHS with the site's links staged in shared memory: the CTA first
// copies the (p1 - p0) N x N link matrices of its site with cp.async (every
// 16-byte chunk in flight at once: one memory round trip instead of a
// dependent chain per row), then thread (p, b) forms row b of point p from
// shared memory, starting
// its row at column (b + k) mod N so that the 16-byte reads of a quarter warp
// fall in distinct banks (N a multiple of 8).
template <class T>
__global__ void __launch_bounds__(576) coarse_1rhs_smem_kernel(const typename cplx_t<T>::type* __restrict__ links,
                                                               int link_pts, int pbase,
                                                               const int32_t* __restrict__ site_map,
                                                               const int32_t* __restrict__ nbr, int dag,
                                                               const typename cplx_t<T>::type* __restrict__ in,
                                                               typename cplx_t<T>::type* __restrict__ out, int V,
                                                               int N, int nrhs, int slot, int p0, int p1, int g5) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int np = p1 - p0, NN = N * N;
  C* Ls = reinterpret_cast<C*>(smem_raw);  // [np][N][N]
  C* X = Ls + (size_t)np * NN;             // [9][N] neighbour vectors
  C* part = X + 9 * N;                     // [9][N] partial rows
  const int t = threadIdx.x;
  const int p = t / N, b = t % N;  // blockDim = 9 N
  const int half = N / 2;
  for (int site = blockIdx.x; site < V; site += gridDim.x) {
    const int64_t lsite = site_map ? site_map[site] : site;
    // every 16-byte chunk of the site's links in flight at once (cp.async),
    // one wait for all of them
    const unsigned char* src = reinterpret_cast<const unsigned char*>(links + (lsite * link_pts + (p0 - pbase)) * NN);
    const int nchunk = (int)(np * NN * sizeof(C) / 16);
    const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(Ls);
    for (int e = t; e < nchunk; e += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + 16u * e), "l"(src + 16 * (size_t)e)
                   : "memory");
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
    if (p >= p0 && p < p1) {
      const int nb = nbr ? nbr[(int64_t)p * V + site] : site;
      C v = in[((int64_t)nb * nrhs + slot) * N + b];
      if (g5 && b >= half) { v.x = -v.x; v.y = -v.y; }
      X[p * N + b] = v;
    }
    __syncthreads();
    C acc{0, 0};
    if (p >= p0 && p < p1) {
      const C* Mp = Ls + (size_t)(p - p0) * NN;
      const C* xp = X + p * N;
      int bb = b;
      if (dag) {  // row b of A^dag: conj(A[bb][b])
        for (int k = 0; k < N; ++k) {
          acc = cmul_add(acc, cconj(Mp[bb * N + b]), xp[bb]);
          bb = bb + 1 == N ? 0 : bb + 1;
        }
      } else {
        const C* row = Mp + b * N;
        for (int k = 0; k < N; ++k) {
          acc = cmul_add(acc, row[bb], xp[bb]);
          bb = bb + 1 == N ? 0 : bb + 1;
        }
      }
    }
    part[p * N + b] = acc;
    __syncthreads();
    if (t < N) {
      C o{0, 0};
      for (int q = p0; q < p1; ++q) {
        o.x += part[q * N + t].x;
        o.y += part[q * N + t].y;
      }
      if (g5 && t >= half) { o.x = -o.x; o.y = -o.y; }
      out[((int64_t)site * nrhs + slot) * N + t] = o;
    }
    __syncthreads();
  }
}

template <class T>
static gmg_status launch_1rhs(const LinkSel& L, const void* in, void* out, int V, int N,
                              int nrhs, int slot, int p0, int p1, int g5, cudaStream_t s) {
  typedef typename cplx_t<T>::type C;
  const int threads = 9 * N;
  KernelTimer kt("coarse_simt", s);
  // links staged in shared memory when they fit two CTAs per SM
  const size_t smem_staged = sizeof(C) * ((size_t)(p1 - p0) * N * N + 18 * (size_t)N);
  if (N % 8 == 0 && smem_staged <= 100 * 1024) {
    if (smem_staged > 48 * 1024)
      GMG_CUDA(cudaFuncSetAttribute(coarse_1rhs_smem_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem_staged));
    coarse_1rhs_smem_kernel<T><<<V, threads, smem_staged, s>>>(
        reinterpret_cast<const C*>(L.links), L.link_pts, L.pbase, L.site_map, L.nbr, L.dag,
        reinterpret_cast<const C*>(in), reinterpret_cast<C*>(out), V, N, nrhs, slot, p0, p1, g5);
    GMG_CUDA(cudaGetLastError());
    return GMG_OK;
  }
  const size_t smem = sizeof(C) * 18 * (size_t)N;
  coarse_1rhs_kernel<T><<<V, threads, smem, s>>>(reinterpret_cast<const C*>(L.links), L.link_pts, L.pbase, L.site_map,
                                                 L.nbr, L.dag, reinterpret_cast<const C*>(in),
                                                 reinterpret_cast<C*>(out), V, N, nrhs, slot, p0, p1, g5);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

// `src`: 0 = the stencil links, 1 = the self-link inverse (one matrix per site,
// addressed as point 8).  V / site_map / nbr: the output geometry (full grid
// when site_map is null and nbr is the handle's table).
gmg_status coarse_apply_simt_ex(gmg_coarse* h, int src, int V, const int32_t* site_map, const int32_t* nbr,
                                bool dag, int p0, int p1, bool g5, int compute, int vec_prec, int nrhs,
                                const void* in, void* out, const int32_t* active, int n_active, cudaStream_t s) {
  const int N = h->N;
  const int R = active ? n_active : nrhs;
  if (R == 0) return GMG_OK;
  LinkSel L{nullptr, src == 1 ? 1 : 9, src == 1 ? 8 : 0, site_map, nbr, dag ? 1 : 0};
  if (compute == GMG_F64) {
    GMG_CHECK(vec_prec == GMG_F64, GMG_ERR_UNSUPPORTED, "F64 compute needs F64 vectors");
    L.links = src == 1 ? h->self_inv.p : h->links_d.p;
  } else if (compute == GMG_F32) {
    GMG_CHECK(vec_prec == GMG_F32, GMG_ERR_UNSUPPORTED, "F32 compute needs F32 vectors");
    GMG_CHECK(src == 1 ? h->self_inv_f_ok : h->links_f_ok, GMG_ERR_STATE,
              "F32 links not prepared (gmg_coarse_prepare)");
    L.links = src == 1 ? h->self_inv_f.p : h->links_f.p;
  } else {
    return fail(GMG_ERR_UNSUPPORTED, "coarse apply: unsupported compute precision for SIMT path");
  }
  GMG_CHECK(L.links != nullptr, GMG_ERR_STATE, "coarse apply: link source not built");
  // One right-hand side: the CUDA-core kernels where a site's links fit their
  // staging buffer (nbasis 24 in FP64, 32 in FP32) and the lattice is small
  // enough to be bound by latency.  FP64 us, CUDA cores / tensor cores: 256
  // sites, nbasis 24: 6.2 / 6.3, nbasis 32: 14 / 10; 768 sites, nbasis 24: 14.4 /
  // 12.3; 4096 sites, nbasis 8: 10.3 / 12.3, nbasis 32: 161 / 98.  FP32: 1024
  // sites, nbasis 32: 16 / 20, nbasis 40: 45 / 31; 4096, nbasis 24: 44 / 38.
  const int64_t vnn = (int64_t)V * N * N;
  if (R == 1 && !active &&
      (compute == GMG_F64 ? N <= 24 && vnn < 768 * 24 * 24 : N <= 32 && vnn < 4096 * 24 * 24)) {
    if (compute == GMG_F64) return launch_1rhs<double>(L, in, out, V, N, nrhs, 0, p0, p1, g5, s);
    return launch_1rhs<float>(L, in, out, V, N, nrhs, 0, p0, p1, g5, s);
  }
  // the sizes the apply takes
  const size_t esz = compute == GMG_F64 ? sizeof(double2) : sizeof(float2);
  GMG_CHECK(R < 4 || ((N + 3) / 4) * ((R + 3) / 4) <= 256, GMG_ERR_UNSUPPORTED,
            "coarse apply: nbasis x nrhs tile too large");
  GMG_CHECK(esz * N * (size_t)(N + R) <= 227 * 1024, GMG_ERR_UNSUPPORTED, "coarse apply: nbasis x nrhs too large");
  if (compute == GMG_F64) return coarse_mma<double>(L, in, out, V, N, nrhs, active, R, p0, p1, g5, nullptr, 0, nullptr, s);
  // FP32 with 28 right-hand sides or more at nbasis 32 to 40, in whole 4 x 4
  // tiles: the FP32 pipe's twice higher rate still wins there (768 sites, nbasis
  // 32, 32 RHS: 65 us against 83 on the FP64 tensor cores; 24 RHS: 64 against 62;
  // nbasis 24, 32 RHS: 52 against 50; nbasis 48: 224 against 168)
  gmg_status st = GMG_OK;
  if (R >= 28 && N >= 32 && N <= 40 && launch_simt_pipe<float, 4, 4>(L, in, out, V, N, nrhs, active, R, p0, p1, g5, s, &st)) return st;
  return coarse_mma<float>(L, in, out, V, N, nrhs, active, R, p0, p1, g5, nullptr, 0, nullptr, s);
}

gmg_status coarse_apply_simt(gmg_coarse* h, int p0, int p1, bool g5, int compute, int vec_prec,
                             int nrhs, const void* in, void* out, const int32_t* active,
                             int n_active, cudaStream_t s) {
  return coarse_apply_simt_ex(h, 0, (int)h->dims.vol(), nullptr, h->nbr.as<int32_t>(), false, p0, p1, g5, compute,
                              vec_prec, nrhs, in, out, active, n_active, s);
}

// FP64 stencil of points [p0, p1) on nsel listed sites (all when sel is null),
// without the points whose bit is set in skip (per site, nullable): the hops
// and the self term of the coarse-operator construction
gmg_status coarse_apply_sel_f64(gmg_coarse* h, int p0, int p1, int nrhs, const double* in, double* out,
                                const int32_t* sel, int nsel, const uint8_t* skip, cudaStream_t s) {
  const LinkSel L{h->links_d.p, 9, 0, nullptr, h->nbr.as<int32_t>(), 0};
  return coarse_mma<double>(L, in, out, (int)h->dims.vol(), h->N, nrhs, nullptr, nrhs, p0, p1, 0, sel, nsel, skip, s);
}

// ---------------------------------------------------------------------------
// ConstructRemainingLinks (...DirsaveLut.h:1164-1196) / ForceHermitian
// (CoarsenedMatrixUpstream.h:956-976) on the exchange layout:
//   A_{dir}(x)[n1][n2] = S(n1,n2) conj(A_{dir+4}(x + e_dir)[n2][n1])
// S = -1 iff n1 and n2 lie in different halves (1 if hermitian).
// ---------------------------------------------------------------------------
__global__ void construct_remaining_kernel(double2* __restrict__ A, const int32_t* __restrict__ nbr,
                                           int V, int N, int hermitian) {
  const int64_t NN = (int64_t)N * N;
  const int64_t total = 4 * (int64_t)V * NN;
  const int half = N / 2;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int n2 = (int)(k % N);
    const int n1 = (int)((k / N) % N);
    const int64_t s = (k / NN) % V;
    const int dir = (int)(k / (NN * V));
    const int sp = nbr[(int64_t)dir * V + s];  // x + e_dir
    double2 v = A[((int64_t)(dir + 4) * V + sp) * NN + (int64_t)n2 * N + n1];
    double f = 1.0;
    if (!hermitian && ((n1 / half + n2 / half) & 1)) f = -1.0;
    A[((int64_t)dir * V + s) * NN + (int64_t)n1 * N + n2] = make_double2(f * v.x, -f * v.y);
  }
}

gmg_status coarse_construct_remaining(gmg_coarse* h, cudaStream_t s) {
  const int V = (int)h->dims.vol();
  const int64_t total = 4 * (int64_t)V * h->N * h->N;
  construct_remaining_kernel<<<grid_for(total, 256), 256, 0, s>>>(
      h->links_ref.as<double2>(), h->nbr.as<int32_t>(), V, h->N, h->hermitian);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

}  // namespace gmg

// ---------------------------------------------------------------------------
// Rework layout map for links (Layout_converters.h:49-56): flat [n1][n2] with
// n = s*Nc_c + c  <->  spin-split [s1][s2][c1][c2].
// ---------------------------------------------------------------------------
namespace gmg {
__global__ void layout_links_kernel(const double2* __restrict__ in, double2* __restrict__ out, int64_t V,
                                    int N, int ncs, int inverse) {
  const int ncc = N / ncs;
  const int64_t NN = (int64_t)N * N;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < V * NN;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = e / NN;
    const int n1 = (int)((e % NN) / N), n2 = (int)(e % N);
    const int s1 = n1 / ncc, c1 = n1 % ncc, s2 = n2 / ncc, c2 = n2 % ncc;
    const int64_t spin = s * NN + ((int64_t)(s1 * ncs + s2) * ncc + c1) * ncc + c2;
    if (!inverse) out[spin] = in[e];
    else out[e] = in[spin];
  }
}

// vectors: flat index n = s * Nc_c + c <-> spin form [s][c] (Layout_converters.h:92-139)
__global__ void layout_vectors_kernel(const double2* __restrict__ in, double2* __restrict__ out, int64_t rows,
                                      int N, int ncs, int inverse) {
  const int ncc = N / ncs;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < rows * N;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = e / N;
    const int n = (int)(e % N), sp = n / ncc, c = n % ncc;
    const int64_t spin = row * N + (int64_t)sp * ncc + c;  // [row][s][c]: the same order as the flat index
    if (!inverse) out[spin] = in[e];
    else out[e] = in[spin];
  }
}
}  // namespace gmg

extern "C" gmg_status gmg_layout_vectors(int64_t rows, int nbasis, int ncs, const double* in, double* out,
                                         int inverse, gmg_stream s) {
  GMG_CHECK(in && out && in != out, GMG_ERR_ARGUMENT, "gmg_layout_vectors: bad pointers");
  GMG_CHECK(rows > 0 && nbasis > 0 && ncs > 0 && nbasis % ncs == 0, GMG_ERR_ARGUMENT,
            "gmg_layout_vectors: nbasis must be a multiple of the coarse spin count");
  const int64_t n = rows * nbasis;
  gmg::layout_vectors_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 32), 256, 0, gmg::S(s)>>>(
      reinterpret_cast<const double2*>(in), reinterpret_cast<double2*>(out), rows, nbasis, ncs, inverse);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

extern "C" gmg_status gmg_layout_links(int64_t V, int nbasis, int ncs, const double* in, double* out,
                                       int inverse, gmg_stream s) {
  GMG_CHECK(in && out && in != out, GMG_ERR_ARGUMENT, "gmg_layout_links: bad pointers");
  GMG_CHECK(V > 0 && nbasis > 0 && ncs > 0 && nbasis % ncs == 0, GMG_ERR_ARGUMENT,
            "gmg_layout_links: nbasis must be a multiple of the coarse spin count");
  const int64_t n = V * nbasis * (int64_t)nbasis;
  gmg::layout_links_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 32), 256, 0, gmg::S(s)>>>(
      reinterpret_cast<const double2*>(in), reinterpret_cast<double2*>(out), V, nbasis, ncs, inverse);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}
