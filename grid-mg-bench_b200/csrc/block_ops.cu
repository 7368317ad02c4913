// block_ops.cu -- block projection and promotion in FP64 and FP32.
//
// Restates blockLutedInnerProduct / blockLutedAxpy / blockLutedOrthonormalise
// (include/CoarsenedMatrixUpstreamImprovedDirsaveLut.h:70-240, multi-RHS form
// ...LutMRHS.h:70-236) as per-block complex GEMMs:
//
//   project   C_c (R x N)  = F_c^T (R x K) conj(V_c)^T (K x N)   K = bv * dof
//   promote   F_c (K x R)  = V_c^T (K x N) C_c (N x R)
//
// (the block orthonormalisation is in ortho.cu)
// The basis is kept block-major, basis_blk[c][i][k], k = sb*dof + a with sb the
// lexicographic in-block site index (CoarseningLookupTableRework.h:156-163),
// so one block's N x K panel is contiguous.  Fine fields stay in the caller's
// [site][rhs][dof] layout and are gathered through blk_sites[c][sb].
#include <algorithm>
#include <type_traits>

#include "f64_mma.cuh"
#include "gmg_internal.cuh"

namespace gmg {

template <class T> struct ctype;
template <> struct ctype<double> { typedef double2 t; };
template <> struct ctype<float> { typedef float2 t; };

// ---------------------------------------------------------------------------
// tables and basis layout
// ---------------------------------------------------------------------------
gmg_status agg_build_tables(gmg_agg* h, cudaStream_t s) {
  const int64_t Vc = h->cdims.vol();
  std::vector<int32_t> t(Vc * h->bv);
  for (int64_t sc = 0; sc < Vc; ++sc) {
    int cc[4];
    int64_t q = sc;
    for (int d = 0; d < 4; ++d) { cc[d] = (int)(q % h->cdims.d[d]); q /= h->cdims.d[d]; }
    for (int sb = 0; sb < h->bv; ++sb) {
      int cb[4], cf[4];
      int r = sb;
      for (int d = 0; d < 4; ++d) { cb[d] = r % h->b[d]; r /= h->b[d]; }
      for (int d = 0; d < 4; ++d) cf[d] = cc[d] * h->b[d] + cb[d];
      int64_t sf = 0;
      for (int d = 3; d >= 0; --d) sf = sf * h->fdims.d[d] + cf[d];
      t[sc * h->bv + sb] = (int32_t)sf;
    }
  }
  GMG_TRY(h->blk_sites.alloc(t.size() * sizeof(int32_t)));
  GMG_CUDA(cudaMemcpyAsync(h->blk_sites.p, t.data(), t.size() * sizeof(int32_t),
                           cudaMemcpyHostToDevice, s));
  GMG_CUDA(cudaStreamSynchronize(s));
  return GMG_OK;
}

// basis [i][site][dof] <-> basis_blk [c][i][sb*dof + a].  Bound by HBM, both sides
// once.  A thread keeps one (c, sb*dof + a), whose place in either layout it works
// out once, and walks basis vectors blockIdx.y, + gridDim.y, ..., eight requests at
// a time (U; one where a thread has few): 32^4 x 12, nbasis 32, 2.32 -> 1.94 ms in and
// 2.28 -> 2.00 ms back, 6.4 to 6.6 TB/s, against one element a thread and step with its
// divisions.
template <bool TO_BLK, int U>
__global__ void __launch_bounds__(256) basis_layout_kernel(const double2* __restrict__ src, double2* __restrict__ dst,
                                                           const int32_t* __restrict__ blk_sites, int64_t Vc, int N,
                                                           int bv, int dof, int64_t Vf) {
  const int64_t K = (int64_t)bv * dof, e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= Vc * K) return;
  const int64_t c = e / K, k = e - c * K, sb = k / dof;
  const int64_t blk = c * N * K + k, nat = blk_sites[c * bv + sb] * (int64_t)dof + (k - sb * dof);
  const double2* in = src + (TO_BLK ? nat : blk);
  double2* out = dst + (TO_BLK ? blk : nat);
  const int64_t si = TO_BLK ? Vf * dof : K, so = TO_BLK ? K : Vf * dof;
  for (int i0 = blockIdx.y; i0 < N; i0 += U * gridDim.y) {
    double2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * (int)gridDim.y < N) v[u] = __ldcs(in + (i0 + u * (int)gridDim.y) * si);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * (int)gridDim.y < N) __stcs(out + (i0 + u * (int)gridDim.y) * so, v[u]);
  }
}

template <bool TO_BLK>
static gmg_status basis_layout(gmg_agg* h, const double2* src, double2* dst, cudaStream_t s) {
  const int64_t Vc = h->cdims.vol(), n = (Vc * h->bv * h->dof + 255) / 256;
  // the basis vectors split over CTAs only while those do not fill the chip (256 sites x
  // 12, nbasis 8, out: 4.1 us by one CTA per 256 elements, 3.5 by eight)
  const int64_t most = std::max<int64_t>(1, 148 * 8 / n);
  int split = (int)std::min<int64_t>((h->N + 7) / 8, most);
  if (n * split < 148 * 2) split = (int)std::min<int64_t>(h->N, most);
  GMG_CHECK(n < ((int64_t)1 << 31), GMG_ERR_UNSUPPORTED, "basis layout: lattice too large");
  auto kern = h->N < 4 * split ? basis_layout_kernel<TO_BLK, 1> : basis_layout_kernel<TO_BLK, 8>;
  kern<<<dim3((unsigned)n, split), 256, 0, s>>>(src, dst, h->blk_sites.as<int32_t>(), Vc, h->N, h->bv, h->dof,
                                                h->fdims.vol());
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

gmg_status agg_basis_to_blocked(gmg_agg* h, const double* basis_dev, cudaStream_t s) {
  const int64_t total = h->cdims.vol() * h->N * (int64_t)h->bv * h->dof;
  GMG_TRY(h->basis_blk.alloc(total * sizeof(double2)));
  GMG_TRY(basis_layout<true>(h, reinterpret_cast<const double2*>(basis_dev), h->basis_blk.as<double2>(), s));
  h->basis_f_ok = false;
  h->basis_tc_ok = false;
  // a new basis: the failure flag of the previous orthonormalisation no longer applies
  if (h->ortho_ws.p) GMG_CUDA(cudaMemsetAsync(h->ortho_ws.p, 0, sizeof(int), s));
  return GMG_OK;
}

gmg_status agg_basis_from_blocked(gmg_agg* h, double* basis_dev, cudaStream_t s) {
  return basis_layout<false>(h, h->basis_blk.as<double2>(), reinterpret_cast<double2*>(basis_dev), s);
}

__global__ void d2f_kernel(const double2* __restrict__ a, float2* __restrict__ b, int64_t n) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    b[e] = make_float2((float)a[e].x, (float)a[e].y);
}

gmg_status agg_prepare_f32(gmg_agg* h, cudaStream_t s) {
  if (h->basis_f_ok) return GMG_OK;
  const int64_t n = h->cdims.vol() * h->N * (int64_t)h->bv * h->dof;
  GMG_TRY(h->basis_blk_f.alloc(n * sizeof(float2)));
  d2f_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 64), 256, 0, s>>>(
      h->basis_blk.as<double2>(), h->basis_blk_f.as<float2>(), n);
  GMG_CUDA(cudaGetLastError());
  h->basis_f_ok = true;
  return GMG_OK;
}

// ---------------------------------------------------------------------------
// project: out[c][r][i] = sum_k conj(V[c][i][k]) F[site(c,k)][r][k % dof]
// on the FP64 tensor cores (f64_mma.cuh), FP64 fields and FP32 ones widened on
// load.  CTA per block; a unit is 8 MT basis vectors and 4 RQ right-hand sides,
// a warp sums the unit over the block's sites ks, ks + KS, ... with the operands
// of the next step requested one step ahead, and the KS warps of a unit add
// their tiles through shared memory in a fixed order.
// What bounds it: the MMA rate (8 N R flops per 16 (N + R) bytes: above about 8
// right-hand sides the arithmetic takes longer than the reads).  The register-
// tiled CUDA-core kernels before it were bound by shared-memory operand reads
// and staging.  32^4, nbasis 32, 32 RHS, 4^4 blocks, FP64:
// 7.27 -> 3.69 ms (28 TFLOP/s of 37); 16^4, nbasis 24, 12 RHS: 534 -> 95 us, in
// FP32 2428 -> 84 us.
// sel (nullable, nsel entries): the in-block site indices the sum runs over,
// the same for every block (a face of the block); without it all bv sites.
// The result goes to out[c * cstr + r * rstr + i * istr].
// ---------------------------------------------------------------------------
template <class Cx> struct ProjArgs {
  const Cx* basis;
  const int32_t* blk_sites;
  const Cx* fine;
  Cx* out;
  int64_t cstr, rstr, istr;
  int N, dof, bv, nrhs;
  const int32_t* sel;
  int nsel;
  // fine[site * fsite + r * frhs + k * fk].  face >= 0: a face field of the
  // Wilson operator's hop `face` instead, sites c * nsel + s, with the upper two
  // spins only; the lower two are phases times upper ones (see face_spin), so
  // that the sum runs over the upper components and conj(v_upper) + phase
  // conj(v_lower): half the MMAs, two sites of 6 components a turn.  32^4, 4^4
  // blocks, nbasis 40, one face of 40 vectors: 1.56 -> 1.34 ms.
  int64_t fsite;
  int frhs, fk, face;
  int units, rchunks, G, KS;
};

constexpr int kProjWarps = 8;
// blocks of so many components (a row of 4 GiB in FP64) take the kernels' forms with
// 64-bit offsets, which need more registers per load
constexpr int64_t kWideBlock = (int64_t)1 << 28;

// The lower spin *low of (1 -+ gamma_mu) psi that is a phase (code 0: 1, 1: i, 2:
// -1, 3: -i) times upper spin s, for hop p (p < 4: +mu, the projector 1 -
// gamma_mu; p >= 4: -mu, 1 + gamma_mu), in the gamma basis of the fine operator.
__device__ __forceinline__ int face_spin(int p, int s, int* low) {
  const int mu = p & 3;
  *low = mu < 2 ? 3 - s : s + 2;
  const int g = mu == 0 ? 3 : mu == 1 ? (*low == 3 ? 2 : 0) : mu == 2 ? (*low == 3 ? 1 : 3) : 0;
  return (g + (p < 4 ? 2 : 0)) & 3;
}

// WIDE: in-block offsets in 64 bits, for blocks of 2^28 components or more
template <class T, int MT, int RQ, bool FACE, bool WIDE = false>
__global__ void __launch_bounds__(32 * kProjWarps) project_mma_kernel(const ProjArgs<typename ctype<T>::t> a) {
  typedef typename ctype<T>::t Cx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int N = a.N, dof = a.dof, ks = warp % a.KS, g = warp / a.KS, u = blockIdx.y * a.G + g;
  const int mc = u / a.rchunks, rc = u - mc * a.rchunks;
  const int kk = lane & 3, part = (lane >> 2) & 1;
  const int64_t c = blockIdx.x, K = (int64_t)a.bv * dof;
  const int nsites = FACE ? (a.nsel + 1) / 2 : a.sel ? a.nsel : a.bv;  // pairs of sites of a face
  double acc[MT][RQ][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int q = 0; q < RQ; ++q) acc[m][q][0] = acc[m][q][1] = 0.0;

  if (u < a.units && ks < nsites) {
    // rows and right-hand sides past the end repeat the last one; their results are not stored
    const Cx* Vb = a.basis + c * N * K;
    const int32_t* blk = a.blk_sites + c * a.bv;
    typedef typename std::conditional<WIDE, uint64_t, uint32_t>::type Off;
    Off row[MT];
    int foff[RQ];
    const Off Kb = (Off)(K * sizeof(Cx));
#pragma unroll
    for (int m = 0; m < MT; ++m) row[m] = min((mc * MT + m) * 8 + (lane >> 2), N - 1);
#pragma unroll
    for (int q = 0; q < RQ; ++q) foff[q] = min((rc * RQ + q) * 4 + (lane >> 3), a.nrhs - 1) * a.frhs;
    const uint32_t s1 = f64mma::second_sign(part, true);
    int low0 = 0, low1 = 0, code0 = 0, code1 = 0;
    if (FACE) {
      code0 = face_spin(a.face, 0, &low0);
      code1 = face_spin(a.face, 1, &low1);
    }
    constexpr int AT = FACE ? 2 * MT : MT;  // FACE: the upper components, then the lower ones
    Cx av[2][AT], fv[2][RQ];
    int s = ks, k4 = 0, kc = kk, left = (nsites - ks + a.KS - 1) / a.KS * ((dof + 3) / 4);
    // the site requested next and the one after it (FACE: the pair's second site is sc)
    auto second = [&](int pair) { return 2 * pair + 1 < a.nsel ? a.sel[2 * pair + 1] : -1; };
    int sb = FACE ? a.sel[2 * s] : a.sel ? a.sel[s] : s, sf = FACE ? s : blk[sb], sc = FACE ? second(s) : 0;
    int sb1 = 0, sf1 = 0, sc1 = 0;
    const Cx *Vp, *Fp;
    auto at_site = [&]() {
      Vp = Vb + (int64_t)sb * dof;
      Fp = a.fine + (FACE ? c * a.nsel + 2 * sf : (int64_t)sf) * a.fsite;
      s += a.KS;
      if (s < nsites) {
        sb1 = FACE ? a.sel[2 * s] : a.sel ? a.sel[s] : s;
        sf1 = FACE ? s : blk[sb1];
        if (FACE) sc1 = second(s);
      }
    };
    auto request = [&](Cx (&A)[AT], Cx (&F)[RQ]) {
      int k = k4 + kk;
      bool in_k = k < dof;
      const Cx *V = Vp, *Ff = Fp;
      if (FACE && k >= 6) {
        k -= 6;
        in_k = sc >= 0;
        if (in_k) {
          V = Vb + (int64_t)sc * dof;
          Ff = Fp + a.fsite;
        }
      }
      auto basis = [&](int m, int at) {
        return in_k ? __ldg(reinterpret_cast<const Cx*>(reinterpret_cast<const char*>(V + at) + (uint64_t)row[m] * Kb))
                    : Cx{0, 0};
      };
#pragma unroll
      for (int m = 0; m < MT; ++m) A[m] = basis(m, k);
      if constexpr (FACE) {
        const int kl = k < 3 ? 3 * low0 + k : 3 * low1 + k - 3;
#pragma unroll
        for (int m = 0; m < MT; ++m) A[MT + m] = basis(m, kl);
      }
#pragma unroll
      for (int q = 0; q < RQ; ++q) F[q] = in_k ? __ldg(Ff + foff[q] + k * a.fk) : Cx{0, 0};
      k4 += 4;
      if (k4 >= dof) {
        k4 = 0;
        sb = sb1;
        sf = sf1;
        sc = sc1;
        at_site();
      }
    };
    auto multiply = [&](const Cx (&A)[AT], const Cx (&F)[RQ]) {
      double b0[RQ], b1[RQ], ax[MT], ay[MT];
#pragma unroll
      for (int q = 0; q < RQ; ++q) f64mma::expand(F[q], part, 0u, s1, b0[q], b1[q]);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        ax[m] = (double)A[m].x;
        ay[m] = (double)A[m].y;
      }
      if constexpr (FACE) {
        // + conj(phase) v_lower, the phase as an exchange of the parts and signs: -i (x + i y) = y - i x
        const int code = kc % 6 < 3 ? code0 : code1;
        const bool swap = code & 1;
        const uint32_t nre = code >= 2 ? 0x80000000u : 0u, nim = nre ^ (swap ? 0x80000000u : 0u);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const Cx l = A[MT + m];
          ax[m] += f64mma::flip(swap ? l.y : l.x, nre);
          ay[m] += f64mma::flip(swap ? l.x : l.y, nim);
        }
        kc = kc + 4 >= dof ? kk : kc + 4;
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < RQ; ++q) f64mma::mma(acc[m][q], ax[m], b0[q]);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < RQ; ++q) f64mma::mma(acc[m][q], ay[m], b1[q]);
    };
    at_site();
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

  auto store = [&](int m, int q, double re, double im) {
    const int i = (mc * MT + m) * 8 + (lane >> 2), r = (rc * RQ + q) * 4 + kk;
    if (i >= N || r >= a.nrhs) return;
    Cx v;
    v.x = re;
    v.y = im;
    a.out[c * a.cstr + r * a.rstr + i * a.istr] = v;
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

template <class T, int MT, int RQ, bool FACE, bool WIDE = false>
static gmg_status launch_project(const ProjArgs<typename ctype<T>::t>& a, int Vc, cudaStream_t s) {
  auto kern = project_mma_kernel<T, MT, RQ, FACE, WIDE>;
  const size_t smem = a.KS == 1 ? 0 : sizeof(double2) * 32 * MT * RQ * (size_t)a.G * a.KS;
  if (smem > 48 * 1024)
    GMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  KernelTimer kt("project", s);
  kern<<<dim3(Vc, (a.units + a.G - 1) / a.G), 32 * a.G * a.KS, smem, s>>>(a);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

// Launch shape of the projection: w quads of right-hand sides per unit, G units
// and KS shares of the sites per CTA.  The grid's time in units of MMA work is
// estimated for every w, with the units of a block in one CTA (their operands
// meet in L1) or in CTAs of their own: CTAs in full waves of C per SM, the last
// wave with what is left; the basis read of a unit counts as half a quad, 0.4
// when shared.  Big tiles run in CTAs of 4 warps, so that two or three CTAs
// overlap each other's ends (32^4, nbasis 32, 32 RHS, FP64: 3.71 ms, 5.12 with
// 8), small tiles and part-filled chips in CTAs of 8 (16^4, nbasis 24, 12 RHS:
// 95 us, 118 with 4).  16^4, nbasis 32, 32 RHS: 290 us with w = 2 and own CTAs,
// 376 with w = 4 and shared ones; 8^4 with 16 blocks, nbasis 24, 24 RHS: 37 us
// with w = 1, 98 with w = 3.  A face reads its basis twice as fast per MMA and
// holds two loads a row: with blocks enough to fill the chip several times over,
// the units of a block share a CTA, tiles of up to 3 quads (32^4, 40 columns:
// 1.34 ms; 1.84 in CTAs of their own, 1.49 with w = 5).
struct ProjShape {
  int w, chunks, G, KS;
};
static ProjShape project_shape(int Vc, int MT, int mchunks, int rq, bool face) {
  ProjShape best{1, rq, 1, kProjWarps};
  double t_best = 1e30;
  face = face && Vc >= 148 * 8;
  for (int w = 1; w <= std::min(face ? 3 : 5, rq); ++w) {
    const int chunks = (rq + w - 1) / w, units = mchunks * chunks;
    const int regs = (40 + 4 * MT * w + 8 * MT + 8 * w + 7) / 8 * 8;
    for (int shared = face ? 1 : 0; shared < 2; ++shared) {
      int warps = MT * w > 10 ? 4 : kProjWarps;
      int G = shared ? std::min(units, warps) : 1;
      int64_t ctas = (int64_t)Vc * ((units + G - 1) / G);
      if (ctas < 2 * 148) {
        warps = kProjWarps;
        G = shared ? std::min(units, warps) : 1;
        ctas = (int64_t)Vc * ((units + G - 1) / G);
      }
      const int C = std::max(1, 65536 / 32 / regs / warps);
      const double work = G * MT * (w + (G > 1 ? 0.4 : 0.5)) * (C > 1 ? 1.0 : 1.25);
      const int64_t rest = ctas % (148 * C);
      const double t = work * (ctas / (148 * C) * C + (rest + 147) / 148);
      if (t <= t_best) {
        t_best = t;
        best = ProjShape{w, chunks, G, warps / G};
      }
    }
  }
  return best;
}

// cmajor: fine is a component-major field [site][dof][nrhs] (else [site][nrhs][dof]);
// FACE: a component-major field of the faces (see ProjArgs)
template <class T, bool FACE = false>
static gmg_status project_mma(gmg_agg* h, const void* basis, int nrhs, const void* fine, bool cmajor, int face,
                              void* out, int64_t cstr, int64_t rstr, int64_t istr, const int32_t* sel, int nsel,
                              cudaStream_t s) {
  typedef typename ctype<T>::t Cx;
  GMG_CHECK(sizeof(Cx) * 4 * h->dof * (size_t)(h->N + nrhs) <= 227 * 1024, GMG_ERR_UNSUPPORTED,
            "project: site dof x (nbasis + nrhs) too large");
  const bool wide = (int64_t)h->bv * h->dof >= kWideBlock;
  const int mt = (h->N + 7) / 8, mchunks = wide ? mt : (mt + 4) / 5, MT = (mt + mchunks - 1) / mchunks;
  const int Vc = (int)h->cdims.vol();
  const ProjShape sh = wide ? ProjShape{1, (nrhs + 3) / 4, 1, kProjWarps}
                            : project_shape(Vc, MT, mchunks, (nrhs + 3) / 4, FACE);
  const ProjArgs<Cx> a{reinterpret_cast<const Cx*>(basis), h->blk_sites.as<int32_t>(),
                       reinterpret_cast<const Cx*>(fine), reinterpret_cast<Cx*>(out), cstr, rstr, istr, h->N, h->dof,
                       h->bv, nrhs, sel, nsel, (int64_t)nrhs * (FACE ? 6 : h->dof), cmajor ? 1 : h->dof,
                       cmajor ? nrhs : 1, face, mchunks * sh.chunks, sh.chunks, sh.G, sh.KS};
  if (wide) return launch_project<T, 1, 1, FACE, true>(a, Vc, s);
  auto by_rq = [&](auto mtc) -> gmg_status {
    constexpr int M = decltype(mtc)::value;
    switch (sh.w) {
      case 1: return launch_project<T, M, 1, FACE>(a, Vc, s);
      case 2: return launch_project<T, M, 2, FACE>(a, Vc, s);
      case 3: return launch_project<T, M, 3, FACE>(a, Vc, s);
      case 4: return launch_project<T, M, 4, FACE>(a, Vc, s);
      default: return launch_project<T, M, 5, FACE>(a, Vc, s);
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

gmg_status agg_project(gmg_agg* h, int compute, int vec_prec, int nrhs, const void* fine, void* coarse,
                       cudaStream_t s) {
  if (compute == GMG_BF16 && vec_prec == GMG_F32) return agg_project_tc(h, nrhs, (const float*)fine, (float*)coarse, s);
  GMG_CHECK(compute == vec_prec, GMG_ERR_UNSUPPORTED, "project: compute and vector precision differ");
  const int64_t N = h->N;
  if (compute == GMG_F64)
    return project_mma<double>(h, h->basis_blk.p, nrhs, fine, false, -1, coarse, nrhs * N, N, 1, nullptr, 0, s);
  if (compute == GMG_F32) {
    GMG_TRY(agg_prepare_f32(h, s));
    return project_mma<float>(h, h->basis_blk_f.p, nrhs, fine, false, -1, coarse, nrhs * N, N, 1, nullptr, 0, s);
  }
  return fail(GMG_ERR_UNSUPPORTED, "project: unsupported precision");
}

// FP64 projection over a subset of every block's sites (sel: nsel in-block
// indices on the device, the same for all blocks; null: all of them), written
// as columns i0 .. i0 + nrhs of the link matrices A[c][i][column].  face >= 0: of
// the face field of the Wilson operator's hop `face` (wilson_face_half).
gmg_status agg_project_links(gmg_agg* h, int nrhs, const double* fine, bool cmajor, int face, double* A, int i0,
                             const int32_t* sel, int nsel, cudaStream_t s) {
  const int64_t N = h->N;
  double2* out = reinterpret_cast<double2*>(A) + i0;
  if (face >= 0)
    return project_mma<double, true>(h, h->basis_blk.p, nrhs, fine, true, face, out, N * N, 1, N, sel, nsel, s);
  return project_mma<double>(h, h->basis_blk.p, nrhs, fine, cmajor, -1, out, N * N, 1, N, sel, nsel, s);
}

// ---------------------------------------------------------------------------
// promote: F[site(c,k)][r][k%dof] = sum_i V[c][i][k] C[c][r][i]
// on the FP64 tensor cores: rows k (8 KT per warp and turn), contraction i.  A
// block's coarse vectors are expanded once per CTA into MMA operand order in
// shared memory; the basis is read straight from global memory, each element
// once per chunk of 4 RQ right-hand sides, one step ahead.
// What bounds it: the MMA rate, as the projection.  32^4, nbasis 32, 32 RHS,
// 4^4 blocks, FP64: 9.64 -> 3.52 ms (29 TFLOP/s of 37); 16^4, nbasis 24, 12 RHS:
// 946 -> 96 us.
// ---------------------------------------------------------------------------
template <class Cx> struct PromArgs {
  const Cx* basis;
  const int32_t* blk_sites;
  const Cx* coarse;
  Cx* fine;
  int N, dof, bv, nrhs, rq;  // rq: quads of the shared-memory table
  int rlim;                  // right-hand sides from `coarse` and `fine` on (nrhs: their stride)
};

// PART: a part of the right-hand sides, the first a.rlim from a.coarse and a.fine on
template <class T, int KT, int RQ, bool WIDE = false, bool PART = false>
__global__ void __launch_bounds__(256) promote_mma_kernel(const PromArgs<typename ctype<T>::t> a) {
  typedef typename ctype<T>::t Cx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* Bs = reinterpret_cast<double2*>(smem_raw);  // [steps][rq][32]: (first, second) operand of every lane
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kk = lane & 3;
  const int N = a.N, dof = a.dof, steps = (N + 3) / 4;
  const int64_t c = blockIdx.x;
  typedef typename std::conditional<WIDE, int64_t, int>::type Idx;
  const Idx K = (Idx)a.bv * dof;
  for (int e = threadIdx.x; e < steps * a.rq * 32; e += blockDim.x) {
    const int l = e & 31, q = (e >> 5) % a.rq, st = (e >> 5) / a.rq;
    const int i = 4 * st + (l & 3), r = q * 4 + (l >> 3), part = (l >> 2) & 1;
    Cx v{0, 0};
    if (i < N && r < (PART ? a.rlim : a.nrhs)) v = a.coarse[(c * a.nrhs + r) * N + i];
    double2 b;
    f64mma::expand(v, part, 0u, f64mma::second_sign(part, false), b.x, b.y);
    Bs[e] = b;
  }
  __syncthreads();
  const Cx* Vb = a.basis + c * N * (int64_t)K;
  const int32_t* blk = a.blk_sites + c * a.bv;
  const Idx ngroups = (K + 8 * KT - 1) / (8 * KT);
  const int nwarps = (blockDim.x >> 5) * gridDim.y;
  const int chunks = a.rq / RQ;
  for (Idx item = blockIdx.y * (blockDim.x >> 5) + warp; item < ngroups * chunks; item += nwarps) {
    const Idx grp = item / chunks;
    const int q0 = (int)(item - grp * chunks) * RQ;
    double acc[KT][RQ][2];
#pragma unroll
    for (int t = 0; t < KT; ++t)
#pragma unroll
      for (int q = 0; q < RQ; ++q) acc[t][q][0] = acc[t][q][1] = 0.0;
    const Idx k0 = grp * 8 * KT + (lane >> 2);
    int sf[KT], at[KT];  // site and component of this lane's rows
    const Cx* Vp[KT];
#pragma unroll
    for (int t = 0; t < KT; ++t) {
      const Idx k = min(k0 + 8 * t, K - 1);
      const int sb = (int)(k / dof);
      sf[t] = blk[sb];
      at[t] = (int)(k - (Idx)sb * dof);
      Vp[t] = Vb + k;
    }
    Cx av[2][KT];
    auto request = [&](Cx (&A)[KT], int st) {
      const int i = 4 * st + kk;
#pragma unroll
      for (int t = 0; t < KT; ++t) A[t] = i < N ? __ldg(Vp[t] + (int64_t)i * K) : Cx{0, 0};
    };
    auto multiply = [&](const Cx (&A)[KT], int st) {
      const double2* B = Bs + (st * a.rq + q0) * 32 + lane;
#pragma unroll
      for (int q = 0; q < RQ; ++q) {
        const double2 b = B[q * 32];
#pragma unroll
        for (int t = 0; t < KT; ++t) f64mma::mma(acc[t][q], (double)A[t].x, b.x);
#pragma unroll
        for (int t = 0; t < KT; ++t) f64mma::mma(acc[t][q], (double)A[t].y, b.y);
      }
    };
    request(av[0], 0);
    for (int st = 0; st < steps; st += 2) {
      if (st + 1 < steps) request(av[1], st + 1);
      multiply(av[0], st);
      if (st + 1 == steps) break;
      if (st + 2 < steps) request(av[0], st + 2);
      multiply(av[1], st + 1);
    }
#pragma unroll
    for (int t = 0; t < KT; ++t) {
      if (k0 + 8 * t >= K) continue;
#pragma unroll
      for (int q = 0; q < RQ; ++q) {
        const int r = (q0 + q) * 4 + kk;
        if (r >= (PART ? a.rlim : a.nrhs)) continue;
        Cx v;
        v.x = acc[t][q][0];
        v.y = acc[t][q][1];
        a.fine[((int64_t)sf[t] * a.nrhs + r) * dof + at[t]] = v;
      }
    }
  }
}

template <class T, int KT, int RQ, bool WIDE = false, bool PART = false>
static gmg_status launch_promote(PromArgs<typename ctype<T>::t> a, int Vc, cudaStream_t s) {
  auto kern = promote_mma_kernel<T, KT, RQ, WIDE, PART>;
  const int launches = PART ? a.rq / RQ : 1;  // PART: a chunk of right-hand sides each
  if (PART) a.rq = RQ;
  const size_t smem = sizeof(double2) * 32 * (size_t)((a.N + 3) / 4) * a.rq;
  if (smem > 48 * 1024)
    GMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // 8 warps per CTA; few blocks are split over several CTAs, up to 6 per SM with
  // 3 turns a warp or more (256 blocks, nbasis 32, 32 RHS: 252 us at 4, 276 at 1;
  // 16 blocks, nbasis 24, 24 RHS: 18 us at 8, 97 at 1).  A block with no more than one
  // item a warp takes CTAs of fewer warps where that keeps more of them busy and on an
  // SM, which then overlap each other's tables and ends (4096 blocks of 2^4 x 12, nbasis
  // 16, 16 RHS, FP32: 180 us with 8, 97 with 2; FP64 nbasis 2, 1 RHS: 24 and 15).
  const int64_t items = ((int64_t)a.bv * a.dof + 8 * KT - 1) / (8 * KT) * (a.rq / RQ);
  int nw = 8;
  if (items <= 8) {
    // registers a thread, as compiled by nvcc 12.9 (a wrong entry costs speed only)
    static const int tab[2][8] = {{88, 112, 128, 144, 128, 112, 120, 120}, {80, 104, 128, 144, 128, 104, 120, 120}};
    const int regs = tab[sizeof(T) == 8 ? 0 : 1][RQ - 1];
    double most = 0.0;
    for (const int n : {8, 6, 4, 3, 2}) {
      const int64_t C = std::max<int64_t>(1, std::min<int64_t>(65536 / (32 * regs * n), 227 * 1024 / (smem + 1024)));
      const double busy = (double)std::min<int64_t>(C, (Vc + 147) / 148) * items / ((items + n - 1) / n);
      if (busy > 1.2 * most) {
        most = busy;
        nw = n;
      }
    }
  }
  const int split = (int)std::max<int64_t>(1, std::min<int64_t>((items + 3 * nw - 1) / (3 * nw), (148 * 48 / nw + Vc - 1) / Vc));
  KernelTimer kt("promote", s);
  for (int k = 0; k < launches; ++k) {
    kern<<<dim3(Vc, split), 32 * nw, smem, s>>>(a);
    a.coarse += (int64_t)4 * RQ * a.N;
    a.fine += (int64_t)4 * RQ * a.dof;
    a.rlim -= 4 * RQ;
  }
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

template <class T>
static gmg_status promote_mma(gmg_agg* h, const void* basis, int nrhs, const void* coarse, void* fine,
                              cudaStream_t s) {
  typedef typename ctype<T>::t Cx;
  GMG_CHECK(sizeof(Cx) * ((size_t)h->N * nrhs + (size_t)h->N * 4 * h->dof) <= 227 * 1024, GMG_ERR_UNSUPPORTED,
            "promote: nbasis x (nrhs + site dof) too large");
  // quads per warp: the fewest padded ones (each chunk reads the basis once
  // more, counted as half a quad)
  const int rq = (nrhs + 3) / 4;
  int w = 1, chunks = rq;
  for (int v = 2; v <= 8; ++v) {
    const int u = (rq + v - 1) / v;
    if (u * (2 * v + 1) <= chunks * (2 * w + 1)) {
      w = v;
      chunks = u;
    }
  }
  PromArgs<Cx> a{reinterpret_cast<const Cx*>(basis), h->blk_sites.as<int32_t>(), reinterpret_cast<const Cx*>(coarse),
                 reinterpret_cast<Cx*>(fine), h->N, h->dof, h->bv, nrhs, w * chunks, nrhs};
  const int Vc = (int)h->cdims.vol();
  if ((int64_t)h->bv * h->dof >= kWideBlock) {
    a.rq = rq;
    return launch_promote<T, 4, 1, true>(a, Vc, s);
  }
  // a table that leaves room for one CTA on an SM only (nbasis above 56, 57 right-hand
  // sides and more) is made by chunk, one launch each, where blocks enough for both wait
  // (4096 blocks of 2^4 x 12, nbasis 64, 64 RHS, FP32: 1490 us with all of it, 1070)
  if (Vc >= 148 * 2 && sizeof(double2) * 32 * (size_t)((h->N + 3) / 4) * a.rq > 112 * 1024)
    return w == 5 ? launch_promote<T, 3, 5, false, true>(a, Vc, s) : launch_promote<T, 2, 8, false, true>(a, Vc, s);
  switch (w) {
    case 1: return launch_promote<T, 4, 1>(a, Vc, s);
    case 2: return launch_promote<T, 4, 2>(a, Vc, s);
    case 3: return launch_promote<T, 4, 3>(a, Vc, s);
    case 4: return launch_promote<T, 4, 4>(a, Vc, s);
    case 5: return launch_promote<T, 3, 5>(a, Vc, s);
    case 6: return launch_promote<T, 2, 6>(a, Vc, s);
    case 7: return launch_promote<T, 2, 7>(a, Vc, s);
    default: return launch_promote<T, 2, 8>(a, Vc, s);
  }
}

gmg_status agg_promote(gmg_agg* h, int compute, int vec_prec, int nrhs, const void* coarse,
                       void* fine, cudaStream_t s) {
  if (compute == GMG_BF16 && vec_prec == GMG_F32) return agg_promote_tc(h, nrhs, (const float*)coarse, (float*)fine, s);
  GMG_CHECK(compute == vec_prec, GMG_ERR_UNSUPPORTED, "promote: compute and vector precision differ");
  if (compute == GMG_F64) return promote_mma<double>(h, h->basis_blk.p, nrhs, coarse, fine, s);
  if (compute == GMG_F32) {
    GMG_TRY(agg_prepare_f32(h, s));
    return promote_mma<float>(h, h->basis_blk_f.p, nrhs, coarse, fine, s);
  }
  return fail(GMG_ERR_UNSUPPORTED, "promote: unsupported precision");
}

}  // namespace gmg
