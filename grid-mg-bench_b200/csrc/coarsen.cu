// coarsen.cu -- Galerkin coarse-operator construction on the GPU (FP64).
//
// Restates CoarsenedMatrix::CoarsenOperator in its direction-saving form
// (include/CoarsenedMatrixUpstreamImprovedDirsaveLut.h:927-1097, multi-RHS
// batching of the fine applies as in ...LutMRHS.h:1004-1101):
//
//   for a batch of basis vectors phi_i (the fine operator sees them as RHS):
//     W_p = Mdir_p phi,               p = 4..7 (disp = -1)
//     A_p(c)[j][i] = sum_{x in c, x_dir mod b == 0} <v_j(x), W_p(x)>
//     W_8 = e*M(e phi) + o*M(o phi)   (block even/odd trick, :1053-1067)
//     A_8(c)[j][i] = sum_{x in c} <v_j(x), W_8(x)>
//   then A_{+mu}(x) = S o A_{-mu}(x+mu)^dag  (ConstructRemainingLinks, :1164-1196)
//
// The fine operator is either the Wilson-clover operator or, for
// coarse-of-coarse, the coarse stencil of the level above (its MdirCalc is the
// "fine" Mdir, ...Lut.h:820-860).
#include <algorithm>

#include "gmg_internal.cuh"

namespace gmg {

// field[sf][r][a] = basis_blk[c][i0 + r][sb*dof + a]
__global__ void basis_gather_kernel(const double2* __restrict__ basis_blk, const int32_t* __restrict__ blk_sites,
                                    double2* __restrict__ field, int64_t Vc, int N, int bv, int dof, int i0,
                                    int nb) {
  const int64_t K = (int64_t)bv * dof;
  const int64_t total = Vc * nb * K;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = e % K;
    const int r = (int)((e / K) % nb);
    const int64_t c = e / (K * nb);
    const int64_t sf = blk_sites[c * bv + k / dof];
    field[(sf * nb + r) * dof + k % dof] = basis_blk[(c * N + i0 + r) * K + k];
  }
}

// The component-major form of a spin-colour field, field[sf][a][r]: a CTA
// transposes kGatherSites sites of a block through shared memory, runs of 16 x
// kGatherSites components in and whole lines of nb right-hand sides out.  (The
// element-wise gather above: 3.13 ms at 32^4 x 40 vectors for 16.1 GB.)
constexpr int kGatherSites = 4;
__global__ void __launch_bounds__(256) basis_gather_cm_kernel(const double2* __restrict__ basis_blk,
                                                              const int32_t* __restrict__ blk_sites,
                                                              double2* __restrict__ field, int N, int bv, int i0,
                                                              int nb) {
  constexpr int KC = 12 * kGatherSites;
  extern __shared__ __align__(16) double2 tile[];  // [KC][nb + 1]
  const int chunks = (bv + kGatherSites - 1) / kGatherSites;
  const int64_t c = blockIdx.x / chunks, K = (int64_t)bv * 12;
  const int sb0 = (int)(blockIdx.x % chunks) * kGatherSites, kc = min(KC, (int)(K - sb0 * 12));
  const double2* src = basis_blk + (c * N + i0) * K + sb0 * 12;
  for (int e = threadIdx.x; e < nb * KC; e += blockDim.x) {
    const int r = e / KC, k = e - r * KC;
    if (k < kc) tile[k * (nb + 1) + r] = src[r * K + k];
  }
  __syncthreads();
  for (int sl = 0; sl * 12 < kc; ++sl) {
    double2* dst = field + (int64_t)blk_sites[c * bv + sb0 + sl] * 12 * nb;
    for (int e = threadIdx.x; e < 12 * nb; e += blockDim.x) {
      const int a = e / nb, r = e - a * nb;
      dst[e] = tile[(sl * 12 + a) * (nb + 1) + r];
    }
  }
}

static int gsz(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>((n + 255) / 256, 1), 148 * 64); }

// The fine operator, the Wilson-clover operator or a coarse stencil, on the
// fields of its own layout: [site][12][r] or [site][r][dof].
struct FineOpRef {
  gmg_wilson* w = nullptr;
  gmg_coarse* c = nullptr;
  int dof() const { return w ? 12 : c->N; }
  const Dims& dims() const { return w ? w->dims : c->dims; }
  // field = basis vectors [i0, i0 + nb)
  gmg_status gather(gmg_agg* agg, int i0, int nb, double* field, cudaStream_t s) const {
    const int64_t Vc = agg->cdims.vol();
    if (w) {
      const size_t smem = sizeof(double2) * 12 * kGatherSites * (nb + 1);
      if (smem > 48 * 1024)
        GMG_CUDA(cudaFuncSetAttribute(basis_gather_cm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      basis_gather_cm_kernel<<<(unsigned)(Vc * ((agg->bv + kGatherSites - 1) / kGatherSites)), 256, smem, s>>>(
          agg->basis_blk.as<double2>(), agg->blk_sites.as<int32_t>(), reinterpret_cast<double2*>(field), agg->N,
          agg->bv, i0, nb);
    } else {
      basis_gather_kernel<<<gsz(Vc * nb * agg->bv * dof()), 256, 0, s>>>(
          agg->basis_blk.as<double2>(), agg->blk_sites.as<int32_t>(), reinterpret_cast<double2*>(field), Vc, agg->N,
          agg->bv, dof(), i0, nb);
    }
    GMG_CUDA(cudaGetLastError());
    return GMG_OK;
  }
  // the hop of point p on the face sites of every block, projected into the links A of p
  gmg_status face(gmg_agg* agg, int p, int nb, const double* in, double* tmp, double* A, int i0, const int32_t* sites,
                  int n, const int32_t* sel, int nsel, cudaStream_t s) const {
    if (w) {
      GMG_TRY(wilson_face_half(w, p, nb, in, tmp, agg->blk_sites.as<int32_t>(), agg->cdims.vol(), agg->bv, sel, nsel, s));
      return agg_project_links(agg, nb, tmp, true, p, A, i0, sel, nsel, s);
    }
    GMG_TRY(coarse_apply_sel_f64(c, p, p + 1, nb, in, tmp, sites, n, nullptr, s));
    return agg_project_links(agg, nb, tmp, false, -1, A, i0, sel, nsel, s);
  }
  // the operator without the hops whose bit is set in hskip (per site), projected into the self links A
  gmg_status self(gmg_agg* agg, int nb, const double* in, double* tmp, double* A, int i0, const uint8_t* hskip,
                  cudaStream_t s) const {
    if (w)
      GMG_TRY(wilson_apply_masked(w, nb, in, tmp, agg->blk_sites.as<int32_t>(), hskip, s));
    else
      GMG_TRY(coarse_apply_sel_f64(c, 0, 9, nb, in, tmp, nullptr, 0, hskip, s));
    return agg_project_links(agg, nb, tmp, w != nullptr, -1, A, i0, nullptr, 0, s);
  }
};

// Workspace of the construction, built on the first call and kept in the
// aggregation (by the coarse-of-coarse form up to kKeptBytes): the batch size comes from the free memory then (two
// fields of it in a third of it, at most 40 GB), the face lists and block
// parities from the geometry.
constexpr size_t kKeptBytes = (size_t)1 << 30;
static gmg_status coarsen_workspace(gmg_agg* agg, cudaStream_t s) {
  if (agg->cw_nb > 0) return GMG_OK;
  const Dims& fd = agg->fdims;
  const int64_t Vf = fd.vol();
  const int N = agg->N, dof = agg->dof;
  size_t free_b = 0, total_b = 0;
  GMG_CUDA(cudaMemGetInfo(&free_b, &total_b));
  const double cap = std::min(40.0e9, (double)free_b / 3.0) / 2.0;
  int nb = N;
  while (nb > 1 && (double)Vf * nb * dof * 16.0 > cap) nb = (nb + 1) / 2;
  if (agg->cw_max_batch > 0) nb = std::min(nb, agg->cw_max_batch);
  const size_t fbytes = sizeof(double2) * (size_t)Vf * nb * dof;
  GMG_TRY(agg->cw_phi.alloc(fbytes));
  GMG_TRY(agg->cw_w.alloc(fbytes));
  std::vector<int32_t> face, sel;
  std::vector<uint8_t> bpar(Vf), hskip(Vf);
  for (int d = 0; d < 4; ++d) {
    agg->cw_nface[d] = 0;
    for (int64_t x = 0; x < Vf; ++x) {
      int64_t t = x;
      int c = 0;
      for (int q = 0; q <= d; ++q) {
        c = (int)(t % fd.d[q]);
        t /= fd.d[q];
      }
      if (c % agg->b[d] == 0) {
        face.push_back((int32_t)x);
        ++agg->cw_nface[d];
      }
    }
    agg->cw_nsel[d] = 0;
    for (int k = 0; k < agg->bv; ++k) {
      int t = k, lc[4];
      for (int q = 0; q < 4; ++q) {
        lc[q] = t % agg->b[q];
        t /= agg->b[q];
      }
      if (lc[d] == 0) {
        sel.push_back(k);
        ++agg->cw_nsel[d];
      }
    }
  }
  for (int64_t x = 0; x < Vf; ++x) {
    int64_t t = x;
    int par = 0;
    for (int q = 0; q < 4; ++q) {
      par += (int)(t % fd.d[q]) / agg->b[q];
      t /= fd.d[q];
    }
    bpar[x] = (uint8_t)(par & 1);
  }
  // hop p = (mu = p mod 4, +1 for p < 4, -1 otherwise), periodic neighbours
  int64_t stride[4] = {1, 1, 1, 1};
  for (int q = 1; q < 4; ++q) stride[q] = stride[q - 1] * fd.d[q - 1];
  for (int64_t x = 0; x < Vf; ++x) {
    uint8_t m = 0;
    for (int p = 0; p < 8; ++p) {
      const int mu = p & 3;
      const int xm = (int)((x / stride[mu]) % fd.d[mu]);
      const int ym = (xm + (p < 4 ? 1 : fd.d[mu] - 1)) % fd.d[mu];
      const int64_t y = x + (int64_t)(ym - xm) * stride[mu];
      if (bpar[y] != bpar[x]) m |= (uint8_t)(1u << p);
    }
    hskip[x] = m;
  }
  GMG_TRY(agg->cw_face.alloc(sizeof(int32_t) * face.size()));
  GMG_TRY(agg->cw_sel.alloc(sizeof(int32_t) * sel.size()));
  GMG_TRY(agg->cw_hskip.alloc(hskip.size()));
  GMG_CUDA(cudaMemcpyAsync(agg->cw_face.p, face.data(), sizeof(int32_t) * face.size(), cudaMemcpyHostToDevice, s));
  GMG_CUDA(cudaMemcpyAsync(agg->cw_sel.p, sel.data(), sizeof(int32_t) * sel.size(), cudaMemcpyHostToDevice, s));
  GMG_CUDA(cudaMemcpyAsync(agg->cw_hskip.p, hskip.data(), hskip.size(), cudaMemcpyHostToDevice, s));
  GMG_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
  agg->cw_nb = nb;
  return GMG_OK;
}

// CoarsenOperator.  Per batch of basis vectors: the backward hop Mdir_p
// evaluated on the face sites only (the only sites its face projection reads),
// and the self term e D e + o D o as one pass of the operator with the hops
// between blocks of opposite parity left out.  At every site the projections
// read, both give the sums of the masked full-lattice form.  Over a coarse
// stencil (8^4 -> 4^4, 2^4 blocks, nbasis 40) that is 7 point applications per
// site instead of the 22 of four full hops and two masked operators: 11.0 ms
// (and up to 40 with its six workspace allocations per call) -> 0.99 ms.
static gmg_status coarsen_faces(gmg_coarse* out, gmg_agg* agg, const FineOpRef& op, cudaStream_t s) {
  const int dof = op.dof();
  GMG_CHECK(agg->dof == dof, GMG_ERR_SHAPE, "coarsen: aggregation site dof differs from the fine operator");
  for (int d = 0; d < 4; ++d) {
    GMG_CHECK(agg->fdims.d[d] == op.dims().d[d], GMG_ERR_SHAPE, "coarsen: fine lattice differs");
    GMG_CHECK(agg->cdims.d[d] == out->dims.d[d], GMG_ERR_SHAPE, "coarsen: coarse lattice differs");
  }
  GMG_CHECK(agg->N == out->N, GMG_ERR_SHAPE, "coarsen: nbasis differs");
  GMG_CHECK(agg->basis_set, GMG_ERR_STATE, "coarsen: basis not set");
  const int N = agg->N;
  const int64_t Vc = out->dims.vol();
  GMG_TRY(out->links_ref.alloc(sizeof(double2) * 9 * Vc * N * N));  // every entry is written below
  GMG_TRY(coarsen_workspace(agg, s));
  // the constructions of one aggregation share its workspace: one on another stream
  // waits for the one before it (its event cannot enter a stream capture)
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GMG_CUDA(cudaStreamIsCapturing(s, &cap));
  if (cap == cudaStreamCaptureStatusNone) {
    if (!agg->cw_done) GMG_CUDA(cudaEventCreateWithFlags(&agg->cw_done, cudaEventDisableTiming));
    GMG_CUDA(cudaStreamWaitEvent(s, agg->cw_done, 0));
  }
  struct Done {
    cudaEvent_t ev;
    cudaStream_t s;
    ~Done() {
      if (ev) cudaEventRecord(ev, s);
    }
  } done{cap == cudaStreamCaptureStatusNone ? agg->cw_done : nullptr, s};
  const int nb = agg->cw_nb;
  double* phi = agg->cw_phi.as<double>();
  double* wf = agg->cw_w.as<double>();
  const int32_t* face = agg->cw_face.as<int32_t>();
  const int32_t* sel = agg->cw_sel.as<int32_t>();
  double2* A = out->links_ref.as<double2>();
  for (int i0 = 0; i0 < N; i0 += nb) {
    const int cur = std::min(nb, N - i0);
    GMG_TRY(op.gather(agg, i0, cur, phi, s));
    int fo = 0, so = 0;
    for (int d = 0; d < 4; ++d) {
      GMG_TRY(op.face(agg, 4 + d, cur, phi, wf, reinterpret_cast<double*>(A + (int64_t)(4 + d) * Vc * N * N), i0,
                      face + fo, agg->cw_nface[d], sel + so, agg->cw_nsel[d], s));
      fo += agg->cw_nface[d];
      so += agg->cw_nsel[d];
    }
    GMG_TRY(op.self(agg, cur, phi, wf, reinterpret_cast<double*>(A + (int64_t)8 * Vc * N * N), i0,
                    agg->cw_hskip.as<uint8_t>(), s));
  }
  GMG_TRY(coarse_construct_remaining(out, s));
  GMG_TRY(coarse_links_to_site_major(out, s));
  out->links_set = true;
  out->links_f_ok = false;
  out->self_inv_ok = out->self_inv_f_ok = false;
  out->links_h.kind = -1;
  return GMG_OK;
}

gmg_status coarsen_wilson(gmg_coarse* out, gmg_agg* agg, gmg_wilson* fine, cudaStream_t s) {
  GMG_CHECK(fine->gauge_set, GMG_ERR_STATE, "coarsen: gauge field not set");
  FineOpRef op;
  op.w = fine;
  return coarsen_faces(out, agg, op, s);
}

gmg_status coarsen_coarse(gmg_coarse* out, gmg_agg* agg, gmg_coarse* fine, cudaStream_t s) {
  GMG_CHECK(fine->links_set, GMG_ERR_STATE, "coarsen: fine links not set");
  FineOpRef op;
  op.c = fine;
  const bool had = agg->cw_nb > 0;
  const gmg_status st = coarsen_faces(out, agg, op, s);
  // unlike the Wilson-clover form this entry returns when the links are built, and
  // gives a large workspace back (8^4 sites of 40 components, nbasis 40, take 0.2 GB;
  // where it is large the construction takes far longer than the allocation)
  const cudaError_t e = cudaStreamSynchronize(s);
  if (!had && agg->cw_phi.bytes + agg->cw_w.bytes > kKeptBytes) {
    agg->cw_phi.free();
    agg->cw_w.free();
    agg->cw_nb = 0;
  }
  GMG_TRY(st);
  GMG_CUDA(e);
  return GMG_OK;
}

}  // namespace gmg
