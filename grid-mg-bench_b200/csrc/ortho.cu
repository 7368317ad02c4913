// ortho.cu -- block orthonormalisation of the aggregation basis (FP64) and the
// orthogonality check.
//
// Restates blockLutedOrthonormalise (include/CoarsenedMatrixUpstreamImprovedDirsaveLut.h:
// 172-240; per-chirality form AggregationKernelsRework.h:266-341) and
// Aggregation::CheckOrthogonal (...LutMRHS.h:326-340).  The reference runs a
// modified Gram-Schmidt per block, one thread per block.  Here each pass is a
// Cholesky QR of every block's N x K panel V_c (K = block sites x site dof):
//
//   G_c = conj(V_c) V_c^T          (N x N Hermitian Gram matrix, G[i][j] = <v_i, v_j>_c)
//   G_c = L L^dag                   (Cholesky, L lower with a positive diagonal)
//   conj(L) W_c = V_c               (forward substitution, one column of V_c at a time)
//
// W_c is orthonormal and lower-triangularly related to V_c with a positive
// diagonal, the properties that fix the result of Gram-Schmidt: a thin QR with
// a positive R diagonal is unique, so both give the same basis up to rounding.
// Cholesky QR loses orthogonality as cond(V_c)^2; when a factorisation breaks
// down (smoothed test vectors can be nearly dependent inside a block) it is
// redone with the diagonal shift of shifted Cholesky QR (Fukaya, Kannan,
// Nakatsukasa, Yamamoto, Yanagisawa, SIAM J. Sci. Comput. 42 (2020)),
// s = 11 (K N + N (N + 1)) u ||V_c||_F^2, which always factors, and that block
// gets two extra plain passes.
//
// Three kernels per pass (nbasis up to 40):
//   gram_kernel      CTA per block: the Gram matrix on the FP64 tensor cores, K
//                    split over the warps; writes the packed lower triangle.
//   factor_kernel    warp per block: the Cholesky factor in shared memory, lane
//                    i owning row i; the shifted retry re-reads the Gram matrix;
//                    writes conj(L) and 1 / diag(L) packed (row i: i + 1 entries).
//   tri_solve_kernel thread per column of V_c: the column in registers, forward
//                    substitution against conj(L) in shared memory (every thread
//                    reads the same entry: a broadcast), the column written back
//                    in place; the next column batch is copied into shared
//                    memory (cp.async) while the current one is solved.  (On
//                    the FP64 tensor cores, a column's rows in the accumulator
//                    layout and the 4 x 4 diagonal blocks inverted, the same
//                    substitution takes 2.36 against 2.86 ms at 32^4 x 32, but
//                    the MMAs' order of summation loses most of a digit on nearly
//                    dependent vectors; with the diagonal blocks solved by
//                    shuffles 3.06 ms.)
// Traffic per pass: the basis read twice and written once (3 x 8 B x 2 x N x K
// per block) plus the small factors; flops 8 K N (N + 1) / 2 for the Gram
// matrix (lower triangle) and the same for the substitution.
//
// Layout: basis_blk [c][i][k] complex128, k = sb * dof + a (one block's panel
// contiguous).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "f64_mma.cuh"
#include "gmg_internal.cuh"

namespace gmg {
namespace ortho {

constexpr int kThreads = 256;
constexpr int kSolveMax = 40;   // largest nbasis of the three-kernel path
constexpr int kFactorWarps = 4;  // blocks (one per warp) per factor CTA

__device__ __forceinline__ double2 cfma_conj(double2 acc, double2 a, double2 b) {  // acc += conj(a) b
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
  return acc;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }

struct Params {
  double2* basis;              // [Vc][N][K]
  double2* gram;               // [Vc][N (N + 1) / 2]: G[i][j], j <= i
  double2* lfac;               // [Vc][N (N + 1) / 2]: conj(L[i][j]) for j < i, (1 / L[i][i], 0) for j = i
  int* need;                   // [Vc]: 1 once a block needed the shifted factorisation
  int* status;                 // 1 when a shifted factorisation failed too
  unsigned long long* maxerr;  // check mode: max |G - 1| (as the bits of a non-negative double)
  int Vc, N, K;
  int pass, passes;
  int whole;  // the wide substitution's CTAs take whole blocks
};

__device__ __forceinline__ bool block_active(const Params& P, int c) { return P.pass < P.passes || P.need[c] != 0; }

// Gram matrices of the blocks (packed lower triangles into P.gram), or in
// CHECK mode the largest |G - 1| over all blocks into P.maxerr.  CTA per block.
// Bound by the FP64 tensor pipe: with R, I the real and imaginary parts of eight
// basis vectors a tile, the lower 8 x 8 tiles of
//   Re G = R R^T + I I^T,  Im G = R I^T - I R^T
// take four MMAs per four values of k (three on the diagonal, where Im G is
// S - S^T, S = R I^T).  A lane's fragments of both parts are one 16-byte load:
// lane (r, q) reads v_(8 X + r)[k + q], a warp 64 contiguous bytes of each vector,
// so nothing is staged in shared memory, and every warp computes all tiles from
// one set of loads, the next KU steps' requests in flight meanwhile; the warps
// split k and their sums are added in a fixed order.  32^4, 4^4 blocks, nbasis 32:
// 2.49 ms (fragments by way of shared memory, 58 % of the pipe) -> 1.98 ms.
// HALF: the last tile holds four vectors at most, their real parts as rows 0 to 3 and
// their imaginary parts as rows 4 to 7, so that it takes two MMAs against another tile and
// one with itself instead of four and three (16^4, 4^4 blocks, nbasis 36: 282 -> 255 us;
// the tiles of the real panel's Gram matrix before took 273).
template <int NT, bool CHECK, bool HALF = false>
__global__ void __launch_bounds__(NT > 4 ? 256 : 384) gram_kernel(Params P) {
  constexpr int KU = NT == 1 ? 8 : NT == 2 ? 4 : 2, NP = NT * (NT + 1) / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* red = reinterpret_cast<double*>(smem_raw);  // [warps][NP][2][64]
  const int c = blockIdx.x;
  if (!CHECK && !block_active(P, c)) return;  // the whole CTA
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int N = P.N, K = P.K, q = lane & 3;
  const double2* row[NT];  // rows past N read row N - 1: their sums are not used
#pragma unroll
  for (int X = 0; X < NT; ++X)
    row[X] = P.basis + ((int64_t)c * N + min(8 * X + (HALF && X == NT - 1 ? (lane >> 2) & 3 : lane >> 2), N - 1)) * K;
  double re[NP][2], im[NP][2];
#pragma unroll
  for (int p = 0; p < NP; ++p) re[p][0] = re[p][1] = im[p][0] = im[p][1] = 0.0;
  double2 f[KU][NT], g[KU][NT];
  auto load = [&](double2 (&d)[KU][NT], int u) {
#pragma unroll
    for (int t = 0; t < KU; ++t) {
      const int k = (u * KU + t) * 4 + q;
#pragma unroll
      for (int X = 0; X < NT; ++X) d[t][X] = k < K ? __ldg(row[X] + k) : make_double2(0.0, 0.0);
    }
  };
  const int units = (K + 4 * KU - 1) / (4 * KU);
  if (w < units) load(f, w);
  for (int u = w; u < units; u += nw) {
    if (u + nw < units) load(g, u + nw);
#pragma unroll
    for (int t = 0; t < KU; ++t) {
      constexpr int NW = HALF ? NT - 1 : NT;  // whole tiles
      if constexpr (HALF) {
        const double h = (lane >> 2) < 4 ? f[t][NW].x : f[t][NW].y;
        constexpr int B = NW * (NW + 1) / 2;
#pragma unroll
        for (int Y = 0; Y < NW; ++Y) {
          f64mma::mma(re[B + Y], h, f[t][Y].x);
          f64mma::mma(im[B + Y], h, f[t][Y].y);
        }
        f64mma::mma(re[B + NW], h, h);
      }
#pragma unroll
      for (int X = 0; X < NW; ++X)
#pragma unroll
        for (int Y = 0; Y <= X; ++Y) {
          f64mma::mma(re[X * (X + 1) / 2 + Y], f[t][X].x, f[t][Y].x);
          f64mma::mma(im[X * (X + 1) / 2 + Y], f[t][X].x, f[t][Y].y);
        }
#pragma unroll
      for (int X = 0; X < NW; ++X)
#pragma unroll
        for (int Y = 0; Y <= X; ++Y) {
          f64mma::mma(re[X * (X + 1) / 2 + Y], f[t][X].y, f[t][Y].y);
          if (Y < X) f64mma::mma(im[X * (X + 1) / 2 + Y], -f[t][X].y, f[t][Y].x);
        }
    }
#pragma unroll
    for (int t = 0; t < KU; ++t)
#pragma unroll
      for (int X = 0; X < NT; ++X) f[t][X] = g[t][X];
  }
  // element (m, n) of a tile: lane (m, n / 2)
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    double* d = red + ((size_t)w * NP + p) * 128 + 2 * lane;
    *reinterpret_cast<double2*>(d) = make_double2(re[p][0], re[p][1]);
    *reinterpret_cast<double2*>(d + 64) = make_double2(im[p][0], im[p][1]);
  }
  __syncthreads();
  double mx = 0.0;
  double2* Gc = P.gram + (int64_t)c * (N * (N + 1) / 2);
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int i = e / N, j = e - i * N;
    if (j > i) continue;
    const int X = i >> 3, Y = j >> 3;
    const double* d = red + (size_t)(X * (X + 1) / 2 + Y) * 128;
    const int at = (i & 7) * 8 + (j & 7), mirror = (j & 7) * 8 + (i & 7);
    double gr = 0.0, gi = 0.0;
    for (int v = 0; v < nw; ++v, d += NP * 128) {
      if (HALF && X == NT - 1) {  // rows 0 to 3 and 4 to 7 (and columns, of the tile with itself)
        gr += d[at] + (X == Y ? d[at + 36] : d[64 + at + 32]);
        gi += (X == Y ? d[at + 4] : d[64 + at]) - d[at + 32];
        continue;
      }
      gr += d[at];
      gi += X == Y ? d[64 + at] - d[64 + mirror] : d[64 + at];
    }
    if (CHECK && i == j) gi = 0.0;  // also where both terms overflowed (the factor takes real diagonals)
    if (CHECK) {
      const double x = gr - (i == j ? 1.0 : 0.0);
      mx = fmax(mx, sqrt(x * x + gi * gi));
    } else {
      Gc[i * (i + 1) / 2 + j] = make_double2(gr, gi);
    }
  }
  if (CHECK) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0)  // non-negative doubles order as integers
      atomicMax(P.maxerr, (unsigned long long)__double_as_longlong(mx));
  }
}

// Cholesky factor of one block's Gram matrix by one warp: G + shift I = L L^dag,
// rows in shared memory at stride N + 1 (lane i owns rows i and i + 32), the
// strict lower triangle of L in place of G, the diagonal in diag[].  Returns
// false when a pivot is not positive (replaced by 1 so that L stays finite).
__device__ bool warp_cholesky(double2* G, double* diag, int N, double shift) {
  const int lane = threadIdx.x & 31, Sp = N + 1;
  bool ok = true;
  for (int j = 0; j < N; ++j) {
    double d = G[j * Sp + j].x + shift;
    if (!(d > 0.0)) {
      ok = false;
      d = 1.0;
    }
    const double dj = sqrt(d), inv = 1.0 / dj;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = lane + 32 * h;
      if (i > j && i < N) {
        const double2 v = G[i * Sp + j];
        G[i * Sp + j] = make_double2(v.x * inv, v.y * inv);
      }
    }
    if (lane == 0) diag[j] = dj;
    __syncwarp();
    // trailing update G[i][k] -= L[i][j] conj(L[k][j]), j < k <= i: lane i walks
    // k in step with the other lanes, so L[k][j] is one broadcast read
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = lane + 32 * h;
      if (i > j && i < N) {
        const double2 a = G[i * Sp + j];
#pragma unroll 4
        for (int k = j + 1; k <= i; ++k) {
          const double2 b = G[k * Sp + j];
          double2 g = G[i * Sp + k];
          g.x -= a.x * b.x + a.y * b.y;
          g.y -= a.y * b.x - a.x * b.y;
          G[i * Sp + k] = g;
        }
      }
    }
    __syncwarp();
  }
  return ok;
}

__global__ void __launch_bounds__(32 * kFactorWarps) factor_kernel(Params P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = P.N, Sp = N + 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * kFactorWarps + w;
  if (c >= P.Vc || !block_active(P, c)) return;  // whole warps leave; no block-wide barrier follows
  double2* G = reinterpret_cast<double2*>(smem_raw) + (size_t)w * N * Sp;
  double* diag = reinterpret_cast<double*>(reinterpret_cast<double2*>(smem_raw) + (size_t)kFactorWarps * N * Sp) +
                 (size_t)w * N;
  const int nl = N * (N + 1) / 2;
  const double2* Gc = P.gram + (int64_t)c * nl;
  auto load = [&]() {
    for (int i = 0; i < N; ++i)
      for (int j = lane; j <= i; j += 32) G[i * Sp + j] = Gc[i * (i + 1) / 2 + j];
    __syncwarp();
  };
  load();
  bool ok = warp_cholesky(G, diag, N, 0.0);
  if (!ok) {
    // shifted Cholesky QR on the same Gram matrix, and two extra passes for this block
    load();
    double tr = 0.0;
    for (int i = lane; i < N; i += 32) tr += G[i * Sp + i].x;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, off);
    const double shift = 11.0 * ((double)P.K * N + (double)N * (N + 1)) * 1.1102230246251565e-16 * tr;
    ok = warp_cholesky(G, diag, N, shift);
    if (lane == 0) {
      P.need[c] = 1;
      if (!ok) atomicExch(P.status, 1);
    }
  }
  double2* Lc = P.lfac + (int64_t)c * nl;
  for (int i = 0; i < N; ++i)
    for (int j = lane; j <= i; j += 32) {
      const double2 v = G[i * Sp + j];
      Lc[i * (i + 1) / 2 + j] = j < i ? make_double2(v.x, -v.y) : make_double2(1.0 / diag[i], 0.0);
    }
}

constexpr int kSolveThreads = 128;  // columns per solve chunk (three CTAs per SM at N = 32)

// W = conj(L)^{-1} V for every column of every block: thread per column, the
// column in registers (NMAX entries, rows >= N unused), conj(L) in shared
// memory; the CTA walks a run of kSolveThreads-column chunks, an equal share of
// all blocks' (with whole blocks a CTA, fewer blocks than CTAs left SMs idle: 108
// blocks of 128 sites x 12, nbasis 20, take 154 us orthonormalised and written back
// against 204, the Gram kernel's gain included), with the next chunk's columns
// copied into shared memory while the current chunk is solved.
// EXACT: nbasis equals NMAX, so that every row bound is a compile-time
// constant (no guards between the row groups' independent products; at
// N = 32 that also frees registers: 176 instead of 214, and 168 without
// spills at three CTAs per SM, tri_solve32_kernel).  C3 (32^4, 4^4 blocks,
// N 32): 3.26 ms with the guards at two CTAs per SM, 2.98 ms without, 2.83 ms
// without at three.
template <int NMAX, bool EXACT>
__device__ __forceinline__ void tri_solve_body(const Params& P) {
  constexpr int NTS = kSolveThreads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* pre = reinterpret_cast<double2*>(smem_raw);  // [NMAX][NTS]: the prefetched columns
  double2* L = pre + NMAX * NTS;                        // packed conj(L) of the current block
  const int N = EXACT ? NMAX : P.N, K = P.K, t = threadIdx.x;
  const int nl = N * (N + 1) / 2;
  const int chunks = (K + NTS - 1) / NTS;
  auto prefetch = [&](bool valid, int c, int ch) {
    const int k = valid ? ch * NTS + t : K;
    if (k < K) {
      const double2* col = P.basis + (int64_t)c * N * K + k;
#pragma unroll
      for (int i = 0; i < NMAX; ++i)
        if (i < N) cp_async16(pre + i * NTS + t, col + (int64_t)i * K);
    }
    cp_async_commit();
  };
  int lc = -1;  // the block whose factor is in L
  auto item = [&](int c, int ch, auto prefetch_next) {
    if (c != lc) {
      __syncthreads();  // every thread is done with the previous block's factor
      const double2* src = P.lfac + (int64_t)c * nl;
      for (int e = t; e < nl; e += NTS) L[e] = src[e];
      __syncthreads();
      lc = c;
    }
    cp_async_wait<0>();  // this thread's columns of the current item (its own slots only)
    const int k = ch * NTS + t;
    double2 w[NMAX];
#pragma unroll
    for (int i = 0; i < NMAX; ++i) w[i] = (i < N && k < K) ? pre[i * NTS + t] : make_double2(0.0, 0.0);
    prefetch_next();  // the slots are free again: copy the next item's columns meanwhile
    if (k < K) {
      // rows in groups of four: the products with the already solved entries
      // (j below the group) are independent across the group's rows, two
      // partial sums each, so eight chains run side by side; then the group's
      // own 4 x 4 triangle in order
#pragma unroll
      for (int i0 = 0; i0 < NMAX; i0 += 4) {
        if (i0 < N) {
          double2 sp[4][2];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            sp[q][0] = (i0 + q < N) ? w[i0 + q] : make_double2(0.0, 0.0);
            sp[q][1] = make_double2(0.0, 0.0);
          }
#pragma unroll
          for (int j = 0; j < i0; ++j) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // s -= conj(L[i][j]) w[j]
              const int i = i0 + q;
              if (i < NMAX && i < N) {  // L holds the N (N + 1) / 2 entries of rows i < N only
                const double2 a = L[i * (i + 1) / 2 + j];
                double2& sq = sp[q][j & 1];
                sq.x = fma(-a.x, w[j].x, sq.x);
                sq.x = fma(a.y, w[j].y, sq.x);
                sq.y = fma(-a.x, w[j].y, sq.y);
                sq.y = fma(-a.y, w[j].x, sq.y);
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + q;
            if (i < NMAX && i < N) {
              const double2* Li = L + i * (i + 1) / 2;
              double2 sq = make_double2(sp[q][0].x + sp[q][1].x, sp[q][0].y + sp[q][1].y);
#pragma unroll
              for (int j = i0; j < i; ++j) {
                const double2 a = Li[j];
                sq.x = fma(-a.x, w[j].x, sq.x);
                sq.x = fma(a.y, w[j].y, sq.x);
                sq.y = fma(-a.x, w[j].y, sq.y);
                sq.y = fma(-a.y, w[j].x, sq.y);
              }
              const double inv = Li[i].x;
              w[i] = make_double2(sq.x * inv, sq.y * inv);
            }
          }
        }
      }
      double2* col = P.basis + (int64_t)c * N * K + k;
#pragma unroll
      for (int i = 0; i < NMAX; ++i)
        if (i < N) col[(int64_t)i * K] = w[i];
    }
  };
  if constexpr (NMAX > 32) {
    // items [it, end): chunk it % chunks of block(it / chunks), a run of all blocks' chunks or
    // whole blocks at the grid's stride.  One index and a division per item: the state of
    // the loop below slowed these instances, whose column alone takes 160 registers (433
    // -> 375 us at 4096 blocks of 192 columns, nbasis 36)
    const int total = P.Vc * chunks, per = (total + (int)gridDim.x - 1) / (int)gridDim.x;
    int it = P.whole ? 0 : min((int)blockIdx.x * per, total);
    const int end = P.whole ? (P.Vc - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * chunks : min(it + per, total);
    auto block = [&](int q) { return P.whole ? (int)blockIdx.x + q * (int)gridDim.x : q; };
    auto active_from = [&](int i) {
      while (i < end && !block_active(P, block(i / chunks))) i = (i / chunks + 1) * chunks;
      return i;
    };
    it = active_from(it);
    prefetch(it < end, block(it / chunks), it % chunks);
    while (it < end) {
      const int q = it / chunks;
      item(block(q), it - q * chunks, [&] {
        it = active_from(it + 1);
        prefetch(it < end, block(it / chunks), it % chunks);
      });
    }
  } else {
    // this CTA's items: n (block c, chunk ch) pairs in order from its first; inactive blocks are passed over
    const int64_t total = (int64_t)P.Vc * chunks, per = (total + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per;
    int n = (int)max((int64_t)0, min(per, total - first)), c = (int)(first / chunks), ch = (int)(first % chunks);
    auto skip = [&](int& n, int& c, int& ch) {
      while (n > 0 && !block_active(P, c)) {
        n -= chunks - ch;
        ++c;
        ch = 0;
      }
    };
    skip(n, c, ch);
    prefetch(n > 0, c, ch);
    while (n > 0) {
      // the item after this one
      int nn = n - 1, nc = c, nch = ch + 1;
      if (nch == chunks) {
        ++nc;
        nch = 0;
      }
      skip(nn, nc, nch);
      item(c, ch, [&] { prefetch(nn > 0, nc, nch); });
      n = nn;
      c = nc;
      ch = nch;
    }
  }
  cp_async_wait<0>();
}

template <int NMAX, bool EXACT>
__global__ void __launch_bounds__(kSolveThreads) tri_solve_kernel(Params P) {
  tri_solve_body<NMAX, EXACT>(P);
}

__global__ void __launch_bounds__(kSolveThreads, 3) tri_solve32_kernel(Params P) { tri_solve_body<32, true>(P); }

// Cholesky G + shift I = L L^dag in place by the whole CTA (strict lower
// triangle of G, row-major N x N; the diagonal goes to diag[]); false to every
// thread when a pivot is not positive (replaced by 1).  Used by the one-CTA-
// per-block path below.
__device__ bool block_cholesky(double2* G, double* diag, int N, double shift, int* fail_s) {
  const int t = threadIdx.x;
  if (t == 0) *fail_s = 0;
  __syncthreads();
  for (int j = 0; j < N; ++j) {
    double d = G[j * N + j].x + shift;
    const bool bad = !(d > 0.0);
    if (bad) d = 1.0;
    const double dj = sqrt(d), inv = 1.0 / dj;
    for (int i = j + 1 + t; i < N; i += kThreads) {
      const double2 v = G[i * N + j];
      G[i * N + j] = make_double2(v.x * inv, v.y * inv);
    }
    if (t == 0) {
      diag[j] = dj;
      if (bad) *fail_s = 1;
    }
    __syncthreads();
    const int m = N - j - 1;
    for (int e = t; e < m * (m + 1) / 2; e += kThreads) {
      int ii = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
      while (ii * (ii + 1) / 2 > e) --ii;
      while ((ii + 1) * (ii + 2) / 2 <= e) ++ii;
      const int kk = e - ii * (ii + 1) / 2;
      const int i = j + 1 + ii, k = j + 1 + kk;
      const double2 a = G[i * N + j], b = G[k * N + j];
      double2 g = G[i * N + k];
      g.x -= a.x * b.x + a.y * b.y;
      g.y -= a.y * b.x - a.x * b.y;
      G[i * N + k] = g;
    }
    __syncthreads();
  }
  return *fail_s == 0;
}

// ---------------------------------------------------------------------------
// one CTA per block for nbasis above the two-kernel path (up to 64): the same
// Cholesky QR with the whole block's transform applied from shared memory
// ---------------------------------------------------------------------------
constexpr int kBigKS = 2;  // sites per K chunk

__device__ void big_gram(const double2* __restrict__ Vb, int N, int64_t K, int dof, double2* VT, double2* G) {
  const int t = threadIdx.x;
  const int NTl = (N + 3) / 4;
  const int ntiles = NTl * NTl;
  const int ti = t % NTl, tj = t / NTl;
  double2 acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = make_double2(0, 0);
  const int KC = kBigKS * dof;
  for (int64_t k0 = 0; k0 < K; k0 += KC) {
    const int kc = (int)((K - k0) < (int64_t)KC ? (K - k0) : (int64_t)KC);
    __syncthreads();
    for (int e = t; e < N * kc; e += blockDim.x) {
      const int i = e / kc, kk = e % kc;
      VT[kk * N + i] = Vb[(int64_t)i * K + k0 + kk];
    }
    __syncthreads();
    if (t < ntiles) {
      for (int kk = 0; kk < kc; ++kk) {
        double2 a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = ti * 4 + q, j = tj * 4 + q;
          a[q] = i < N ? VT[kk * N + i] : make_double2(0, 0);
          b[q] = j < N ? VT[kk * N + j] : make_double2(0, 0);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[x][y] = cfma_conj(acc[x][y], a[x], b[y]);
      }
    }
  }
  __syncthreads();
  if (t < ntiles) {
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int i = ti * 4 + x, j = tj * 4 + y;
        if (i < N && j < N) G[i * N + j] = acc[x][y];
      }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kThreads) big_ortho_kernel(double2* __restrict__ basis, int Vc, int N, int dof,
                                                             int bv, int passes, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* G = reinterpret_cast<double2*>(smem_raw);  // [N][N]  Gram, then L
  double2* Li = G + N * N;                             // [N][N]  conj(L^{-1})
  double* diag = reinterpret_cast<double*>(Li + N * N);
  double2* VT = reinterpret_cast<double2*>(diag + N + (N & 1));  // [KC][N] staging
  __shared__ int fail_s;
  __shared__ double trace_s;
  const int64_t K = (int64_t)bv * dof;
  const int t = threadIdx.x;
  for (int c = blockIdx.x; c < Vc; c += gridDim.x) {
    double2* Vb = basis + (int64_t)c * N * K;
    int extra = 0;
    for (int pass = 0; pass < passes + extra; ++pass) {
      big_gram(Vb, N, K, dof, VT, G);
      if (!block_cholesky(G, diag, N, 0.0, &fail_s)) {
        big_gram(Vb, N, K, dof, VT, G);
        if (t == 0) {
          double tr = 0.0;
          for (int i = 0; i < N; ++i) tr += G[i * N + i].x;
          trace_s = tr;
        }
        __syncthreads();
        const double shift = 11.0 * ((double)K * N + (double)N * (N + 1)) * 1.1102230246251565e-16 * trace_s;
        if (!block_cholesky(G, diag, N, shift, &fail_s) && t == 0) atomicExch(status, 1);
        if (extra < 2) extra = 2;
      }
      // conj(L^{-1}) column by column (one thread per column)
      for (int j = t; j < N; j += blockDim.x) {
        for (int i = 0; i < N; ++i) Li[i * N + j] = make_double2(0, 0);
        Li[j * N + j] = make_double2(1.0 / diag[j], 0.0);
        for (int i = j + 1; i < N; ++i) {
          double2 sacc = make_double2(0, 0);
          for (int k = j; k < i; ++k) {
            const double2 a = k == i ? make_double2(diag[i], 0.0) : G[i * N + k], x = Li[k * N + j];
            sacc.x += a.x * x.x - a.y * x.y;
            sacc.y += a.x * x.y + a.y * x.x;
          }
          const double inv = 1.0 / diag[i];
          Li[i * N + j] = make_double2(-sacc.x * inv, -sacc.y * inv);
        }
        for (int i = j; i < N; ++i) Li[i * N + j].y = -Li[i * N + j].y;
      }
      __syncthreads();
      const int KC = kBigKS * dof;
      for (int64_t k0 = 0; k0 < K; k0 += KC) {
        const int kc = (int)((K - k0) < (int64_t)KC ? (K - k0) : (int64_t)KC);
        __syncthreads();
        for (int e = t; e < N * kc; e += blockDim.x) {
          const int i = e / kc, kk = e % kc;
          VT[kk * N + i] = Vb[(int64_t)i * K + k0 + kk];
        }
        __syncthreads();
        for (int e = t; e < N * kc; e += blockDim.x) {
          const int i = e / kc, kk = e % kc;
          double2 acc = make_double2(0, 0);
          for (int j = 0; j <= i; ++j) {
            const double2 l = Li[i * N + j], v = VT[kk * N + j];
            acc.x = fma(l.x, v.x, acc.x);
            acc.x = fma(-l.y, v.y, acc.x);
            acc.y = fma(l.x, v.y, acc.y);
            acc.y = fma(l.y, v.x, acc.y);
          }
          Vb[(int64_t)i * K + k0 + kk] = acc;
        }
      }
      __syncthreads();
    }
  }
}

// the orthogonality check above nbasis 40: one CTA per block, max |G - 1|
__global__ void __launch_bounds__(kThreads) big_check_kernel(const double2* __restrict__ basis, int Vc, int N, int dof,
                                                             int bv, unsigned long long* __restrict__ maxerr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* G = reinterpret_cast<double2*>(smem_raw);  // [N][N]
  double2* VT = G + N * N;                             // [KC][N] staging
  const int64_t K = (int64_t)bv * dof;
  double mx = 0.0;
  for (int c = blockIdx.x; c < Vc; c += gridDim.x) {
    big_gram(basis + (int64_t)c * N * K, N, K, dof, VT, G);
    for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
      const int i = e / N, j = e % N;
      const double re = G[e].x - (i == j ? 1.0 : 0.0), im = G[e].y;
      mx = fmax(mx, sqrt(re * re + im * im));
    }
    __syncthreads();
  }
  atomicMax(maxerr, (unsigned long long)__double_as_longlong(mx));
}

static int num_sms() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// workspace: [status int + max error][need int Vc][Gram Vc x N (N + 1) / 2][conj(L) same]
static gmg_status workspace(gmg_agg* h, Params* P) {
  const int64_t Vc = h->cdims.vol();
  const size_t head = 256, need_b = (size_t)(Vc * sizeof(int) + 255) / 256 * 256;
  const size_t lf_b = sizeof(double2) * (size_t)Vc * (h->N * (h->N + 1) / 2);
  const void* before = h->ortho_ws.p;
  GMG_TRY(h->ortho_ws.alloc(head + need_b + 2 * lf_b));
  char* p = h->ortho_ws.as<char>();
  if (p != before) GMG_CUDA(cudaMemset(p, 0, head));  // fresh memory: no failure recorded yet
  P->basis = h->basis_blk.as<double2>();
  P->status = reinterpret_cast<int*>(p);
  P->maxerr = reinterpret_cast<unsigned long long*>(p + 8);
  P->need = reinterpret_cast<int*>(p + head);
  P->gram = reinterpret_cast<double2*>(p + head + need_b);
  P->lfac = reinterpret_cast<double2*>(p + head + need_b + lf_b);
  P->Vc = (int)Vc;
  P->N = h->N;
  P->K = h->bv * h->dof;
  P->pass = 0;
  P->whole = 0;
  P->passes = 1;
  return GMG_OK;
}

template <int NT, bool CHECK, bool HALF = false>
static gmg_status launch_gram_nt(const Params& P, cudaStream_t s) {
  // four warps a block; eight where the blocks alone leave the chip's warps idle
  const int nw = P.Vc < num_sms() * 4 ? 8 : 4;
  const size_t smem = sizeof(double) * 128 * (NT * (NT + 1) / 2) * nw;
  auto kern = gram_kernel<NT, CHECK, HALF>;
  GMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<P.Vc, 32 * nw, smem, s>>>(P);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

template <bool CHECK>
static gmg_status launch_gram(const Params& P, cudaStream_t s) {
  switch ((P.N + 7) / 8) {
    case 1: return launch_gram_nt<1, CHECK>(P, s);
    case 2: return launch_gram_nt<2, CHECK>(P, s);
    case 3: return launch_gram_nt<3, CHECK>(P, s);
    case 4: return launch_gram_nt<4, CHECK>(P, s);
    case 5:
      if constexpr (!CHECK)
        if (P.N <= 36) return launch_gram_nt<5, CHECK, true>(P, s);
      return launch_gram_nt<5, CHECK>(P, s);
    default: return fail(GMG_ERR_UNSUPPORTED, "orthonormalise: nbasis above the tensor-core Gram path");
  }
}

static gmg_status launch_factor(const Params& P, cudaStream_t s) {
  const size_t smem = (sizeof(double2) * (size_t)P.N * (P.N + 1) + sizeof(double) * P.N) * kFactorWarps;
  GMG_CUDA(cudaFuncSetAttribute(factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  factor_kernel<<<(P.Vc + kFactorWarps - 1) / kFactorWarps, 32 * kFactorWarps, smem, s>>>(P);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

template <int NMAX>
static gmg_status launch_solve(const Params& P, cudaStream_t s) {
  const size_t smem = sizeof(double2) * ((size_t)NMAX * kSolveThreads + (size_t)P.N * (P.N + 1) / 2);
  void (*kern)(Params) = tri_solve_kernel<NMAX, false>;
  if (P.N == NMAX) {
    if constexpr (NMAX == 32)
      kern = tri_solve32_kernel;
    else
      kern = tri_solve_kernel<NMAX, true>;
  }
  GMG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1;
  GMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSolveThreads, smem));
  const int64_t chunks = (P.K + kSolveThreads - 1) / kSolveThreads, items = P.Vc * chunks;
  const int64_t slots = num_sms() * std::max(per_sm, 1), by_block = std::min<int64_t>(P.Vc, slots);
  int64_t grid = std::min<int64_t>(items, slots);
  // nbasis above 32: whole blocks at the grid's stride, whose CTAs walk the rows side by side, unless that
  // takes a CTA a fifth more chunks than equal runs of them (24^4, 1296 blocks of 4^4,
  // nbasis 40: 1509 us, in runs 1705; 16^4, 256 blocks, nbasis 32: 220, in runs 200; 81
  // blocks, nbasis 40: 195, in runs 113)
  Params Q = P;
  Q.whole = NMAX > 32 && 5 * ((P.Vc + by_block - 1) / by_block * chunks) <= 6 * ((items + grid - 1) / grid);
  if (Q.whole) grid = by_block;
  kern<<<(int)grid, kSolveThreads, smem, s>>>(Q);
  GMG_CUDA(cudaGetLastError());
  return GMG_OK;
}

static gmg_status solve(const Params& P, cudaStream_t s) {
  if (P.N <= 8) return launch_solve<8>(P, s);
  if (P.N <= 16) return launch_solve<16>(P, s);
  if (P.N <= 24) return launch_solve<24>(P, s);
  if (P.N <= 32) return launch_solve<32>(P, s);
  return launch_solve<40>(P, s);
}

}  // namespace ortho

gmg_status agg_orthonormalise(gmg_agg* h, int passes, cudaStream_t s) {
  using namespace ortho;
  const int N = h->N;
  Params P;
  GMG_TRY(workspace(h, &P));
  const int Vc = P.Vc;
  GMG_CUDA(cudaMemsetAsync(P.status, 0, sizeof(int), s));
  if (N > kSolveMax) {
    GMG_CHECK(N <= 64, GMG_ERR_UNSUPPORTED, "orthonormalise: nbasis > 64");
    const size_t smem = sizeof(double2) * ((size_t)2 * N * N + (size_t)kBigKS * h->dof * N) +
                        sizeof(double) * (N + (N & 1));
    GMG_CHECK(smem <= 227 * 1024, GMG_ERR_UNSUPPORTED, "orthonormalise: nbasis x site dof too large");
    GMG_CUDA(cudaFuncSetAttribute(big_ortho_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KernelTimer kt("ortho", s);
    big_ortho_kernel<<<std::min(Vc, num_sms() * 8), kThreads, smem, s>>>(h->basis_blk.as<double2>(), Vc, N, h->dof,
                                                                        h->bv, passes, P.status);
    GMG_CUDA(cudaGetLastError());
  } else {
    GMG_CUDA(cudaMemsetAsync(P.need, 0, sizeof(int) * Vc, s));
    P.passes = passes;
    KernelTimer kt("ortho", s);
    // passes + 2 rounds: the last two only touch blocks that needed the shift
    for (int pass = 0; pass < passes + 2; ++pass) {
      P.pass = pass;
      {
        KernelTimer k1("ortho_gram", s);
        GMG_TRY(launch_gram<false>(P, s));
      }
      {
        KernelTimer k2("ortho_factor", s);
        GMG_TRY(launch_factor(P, s));
      }
      KernelTimer k3("ortho_solve", s);
      GMG_TRY(solve(P, s));
    }
  }
  h->basis_f_ok = false;
  h->basis_tc_ok = false;
  return GMG_OK;
}

gmg_status agg_check_orthogonal(gmg_agg* h, double* max_err, cudaStream_t s) {
  using namespace ortho;
  Params P;
  GMG_TRY(workspace(h, &P));
  GMG_CUDA(cudaMemsetAsync(P.maxerr, 0, sizeof(unsigned long long), s));
  if (h->N > kSolveMax) {
    const size_t smem = sizeof(double2) * ((size_t)h->N * h->N + (size_t)kBigKS * h->dof * h->N);
    GMG_CHECK(smem <= 227 * 1024, GMG_ERR_UNSUPPORTED, "check orthogonal: nbasis x site dof too large");
    GMG_CUDA(cudaFuncSetAttribute(big_check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    big_check_kernel<<<std::min(P.Vc, num_sms() * 8), kThreads, smem, s>>>(h->basis_blk.as<double2>(), P.Vc, h->N,
                                                                          h->dof, h->bv, P.maxerr);
    GMG_CUDA(cudaGetLastError());
  } else {
    GMG_TRY(launch_gram<true>(P, s));
  }
  unsigned long long v = 0;
  int st = 0;
  GMG_CUDA(cudaMemcpyAsync(&v, P.maxerr, sizeof(v), cudaMemcpyDeviceToHost, s));
  GMG_CUDA(cudaMemcpyAsync(&st, P.status, sizeof(int), cudaMemcpyDeviceToHost, s));
  GMG_CUDA(cudaStreamSynchronize(s));
  double r;
  memcpy(&r, &v, sizeof(r));
  *max_err = r;
  if (st) return fail(GMG_ERR_NONFINITE, "orthonormalise: a block Gram matrix was singular even with the shift");
  return GMG_OK;
}

}  // namespace gmg
