// DG block Jacobi (PartialDGOperator::DiagonalBlocks, src/partial.cpp:265-298,
// factored as in src/linear.cpp:198-202 and applied by
// LinearSolver::Impl::Precondition, src/linear.cpp:66-75) as explicit inverses:
// every cell block is inverted in registers (eg_cellinv.cuh: one SM per cell
// for k <= 5; eg_cluster.cu: a cluster per cell above) and stored column-major,
// so that the apply streams each inverse once with full sectors and has no
// dependent steps. A block whose inverse the elimination cannot vouch for is
// inverted again through its LU with row pivoting.
//
// Measured against the Gauss-Jordan record (k = 3..5) and the LU sweeps (k >=
// 6) this replaces, with the solve in one kernel: a Newton update at 96x80 Q4
// 13.6 -> 10.0 ms.
#include <algorithm>

#include "eg_cellinv.cuh"
#include "eg_internal.h"

namespace eg {
namespace {

template <int Q, int WR, int WC, int DED, int MINB>
__global__ void __launch_bounds__(32 * (WR * WC + DED), MINB)
    dg_inverse_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u, double *inv,
                      int *redo, int *redo_count) {
  using C = InvCfg<Q, WR, WC, DED>;
  constexpr int M = C::M;
  __shared__ STab<Q> st;
  __shared__ __align__(16) double us[M], UT[16 * Q], FM[4 * Q * kFaceStride], tiles[256], J[kJacStride * Q * Q];
  __shared__ int bad;
  extern __shared__ __align__(16) double A[];
  load_tables<Q>(st, tab);
  for (int e = blockIdx.x; e < g.n; e += gridDim.x) {
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += C::THREADS) us[i] = u[(size_t)e * M + i];
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    cell_traces<Q>(st, us, UT);
    node_jacobians<Q>(J, st, us, g);
    __syncthreads();
    dg_face_matrices<Q, kFaceStride>(UT, FM, g, fz, e);
    __syncthreads();
    assemble_cell<C, Q>(A, st, J, FM, g);
    __syncthreads();
    double acc[C::TR][C::TC][2];
    load_tiles<C>(acc, A);
    __syncthreads();  // the panels take the matrix's place
    invert_tiles<C>(acc, A, tiles, &bad);
    if (bad) {
      if (threadIdx.x == 0) redo[atomicAdd(redo_count, 1)] = e;
      continue;
    }
    store_tiles<C>(acc, A);
    __syncthreads();
    double2 *dst = reinterpret_cast<double2 *>(inv + (size_t)e * M * M);
    for (int i = threadIdx.x; i < M * M / 2; i += C::THREADS)
      dst[i] = *reinterpret_cast<const double2 *>(A + (size_t)(2 * i / M) * C::LDA + 2 * i % M);
  }
}

// The listed cells' inverses from the LU with row pivoting of the block
// (applied to the identity), the block in a slab of global memory per CTA.
template <int Q>
__global__ void __launch_bounds__(256)
    dg_inverse_lu_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                         double *inv, double *work, const int *__restrict__ list, int count, int *err) {
  constexpr int M = 4 * Q * Q;
  __shared__ STab<Q> st;
  __shared__ double us[M], UT[16 * Q], FM[64 * Q], inv_piv[M], bcast[2];
  __shared__ int piv_s[M];
  load_tables<Q>(st, tab);
  double *A = work + (size_t)blockIdx.x * M * M;
  for (int item = blockIdx.x; item < count; item += gridDim.x) {
    const int e = list[item];
    double *R = inv + (size_t)e * M * M;
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) us[i] = u[(size_t)e * M + i];
    __syncthreads();
    cell_traces<Q>(st, us, UT);
    __syncthreads();
    dg_face_matrices<Q>(UT, FM, g, fz, e);
    __syncthreads();
    build_cell_matrix<Q>(A, M, st, us, FM, g);
    for (int i = threadIdx.x; i < M * M; i += blockDim.x) R[i] = i / M == i % M ? 1. : 0.;
    __syncthreads();
    const bool ok = cta_lu_solve<(M + 31) / 32>(A, M, R, M, M, M, piv_s, inv_piv, bcast);
    if (!ok && threadIdx.x == 0) raise_err(err, DERR_SINGULAR_JACOBI);
  }
}

// x_e = A_e^{-1} b_e, inverses column-major: one warp per cell, lane l holds
// rows 2l, 2l+1 (+ 64 s); the right-hand side is staged per warp in shared
// memory and broadcast column by column.
template <int M>
__global__ void __launch_bounds__(256) block_inverse_cm_apply_kernel(const double *__restrict__ inv, int nblocks,
                                                                     const double *__restrict__ b,
                                                                     double *__restrict__ x,
                                                                     const int *__restrict__ skip) {
  if (skip != nullptr && *skip) return;  // speculative Arnoldi step after convergence
  constexpr int S = (M + 63) / 64;
  __shared__ double bs[8][M];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = blockIdx.x * 8 + warp;
  if (blk >= nblocks) return;  // warp-uniform; nothing below synchronises the CTA
  for (int i = lane; i < M; i += 32) bs[warp][i] = b[(size_t)blk * M + i];
  __syncwarp();
  const double *A = inv + (size_t)blk * M * M;
  double acc[S][2];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s][0] = acc[s][1] = 0.;
#pragma unroll 4
  for (int c = 0; c < M; ++c) {
    const double bc = bs[warp][c];
    const double2 *col = reinterpret_cast<const double2 *>(A + (size_t)c * M);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r2 = lane + 32 * s;  // row pair
      if (2 * r2 < M) {
        const double2 v = __ldcs(col + r2);
        acc[s][0] = fma(v.x, bc, acc[s][0]);
        acc[s][1] = fma(v.y, bc, acc[s][1]);
      }
    }
  }
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int r2 = lane + 32 * s;
    if (2 * r2 < M) reinterpret_cast<double2 *>(x + (size_t)blk * M)[r2] = make_double2(acc[s][0], acc[s][1]);
  }
}

template <int Q, int WR, int WC, int DED, int MINB>
void launch_inverse(Ctx &c, const double *u) {
  using C = InvCfg<Q, WR, WC, DED>;
  constexpr size_t dyn = sizeof(double) * (size_t)C::REGION;
  auto kern = dg_inverse_kernel<Q, WR, WC, DED, MINB>;
  EG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  const int grid = std::min(c.n, device_sms() * MINB);
  kern<<<grid, C::THREADS, dyn, c.stream>>>(c.geo, c.tab, Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, c.pc_dg,
                                            c.redo, c.derr + 3);
}

}  // namespace

void launch_dg_inverse(Ctx &c, const double *u) {
  c.ensure_pc_dg();
  c.clear_redo();
  {
    ProfScope ps(c, EG_K_DG_JACOBI, 1);
    switch (c.q) {  // shapes as in the condensation, which does the same inversion
      case 1: launch_inverse<1, 1, 1, 0, 16>(c, u); break;
      case 2: launch_inverse<2, 1, 1, 0, 16>(c, u); break;
      case 3: launch_inverse<3, 1, 1, 0, 8>(c, u); break;
      case 4: launch_inverse<4, 2, 2, 0, 4>(c, u); break;
      case 5: launch_inverse<5, 2, 2, 0, 2>(c, u); break;
      case 6: launch_inverse<6, 5, 3, 1, 1>(c, u); break;
      default: launch_dg_inverse_cluster(c, u);
    }
    EG_CUDA(cudaGetLastError());
  }
  c.check_device_error();
  const int count = c.redo_count();
  if (count == 0) return;
  ProfScope ps(c, EG_K_DG_JACOBI, 1);
  c.ensure_work_cell(std::min(c.n, device_sms()));
  const int grid = std::min(count, c.work_slots);
  EG_DISPATCH_Q(c.q, (dg_inverse_lu_kernel<Q><<<grid, 256, 0, c.stream>>>(
                         c.geo, c.tab, Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, c.pc_dg, c.work_cell, c.redo,
                         count, c.derr)));
  EG_CUDA(cudaGetLastError());
  c.check_device_error();
}

void launch_dg_inverse_apply(Ctx &c, const double *b, double *x) {
  ProfScope ps(c, EG_K_PC_APPLY, 1);
  const int grid = (c.n + 7) / 8;
  EG_DISPATCH_Q(c.q, (block_inverse_cm_apply_kernel<4 * Q * Q><<<grid, 256, 0, c.stream>>>(c.pc_dg, c.n, b, x, c.skip)));
  EG_CUDA(cudaGetLastError());
}

}  // namespace eg
