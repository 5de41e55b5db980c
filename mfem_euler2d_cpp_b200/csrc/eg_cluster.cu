// Cell inverses at k = 6..8, where the matrix (307 KB at k = 6, 840 KB at
// k = 8) is larger than an SM's registers: a thread-block cluster holds one,
// every CTA the column tiles rank, rank + CL, ... of it in registers.
//
// The elimination is that of eg_cellinv.cuh. A panel's column belongs to one
// CTA, which writes it into the shared memory of all (12 to 21 KB over the
// SM-to-SM network per panel); a panel's pivot rows stay local, each CTA having
// its own columns of them. The CTA that owns the next pivot block's column
// inverts it and sends the inverse around. One cluster barrier per panel.
//
// Against the slab kernel this replaces (one CTA per cell, the system in L2, a
// search over all rows per column) the matrix crosses no memory during the
// elimination.
#include <cooperative_groups.h>

#include <algorithm>

#include "eg_condense.cuh"
#include "eg_internal.h"

namespace cg = cooperative_groups;

namespace eg {
namespace {

template <int Q, int WR_, int WC_, int CL_, int DED_>
struct ClCfg {
  static constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, MT = (M + 7) / 8, CL = CL_;
  // DED as in InvCfg
  static constexpr int WR = WR_, WC = WC_, DED = DED_, NW = WR * WC, THREADS = 32 * (NW + DED);
  static constexpr int CT = (MT + CL - 1) / CL;                           // column tiles per CTA
  static constexpr int TR = (MT + WR - 1) / WR, TC = (CT + WC - 1) / WC;  // tiles per warp
  static constexpr int PR = 8 * TR * WR, PC = 8 * TC * WC;
  static constexpr int TS = PC % 16 == 0 ? PC + 8 : PC;  // as in InvCfg
  static constexpr int PANELS = 2 * (8 * PR + 8 * TS);
};

// acc: the CTA's tiles (rows wr + a WR, global columns rank + CL (wc + b WC))
// of the matrix, identity on the padding; on return, of its inverse. panels,
// tiles as in invert_tiles, at the same offsets in every CTA; *bad is set in
// every CTA when the elimination cannot vouch for the result. Ends with a
// cluster barrier.
template <class C>
__device__ __forceinline__ void invert_tiles_cluster(double (&acc)[C::TR][C::TC][2], double *panels, double *tiles,
                                                     int *bad, cg::cluster_group &cluster) {
  constexpr int MT = C::MT, PR = C::PR, TS = C::TS, WR = C::WR, WC = C::WC, TR = C::TR, TC = C::TC, CL = C::CL;
  const int rank = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % WR, wc = warp / WR;
  const int gq = lane >> 2, tq = lane & 3;
  double *Tis = tiles + 128;
  const bool tiles_here = C::DED == 0 || warp < C::NW;
  bool fine = true;
  const auto pan = [&](int buf) { return panels + buf * (8 * PR + 8 * TS); };
  const auto top = [&](int buf) { return panels + buf * (8 * PR + 8 * TS) + 8 * PR; };
  const auto publish = [&](int nxt, int buf) {
    const int lt = nxt / CL;
    if (nxt % CL == rank && lt % WC == wc) {
#pragma unroll
      for (int b = 0; b < TC; ++b)
        if (wc + b * WC == lt) {
          double *P = pan(buf) + gq * 8 + 2 * tq;
#pragma unroll 1
          for (int r = 0; r < CL; ++r) {
            double *Pr = cluster.map_shared_rank(P, r);
#pragma unroll
            for (int a = 0; a < TR; ++a) {
              const bool diag = wr + a * WR == nxt;
              *reinterpret_cast<double2 *>(Pr + (wr + a * WR) * 64) =
                  make_double2(diag ? (gq == 2 * tq ? 1. : 0.) : -acc[a][b][0],
                               diag ? (gq == 2 * tq + 1 ? 1. : 0.) : -acc[a][b][1]);
            }
          }
        }
    }
    if (nxt % WR == wr) {
#pragma unroll
      for (int a = 0; a < TR; ++a)
        if (wr + a * WR == nxt) {
          double *W = top(buf) + gq * TS + 2 * tq;
#pragma unroll
          for (int b = 0; b < TC; ++b)
            *reinterpret_cast<double2 *>(W + (wc + b * WC) * 8) = make_double2(acc[a][b][0], acc[a][b][1]);
        }
    }
  };
  const auto publish_diagonal = [&](int i, int buf) {
    const int lt = i / CL;
    if (i % CL != rank || i % WR != wr || lt % WC != wc) return;
#pragma unroll
    for (int a = 0; a < TR; ++a)
      if (wr + a * WR == i) {
#pragma unroll
        for (int b = 0; b < TC; ++b)
          if (wc + b * WC == lt)
            *reinterpret_cast<double2 *>(tiles + buf * 64 + gq * 8 + 2 * tq) = make_double2(acc[a][b][0], acc[a][b][1]);
      }
  };
  // the warp's inverse pivot block, to every CTA
  const auto send_inverse = [&](double *Ti) {
    __syncwarp();
    const double2 v = *reinterpret_cast<const double2 *>(Ti + 2 * lane);
#pragma unroll 1
    for (int r = 0; r < CL; ++r)
      if (r != rank) *reinterpret_cast<double2 *>(cluster.map_shared_rank(Ti + 2 * lane, r)) = v;
  };
  if (tiles_here) {
    publish(0, 0);
    publish_diagonal(0, 1);
    publish_diagonal(1, 0);
  }
  cluster.sync();
  if (rank == 0 && warp == 0) {
    Invert8 inv;
    inv.v0 = tiles[64 + gq * 8 + 2 * tq];
    inv.v1 = tiles[64 + gq * 8 + 2 * tq + 1];
    inv.run(Tis);
    send_inverse(Tis);
    fine = inv.ok;
  }
  cluster.sync();
#pragma unroll 1
  for (int p = 0; p < MT; ++p) {
    const int buf = p & 1;
    const double ti0 = Tis[buf * 64 + gq * 8 + tq], ti1 = Tis[buf * 64 + gq * 8 + tq + 4];
    const double *P = pan(buf) + gq * 8 + 2 * tq, *W = top(buf) + tq * TS + gq;
    const auto pivot_rows = [&](int lt, double &b0, double &b1) {
      const bool pc = rank + CL * lt == p;
      const double t0 = pc ? (gq == tq ? 1. : 0.) : lds_one(W + lt * 8);
      const double t1 = pc ? (gq == tq + 4 ? 1. : 0.) : lds_one(W + 4 * TS + lt * 8);
      b0 = b1 = 0.;
      dmma_m8n8k4(b0, b1, t0, ti0);
      dmma_m8n8k4(b0, b1, t1, ti1);
      fine = fine && (pc || (fabs(b0) <= kMaxB && fabs(b1) <= kMaxB));
    };
    if (p + 1 < MT && (p + 1) % CL == rank && warp == (C::DED ? C::NW : ((p + 1) / CL) % C::NW)) {
      double b0, b1;
      pivot_rows((p + 1) / CL, b0, b1);
      const double2 w = *reinterpret_cast<const double2 *>(P + (p + 1) * 64);
      const double2 t = *reinterpret_cast<const double2 *>(tiles + buf * 64 + gq * 8 + 2 * tq);
      Invert8 inv;
      inv.v0 = t.x;
      inv.v1 = t.y;
      dmma_m8n8k4(inv.v0, inv.v1, w.x, b0);
      dmma_m8n8k4(inv.v0, inv.v1, w.y, b1);
      inv.run(Tis + (buf ^ 1) * 64);
      send_inverse(Tis + (buf ^ 1) * 64);
      fine = fine && inv.ok;
    }
    if (tiles_here) {
      if (p % CL == rank && (p / CL) % WC == wc) {
#pragma unroll
        for (int b = 0; b < TC; ++b)
          if (wc + b * WC == p / CL) {
#pragma unroll
            for (int a = 0; a < TR; ++a) acc[a][b][0] = acc[a][b][1] = 0.;
          }
      }
      if (p % WR == wr) {
#pragma unroll
        for (int a = 0; a < TR; ++a)
          if (wr + a * WR == p) {
#pragma unroll
            for (int b = 0; b < TC; ++b) acc[a][b][0] = acc[a][b][1] = 0.;
          }
      }
      double b0, b1;
      pivot_rows(wc, b0, b1);
#pragma unroll
      for (int b = 0; b < TC; ++b) {
        double n0 = 0., n1 = 0.;
#pragma unroll
        for (int a = 0; a < TR; a += 2) {
          const double2 w = lds_pair(P + (wr + a * WR) * 64);
          if (a + 1 < TR) {
            const double2 x = lds_pair(P + (wr + (a + 1) * WR) * 64);
            dmma_m8n8k4(acc[a][b][0], acc[a][b][1], w.x, b0);
            dmma_m8n8k4(acc[a + 1][b][0], acc[a + 1][b][1], x.x, b0);
            dmma_m8n8k4(acc[a][b][0], acc[a][b][1], w.y, b1);
            dmma_m8n8k4(acc[a + 1][b][0], acc[a + 1][b][1], x.y, b1);
          } else {
            dmma_m8n8k4(acc[a][b][0], acc[a][b][1], w.x, b0);
            dmma_m8n8k4(acc[a][b][0], acc[a][b][1], w.y, b1);
          }
          if (b + 1 < TC && a == 0) pivot_rows(wc + (b + 1) * WC, n0, n1);
        }
        b0 = n0;
        b1 = n1;
      }
      publish(p + 1, buf ^ 1);
      publish_diagonal(p + 2, buf ^ 1);
    }
    cluster.sync();
  }
  if (!fine)
    for (int r = 0; r < CL; ++r) *cluster.map_shared_rank(bad, r) = 1;
  cluster.sync();
}

// The CTA's tiles of the cell matrix, assembled in registers (the entries of
// assemble_cell), identity on the padding.
template <class C, int Q>
__device__ __forceinline__ void assemble_tiles(double (&acc)[C::TR][C::TC][2], const STab<Q> &st, const double *J,
                                               const double *FM, const Geo &g, int rank) {
  constexpr int M = C::M;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % C::WR, wc = warp / C::WR;
  const int gq = lane >> 2, tq = lane & 3;
  const double sx = g.dt * g.hy / g.area, sy = g.dt * g.hx / g.area;
#pragma unroll
  for (int a = 0; a < C::TR; ++a) {
    const int row = (wr + a * C::WR) * 8 + gq, i = row >> 2, c = row & 3, ix = i % Q, iy = i / Q;
#pragma unroll
    for (int b = 0; b < C::TC; ++b) {
      const int col = (rank + C::CL * (wc + b * C::WC)) * 8 + 2 * tq, jn = col >> 2, d = col & 3, jx = jn % Q, jy = jn / Q;
      double v0 = row == col ? 1. : 0., v1 = row == col + 1 ? 1. : 0.;
      if (row < M && col < M) {
        const double im = st.inv_mass(i);
        if (iy == jy) {
          const double e = im * sx * st.ew(jy), gd = im * st.tdx(jx, ix);
          const double f0 = e * (st.fb(0, jy, ix) * st.fb(0, jy, jx)), f1 = e * (st.fb(1, jy, ix) * st.fb(1, jy, jx));
          const double *j = J + kJacStride * jn + 4 * d + c, *m0 = FM + jy * kFaceStride + 4 * d + c,
                       *m1 = FM + (Q + jy) * kFaceStride + 4 * d + c;
          v0 += gd * j[0] + (f0 * m0[0] + f1 * m1[0]);
          v1 += gd * j[4] + (f0 * m0[4] + f1 * m1[4]);
        }
        if (ix == jx) {
          const double e = im * sy * st.ew(jx), gd = im * st.tdy(jy, iy);
          const double f2 = e * (st.fb(2, jx, iy) * st.fb(2, jx, jy)), f3 = e * (st.fb(3, jx, iy) * st.fb(3, jx, jy));
          const double *j = J + kJacStride * jn + 16 + 4 * d + c, *m2 = FM + (2 * Q + jx) * kFaceStride + 4 * d + c,
                       *m3 = FM + (3 * Q + jx) * kFaceStride + 4 * d + c;
          v0 += gd * j[0] + (f2 * m2[0] + f3 * m3[0]);
          v1 += gd * j[4] + (f2 * m2[4] + f3 * m3[4]);
        }
      }
      acc[a][b][0] = v0;
      acc[a][b][1] = v1;
    }
  }
}

// The CTA's columns of the inverse to global memory, column-major, stride M.
template <class C>
__device__ __forceinline__ void write_tiles(const double (&acc)[C::TR][C::TC][2], double *S, int rank) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % C::WR, wc = warp / C::WR;
  const int gq = lane >> 2, tq = lane & 3;
  if (C::DED && warp >= C::NW) return;
#pragma unroll
  for (int a = 0; a < C::TR; ++a)
#pragma unroll
    for (int b = 0; b < C::TC; ++b) {
      const int row = (wr + a * C::WR) * 8 + gq, col = (rank + C::CL * (wc + b * C::WC)) * 8 + 2 * tq;
      if (row < C::M && col < C::M) {
        __stcg(S + (size_t)col * C::M + row, acc[a][b][0]);
        __stcg(S + (size_t)(col + 1) * C::M + row, acc[a][b][1]);
      }
    }
}

// Row r of V B for the four sides (lift_row), V in global memory.
template <int Q>
__device__ __forceinline__ void lift_row_global(const double *lift, const double *V, int ld, int jc, double (&x)[4]) {
  const int jj = jc >> 2, c = jc & 3;
  double vx[Q], vy[Q];
#pragma unroll
  for (int l = 0; l < Q; ++l) {
    vx[l] = __ldcg(V + (size_t)(4 * (jj * Q + l) + c) * ld);
    vy[l] = __ldcg(V + (size_t)(4 * (l * Q + jj) + c) * ld);
  }
  x[0] = x[1] = x[2] = x[3] = 0.;
#pragma unroll
  for (int l = 0; l < Q; ++l) {
    x[0] += lift[jj * Q + l] * vx[l];
    x[1] += lift[(Q + jj) * Q + l] * vx[l];
    x[2] += lift[(2 * Q + jj) * Q + l] * vy[l];
    x[3] += lift[(3 * Q + jj) * Q + l] * vy[l];
  }
}

// Condensation of a cell per cluster. After the inversion A^{-1} goes to the
// cluster's scratch (L2-resident: 22 to 28 MB over all clusters) and the CTAs
// share the outputs: the columns of X, the rows of y, the four sides' C_s R_s
// A^{-1} and panels.
template <int Q, int WR, int WC, int CL, int DED>
__global__ void __launch_bounds__(32 * (WR * WC + DED), 1)
    condense_cluster_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                            const double *__restrict__ r, double *XY, double *Cb, double *sf_out, double *contrib,
                            double *panels, double *scratch, int *redo, int *redo_count) {
  using C = ClCfg<Q, WR, WC, CL, DED>;
  constexpr int M = C::M, T = C::T, NR = 4 * T + 1, TS = T + 2;
  __shared__ CondenseInvShared<Q> sh;
  __shared__ __align__(16) double tiles[256];
  extern __shared__ __align__(16) double dyn[];
  double *J = dyn + C::PANELS, *aux = J;  // the node Jacobians, later one side's C_s R_s A^{-1}
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), cid = blockIdx.x / CL, ncl = gridDim.x / CL;
  double *S = scratch + (size_t)cid * M * M;
  load_tables<Q>(sh.st, tab);
  for (int e = cid; e < g.n; e += ncl) {
    __syncthreads();
    condense_cell_data<Q>(sh, g, fz, u, r, Cb, sf_out, J, e, rank == 0);
    double acc[C::TR][C::TC][2];
    assemble_tiles<C, Q>(acc, sh.st, J, sh.FM, g, rank);
    // ends with a cluster barrier before any CTA's panels are written by another
    cluster.sync();
    invert_tiles_cluster<C>(acc, dyn, tiles, &sh.bad, cluster);
    if (sh.bad) {  // the same in every CTA
      if (rank == 0 && threadIdx.x == 0) redo[atomicAdd(redo_count, 1)] = e;
      cluster.sync();  // every CTA has read its flag
      continue;
    }
    write_tiles<C>(acc, S, rank);
    cluster.sync();
    double *X = XY + (size_t)e * M * NR;
    for (int t = threadIdx.x; t < M * ((T + CL - 1) / CL); t += blockDim.x) {
      const int row = t % M, jc = rank + CL * (t / M);
      if (jc >= T) break;
      double x[4];
      lift_row_global<Q>(sh.lift, S + row, M, jc, x);
#pragma unroll
      for (int s = 0; s < 4; ++s) X[(size_t)(s * T + jc) * M + row] = x[s];
    }
    // y = A^{-1} r on the rows [r0, r1), NG threads to a row
    {
      constexpr int RY = (M + CL - 1) / CL, NG = C::THREADS / RY > 8 ? 8 : C::THREADS / RY;
      const int row = rank * RY + (int)threadIdx.x % RY, part = (int)threadIdx.x / RY;
      double y = 0.;
      if (part < NG && row < M) {
#pragma unroll 8
        for (int c = part; c < M; c += NG) y += __ldcg(S + (size_t)c * M + row) * sh.rs[c];
      }
      __syncthreads();
      double *part_y = dyn;  // the panels are not in use
      if (part < NG) part_y[part * RY + threadIdx.x % RY] = y;
      __syncthreads();
      if (part == 0 && row < M) {
        double t = 0.;
        for (int k = 0; k < NG; ++k) t += part_y[k * RY + threadIdx.x];
        X[(size_t)(4 * T) * M + row] = t;
        *cluster.map_shared_rank(&sh.y[row], 0) = t;
      }
    }
    for (int s = rank; s < 4; s += CL) {
      __syncthreads();
      for (int t = threadIdx.x; t < Q * M; t += blockDim.x) {
        const int jj = t / M, col = t % M;
        double2 p0[Q], p1[Q];
#pragma unroll
        for (int l = 0; l < Q; ++l) {
          const double2 *p = reinterpret_cast<const double2 *>(S + (size_t)col * M + 4 * line_node<Q>(s, jj, l));
          p0[l] = __ldcg(p);
          p1[l] = __ldcg(p + 1);
        }
        double v[4] = {0., 0., 0., 0.};
#pragma unroll
        for (int l = 0; l < Q; ++l) {
          const double f = sh.st.fb(s, jj, l);
          v[0] += f * p0[l].x;
          v[1] += f * p0[l].y;
          v[2] += f * p1[l].x;
          v[3] += f * p1[l].y;
        }
        const double *cb = sh.CB + (s * Q + jj) * kFaceStride;
        double o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] = (cb[c] * v[0] + cb[c + 4] * v[1]) + (cb[c + 8] * v[2] + cb[c + 12] * v[3]);
        double2 *dst = reinterpret_cast<double2 *>(aux + (size_t)col * TS + 4 * jj);
        dst[0] = make_double2(o[0], o[1]);
        dst[1] = make_double2(o[2], o[3]);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < T * T; t += blockDim.x) {
        const int row = t % T, jc = t / T;
        double x[4];
        lift_row<Q>(sh.lift, aux + row, TS, jc, x);
#pragma unroll
        for (int o = 0; o < 4; ++o) panels[(((size_t)e * 16 + s * 4 + o) * T + jc) * T + row] = x[o];
      }
    }
    cluster.sync();  // y is complete in rank 0; the scratch and the flags may be written again
    if (rank == 0)
      for (int t = threadIdx.x; t < 4 * Q; t += blockDim.x) {  // C_s R_s y (src/condensation.cpp:141-142)
        double v[4] = {0., 0., 0., 0.};
        for (int l = 0; l < Q; ++l) {
          const double f = sh.st.fb(t / Q, t % Q, l);
          const double *p = sh.y + 4 * line_node<Q>(t / Q, t % Q, l);
#pragma unroll
          for (int d = 0; d < 4; ++d) v[d] += f * p[d];
        }
        const double *cb = sh.CB + t * kFaceStride;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          contrib[(size_t)e * 4 * T + 4 * t + c] = (cb[c] * v[0] + cb[c + 4] * v[1]) + (cb[c + 8] * v[2] + cb[c + 12] * v[3]);
      }
  }
  cluster.sync();  // no CTA leaves while another may write to its shared memory
}

// Explicit DG block-Jacobi inverses, column-major.
template <int Q, int WR, int WC, int CL, int DED>
__global__ void __launch_bounds__(32 * (WR * WC + DED), 1)
    dg_inverse_cluster_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                              double *inv, int *redo, int *redo_count) {
  using C = ClCfg<Q, WR, WC, CL, DED>;
  constexpr int M = C::M;
  __shared__ STab<Q> st;
  __shared__ __align__(16) double us[M], UT[16 * Q], FM[4 * Q * kFaceStride], tiles[256];
  __shared__ int bad;
  extern __shared__ __align__(16) double dyn[];
  double *J = dyn + C::PANELS;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), cid = blockIdx.x / CL, ncl = gridDim.x / CL;
  load_tables<Q>(st, tab);
  for (int e = cid; e < g.n; e += ncl) {
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) us[i] = u[(size_t)e * M + i];
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    cell_traces<Q>(st, us, UT);
    node_jacobians<Q>(J, st, us, g);
    __syncthreads();
    dg_face_matrices<Q, kFaceStride>(UT, FM, g, fz, e);
    __syncthreads();
    double acc[C::TR][C::TC][2];
    assemble_tiles<C, Q>(acc, st, J, FM, g, rank);
    cluster.sync();
    invert_tiles_cluster<C>(acc, dyn, tiles, &bad, cluster);
    if (bad) {
      if (rank == 0 && threadIdx.x == 0) redo[atomicAdd(redo_count, 1)] = e;
    } else {
      write_tiles<C>(acc, inv + (size_t)e * M * M, rank);
    }
    cluster.sync();  // every CTA has read its flag
  }
}

// Clusters of the kernel resident at once, and a launch of at most that many.
template <class Kern, class... Args>
void launch_cluster(Kern kern, int CL, int threads, size_t dyn, int clusters, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)CL;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(clusters * CL));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  EG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}
template <class Kern>
int resident_clusters(Kern kern, int CL, int threads, size_t dyn) {
  EG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)CL;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(64 * CL));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = dyn;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  EG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
  if (n < 1) fail(EG_ERR_CUDA, "no cluster of the cell inverse fits the device");
  return n;
}

template <int Q, int WR, int WC, int CL, int DED>
void condense_launch(Ctx &c, const double *u, const double *r) {
  using C = ClCfg<Q, WR, WC, CL, DED>;
  constexpr int AUX = kJacStride * C::P > C::M * (C::T + 2) ? kJacStride * C::P : C::M * (C::T + 2);
  constexpr size_t dyn = sizeof(double) * (size_t)(C::PANELS + AUX);
  auto kern = condense_cluster_kernel<Q, WR, WC, CL, DED>;
  const int clusters = std::min(c.n, resident_clusters(kern, CL, C::THREADS, dyn));
  if (c.work_gj == nullptr || c.work_gj_slots < clusters) {
    c.work_gj = c.alloc_n<double>((size_t)clusters * C::M * C::M);
    c.work_gj_slots = clusters;
  }
  launch_cluster(kern, CL, C::THREADS, dyn, clusters, c.stream, c.geo, (const double *)c.tab,
                 Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, r, c.XY, c.Cb, c.sf, c.contrib, c.panels, c.work_gj,
                 c.redo, c.derr + 3);
}
template <int Q, int WR, int WC, int CL, int DED>
void dg_launch(Ctx &c, const double *u) {
  using C = ClCfg<Q, WR, WC, CL, DED>;
  constexpr size_t dyn = sizeof(double) * (size_t)(C::PANELS + kJacStride * C::P);
  auto kern = dg_inverse_cluster_kernel<Q, WR, WC, CL, DED>;
  const int clusters = std::min(c.n, resident_clusters(kern, CL, C::THREADS, dyn));
  launch_cluster(kern, CL, C::THREADS, dyn, clusters, c.stream, c.geo, (const double *)c.tab,
                 Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, c.pc_dg, c.redo, c.derr + 3);
}

}  // namespace

// Shapes: the fewest CTAs whose registers hold the tiles (k = 6: 35 tiles for
// each of 10 warps and one more for the pivot blocks; k = 7: 16 for 16; k = 8:
// 28 for 12). What a panel needs besides is spilled in part: 518 bytes stored
// and 1416 loaded at k = 6 (140 of 168 registers are tiles), 48 and 216 at k =
// 7, 116 and 688 at k = 8. Clusters of 2 fill all 148 SMs, of 4 and 6 132.
// Condensation with a warp for the pivot blocks against tile warps in turn:
// 8.10 against 9.12 ms at k = 6 (64x64 cells), but 5.21 against 4.74 at k = 7
// and 13.3 against 11.8 at k = 8 (32x32), where it costs the others registers.
void launch_condense_cluster(Ctx &c, const double *u, const double *r) {
  switch (c.q) {
    case 7: condense_launch<7, 5, 2, 2, 1>(c, u, r); break;
    case 8: condense_launch<8, 4, 4, 4, 0>(c, u, r); break;
    case 9: condense_launch<9, 6, 2, 6, 0>(c, u, r); break;
    default: fail(EG_ERR_INVALID, "unsupported degree");
  }
}
void launch_dg_inverse_cluster(Ctx &c, const double *u) {
  switch (c.q) {
    case 7: dg_launch<7, 5, 2, 2, 1>(c, u); break;
    case 8: dg_launch<8, 4, 4, 4, 0>(c, u); break;
    case 9: dg_launch<9, 6, 2, 6, 0>(c, u); break;
    default: fail(EG_ERR_INVALID, "unsupported degree");
  }
}

}  // namespace eg
