// Static condensation kernels of the hybridised (HDG) Newton update.
//
// Device layout per cell e (m = 4p, t = 4q):
//   XY[e]      m x (4t+1) column-major: columns 0..4t-1 are X_e = A_e^{-1} B_e,
//              column 4t is y_e = A_e^{-1} r_e  (src/condensation.cpp:131-148);
//   Cb[e]      4q flux blocks C (4x4 column-major) of the face restriction;
//   sf[e]      4q lift scalars of B;
//   contrib[e] 4t face contributions of the last per-cell pass, combined per
//              face by a second pass (two contributions per face, no atomics,
//              deterministic).
#include <algorithm>

#include "eg_cellmat.cuh"
#include "eg_condense.cuh"
#include "eg_internal.h"

namespace eg {

// Shared-memory budget for the dense cell system (227 KB per CTA minus the
// static tables and staging arrays).
constexpr size_t kCellSmemBudget = 200 * 1024;
template <int Q>
__host__ __device__ constexpr int condense_mode() {
  // 0: A and [B|r] in shared memory; 1: A in shared memory, [B|r] in XY;
  // 2: A in a global workspace slab, [B|r] in XY.
  constexpr size_t M = 4 * Q * Q, NR = 16 * Q + 1;
  return sizeof(double) * M * (M + NR) <= kCellSmemBudget ? 0
         : (sizeof(double) * M * M <= kCellSmemBudget ? 1 : 2);
}
template <int Q>
__host__ __device__ constexpr size_t condense_dyn_bytes() {
  constexpr int M = 4 * Q * Q, NR = 16 * Q + 1;
  return condense_mode<Q>() == 0 ? sizeof(double) * (size_t)M * (M + NR)
                                 : (condense_mode<Q>() == 1 ? sizeof(double) * (size_t)M * M : 0);
}

// ---------------------------------------------------------- condensation
// Per-cell staging shared by both condensation kernels.
template <int Q>
struct CondenseShared {
  static constexpr int M = 4 * Q * Q;
  STab<Q> st;
  double us[M], UT[16 * Q], FM[4 * Q * 16], SF[4 * Q], CB[4 * Q * 16];
  int piv_s[M];
  double inv_piv[M];
  double bcast[2];
};

// Assemble the cell system: A (m x m) and [B | r_e] (m x (4t+1)), both
// column-major, A with leading dimension ld and [B | r_e] with ldr (ld when
// not given); also store C and the B scalars.
template <int Q>
__device__ void condense_build(CondenseShared<Q> &sh, const Geo &g, const Frozen &fz,
                               const double *__restrict__ u, const double *__restrict__ r, double *Cb,
                               double *sf_out, double *A, double *R, int e, int ld = 4 * Q * Q, int ldr = -1) {
  if (ldr < 0) ldr = ld;
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, NR = 4 * T + 1;
  const STab<Q> &st = sh.st;
  for (int i = threadIdx.x; i < M; i += blockDim.x) sh.us[i] = u[(size_t)e * M + i];
  __syncthreads();
  for (int task = threadIdx.x; task < 4 * Q; task += blockDim.x) {
    const int s = task / Q, j = task % Q;
    double o[4] = {0., 0., 0., 0.};
    for (int l = 0; l < Q; ++l) {
      const double f = st.fb(s, j, l);
      const double *v = sh.us + 4 * line_node<Q>(s, j, l);
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] += f * v[c];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) sh.UT[task * 4 + c] = o[c];
  }
  __syncthreads();
  // HDG face matrices (src/problem.cpp:661-699): derivative = sign J(U_own)
  // + stab I with stab = a (own left) or b (own right); C = -ew derivative;
  // B lift scalar = -dt len/|K| ew (a or b) (problem.cpp:622-630).
  for (int task = threadIdx.x; task < 4 * Q; task += blockDim.x) {
    const int s = task / Q, j = task % Q;
    const bool L = side_is_left(s);
    const int f = cell_face(e, s, g.nx, g.ny);
    const int fi = f * Q + j;
    const double stab = L ? fz.a[fi] : fz.b[fi];
    double jm[16];
    jacobian(sh.UT + 4 * task, s < 2 ? 0 : 1, g.gm1, jm);
    const double nsign = L ? 1. : -1.;
    const double ewj = st.ew(j);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const double v = nsign * jm[k] + ((k % 5) == 0 ? stab : 0.);
      sh.FM[task * 16 + k] = v;
      const double cv = -ewj * v;
      sh.CB[task * 16 + k] = cv;
      Cb[((size_t)e * 4 * Q + task) * 16 + k] = cv;
    }
    const double len = s < 2 ? g.hy : g.hx;
    const double scale = g.dt * len / g.area * ewj;
    const double sv = -scale * stab;
    sh.SF[task] = sv;
    sf_out[(size_t)e * 4 * Q + task] = sv;
  }
  __syncthreads();
  build_cell_matrix<Q>(A, ld, st, sh.us, sh.FM, g);
  if (R == nullptr) return;  // the caller forms [B | r_e] itself (lift_entry)
  for (int col = threadIdx.x; col < NR; col += blockDim.x) {
    double *rc = R + (size_t)col * ldr;
    if (col < 4 * T) {
      for (int i = 0; i < M; ++i) rc[i] = 0.;
      const int s = col / T, jj = (col % T) >> 2, c = col & 3;
      const double sv = sh.SF[s * Q + jj];
      for (int l = 0; l < Q; ++l) {
        const int i = line_node<Q>(s, jj, l);
        rc[4 * i + c] = st.fb(s, jj, l) * st.inv_mass(i) * sv;
      }
    } else {
      for (int i = 0; i < M; ++i) rc[i] = r[(size_t)e * M + i];
    }
  }
}

// Outputs of a solved cell: X|y to XY (unless already there), rhs
// contributions C_e y_e (src/condensation.cpp:141-142) and the Schur Jacobi
// panels C_s X_s (src/operators.cpp:7-26, 295-301).
template <int Q>
__device__ void condense_epilogue(const CondenseShared<Q> &sh, const double *R, bool copy_out, double *XY,
                                  double *contrib, double *panels, int npan, int e) {
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, NR = 4 * T + 1;
  const STab<Q> &st = sh.st;
  if (copy_out) {
    double *dst = XY + (size_t)e * M * NR;
    for (int i = threadIdx.x; i < M * NR; i += blockDim.x) dst[i] = R[i];
  }
  const double *y = R + (size_t)(4 * T) * M;
  for (int o = threadIdx.x; o < 4 * T; o += blockDim.x) {
    const int s = o / T, jj = (o % T) >> 2, c = o & 3;
    double val[4] = {0., 0., 0., 0.};
    for (int l = 0; l < Q; ++l) {
      const double f = st.fb(s, jj, l);
      const double *yv = y + 4 * line_node<Q>(s, jj, l);
#pragma unroll
      for (int d = 0; d < 4; ++d) val[d] += f * yv[d];
    }
    const double *cb = sh.CB + (s * Q + jj) * 16;
    double res = 0.;
#pragma unroll
    for (int d = 0; d < 4; ++d) res += cb[c + 4 * d] * val[d];
    contrib[(size_t)e * 4 * T + o] = res;
  }
  if (panels) {
    // the 4 diagonal panels, or all 16 ([s][o]) where the Schur action uses them
    const bool all16 = npan == 16;
    for (int o = threadIdx.x; o < npan * T * T; o += blockDim.x) {
      const int pan = o / (T * T), rem = o % (T * T);
      const int s = all16 ? pan >> 2 : pan, so = all16 ? pan & 3 : pan;
      const int row = rem % T, cc = rem / T;
      const int jj = row >> 2, c = row & 3;
      const double *xc = R + (size_t)(so * T + cc) * M;
      double val[4] = {0., 0., 0., 0.};
      for (int l = 0; l < Q; ++l) {
        const double f = st.fb(s, jj, l);
        const double *xv = xc + 4 * line_node<Q>(s, jj, l);
#pragma unroll
        for (int d = 0; d < 4; ++d) val[d] += f * xv[d];
      }
      const double *cb = sh.CB + (s * Q + jj) * 16;
      double res = 0.;
#pragma unroll
      for (int d = 0; d < 4; ++d) res += cb[c + 4 * d] * val[d];
      panels[(size_t)e * npan * T * T + o] = res;
    }
  }
}

// Generic condensation (any degree): CTA-cooperative LU on shared or global
// memory (StreamCondense, src/condensation.cpp:131-148).
template <int Q>
__global__ void __launch_bounds__(256)
    condense_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                    const double *__restrict__ r, double *XY, double *Cb, double *sf_out,
                    double *contrib, double *panels, double *work, const int *__restrict__ list, int count,
                    int *err) {
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, NR = 4 * T + 1;
  constexpr int MODE = condense_mode<Q>();
  __shared__ CondenseShared<Q> sh;
  extern __shared__ double dyn[];
  load_tables<Q>(sh.st, tab);
  for (int item = blockIdx.x; item < count; item += gridDim.x) {
    const int e = list[item];
    __syncthreads();
    double *A = MODE < 2 ? dyn : work + (size_t)blockIdx.x * M * M;
    double *R = MODE == 0 ? dyn + (size_t)M * M : XY + (size_t)e * M * NR;
    condense_build<Q>(sh, g, fz, u, r, Cb, sf_out, A, R, e);
    __syncthreads();
    const bool ok = cta_lu_solve<(M + 31) / 32>(A, M, R, M, M, NR, sh.piv_s, sh.inv_piv, sh.bcast);
    if (!ok) {
      if (threadIdx.x == 0) raise_err(err, DERR_SINGULAR_CELL);
      continue;
    }
    condense_epilogue<Q>(sh, R, MODE == 0, XY, contrib, panels, g.npan, e);
  }
}

// --------------------------------------- condensation (k <= 5): cell inverses
// Per cell: A is assembled in shared memory, inverted in registers by the
// block Gauss-Jordan of eg_cellinv.cuh, and written back; X = A^{-1} B, y and
// the panels follow from the inverse, since a column of B has q entries (the
// nodes of one line, weighted by `lift`). For m <= 144 that takes fewer flops
// than eliminating the 4t + 1 right-hand sides (2 m^3 against m^3 + 2 m^2
// (4t + 1): 2.0 against 2.6 M at k = 4), needs no registers for them, and the
// matrix fits an SM twice at k = 4.
// Bound by the FP64 tensor pipe while a cell is inverted and by shared memory
// while it is assembled and its panels are formed; several cells per SM overlap
// the two. Whole condensation, against the elimination of the right-hand sides
// this replaces, ms: k = 1 0.25 -> 0.107, k = 2 0.82 -> 0.39, k = 3 2.09 ->
// 1.01, k = 4 5.81 -> 3.47 (128x128 cells), k = 5 4.16 -> 2.11 (64x64).
// Without the padded strides (kJacStride, kFaceStride, TS; k = 4, 64x64) 1.07,
// with them 0.90.
template <int Q, int WR, int WC>
__host__ __device__ constexpr int condense_inv_aux() {  // doubles of J, later of one side's C R A^{-1}
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q;
  return kJacStride * P > M * (T + 2) ? kJacStride * P : M * (T + 2);
}

template <int Q, int WR, int WC, int DED, int MINB>
__global__ void __launch_bounds__(32 * (WR * WC + DED), MINB)
    condense_inv_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                        const double *__restrict__ r, double *XY, double *Cb, double *sf_out, double *contrib,
                        double *panels, int *redo, int *redo_count) {
  using C = InvCfg<Q, WR, WC, DED>;
  // TS: stride of C_s R_s A^{-1}; T + 2 is twice an odd number, so 16-byte
  // stores with lanes over columns use all banks
  constexpr int M = C::M, T = C::T, NR = 4 * T + 1, LDA = C::LDA, TS = T + 2;
  __shared__ CondenseInvShared<Q> sh;
  __shared__ __align__(16) double tiles[256];
  extern __shared__ __align__(16) double A[];
  double *aux = A + C::REGION;
  load_tables<Q>(sh.st, tab);
  for (int e = blockIdx.x; e < g.n; e += gridDim.x) {
    __syncthreads();
    condense_cell_data<Q>(sh, g, fz, u, r, Cb, sf_out, aux, e);
    assemble_cell<C, Q>(A, sh.st, aux, sh.FM, g);
    __syncthreads();
    double acc[C::TR][C::TC][2];
    load_tiles<C>(acc, A);
    __syncthreads();  // the panels take the matrix's place
    invert_tiles<C>(acc, A, tiles, &sh.bad);
    if (sh.bad) {
      if (threadIdx.x == 0) redo[atomicAdd(redo_count, 1)] = e;
      continue;
    }
    store_tiles<C>(acc, A);
    __syncthreads();
    double *X = XY + (size_t)e * M * NR;
    for (int t = threadIdx.x; t < M * T; t += blockDim.x) {
      const int row = t % M, jc = t / M;
      double x[4];
      lift_row<Q>(sh.lift, A + row, LDA, jc, x);
#pragma unroll
      for (int s = 0; s < 4; ++s) X[(size_t)(s * T + jc) * M + row] = x[s];
    }
    for (int row = threadIdx.x; row < M; row += blockDim.x) {
      double y[4] = {0., 0., 0., 0.};
#pragma unroll 4
      for (int c = 0; c < M; c += 4)
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] += A[row + (size_t)(c + k) * LDA] * sh.rs[c + k];
      const double v = (y[0] + y[1]) + (y[2] + y[3]);
      sh.y[row] = v;
      X[(size_t)(4 * T) * M + row] = v;
    }
    // one side at a time: C_s R_s A^{-1} (t x m, in aux), then its panels
    for (int s = 0; s < 4; ++s) {
      __syncthreads();
      for (int t = threadIdx.x; t < Q * M; t += blockDim.x) {
        const int jj = t / M, col = t % M;
        double v[4] = {0., 0., 0., 0.};
#pragma unroll
        for (int l = 0; l < Q; ++l) {
          const double f = sh.st.fb(s, jj, l);
          const double2 *p = reinterpret_cast<const double2 *>(A + (size_t)col * LDA + 4 * line_node<Q>(s, jj, l));
          const double2 p0 = p[0], p1 = p[1];
          v[0] += f * p0.x;
          v[1] += f * p0.y;
          v[2] += f * p1.x;
          v[3] += f * p1.y;
        }
        const double *cb = sh.CB + (s * Q + jj) * kFaceStride;
        double o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] = (cb[c] * v[0] + cb[c + 4] * v[1]) + (cb[c + 8] * v[2] + cb[c + 12] * v[3]);
        double2 *dst = reinterpret_cast<double2 *>(aux + (size_t)col * TS + 4 * jj);
        dst[0] = make_double2(o[0], o[1]);
        dst[1] = make_double2(o[2], o[3]);
      }
      if (s == 0) {
        // C_s R_s y of every side (src/condensation.cpp:141-142)
        for (int t = threadIdx.x; t < 4 * Q; t += blockDim.x) {
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
            contrib[(size_t)e * 4 * T + 4 * t + c] =
                (cb[c] * v[0] + cb[c + 4] * v[1]) + (cb[c + 8] * v[2] + cb[c + 12] * v[3]);
        }
      }
      __syncthreads();
      for (int t = threadIdx.x; t < T * T; t += blockDim.x) {
        const int row = t % T, jc = t / T;
        double x[4];
        lift_row<Q>(sh.lift, aux + row, TS, jc, x);
        if (g.npan == 16) {
#pragma unroll
          for (int o = 0; o < 4; ++o) panels[(((size_t)e * 16 + s * 4 + o) * T + jc) * T + row] = x[o];
        } else {
          panels[(((size_t)e * 4 + s) * T + jc) * T + row] = x[s];
        }
      }
    }
  }
}

// -------------------------------------------------- Schur action / recovery
// Per cell: gather the 4t trace values, mid = X_e v_e (GEMV streaming X once),
// then either restrict with C (Schur action, src/operators.cpp:166-178) or
// write du = -mid - y (Recover, src/condensation.cpp:28-41, 154-163).
template <int Q, bool RECOVER>
__global__ void __launch_bounds__(128)
    cell_gemv_kernel(Geo g, const double *__restrict__ tab, const double *__restrict__ XY,
                     const double *__restrict__ Cb, const double *__restrict__ v,
                     double *__restrict__ out, const int *__restrict__ skip) {
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, NR = 4 * T + 1;
  if (skip != nullptr && *skip) return;  // speculative Arnoldi step after convergence
  __shared__ STab<Q> st;
  __shared__ double vl[4 * T], mid[M];
  load_tables<Q>(st, tab);
  for (int e = blockIdx.x; e < g.n; e += gridDim.x) {
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * T; i += blockDim.x) {
      const int s = i / T;
      vl[i] = v[(size_t)cell_face(e, s, g.nx, g.ny) * T + (i % T)];
    }
    __syncthreads();
    const double *X = XY + (size_t)e * M * NR;
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      double acc = 0.;
#pragma unroll 8
      for (int col = 0; col < 4 * T; ++col) acc += X[(size_t)col * M + i] * vl[col];
      if (RECOVER) {
        out[(size_t)e * M + i] = -acc - X[(size_t)(4 * T) * M + i];
      } else {
        mid[i] = acc;
      }
    }
    if (!RECOVER) {
      __syncthreads();
      for (int o = threadIdx.x; o < 4 * T; o += blockDim.x) {
        const int s = o / T, jj = (o % T) >> 2, c = o & 3;
        double val[4] = {0., 0., 0., 0.};
        for (int l = 0; l < Q; ++l) {
          const double f = st.fb(s, jj, l);
          const double *mv = mid + 4 * line_node<Q>(s, jj, l);
#pragma unroll
          for (int d = 0; d < 4; ++d) val[d] += f * mv[d];
        }
        const double *cb = Cb + ((size_t)e * 4 * Q + s * Q + jj) * 16;
        double res = 0.;
#pragma unroll
        for (int d = 0; d < 4; ++d) res += cb[c + 4 * d] * val[d];
        out[(size_t)e * 4 * T + o] = res;
      }
    }
  }
}

// Schur action from the 16 panels of a cell (degrees with
// schur_panels_full, and every degree with element or full assembly, where the
// panels are the element entries C X of src/condensation.cpp:143-146):
// contrib[e][s] = sum_o (C_s X_o) v_o, the same product as the C restriction
// of X v (src/operators.cpp:166-178) with the C X panels formed once per
// condensation, so that each apply streams 16 t^2 doubles per cell instead of
// m x 4t. One thread per output (s, row); consecutive rows read consecutive
// panel entries.
template <int Q>
__global__ void __launch_bounds__(((16 * Q + 31) / 32) * 32)
    panel_gemv_kernel(Geo g, const double *__restrict__ panels, const double *__restrict__ v,
                      double *__restrict__ out, const int *__restrict__ skip) {
  constexpr int T = 4 * Q, TT = T * T;
  if (skip != nullptr && *skip) return;  // speculative Arnoldi step after convergence
  __shared__ double vl[4 * T];
  const int o = threadIdx.x, s = o / T, row = o % T;
  for (int e = blockIdx.x; e < g.n; e += gridDim.x) {
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * T; i += blockDim.x)
      vl[i] = v[(size_t)cell_face(e, i / T, g.nx, g.ny) * T + (i % T)];
    __syncthreads();
    if (o < 4 * T) {
      const double *P = panels + ((size_t)e * 16 + s * 4) * TT + row;
      double acc = 0.;
#pragma unroll 8
      for (int k = 0; k < 4 * T; ++k) acc += P[(size_t)(k / T) * TT + (k % T) * T] * vl[k];
      out[(size_t)e * 4 * T + o] = acc;
    }
  }
}

// y_f = D_f v_f - contrib[L][ls] - contrib[R][rs]  (one thread per trace dof)
__global__ void face_combine_kernel(int nx, int ny, int T, int nl, const double *__restrict__ D,
                                    const double *__restrict__ v, const double *__restrict__ contrib,
                                    double sign_v, double *__restrict__ y, const int *__restrict__ skip) {
  if (skip != nullptr && *skip) return;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nl) return;
  const int f = idx / T, i = idx % T;
  const int L = f >> 1, ls = (f & 1) ? 3 : 1;
  const int R = neighbour(L, ls, nx, ny), rs = ls - 1;
  const double base = D ? D[idx] * v[idx] : 0.;
  y[idx] = sign_v * ((base - contrib[(size_t)L * 4 * T + ls * T + i]) -
                     contrib[(size_t)R * 4 * T + rs * T + i]);
}

// er = -B (eq / D) (RecoveredResidual, src/stepper.cpp:10-26); one thread per
// (cell, node).
template <int Q>
__global__ void __launch_bounds__(256)
    recovered_residual_kernel(Geo g, const double *__restrict__ tab, const double *__restrict__ sf,
                              const double *__restrict__ D, const double *__restrict__ eq,
                              double *__restrict__ er) {
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q;
  __shared__ STab<Q> st;
  load_tables<Q>(st, tab);
  __syncthreads();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= g.n * P) return;
  const int e = idx / P, node = idx % P, ix = node % Q, iy = node / Q;
  const double im = st.inv_mass(node);
  double acc[4] = {0., 0., 0., 0.};
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int j = s < 2 ? iy : ix, l = s < 2 ? ix : iy;
    const int f = cell_face(e, s, g.nx, g.ny);
    const double wgt = st.fb(s, j, l) * im;
    const double a = sf[(size_t)e * 4 * Q + s * Q + j];
    const size_t base = (size_t)f * T + 4 * j;
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] += wgt * (a * (eq[base + c] / D[base + c]));
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) er[(size_t)e * M + 4 * node + c] = -acc[c];
}

// Schur block-Jacobi: S_ff = D_f - P_L - P_R (ElementOperator::DiagonalBlocks
// src/operators.cpp:275-303). With factor set, the block is inverted through
// its pivoted LU (LUFactors, src/linear.cpp:198-202) applied to the identity,
// and the explicit inverse is stored so the preconditioner apply is a
// coalesced batched GEMV instead of two dependent triangular sweeps.
template <int T>
__global__ void __launch_bounds__(64)
    schur_jacobi_kernel(int nx, int ny, int nf, int npan, const double *__restrict__ D,
                        const double *__restrict__ panels, double *blocks, int *pivots, bool factor,
                        int *err) {
  __shared__ double S[T * T], Inv[T * T];
  __shared__ int piv_s[T];
  __shared__ double inv_piv[T];
  __shared__ double bcast[2];
  for (int f = blockIdx.x; f < nf; f += gridDim.x) {
    __syncthreads();
    const int L = f >> 1, ls = (f & 1) ? 3 : 1;
    const int R = neighbour(L, ls, nx, ny), rs = ls - 1;
    // diagonal panels C_s X_s of the two cells (panel s*5 of 16 where all are kept)
    const bool all16 = npan == 16;
    const double *pl = panels + (all16 ? (size_t)L * 16 + ls * 5 : (size_t)L * 4 + ls) * T * T;
    const double *pr = panels + (all16 ? (size_t)R * 16 + rs * 5 : (size_t)R * 4 + rs) * T * T;
    for (int o = threadIdx.x; o < T * T; o += blockDim.x) {
      const int row = o % T, col = o / T;
      const double d = row == col ? D[(size_t)f * T + row] : 0.;
      S[o] = (d - pl[o]) - pr[o];
      Inv[o] = row == col ? 1. : 0.;
    }
    __syncthreads();
    const double *out = S;
    if (factor) {
      const bool ok = cta_lu_solve<(T + 31) / 32>(S, T, Inv, T, T, T, piv_s, inv_piv, bcast);
      if (!ok && threadIdx.x == 0) raise_err(err, DERR_SINGULAR_JACOBI);
      out = Inv;
    }
    for (int i = threadIdx.x; i < T; i += blockDim.x) pivots[(size_t)f * T + i] = factor ? piv_s[i] : i;
    for (int o = threadIdx.x; o < T * T; o += blockDim.x) blocks[(size_t)f * T * T + o] = out[o];
  }
}

// The same blocks inverted by one warp per face for T <= 32: lane r holds row
// r of [S | I] in registers and Gauss-Jordan runs with partial pivoting over
// the rows not yet used as pivot rows (largest magnitude, first row on ties,
// NaN never chosen; a zero pivot is singular, as in LU with row exchanges).
// Rows never move: the pivot row of step k ends up holding row k of S^{-1}.
// The pivot search is three warp reductions on IEEE bit patterns and the
// normalised pivot row is broadcast by shuffles, so no step needs a barrier.
// `pivots` receives the pivot row of every step.
template <int T>
__global__ void __launch_bounds__(128)
    schur_jacobi_warp_kernel(int nx, int ny, int nf, int npan, const double *__restrict__ D,
                             const double *__restrict__ panels, double *blocks, int *pivots, bool factor,
                             int *err) {
  static_assert(T <= 32, "one row per lane");
  constexpr unsigned long long kAbs = 0x7fffffffffffffffull, kInf = 0x7ff0000000000000ull;
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int f = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); f < nf; f += nwarps) {
    const int L = f >> 1, ls = (f & 1) ? 3 : 1;
    const int R = neighbour(L, ls, nx, ny), rs = ls - 1;
    // diagonal panels C_s X_s of the two cells (panel s*5 of 16 where all are kept)
    const bool all16 = npan == 16;
    const double *pl = panels + (all16 ? (size_t)L * 16 + ls * 5 : (size_t)L * 4 + ls) * T * T;
    const double *pr = panels + (all16 ? (size_t)R * 16 + rs * 5 : (size_t)R * 4 + rs) * T * T;
    const bool row_ok = lane < T;
    const double d = row_ok ? D[(size_t)f * T + lane] : 0.;
    double sr[T], xr[T];
#pragma unroll
    for (int c = 0; c < T; ++c) {
      sr[c] = row_ok ? ((lane == c ? d : 0.) - pl[c * T + lane]) - pr[c * T + lane] : 0.;
      xr[c] = lane == c ? 1. : 0.;
    }
    double *out = blocks + (size_t)f * T * T;  // column-major
    if (!factor) {
      if (row_ok) {
#pragma unroll
        for (int c = 0; c < T; ++c) out[c * T + lane] = sr[c];
        pivots[(size_t)f * T + lane] = lane;
      }
      continue;
    }
    bool un = row_ok;
    int pos = 0;
    bool singular = false;
#pragma unroll
    for (int k = 0; k < T; ++k) {
      double sk = 0.;
#pragma unroll
      for (int c = 0; c < T; ++c)
        if (c == k) sk = sr[c];
      const unsigned long long bits = (unsigned long long)__double_as_longlong(sk) & kAbs;
      const bool cand = un && bits <= kInf;
      const unsigned hi = cand ? (unsigned)(bits >> 32) : 0u, lo = cand ? (unsigned)bits : 0u;
      const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
      const bool c1 = cand && hi == mhi;
      const unsigned mlo = __reduce_max_sync(0xffffffffu, c1 ? lo : 0u);
      const unsigned pw = __reduce_min_sync(0xffffffffu, c1 && lo == mlo ? (unsigned)lane : 32u);
      // a zero pivot (warp-uniform) marks the block singular; the remaining
      // steps run on row 0 and their results are discarded
      const bool zero = pw >= 32u || (mhi == 0u && mlo == 0u);
      singular = singular || zero;
      const int p = zero ? 0 : (int)pw;
      const double l = sk;
      const double ip = 1.0 / __shfl_sync(0xffffffffu, l, p);
      const bool me = lane == p;
#pragma unroll
      for (int c = 0; c < T; ++c) {
        if (c > k) {
          const double v = __shfl_sync(0xffffffffu, sr[c], p) * ip;
          sr[c] = me ? v : sr[c] - l * v;
        }
      }
#pragma unroll
      for (int c = 0; c < T; ++c) {
        const double v = __shfl_sync(0xffffffffu, xr[c], p) * ip;
        xr[c] = me ? v : xr[c] - l * v;
      }
#pragma unroll
      for (int c = 0; c < T; ++c)
        if (c == k) sr[c] = me ? 1. : 0.;
      if (me) {
        un = false;
        pos = k;
      }
    }
    if (singular) {
      if (lane == 0) raise_err(err, DERR_SINGULAR_JACOBI);
      continue;
    }
    if (row_ok) {
#pragma unroll
      for (int c = 0; c < T; ++c) out[c * T + pos] = xr[c];
      pivots[(size_t)f * T + pos] = lane;
    }
  }
}

// x_b = Inv_b b_b for column-major BS x BS inverses: one thread per output
// row, so that neighbouring threads read neighbouring entries of a column; the
// column loop unrolls and all of a row's loads are in flight together.
template <int BS>
__global__ void __launch_bounds__(256) block_gemv_kernel(const double *__restrict__ inv, int nblocks,
                                                         const double *__restrict__ b, double *__restrict__ x) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (long long)nblocks * BS) return;
  const int blk = (int)(id / BS), row = (int)(id % BS);
  const double *a = inv + (size_t)blk * BS * BS + row;
  const double *bb = b + (size_t)blk * BS;
  double acc = 0.;
#pragma unroll
  for (int c = 0; c < BS; ++c) acc += a[c * BS] * bb[c];
  x[id] = acc;
}

// ================================================================ launchers
template <int Q, int WR, int WC, int DED, int MINB>
static void launch_condense_inv(Ctx &c, const double *u, const double *r) {
  using C = InvCfg<Q, WR, WC, DED>;
  constexpr size_t dyn = sizeof(double) * (size_t)(C::REGION + condense_inv_aux<Q, WR, WC>());
  auto kern = condense_inv_kernel<Q, WR, WC, DED, MINB>;
  EG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  const int grid = std::min(c.n, device_sms() * MINB);
  kern<<<grid, C::THREADS, dyn, c.stream>>>(c.geo, c.tab, Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, r, c.XY, c.Cb,
                                            c.sf, c.contrib, c.panels, c.redo, c.derr + 3);
}

// rhs_f = contrib_L + contrib_R (s.rhs = 0; rhs[ids] += C y)
static void launch_condensed_rhs(Ctx &c) {
  face_combine_kernel<<<(c.nl + 255) / 256, 256, 0, c.stream>>>(c.desc.nx, c.desc.ny, c.t, c.nl, nullptr, c.rhs,
                                                                c.contrib, -1.0, c.rhs, nullptr);
  EG_CUDA(cudaGetLastError());
}

// The cells whose inverse the kernels above could not vouch for, by LU with
// partial pivoting; `count` of them in c.redo.
static void condense_redo(Ctx &c, const double *u, const double *r, int count) {
  ProfScope ps(c, EG_K_CONDENSE, 2);
  const int grid = std::min(count, device_sms());
  EG_DISPATCH_Q(c.q, {
    constexpr size_t dyn = condense_dyn_bytes<Q>();
    auto kern = condense_kernel<Q>;
    if (dyn > 48 * 1024) EG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    if (condense_mode<Q>() == 2) c.ensure_work_cell(std::min(c.n, device_sms()));
    kern<<<grid, 256, dyn, c.stream>>>(c.geo, c.tab, Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, u, r, c.XY, c.Cb,
                                       c.sf, c.contrib, c.panels, c.work_cell, c.redo, count, c.derr);
  });
  EG_CUDA(cudaGetLastError());
  launch_condensed_rhs(c);
}

// Warps per cell and cells per SM: one warp holds the tiles up to k = 2, four
// at k = 3 and 4, with as many cells per SM as registers and shared memory
// allow (two warps at k = 2: 0.47 instead of 0.39 ms; four and one for the
// pivot blocks at k = 3: 1.19 instead of 1.01). At k = 5 one cell fills the SM,
// and the warp for the pivot blocks pays: 2.11 against 2.24 ms (2 x 5 tile warps
// instead of 5 x 3: 2.16). From k = 6 on a cell takes a cluster.
void condense_launch(Ctx &c, const double *u, const double *r) {
  c.ensure_hdg();
  c.clear_redo();
  {
    ProfScope ps(c, EG_K_CONDENSE, 2);
    switch (c.q) {
      case 1: launch_condense_inv<1, 1, 1, 0, 16>(c, u, r); break;
      case 2: launch_condense_inv<2, 1, 1, 0, 16>(c, u, r); break;
      case 3: launch_condense_inv<3, 1, 1, 0, 8>(c, u, r); break;
      case 4: launch_condense_inv<4, 2, 2, 0, 4>(c, u, r); break;
      case 5: launch_condense_inv<5, 2, 2, 0, 2>(c, u, r); break;
      case 6: launch_condense_inv<6, 5, 3, 1, 1>(c, u, r); break;
      default: launch_condense_cluster(c, u, r);
    }
    EG_CUDA(cudaGetLastError());
    launch_condensed_rhs(c);
  }
  c.condensed = true;
}

bool condense_finish(Ctx &c, const double *u, const double *r) {
  const int count = c.redo_count();
  if (count == 0) {
    c.raise_device_error();
    return false;
  }
  // an error raised so far is of work on the unfinished system
  EG_CUDA(cudaMemsetAsync(c.derr, 0, sizeof(int), c.stream));
  condense_redo(c, u, r, count);
  c.check_device_error();
  return true;
}

void condense(Ctx &c, const double *u, const double *r) {
  condense_launch(c, u, r);
  c.fetch_status();
  condense_finish(c, u, r);
}

void launch_schur_apply(Ctx &c, const double *v, double *y) {
  ProfScope ps(c, EG_K_SCHUR_APPLY, 2);
  const int grid = std::min(c.n, device_sms() * 16);
  if (c.geo.npan == 16) {
    switch (c.q) {
#define EG_PG(QQ)                                                                                          \
  case QQ:                                                                                                 \
    panel_gemv_kernel<QQ><<<grid, ((16 * QQ + 31) / 32) * 32, 0, c.stream>>>(c.geo, c.panels, v, c.contrib, \
                                                                            c.skip);                       \
    break;
      EG_PG(1) EG_PG(2) EG_PG(3) EG_PG(4) EG_PG(5) EG_PG(6) EG_PG(7) EG_PG(8) EG_PG(9)
#undef EG_PG
      default:
        fail(EG_ERR_INVALID, "unsupported degree");
    }
  } else {
    EG_DISPATCH_Q(c.q, (cell_gemv_kernel<Q, false><<<grid, 128, 0, c.stream>>>(c.geo, c.tab, c.XY, c.Cb,
                                                                              v, c.contrib, c.skip)));
  }
  EG_CUDA(cudaGetLastError());
  const int blocks = (c.nl + 255) / 256;
  face_combine_kernel<<<blocks, 256, 0, c.stream>>>(c.desc.nx, c.desc.ny, c.t, c.nl, c.D, v,
                                                    c.contrib, 1.0, y, c.skip);
  EG_CUDA(cudaGetLastError());
}

void launch_recover(Ctx &c, const double *lam, double *du) {
  ProfScope ps(c, EG_K_RECOVER, 1);
  const int grid = std::min(c.n, device_sms() * 16);
  EG_DISPATCH_Q(c.q, (cell_gemv_kernel<Q, true><<<grid, 128, 0, c.stream>>>(c.geo, c.tab, c.XY, c.Cb,
                                                                           lam, du, nullptr)));
  EG_CUDA(cudaGetLastError());
}

void launch_recovered_residual(Ctx &c, const double *eq, double *er) {
  const int total = c.n * c.p;
  ProfScope ps(c, EG_K_RECOVERED_RESIDUAL, 1);
  EG_DISPATCH_Q(c.q, (recovered_residual_kernel<Q><<<(total + 255) / 256, 256, 0, c.stream>>>(
                         c.geo, c.tab, c.sf, c.D, eq, er)));
  EG_CUDA(cudaGetLastError());
}

void launch_block_inverse_apply(Ctx &c, const double *inv, int nblocks, int bs, const double *b, double *x) {
  ProfScope ps(c, EG_K_PC_APPLY, 1);
  const long long total = (long long)nblocks * bs;
  const unsigned grid = (unsigned)((total + 255) / 256);
  switch (bs) {
#define EG_BG(BB)                                                                                  \
  case BB:                                                                                         \
    block_gemv_kernel<BB><<<grid, 256, 0, c.stream>>>(inv, nblocks, b, x);                         \
    break;
    EG_BG(4) EG_BG(8) EG_BG(12) EG_BG(16) EG_BG(20) EG_BG(24) EG_BG(28) EG_BG(32) EG_BG(36)
#undef EG_BG
    default:
      fail(EG_ERR_INVALID, "unsupported trace block size");
  }
  EG_CUDA(cudaGetLastError());
}

void launch_schur_jacobi(Ctx &c, bool factor) {
  c.ensure_pc_hdg();
  ProfScope ps(c, EG_K_SCHUR_JACOBI, 1);
  const int grid = std::min(c.nf, device_sms() * 32);
  const int wgrid = std::min((c.nf + 3) / 4, device_sms() * 32);  // 4 warps (faces) per CTA
  switch (c.t) {
#define EG_SJW(TT)                                                                                     \
  case TT:                                                                                             \
    schur_jacobi_warp_kernel<TT><<<wgrid, 128, 0, c.stream>>>(c.desc.nx, c.desc.ny, c.nf, c.geo.npan, c.D, c.panels, \
                                                              c.pc_hdg, c.piv_hdg, factor, c.derr);      \
    break;
    EG_SJW(4) EG_SJW(8) EG_SJW(12) EG_SJW(16) EG_SJW(20) EG_SJW(24) EG_SJW(28) EG_SJW(32)
#undef EG_SJW
    case 36:
      schur_jacobi_kernel<36><<<grid, 64, 0, c.stream>>>(c.desc.nx, c.desc.ny, c.nf, c.geo.npan, c.D, c.panels, c.pc_hdg,
                                                         c.piv_hdg, factor, c.derr);
      break;
    default:
      fail(EG_ERR_INVALID, "unsupported trace block size");
  }
  EG_CUDA(cudaGetLastError());
}

}  // namespace eg

// Element-wise pivot_reciprocal of n values (host arrays), for the test that
// bounds it against IEEE division.
namespace eg {
namespace {
__global__ void pivot_reciprocal_kernel(long long n, const double *__restrict__ x, double *__restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = pivot_reciprocal(x[i]);
}
}  // namespace
}  // namespace eg

extern "C" int eg_check_pivot_reciprocal(const double *x, double *y, long long n) {
  if (!x || !y || n <= 0) return EG_ERR_INVALID;
  double *d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * 2 * (size_t)n) != cudaSuccess) {
    cudaGetLastError();
    return EG_ERR_OUT_OF_MEMORY;
  }
  cudaError_t e = cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    eg::pivot_reciprocal_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 1024), 256>>>(n, d, d + n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return EG_ERR_CUDA;
  }
  return EG_OK;
}
