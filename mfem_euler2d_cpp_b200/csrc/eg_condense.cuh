// Per-cell pieces of the HDG condensation shared by the kernels that invert a
// cell on one SM (eg_hdg.cu) and on a cluster of SMs (eg_cluster.cu). Not part
// of the public C-ABI.
#pragma once
#include "eg_cellinv.cuh"

namespace eg {

template <int Q>
struct CondenseInvShared {
  static constexpr int M = 4 * Q * Q;
  STab<Q> st;
  alignas(16) double us[M], rs[M], y[M], UT[16 * Q], FM[4 * Q * kFaceStride], CB[4 * Q * kFaceStride], SF[4 * Q], lift[4 * Q * Q];
  int bad;
};

// Traces, face matrices FM = sign J(U_own) + stab I (stab = a or b), flux
// blocks C = -ew FM and lift scalars B = -dt len/|K| ew stab of a cell
// (src/problem.cpp:622-630, 661-699), C and B also to global memory when
// `store`; the node Jacobians go to J.
template <int Q>
__device__ __forceinline__ void condense_cell_data(CondenseInvShared<Q> &sh, const Geo &g, const Frozen &fz,
                                                   const double *__restrict__ u, const double *__restrict__ r, double *Cb,
                                                   double *sf_out, double *J, int e, bool store = true) {
  constexpr int M = 4 * Q * Q;
  for (int i = threadIdx.x; i < M; i += blockDim.x) {
    sh.us[i] = u[(size_t)e * M + i];
    sh.rs[i] = r[(size_t)e * M + i];
  }
  if (threadIdx.x == 0) sh.bad = 0;
  __syncthreads();
  cell_traces<Q>(sh.st, sh.us, sh.UT);
  node_jacobians<Q>(J, sh.st, sh.us, g);
  __syncthreads();
  for (int task = threadIdx.x; task < 4 * Q; task += blockDim.x) {
    const int s = task / Q, j = task % Q;
    const bool L = side_is_left(s);
    const int fi = cell_face(e, s, g.nx, g.ny) * Q + j;
    const double stab = L ? fz.a[fi] : fz.b[fi], ewj = sh.st.ew(j), nsign = L ? 1. : -1.;
    double jm[16];
    jacobian_axis(sh.UT + 4 * task, s >> 1, g.gm1, jm);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const double v = nsign * jm[k] + ((k % 5) == 0 ? stab : 0.);
      sh.FM[task * kFaceStride + k] = v;
      sh.CB[task * kFaceStride + k] = -ewj * v;
    }
    const double sv = -(g.dt * (s < 2 ? g.hy : g.hx) / g.area * ewj) * stab;
    sh.SF[task] = sv;
    if (store) sf_out[(size_t)e * 4 * Q + task] = sv;
    for (int l = 0; l < Q; ++l) {
      const int i = line_node<Q>(s, j, l);
      sh.lift[task * Q + l] = sh.st.fb(s, j, l) * sh.st.inv_mass(i) * sv;
    }
  }
  __syncthreads();
  if (store)
    for (int i = threadIdx.x; i < 64 * Q; i += blockDim.x) Cb[(size_t)e * 64 * Q + i] = sh.CB[i / 16 * kFaceStride + i % 16];
}

// Row r of V B for the four sides, from a matrix V whose column c starts at V
// + c * ld: entry jc = 4 jj + c of every side is a weighted sum over the
// x-line (sides 0, 1) or the y-line (sides 2, 3) through face point jj.
template <int Q>
__device__ __forceinline__ void lift_row(const double *lift, const double *V, int ld, int jc, double (&x)[4]) {
  const int jj = jc >> 2, c = jc & 3;
  x[0] = x[1] = x[2] = x[3] = 0.;
#pragma unroll
  for (int l = 0; l < Q; ++l) {
    const double vx = V[(size_t)(4 * (jj * Q + l) + c) * ld], vy = V[(size_t)(4 * (l * Q + jj) + c) * ld];
    x[0] += lift[jj * Q + l] * vx;
    x[1] += lift[(Q + jj) * Q + l] * vx;
    x[2] += lift[(2 * Q + jj) * Q + l] * vy;
    x[3] += lift[(3 * Q + jj) * Q + l] * vy;
  }
}

}  // namespace eg
