// Restarted CGS2 GMRES with block Jacobi as one cooperative kernel: the whole
// solve (LinearSolver::Impl, src/linear.cpp:76-157) runs in a single launch,
// one CTA per SM at most, with grid barriers between its phases.
//
// Why: an Arnoldi step of the host-driven loop (eg_krylov.cu) is seven
// launches (preconditioner, two operator kernels, three CGS passes,
// normalisation), each with its own ramp-up and a last-block reduction tail,
// and one host round trip per four steps. Below about 1e5 unknowns nearly all
// of the step is that latency. Measured, whole Newton updates before and after:
// 8x8 Q2 1.83 -> 0.72 ms (30 steps), DG 63x45 Q1 1.78 -> 0.86; at 128x128 Q4 a
// step takes 0.202 ms, 0.74 of the copy bandwidth for the operator's bytes.
//
// One step, with CTA b owning the cells [e0, e1) and the vector entries of
// those cells (HDG: their faces 2e and 2e + 1; DG: their nodes):
//   operator    contributions of the CTA's cells (HDG) or
//               values of its faces (DG), then its cells    | grid barrier
//   pass 1      w = A z on the CTA's entries; V^T M w        | grid barrier
//   pass 2      w -= V h; V^T M w and w^T M w                | grid barrier
//   pass 3      w -= V h2; V_{j+1} = w / |w|; z = P V_{j+1}  | grid barrier
// Sums are formed per CTA, published and added by every CTA in the same fixed
// order, so all CTAs hold the same Hessenberg column and take the same
// decisions; the result is bitwise reproducible for a given problem and
// device. |w| after pass 3 is sqrt(w'^T M w' - |h2|^2) with w' the vector
// after pass 2 (Pythagoras: h2 are the coefficients of its M-orthogonal
// projection); where that difference cancels (|h2|^2 above a quarter of
// w'^T M w') the norm is formed by a reduction of its own instead.
//
// Barriers are bounded in time: a CTA that waits longer than the limit
// records DERR_WAIT_LIMIT and sets the abort word, and every CTA leaves at its
// next barrier.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "eg_internal.h"

namespace eg {
namespace {

constexpr int kGT = 512;          // threads per CTA
constexpr int kGW = kGT / 32;     // warps per CTA
constexpr int kGC = 24;           // most basis columns kept in registers (restart <= kGC)

struct GridBar {
  unsigned *count;  // arrivals since the launch (zeroed before it)
  int *abort;
  int *err;
  unsigned long long limit_ns;
  int starve;  // test setting: no barrier is ever met
};

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier of all CTAs of the launch; `target` counts the arrivals this CTA has
// waited for so far. Returns false, CTA-uniformly, once the launch is aborted.
__device__ __forceinline__ bool grid_barrier(const GridBar &b, unsigned &target) {
  __shared__ int ok;
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.count) : "memory");
    const unsigned want = b.starve ? target + 1u : target;
    unsigned long long t0 = 0;
    int good = 1;
    for (unsigned it = 0;; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(b.count) : "memory");
      if ((int)(v - want) >= 0) break;
      if ((it & 255u) == 255u) {
        if (*(volatile int *)b.abort) {
          good = 0;
          break;
        }
        const unsigned long long now = gtimer();
        if (t0 == 0) t0 = now;
        if (now - t0 > b.limit_ns) {
          atomicExch(b.abort, 1);
          raise_err(b.err, DERR_WAIT_LIMIT);
          good = 0;
          break;
        }
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Sums of NC per-lane values over a warp with the values halved at every
// exchange (NC - 1 + log2(32 / NC) shuffles instead of 5 NC): returns the sum
// of column `col` of the lane, NC a power of two.
template <int NC>
__device__ __forceinline__ double warp_sum_columns(double (&v)[NC], int &col) {
  const int lane = threadIdx.x & 31;
  int off = 16;
  col = 0;
#pragma unroll
  for (int n = NC; n > 1; n >>= 1, off >>= 1) {
    const bool up = (lane & off) != 0;
    const int half = n / 2;
#pragma unroll
    for (int k = 0; k < NC / 2; ++k)
      if (k < half) {
        const double send = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    if (up) col += half;
  }
  double s = v[0];
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}
__device__ __forceinline__ double warp_sum(double s) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

struct SolveShared {
  double h[(kGC + 1) * kGC];  // column-major, leading dimension kGC + 1
  double g[kGC + 1], cs[kGC], sn[kGC], y[kGC];
  double h1[kGC + 1], h2[kGC + 1];  // first and second projections; [ncols]: the norm
  double red[kGW][kGC + 1];
  double mt[2 * EG_MAX_P];
  int stop, err;
};

// Adds the CTA's columns acc[0..nc) (and `extra` as column nc when with_extra)
// and publishes them: partials[col * gridDim + cta].
template <int NC>
__device__ __forceinline__ void publish_columns(SolveShared &sh, double (&acc)[NC], int nc, bool with_extra,
                                                double extra, double *partials) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (NC == 24) {
    double lo[16], hi[8];
#pragma unroll
    for (int k = 0; k < 16; ++k) lo[k] = acc[k];
#pragma unroll
    for (int k = 0; k < 8; ++k) hi[k] = acc[16 + k];
    int c0, c1;
    const double s0 = warp_sum_columns<16>(lo, c0), s1 = warp_sum_columns<8>(hi, c1);
    if ((lane & 1) == 0) sh.red[warp][c0] = s0;
    if ((lane & 3) == 0) sh.red[warp][16 + c1] = s1;
  } else {
    int c0;
    const double s0 = warp_sum_columns<NC>(acc, c0);
    if ((lane & (32 / NC - 1)) == 0) sh.red[warp][c0] = s0;
  }
  __syncwarp();
  if (with_extra) {
    extra = warp_sum(extra);
    if (lane == 0) sh.red[warp][nc] = extra;  // column nc of the padding is not used
  }
  __syncthreads();
  const int total = nc + (with_extra ? 1 : 0);
  if ((int)threadIdx.x < total) {
    double t[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int w = 0; w < kGW; ++w) t[w & 3] += sh.red[w][threadIdx.x];
    __stcg(partials + (size_t)threadIdx.x * gridDim.x + blockIdx.x, (t[0] + t[1]) + (t[2] + t[3]));
  }
}
// The same for one value.
__device__ __forceinline__ void publish_one(SolveShared &sh, double v, double *partials) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh.red[warp][0] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.;
    for (int w = 0; w < kGW; ++w) t += sh.red[w][0];
    __stcg(partials + blockIdx.x, t);
  }
}
// out[c] = sum of the published column c over the CTAs, in the same order in
// every CTA (lane l adds CTAs l, l + 32, ..., then a warp tree).
__device__ __forceinline__ void collect_columns(int total, const double *partials, double *out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
  for (int c = warp; c < total; c += kGW) {
    const double *p = partials + (size_t)c * G;
    double t = 0.;
    for (int b = lane; b < G; b += 32) t += __ldcg(p + b);
    t = warp_sum(t);
    if (lane == 0) out[c] = t;
  }
  __syncthreads();
}

// --------------------------------------------------------------- operators
// HDG Schur action and Schur block Jacobi. PAN: from the 16 panels C_s X_o of
// a cell (16 t^2 entries); otherwise from X (m x 4t) and the restriction C.
// S warps share a cell (S a power of two, so that a CTA with few cells still
// has most of its warps loading): each takes a slice of the 4t columns and
// the slices are added in shared memory.
template <int Q, class T, bool PAN>
struct HdgOp {
  using Real = T;
  static constexpr int P = Q * Q, M = 4 * P, TT = 4 * Q, K = 4 * TT;  // TT: trace entries per face
  static constexpr int ROWS = PAN ? K : M, RO = (ROWS + 31) / 32;
  // columns whose loads are in flight together: a warp with a whole cell (UN),
  // and one with a slice of it (UC; predicated, so short slices are one round)
  static constexpr int UN = RO <= 2 ? 16 : 8, UC = RO <= 3 ? 9 : RO == 4 ? 7 : 5;
  struct Args {
    Geo g;
    const double *tab, *Cb;
    const T *act;      // panels, or X
    size_t cell_stride;  // entries of act per cell
    const T *D, *pc;   // pc: block inverses, column-major
    T *contrib;
    int split;         // S
  };
  struct Shared {
    T v[kGW][K];
    T part[kGW][ROWS];
    double fb[PAN ? 1 : 4 * P];
  };
  static __device__ __forceinline__ void setup(const Args &a, Shared &sh) {
    if constexpr (!PAN)
      for (int i = threadIdx.x; i < 4 * P; i += blockDim.x) sh.fb[i] = a.tab[TabLayout<Q>::FB + i];
  }
  // entries [0, K) of C_e X_e v_e from mid = X_e v_e
  static __device__ __forceinline__ T restrict_entry(const Args &a, const Shared &sh, const T *mid, int e, int o) {
    const int s = o / TT, jj = (o % TT) >> 2, c = o & 3;
    T val[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int l = 0; l < Q; ++l) {
      const T f = (T)sh.fb[(s * Q + jj) * Q + l];
      const T *mv = mid + 4 * line_node<Q>(s, jj, l);
#pragma unroll
      for (int d = 0; d < 4; ++d) val[d] += f * mv[d];
    }
    const double *cb = a.Cb + ((size_t)e * 4 * Q + s * Q + jj) * 16;
    T res = T(0);
#pragma unroll
    for (int d = 0; d < 4; ++d) res += (T)cb[c + 4 * d] * val[d];
    return res;
  }
  // contributions of the cells [e0, e1) for the trace vector x
  static __device__ __forceinline__ bool apply(const Args &a, Shared &sh, const T *x, T *, int e0, int e1,
                                               const GridBar &bar, unsigned &target) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int S = a.split, slots = kGW / S, slice = warp % S, slot = warp / S;
    const int kper = (K + S - 1) / S, k0 = min(K, slice * kper), k1 = min(K, k0 + kper);
    const int rounds = (e1 - e0 + slots - 1) / slots;
    for (int rd = 0; rd < rounds; ++rd) {
      const int e = e0 + rd * slots + slot;
      const bool on = e < e1;
      if (on) {
        T *sv = sh.v[warp];
        const T *A = a.act + (size_t)e * a.cell_stride;
        T acc[RO];
        const T *base[RO];
#pragma unroll
        for (int r = 0; r < RO; ++r) {
          const int o = min(lane + 32 * r, ROWS - 1);
          acc[r] = T(0);
          base[r] = PAN ? A + (size_t)(o / TT) * 4 * TT * TT + o % TT : A + o;
        }
        // column k of the panel row (s, .) is panel o = k / t, column k % t:
        // consecutive columns are t (PAN) or m entries apart
        constexpr int LD = PAN ? TT : M;
        const auto gather = [&] {
          for (int i = k0 + lane; i < k1; i += 32)
            sv[i] = __ldcg(x + (size_t)cell_face(e, i / TT, a.g.nx, a.g.ny) * TT + (i % TT));
          __syncwarp();
        };
        if (S == 1) {
          gather();
#pragma unroll UN
          for (int k = 0; k < K; ++k) {
            const T xv = sv[k];
#pragma unroll
            for (int r = 0; r < RO; ++r)
              if (lane + 32 * r < ROWS) acc[r] += __ldcs(base[r] + (size_t)k * LD) * xv;
          }
        } else {
          T col[UC][RO];
          for (int k = k0; k < k1; k += UC) {
#pragma unroll
            for (int u = 0; u < UC; ++u)
#pragma unroll
              for (int r = 0; r < RO; ++r)
                col[u][r] = (k + u < k1 && lane + 32 * r < ROWS) ? __ldcs(base[r] + (size_t)(k + u) * LD) : T(0);
            if (k == k0) gather();
#pragma unroll
            for (int u = 0; u < UC; ++u) {
              const T xv = sv[min(k + u, k1 - 1)];
#pragma unroll
              for (int r = 0; r < RO; ++r) acc[r] += col[u][r] * xv;
            }
          }
        }
        if (PAN && S == 1) {
#pragma unroll
          for (int r = 0; r < RO; ++r)
            if (lane + 32 * r < ROWS) __stcg(a.contrib + (size_t)e * K + lane + 32 * r, acc[r]);
        } else {
#pragma unroll
          for (int r = 0; r < RO; ++r)
            if (lane + 32 * r < ROWS) sh.part[warp][lane + 32 * r] = acc[r];
        }
        __syncwarp();
        if (!PAN && S == 1)
          for (int o = lane; o < K; o += 32)
            __stcg(a.contrib + (size_t)e * K + o, restrict_entry(a, sh, sh.part[warp], e, o));
        __syncwarp();
      }
      if (S > 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < slots * ROWS; i += blockDim.x) {
          const int sl = i / ROWS, o = i % ROWS, ee = e0 + rd * slots + sl;
          if (ee < e1) {
            T t = sh.part[sl * S][o];
            for (int k = 1; k < S; ++k) t += sh.part[sl * S + k][o];
            if (PAN)
              __stcg(a.contrib + (size_t)ee * K + o, t);
            else
              sh.part[sl * S][o] = t;
          }
        }
        __syncthreads();
        if constexpr (!PAN) {
          for (int i = threadIdx.x; i < slots * K; i += blockDim.x) {
            const int sl = i / K, o = i % K, ee = e0 + rd * slots + sl;
            if (ee < e1) __stcg(a.contrib + (size_t)ee * K + o, restrict_entry(a, sh, sh.part[sl * S], ee, o));
          }
          __syncthreads();
        }
      }
    }
    return grid_barrier(bar, target);
  }
  // entry i of A x once the contributions are complete
  static __device__ __forceinline__ T value(const Args &a, const T *x, const T *, int i) {
    const int f = i / TT, r = i % TT;
    const int L = f >> 1, ls = (f & 1) ? 3 : 1;
    const int R = neighbour(L, ls, a.g.nx, a.g.ny), rs = ls - 1;
    return (a.D[i] * x[i] - __ldcg(a.contrib + (size_t)L * K + ls * TT + r)) -
           __ldcg(a.contrib + (size_t)R * K + rs * TT + r);
  }
  // z = P v on the entries [i0, i1) (whole blocks); v was written by this CTA
  static __device__ __forceinline__ void precondition(const Args &a, Shared &, const T *v, T *z, int, int, int i0,
                                                      int i1) {
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
      const int f = i / TT, r = i % TT;
      const T *inv = a.pc + (size_t)f * TT * TT + r, *b = v + (size_t)f * TT;
      T acc = T(0);
#pragma unroll
      for (int c = 0; c < TT; ++c) acc += __ldcs(inv + c * TT) * b[c];
      __stcg(z + i, acc);
    }
  }
};

// DG partial assembly (the cached Jacobians of dg_refresh_*_kernel, eg_cell.cu)
// and explicit cell-block inverses. The face values of the CTA's own faces come
// first (each face point once), a grid barrier, then the cells, whose values
// stay in w. S warps share a cell's inverse, as above.
template <int Q>
struct DgOp {
  using Real = double;
  static constexpr int P = Q * Q, M = 4 * P, CPB = (kGT / P) < 64 ? kGT / P : 64;
  static constexpr int R2 = (M / 2 + 31) / 32;  // row pairs per lane
  struct Args {
    Geo g;
    const double *tab, *vol, *face, *inv;
    double *hface;
    int split;  // S
  };
  struct Shared {
    double fb[4 * P], tdx[P], tdy[P], im[P], ew[Q];
    union {
      struct {
        double fx[CPB][P][4], fy[CPB][P][4], hs[CPB][4 * Q][4];
      } cell;
      struct {
        double v[kGW][M], part[kGW][M];
      } pc;
    };
  };
  static __device__ __forceinline__ void setup(const Args &a, Shared &sh) {
    using L = TabLayout<Q>;
    for (int i = threadIdx.x; i < 4 * P; i += blockDim.x) sh.fb[i] = a.tab[L::FB + i];
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      sh.tdx[i] = a.tab[L::TDX + i];
      sh.tdy[i] = a.tab[L::TDY + i];
      sh.im[i] = a.tab[L::IM + i];
    }
    for (int i = threadIdx.x; i < Q; i += blockDim.x) sh.ew[i] = a.tab[L::EW + i];
  }
  // trace of x on side s of cell c at face point j
  static __device__ __forceinline__ void trace(const Shared &sh, const double *x, int c, int s, int j, double (&o)[4]) {
    const double2 *cell = reinterpret_cast<const double2 *>(x + (size_t)c * M);
    o[0] = o[1] = o[2] = o[3] = 0.;
#pragma unroll
    for (int l = 0; l < Q; ++l) {
      const double f = sh.fb[(s * Q + j) * Q + l];
      const int node = line_node<Q>(s, j, l);
      const double2 v0 = __ldcg(cell + 2 * node), v1 = __ldcg(cell + 2 * node + 1);
      o[0] += f * v0.x;
      o[1] += f * v0.y;
      o[2] += f * v1.x;
      o[3] += f * v1.y;
    }
  }
  static __device__ __forceinline__ bool apply(const Args &a, Shared &sh, const double *x, double *w, int e0, int e1,
                                               const GridBar &bar, unsigned &target) {
    const Geo &g = a.g;
    const long long nq = (long long)g.nf * Q, np = (long long)g.n * P;
    for (int idx = 2 * e0 * Q + (int)threadIdx.x; idx < 2 * e1 * Q; idx += blockDim.x) {
      const int f = idx / Q, j = idx % Q, L = f >> 1, axis = f & 1, sl = axis ? 3 : 1;
      double cf[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) cf[k] = __ldcs(a.face + k * nq + idx);
      double xl[4], xr[4], h[4] = {0., 0., 0., 0.};
      trace(sh, x, L, sl, j, xl);
      trace(sh, x, neighbour(L, sl, g.nx, g.ny), sl - 1, j, xr);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) h[r] += cf[r + 4 * c] * xl[c] + cf[16 + r + 4 * c] * xr[c];
      const double scale = g.dt * (axis == 0 ? g.hy : g.hx) / g.area * sh.ew[j];
      double2 *o = reinterpret_cast<double2 *>(a.hface) + (size_t)idx * 2;
      __stcg(o, make_double2(scale * h[0], scale * h[1]));
      __stcg(o + 1, make_double2(scale * h[2], scale * h[3]));
    }
    if (!grid_barrier(bar, target)) return false;
    const int lc = threadIdx.x / P, node = threadIdx.x % P, ix = node % Q, iy = node / Q;
    for (int eb = e0; eb < e1; eb += CPB) {
      const int e = eb + lc;
      const bool on = lc < CPB && e < e1;
      double xx[4];
      if (on) {
        const double2 *xv = reinterpret_cast<const double2 *>(x + (size_t)e * M + 4 * node);
        const double2 x0 = __ldcg(xv), x1 = __ldcg(xv + 1);
        xx[0] = x0.x;
        xx[1] = x0.y;
        xx[2] = x1.x;
        xx[3] = x1.y;
        const long long idx = (long long)e * P + node;
        double fx[4] = {0., 0., 0., 0.}, fy[4] = {0., 0., 0., 0.};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            fx[r] += __ldcs(a.vol + (r + 4 * c) * np + idx) * xx[c];
            fy[r] += __ldcs(a.vol + (16 + r + 4 * c) * np + idx) * xx[c];
          }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          sh.cell.fx[lc][node][c] = fx[c];
          sh.cell.fy[lc][node][c] = fy[c];
        }
        for (int task = node; task < 4 * Q; task += P) {
          const int s = task / Q, j = task % Q;
          const double2 *h = reinterpret_cast<const double2 *>(a.hface) + ((size_t)cell_face(e, s, g.nx, g.ny) * Q + j) * 2;
          const double2 h0 = __ldcg(h), h1 = __ldcg(h + 1);
          const double sg = side_is_left(s) ? 1. : -1.;
          sh.cell.hs[lc][task][0] = sg * h0.x;
          sh.cell.hs[lc][task][1] = sg * h0.y;
          sh.cell.hs[lc][task][2] = sg * h1.x;
          sh.cell.hs[lc][task][3] = sg * h1.y;
        }
      }
      __syncthreads();
      if (on) {
        double acc[4] = {0., 0., 0., 0.};
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const double dx = sh.tdx[k * Q + ix], dy = sh.tdy[k * Q + iy];
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[c] += dx * sh.cell.fx[lc][iy * Q + k][c] + dy * sh.cell.fy[lc][k * Q + ix][c];
        }
        const double w0 = sh.fb[iy * Q + ix], w1 = sh.fb[(Q + iy) * Q + ix], w2 = sh.fb[(2 * Q + ix) * Q + iy],
                     w3 = sh.fb[(3 * Q + ix) * Q + iy], im = sh.im[node];
        double o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const double fc = w0 * sh.cell.hs[lc][iy][c] + w1 * sh.cell.hs[lc][Q + iy][c] +
                            w2 * sh.cell.hs[lc][2 * Q + ix][c] + w3 * sh.cell.hs[lc][3 * Q + ix][c];
          o[c] = im * (fc - acc[c]) + xx[c];
        }
        double2 *wv = reinterpret_cast<double2 *>(w + (size_t)e * M + 4 * node);
        wv[0] = make_double2(o[0], o[1]);
        wv[1] = make_double2(o[2], o[3]);
      }
      __syncthreads();
    }
    return true;
  }
  static __device__ __forceinline__ double value(const Args &, const double *, const double *w, int i) { return w[i]; }
  static __device__ __forceinline__ void precondition(const Args &a, Shared &sh, const double *v, double *z, int e0,
                                                      int e1, int, int) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int S = a.split, slots = kGW / S, slice = warp % S, slot = warp / S;
    const int kper = (M + S - 1) / S, k0 = min(M, slice * kper), k1 = min(M, k0 + kper);
    const int rounds = (e1 - e0 + slots - 1) / slots;
    for (int rd = 0; rd < rounds; ++rd) {
      const int e = e0 + rd * slots + slot;
      const bool on = e < e1;
      double acc[R2][2];
      if (on) {
        double *sv = sh.pc.v[warp];
        for (int i = k0 + lane; i < k1; i += 32) sv[i] = v[(size_t)e * M + i];
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R2; ++r) acc[r][0] = acc[r][1] = 0.;
        const double2 *A = reinterpret_cast<const double2 *>(a.inv + (size_t)e * M * M);
#pragma unroll R2 <= 2 ? 8 : 4
        for (int k = k0; k < k1; ++k) {
          const double xv = sv[k];
#pragma unroll
          for (int r = 0; r < R2; ++r)
            if (lane + 32 * r < M / 2) {
              const double2 m = __ldcs(A + (size_t)k * (M / 2) + lane + 32 * r);
              acc[r][0] = fma(m.x, xv, acc[r][0]);
              acc[r][1] = fma(m.y, xv, acc[r][1]);
            }
        }
      }
      if (S == 1) {
        if (on) {
#pragma unroll
          for (int r = 0; r < R2; ++r)
            if (lane + 32 * r < M / 2)
              __stcg(reinterpret_cast<double2 *>(z + (size_t)e * M) + lane + 32 * r, make_double2(acc[r][0], acc[r][1]));
        }
        __syncwarp();
        continue;
      }
      // the S warps of a cell meet at a barrier of their own
      if (on) {
#pragma unroll
        for (int r = 0; r < R2; ++r)
          if (lane + 32 * r < M / 2)
            *reinterpret_cast<double2 *>(&sh.pc.part[warp][2 * (lane + 32 * r)]) = make_double2(acc[r][0], acc[r][1]);
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(32 * S) : "memory");
      if (on)
        for (int i = slice * 32 + lane; i < M; i += 32 * S) {
          double t[2] = {sh.pc.part[slot * S][i], sh.pc.part[slot * S + 1][i]};
          for (int k = 2; k < S; k += 2) {
            t[0] += sh.pc.part[slot * S + k][i];
            t[1] += sh.pc.part[slot * S + k + 1][i];
          }
          __stcg(z + (size_t)e * M + i, t[0] + t[1]);
        }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(32 * S) : "memory");
    }
  }
};

// ------------------------------------------------------------------ passes
// Pass 1 (MODE 0): w from the operator, columns V^T M w.
// Pass 2 (MODE 1): w -= V h, columns V^T M w and w^T M w.
template <int NC, int MODE, class Op>
__device__ __forceinline__ void cgs_pass(SolveShared &sh, const typename Op::Args &oa, const typename Op::Real *z,
                                         typename Op::Real *w, const typename Op::Real *V, size_t ldv, int nc, int i0,
                                         int i1, int period, double *partials) {
  using T = typename Op::Real;
  double acc[NC], nrm = 0.;
#pragma unroll
  for (int k = 0; k < NC; ++k) acc[k] = 0.;
  for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
    T v[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = k < nc ? V[(size_t)k * ldv + i] : T(0);
    T wi;
    if (MODE == 0) {
      wi = Op::value(oa, z, w, i);
    } else {
      double comb = 0.;
      wi = w[i];
#pragma unroll
      for (int k = 0; k < NC; ++k)
        if (k < nc) comb += (double)v[k] * sh.h1[k];
      wi = (T)((double)wi - comb);
    }
    w[i] = wi;
    const double wm = sh.mt[(i % period) >> 2] * (double)wi;
    if (MODE == 1) nrm += wm * (double)wi;
#pragma unroll
    for (int k = 0; k < NC; ++k) acc[k] += (double)v[k] * wm;
  }
  publish_columns<NC>(sh, acc, nc, MODE == 1, nrm, partials);
}
// Pass 3: w -= V h2; returns the CTA's part of w^T M w.
template <int NC, class T>
__device__ __forceinline__ double cgs_final(SolveShared &sh, T *w, const T *V, T *vnext, size_t ldv, int nc, int i0, int i1,
                                            int period, double scale) {
  double nrm = 0.;
  for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
    T v[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = k < nc ? V[(size_t)k * ldv + i] : T(0);
    double comb = 0.;
    const T wi = w[i];
#pragma unroll
    for (int k = 0; k < NC; ++k)
      if (k < nc) comb += (double)v[k] * sh.h2[k];
    const T wn = (T)((double)wi - comb);
    if (vnext)
      vnext[i] = (T)((double)wn * scale);
    else
      w[i] = wn;
    nrm += sh.mt[(i % period) >> 2] * (double)wn * (double)wn;
  }
  return nrm;
}

// Givens rotations of Hessenberg column j and the convergence test
// (src/linear.cpp:123-136), by one thread.
__device__ __forceinline__ void givens_column(SolveShared &sh, int j, double next, double abs_tol) {
  double *hc = sh.h + (size_t)(kGC + 1) * j;
  for (int i = 0; i < j; ++i) {
    const double u = hc[i], v = hc[i + 1];
    hc[i] = sh.cs[i] * u + sh.sn[i] * v;
    hc[i + 1] = -sh.sn[i] * u + sh.cs[i] * v;
  }
  const double d = hypot(hc[j], hc[j + 1]);
  if (!(isfinite(d) && d > 0)) {
    sh.err = 1;
    sh.stop = 1;
    return;
  }
  const double c = hc[j] / d, s = hc[j + 1] / d;
  hc[j] = d;
  hc[j + 1] = 0.;
  const double gj = sh.g[j];
  sh.cs[j] = c;
  sh.sn[j] = s;
  sh.g[j + 1] = -s * gj;
  sh.g[j] = c * gj;
  sh.stop = (fabs(sh.g[j + 1]) <= abs_tol || next <= DBL_MIN) ? 1 : 0;
}

#define EG_BY_COLUMNS(nc, CALL)                    \
  do {                                             \
    if ((nc) <= 4) { constexpr int NC = 4; CALL; } \
    else if ((nc) <= 8) { constexpr int NC = 8; CALL; } \
    else if ((nc) <= 16) { constexpr int NC = 16; CALL; } \
    else { constexpr int NC = 24; CALL; }          \
  } while (0)

template <class T>
struct SolveArgs {
  int cells, per_cell, R, period, limit, zero_guess;
  double tol, rhs_norm;
  const T *rhs;
  T *x, *res, *w, *z, *comb, *V;
  size_t ldv;
  const double *mtab;
  double *partials;  // 3 x (kGC + 1) x gridDim
  GridBar bar;
  GmresCtl *ctl;     // out: count, err, next (the residual norm)
};

template <class Op>
__global__ void __launch_bounds__(kGT, 1) gmres_kernel(typename Op::Args oa, SolveArgs<typename Op::Real> s) {
  using T = typename Op::Real;
  __shared__ SolveShared sh;
  extern __shared__ __align__(16) unsigned char dyn[];
  typename Op::Shared &osh = *reinterpret_cast<typename Op::Shared *>(dyn);
  const int G = gridDim.x, b = blockIdx.x;
  const int e0 = (int)((long long)s.cells * b / G), e1 = (int)((long long)s.cells * (b + 1) / G);
  const int i0 = e0 * s.per_cell, i1 = e1 * s.per_cell;
  unsigned target = 0;
  double *part0 = s.partials, *part1 = part0 + (size_t)(kGC + 1) * G, *part2 = part1 + (size_t)(kGC + 1) * G;
  Op::setup(oa, osh);
  for (int i = threadIdx.x; i < s.period / 4; i += blockDim.x) sh.mt[i] = s.mtab[i];
  if (threadIdx.x == 0) sh.stop = sh.err = 0;
  __syncthreads();
  // res = rhs - A x for a given guess; norm over the grid
  const auto true_residual = [&](double &norm) -> bool {
    if (!Op::apply(oa, osh, s.x, s.w, e0, e1, s.bar, target)) return false;
    double nrm = 0.;
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
      const T r = s.rhs[i] - Op::value(oa, s.x, s.w, i);
      s.res[i] = r;
      nrm += sh.mt[(i % s.period) >> 2] * (double)r * (double)r;
    }
    publish_one(sh, nrm, part2);
    if (!grid_barrier(s.bar, target)) return false;
    collect_columns(1, part2, sh.h1);
    norm = sqrt(sh.h1[0]);
    __syncthreads();
    return true;
  };
  double residual_norm = s.rhs_norm;
  if (s.zero_guess) {
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
      s.x[i] = T(0);
      s.res[i] = s.rhs[i];
    }
  } else if (!true_residual(residual_norm)) {
    return;
  }
  int iterations = 0, err = 0;
  while (iterations < s.limit) {
    const double beta = residual_norm;
    if (beta <= s.tol * s.rhs_norm) break;
    const double inv_beta = 1 / beta, abs_tol = s.tol * s.rhs_norm;
    for (int i = threadIdx.x; i < (kGC + 1) * kGC; i += blockDim.x) sh.h[i] = 0.;
    for (int i = threadIdx.x; i <= kGC; i += blockDim.x) sh.g[i] = i == 0 ? beta : 0.;
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) s.V[i] = (T)((double)s.res[i] * inv_beta);
    __syncthreads();
    Op::precondition(oa, osh, s.V, s.z, e0, e1, i0, i1);
    if (!grid_barrier(s.bar, target)) return;
    int count = 0;
    for (int j = 0; j < s.R && iterations < s.limit; ++j) {
      const int nc = j + 1;
      if (!Op::apply(oa, osh, s.z, s.w, e0, e1, s.bar, target)) return;
      EG_BY_COLUMNS(nc, (cgs_pass<NC, 0, Op>(sh, oa, s.z, s.w, s.V, s.ldv, nc, i0, i1, s.period, part0)));
      if (!grid_barrier(s.bar, target)) return;
      collect_columns(nc, part0, sh.h1);
      EG_BY_COLUMNS(nc, (cgs_pass<NC, 1, Op>(sh, oa, s.z, s.w, s.V, s.ldv, nc, i0, i1, s.period, part1)));
      if (!grid_barrier(s.bar, target)) return;
      collect_columns(nc + 1, part1, sh.h2);
      double d4[4] = {0., 0., 0., 0.};
#pragma unroll
      for (int k = 0; k < kGC; ++k)
        if (k < nc) d4[k & 3] += sh.h2[k] * sh.h2[k];
      const double drop = (d4[0] + d4[1]) + (d4[2] + d4[3]);
      double next = sqrt(fmax(sh.h2[nc] - drop, 0.));
      T *vnext = s.V + (size_t)(j + 1) * s.ldv;
      const bool direct = drop <= .25 * sh.h2[nc];  // CTA- and grid-uniform
      if (!direct) {
        double nrm = 0.;
        EG_BY_COLUMNS(nc, (nrm = cgs_final<NC, T>(sh, s.w, s.V, nullptr, s.ldv, nc, i0, i1, s.period, 0.)));
        publish_one(sh, nrm, part2);
        if (!grid_barrier(s.bar, target)) return;
        collect_columns(1, part2, sh.red[0]);
        next = sqrt(sh.red[0][0]);
        __syncthreads();
      }
      if (threadIdx.x == kGT - 32) {
        double *hc = sh.h + (size_t)(kGC + 1) * j;
        for (int k = 0; k < nc; ++k) hc[k] = sh.h1[k] + sh.h2[k];
        hc[nc] = next;
        givens_column(sh, j, next, abs_tol);
      }
      if (next > 0) {
        const double scale = 1 / next;
        if (direct) {
          EG_BY_COLUMNS(nc, (cgs_final<NC, T>(sh, s.w, s.V, vnext, s.ldv, nc, i0, i1, s.period, scale)));
        } else {
          for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) vnext[i] = (T)((double)s.w[i] * scale);
        }
      }
      __syncthreads();
      if (sh.err) {
        err = 1;
        break;
      }
      ++iterations;
      count = nc;
      if (sh.stop || nc == s.R || iterations == s.limit) break;
      Op::precondition(oa, osh, vnext, s.z, e0, e1, i0, i1);
      if (!grid_barrier(s.bar, target)) return;
    }
    if (err) break;
    // Krylov coefficients (src/linear.cpp:138-142), column by column
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      double gv = lane < count ? sh.g[lane] : 0.;
      for (int i = count - 1; i >= 0; --i) {
        const double yi = __shfl_sync(0xffffffffu, gv, i) / sh.h[i + (kGC + 1) * i];
        if (lane == i) sh.y[i] = yi;
        if (lane < i) gv -= sh.h[lane + (kGC + 1) * i] * yi;
      }
    }
    __syncthreads();
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
      double sum = 0.;
#pragma unroll 4
      for (int c = 0; c < count; ++c) sum += (double)s.V[(size_t)c * s.ldv + i] * sh.y[c];
      s.comb[i] = (T)sum;
    }
    __syncthreads();
    // z is free here: the last apply of this cycle is behind a barrier
    Op::precondition(oa, osh, s.comb, s.z, e0, e1, i0, i1);
    __syncthreads();
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) s.x[i] += __ldcg(s.z + i);
    if (!grid_barrier(s.bar, target)) return;
    if (!true_residual(residual_norm)) return;
    if (!isfinite(residual_norm)) {
      err = 2;
      break;
    }
  }
  if (b == 0 && threadIdx.x == 0) {
    s.ctl->count = iterations;
    s.ctl->err = err;
    s.ctl->next = residual_norm;
  }
}

// CTAs of a solve over `cells` cells whose operator streams `bytes` per step on
// vectors of N entries: one per 256 KB or 444 entries, at least 16, at most
// one per SM, and no CTA with a nearly idle second round of cells. More CTAs
// than that shorten a small solve by a few per cent and keep other instances
// off the SMs: measured per step at 16x16 Q3 20.5, 17.5, 16.0,
// 16.5 us with 16, 32, 64, 148 CTAs; 32x32 Q2 26.9, 19.7, 18.3 us with 32, 64,
// 148; 64x64 Q1 34.9, 26.0 us with 64, 148; 20x20 Q8 37.2, 32.0, 30.6 us with
// 64, 100, 148; a batch of six instances of 400 to 1024 cells takes 104 ms with
// 148 CTAs each, 72 to 75 ms with 37 to 74.
int solve_grid(int cells, double bytes, int N) {
  const double want = std::max(16., std::max(bytes / 262144., N / 444.));
  const int cap = std::min(device_sms(), cells);
  const int grid = std::max(1, (int)std::min<double>(cap, std::ceil(want)));
  int per = (cells + grid - 1) / grid;  // no more CTAs than the fullest ones need
  if (per > kGW && per < 2 * kGW && (cells + kGW - 1) / kGW <= cap) per = kGW;
  return (cells + per - 1) / per;
}

template <class Op>
double launch_solve(Ctx &c, typename Op::Args &oa, SolveArgs<typename Op::Real> &s, int grid, int *count) {
  EG_CUDA(cudaMemsetAsync(s.bar.count, 0, sizeof(unsigned) + sizeof(int), c.stream));
  {
    ProfScope ps(c, EG_K_KRYLOV, 1);
    void *params[] = {&oa, &s};
    constexpr size_t dyn = sizeof(typename Op::Shared);
    if (dyn > 32 * 1024)
      EG_CUDA(cudaFuncSetAttribute(gmres_kernel<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    EG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(gmres_kernel<Op>), grid, kGT, params, dyn,
                                        c.stream));
  }
  EG_CUDA(cudaMemcpyAsync(c.hctl, c.ctl, sizeof(GmresCtl), cudaMemcpyDeviceToHost, c.stream));
  c.check_device_error();
  *count = c.hctl->count;
  if (c.hctl->err == 1) fail(EG_ERR_GMRES_BREAKDOWN, "GMRES Arnoldi breakdown");
  if (c.hctl->err == 2) fail(EG_ERR_GMRES_NONFINITE, "Nonfinite GMRES residual");
  return c.hctl->next;
}

template <class T>
SolveArgs<T> solve_args(Ctx &c, const KrylovBufs<T> &kb, const T *rhs, T *x, double tol, int limit, bool zero_guess,
                        double rhs_norm, int N) {
  c.need(c.solve_bar, 2);
  c.need(c.solve_partials, (size_t)3 * (kGC + 1) * device_sms());
  SolveArgs<T> s{};
  s.R = std::min(N, kb.R);
  s.limit = limit;
  s.zero_guess = zero_guess;
  s.tol = tol;
  s.rhs_norm = rhs_norm;
  s.rhs = rhs;
  s.x = x;
  s.res = kb.res;
  s.w = kb.w;
  s.z = kb.z;
  s.comb = kb.comb;
  s.V = kb.V;
  s.ldv = kb.ld;
  s.partials = c.solve_partials;
  s.bar = GridBar{c.solve_bar, reinterpret_cast<int *>(c.solve_bar + 1), c.derr, c.ilu_wait_limit_ns, c.ilu_starve};
  s.ctl = c.ctl;
  return s;
}

template <int Q, class T, bool PAN>
double solve_hdg(Ctx &c, const KrylovBufs<T> &kb, const T *act, const T *D, const T *pc, T *contrib, const T *rhs,
                 T *x, double tol, int limit, bool zero_guess, double rhs_norm, int *count) {
  using Op = HdgOp<Q, T, PAN>;
  const size_t stride = PAN ? (size_t)16 * c.t * c.t
                            : (sizeof(T) == 8 ? (size_t)c.m * (4 * c.t + 1) : (size_t)c.m * 4 * c.t);
  const int grid = solve_grid(c.n, (double)c.n * Op::ROWS * Op::K * sizeof(T), c.nl);
  const int per = (c.n + grid - 1) / grid;
  int split = 1;
  while (split < kGW && 2 * split * per <= kGW) split *= 2;
  typename Op::Args oa{c.geo, c.tab, c.Cb, act, stride, D, pc, contrib, split};
  SolveArgs<T> s = solve_args(c, kb, rhs, x, tol, limit, zero_guess, rhs_norm, c.nl);
  s.cells = c.n;
  s.per_cell = 2 * c.t;
  s.period = 2 * c.t;
  s.mtab = c.mtab_hdg;
  return launch_solve<Op>(c, oa, s, grid, count);
}

template <int Q>
double solve_dg(Ctx &c, const KrylovBufs<double> &kb, const double *rhs, double *x, double tol, int limit,
                bool zero_guess, double rhs_norm, int *count) {
  using Op = DgOp<Q>;
  c.need(c.dgc_h, (size_t)4 * c.nf * c.q);
  const int grid = solve_grid(c.n, 8. * c.n * ((double)c.m * c.m + 32 * c.p + 64 * c.q), c.nu);
  const int per = (c.n + grid - 1) / grid;
  // warps per cell of the block apply: the fewest whose last round of cells
  // wastes less than a twentieth of the warps
  int split = 1;
  while (split < kGW && 20 * (((per * split + kGW - 1) / kGW) * kGW - per * split) > per * split) split *= 2;
  typename Op::Args oa{c.geo, c.tab, c.dgc_vol, c.dgc_face, c.pc_dg, c.dgc_h, split};
  SolveArgs<double> s = solve_args(c, kb, rhs, x, tol, limit, zero_guess, rhs_norm, c.nu);
  s.cells = c.n;
  s.per_cell = c.m;
  s.period = c.m;
  s.mtab = c.mtab_dg;
  return launch_solve<Op>(c, oa, s, grid, count);
}

template <class T>
double solve_hdg_q(Ctx &c, const KrylovBufs<T> &kb, const T *act, const T *D, const T *pc, T *contrib, const T *rhs,
                   T *x, double tol, int limit, bool zero_guess, double rhs_norm, int *count) {
#define EG_SOLVE(QQ, PAN)                                                                                        \
  return solve_hdg<QQ, T, PAN>(c, kb, act, D, pc, contrib, rhs, x, tol, limit, zero_guess, rhs_norm, count)
  if (c.geo.npan == 16) {
    EG_DISPATCH_Q(c.q, EG_SOLVE(Q, true));
  } else {
    switch (c.q) {
      case 1: EG_SOLVE(1, false);
      case 2: EG_SOLVE(2, false);
      case 3: EG_SOLVE(3, false);
      case 4: EG_SOLVE(4, false);
      default: break;
    }
  }
#undef EG_SOLVE
  fail(EG_ERR_INVALID, "unsupported degree");
}

}  // namespace

bool fused_solve_supported(const Ctx &c, int R) { return R <= kGC && c.opts.precond == EG_PC_BLOCK_JACOBI; }

double fused_solve_hdg(Ctx &c, const KrylovBufs<double> &kb, const double *rhs, double *x, double tol, int limit,
                       bool zero_guess, double rhs_norm, int *count) {
  return solve_hdg_q<double>(c, kb, c.geo.npan == 16 ? c.panels : c.XY, c.D, c.pc_hdg, c.contrib, rhs, x, tol, limit,
                             zero_guess, rhs_norm, count);
}
double fused_solve_dg(Ctx &c, const KrylovBufs<double> &kb, const double *rhs, double *x, double tol, int limit,
                      bool zero_guess, double rhs_norm, int *count) {
  EG_DISPATCH_Q(c.q, return solve_dg<Q>(c, kb, rhs, x, tol, limit, zero_guess, rhs_norm, count));
  fail(EG_ERR_INVALID, "unsupported degree");
}
double fused_solve_hdg_f32(Ctx &c, const KrylovBufs<float> &kb, const float *rhs, float *x, double tol, int limit,
                           double rhs_norm, int *count) {
  return solve_hdg_q<float>(c, kb, c.Xf, c.Df, c.pcf, c.contribf, rhs, x, tol, limit, true, rhs_norm, count);
}

}  // namespace eg
