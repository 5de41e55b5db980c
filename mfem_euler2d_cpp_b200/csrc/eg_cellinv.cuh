// Inverse of a cell matrix held in registers, shared by the HDG condensation
// (eg_hdg.cu) and the DG block-Jacobi inverses (eg_dginv.cu). Not part of the
// public C-ABI.
//
// The M x M matrix is a grid of 8 x 8 tiles in the accumulator layout of the
// FP64 MMA; warp (wr, wc) of WR x WC owns the tiles (wr + a WR, wc + b WC).
// It is inverted in place by block Gauss-Jordan with the 8 x 8 diagonal
// blocks as pivots in their natural order:
//   B_j  = T^{-1} A_pj  (B_p = T^{-1}),   A_pj <- B_j,
//   A_ij <- A_ij - A_ip B_j  (A_ip taken as zero in the pivot column), i != p.
// Rows are exchanged only inside a pivot block (partial pivoting in its
// inversion). That is enough for these matrices: they are I plus a dissipative
// upwind operator, so the entries of B stay of order one (below 7 for k = 1..8
// at CFL 0.5 to 1000) and the inverse is as accurate as one with full partial
// pivoting. It is checked, not assumed: a cell with an entry of B above kMaxB,
// or a pivot that is zero or not finite, is reported, and its caller solves it
// again by LU with partial pivoting over the whole matrix.
//
// What bounds it: 2 M^3 flops on the FP64 tensor pipe. A search over all rows
// (the LU's pivots) is a serial chain of about 2.6k cycles per 4 columns that
// no other warp can work under; here a panel is 8 columns, its pivot block is
// known in advance, and one warp inverts it (about 2k cycles) as soon as the
// previous panel has updated its tile, while the others finish that panel.
#pragma once
#include "eg_cellmat.cuh"

namespace eg {

// D = C + A B on the FP64 tensor pipe: m8n8k4, A row-major 8x4 (one element
// per lane: row lane/4, column lane%4), B column-major 4x8 (row lane%4,
// column lane/4), C/D 8x8 (two elements per lane: row lane/4, columns
// 2*(lane%4) and 2*(lane%4)+1).
__device__ __forceinline__ void dmma_m8n8k4(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Reciprocal of a pivot: hardware estimate refined by two Newton-Raphson
// steps r <- r + r (1 - x r) (quadratic convergence from the ~2^-20 estimate;
// result within one unit in the last place of 1/x). The estimate flushes
// subnormal inputs and results to zero, so magnitudes outside
// [2^-1020, 2^1020] (and zero, infinities, NaN) take IEEE division instead.
__device__ __forceinline__ double pivot_reciprocal(double x) {
  const double ax = fabs(x);
  if (!(ax >= 0x1p-1020 && ax <= 0x1p+1020)) return 1.0 / x;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}

// A shared-memory pair that the compiler may not keep in registers for the next
// column of tiles: those registers hold the matrix. The clobber keeps the load
// behind the stores and barriers before it.
__device__ __forceinline__ double2 lds_pair(const double *p) {
  double2 v;
  asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}

__device__ __forceinline__ double lds_one(const double *p) {
  double v;
  asm volatile("ld.volatile.shared.f64 %0, [%1];"
               : "=d"(v)
               : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}

constexpr double kMaxB = 64.;

// Strides in doubles of a node's two Jacobians and of a face point's 4x4 matrix
// in shared memory: 16-byte accesses by lanes over nodes and columns then use
// all banks (at 32 and 16 every node started in the same one).
constexpr int kJacStride = 34, kFaceStride = 18;

template <int Q, int WR_, int WC_, int DED_ = 0>
struct InvCfg {
  static constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, MT = (M + 7) / 8;
  // DED: one more warp, without tiles, inverts the pivot blocks (where the
  // registers allow it); otherwise the tile warps take turns
  static constexpr int WR = WR_, WC = WC_, DED = DED_, NW = WR * WC, THREADS = 32 * (NW + DED);
  static constexpr int TR = (MT + WR - 1) / WR, TC = (MT + WC - 1) / WC;  // tiles per warp
  // stride of the matrix in shared memory: LDA % 8 in {2, 6} makes a warp's
  // 8x8 tile accesses, and 16-byte accesses with lanes over columns, conflict-free
  static constexpr int LDA = (M % 8 == 0 || M % 8 == 4) ? M + 2 : M + 1;
  static_assert(LDA % 8 == 2 || LDA % 8 == 6, "tile accesses");
  static constexpr int PR = 8 * TR * WR, PC = 8 * TC * WC;  // rows and columns padded to whole warp grids
  // stride of the pivot rows: 64 bytes past a multiple of 128, so that the four
  // rows an operand load touches use all banks
  static constexpr int TS = PC % 16 == 0 ? PC + 8 : PC;
  static constexpr int PANELS = 2 * (PR * 8 + 8 * TS);  // doubles of the double-buffered panel and pivot rows
  static constexpr int REGION = LDA * M > PANELS ? LDA * M : PANELS;
};

// Inverse of an 8x8 block T by one warp: Gauss-Jordan in place with partial
// pivoting, lane 4 r + q holding T[r][2q], T[r][2q + 1]; rows never move. No
// reciprocal sits on the chain of eight dependent steps: a step scales every
// other row by the pivot's significand (its power of two is taken out exactly)
// instead of dividing the pivot row, and each row is divided once at the end
// by the product it has collected. The steps are branch-free, so that the
// compiler can place them between the MMAs of an update (180 cycles of latency
// each, 1800 in all when nothing else runs).
struct Invert8 {
  double v0, v1, d = 1.;
  double unit = 1.;  // what the rows not yet used have been scaled by
  int row = 0, c0 = 0, c1 = 0;
  bool used = false, ok = true;
  template <int K>
  __device__ __forceinline__ void step() {
    const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const double ck = __shfl_sync(0xffffffffu, (K & 1) ? v1 : v0, (lane & 28) | (K >> 1));
    const unsigned hi = (unsigned)__double2hiint(ck) & 0x7fffffffu;
    // magnitudes within 2^-17 of each other tie, to the first row
    const unsigned key = (!used && hi < 0x7ff00000u) ? ((hi & ~7u) | (unsigned)(7 - gq)) : 0u;
    const unsigned mb = __reduce_max_sync(0xffffffffu, key);
    ok = ok && mb >= 0x00100008u && mb < 0x7fe00000u;
    const int pr = 7 - (int)(mb & 7u);
    const double pv = __shfl_sync(0xffffffffu, ck, 4 * pr);
    const double r0 = __shfl_sync(0xffffffffu, v0, 4 * pr + tq), r1 = __shfl_sync(0xffffffffu, v1, 4 * pr + tq);
    const double sc = __hiloint2double((int)(0x7fe00000u - (mb & 0x7ff00000u)), 0);  // 2^-exponent(pivot)
    const double pn = pv * sc, cn = ck * sc, cu = -cn * unit;
    const bool piv = gq == pr, mine0 = (K >> 1) == tq && !(K & 1), mine1 = (K >> 1) == tq && (K & 1);
    c0 = mine0 ? pr : c0;
    c1 = mine1 ? pr : c1;
    const double n0 = fma(pn, v0, -(cn * r0)), n1 = fma(pn, v1, -(cn * r1));
    v0 = piv ? (mine0 ? unit : v0) : (mine0 ? cu : n0);
    v1 = piv ? (mine1 ? unit : v1) : (mine1 ? cu : n1);
    d = piv ? pv : (used ? d * pn : d);
    row = piv ? K : row;
    used = used || piv;
    unit *= pn;
  }
  // row-major inverse into the warp's Ti
  __device__ __forceinline__ void run(double *Ti) {
    step<0>();
    step<1>();
    step<2>();
    step<3>();
    step<4>();
    step<5>();
    step<6>();
    step<7>();
    const double id = pivot_reciprocal(d);
    Ti[row * 8 + c0] = v0 * id;
    Ti[row * 8 + c1] = v1 * id;
    __syncwarp();
  }
};

// acc: the CTA's tiles of the matrix, identity on the padding; on return, of
// its inverse. panels: C::PANELS doubles of shared memory, tiles: 256 more.
// Sets *bad (shared) when the elimination cannot vouch for the result. Ends
// with a CTA barrier.
//
// One barrier per panel. At its start one warp (C::DED, or another one each
// panel) forms the next pivot block from the published tile (before this panel's update)
// and inverts it; a tile warp then joins the update. The update has no branches: the
// pivot column and row are set to zero first, the panel's pivot rows hold the
// identity, and the right operand of the pivot column is the identity. Tiles
// are updated in pairs, so that the two MMAs of a tile are not back to back
// (26 cycles from one to the other, 16 between two of different tiles).
template <class C>
__device__ __forceinline__ void invert_tiles(double (&acc)[C::TR][C::TC][2], double *panels, double *tiles, int *bad) {
  constexpr int MT = C::MT, PR = C::PR, TS = C::TS, WR = C::WR, WC = C::WC, TR = C::TR, TC = C::TC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % WR, wc = warp / WR;
  const int gq = lane >> 2, tq = lane & 3;
  double *Tis = tiles + 128;  // the inverse pivot blocks, double-buffered like the rest
  const bool tiles_here = C::DED == 0 || warp < C::NW;
  bool fine = true;
  // panel columns (negated), [row][8]; pivot rows, [8][TS]; the next diagonal tile, [8][8]
  const auto pan = [&](int buf) { return panels + buf * (8 * PR + 8 * TS); };
  const auto top = [&](int buf) { return panels + buf * (8 * PR + 8 * TS) + 8 * PR; };
  const auto publish = [&](int nxt, int buf) {
    if (nxt % WC == wc) {
#pragma unroll
      for (int b = 0; b < TC; ++b)
        if (wc + b * WC == nxt) {
          double *P = pan(buf) + gq * 8 + 2 * tq;
#pragma unroll
          for (int a = 0; a < TR; ++a)
            *reinterpret_cast<double2 *>(P + (wr + a * WR) * 64) = make_double2(-acc[a][b][0], -acc[a][b][1]);
          if (nxt % WR == wr)
            *reinterpret_cast<double2 *>(P + nxt * 64) =
                make_double2(gq == 2 * tq ? 1. : 0., gq == 2 * tq + 1 ? 1. : 0.);
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
    if (i % WR != wr || i % WC != wc) return;
#pragma unroll
    for (int a = 0; a < TR; ++a)
#pragma unroll
      for (int b = 0; b < TC; ++b)
        // the same tile by both indices (a known pair when WR == WC)
        if ((WR != WC || a == b) && wr + a * WR == i && wc + b * WC == i)
          *reinterpret_cast<double2 *>(tiles + buf * 64 + gq * 8 + 2 * tq) = make_double2(acc[a][b][0], acc[a][b][1]);
  };
  if (tiles_here) {
    publish(0, 0);
    publish_diagonal(0, 1);
    publish_diagonal(1, 0);
  }
  __syncthreads();
  if (warp == 0) {
    Invert8 inv;
    inv.v0 = tiles[64 + gq * 8 + 2 * tq];
    inv.v1 = tiles[64 + gq * 8 + 2 * tq + 1];
    inv.run(Tis);
    fine = inv.ok;
  }
  __syncthreads();
#pragma unroll 1
  for (int p = 0; p < MT; ++p) {
    const int buf = p & 1;
    const double ti0 = Tis[buf * 64 + gq * 8 + tq], ti1 = Tis[buf * 64 + gq * 8 + tq + 4];
    const double *P = pan(buf) + gq * 8 + 2 * tq, *W = top(buf) + tq * TS + gq;
    // rows 2 tq and 2 tq + 1 of B = T^{-1} A_p,ct, column gq: the transposed
    // product, whose accumulator layout is the operand layout the update needs
    const auto pivot_rows = [&](int ct, double &b0, double &b1) {
      const bool pc = ct == p;
      const double t0 = pc ? (gq == tq ? 1. : 0.) : W[ct * 8];
      const double t1 = pc ? (gq == tq + 4 ? 1. : 0.) : W[4 * TS + ct * 8];
      b0 = b1 = 0.;
      dmma_m8n8k4(b0, b1, t0, ti0);
      dmma_m8n8k4(b0, b1, t1, ti1);
      fine = fine && (pc || (fabs(b0) <= kMaxB && fabs(b1) <= kMaxB));
    };
    if (warp == (C::DED ? C::NW : (p + 1) % C::NW) && p + 1 < MT) {
      double b0, b1;
      pivot_rows(p + 1, b0, b1);
      const double2 w = *reinterpret_cast<const double2 *>(P + (p + 1) * 64);
      const double2 t = *reinterpret_cast<const double2 *>(tiles + buf * 64 + gq * 8 + 2 * tq);
      Invert8 inv;
      inv.v0 = t.x;
      inv.v1 = t.y;
      dmma_m8n8k4(inv.v0, inv.v1, w.x, b0);
      dmma_m8n8k4(inv.v0, inv.v1, w.y, b1);
      inv.run(Tis + (buf ^ 1) * 64);
      fine = fine && inv.ok;
    }
    if (tiles_here) {
      if (p % WC == wc) {
#pragma unroll
        for (int b = 0; b < TC; ++b)
          if (wc + b * WC == p) {
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
        // the next column's rows of B are formed between this column's updates
        const int cn = wc + (b + 1 < TC ? b + 1 : b) * WC;
        const bool pc = cn == p;
        double t0 = lds_one(W + cn * 8), t1 = lds_one(W + 4 * TS + cn * 8), n0 = 0., n1 = 0.;
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
          if (b + 1 < TC && a == 0) dmma_m8n8k4(n0, n1, pc ? (gq == tq ? 1. : 0.) : t0, ti0);
          if (b + 1 < TC && (a == 2 || TR <= 2)) dmma_m8n8k4(n0, n1, pc ? (gq == tq + 4 ? 1. : 0.) : t1, ti1);
        }
        if (b + 1 < TC) {
          fine = fine && (pc || (fabs(n0) <= kMaxB && fabs(n1) <= kMaxB));
          b0 = n0;
          b1 = n1;
        }
      }
      publish(p + 1, buf ^ 1);
      publish_diagonal(p + 2, buf ^ 1);
    }
    __syncthreads();
  }
  if (!fine) *bad = 1;
  __syncthreads();
}

// Tiles of the matrix A (shared memory, column-major, stride C::LDA), identity
// on the padding, and back.
template <class C>
__device__ __forceinline__ void load_tiles(double (&acc)[C::TR][C::TC][2], const double *A) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % C::WR, wc = warp / C::WR;
  const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
  for (int a = 0; a < C::TR; ++a)
#pragma unroll
    for (int b = 0; b < C::TC; ++b) {
      const int row = (wr + a * C::WR) * 8 + gq, col = (wc + b * C::WC) * 8 + 2 * tq;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        acc[a][b][h] = (row < C::M && col + h < C::M) ? A[row + (size_t)(col + h) * C::LDA]
                                                      : (row == col + h ? 1. : 0.);
    }
}
template <class C>
__device__ __forceinline__ void store_tiles(const double (&acc)[C::TR][C::TC][2], double *A) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wr = warp % C::WR, wc = warp / C::WR;
  const int gq = lane >> 2, tq = lane & 3;
  if (C::DED && warp >= C::NW) return;
#pragma unroll
  for (int a = 0; a < C::TR; ++a)
#pragma unroll
    for (int b = 0; b < C::TC; ++b) {
      const int row = (wr + a * C::WR) * 8 + gq, col = (wc + b * C::WC) * 8 + 2 * tq;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (row < C::M && col + h < C::M) A[row + (size_t)(col + h) * C::LDA] = acc[a][b][h];
    }
}

// Column-major 4x4 flux Jacobian in the direction `axis` (EulerGas::jacobian,
// src/physics.cpp:18-39), by arithmetic on the unit normal: threads of a warp
// with different axes do not diverge.
__device__ __forceinline__ void jacobian_axis(const double *u, int axis, double gm1, double j[16]) {
  const double nx = axis == 0 ? 1. : 0., ny = 1. - nx;
  const double inv = 1. / u[0], vx = u[1] * inv, vy = u[2] * inv, vn = axis == 0 ? vx : vy;
  const double hd = (u[3] + gm1 * (u[3] - .5 * (u[1] * u[1] + u[2] * u[2]) * inv)) * inv;
  const double p0 = .5 * gm1 * (vx * vx + vy * vy), p1 = -gm1 * vx, p2 = -gm1 * vy;
  j[0] = 0.;
  j[1] = nx * p0 - vx * vn;
  j[2] = ny * p0 - vy * vn;
  j[3] = vn * (p0 - hd);
  j[4] = nx;
  j[5] = nx * (p1 + vx) + vn;
  j[6] = ny * p1 + nx * vy;
  j[7] = vn * p1 + nx * hd;
  j[8] = ny;
  j[9] = nx * p2 + ny * vx;
  j[10] = ny * (p2 + vy) + vn;
  j[11] = vn * p2 + ny * hd;
  j[12] = 0.;
  j[13] = nx * gm1;
  j[14] = ny * gm1;
  j[15] = vn * gm1 + vn;
}

// Flux Jacobians of the cell's nodes, J[node * kJacStride + 16 axis + k]
// (column-major 4x4), scaled by -dt w of the node.
template <int Q>
__device__ __forceinline__ void node_jacobians(double *J, const STab<Q> &st, const double *us, const Geo &g) {
  for (int t = threadIdx.x; t < 2 * Q * Q; t += blockDim.x) {
    const int node = t >> 1, axis = t & 1;
    double j[16];
    jacobian_axis(us + 4 * node, axis, g.gm1, j);
    const double s = -g.dt * st.w(node);
#pragma unroll
    for (int k = 0; k < 16; ++k) J[node * kJacStride + 16 * axis + k] = s * j[k];
  }
}

// The cell matrix of build_cell_matrix (eg_cellmat.cuh), one column of a 4x4
// node block per thread: node jn meets the nodes on its x-line and y-line only,
// 2 q - 1 of q^2; the other blocks are zero. Lanes run over the columns, which
// keeps the stores free of bank conflicts (a whole block per thread: 16-way).
// J from node_jacobians. Starts with a CTA barrier between the zeros and the
// blocks and needs one before use.
template <class C, int Q>
__device__ __forceinline__ void assemble_cell(double *A, const STab<Q> &st, const double *J, const double *FM,
                                              const Geo &g) {
  constexpr int M = C::M, LDA = C::LDA, L = 2 * Q - 1;
  double2 *A2 = reinterpret_cast<double2 *>(A);
  for (int i = threadIdx.x; i < LDA * M / 2; i += blockDim.x) A2[i] = make_double2(0., 0.);
  __syncthreads();
  const double sx = g.dt * g.hy / g.area, sy = g.dt * g.hx / g.area;
  for (int t = threadIdx.x; t < M * L; t += blockDim.x) {
    // pos < Q: x-line node pos; else the y-line node pos - Q, past the own one
    const int col = t % M, pos = t / M, jn = col >> 2, d = col & 3, jx = jn % Q, jy = jn / Q;
    const bool xl = pos < Q, own = xl && pos == jx;
    const int iy0 = pos - Q, ix = xl ? pos : jx, iy = xl ? jy : iy0 + (iy0 >= jy ? 1 : 0);
    const int i = iy * Q + ix;
    const double im = st.inv_mass(i);
    double v[4] = {own && d == 0 ? 1. : 0., own && d == 1 ? 1. : 0., own && d == 2 ? 1. : 0., own && d == 3 ? 1. : 0.};
    const auto line = [&](double gd, double w0, double w1, const double *j, const double *m0, const double *m1) {
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const double2 a = *reinterpret_cast<const double2 *>(j + k), b = *reinterpret_cast<const double2 *>(m0 + k),
                      c = *reinterpret_cast<const double2 *>(m1 + k);
        v[k] += gd * a.x + (w0 * b.x + w1 * c.x);
        v[k + 1] += gd * a.y + (w0 * b.y + w1 * c.y);
      }
    };
    const double *j = J + kJacStride * jn + 4 * d, *m = FM + 4 * d;
    if (xl) {
      const double e = im * sx * st.ew(jy), f0 = st.fb(0, jy, ix) * st.fb(0, jy, jx), f1 = st.fb(1, jy, ix) * st.fb(1, jy, jx);
      line(im * st.tdx(jx, ix), e * f0, e * f1, j, m + kFaceStride * jy, m + kFaceStride * (Q + jy));
    }
    if (!xl || own) {
      const double e = im * sy * st.ew(jx), f2 = st.fb(2, jx, iy) * st.fb(2, jx, jy), f3 = st.fb(3, jx, iy) * st.fb(3, jx, jy);
      line(im * st.tdy(jy, iy), e * f2, e * f3, j + 16, m + kFaceStride * (2 * Q + jx), m + kFaceStride * (3 * Q + jx));
    }
    double2 *a = reinterpret_cast<double2 *>(A + (size_t)col * LDA + 4 * i);
    a[0] = make_double2(v[0], v[1]);
    a[1] = make_double2(v[2], v[3]);
  }
}

}  // namespace eg
