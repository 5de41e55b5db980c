// Block ILU(0) preconditioner on the DG cell graph or the condensed HDG face
// graph, natural ordering (FixedBlockILU, src/block_ilu.cpp:10-109;
// Problem::SolverGraph, src/block_ilu.cpp:110-124).
//
// Structure (host, once per context and form): BSR rows in natural order with
// sorted block columns, the diagonal entry of each row, and for every
// strictly lower entry (i,k) the (target i,j ; upper k,j) products that ILU(0)
// retains (block_ilu.cpp:46-57).
//
// Numeric fill (every refresh): DG blocks are the cell Jacobian blocks and the
// face couplings of PartialDGOperator::FillBlocks (src/partial.cpp:140-170);
// HDG blocks are D - sum over cells of the panels C_s X_{s,o}
// (ElementOperator::FillBlocks, src/operators.cpp:48-74), summed in cell order.
//
// Factor and apply are dependency-driven sweeps, one cooperative launch each.
// Rows are grouped in chunks of one grid row (2nx faces or nx cells); chunk c
// belongs to CTA c mod G, and every CTA walks its rows in increasing
// (forward, factor) or decreasing (backward) order. A CTA publishes how many
// of its rows are final in one 64-bit counter tagged with the launch's epoch;
// a row waits only for rows earlier in the sweep order, which co-resident
// CTAs own, so no wait can depend on itself. Every wait is bounded: when no row
// of the launch has been finished for IluPlan::wait_limit_ns, far above the
// time of a row, the kernel records DERR_WAIT_LIMIT, sets the abort word, and
// all CTAs leave at their next wait (after their own bulk copies have landed).
//
// The factor stores the explicit inverse of each factored diagonal block
// (pivoted LU applied to the identity), so RightSolve becomes a product with
// it and the backward solve a block GEMV; the arithmetic is the reference's up
// to rounding.
#include <algorithm>
#include <vector>

#include "eg_bulk.cuh"
#include "eg_cellinv.cuh"
#include "eg_internal.h"

namespace eg {
namespace {

constexpr unsigned kCopySpinLimit = 1u << 16;   // try_wait itself suspends between polls
constexpr unsigned kDrainSpinLimit = 1u << 24;  // abort path: let an issued copy land
constexpr int kStageBlocks = 4;             // blocks staged per warp and row
constexpr int kStageMaxB = 36;              // larger blocks are read from global memory
constexpr size_t kSweepSmemBudget = 210 * 1024;
constexpr size_t kFactorSmemBudget = 220 * 1024;
constexpr size_t kRingBytes = 48 * 1024;    // shared-memory ring of finished rows per CTA

// ------------------------------------------------------------ sync helpers
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_volatile(const int *p) { return *(const volatile int *)p; }

__device__ __forceinline__ void give_up(int *abort, int *err) {
  atomicExch(abort, 1);
  raise_err(err, DERR_WAIT_LIMIT);
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits are bounded in time. A poll reads the awaited word only: the abort word
// and the global timer, each a round trip to L2 (about 700 cycles), are looked
// at every 32 or 256 polls.
constexpr unsigned kCheckGlobal = 31, kCheckLocal = 255;
// The bound is on time without a finished row anywhere in the launch, not on the
// wait: the last CTA waits for the whole wavefront (more than a second on 16 x
// 16 cells at k = 8). Every CTA's count of rows stands in `progress`; the counts
// are added up only when the limit has passed, so a wait that nothing will end
// gives up after two limits at most.
struct WaitBound {
  const unsigned long long *progress;
  int *abort, *err;
  unsigned long long limit_ns;
};
struct WaitClock {
  unsigned long long t0 = 0, rows = 0;  // 0: not read, not added up yet
};
__device__ __forceinline__ bool out_of_time(WaitClock &w, const WaitBound &b) {
  if (ld_volatile(b.abort)) return true;
  const unsigned long long now = global_ns();
  if (w.t0 == 0) w.t0 = now;
  if (now - w.t0 <= b.limit_ns) return false;
  // counts with their launch's epoch on top: a count only grows
  unsigned long long rows = 1;
#pragma unroll 1
  for (int g = 0; g < (int)gridDim.x; ++g) rows += *(const volatile unsigned long long *)(b.progress + g);
  if (rows == w.rows) {
    give_up(b.abort, b.err);
    return true;
  }
  w.rows = rows;
  w.t0 = now;
  return false;
}
// Kept out of the sweeps: inlined into their waits it took 4% of an apply at
// 48x48 Q4 (425 against 409 us).
__device__ __noinline__ bool out_of_time_call(WaitClock &w, const WaitBound &b) { return out_of_time(w, b); }
// Bounded wait until *p >= target (another CTA's progress).
__device__ bool wait_progress(const unsigned long long *p, unsigned long long target, const WaitBound &b) {
  WaitClock w;
  for (unsigned it = 1;; ++it) {
    if (ld_acquire(p) >= target) return true;
    if ((it & kCheckGlobal) == 0 && out_of_time(w, b)) return false;
  }
}
// Bounded wait until the CTA's own published row count reaches target.
__device__ bool wait_local(const volatile unsigned *count, unsigned target, const WaitBound &b) {
  WaitClock w;
  for (unsigned it = 1;; ++it) {
    if (*count >= target) return true;
    if ((it & kCheckLocal) == 0 && out_of_time_call(w, b)) return false;
  }
}
// The progress value a wait needs: `starve` (a test setting) asks for one no
// CTA ever publishes, so every wait on another CTA runs out.
__device__ __forceinline__ unsigned long long need(unsigned long long tag, int slot, int starve) {
  return starve ? ~0ull : (tag | (unsigned long long)(slot + 1));
}

// ------------------------------------------------------------- scheduling
// Rows of one sweep, host-built for a fixed grid G: chunk c (one grid row of
// faces or cells) belongs to CTA c mod G, whose slots walk its rows in
// increasing (forward, factor) or decreasing (backward) order. For every
// slot the table holds (row, first entry, entry count) and, for each entry
// the sweep reads, its producer (owner CTA << 22 | owner slot) and row.
constexpr int kMaxDeps = 8;
constexpr int kOwnerShift = 22;
constexpr int kSlotMask = (1 << kOwnerShift) - 1;

__device__ __forceinline__ void publish_max(unsigned long long *p, unsigned long long v) {
  asm volatile("red.release.gpu.global.max.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// ------------------------------------------------------------ sweep kernel
struct SweepArgs {
  int B, ring;
  const int *slot_ptr;
  const int4 *meta;
  const int2 *deps;
  const double *data, *dinv;
  const double *in;  // forward: b; backward: the forward result w
  double *out;       // forward: w; backward: x
  unsigned long long *progress;
  int *abort, *err;
  unsigned long long tag;
  unsigned long long limit_ns;  // bound of the waits (WaitBound)
  int starve;        // test setting: waits on other CTAs can never be met
  ulonglong2 *slots;      // small blocks: the rows' values for other CTAs
  unsigned epoch;
};

// FixedBlockILU::Mult (src/block_ilu.cpp:88-109). Forward: w_i = b_i -
// sum_{j<i} L_ij w_j. Backward: x_i = U_ii^{-1} (w_i - sum_{j>i} U_ij x_j).
// One warp per row (lanes own block rows r = lane + 32 s); the W warps of a
// CTA keep W rows and their block copies in flight. A finished row goes to a
// shared-memory ring (read by later rows of the same CTA) and to global
// memory; the CTA's own count is published first, then, off the local chain,
// the release of the global counter that other CTAs poll. For blocks above
// kStageMaxB, read from global memory; smaller ones take the kernel below.
template <int S, bool BACK>
__global__ void __launch_bounds__(256, 1) ilu_sweep_kernel(SweepArgs a) {
  extern __shared__ __align__(128) double smem[];
  __shared__ unsigned done_local;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int g = blockIdx.x, B = a.B;
  const size_t BB = (size_t)B * B;
  const int p0 = a.slot_ptr[g], nslots = a.slot_ptr[g + 1] - p0;
  const WaitBound wb{a.progress, a.abort, a.err, a.limit_ns};
  double *vb = smem + (size_t)warp * 32 * S;
  double *ring = smem + (size_t)W * 32 * S;
  if (threadIdx.x == 0) done_local = 0;
  __syncthreads();
  volatile unsigned *dl = &done_local;
  int4 nm = make_int4(0, 0, 0, 0);
  int2 nd[kMaxDeps];
  auto fetch = [&](int slot) {
    if (slot < nslots) {
      nm = a.meta[p0 + slot];
#pragma unroll
      for (int k = 0; k < kMaxDeps; ++k) nd[k] = a.deps[(size_t)(p0 + slot) * kMaxDeps + k];
    }
  };
  fetch(warp);
  for (int slot = warp; slot < nslots; slot += W) {
    const int i = nm.x, e0 = nm.y, ne = nm.z;
    int2 dep[kMaxDeps];
#pragma unroll
    for (int k = 0; k < kMaxDeps; ++k) dep[k] = nd[k];
    fetch(slot + W);  // the next row's schedule is in flight during this row
    double acc[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = lane + 32 * s;
      acc[s] = r < B ? __ldcg(a.in + (size_t)i * B + r) : 0.;
    }
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kMaxDeps; ++k) {
      if (k < ne && ok) {
        const int owner = dep[k].x >> kOwnerShift, js = dep[k].x & kSlotMask, j = dep[k].y;
        const bool local = owner == g;
        ok = local ? wait_local(dl, (unsigned)js + 1, wb)
                   : wait_progress(a.progress + owner, need(a.tag, js, a.starve), wb);
        // lanes that give up and lanes that do not may not part before a warp barrier
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
          __threadfence_block();
          const bool in_ring = local && slot - js <= a.ring - W;
          const double *src = ring + (size_t)(js & (a.ring - 1)) * B;
          for (int r = lane; r < B; r += 32) vb[r] = in_ring ? src[r] : __ldcg(a.out + (size_t)j * B + r);
          __syncwarp();
          const double *A = a.data + (size_t)(e0 + k) * BB;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const int r = lane + 32 * s;
            if (r < B) {
              // four partial sums: B is a multiple of 4, and one chain of B
              // dependent products would be most of a row's time
              double t[4] = {acc[s], 0., 0., 0.};
              for (int cc = 0; cc < B; cc += 4)
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) t[k4] -= A[(size_t)(cc + k4) * B + r] * vb[cc + k4];
              acc[s] = (t[0] + t[1]) + (t[2] + t[3]);
            }
          }
          __syncwarp();
        }
      }
    }
    if (!ok) return;
    if (BACK) {
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int r = lane + 32 * s;
        if (r < B) vb[r] = acc[s];
      }
      __syncwarp();
      const double *Di = a.dinv + (size_t)i * BB;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int r = lane + 32 * s;
        if (r < B) {
          double t[4] = {0., 0., 0., 0.};
          for (int cc = 0; cc < B; cc += 4)
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) t[k4] += Di[(size_t)(cc + k4) * B + r] * vb[cc + k4];
          acc[s] = (t[0] + t[1]) + (t[2] + t[3]);
        }
      }
      __syncwarp();
    }
    double *rs = ring + (size_t)(slot & (a.ring - 1)) * B;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = lane + 32 * s;
      if (r < B) {
        a.out[(size_t)i * B + r] = acc[s];
        rs[r] = acc[s];
      }
    }
    __threadfence_block();
    __syncwarp();
    int pub = 1;
    if (lane == 0) {
      pub = wait_local(dl, (unsigned)slot, wb);  // rows are published in order
      if (pub) {
        *dl = (unsigned)slot + 1;
        publish_max(a.progress + g, a.tag | (unsigned long long)(slot + 1));
      }
    }
    if (!__shfl_sync(0xffffffffu, pub, 0)) return;
  }
}

// A row's values for other CTAs travel as self-validating words: each 64-bit
// word of a slot carries 32 bits of a value and the sweep's epoch, so a reader
// polls the values themselves (one trip through L2) instead of a counter that
// is released behind a fence and then the values (three). The two words are the
// elements of a 64-bit vector access: the memory model makes an element one
// access and promises nothing for the vector, so each word carries the epoch.
__device__ __forceinline__ void put_slot(ulonglong2 *p, double v, unsigned ep) {
  const unsigned long long e = (unsigned long long)ep << 32, b = (unsigned long long)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
               : "memory");
}
__device__ __forceinline__ bool get_slot(const ulonglong2 *p, unsigned ep, double &v) {
  unsigned long long lo, hi;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
  v = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
  return (unsigned)(lo >> 32) == ep && (unsigned)(hi >> 32) == ep;
}

// The sweep for blocks of at most kStageMaxB (every HDG degree, DG up to k =
// 2), the block size known at compile time. What bounds it is the chain of
// dependent rows: a grid row of faces starts three to five rows behind its
// neighbour, so a sweep is ny times (a few rows + one hand-over between CTAs).
// A row's products are four partial sums each, unrolled; its neighbours' rows
// in other CTAs are polled together and folded in before its own CTA's.
// 48x48 Q4, forward and backward sweep: 1190 us with the counters and run-time
// block sizes of the kernel above, 404 here.
template <int B, bool BACK>
__global__ void __launch_bounds__(256, 1) ilu_sweep_small_kernel(SweepArgs a) {
  constexpr int S = (B + 31) / 32, BB = B * B;
  extern __shared__ __align__(128) double smem[];
  __shared__ unsigned done_local;
  __shared__ __align__(8) unsigned long long bars[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int g = blockIdx.x;
  const int p0 = a.slot_ptr[g], nslots = a.slot_ptr[g + 1] - p0;
  const WaitBound wb{a.progress, a.abort, a.err, a.limit_ns};
  double *stage = smem + (size_t)warp * kStageBlocks * BB;
  double *vb = smem + (size_t)W * kStageBlocks * BB + (size_t)warp * kMaxDeps * B;
  double *ring = smem + (size_t)W * (kStageBlocks * BB + kMaxDeps * B);
  if (threadIdx.x == 0) done_local = 0;
  if (lane == 0) mbar_init(&bars[warp]);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  volatile unsigned *dl = &done_local;
  unsigned phase = 0;
  int4 nm = make_int4(0, 0, 0, 0);
  int2 nd[kMaxDeps];
  auto fetch = [&](int slot) {
    if (slot < nslots) {
      nm = a.meta[p0 + slot];
#pragma unroll
      for (int k = 0; k < kMaxDeps; ++k) nd[k] = a.deps[(size_t)(p0 + slot) * kMaxDeps + k];
    }
  };
  fetch(warp);
  for (int slot = warp; slot < nslots; slot += W) {
    const int i = nm.x, e0 = nm.y, ne = nm.z;
    int2 dep[kMaxDeps];
#pragma unroll
    for (int k = 0; k < kMaxDeps; ++k) dep[k] = nd[k];
    const int nst = min(ne, BACK ? kStageBlocks - 1 : kStageBlocks);
    const bool copy = nst > 0 || BACK;
    if (copy && lane == 0) {
      const unsigned bytes = (unsigned)(sizeof(double) * BB * (nst + (BACK ? 1 : 0)));
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect(&bars[warp], bytes);
      if (nst) bulk_load(stage, a.data + (size_t)e0 * BB, (unsigned)(sizeof(double) * BB * nst), &bars[warp]);
      if (BACK)
        bulk_load(stage + (size_t)nst * BB, a.dinv + (size_t)i * BB, (unsigned)(sizeof(double) * BB), &bars[warp]);
    }
    fetch(slot + W);  // the next row's schedule is in flight during this row
    double acc[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = lane + 32 * s;
      acc[s] = r < B ? __ldcg(a.in + (size_t)i * B + r) : 0.;
    }
    // values of the rows other CTAs own, all polled together
    bool ok = true;
    unsigned missing = 0u;  // one bit per dependency still to come (per lane)
#pragma unroll
    for (int k = 0; k < kMaxDeps; ++k)
      if (k < ne && (dep[k].x >> kOwnerShift) != g) missing |= 1u << k;
    {
      const unsigned want = a.starve ? a.epoch + 1u : a.epoch;
      WaitClock clock;
      for (unsigned it = 1; __any_sync(0xffffffffu, missing != 0u); ++it) {
#pragma unroll
        for (int k = 0; k < kMaxDeps; ++k)
          if ((missing >> k) & 1u) {
            bool got = true;
            double v[S];
#pragma unroll
            for (int s = 0; s < S; ++s) {
              const int r = lane + 32 * s;
              v[s] = 0.;
              if (r < B) got = get_slot(a.slots + (size_t)dep[k].y * B + r, want, v[s]) && got;
            }
            if (got) {
              missing &= ~(1u << k);
#pragma unroll
              for (int s = 0; s < S; ++s)
                if (lane + 32 * s < B) vb[k * B + lane + 32 * s] = v[s];
            }
          }
        if ((it & kCheckGlobal) == 0) {
          int late = 0;
          if (lane == 0) late = out_of_time_call(clock, wb);
          if (__shfl_sync(0xffffffffu, late, 0)) {
            ok = false;
            break;
          }
        }
      }
    }
    if (copy) {
      if (!mbar_wait(&bars[warp], phase, kCopySpinLimit)) {
        give_up(a.abort, a.err);
        // let the copy land before the CTA can exit; if even the longer drain
        // bound runs out, the copy may still write this CTA's shared memory:
        // err[2] tells the host that the context can no longer be trusted
        if (!mbar_wait(&bars[warp], phase, kDrainSpinLimit) && lane == 0) atomicExch(a.err + 2, 1);
        return;
      }
      phase ^= 1u;
    }
    if (!ok) return;
    __syncwarp();
    // the lane's rows of a block, read before the vector is there
    double ar[S][B];
    const auto load_block = [&](const double *A) {
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int cc = 0; cc < B; ++cc) ar[s][cc] = lane + 32 * s < B ? A[cc * B + lane + 32 * s] : 0.;
    };
    const auto product = [&](const double *v, double sign) {
      double t[S][4];
#pragma unroll
      for (int s = 0; s < S; ++s) t[s][0] = t[s][1] = t[s][2] = t[s][3] = 0.;
#pragma unroll
      for (int cc = 0; cc < B; cc += 4) {
        const double2 a = *reinterpret_cast<const double2 *>(v + cc), b = *reinterpret_cast<const double2 *>(v + cc + 2);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          t[s][0] = fma(ar[s][cc], a.x, t[s][0]);
          t[s][1] = fma(ar[s][cc + 1], a.y, t[s][1]);
          t[s][2] = fma(ar[s][cc + 2], b.x, t[s][2]);
          t[s][3] = fma(ar[s][cc + 3], b.y, t[s][3]);
        }
      }
#pragma unroll
      for (int s = 0; s < S; ++s) acc[s] = fma(sign, (t[s][0] + t[s][1]) + (t[s][2] + t[s][3]), acc[s]);
    };
#pragma unroll
    for (int k = 0; k < kMaxDeps; ++k)
      if (k < ne && (dep[k].x >> kOwnerShift) != g) {
        load_block(k < nst ? stage + (size_t)k * BB : a.data + (size_t)(e0 + k) * BB);
        product(vb + k * B, -1.);
      }
    // the CTA's own rows, the ones finished first in front; a lane whose wait
    // gives up goes on with whatever the ring holds, so that the warp reaches
    // its barriers together, and all leave behind the last row
#pragma unroll
    for (int k0 = 0; k0 < kMaxDeps; ++k0) {
      const int k = BACK ? kMaxDeps - 1 - k0 : k0;
      if (k < ne && (dep[k].x >> kOwnerShift) == g) {
        const int js = dep[k].x & kSlotMask;
        load_block(k < nst ? stage + (size_t)k * BB : a.data + (size_t)(e0 + k) * BB);
        ok = wait_local(dl, (unsigned)js + 1, wb) && ok;
        __threadfence_block();
        const double *v = ring + (size_t)(js & (a.ring - 1)) * B;
        if (slot - js > a.ring - W) {  // gone from the ring
          for (int r = lane; r < B; r += 32) vb[k * B + r] = __ldcg(a.out + (size_t)dep[k].y * B + r);
          __syncwarp();
          v = vb + k * B;
        }
        product(v, -1.);
      }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) return;
    if (BACK) {
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (lane + 32 * s < B) vb[lane + 32 * s] = acc[s];
      load_block(stage + (size_t)nst * BB);
      __syncwarp();
#pragma unroll
      for (int s = 0; s < S; ++s) acc[s] = 0.;
      product(vb, 1.);
    }
    double *rs = ring + (size_t)(slot & (a.ring - 1)) * B;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = lane + 32 * s;
      if (r < B) rs[r] = acc[s];
    }
    __threadfence_block();
    // behind the fence, which would wait for them: other CTAs check the words
    // themselves, and this CTA reads `out` only for rows that left the ring,
    // whose warp has fenced again for its next row since (ring >= 4 W)
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int r = lane + 32 * s;
      if (r < B) {
        put_slot(a.slots + (size_t)i * B + r, acc[s], a.epoch);
        a.out[(size_t)i * B + r] = acc[s];
      }
    }
    __syncwarp();
    int pub = 1;
    if (lane == 0) {
      pub = wait_local(dl, (unsigned)slot, wb);  // rows are published in order
      if (pub) {
        *dl = (unsigned)slot + 1;
        // for the bound of the waits only: no fence, nothing is read behind it (at
        // every row the store took 1.5% of an update at 48x48 Q4)
        if ((slot & 15) == 15 || slot + 1 == nslots)
          *(volatile unsigned long long *)(a.progress + g) = a.tag | (unsigned long long)(slot + 1);
      }
    }
    if (!__shfl_sync(0xffffffffu, pub, 0)) return;
  }
}

// ----------------------------------------------------------- factor kernel
struct FactorArgs {
  int B, maxrow, maxupd, maxl, maxtot;
  int ahead;          // small blocks: the next row's blocks have a buffer of their own
  const int *slot_ptr;
  const int4 *meta;   // forward schedule: (row, first lower entry, lower count)
  const int2 *deps;
  const int *row, *diag, *upd_ptr, *upd;
  double *data, *dinv, *work;
  unsigned long long *progress;
  int *abort, *err;
  unsigned long long tag;
  unsigned long long limit_ns;  // bound of the waits (WaitBound)
  int starve;                   // test setting: waits on other CTAs can never be met
};

// FixedBlockILU::Factor (src/block_ilu.cpp:74-87), one CTA per row: for each
// lower entry (i,k) in column order, L_ik = A_ik U_kk^{-1}, then A_ij -= L_ik
// U_kj over the retained products; finally the pivoted LU of the diagonal
// block, stored as its explicit inverse. With SMEM the row's blocks, U_kk^{-1}
// and the U_kj of one step are staged in shared memory.
template <int RMAX, bool SMEM>
__global__ void __launch_bounds__(256, 1) ilu_factor_kernel(FactorArgs a) {
  extern __shared__ __align__(16) double fsm[];
  __shared__ int piv_s[32 * RMAX];
  __shared__ double inv_piv[32 * RMAX];
  __shared__ double bcast[2];
  __shared__ int stop;
  const int B = a.B;
  const int BB = B * B;
  const int g = blockIdx.x, p0 = a.slot_ptr[g], nslots = a.slot_ptr[g + 1] - p0;
  const WaitBound wb{a.progress, a.abort, a.err, a.limit_ns};
  double *Lt, *Sd, *Inv, *rowblk = nullptr, *Dk = nullptr, *Ub = nullptr;
  if (SMEM) {
    rowblk = fsm;                         // the row's blocks (maxrow)
    Dk = rowblk + (size_t)a.maxrow * BB;  // U_kk^{-1}
    Ub = Dk + BB;                         // the U_kj of one step (maxupd)
    Lt = Ub + (size_t)a.maxupd * BB;
  } else {
    Lt = a.work + (size_t)g * 3 * BB;
  }
  Sd = Lt + BB;
  Inv = Sd + BB;
  for (int slot = 0; slot < nslots; ++slot) {
    const int4 m = a.meta[p0 + slot];
    const int i = m.x, rb = a.row[i], re = a.row[i + 1], di = a.diag[i];
    if (threadIdx.x == 0) {
      int ok = 1;
      for (int k = 0; k < m.z && ok; ++k) {
        const int2 d = a.deps[(size_t)(p0 + slot) * kMaxDeps + k];
        const int owner = d.x >> kOwnerShift, js = d.x & kSlotMask;
        if (owner != g)
          ok = wait_progress(a.progress + owner, need(a.tag, js, a.starve), wb);
      }
      stop = !ok;
    }
    if (SMEM)
      for (int o = threadIdx.x; o < (re - rb) * BB; o += blockDim.x) rowblk[o] = a.data[(size_t)rb * BB + o];
    __syncthreads();
    if (stop) return;
    for (int ik = rb; ik < di; ++ik) {
      const int kk = a.deps[(size_t)(p0 + slot) * kMaxDeps + (ik - rb)].y;
      const int u0 = a.upd_ptr[ik], nu = a.upd_ptr[ik + 1] - u0;
      double *Aik = SMEM ? rowblk + (size_t)(ik - rb) * BB : a.data + (size_t)ik * BB;
      const double *Dsrc = a.dinv + (size_t)kk * BB;
      if (SMEM) {
        for (int o = threadIdx.x; o < BB; o += blockDim.x) Dk[o] = __ldcg(Dsrc + o);
        for (int t = threadIdx.x; t < nu * BB; t += blockDim.x)
          Ub[t] = __ldcg(a.data + (size_t)a.upd[2 * (u0 + t / BB) + 1] * BB + t % BB);
        __syncthreads();
      }
      for (int o = threadIdx.x; o < BB; o += blockDim.x) {
        const int r = o % B, cc = o / B;
        double sum = 0.;
        if (SMEM) {
          for (int s = 0; s < B; ++s) sum += Aik[(size_t)s * B + r] * Dk[(size_t)cc * B + s];
        } else {
          for (int s = 0; s < B; ++s) sum += Aik[(size_t)s * B + r] * __ldcg(Dsrc + (size_t)cc * B + s);
        }
        Lt[o] = sum;
      }
      __syncthreads();
      for (int o = threadIdx.x; o < BB; o += blockDim.x) Aik[o] = Lt[o];
      for (int t = threadIdx.x; t < nu * BB; t += blockDim.x) {
        const int uu = t / BB, o = t % BB;
        const int r = o % B, cc = o / B;
        const int target = a.upd[2 * (u0 + uu)];
        double *T = SMEM ? rowblk + (size_t)(target - rb) * BB : a.data + (size_t)target * BB;
        double sum = 0.;
        if (SMEM) {
          const double *U = Ub + (size_t)uu * BB;
          for (int s = 0; s < B; ++s) sum += Lt[(size_t)s * B + r] * U[(size_t)cc * B + s];
        } else {
          const double *U = a.data + (size_t)a.upd[2 * (u0 + uu) + 1] * BB;
          for (int s = 0; s < B; ++s) sum += Lt[(size_t)s * B + r] * __ldcg(U + (size_t)cc * B + s);
        }
        T[o] -= sum;
      }
      __syncthreads();
    }
    const double *Ad = SMEM ? rowblk + (size_t)(di - rb) * BB : a.data + (size_t)di * BB;
    for (int o = threadIdx.x; o < BB; o += blockDim.x) {
      Sd[o] = Ad[o];
      Inv[o] = (o % B) == (o / B) ? 1. : 0.;
    }
    __syncthreads();
    const bool ok = cta_lu_solve<RMAX>(Sd, B, Inv, B, B, B, piv_s, inv_piv, bcast);
    if (!ok && threadIdx.x == 0) raise_err(a.err, DERR_SINGULAR_ILU);
    double *Di = a.dinv + (size_t)i * BB;
    for (int o = threadIdx.x; o < BB; o += blockDim.x) Di[o] = Inv[o];
    if (SMEM)
      for (int o = threadIdx.x; o < (re - rb) * BB; o += blockDim.x) a.data[(size_t)rb * BB + o] = rowblk[o];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) publish_max(a.progress + g, a.tag | (unsigned long long)(slot + 1));
  }
}

// One 8x8 tile of sign X Y added to (d0, d1), B x B blocks column-major in
// shared memory, zero beyond B. Free of bank conflicts: B % 8 == 4, or the rows
// of a tile are next to each other.
template <int B>
__device__ __forceinline__ void block_tile(double &d0, double &d1, const double *X, const double *Y, int tr, int tc,
                                           double sign) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3, r = 8 * tr + gq, c = 8 * tc + gq;
#pragma unroll
  for (int s = 0; s < B; s += 4)
    dmma_m8n8k4(d0, d1, r < B ? sign * X[(s + tq) * B + r] : 0., c < B ? Y[c * B + s + tq] : 0.);
}

// Factor for blocks of at most 32 (every HDG degree below 8): the arithmetic
// of ilu_factor_kernel with the block size known at compile time. One CTA per
// row as there; the chain of rows bounds it, so what counts is the latency of a
// row. Its schedule and (where they fit twice) its blocks are fetched while the
// row before inverts its diagonal block, all blocks of its neighbours (inverse
// diagonals and retained U) are read in one round, products run on the FP64
// tensor pipe, and the diagonal block is inverted by one warp in registers, a
// row per lane: Gauss-Jordan in place with row pivoting, no barrier in its
// steps, the search for the next pivot under the other columns' update.
// 48x48 Q4: 16.3 ms with the kernel above, 3.6 here (5.8 with a row fetched when
// its turn came and products by FMAs out of shared memory). The kernel above
// keeps B = 36, whose rows do not fit one warp's lanes.
template <int B>
__global__ void __launch_bounds__(512, 1) ilu_factor_small_kernel(FactorArgs a) {
  constexpr int BB = B * B, MT = (B + 7) / 8, TILES = MT * MT;
  extern __shared__ __align__(16) double fsm[];
  __shared__ int stop;
  __shared__ int4 s_row[2];  // row, lower count, first entry, entries
  __shared__ int2 s_dep[2][kMaxDeps], s_upd[2][kMaxDeps * kMaxDeps];  // updates: (target entry in the row, U entry)
  __shared__ int s_ptr[2][kMaxDeps + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int g = blockIdx.x, p0 = a.slot_ptr[g], nslots = a.slot_ptr[g + 1] - p0;
  const WaitBound wb{a.progress, a.abort, a.err, a.limit_ns};
  double *rows = fsm;                                      // a.ahead + 1 buffers for a row's blocks (maxrow)
  double *Dk = rows + (size_t)(a.ahead + 1) * a.maxrow * BB;  // U_kk^{-1} of the lower neighbours (maxl)
  double *Ub = Dk + (size_t)a.maxl * BB;                   // their retained U_kj (maxtot)
  double *Lt = Ub + (size_t)a.maxtot * BB;
  const auto row_blocks = [&](int slot) { return rows + (size_t)(slot & a.ahead) * a.maxrow * BB; };
  const auto load_row = [&](int slot, int rb, int nb, int t, int nt) {
    const double2 *src = reinterpret_cast<const double2 *>(a.data + (size_t)rb * BB);
    double2 *dst = reinterpret_cast<double2 *>(row_blocks(slot));
    for (int o = t; o < nb * BB / 2; o += nt) dst[o] = src[o];
  };
  // the schedule of a row, by threads t of nt >= 64
  const auto fetch = [&](int slot, int t, int nt) {
    const int buf = slot & 1;
    const int4 m = a.meta[p0 + slot];
    const int rb = a.row[m.x], nb = a.row[m.x + 1] - rb, u0 = a.upd_ptr[rb], ntot = a.upd_ptr[rb + m.z] - u0;
    if (t == 0) s_row[buf] = make_int4(m.x, m.z, rb, nb);
    if (t < m.z) s_dep[buf][t] = a.deps[(size_t)(p0 + slot) * kMaxDeps + t];
    if (t <= m.z) s_ptr[buf][t] = a.upd_ptr[rb + t] - u0;
    if (t < ntot) s_upd[buf][t] = make_int2(a.upd[2 * (u0 + t)] - rb, a.upd[2 * (u0 + t) + 1]);
    if (a.ahead) load_row(slot, rb, nb, t, nt);
  };
  if (nslots > 0) fetch(0, threadIdx.x, blockDim.x);
  __syncthreads();
  for (int slot = 0; slot < nslots; ++slot) {
    const int buf = slot & 1;
    const int i = s_row[buf].x, nl = s_row[buf].y, rb = s_row[buf].z, nb = s_row[buf].w;
    double *rowblk = row_blocks(slot);
    if (!a.ahead) load_row(slot, rb, nb, threadIdx.x, blockDim.x);
    if (threadIdx.x == 0) {
      int ok = 1;
      for (int k = 0; k < nl && ok; ++k) {
        const int2 d = s_dep[buf][k];
        const int owner = d.x >> kOwnerShift, js = d.x & kSlotMask;
        if (owner != g)
          ok = wait_progress(a.progress + owner, need(a.tag, js, a.starve), wb);
      }
      stop = !ok;
    }
    __syncthreads();
    if (stop) return;
    const int ntot = s_ptr[buf][nl];
    for (int o = threadIdx.x; o < (nl + ntot) * (BB / 2); o += blockDim.x) {
      const int blk = o / (BB / 2), e = o % (BB / 2);
      const double *src = blk < nl ? a.dinv + (size_t)s_dep[buf][blk].y * BB
                                   : a.data + (size_t)s_upd[buf][blk - nl].y * BB;
      double *dst = blk < nl ? Dk + (size_t)blk * BB : Ub + (size_t)(blk - nl) * BB;
      reinterpret_cast<double2 *>(dst)[e] = __ldcg(reinterpret_cast<const double2 *>(src) + e);
    }
    __syncthreads();
    const int gq = lane >> 2, tq = lane & 3;
    for (int k = 0; k < nl; ++k) {
      const int v0 = s_ptr[buf][k], nu = s_ptr[buf][k + 1] - v0;
      double *Aik = rowblk + (size_t)k * BB;
      for (int t = warp; t < TILES; t += nwarps) {
        const int tr = t % MT, tc = t / MT, r = 8 * tr + gq, c = 8 * tc + 2 * tq;
        double d0 = 0., d1 = 0.;
        block_tile<B>(d0, d1, Aik, Dk + (size_t)k * BB, tr, tc, 1.);
        if (r < B && c < B) {  // c + 1 too: B is even
          Lt[c * B + r] = d0;
          Lt[(c + 1) * B + r] = d1;
        }
      }
      __syncthreads();
      for (int t = warp; t < nu * TILES; t += nwarps) {
        const int uu = v0 + t / TILES, tr = t % MT, tc = t % TILES / MT, r = 8 * tr + gq, c = 8 * tc + 2 * tq;
        double *T = rowblk + (size_t)s_upd[buf][uu].x * BB + c * B + r;
        const bool in = r < B && c < B;
        double d0 = in ? T[0] : 0., d1 = in ? T[B] : 0.;
        block_tile<B>(d0, d1, Lt, Ub + (size_t)uu * BB, tr, tc, -1.);
        if (in) {
          T[0] = d0;
          T[B] = d1;
        }
      }
      for (int o = threadIdx.x; o < BB; o += blockDim.x) Aik[o] = Lt[o];
      __syncthreads();
    }
    if (warp == 0) {
      const double *Ad = rowblk + (size_t)nl * BB;
      double w[B];
#pragma unroll
      for (int c = 0; c < B; ++c) w[c] = lane < B ? Ad[c * B + lane] : 0.;
      bool un = lane < B, singular = false;
      int pos = 0, mycol = 0;  // the step whose pivot row this lane is; the pivot row of step `lane`
      const auto search = [&](double x) {
        // largest magnitude (within 2^-15), first row on ties
        const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
        const unsigned key = (un && hi < 0x7ff00000u) ? ((hi & ~31u) | (unsigned)(31 - lane)) : 0u;
        return __reduce_max_sync(0xffffffffu, key);
      };
      unsigned mb = search(w[0]);
#pragma unroll
      for (int k = 0; k < B; ++k) {
        singular = singular || (mb >> 5) == 0u;
        const int p = 31 - (int)(mb & 31u);
        const bool me = lane == p;
        const double ip = 1.0 / __shfl_sync(0xffffffffu, w[k], p), l = w[k];
        mycol = lane == k ? p : mycol;
        pos = me ? k : pos;
        un = un && !me;
#pragma unroll
        for (int c0 = 1; c0 < B; ++c0) {
          const int c = (k + c0) % B;  // the next pivot's column first
          const double v = __shfl_sync(0xffffffffu, w[c], p) * ip;
          w[c] = me ? v : fma(-l, v, w[c]);
          if (c0 == 1 && k + 1 < B) mb = search(w[c]);
        }
        w[k] = me ? ip : -l * ip;
      }
      if (singular && lane == 0) raise_err(a.err, DERR_SINGULAR_ILU);
      double *Di = a.dinv + (size_t)i * BB;
#pragma unroll
      for (int c = 0; c < B; ++c) {
        const int col = __shfl_sync(0xffffffffu, mycol, c);
        if (lane < B) Di[col * B + pos] = w[c];
      }
    } else {
      double2 *dst = reinterpret_cast<double2 *>(a.data + (size_t)rb * BB);
      for (int o = threadIdx.x - 32; o < nb * BB / 2; o += blockDim.x - 32)
        dst[o] = reinterpret_cast<const double2 *>(rowblk)[o];
      if (slot + 1 < nslots) fetch(slot + 1, threadIdx.x - 32, blockDim.x - 32);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) publish_max(a.progress + g, a.tag | (unsigned long long)(slot + 1));
  }
}

// ------------------------------------------------------------ fill kernels
// HDG: all 16 panels C_s R_s X_{:,o} of every cell (FaceCoupling::Panel,
// src/operators.cpp:7-26), layout [cell][s][o][t x t column-major].
template <int Q>
__global__ void __launch_bounds__(256)
    ilu_panels_kernel(Geo g, const double *__restrict__ tab, const double *__restrict__ XY,
                      const double *__restrict__ Cb, double *__restrict__ panels16) {
  constexpr int P = Q * Q, M = 4 * P, T = 4 * Q, NR = 4 * T + 1, TT = T * T;
  __shared__ STab<Q> st;
  load_tables<Q>(st, tab);
  __syncthreads();
  const long long total = (long long)g.n * 16 * TT;
  for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(o / (16 * TT)), rem = (int)(o % (16 * TT));
    const int pan = rem / TT, r2 = rem % TT;
    const int row = r2 % T, cc = r2 / T;
    const int s = pan >> 2, so = pan & 3, jj = row >> 2, c = row & 3;
    const double *xc = XY + (size_t)e * M * NR + (size_t)(so * T + cc) * M;
    double val[4] = {0., 0., 0., 0.};
    for (int l = 0; l < Q; ++l) {
      const double f = st.fb(s, jj, l);
      const double *xv = xc + 4 * line_node<Q>(s, jj, l);
#pragma unroll
      for (int d = 0; d < 4; ++d) val[d] += f * xv[d];
    }
    const double *cb = Cb + ((size_t)e * 4 * Q + s * Q + jj) * 16;
    double res = 0.;
#pragma unroll
    for (int d = 0; d < 4; ++d) res += cb[c + 4 * d] * val[d];
    panels16[o] = res;
  }
}

// HDG block (f, g) = delta_fg D_f - sum over cells holding both faces of the
// cell's panel (side of f, side of g), in cell order (operators.cpp:48-74).
__global__ void __launch_bounds__(256)
    ilu_fill_hdg_kernel(int nnzb, int T, const int *__restrict__ erow, const int *__restrict__ col,
                        const int *__restrict__ fill_ptr, const int *__restrict__ fill_src,
                        const double *__restrict__ D, const double *__restrict__ panels16,
                        double *__restrict__ data) {
  const int TT = T * T;
  const long long total = (long long)nnzb * TT;
  for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(o / TT), r2 = (int)(o % TT);
    const int row = r2 % T, cc = r2 / T;
    const int f = erow[b];
    double v = (f == col[b] && row == cc) ? D[(size_t)f * T + row] : 0.;
    for (int p = fill_ptr[b]; p < fill_ptr[b + 1]; ++p) v = v - panels16[(size_t)fill_src[p] * TT + r2];
    data[o] = v;
  }
}

// DG blocks (PartialDGOperator::FillBlocks, src/partial.cpp:140-170): the
// diagonal is the cell block of block Jacobi; an off-diagonal block (a, b)
// holds, for every face joining a and b (in face order), +scale M^-1 phi phi jr
// when a is the face's left cell and -scale M^-1 phi phi jl when it is the
// right one. One CTA per block.
template <int Q>
__global__ void __launch_bounds__(256)
    ilu_fill_dg_kernel(Geo g, const double *__restrict__ tab, Frozen fz, const double *__restrict__ u,
                       int nnzb, const int *__restrict__ erow, const int *__restrict__ col,
                       const int *__restrict__ fill_ptr, const int *__restrict__ fill_src, double *data) {
  constexpr int P = Q * Q, M = 4 * P;
  __shared__ STab<Q> st;
  __shared__ double us[M], UT[16 * Q], FM[4 * Q * 16];
  load_tables<Q>(st, tab);
  for (int b = blockIdx.x; b < nnzb; b += gridDim.x) {
    __syncthreads();
    const int ea = erow[b], eb = col[b];
    double *A = data + (size_t)b * M * M;
    if (ea == eb) {
      for (int i = threadIdx.x; i < M; i += blockDim.x) us[i] = u[(size_t)ea * M + i];
      __syncthreads();
      cell_traces<Q>(st, us, UT);
      __syncthreads();
      dg_face_matrices<Q>(UT, FM, g, fz, ea);
      __syncthreads();
      build_cell_matrix<Q>(A, M, st, us, FM, g);
      continue;
    }
    for (int o = threadIdx.x; o < M * M; o += blockDim.x) A[o] = 0.;
    __syncthreads();
    for (int p = fill_ptr[b]; p < fill_ptr[b + 1]; ++p) {
      const int code = fill_src[p];
      const int f = code >> 1;
      const bool right = (code & 1) != 0;  // block row cell is the face's right cell
      const int L = f >> 1, axis = f & 1, ls = axis ? 3 : 1, rs = ls - 1;
      const int R = neighbour(L, ls, g.nx, g.ny);
      const int ts = right ? rs : ls, trs = right ? ls : rs, tc = right ? L : R;
      const double len = axis ? g.hx : g.hy;
      for (int j = threadIdx.x; j < Q; j += blockDim.x) {
        double tr[4], jm[16];
        trace4<Q>(st, u, tc, trs, j, tr);
        jacobian(tr, axis, g.gm1, jm);
        const int fi = f * Q + j;
        const double wgt = right ? fz.lw[fi] : fz.rw[fi], pen = right ? fz.pen[fi] : -fz.pen[fi];
#pragma unroll
        for (int k = 0; k < 16; ++k) FM[j * 16 + k] = wgt * jm[k] + ((k % 5) == 0 ? pen : 0.);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < Q * Q * Q * 16; t += blockDim.x) {
        const int j = t / (Q * Q * 16), rem = t % (Q * Q * 16);
        const int li = rem / (Q * 16), lk = (rem / 16) % Q, cd = rem % 16, c = cd & 3, d = cd >> 2;
        const int i = line_node<Q>(ts, j, li), kk = line_node<Q>(trs, j, lk);
        const double scale = g.dt * len / g.area * st.ew(j);
        const double w = (right ? -scale : scale) * st.inv_mass(i) * st.fb(ts, j, li) * st.fb(trs, j, lk);
        A[(size_t)(4 * kk + d) * M + 4 * i + c] += w * FM[j * 16 + c + 4 * d];
      }
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------ host: plan
template <class Kern>
int per_sm(Kern kern, int block, size_t smem) {
  // The opt-in is the most the kernel can have, not smem: it belongs to the
  // function, and the sizes differ between meshes (a factor row has more updates
  // on 3 x 3 cells than on 12 x 10), so one context would lower another's.
  if (smem > 0) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa{};
    EG_CUDA(cudaGetDevice(&dev));
    EG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    EG_CUDA(cudaFuncGetAttributes(&fa, kern));
    EG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
  }
  int n = 0;
  EG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, block, smem));
  return n;
}

template <int S>
int sweep_occupancy(int block, size_t smem) {
  return std::min(per_sm(ilu_sweep_kernel<S, false>, block, smem), per_sm(ilu_sweep_kernel<S, true>, block, smem));
}
int sweep_occupancy_dispatch(int S, int block, size_t smem) {
  switch (S) {
    case 2: return sweep_occupancy<2>(block, smem);
    case 3: return sweep_occupancy<3>(block, smem);
    case 4: return sweep_occupancy<4>(block, smem);
    case 5: return sweep_occupancy<5>(block, smem);
    case 6: return sweep_occupancy<6>(block, smem);
    case 7: return sweep_occupancy<7>(block, smem);
    case 8: return sweep_occupancy<8>(block, smem);
    case 9: return sweep_occupancy<9>(block, smem);
    case 10: return sweep_occupancy<10>(block, smem);
    case 11: return sweep_occupancy<11>(block, smem);
    default: fail(EG_ERR_INVALID, "unsupported block size");
  }
}
// the block sizes of the compile-time kernels: every HDG degree, DG up to k = 2
#define EG_ILU_SMALL(B, CALL)                                         \
  switch (B) {                                                        \
    case 4: { constexpr int BS = 4; CALL; } break;                    \
    case 8: { constexpr int BS = 8; CALL; } break;                    \
    case 12: { constexpr int BS = 12; CALL; } break;                  \
    case 16: { constexpr int BS = 16; CALL; } break;                  \
    case 20: { constexpr int BS = 20; CALL; } break;                  \
    case 24: { constexpr int BS = 24; CALL; } break;                  \
    case 28: { constexpr int BS = 28; CALL; } break;                  \
    case 32: { constexpr int BS = 32; CALL; } break;                  \
    case 36: { constexpr int BS = 36; CALL; } break;                  \
    default: fail(EG_ERR_INVALID, "unsupported block size");          \
  }
bool factor_small(int B) { return B <= 32; }
int small_sweep_occupancy(int B, int block, size_t smem) {
  EG_ILU_SMALL(B, return std::min(per_sm(ilu_sweep_small_kernel<BS, false>, block, smem),
                                  per_sm(ilu_sweep_small_kernel<BS, true>, block, smem)));
  return 0;
}
int small_factor_occupancy(int B, size_t smem) {
  EG_ILU_SMALL(B, if constexpr (BS <= 32) return per_sm(ilu_factor_small_kernel<BS>, 512, smem));
  return 0;
}
int factor_occupancy(int B, bool staged, size_t smem) {
  if (staged && factor_small(B)) return small_factor_occupancy(B, smem);
  if (staged)
    return per_sm(ilu_factor_kernel<2, true>, 256, smem);
  switch ((B + 31) / 32) {
    case 2: return per_sm(ilu_factor_kernel<2, false>, 256, 0);
    case 3: return per_sm(ilu_factor_kernel<3, false>, 256, 0);
    case 4: return per_sm(ilu_factor_kernel<4, false>, 256, 0);
    case 5: return per_sm(ilu_factor_kernel<5, false>, 256, 0);
    case 6: return per_sm(ilu_factor_kernel<6, false>, 256, 0);
    case 7: return per_sm(ilu_factor_kernel<7, false>, 256, 0);
    case 8: return per_sm(ilu_factor_kernel<8, false>, 256, 0);
    case 9: return per_sm(ilu_factor_kernel<9, false>, 256, 0);
    case 10: return per_sm(ilu_factor_kernel<10, false>, 256, 0);
    case 11: return per_sm(ilu_factor_kernel<11, false>, 256, 0);
    default: fail(EG_ERR_INVALID, "unsupported block size");
  }
}

void build_plan(Ctx &c, int form) {
  IluPlan &P = c.ilu[form];
  if (P.built) return;
  const bool hdg = form == EG_FORM_HDG;
  const int nx = c.desc.nx, ny = c.desc.ny;
  P.rows = hdg ? c.nf : c.n;
  P.B = hdg ? c.t : c.m;
  P.chunk = hdg ? 2 * nx : nx;
  P.chunks = ny;
  // Problem::SolverGraph (src/block_ilu.cpp:110-124) plus the row itself
  std::vector<std::vector<int>> graph(P.rows);
  if (hdg) {
    for (int e = 0; e < c.n; ++e)
      for (int s = 0; s < 4; ++s)
        for (int o = 0; o < 4; ++o) graph[cell_face(e, s, nx, ny)].push_back(cell_face(e, o, nx, ny));
  } else {
    for (int e = 0; e < c.n; ++e) graph[e].push_back(e);
    for (int f = 0; f < c.nf; ++f) {
      const int L = f >> 1, R = neighbour(L, (f & 1) ? 3 : 1, nx, ny);
      graph[L].push_back(R);
      graph[R].push_back(L);
    }
  }
  std::vector<int> row(1, 0), col, diag(P.rows), erow;
  for (int i = 0; i < P.rows; ++i) {
    auto &r = graph[i];
    r.push_back(i);
    std::sort(r.begin(), r.end());
    r.erase(std::unique(r.begin(), r.end()), r.end());
    for (int j : r) {
      if (j == i) diag[i] = (int)col.size();
      col.push_back(j);
      erow.push_back(i);
    }
    row.push_back((int)col.size());
  }
  P.nnzb = (int)col.size();
  // retained ILU(0) products (src/block_ilu.cpp:46-57)
  std::vector<int> upd_ptr(1, 0), upd;
  P.maxupd = 1;
  for (int i = 0; i < P.rows; ++i) {
    for (int ik = row[i]; ik < row[i + 1]; ++ik) {
      int count = 0;
      if (ik < diag[i]) {
        const int k = col[ik];
        int ij = ik + 1, kj = diag[k] + 1;
        while (ij < row[i + 1] && kj < row[k + 1]) {
          if (col[ij] < col[kj]) {
            ++ij;
          } else if (col[kj] < col[ij]) {
            ++kj;
          } else {
            upd.push_back(ij);
            upd.push_back(kj);
            ++count;
            ++ij;
            ++kj;
          }
        }
      }
      P.maxupd = std::max(P.maxupd, count);
      upd_ptr.push_back((int)upd.size() / 2);
    }
  }
  auto at = [&](int i, int j) {
    const auto it = std::lower_bound(col.begin() + row[i], col.begin() + row[i + 1], j);
    return (int)(it - col.begin());
  };
  // fill contributions per entry
  std::vector<std::vector<int>> contrib(P.nnzb);
  if (hdg) {
    for (int e = 0; e < c.n; ++e)
      for (int s = 0; s < 4; ++s)
        for (int o = 0; o < 4; ++o)
          contrib[at(cell_face(e, s, nx, ny), cell_face(e, o, nx, ny))].push_back(e * 16 + s * 4 + o);
  } else {
    for (int f = 0; f < c.nf; ++f) {
      const int L = f >> 1, R = neighbour(L, (f & 1) ? 3 : 1, nx, ny);
      contrib[at(L, R)].push_back(2 * f);
      contrib[at(R, L)].push_back(2 * f + 1);
    }
  }
  std::vector<int> fill_ptr(1, 0), fill_src;
  for (auto &v : contrib) {
    fill_src.insert(fill_src.end(), v.begin(), v.end());
    fill_ptr.push_back((int)fill_src.size());
  }
  if (fill_src.empty()) fill_src.push_back(0);
  if (upd.empty()) upd.push_back(0);
  P.maxl = P.maxu = P.maxrow = 0;
  P.maxtot = 1;
  for (int i = 0; i < P.rows; ++i) {
    P.maxl = std::max(P.maxl, diag[i] - row[i]);
    P.maxtot = std::max(P.maxtot, upd_ptr[diag[i]] - upd_ptr[row[i]]);
    P.maxu = std::max(P.maxu, row[i + 1] - diag[i] - 1);
    P.maxrow = std::max(P.maxrow, row[i + 1] - row[i]);
  }
  if (P.maxl > kMaxDeps || P.maxu > kMaxDeps) fail(EG_ERR_INVALID, "block ILU row too long");
  // launch shapes; every CTA of a sweep must be resident (cooperative launch)
  const int sms = device_sms();
  const size_t BB = (size_t)P.B * P.B;
  const int S = (P.B + 31) / 32;
  P.staged = P.B <= kStageMaxB ? 1 : 0;
  P.ring = 1;
  while ((size_t)(2 * P.ring) * P.B * sizeof(double) <= kRingBytes) P.ring *= 2;
  int W = 8;
  auto sweep_smem = [&](int w) {
    return sizeof(double) * ((size_t)w * (P.staged ? kStageBlocks * BB + kMaxDeps * P.B : 32 * S) +
                             (size_t)P.ring * P.B);
  };
  while (W > 1 && sweep_smem(W) > kSweepSmemBudget) --W;
  if (P.ring < (P.staged ? 4 : 2) * W) fail(EG_ERR_INVALID, "block ILU ring too small");
  P.sweep_warps = W;
  P.sweep_smem = sweep_smem(W);
  const auto factor_smem = [&](int row_buffers) {
    return sizeof(double) * BB * (size_t)(row_buffers * P.maxrow + P.maxl + P.maxtot + 1);
  };
  P.ahead = factor_small(P.B) && factor_smem(2) <= kFactorSmemBudget ? 1 : 0;
  P.factor_smem = !P.staged          ? 0
                  : factor_small(P.B) ? factor_smem(P.ahead + 1)
                                      : sizeof(double) * BB * (size_t)(P.maxrow + P.maxupd + 4);
  if (P.staged && P.maxtot > kMaxDeps * kMaxDeps) fail(EG_ERR_INVALID, "block ILU row too long");
  const int occ = std::min(P.staged ? small_sweep_occupancy(P.B, 32 * W, P.sweep_smem)
                                    : sweep_occupancy_dispatch(S, 32 * W, P.sweep_smem),
                           factor_occupancy(P.B, P.staged != 0, P.factor_smem));
  if (occ < 1) fail(EG_ERR_INVALID, "block ILU kernels do not fit on an SM");
  const int G = std::min(P.chunks, std::min(occ, 2) * sms);
  P.grid_sweep = P.grid_factor = G;
  // schedules (the forward one is also the factor's)
  auto upload = [&](const std::vector<int> &v) {
    int *d = c.alloc_n<int>(v.size());
    EG_CUDA(cudaMemcpyAsync(d, v.data(), sizeof(int) * v.size(), cudaMemcpyHostToDevice, c.stream));
    c.sync();  // the host vector is local
    return d;
  };
  for (int back = 0; back < 2; ++back) {
    std::vector<int> slot_ptr(G + 1, 0), owner_of(P.rows), slot_of(P.rows);
    std::vector<std::vector<int>> rows_of(G);
    for (int g = 0; g < G; ++g) {
      std::vector<int> chunks;
      for (int ch = g; ch < P.chunks; ch += G) chunks.push_back(ch);
      if (back) std::reverse(chunks.begin(), chunks.end());
      for (int ch : chunks)
        for (int o = 0; o < P.chunk; ++o) {
          const int i = ch * P.chunk + (back ? P.chunk - 1 - o : o);
          owner_of[i] = g;
          slot_of[i] = (int)rows_of[g].size();
          rows_of[g].push_back(i);
        }
      slot_ptr[g + 1] = slot_ptr[g] + (int)rows_of[g].size();
    }
    if (slot_ptr[G] != P.rows) fail(EG_ERR_INVALID, "block ILU schedule does not cover the rows");
    std::vector<int> meta((size_t)P.rows * 4, 0), deps((size_t)P.rows * kMaxDeps * 2, 0);
    for (int g = 0; g < G; ++g)
      for (size_t s = 0; s < rows_of[g].size(); ++s) {
        const int i = rows_of[g][s];
        const size_t pos = (size_t)slot_ptr[g] + s;
        const int e0 = back ? diag[i] + 1 : row[i], e1 = back ? row[i + 1] : diag[i];
        meta[pos * 4] = i;
        meta[pos * 4 + 1] = e0;
        meta[pos * 4 + 2] = e1 - e0;
        for (int e = e0; e < e1; ++e) {
          const int j = col[e], k = e - e0;
          // a row reads only rows that come earlier in its own CTA's order
          if (owner_of[j] == g && slot_of[j] >= (int)s) fail(EG_ERR_INVALID, "block ILU schedule order");
          if (slot_of[j] > kSlotMask) fail(EG_ERR_INVALID, "block ILU schedule too long");
          deps[(pos * kMaxDeps + k) * 2] = (owner_of[j] << kOwnerShift) | slot_of[j];
          deps[(pos * kMaxDeps + k) * 2 + 1] = j;
        }
      }
    P.slot_ptr[back] = upload(slot_ptr);
    P.meta[back] = upload(meta);
    P.deps[back] = upload(deps);
  }
  P.row = upload(row);
  P.col = upload(col);
  P.diag = upload(diag);
  P.erow = upload(erow);
  P.upd_ptr = upload(upd_ptr);
  P.upd = upload(upd);
  P.fill_ptr = upload(fill_ptr);
  P.fill_src = upload(fill_src);
  P.data = c.alloc_n<double>((size_t)P.nnzb * BB);
  P.dinv = c.alloc_n<double>((size_t)P.rows * BB);
  P.w = c.alloc_n<double>((size_t)P.rows * P.B);
  if (P.staged) {
    const size_t bytes = sizeof(ulonglong2) * (size_t)P.rows * P.B;
    P.slots = c.alloc(bytes);
    EG_CUDA(cudaMemsetAsync(P.slots, 0, bytes, c.stream));
  }
  // the condensation keeps all 16 panels per cell where the Schur action
  // streams them (same layout and arithmetic); otherwise the fill forms them
  if (hdg && c.geo.npan != 16) P.panels16 = c.alloc_n<double>((size_t)c.n * 16 * BB);
  if (!P.staged) P.work = c.alloc_n<double>((size_t)G * 3 * BB);
  P.progress = c.alloc_n<unsigned long long>(G);
  EG_CUDA(cudaMemsetAsync(P.progress, 0, sizeof(unsigned long long) * G, c.stream));
  P.abort = c.alloc_n<int>(1);
  EG_CUDA(cudaMemsetAsync(P.abort, 0, sizeof(int), c.stream));
  P.epoch = 0;
  P.wait_limit_ns = c.ilu_wait_limit_ns;
  P.starve = c.ilu_starve;
  P.built = true;
}

template <class Kern, class Args>
void launch_coop(Kern kern, int grid, int block, size_t smem, cudaStream_t s, Args &args) {
  void *params[] = {&args};
  EG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kern), grid, block, params, smem, s));
}

template <int S, bool BACK>
void sweep(Ctx &c, IluPlan &P, const double *in, double *out) {
  SweepArgs a{};
  a.B = P.B;
  a.ring = P.ring;
  a.slot_ptr = P.slot_ptr[BACK];
  a.meta = reinterpret_cast<const int4 *>(P.meta[BACK]);
  a.deps = reinterpret_cast<const int2 *>(P.deps[BACK]);
  a.data = P.data;
  a.dinv = P.dinv;
  a.in = in;
  a.out = out;
  a.progress = P.progress;
  a.abort = P.abort;
  a.err = c.derr;
  a.tag = (unsigned long long)(++P.epoch) << 32;
  a.limit_ns = P.wait_limit_ns;
  a.starve = P.starve;
  a.slots = static_cast<ulonglong2 *>(P.slots);
  a.epoch = P.epoch;
  if constexpr (S <= 2) {
    if (P.staged) {
      EG_ILU_SMALL(P.B, launch_coop(ilu_sweep_small_kernel<BS, BACK>, P.grid_sweep, 32 * P.sweep_warps, P.sweep_smem,
                                    c.stream, a));
      return;
    }
  }
  if constexpr (S >= 2)
    launch_coop(ilu_sweep_kernel<S, BACK>, P.grid_sweep, 32 * P.sweep_warps, P.sweep_smem, c.stream, a);
}

template <bool BACK>
void sweep_dispatch(Ctx &c, IluPlan &P, const double *in, double *out) {
  switch ((P.B + 31) / 32) {
    case 1: sweep<1, BACK>(c, P, in, out); break;
    case 2: sweep<2, BACK>(c, P, in, out); break;
    case 3: sweep<3, BACK>(c, P, in, out); break;
    case 4: sweep<4, BACK>(c, P, in, out); break;
    case 5: sweep<5, BACK>(c, P, in, out); break;
    case 6: sweep<6, BACK>(c, P, in, out); break;
    case 7: sweep<7, BACK>(c, P, in, out); break;
    case 8: sweep<8, BACK>(c, P, in, out); break;
    case 9: sweep<9, BACK>(c, P, in, out); break;
    case 10: sweep<10, BACK>(c, P, in, out); break;
    case 11: sweep<11, BACK>(c, P, in, out); break;
    default: fail(EG_ERR_INVALID, "unsupported block size");
  }
}

template <int RMAX, bool SMEM>
void factor_launch(Ctx &c, IluPlan &P) {
  FactorArgs a{};
  a.B = P.B;
  a.maxrow = P.maxrow;
  a.maxupd = P.maxupd;
  a.slot_ptr = P.slot_ptr[0];
  a.meta = reinterpret_cast<const int4 *>(P.meta[0]);
  a.deps = reinterpret_cast<const int2 *>(P.deps[0]);
  a.row = P.row;
  a.diag = P.diag;
  a.upd_ptr = P.upd_ptr;
  a.upd = P.upd;
  a.data = P.data;
  a.dinv = P.dinv;
  a.work = P.work;
  a.progress = P.progress;
  a.abort = P.abort;
  a.err = c.derr;
  a.tag = (unsigned long long)(++P.epoch) << 32;
  a.limit_ns = P.wait_limit_ns;
  a.starve = P.starve;
  a.maxl = P.maxl;
  a.ahead = P.ahead;
  a.maxtot = P.maxtot;
  if (SMEM && factor_small(P.B)) {
    EG_ILU_SMALL(P.B, if constexpr (BS <= 32)
                          launch_coop(ilu_factor_small_kernel<BS>, P.grid_factor, 512, P.factor_smem, c.stream, a));
    return;
  }
  launch_coop(ilu_factor_kernel<RMAX, SMEM>, P.grid_factor, 256, SMEM ? P.factor_smem : 0, c.stream, a);
}

void factor_dispatch(Ctx &c, IluPlan &P) {
  if (P.staged) {
    factor_launch<2, true>(c, P);
    return;
  }
  switch ((P.B + 31) / 32) {
    case 2: factor_launch<2, false>(c, P); break;
    case 3: factor_launch<3, false>(c, P); break;
    case 4: factor_launch<4, false>(c, P); break;
    case 5: factor_launch<5, false>(c, P); break;
    case 6: factor_launch<6, false>(c, P); break;
    case 7: factor_launch<7, false>(c, P); break;
    case 8: factor_launch<8, false>(c, P); break;
    case 9: factor_launch<9, false>(c, P); break;
    case 10: factor_launch<10, false>(c, P); break;
    case 11: factor_launch<11, false>(c, P); break;
    default: fail(EG_ERR_INVALID, "unsupported block size");
  }
}

// Numeric blocks of the plan's structure into dst (nnzb x B^2, column-major).
void fill_blocks(Ctx &c, int form, IluPlan &P, double *dst) {
  const bool hdg = form == EG_FORM_HDG;
  const int sms = device_sms();
  if (hdg) {
    const double *pan16 = c.geo.npan == 16 ? c.panels : P.panels16;
    if (c.geo.npan != 16) {
      const long long np = (long long)c.n * 16 * c.t * c.t;
      const int grid = (int)std::min<long long>((np + 255) / 256, (long long)sms * 16);
      EG_DISPATCH_Q(c.q, (ilu_panels_kernel<Q><<<grid, 256, 0, c.stream>>>(c.geo, c.tab, c.XY, c.Cb, P.panels16)));
      EG_CUDA(cudaGetLastError());
    }
    const long long ne = (long long)P.nnzb * c.t * c.t;
    const int g2 = (int)std::min<long long>((ne + 255) / 256, (long long)sms * 16);
    ilu_fill_hdg_kernel<<<g2, 256, 0, c.stream>>>(P.nnzb, c.t, P.erow, P.col, P.fill_ptr, P.fill_src, c.D,
                                                  pan16, dst);
  } else {
    const int grid = std::min(P.nnzb, sms * 8);
    EG_DISPATCH_Q(c.q, (ilu_fill_dg_kernel<Q><<<grid, 256, 0, c.stream>>>(
                           c.geo, c.tab, Frozen{c.fa, c.fbb, c.flw, c.frw, c.fpen}, c.u, P.nnzb, P.erow, P.col,
                           P.fill_ptr, P.fill_src, dst)));
  }
  EG_CUDA(cudaGetLastError());
}

// y = A x for an assembled block-sparse operator: one thread per scalar row;
// blocks are column-major, so consecutive rows of a block read adjacent
// entries, and block columns come in increasing order (the column order of
// the assembled CSR rows, src/operators.cpp:180-238).
__global__ void __launch_bounds__(256)
    bsr_spmv_kernel(int rows, int B, const int *__restrict__ rowp, const int *__restrict__ col,
                    const double *__restrict__ data, const double *__restrict__ x, double *__restrict__ y,
                    const int *__restrict__ skip) {
  if (skip != nullptr && *skip) return;  // speculative Arnoldi step after convergence
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (long long)rows * B) return;
  const int i = (int)(id / B), r = (int)(id % B);
  const size_t BB = (size_t)B * B;
  double acc = 0.;
  for (int k = rowp[i]; k < rowp[i + 1]; ++k) {
    const double *a = data + (size_t)k * BB + r;
    const double *xv = x + (size_t)col[k] * B;
#pragma unroll 4
    for (int j = 0; j < B; ++j) acc += a[(size_t)j * B] * xv[j];
  }
  y[id] = acc;
}

}  // namespace

void ilu_refresh(Ctx &c, int form, bool factor) {
  build_plan(c, form);
  IluPlan &P = c.ilu[form];
  const bool hdg = form == EG_FORM_HDG;
  if (hdg && !c.condensed) fail(EG_ERR_INVALID, "Schur preconditioner requires a condensation");
  ProfScope ps(c, hdg ? EG_K_SCHUR_JACOBI : EG_K_DG_JACOBI, factor ? 3 : 2);
  EG_CUDA(cudaMemsetAsync(P.abort, 0, sizeof(int), c.stream));
  fill_blocks(c, form, P, P.data);
  if (factor) factor_dispatch(c, P);
}

// ElementOperator::Assemble (src/operators.cpp:180-238) for full assembly and
// the element-assembled DG Jacobian (Problem::DG, src/problem.cpp:552-588):
// the blocks the ILU(0) fill sums (FillBlocks), left unfactored.
void assemble_blocks(Ctx &c, int form) {
  const bool hdg = form == EG_FORM_HDG;
  if (hdg && !c.condensed) fail(EG_ERR_INVALID, "assembled Schur operator requires a condensation");
  build_plan(c, form);
  IluPlan &P = c.ilu[form];
  ProfScope ps(c, EG_K_VECTOR, 2);
  if (c.opts.precond == EG_PC_BLOCK_ILU0) {
    if (!P.asm_own) P.asm_own = c.alloc_n<double>((size_t)P.nnzb * P.B * P.B);
    P.asmd = P.asm_own;
  } else {
    P.asmd = P.data;  // unused by block Jacobi
  }
  fill_blocks(c, form, P, P.asmd);
}

void launch_assembled_apply(Ctx &c, int form, const double *x, double *y) {
  IluPlan &P = c.ilu[form];
  if (!P.built || !P.asmd) fail(EG_ERR_INVALID, "no assembled operator");
  ProfScope ps(c, form == EG_FORM_HDG ? EG_K_SCHUR_APPLY : EG_K_DG_APPLY, 2);
  const long long total = (long long)P.rows * P.B;
  bsr_spmv_kernel<<<(unsigned)((total + 255) / 256), 256, 0, c.stream>>>(P.rows, P.B, P.row, P.col, P.asmd, x,
                                                                         y, c.skip);
  EG_CUDA(cudaGetLastError());
}

void launch_ilu_apply(Ctx &c, int form, const double *b, double *x) {
  IluPlan &P = c.ilu[form];
  if (!P.built) fail(EG_ERR_INVALID, "no preconditioner built");
  ProfScope ps(c, EG_K_PC_APPLY, 2);
  // a sweep that gave up leaves the abort word set; every apply starts clear
  EG_CUDA(cudaMemsetAsync(P.abort, 0, sizeof(int), c.stream));
  sweep_dispatch<false>(c, P, b, P.w);
  sweep_dispatch<true>(c, P, P.w, x);
}

}  // namespace eg
