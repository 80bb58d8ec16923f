// CUDA kernels of the Newton inner loop (sm_103a).
//
//  * first_factor  - the reference's first numeric factorization with its
//                    threshold pivot rule (crates/sim-core/src/native_klu.rs:
//                    1194-1382), one warp walking the columns in order; it
//                    discovers the pivot sequence. k_first_factor_s keeps the
//                    working column and each column's update operands in
//                    shared memory; k_first_factor is the fallback for blocks
//                    too large for that. From 16 rows on the host runs the
//                    same pass as refactorizations in their pivot-pass mode
//                    (PivotCheck) instead, and these kernels only when that
//                    does not settle.
//  * refactor      - left-looking refactorization with frozen pivots. Warps
//                    take columns in increasing order from an atomic counter
//                    and wait for exactly the columns they depend on (the U
//                    pattern), so independent columns run concurrently
//                    without level barriers; a warp's column sits in shared
//                    memory while it is updated. k_refactor_cta is the same
//                    in one block, for small plans.
//  * solve         - the forward (L) and backward (U) substitutions and the
//                    BTF block coupling, and A^T y = g for the adjoint.
//                    k_solve_steps runs them as a step program in one block
//                    (solution vector in shared memory), k_solve_cta sweeps
//                    the columns in one block; k_solve and k_tsolve run one
//                    warp per row task driven by per-row flags (large plans).
//  * stamp         - one thread per device instance writes its conductances
//                    into the raw CSC slots given by the stamp-to-slot map and
//                    its currents into per-contribution slots; a second pass
//                    sums the right-hand side row by row in stamping order.
//  * newton_update - convergence test, damping and the iterate update of
//                    crates/sim-core/src/newton.rs:93-107, 187-201.
//  * batch_newton  - batched Newton over many circuit instances, one warp per
//                    instance (or 2, 4 per warp for small programs) with the
//                    instance's whole state in shared memory; in use when the
//                    warp-per-instance kernel (cont.cu) is off, behind the
//                    lane kernel (lanes.cu) or alone.
//
// All floating-point work of the single-circuit kernels is FP64 and compiled
// without multiply-add contraction, so every product is rounded before it is
// added exactly as in the reference; their factor and solve results are
// bit-identical to a scalar CPU evaluation in the reference's order. The
// batched kernels use fused multiply-adds and agree with the oracle within
// the Newton tolerance.
#include <algorithm>
#include <cstdio>

#include "batch_common.cuh"
#include "device.cuh"
#include "kernels.cuh"

namespace gk {

namespace {
constexpr unsigned FULL = 0xffffffffu;

// --------------------------------------------------------------- first factor
__global__ void k_first_factor(DPlan P, const double* __restrict__ ax, double* lu,
                               double* work, int* rperm, int* rinv, double tol,
                               int* status) {
  const int lane = threadIdx.x;
  const int n = P.n;
  for (int i = lane; i < n; i += 32) {
    int b0 = P.block_ptr[P.pos_block[i]];
    rperm[i] = i - b0;
    rinv[i] = i - b0;
    work[i] = 0.0;
  }
  __syncwarp();
  for (int k = 0; k < n; ++k) {
    const int b0 = P.block_ptr[P.pos_block[k]];
    const int s0 = P.col_ptr[k], ds = P.dslot[k], s1 = P.col_ptr[k + 1];
    const int t0 = P.pcol_ptr[k], t1 = P.pcol_ptr[k + 1];
    if (P.col_single[k]) {
      if (lane == 0) {
        double d = 0.0;
        for (int t = t0; t < t1; ++t) d += ax[P.pcol_raw[t]];
        lu[ds] = perturb(d, true);
      }
      __syncwarp();
      continue;
    }
    if (lane == 0)  // duplicates accumulate in CSC order
      for (int t = t0; t < t1; ++t) {
        int w = b0 + rinv[b0 + P.pcol_q[t]];
        work[w] += ax[P.pcol_raw[t]];
      }
    __syncwarp();
    for (int s = s0; s < ds; ++s) {
      const int j = P.slot_row[s];
      const double u = work[j];
      if (u != 0.0) {
        const int q1 = P.col_ptr[j + 1];
        for (int q = P.dslot[j] + 1 + lane; q < q1; q += 32) {
          int r = P.slot_row[q];
          work[r] = work[r] - lu[q] * u;
        }
      }
      __syncwarp();
    }
    // threshold pivot search inside the symbolic pattern: the first row with
    // the largest magnitude wins; the diagonal wins ties
    const double dabs = fabs(work[k]);
    double best = -1.0;
    int bidx = 0x7fffffff;
    for (int q = ds + 1 + lane; q < s1; q += 32) {
      double v = fabs(work[P.slot_row[q]]);
      if (v > best) {
        best = v;
        bidx = q;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      double ov = __shfl_down_sync(FULL, best, off);
      int oi = __shfl_down_sync(FULL, bidx, off);
      if (ov > best || (ov == best && oi < bidx)) {
        best = ov;
        bidx = oi;
      }
    }
    best = __shfl_sync(FULL, best, 0);
    bidx = __shfl_sync(FULL, bidx, 0);
    if (lane == 0 && bidx != 0x7fffffff && best > dabs && dabs < tol * best) {
      const int mr = P.slot_row[bidx];
      double tmp = work[k];
      work[k] = work[mr];
      work[mr] = tmp;
      int ok = rperm[k], om = rperm[mr];
      rperm[k] = om;
      rperm[mr] = ok;
      rinv[b0 + ok] = mr - b0;
      rinv[b0 + om] = k - b0;
    }
    __syncwarp();
    for (int s = s0 + lane; s < ds; s += 32) lu[s] = work[P.slot_row[s]];
    const double diag = perturb(work[k], false);
    if (lane == 0) lu[ds] = diag;
    for (int q = ds + 1 + lane; q < s1; q += 32) lu[q] = work[P.slot_row[q]] / diag;
    __syncwarp();
    if (lane == 0)
      for (int t = t0; t < t1; ++t) work[b0 + rinv[b0 + P.pcol_q[t]]] = 0.0;
    for (int q = s0 + lane; q < s1; q += 32) work[P.slot_row[q]] = 0.0;
    __syncwarp();
    if (lane == 0) work[k] = 0.0;
    __syncwarp();
  }
  (void)status;
}

// The same first factorization with the working column, the block's row
// inverse and the operands of each column's updates in shared memory. The
// operations and their order are those of k_first_factor (and therefore the
// reference's); only where the operands sit differs. Per column:
//   1. A(:,k) is loaded by all lanes and lane 0 adds it into the working
//      column in CSC order;
//   2. the U entries are taken in chunks of 32, and a chunk in runs whose
//      L columns (rows and values, all of them final) fit the buffer: a run's
//      operands are copied into shared memory by cp.async, every lane issuing
//      its copies at once, and its updates then run in order out of shared
//      memory;
//   3. the threshold pivot search, the swap and the scaling follow.
// Shared layout: work[maxblk] f64, bl[cap] f64, rinv[maxblk] i32, br[cap]
// i32, kpat[kcap] i32, then the chunk table.
constexpr int kPatCap = 1024;

__device__ __forceinline__ void cp_async4(void* sdst, const void* gsrc) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__global__ void k_first_factor_s(DPlan P, const double* __restrict__ ax, double* lu,
                                 int* rperm, int* rinv, double tol, int maxblk, int cap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* const work = reinterpret_cast<double*>(smem_raw);
  double* const bl = work + maxblk;
  int* const srinv = reinterpret_cast<int*>(bl + cap);
  int* const br = srinv + maxblk;
  int* const kpat = br + cap;
  int* const soff = kpat + kPatCap;  // [33]
  int* const sq0 = soff + 33;        // [32]
  int* const sj = sq0 + 32;          // [32]
  const int lane = threadIdx.x;
  const int n = P.n;
  for (int i = lane; i < n; i += 32) rperm[i] = i - P.block_ptr[P.pos_block[i]];
  for (int i = lane; i < maxblk; i += 32) work[i] = 0.0;
  for (int b = 0; b < P.nblocks; ++b) {
    const int b0 = P.block_ptr[b], b1 = P.block_ptr[b + 1];
    for (int i = lane; i < b1 - b0; i += 32) srinv[i] = i;
    __syncwarp();
    for (int k = b0; k < b1; ++k) {
      const int s0 = P.col_ptr[k], ds = P.dslot[k], s1 = P.col_ptr[k + 1];
      const int t0 = P.pcol_ptr[k], t1 = P.pcol_ptr[k + 1];
      if (P.col_single[k]) {
        double d = 0.0;
        for (int tc = t0; tc < t1; tc += 32) {
          const double v = tc + lane < t1 ? ax[P.pcol_raw[tc + lane]] : 0.0;
          const int cnt = min(32, t1 - tc);
          for (int i = 0; i < cnt; ++i) d += __shfl_sync(FULL, v, i);
        }
        if (lane == 0) lu[ds] = perturb(d, true);
        continue;
      }
      const bool staged = s1 - s0 <= kPatCap;
      if (staged)
        for (int s = s0 + lane; s < s1; s += 32) cp_async4(&kpat[s - s0], &P.slot_row[s]);
      // 1. A(:,k), duplicates added in CSC order
      for (int tc = t0; tc < t1; tc += 32) {
        int q = 0;
        double v = 0.0;
        if (tc + lane < t1) {
          q = P.pcol_q[tc + lane];
          v = ax[P.pcol_raw[tc + lane]];
        }
        const int cnt = min(32, t1 - tc);
        for (int i = 0; i < cnt; ++i) {
          const int qi = __shfl_sync(FULL, q, i);
          const double vi = __shfl_sync(FULL, v, i);
          if (lane == 0) work[srinv[qi]] += vi;
        }
      }
      cp_async_wait_all();
      __syncwarp();
      auto row = [&](int s) { return staged ? kpat[s - s0] : P.slot_row[s]; };
      // 2. updates by the U entries, in order
      for (int sc = s0; sc < ds; sc += 32) {
        const int cnt = min(32, ds - sc);
        int j = 0, q0 = 0, len = 0;
        if (lane < cnt) {
          j = row(sc + lane);
          q0 = P.dslot[j] + 1;
          len = P.col_ptr[j + 1] - q0;
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        soff[lane] = incl - len;
        sq0[lane] = q0;
        sj[lane] = j;
        if (lane == 31) soff[32] = total;
        __syncwarp();
        // runs of consecutive U entries whose operands fit the buffer
        for (int i0 = 0; i0 < cnt;) {
          int i1 = i0 + 1;
          while (i1 < cnt && soff[i1 + 1] - soff[i0] <= cap) ++i1;
          const int e0 = soff[i0], e1 = soff[i1];
          if (e1 - e0 <= cap) {
            int si = i0;
            for (int e = e0 + lane; e < e1; e += 32) {
              while (soff[si + 1] <= e) ++si;
              const int q = sq0[si] + (e - soff[si]);
              cp_async4(&br[e - e0], &P.slot_row[q]);
              cp_async8(&bl[e - e0], &lu[q]);
            }
            cp_async_wait_all();
            __syncwarp();
            for (int i = i0; i < i1; ++i) {
              const double u = work[sj[i] - b0];
              if (u != 0.0) {
                const int ea = soff[i] - e0, eb = soff[i + 1] - e0;
                for (int e = ea + lane; e < eb; e += 32) {
                  const int r = br[e] - b0;
                  work[r] = work[r] - bl[e] * u;
                }
              }
              __syncwarp();
            }
          } else {  // one L column longer than the buffer: straight from memory
            const double u = work[sj[i0] - b0];
            const int qa = sq0[i0], qb = qa + (e1 - e0);
            if (u != 0.0)
              for (int q = qa + lane; q < qb; q += 32) {
                const int r = P.slot_row[q] - b0;
                work[r] = work[r] - lu[q] * u;
              }
            __syncwarp();
          }
          i0 = i1;
        }
      }
      // 3. threshold pivot search inside the symbolic pattern: the first row
      // with the largest magnitude wins; the diagonal wins ties
      const double dabs = fabs(work[k - b0]);
      double best = -1.0;
      int bidx = 0x7fffffff;
      for (int q = ds + 1 + lane; q < s1; q += 32) {
        const double v = fabs(work[row(q) - b0]);
        if (v > best) {
          best = v;
          bidx = q;
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_down_sync(FULL, best, off);
        const int oi = __shfl_down_sync(FULL, bidx, off);
        if (ov > best || (ov == best && oi < bidx)) {
          best = ov;
          bidx = oi;
        }
      }
      best = __shfl_sync(FULL, best, 0);
      bidx = __shfl_sync(FULL, bidx, 0);
      if (lane == 0 && bidx != 0x7fffffff && best > dabs && dabs < tol * best) {
        const int mr = row(bidx);
        const double tmp = work[k - b0];
        work[k - b0] = work[mr - b0];
        work[mr - b0] = tmp;
        const int ok = rperm[k], om = rperm[mr];
        rperm[k] = om;
        rperm[mr] = ok;
        srinv[ok] = mr - b0;
        srinv[om] = k - b0;
      }
      __syncwarp();
      for (int s = s0 + lane; s < ds; s += 32) lu[s] = work[row(s) - b0];
      const double diag = perturb(work[k - b0], false);
      if (lane == 0) lu[ds] = diag;
      for (int q = ds + 1 + lane; q < s1; q += 32) lu[q] = work[row(q) - b0] / diag;
      __syncwarp();
      for (int t = t0 + lane; t < t1; t += 32) work[srinv[P.pcol_q[t]]] = 0.0;
      for (int q = s0 + lane; q < s1; q += 32) work[row(q) - b0] = 0.0;
      __syncwarp();
      if (lane == 0) work[k - b0] = 0.0;
      __syncwarp();
    }
    for (int i = lane; i < b1 - b0; i += 32) rinv[b0 + i] = srinv[i];
    __syncwarp();
  }
}

// --------------------------------------------------------------- refactor
// The updates of a column: for its U entries s in order, of columns j, the
// slots upd_dst of the column lose u * l(q) for every L slot q of column j.
// The values and the destinations reach the warp through a ring of
// asynchronous copies, cut into pieces of up to 64 slots that start on an even
// slot (16 bytes); a piece's header {s, first slot, rows lo, hi and offset of
// the destinations, column} lies before them. The entries' ranges are read 32
// at a time, one per lane, two groups ahead. The operations and their order
// are the reference's.
constexpr int kPiece = 64;
constexpr int kDstBytes = 288;  // 64 destinations behind up to 3 others
constexpr int kGridRing = 8;    // pieces in flight per column
constexpr int kGridStage = 16 + kDstBytes + 8 * kPiece;
constexpr int kCtaRing = 4;
constexpr int kCtaStage = 16 + kDstBytes;  // the values are in shared memory
constexpr int kColCap = 4096;   // slots of a column kept in shared memory

// The grid kernel has no completion flags: every value of lu is preset to
// kUnset (all bits one, a NaN; a computed value with these bits is stored as
// another NaN) and a reader that finds it polls the value itself. One trip
// through L2 per dependency instead of three (fence, flag, value).
__device__ __forceinline__ bool unset(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ double ld_relaxed(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_set(double* p, double v) {
  if (unset(v)) v = __longlong_as_double(0x7fffffffffffffffll);
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_cta(const unsigned* p) {
  unsigned v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cta(unsigned* p, unsigned v) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// 16 bytes to shared memory, the first n of them from memory, the rest zero.
__device__ __forceinline__ void cp_async16(void* d, const void* g, int n) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(d);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(g), "r"(n) : "memory");
}

// The pieces of a column's updates in order, handed out one at a time (by all
// lanes alike): entries [s0, ds), those without L slots left out.
struct Pieces {
  const DPlan& P;
  int ds, sc, part;
  int j0, j1, j2, qa, qb, up, nqa, nqb, nup;  // this lane's entry of the group and of the next
  unsigned mask;                              // entries of the group not yet handed out
  __device__ __forceinline__ int row_of(int s) const { return s < ds ? P.slot_row[s] : -1; }
  __device__ __forceinline__ void range_of(int s, int j, int& a, int& b, int& u) const {
    a = b = u = 0;
    if (j >= 0) {
      a = P.dslot[j] + 1;
      b = P.col_ptr[j + 1];
      u = P.upd_ptr[s];
    }
  }
  __device__ __forceinline__ Pieces(const DPlan& P_, int s0, int ds_)
      : P(P_), ds(ds_), sc(s0), part(0) {
    const int lane = threadIdx.x & 31;
    j0 = row_of(s0 + lane);
    j1 = row_of(s0 + 32 + lane);
    j2 = row_of(s0 + 64 + lane);
    range_of(s0 + lane, j0, qa, qb, up);
    range_of(s0 + 32 + lane, j1, nqa, nqb, nup);
    mask = __ballot_sync(FULL, qb > qa);
    skip_empty();
  }
  __device__ __forceinline__ void skip_empty() {
    const int lane = threadIdx.x & 31;
    while (mask == 0 && sc + 32 < ds) {
      sc += 32;
      j0 = j1;
      qa = nqa;
      qb = nqb;
      up = nup;
      j1 = j2;
      range_of(sc + 32 + lane, j1, nqa, nqb, nup);
      j2 = row_of(sc + 64 + lane);
      mask = __ballot_sync(FULL, qb > qa);
    }
  }
  __device__ __forceinline__ bool more() const { return mask != 0; }
  // Starts the copies of the next piece into stage st (the values only when
  // there is a lu in memory) and returns its header.
  __device__ __forceinline__ int4 next(unsigned char* st, const double* lu) {
    const int lane = threadIdx.x & 31;
    const int i = __ffs(mask) - 1;
    const int a = __shfl_sync(FULL, qa, i), b = __shfl_sync(FULL, qb, i);
    const int u = __shfl_sync(FULL, up, i), j = __shfl_sync(FULL, j0, i);
    const int base = (a & ~1) + kPiece * part;
    const int lo = max(a - base, 0), hi = min(b - base, kPiece);
    const int d0 = u + base + lo - a, da = d0 & ~3, dend = u + base + hi - a;
    if (da + 4 * lane < dend)
      cp_async16(st + 16 + 16 * lane, P.upd_dst + da + 4 * lane,
                 min(16, 4 * (dend - da) - 16 * lane));
    if (lu != nullptr && 2 * lane < hi)  // lu is padded by a value
      cp_async16(st + 16 + kDstBytes + 16 * lane, lu + base + 2 * lane, 16);
    const int4 h = make_int4(sc + i, base, lo | hi << 8 | ((d0 & 3) - lo + 128) << 16, j);
    if (base + kPiece >= b) {
      mask &= mask - 1;
      part = 0;
    } else {
      ++part;
    }
    return h;
  }
};

// One piece as a warp holds it: a0, a1 this lane's rows, their destinations
// and values.
struct Piece {
  int4 h;
  int e0, e1;
  bool a0, a1, two;
  double v0, v1;
  __device__ __forceinline__ void read(const unsigned char* st, bool values) {
    const int lane = threadIdx.x & 31;
    h = *reinterpret_cast<const int4*>(st);
    const int lo = h.z & 255, hi = (h.z >> 8) & 255;
    const int* const dst = reinterpret_cast<const int*>(st + 16) + (((h.z >> 16) & 255) - 128);
    a0 = lane >= lo && lane < hi;  // lo is 0 or 1
    a1 = lane + 32 < hi;
    two = hi > 32;
    e0 = a0 ? dst[lane] : 0;
    e1 = a1 ? dst[lane + 32] : 0;
    if (values) {
      const double* const val = reinterpret_cast<const double*>(st + 16 + kDstBytes);
      v0 = a0 ? val[lane] : 0.0;
      v1 = a1 ? val[lane + 32] : 0.0;
    }
  }
};

// The updates of the column in slots [s0, ds) of a factor in shared memory
// (indexed by slot), completion flags in `done`, by one warp that copies its
// own pieces. Returns false when a wait gave up.
__device__ __forceinline__ bool block_updates(const DPlan& P, int s0, int ds, double* lu,
                                              const unsigned* done, unsigned char* ring,
                                              int* status) {
  const int lane = threadIdx.x & 31;
  Pieces todo(P, s0, ds);
  int live = 0, head = 0, tail = 0;
  auto issue = [&]() {
    if (todo.more()) {
      unsigned char* const st = ring + tail * kCtaStage;
      const int4 h = todo.next(st, nullptr);
      if (lane == 0) *reinterpret_cast<int4*>(st) = h;
      todo.skip_empty();
      tail = tail + 1 == kCtaRing ? 0 : tail + 1;
      ++live;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < kCtaRing; ++i) issue();
  Piece nx;
  auto read = [&]() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kCtaRing - 1) : "memory");  // the oldest has landed
    __syncwarp();
    nx.read(ring + head * kCtaStage, false);
  };
  bool ok = true;
  if (live > 0) read();
  while (live > 0) {
    const Piece p = nx;
    const double u = lu[p.h.x];
    double c0 = 0.0, c1 = 0.0;
    if (p.a0) c0 = lu[p.e0];
    if (p.two && p.a1) c1 = lu[p.e1];
    __syncwarp();  // the piece is read by all lanes: the next one takes its stage
    head = head + 1 == kCtaRing ? 0 : head + 1;
    --live;
    issue();
    if (live > 0) read();
    unsigned spins = 0;
    while (!__all_sync(FULL, ld_acquire_cta(&done[p.h.w]) != 0u)) {
      ++spins;
      bool stop = spins > P.spin_limit;
      if (stop && lane == 0) atomicCAS(status, DS_OK, DS_TIMEOUT);
      if ((spins & 1023u) == 0 && *(volatile int*)status != DS_OK) stop = true;
      if (__any_sync(FULL, stop)) {
        ok = false;
        break;
      }
      if (spins > 256) __nanosleep(20);  // shared-memory polls first
    }
    if (!ok) break;
    if (bt::nonzero(u)) {  // the same in every lane
      if (p.a0) lu[p.e0] = sub(c0, mul(lu[p.h.y + lane], u));
      if (p.two && p.a1) lu[p.e1] = sub(c1, mul(lu[p.h.y + lane + 32], u));
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  return ok;
}

// The L values of a column: C[q] / diag for q in (ds, s1), correctly rounded,
// handed to put(q, value). Division by an invariant integer (Granlund and
// Montgomery, PLDI 1994) on the significands: FP64 takes about ten operations
// of 64 cycles a division (620 cycles for 32 rows, one after another), the
// integer unit two products once the reciprocal stands.
//   w   2^116 / mb less at most 32, mb the divisor's significand in
//       [2^52, 2^53): a 24-bit reciprocal and two Newton steps in fixed point
//   q   floor(2^57 ma / mb), first as the high word of (ma << 5) w, then with
//       the remainder's correction; rounded to 53 bits, ties to even
// Zeros keep their sign; operands far from 1 and the non-finite are divided.
__device__ __forceinline__ unsigned long long significand(double v) {
  return ((unsigned long long)__double_as_longlong(v) & 0xfffffffffffffull) | (1ull << 52);
}
__device__ __forceinline__ int exponent(double v) {
  return (int)(((unsigned)__double2hiint(v) >> 20) & 0x7ffu);
}
__device__ __forceinline__ unsigned long long fixed_reciprocal(unsigned long long mb) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;"
      : "=f"(r)
      : "f"(__uint_as_float(0x3f800000u | (unsigned)(mb >> 29 & 0x7fffffu))));
  const unsigned long long x0 = __float2uint_rz(r * 4294967296.0f);  // saturates below 1
  const long long e1 = (long long)(0x8000000000000000ull - __umul64hi(mb << 11, x0 << 32));
  const unsigned long long x1 =
      (x0 << 32) + (unsigned long long)(((long long)x0 * (e1 >> 12)) >> 19);
  const long long e2 = (long long)(0x8000000000000000ull - __umul64hi(mb << 11, x1));
  return x1 + (unsigned long long)(((long long)(x1 >> 32) * e2) >> 31) - 16;
}
__device__ __forceinline__ double fixed_divide(double a, double b, unsigned long long mb,
                                               unsigned long long w) {
  const unsigned long long ma = significand(a);
  int e = exponent(a) - exponent(b);
  unsigned long long q = __umul64hi(ma << 5, w);
  unsigned long long r = (ma << 57) - q * mb;
  if (r >= mb) {
    q += 1;
    r -= mb;
  }
  if (q < (1ull << 57)) {
    q <<= 1;
    e -= 1;
  }
  const unsigned long long t = q | (r != 0 ? 1ull : 0ull);
  const unsigned long long m = (t + 15 + (t >> 5 & 1)) >> 5;
  const unsigned long long sign =
      (unsigned long long)(__double_as_longlong(a) ^ __double_as_longlong(b)) & (1ull << 63);
  return __longlong_as_double(
      (long long)(sign | (((unsigned long long)(e + 1022) << 52) + m)));
}
template <class Get, class Put>
__device__ __forceinline__ void scale_column(int ds, int s1, double diag, Get get, Put put) {
  const int lane = threadIdx.x & 31;
  const unsigned long long mb = significand(diag), w = fixed_reciprocal(mb);
  const bool inside = (unsigned)(exponent(diag) - (1023 - 400)) <= 800u;
  for (int q = ds + 1 + lane; q - lane < s1; q += 32) {
    const double a = q < s1 ? get(q) : 1.0;
    const bool zero = !bt::nonzero(a);
    const bool fast = inside && (zero || (unsigned)(exponent(a) - (1023 - 500)) <= 1000u);
    double v;
    if (__all_sync(FULL, fast)) {
      v = fixed_divide(a, diag, mb, w);
      if (zero)
        v = __longlong_as_double((__double_as_longlong(a) ^ __double_as_longlong(diag)) &
                                 (long long)(1ull << 63));
    } else {
      v = a / diag;
    }
    if (q < s1) put(q, v);
  }
}

// Pivot-pass mode of the refactorization (PivotCheck): the first
// factorization's threshold rule on column k's finished values - the first L
// slot of largest magnitude takes the pivot when it beats the diagonal and
// the diagonal is below tol times it - written to want[k]; then the
// candidate's row is swapped into the pivot. get(q) / put(q, v) access the
// column by slot.
template <class Get, class Put>
__device__ __forceinline__ void pivot_check(const PivotCheck& pc, int k, int ds, int s1,
                                            bool single, Get get, Put put) {
  const int lane = threadIdx.x & 31;
  double best = -1.0;
  int bq = 0x7fffffff;
  if (!single)
    for (int q = ds + 1 + lane; q < s1; q += 32) {
      const double v = fabs(get(q));
      if (v > best) {
        best = v;
        bq = q;
      }
    }
  for (int off = 16; off > 0; off >>= 1) {
    const double ov = __shfl_down_sync(FULL, best, off);
    const int oq = __shfl_down_sync(FULL, bq, off);
    if (ov > best || (ov == best && oq < bq)) {
      best = ov;
      bq = oq;
    }
  }
  if (lane == 0) {
    const double dabs = fabs(get(ds));
    pc.want[k] = (!single && bq != 0x7fffffff && best > dabs && dabs < pc.tol * best) ? bq : -1;
    const int c = pc.cand[k];
    if (c > ds && c < s1) {
      const double t = get(ds);
      put(ds, get(c));
      put(c, t);
    }
  }
  __syncwarp();
}

// The grid kernel: a pair of warps per column. The loader takes the columns in
// P.order and copies their pieces; the computing warp holds the column in shared
// memory (in `big` when it is longer than colcap) and does nothing but the
// arithmetic, so a piece costs it about 30 instructions and the latency of a
// multiply, a subtract and two trips to shared memory. Stage protocol: `full`
// counts the loader's 32 copy completions and its header, `empty` the computing
// warp; a stage marked last is released when its column is stored, and only
// then the loader takes another column, so the lowest unfinished column is
// always at work. The column counter lies behind the values, so one fill
// presets both: it starts at the largest unsigned. A wait that gives up ends the
// pair (`dead`) and sets the status, which ends the others.
//
// What bounds it: the chain of dependent columns, about 1 us a column (the last
// update 350 cycles, the reciprocal and the first 32 quotients 820, store to
// load through L2 900), and for the hub columns 800 cycles a piece. Measured
// against one warp per column, flags, one entry's loads ahead and FP64
// compares and divisions: 32 x 32 mesh (n 1026, 25 k slots) 353 -> 178 us,
// 48 x 48 740 -> 353 us, 120 x 120 with 1000 inverters (n 15,403, 670 k slots)
// 4.2 -> 1.6 ms.
constexpr int kStart = -1, kEnd = -2, kNone = -3;  // header.z of a stage that is no piece
constexpr int kLast = 1 << 24;  // in a piece's header.z
constexpr int kPairs = 4;       // per block

__device__ __forceinline__ void bar_init(unsigned b, int n) {
  asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned b) {
  asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(b) : "memory");
}
__device__ __forceinline__ void bar_arrive_copies(unsigned b) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(b) : "memory");
}
// Waits for the end of a barrier's phase; false when the pair has given up
// (dead, where there is one) or the wait runs out.
__device__ __forceinline__ bool bar_wait(unsigned b, unsigned parity, volatile int* dead,
                                         unsigned limit) {
  for (unsigned spins = 0;; ++spins) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(b), "r"(parity)
        : "memory");
    if (__all_sync(FULL, done)) return true;
    if (__any_sync(FULL, (dead != nullptr && *dead != 0) || spins >= limit)) return false;
    if (spins > 256) __nanosleep(100);
  }
}
// Ends the pair, and through the status the pairs that wait for its column.
__device__ __forceinline__ void give_up(volatile int* dead, int* status) {
  if ((threadIdx.x & 31) == 0) {
    *dead = 1;
    atomicCAS(status, DS_OK, DS_TIMEOUT);
  }
}

struct Stages {
  unsigned char* ring;
  unsigned bars;  // full[kGridRing], then empty[kGridRing]
  int st = 0;
  unsigned ph = 0;
  __device__ __forceinline__ unsigned char* at() const { return ring + st * kGridStage; }
  __device__ __forceinline__ unsigned full() const { return bars + 8 * st; }
  __device__ __forceinline__ unsigned empty() const { return bars + 8 * (kGridRing + st); }
  __device__ __forceinline__ void advance() {
    if (++st == kGridRing) {
      st = 0;
      ph ^= 1u;
    }
  }
};

// Returns false when a wait gave up.
__device__ __forceinline__ bool load_columns(const DPlan& P, const double* lu, unsigned* counter,
                                             Stages S, volatile int* dead) {
  const int lane = threadIdx.x & 31;
  auto publish = [&](int4 h) {  // after the stage's copies
    if (lane == 0) *reinterpret_cast<int4*>(S.at()) = h;
    bar_arrive_copies(S.full());
    if (lane == 0) bar_arrive(S.full());
  };
  while (true) {
    int k = 0;
    if (lane == 0) k = (int)(atomicAdd(counter, 1u) + 1u);
    k = __shfl_sync(FULL, k, 0);
    if (!bar_wait(S.empty(), S.ph ^ 1u, dead, P.pair_limit)) return false;
    if (k >= P.n) {
      publish(make_int4(0, 0, kEnd, 0));
      return true;
    }
    k = P.order[k];
    const int s0 = P.col_ptr[k], ds = P.dslot[k], s1 = P.col_ptr[k + 1];
    const int single = P.col_single[k];
    if (lane == 0) *reinterpret_cast<int4*>(S.at() + 16) = make_int4(s1, single, 0, 0);
    publish(make_int4(s0, ds, kStart, k));
    S.advance();
    Pieces todo(P, s0, ds);
    bool more = todo.more();
    do {
      if (!bar_wait(S.empty(), S.ph ^ 1u, dead, P.pair_limit)) return false;
      int4 h = make_int4(0, 0, kNone, 0);
      if (more) {
        h = todo.next(S.at(), lu);
        todo.skip_empty();
        more = todo.more();
        if (!more) h.z |= kLast;
      }
      publish(h);
      if (!more && !bar_wait(S.empty(), S.ph, dead, P.pair_limit)) return false;
      S.advance();
    } while (more);
  }
}

// The computing warp's updates of one column; S stands at its first piece.
// Leaves S at the column's last stage, not yet released.
template <bool kStaged>
__device__ __forceinline__ bool grid_updates(const DPlan& P, double* C, const double* lu,
                                             Stages& S, int* status, volatile int* dead) {
  const int lane = threadIdx.x & 31;
  auto at = [&](int s) { return kStaged ? C[s] : ld_cg(&C[s]); };
  Piece nx;
  auto read = [&]() {
    if (!bar_wait(S.full(), S.ph, dead, P.pair_limit)) return false;
    nx.read(S.at(), true);
    __syncwarp();
    if ((nx.h.z & kLast) == 0) {
      if (lane == 0) bar_arrive(S.empty());
      S.advance();
    }
    return true;
  };
  if (!read()) return false;
  if (nx.h.z < 0) return true;  // no updates
  while (true) {
    // all that does not depend on the values comes before the wait for them
    const Piece p = nx;
    const bool last = (p.h.z & kLast) != 0;
    double x0 = p.v0, x1 = p.v1;
    const double u = at(p.h.x);
    double c0 = 0.0, c1 = 0.0;
    if (p.a0) c0 = at(p.e0);
    if (p.two && p.a1) c1 = at(p.e1);
    if (!last && !read()) return false;
    bool w0 = p.a0 && unset(x0), w1 = p.a1 && unset(x1);
    unsigned spins = 0;
    while (__any_sync(FULL, w0 || w1)) {
      if (w0) {
        x0 = ld_relaxed(lu + p.h.y + lane);
        w0 = unset(x0);
      }
      if (w1) {
        x1 = ld_relaxed(lu + p.h.y + lane + 32);
        w1 = unset(x1);
      }
      ++spins;
      bool stop = spins > P.spin_limit && (w0 || w1);
      if (stop) atomicCAS(status, DS_OK, DS_TIMEOUT);
      if ((spins & 63u) == 0 && *(volatile int*)status != DS_OK) stop = true;
      if (__any_sync(FULL, stop)) return false;
      if (spins > 64) __nanosleep(64);  // a poll is a trip through L2
    }
    if (bt::nonzero(u)) {  // the same in every lane
      const double m0 = mul(x0, u);
      if (p.a0) C[p.e0] = sub(c0, m0);
      if (p.two) {
        const double m1 = mul(x1, u);
        if (p.a1) C[p.e1] = sub(c1, m1);
      }
    }
    __syncwarp();
    if (last) return true;
  }
}

__global__ void k_preset(double* lu, long long n, const int* skip) {
  if (__ldcg(skip) != 0) return;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
    lu[i] = __longlong_as_double(-1ll);
}

__global__ void __launch_bounds__(64 * kPairs) k_refactor(DPlan P, const double* __restrict__ ax,
                                                          double* lu, double* big, int colcap,
                                                          int* status, PivotCheck pc) {
  if (P.skip != nullptr && __ldcg(P.skip) != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[kPairs][2 * kGridRing];
  __shared__ int dead_flag[kPairs];
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % kPairs;
  const bool loader = (threadIdx.x >> 5) >= kPairs;
  volatile int* const dead = &dead_flag[w];
  double* const cbuf =
      reinterpret_cast<double*>(smem_raw + kPairs * kGridRing * kGridStage) + w * colcap;
  Stages S;
  S.ring = smem_raw + w * (kGridRing * kGridStage);
  S.bars = (unsigned)__cvta_generic_to_shared(&bars[w][0]);
  if (!loader && lane == 0) {
    for (int i = 0; i < kGridRing; ++i) {
      bar_init(S.bars + 8 * i, 33);
      bar_init(S.bars + 8 * (kGridRing + i), 1);
    }
    *dead = 0;
  }
  __syncthreads();
  if (loader) {
    if (!load_columns(P, lu, reinterpret_cast<unsigned*>(lu + P.nslots + 2), S, dead))
      give_up(dead, status);
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  while (true) {
    if (!bar_wait(S.full(), S.ph, dead, P.pair_limit)) {
      give_up(dead, status);
      return;
    }
    const int4 h = *reinterpret_cast<const int4*>(S.at());
    if (h.z == kEnd) return;
    const int4 h1 = *reinterpret_cast<const int4*>(S.at() + 16);
    const int s0 = h.x, ds = h.y, k = h.w, s1 = h1.x;
    const bool staged = s1 - s0 <= colcap, single = h1.y != 0;
    double* const C = staged ? cbuf - s0 : big;  // the column, indexed by slot
    __syncwarp();
    if (lane == 0) bar_arrive(S.empty());
    S.advance();
    // A(:,k) into the column's slots; duplicates summed in CSC order
    for (int s = s0 + lane; s < s1; s += 32) {
      double v = 0.0;
      for (int t = P.amap_ptr[s]; t < P.amap_ptr[s + 1]; ++t) v += ax[P.amap_idx[t]];
      C[s] = v;
    }
    __syncwarp();
    if (!(staged ? grid_updates<true>(P, cbuf - s0, lu, S, status, dead)
                 : grid_updates<false>(P, big, lu, S, status, dead))) {
      give_up(dead, status);
      return;
    }
    if (pc.want != nullptr)
      pivot_check(
          pc, k, ds, s1, single, [&](int q) { return staged ? C[q] : ld_cg(&C[q]); },
          [&](int q, double v) { C[q] = v; });
    const double diag = bt::perturb_bits(staged ? C[ds] : ld_cg(&C[ds]), single);
    scale_column(
        ds, s1, diag, [&](int q) { return staged ? C[q] : ld_cg(&C[q]); },
        [&](int q, double v) { st_set(&lu[q], v); });
    for (int q = s0 + lane; q < ds; q += 32) lu[q] = staged ? C[q] : ld_cg(&C[q]);
    if (lane == 0) lu[ds] = diag;
    __syncwarp();
    if (lane == 0) bar_arrive(S.empty());
    S.advance();
  }
}

// --------------------------------------------------------------- solve
// v - sum_e coef(e) * val(dep(e)) over e in [e0, e1), subtracted in order.
// Each lane waits for and multiplies one entry of a 32-entry chunk; lane 0
// then subtracts the rounded products in order.
template <class Coef, class Dep>
__device__ __forceinline__ bool ordered_dot(double& v, int e0, int e1, Coef coef, Dep dep,
                                            const unsigned* flag, const double* val,
                                            unsigned epoch, int* status, unsigned limit) {
  const int lane = threadIdx.x & 31;
  for (int base = e0; base < e1; base += 32) {
    const int e = base + lane;
    double prod = 0.0;
    int ok = 1;
    if (e < e1) {
      const int d = dep(e);
      ok = wait_flag(&flag[d], epoch, status, limit);
      if (ok) prod = coef(e) * ld_cg(&val[d]);
    }
    if (!__all_sync(FULL, ok)) return false;
    const int cnt = min(32, e1 - base);
    for (int t = 0; t < cnt; ++t) {
      double pt = __shfl_sync(FULL, prod, t);
      v = v - pt;
    }
  }
  return true;
}

__global__ void k_solve(DPlan P, const double* __restrict__ rhs, const double* __restrict__ ax,
                        const double* __restrict__ lu, double* z, double* x, double* out,
                        unsigned* zflag, unsigned* xflag, unsigned epoch, unsigned* counter,
                        int* status) {
  if (P.skip != nullptr && __ldcg(P.skip) != 0) return;
  const int lane = threadIdx.x & 31;
  while (true) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(counter, 1u);
    t = __shfl_sync(FULL, t, 0);
    if (t >= P.ntask) return;
    const int code = P.task[t];
    const int i = code >> 1;
    if ((code & 1) == 0) {  // forward: block coupling, then L
      double v = rhs[P.in_row[i]];
      bool ok = ordered_dot(
          v, P.offd_ptr[i], P.offd_ptr[i + 1], [&](int e) { return ax[P.offd_raw[e]]; },
          [&](int e) { return P.offd_col[e]; }, xflag, x, epoch, status, P.spin_limit);
      if (ok)
        ok = ordered_dot(
            v, P.lrow_ptr[i], P.lrow_ptr[i + 1], [&](int e) { return lu[P.lrow_slot[e]]; },
            [&](int e) { return P.lrow_col[e]; }, zflag, z, epoch, status, P.spin_limit);
      if (!ok) return;
      if (lane == 0) {
        z[i] = v;
        __threadfence();
        st_release(&zflag[i], epoch);
      }
    } else {  // backward: U
      int ok = 1;
      if (lane == 0) ok = wait_flag(&zflag[i], epoch, status, P.spin_limit);
      if (!__shfl_sync(FULL, ok, 0)) return;
      double v = ld_cg(&z[i]);
      ok = ordered_dot(
          v, P.urow_ptr[i], P.urow_ptr[i + 1], [&](int e) { return lu[P.urow_slot[e]]; },
          [&](int e) { return P.urow_col[e]; }, xflag, x, epoch, status, P.spin_limit);
      if (!ok) return;
      if (lane == 0) {
        v = v / lu[P.dslot[i]];
        x[i] = v;
        out[P.out_col[i]] = v;
        __threadfence();
        st_release(&xflag[i], epoch);
      }
    }
  }
}

// A^T y = g with the same factors: U^T forward (U columns as rows), then
// L^T backward (L columns as rows). Task codes as in k_solve; the input is
// indexed by original column and the output by original row.
__global__ void k_tsolve(DPlan P, const double* __restrict__ g, const double* __restrict__ ax,
                         const double* __restrict__ lu, double* z, double* x, double* out,
                         unsigned* zflag, unsigned* xflag, unsigned epoch, unsigned* counter,
                         int* status) {
  const int lane = threadIdx.x & 31;
  while (true) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(counter, 1u);
    t = __shfl_sync(FULL, t, 0);
    if (t >= P.ntask) return;
    const int code = P.task[t];
    const int k = code >> 1;
    if ((code & 1) == 0) {  // coupling^T, then U^T row k = U column k
      double v = g[P.out_col[k]];
      bool ok = ordered_dot(
          v, P.offdT_ptr[k], P.offdT_ptr[k + 1], [&](int e) { return ax[P.offdT_raw[e]]; },
          [&](int e) { return P.offdT_row[e]; }, xflag, x, epoch, status, P.spin_limit);
      if (ok)
        ok = ordered_dot(
            v, P.col_ptr[k], P.dslot[k], [&](int e) { return lu[e]; },
            [&](int e) { return P.slot_row[e]; }, zflag, z, epoch, status, P.spin_limit);
      if (!ok) return;
      if (lane == 0) {
        v = v / lu[P.dslot[k]];
        z[k] = v;
        __threadfence();
        st_release(&zflag[k], epoch);
      }
    } else {  // L^T row k = L column k
      int ok = 1;
      if (lane == 0) ok = wait_flag(&zflag[k], epoch, status, P.spin_limit);
      if (!__shfl_sync(FULL, ok, 0)) return;
      double v = ld_cg(&z[k]);
      ok = ordered_dot(
          v, P.dslot[k] + 1, P.col_ptr[k + 1], [&](int e) { return lu[e]; },
          [&](int e) { return P.slot_row[e]; }, xflag, x, epoch, status, P.spin_limit);
      if (!ok) return;
      if (lane == 0) {
        x[k] = v;
        out[P.in_row[k]] = v;
        __threadfence();
        st_release(&xflag[k], epoch);
      }
    }
  }
}

// --------------------------------------------------------------- one-block factor and solve
// For factorizations small enough that one SM does their arithmetic faster
// than the dependency hops of the grid-wide kernels cost, the refactor and
// the solve run in one thread block, where a hop is a shared-memory flag (or
// a warp barrier) instead of a round trip through L2.

// k_refactor in one block, with the factor itself in shared memory: the
// column code is k_refactor's (same operations, same order); completion flags
// live in shared memory, so a warp waiting for a column sees it finish within
// a few hundred cycles. All warps of the block are resident and a warp only
// waits for columns handed out before its own, so the warp holding the lowest
// unfinished column always proceeds. Shared: lu[nslots] f64, the warps' rings,
// done[n] u32.
__global__ void __launch_bounds__(1024) k_refactor_cta(DPlan P, const double* __restrict__ ax,
                                                       double* lu_out, int* status,
                                                       PivotCheck pc) {
  if (P.skip != nullptr && __ldcg(P.skip) != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* const lu = reinterpret_cast<double*>(smem_raw);
  unsigned char* const rings = smem_raw + (((size_t)8 * P.nslots + 15) & ~(size_t)15);
  unsigned* const sdone = reinterpret_cast<unsigned*>(rings + (blockDim.x >> 5) * (kCtaRing * kCtaStage));
  unsigned char* const ring = rings + (threadIdx.x >> 5) * (kCtaRing * kCtaStage);
  __shared__ unsigned snext;
  const int lane = threadIdx.x & 31;
  const int n = P.n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sdone[i] = 0u;
  if (threadIdx.x == 0) snext = 0u;
  __syncthreads();
  while (true) {
    int k = 0;
    if (lane == 0) k = (int)atomicAdd(&snext, 1u);
    k = __shfl_sync(FULL, k, 0);
    if (k >= n) break;
    const int s0 = P.col_ptr[k], ds = P.dslot[k], s1 = P.col_ptr[k + 1];
    const bool single = P.col_single[k] != 0;
    for (int s = s0 + lane; s < s1; s += 32) {
      double v = 0.0;
      for (int t = P.amap_ptr[s]; t < P.amap_ptr[s + 1]; ++t) v += ax[P.amap_idx[t]];
      lu[s] = v;
    }
    __syncwarp();
    if (!block_updates(P, s0, ds, lu, sdone, ring, status)) break;
    if (pc.want != nullptr)
      pivot_check(
          pc, k, ds, s1, single, [&](int q) { return lu[q]; },
          [&](int q, double v) { lu[q] = v; });
    const double diag = bt::perturb_bits(lu[ds], single);
    scale_column(
        ds, s1, diag, [&](int q) { return lu[q]; }, [&](int q, double v) { lu[q] = v; });
    __syncwarp();
    if (lane == 0) lu[ds] = diag;
    __syncwarp();
    if (lane == 0) st_release_cta(&sdone[k], 1u);
  }
  __syncthreads();
  for (int s = threadIdx.x; s < P.nslots; s += blockDim.x) lu_out[s] = lu[s];
}

// The solve of k_solve in one block, column by column: the forward sweep
// takes the L columns in ascending order and subtracts l(r,j) x(j) from each
// row r below, the backward sweep the U columns in descending order, so every
// row receives its terms in the order of its row lists (L ascending, U
// descending) - the reference's order - and the results are those of k_solve
// bit for bit. The block coupling of a BTF block is subtracted, row by row in
// its list order, before the block's first column.
//
// Warp 0 does the arithmetic; the other warps copy the factor's slots (rows
// and values) chunk by chunk into a double buffer ahead of it. The host cuts
// the sweeps into chunks of contiguous slots (CtaSolve in capi.cu):
//   chunk c: cs_chunk[4c..4c+3] = slot_lo, slot_hi, op_lo, op_hi
//   op o:    cs_op[3o..3o+2]    = kind | direct << 2, a, b
// kind 0: coupling of rows [a, b); 1: forward over columns [a, b); 2:
// backward over columns [a, b); direct: a column larger than a chunk, read
// from memory. Shared: w[n] f64, 2 x chunk values f64, then (i32) 2 x chunk
// rows, col_ptr[n+1], dslot[n], offd_ptr[n+1] (when there is coupling).
//
// With grouped != 0 the block is one of P.cs_ngrp: it solves rows [r0, r1)
// (whole uncoupled BTF blocks) with its own chunk range; the shared arrays
// then cover only those rows and are indexed by position - r0.
__global__ void __launch_bounds__(256) k_solve_cta(DPlan P, const double* __restrict__ rhs,
                                                   const double* __restrict__ ax,
                                                   const double* __restrict__ lu, double* out,
                                                   int chunk, int grouped) {
  if (P.skip != nullptr && __ldcg(P.skip) != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31;
  int r0 = 0, r1 = P.n, c0 = 0, c1 = P.cs_nchunk;
  const int *CH = P.cs_chunk, *OP = P.cs_op;
  if (grouped) {
    const int* g = P.cs_grp + 4 * blockIdx.x;
    r0 = g[0];
    r1 = g[1];
    c0 = g[2];
    c1 = g[3];
    CH = P.cs_gchunk;
    OP = P.cs_gop;
  }
  const int m = r1 - r0;
  const bool coupled = P.noffd > 0;
  double* const w = reinterpret_cast<double*>(smem_raw);
  double* const bval = w + m;
  int* const brow = reinterpret_cast<int*>(bval + 2 * chunk);
  int* const scp = brow + 2 * chunk;
  int* const sds = scp + m + 1;
  int* const sop = sds + m;
  for (int i = tid; i <= m; i += blockDim.x) {
    cp_async4(&scp[i], &P.col_ptr[r0 + i]);
    if (i < m) cp_async4(&sds[i], &P.dslot[r0 + i]);
    if (coupled) cp_async4(&sop[i], &P.offd_ptr[r0 + i]);
  }
  for (int i = tid; i < m; i += blockDim.x) w[i] = rhs[P.in_row[r0 + i]];
  cp_async_wait_all();
  const int nprod = blockDim.x - 32;
  auto load = [&](int c) {
    const int lo = CH[4 * c], hi = CH[4 * c + 1];
    double* const bv = bval + (c & 1) * chunk;
    int* const br = brow + (c & 1) * chunk;
    for (int s = lo + tid - 32; s < hi; s += nprod) {  // all copies in flight at once
      cp_async8(&bv[s - lo], &lu[s]);
      cp_async4(&br[s - lo], &P.slot_row[s]);
    }
    cp_async_wait_all();
  };
  if (tid >= 32 && c1 > c0) load(c0);
  __syncthreads();
  for (int c = c0; c < c1; ++c) {
    if (tid >= 32) {
      if (c + 1 < c1) load(c + 1);
    } else {
      const int lo = CH[4 * c], o0 = CH[4 * c + 2], o1 = CH[4 * c + 3];
      const double* const bv = bval + (c & 1) * chunk - lo;  // indexed by slot
      const int* const br = brow + (c & 1) * chunk - lo;
      for (int o = o0; o < o1; ++o) {
        const int code = OP[3 * o], a = OP[3 * o + 1] - r0, b = OP[3 * o + 2] - r0;
        // forward: L columns ascending. The next column's range is read, and
        // this column's first rows and values are loaded, before the value
        // of x(j) is: only the subtraction waits for the previous column.
        auto fwd = [&](const auto* V, const auto* R) {
          int q0 = sds[a] + 1, q1 = scp[a + 1];
          for (int j = a; j < b; ++j) {
            const int cq0 = q0, cq1 = q1;
            if (j + 1 < b) {
              q0 = sds[j + 1] + 1;
              q1 = scp[j + 2];
            }
            const int q = cq0 + lane;
            int r = 0;
            double v = 0.0;
            if (q < cq1) {
              r = R[q] - r0;
              v = V[q];
            }
            const double xj = w[j];
            if (q < cq1) w[r] = w[r] - v * xj;
            for (int qq = q + 32; qq < cq1; qq += 32) {
              const int rr = R[qq] - r0;
              w[rr] = w[rr] - V[qq] * xj;
            }
            __syncwarp();
          }
        };
        // backward: U columns descending
        auto bwd = [&](const auto* V, const auto* R) {
          for (int j = b - 1; j >= a; --j) {
            const int ds = sds[j], q = scp[j] + lane;
            int r = 0;
            double v = 0.0;
            if (q < ds) {
              r = R[q] - r0;
              v = V[q];
            }
            const double xj = w[j] / V[ds];
            if (q < ds) w[r] = w[r] - v * xj;
            for (int qq = q + 32; qq < ds; qq += 32) {
              const int rr = R[qq] - r0;
              w[rr] = w[rr] - V[qq] * xj;
            }
            __syncwarp();
            if (lane == 0) w[j] = xj;
          }
        };
        // separate instantiations keep the buffered sweeps on shared-memory
        // loads (a pointer that may be either space would make them generic)
        if ((code & 3) == 0) {  // coupling to the blocks solved before
          for (int i = a + lane; i < b; i += 32) {
            double v = w[i];
            for (int e = sop[i]; e < sop[i + 1]; ++e)
              v = v - ax[P.offd_raw[e]] * w[P.offd_col[e] - r0];
            w[i] = v;
          }
        } else if ((code & 3) == 1) {
          if (code & 4)
            fwd(lu, P.slot_row);
          else
            fwd(bv, br);
        } else {
          if (code & 4)
            bwd(lu, P.slot_row);
          else
            bwd(bv, br);
        }
        __syncwarp();
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < m; i += blockDim.x) out[P.out_col[r0 + i]] = w[i];
}

// The solve as a step program, one thread block, the solution vector in
// shared memory. The pivots' reciprocals come first (n divisions in
// parallel); then four compute warps run the rows - the operations the column
// sweeps perform, in the reference's order for every row of the system (each
// update a separately rounded product and difference, the pivot division
// exact), one per thread - while eight loader warps fetch the next chunk's
// operations and matrix values into the other half of a shared double
// buffer.
//
// Both kinds of operation are one formula: p = v T[s], r = c p + T[d] in one
// rounding, with v the matrix value and c = -1 for an update (r = T[d] - p).
// A division a / b is Markstein's correction (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990) from the correctly rounded reciprocal y = 1/b: with s = d,
// v = y and c = -b, p is within an ulp of a / b, r = a - b p is exact and
// r y + p is the correctly rounded quotient; only rows with a division spend
// that third operation. Operands or a quotient near the ends of the exponent
// range (zeros, subnormals, infinities, NaN included) take the division
// itself; the tests are integer operations on the exponents of a, b and y
// (the quotient's is the sum of a's and y's, or one more), so none waits for
// an FP64 result.
//
// A step costs its latency: a shared load, two dependent FP64 operations (64
// cycles each, and 50 more until anything but an FP64 operation sees the
// result), a shared store and, when more than one warp is at it, the
// barrier. Compute warps that fetch from global memory themselves, however
// far ahead, take 430 to 620 cycles a step (a warp's few scoreboards are
// shared by the loads in flight and the FP64 results), hence the loader
// warps; with 128 loader threads the loads set the pace, 256 to 896 take the
// same time. Measured against one set of 128 threads that loads two steps
// ahead and no chains, per solve: 32x32 diode mesh 274 -> 119 us, 48x48 589 ->
// 235 us, 120x120 mesh with 1000 inverters 8.26 -> 1.97 ms; its transpose
// solve, a grid kernel before, 19.4 -> 1.97 ms.
constexpr int kSolveLoaders = 256, kLoadBatch = 4;
constexpr int kSolveStepsThreads = kSolveRow + kSolveLoaders;
// flags in a slot's destination address (a multiple of 8 otherwise)
constexpr unsigned kSlotDivRow = 1u, kSlotLast = 2u, kSlotDiv = 4u;
constexpr unsigned kSlotSlow = 1u;  // in its source address

__device__ __forceinline__ double lds_f64(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_f64(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ unsigned exponent_of(double a) {
  return (unsigned)(__double2hiint(a) >> 20) & 0x7ffu;
}

// The slots of a large program as the rows read them (values and factor; the
// addresses, from the solution's base, of destination and source with their
// flags), laid out by the whole grid ahead of the solve.
__global__ void k_solve_slots(SolveSched S, int n, const double* __restrict__ ax,
                              const double* __restrict__ lu, const int* skip) {
  if (skip != nullptr && __ldcg(skip) != 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.nslots) return;
  const int4 o = __ldg(S.ops + i);
  const int kind = o.w & 3;
  const bool div = kind == 1, none = kind == 3;
  const double m = none ? 0.0 : (kind == 2 ? ax : lu)[o.z], y = div ? 1.0 / m : 0.0;
  const bool slow = div && (exponent_of(m) - 64u > 1919u || exponent_of(y) - 64u > 1919u);
  S.vc[i] = make_double2(div ? y : m, div ? -m : (none ? 0.0 : -1.0));
  S.ad[i] =
      make_uint2(8u * (unsigned)(none ? n : o.x) | (unsigned)(o.w >> 2) | (div ? kSlotDiv : 0u),
                 8u * (unsigned)(none ? n : o.y) | (slow ? kSlotSlow : 0u));
}

// n bytes (a multiple of 16) from memory to shared memory, counted by barrier b.
__device__ __forceinline__ void bulk_copy(unsigned d, const void* g, unsigned n, unsigned b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          d),
      "l"(g), "r"(n), "r"(b)
      : "memory");
}

// Whether `ok` holds in all four compute warps (their barrier, as bar.sync 1).
__device__ __forceinline__ bool all_rows(bool ok) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1u : 0u)
      : "memory");
  return r != 0;
}

// kStaged (programs of kSolveStaged slots or more): the slots come ready from
// k_solve_slots, a chunk in two bulk copies by one warp, and the loads of eight
// loader warps no longer share the SM's load unit with the rows (measured at
// kSolveStaged). A wait for a chunk that runs out ends the solve (DS_TIMEOUT): the
// compute warps agree on it, as one that left alone would be missing at the
// others' barriers, and the copying warp stays until its last copies have landed.
template <bool kStaged>
__global__ void __launch_bounds__(kStaged ? kSolveRow + 32 : kSolveStepsThreads)
    k_solve_steps(SolveSched S, int n, const int* __restrict__ in, const int* __restrict__ outp,
                  const int* __restrict__ dslot, const double* __restrict__ rhs,
                  const double* __restrict__ ax, const double* __restrict__ lu, double* rec,
                  double* out, const int* skip, int* status, unsigned pair_limit) {
  if (skip != nullptr && __ldcg(skip) != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* const T = reinterpret_cast<double*>(smem_raw);  // the solution, a spare entry at n
  double2* const svc = reinterpret_cast<double2*>(T + ((n + 2) & ~1));  // (v, c) of every slot
  uint2* const sad = reinterpret_cast<uint2*>(svc + 2 * S.chunk);  // destination, source address
  int2* const sseg = reinterpret_cast<int2*>(sad + 2 * S.chunk);   // segments, an end mark
  const unsigned T0 = (unsigned)__cvta_generic_to_shared(T);
  const int tid = threadIdx.x, lane = tid & 31;
  __shared__ __align__(8) unsigned long long bars[4];  // a half is full, 2: is free
  __shared__ int dead_flag;
  volatile int* const dead = &dead_flag;
  const unsigned bar0 = (unsigned)__cvta_generic_to_shared(bars);
  const unsigned A0 = kStaged ? T0 : 0u;  // what the slots' addresses count from
  for (int i = tid; i < n; i += blockDim.x) {
    T[i] = rhs[in[i]];
    if (!kStaged) rec[i] = 1.0 / lu[dslot[i]];
  }
  if (tid == 0) {
    T[n] = 0.0;
    if (kStaged) {
      for (int i = 0; i < 4; ++i) bar_init(bar0 + 8 * i, i < 2 ? 1 : kSolveRow / 32);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      *dead = 0;
    }
  }
  __syncthreads();
  // chunk c into its half of the buffer, by the threads from tid0 on:
  // kLoadBatch operations' loads in flight together, then their values'
  auto load = [&](int c, int tid0) {
    const int4 C = __ldg(S.chunks + c);
    const int h = (c & 1) * S.chunk, hs = (c & 1) * (kSolveSegs + 1), nt = blockDim.x - tid0;
    for (int i = tid - tid0; i <= C.w; i += nt)
      sseg[hs + i] = i < C.w ? __ldg(S.segs + C.z + i) : make_int2(3, -1);
    for (int i0 = tid - tid0; i0 < C.y; i0 += kLoadBatch * nt) {
      int4 o[kLoadBatch];
      double m[kLoadBatch], y[kLoadBatch];
#pragma unroll
      for (int u = 0; u < kLoadBatch; ++u)
        o[u] = i0 + u * nt < C.y ? __ldg(S.ops + C.x + i0 + u * nt) : make_int4(0, 0, 0, 3);
#pragma unroll
      for (int u = 0; u < kLoadBatch; ++u) {
        const int kind = o[u].w & 3;
        m[u] = kind != 3 ? __ldg((kind == 2 ? ax : lu) + o[u].z) : 0.0;
        y[u] = kind == 1 ? __ldcg(rec + o[u].x) : 0.0;  // written above by this block
      }
#pragma unroll
      for (int u = 0; u < kLoadBatch; ++u) {
        const int i = i0 + u * nt, kind = o[u].w & 3;
        if (i >= C.y) break;
        const bool div = kind == 1, none = kind == 3;
        const bool slow =
            div && (exponent_of(m[u]) - 64u > 1919u || exponent_of(y[u]) - 64u > 1919u);
        svc[h + i] = make_double2(div ? y[u] : m[u], div ? -m[u] : (none ? 0.0 : -1.0));
        sad[h + i] =
            make_uint2((T0 + 8u * (unsigned)(none ? n : o[u].x)) | (unsigned)(o[u].w >> 2) |
                           (div ? kSlotDiv : 0u),
                       (T0 + 8u * (unsigned)(none ? n : o[u].y)) | (slow ? kSlotSlow : 0u));
      }
    }
  };
  // one chain: 32 products, then their differences in order (every lane
  // computes them); terms fetched two chunks ahead, values one
  auto run_chain = [&](int4 o) {
    const int2 nt = make_int2(0, 0);
    const int2* const tp = S.terms + o.y;
    auto value = [&](int z) { return __ldg(z < 0 ? ax + ~z : lu + z); };
    double v = T[o.x];
    int2 t0 = lane < o.z ? __ldg(tp + lane) : nt;
    int2 t1 = lane + 32 < o.z ? __ldg(tp + lane + 32) : nt;
    double c0 = lane < o.z ? value(t0.y) : 0.0;
    for (int b = 0; b < o.z; b += 32) {
      const double c1 = b + 32 + lane < o.z ? value(t1.y) : 0.0;
      const int2 t2 = b + 64 + lane < o.z ? __ldg(tp + b + 64 + lane) : nt;
      const double p = __dmul_rn(c0, T[t0.x]);
      const int cnt = min(32, o.z - b);
      if (cnt == 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v = __dsub_rn(v, __shfl_sync(FULL, p, i));
      } else {
        for (int i = 0; i < cnt; ++i) v = __dsub_rn(v, __shfl_sync(FULL, p, i));
      }
      t0 = t1;
      t1 = t2;
      c0 = c1;
    }
    if (lane == 0) T[o.x] = v;
  };
  // one slot's operation
  auto exec = [&](uint2 a, double2 vc) {
    const unsigned da = A0 + (a.x & ~7u);
    const double td = lds_f64(da), ts = lds_f64(A0 + (a.y & ~7u));
    const double p = vc.x * ts;
    double r = fma(vc.y, p, td);
    if (a.x & kSlotDivRow) {
      const double q = fma(r, vc.x, p);
      if (a.x & kSlotDiv) {
        const unsigned ea = exponent_of(td);
        r = q;
        if ((a.y & kSlotSlow) || ea - 64u > 1919u || ea + exponent_of(vc.x) - 1088u > 1917u)
          r = td / -vc.y;
      }
    }
    sts_f64(da, r);
  };
  if (!kStaged && S.nchunks > 0) load(0, 0);
  __syncthreads();
  if (kStaged && tid >= kSolveRow) {  // the copying warp
    const int2 end = make_int2(3, -1);
    int c = 0;  // chunks issued
    for (; c < S.nchunks; ++c) {
      const int h = c & 1;
      const int4 C = __ldg(S.chunks + c);
      const int2 s0 = lane < C.w ? __ldg(S.segs + C.z + lane) : end;
      const int2 s1 = lane + 32 < C.w ? __ldg(S.segs + C.z + lane + 32) : end;
      if (!bar_wait(bar0 + 8 * (2 + h), (c >> 1 & 1) ^ 1u, dead, pair_limit)) {
        give_up(dead, status);
        break;
      }
      int2* const sg = sseg + h * (kSolveSegs + 1);
      sg[lane] = s0;
      sg[lane + 32] = s1;
      if (lane == 0) sg[64] = end;
      __syncwarp();
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(bar0 + 8 * h),
                     "r"(24 * C.y)
                     : "memory");
        if (C.y > 0) {
          bulk_copy((unsigned)__cvta_generic_to_shared(svc + h * S.chunk), S.vc + C.x, 16 * C.y,
                    bar0 + 8 * h);
          bulk_copy((unsigned)__cvta_generic_to_shared(sad + h * S.chunk), S.ad + C.x, 8 * C.y,
                    bar0 + 8 * h);
        }
      }
      __syncwarp();
    }
    for (int q = max(c - 2, 0); q < c; ++q)  // the last copy into either half
      bar_wait(bar0 + 8 * (q & 1), q >> 1 & 1, nullptr, 8 * kSpinLimit);
  }
  for (int c = 0; c < S.nchunks; ++c) {
    if (kStaged) {
      if (tid >= kSolveRow) break;
      if (!all_rows(bar_wait(bar0 + 8 * (c & 1), c >> 1 & 1, dead, pair_limit))) {
        give_up(dead, status);
        break;
      }
    }
    if (!kStaged && tid >= kSolveRow) {
      if (c + 1 < S.nchunks) load(c + 1, kSolveRow);
    } else {
      const int2* seg = sseg + (c & 1) * (kSolveSegs + 1);
      int base = (c & 1) * S.chunk;
      int2 next = *seg;
      while ((next.x & 3) != 3) {
        const int2 g = next;
        next = *++seg;
        const int kind = g.x & 3, cnt = g.x >> 2;
        if (kind == kSolveSegSolo) {
          // two register sets, each slot's operands read a row ahead
          if (tid < 32) {
            const uint2* pa = sad + base + lane;
            const double2* pv = svc + base + lane;
            uint2 a0 = pa[0], a1 = a0;
            double2 v0 = pv[0], v1 = v0;
            int q = 0;
            for (; q + 2 <= cnt; q += 2) {
              a1 = pa[32];
              v1 = pv[32];
              exec(a0, v0);
              __syncwarp();
              pa += 64;
              pv += 64;
              if (q + 2 < cnt) {
                a0 = pa[0];
                v0 = pv[0];
              }
              exec(a1, v1);
              __syncwarp();
            }
            if (q < cnt) exec(a0, v0);
          }
          base += 32 * cnt;
          asm volatile("bar.sync 1, 128;" ::: "memory");
        } else if (kind == kSolveSegWide) {
          const bool on = tid < S.width;
          const uint2* pa = sad + base + (on ? tid : 0);
          const double2* pv = svc + base + (on ? tid : 0);
          uint2 a0 = pa[0], a1 = a0;
          double2 v0 = pv[0], v1 = v0;
          for (int q = 0; q < cnt; ++q) {
            pa += S.width;
            pv += S.width;
            if (q + 1 < cnt) {
              a1 = *pa;
              v1 = *pv;
            }
            if (on) exec(a0, v0);
            if (a0.x & kSlotLast) asm volatile("bar.sync 1, 128;" ::: "memory");
            a0 = a1;
            v0 = v1;
          }
          base += S.width * cnt;
        } else {
          for (int m = tid >> 5; m < cnt; m += kSolveRow >> 5) run_chain(__ldg(S.chains + g.y + m));
          asm volatile("bar.sync 1, 128;" ::: "memory");
        }
      }
    }
    if (kStaged) {  // the half is free (the rows ordered themselves where it matters)
      __syncwarp();
      if (lane == 0) bar_arrive(bar0 + 8 * (2 + (c & 1)));
    } else {
      __syncthreads();
    }
  }
  if (kStaged) __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) out[outp[i]] = T[i];
}

// The step program of a solution that fills the shared memory: each thread
// reads its operation, its matrix value and (for a division) its reciprocal
// from memory two steps ahead, none of which depends on the solution; a barrier
// a step. The quotients are k_solve_steps' (Markstein). 430 to 620 cycles a step.
constexpr int kSolveListThreads = 128;

__device__ __forceinline__ double div_markstein(double a, double b, double y) {
  const double q = a * y;
  if (exponent_of(a) - 64u > 1919u || exponent_of(b) - 64u > 1919u || exponent_of(q) - 64u > 1919u)
    return a / b;
  const double r = fma(-b, q, a);
  return fma(r, y, q);
}

struct ListOp {
  int4 o;
  double v, y;
};

__global__ void __launch_bounds__(kSolveListThreads)
    k_solve_list(SolveSched S, int n, const int* __restrict__ in, const int* __restrict__ outp,
                 const int* __restrict__ dslot, const double* __restrict__ rhs,
                 const double* __restrict__ ax, const double* __restrict__ lu, double* rec,
                 double* out, const int* skip) {
  if (skip != nullptr && __ldcg(skip) != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* const T = reinterpret_cast<double*>(smem_raw);
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += blockDim.x) {
    T[i] = rhs[in[i]];
    rec[i] = 1.0 / lu[dslot[i]];
  }
  __syncthreads();
  const int* const sp = S.ptr;
  const int ns = S.nsteps, nops = sp[ns];
  auto fetch = [&](int p) {
    ListOp f{make_int4(0, -1, 0, 3), 0.0, 0.0};
    if (p < nops) {
      f.o = __ldg(S.list + p);
      f.v = f.o.w == 2 ? __ldg(ax + f.o.z) : __ldg(lu + f.o.z);
      if (f.o.w == 1) f.y = __ldcg(rec + f.o.x);  // written above by this block
    }
    return f;
  };
  auto exec = [&](const ListOp& f) {
    const int d = f.o.x;
    if (f.o.w == 1)
      T[d] = div_markstein(T[d], f.v, f.y);
    else if (f.o.w != 3)
      T[d] = __dsub_rn(T[d], __dmul_rn(f.v, T[f.o.y]));
  };
  int s0 = sp[0], s1 = sp[min(1, ns)], s2 = sp[min(2, ns)], s3 = sp[min(3, ns)];
  ListOp f0 = fetch(s0 + tid), f1 = fetch(s1 + tid);
  for (int t = 0; t < ns; ++t) {
    const ListOp f2 = fetch(s2 + tid);
    const int s4 = sp[min(t + 4, ns)];
    if (s0 + tid < s1) exec(f0);
    for (int p = s0 + tid + kSolveListThreads; p < s1; p += kSolveListThreads) exec(fetch(p));
    __syncthreads();
    s0 = s1;
    s1 = s2;
    s2 = s3;
    s3 = s4;
    f0 = f1;
    f1 = f2;
  }
  for (int i = tid; i < n; i += blockDim.x) out[outp[i]] = T[i];
}

// --------------------------------------------------------------- devices
// Level-1 MOSFET exactly as the reference evaluates it
// (crates/sim-devices/src/bsim/evaluate.rs:285-356 via mod.rs:440-455).
__device__ void mos_reference(const double* p, double vd, double vg, double vs, double& gm,
                              double& gds, double& ieq) {
  const double lambda = 0.02, gmin_dev = 1e-12;
  const bool pm = p[0] != 0.0;
  const double beta = p[2] * 1e-4 * ((3.9 * 8.854e-12) / p[3]);
  double vdi = pm ? -vs : vd, vgi = pm ? -vg : vg, vsi = pm ? -vd : vs;
  double vgs = vgi - vsi, vds = vdi - vsi;
  if (vds < 0.0) {
    vds = -vds;
    vgs = vgi - vdi;
  }
  const double vth = pm ? -fabs(p[1]) : fabs(p[1]);
  const double beff = beta * p[4] / p[5];
  double ids;
  if (vgs <= vth) {
    ids = 0.0;
    gm = 0.0;
    gds = gmin_dev;
  } else if (vds < vgs - vth) {
    ids = beff * ((vgs - vth) * vds - 0.5 * vds * vds);
    gm = beff * vds;
    gds = fmax(beff * ((vgs - vth) - vds), gmin_dev);
  } else {
    const double t = vgs - vth;
    ids = 0.5 * beff * (t * t) * (1.0 + lambda * vds);
    gm = beff * (vgs - vth) * (1.0 + lambda * vds);
    gds = fmax(0.5 * beff * (t * t) * lambda, gmin_dev);
  }
  const double ids_s = pm ? -ids : ids;
  ieq = ids_s - gm * (vg - vs) - gds * (vd - vs);
}

// Level-1 MOSFET in the Shichman-Hodges form (the (1 + lambda vds) factor in
// both regions, so the current is continuous where they meet) with a
// self-consistent linearisation: drain current and its partials with respect
// to (vg, vd, vs).
__device__ void mos_consistent(const double* p, double vd, double vg, double vs, double& id,
                               double& ddg, double& ddd, double& dds, double gmin_dev) {
  const double lambda = 0.02;
  const double pol = p[0] != 0.0 ? -1.0 : 1.0;
  const double beta = p[2] * 1e-4 * ((3.9 * 8.854e-12) / p[3]);
  const double vgs = pol * (vg - vs), vds = pol * (vd - vs);
  const bool rev = vds < 0.0;
  const double vgse = rev ? vgs - vds : vgs, vdse = rev ? -vds : vds;
  const double vth = fabs(p[1]);
  const double beff = beta * p[4] / p[5];
  double ids, gm, gds;
  if (vgse <= vth) {
    ids = 0.0;
    gm = 0.0;
    gds = gmin_dev;
  } else if (vdse < vgse - vth) {  // Shichman-Hodges: (1 + lambda vds) here too
    const double k = 1.0 + lambda * vdse;
    const double q = (vgse - vth) * vdse - 0.5 * vdse * vdse;
    ids = beff * q * k;
    gm = beff * vdse * k;
    gds = fmax(beff * ((vgse - vth) - vdse) * k + lambda * beff * q, gmin_dev);
  } else {
    const double t = vgse - vth;
    ids = 0.5 * beff * (t * t) * (1.0 + lambda * vdse);
    gm = beff * (vgse - vth) * (1.0 + lambda * vdse);
    gds = fmax(0.5 * beff * (t * t) * lambda, gmin_dev);
  }
  if (!rev) {
    id = pol * ids;
    ddg = gm;
    ddd = gds;
    dds = -(gm + gds);
  } else {
    id = -pol * ids;
    ddg = -gm;
    ddd = gm + gds;
    dds = -gds;
  }
}

// One device's matrix inserts (in the reference's insert order) and its
// right-hand-side contributions. Returns the number of matrix values.
// gdev is the level-1 conductance floor of the consistent model: 1e-12 as
// the reference's evaluator uses, or 0 for the exact Jacobian of the
// residual (the floor cancels in the residual but not in the matrix).
template <class XGet>
__device__ __forceinline__ int eval_device(int type, const int* nd, const double* p, XGet xg,
                                           double gmin, double scale, double dt, double vprev,
                                           double be_sign, double* m, double* r, int& nr,
                                           double gdev = 1e-12) {
  nr = 0;
  switch (type) {
    case 0: {  // R
      const double g = 1.0 / p[0];
      m[0] = g;
      m[1] = g;
      m[2] = -g;
      m[3] = -g;
      return 4;
    }
    case 1: {  // V
      m[0] = 1.0;
      m[1] = -1.0;
      m[2] = 1.0;
      m[3] = -1.0;
      r[0] = p[0] * scale;
      nr = 1;
      return 4;
    }
    case 2: {  // I
      const double v = p[0] * scale;
      r[0] = -v;
      r[1] = v;
      nr = 2;
      return 0;
    }
    case 3: {  // D, crates/sim-core/src/stamp.rs:351-387
      const double gf = gmin > 0.0 ? gmin : 1e-12;
      const double vt = 0.02585 * p[1];
      const double vd = xg(nd[0]) - xg(nd[1]);
      const double e = exp(vd / vt);
      const double id = p[0] * (e - 1.0);
      const double gd = (p[0] / vt) * e;
      const double g = fmax(gd, gf);
      const double ieq = id - gd * vd;
      m[0] = g;
      m[1] = g;
      m[2] = -g;
      m[3] = -g;
      r[0] = -ieq;
      r[1] = ieq;
      nr = 2;
      return 4;
    }
    case 4: {  // M, crates/sim-core/src/stamp.rs:511-545
      const double gf = gmin > 0.0 ? gmin : 1e-12;
      double gm, gds, ieq;
      mos_reference(p, xg(nd[0]), xg(nd[1]), xg(nd[2]), gm, gds, ieq);
      gds = fmax(gds, gf);
      m[0] = gds;
      m[1] = gds;
      m[2] = -gds;
      m[3] = -gds;
      m[4] = gm;
      m[5] = -gm;
      m[6] = -gm;
      m[7] = gm;
      r[0] = -ieq;
      r[1] = ieq;
      nr = 2;
      return 8;
    }
    case 6: {  // MC: same 8 inserts, exact partials
      const double vd = xg(nd[0]), vg = xg(nd[1]), vs = xg(nd[2]);
      double id, ddg, ddd, dds;
      mos_consistent(p, vd, vg, vs, id, ddg, ddd, dds, gdev);
      const double ieq = id - (ddg * vg + ddd * vd + dds * vs);
      m[0] = ddd;
      m[1] = -dds;
      m[2] = dds;
      m[3] = -ddd;
      m[4] = ddg;
      m[5] = 0.0;
      m[6] = -ddg;
      m[7] = 0.0;
      r[0] = -ieq;
      r[1] = ieq;
      nr = 2;
      return 8;
    }
    case 5: {  // C: backward Euler companion in transient, open in DC
      if (dt <= 0.0) return 0;
      const double g = p[0] / dt;
      const double ieq = g * vprev;
      m[0] = g;
      m[1] = g;
      m[2] = -g;
      m[3] = -g;
      r[0] = be_sign * ieq;
      r[1] = -be_sign * ieq;
      nr = 2;
      return 4;
    }
  }
  return 0;
}

__device__ __forceinline__ void stamp_device(const DCircuit& C, int d, const double* x, int xlen,
                                             double gmin, double scale, double dt,
                                             const double* cap_v, double be_sign, double* ax,
                                             double* rhs_c, double gdev) {
  const int* nd = C.nodes + 4 * d;
  auto xg = [&](int i) { return (i >= 0 && i < xlen) ? x[i] : 0.0; };
  double m[8], r[2];
  int nr;
  const double vprev = cap_v ? cap_v[d] : 0.0;
  const int nm = eval_device(C.type[d], nd, C.p + 6 * d, xg, gmin, scale, dt, vprev, be_sign,
                             m, r, nr, gdev);
  const int* raw = C.raw + 8 * d;
  for (int e = 0; e < nm; ++e)
    if (raw[e] >= 0) ax[raw[e]] = m[e];
  const int* rs = C.rhs_slot + 2 * d;
  for (int e = 0; e < nr; ++e)
    if (rs[e] >= 0) rhs_c[rs[e]] = r[e];
}

__global__ void k_stamp(DCircuit C, const double* __restrict__ x, int xlen, double gmin,
                        double scale, double dt, const double* __restrict__ cap_v,
                        double be_sign, double* ax, double* rhs_c, double gdev) {
  if (C.skip != nullptr && __ldcg(C.skip) != 0) return;
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d == 0 && C.pin_raw >= 0) ax[C.pin_raw] = 1.0;
  if (d >= C.ndev) return;
  stamp_device(C, d, x, xlen, gmin, scale, dt, cap_v, be_sign, ax, rhs_c, gdev);
}

// k_stamp and k_rhs_sum in one block, for circuits of up to kStampBlock devices: one
// launch instead of two. Measured, both kernels against this one: 33 devices 6.6 and
// 5.2 us, 530 devices 7.0 and 6.1 us, and a gap between launches less; a whole Newton
// iteration, 30 devices 55.8 and 51.0 us, 498 145.1 and 143.4, 948 190.7 and 189.1,
// 1130 230.8 and 232.1, 1772 301.1 and 303.8.
__global__ void __launch_bounds__(512) k_stamp_block(DCircuit C, const double* __restrict__ x,
                                                     int xlen, double gmin, double scale,
                                                     double dt, const double* __restrict__ cap_v,
                                                     double be_sign, double* ax, double* rhs_c,
                                                     double* rhs, double gdev) {
  if (C.skip != nullptr && __ldcg(C.skip) != 0) return;
  const int tid = threadIdx.x;
  if (tid == 0 && C.pin_raw >= 0) ax[C.pin_raw] = 1.0;
  for (int d = tid; d < C.ndev; d += blockDim.x)
    stamp_device(C, d, x, xlen, gmin, scale, dt, cap_v, be_sign, ax, rhs_c, gdev);
  __syncthreads();
  for (int i = tid; i < C.n; i += blockDim.x) {
    double v = 0.0;
    for (int t = C.rhs_ptr[i]; t < C.rhs_ptr[i + 1]; ++t) v += rhs_c[C.rhs_src[t]];
    rhs[i] = v;
  }
}

// dL/dp of every device at a DC solution x, given the adjoint lambda
// (A^T lambda = dL/dx): dL/dp = -lambda^T dF/dp with F(x, p) = A(x) x - b(x)
// the stamped KCL residual. p is the resistance for R, the value for V and
// I, Is for D, and VTO for the MOSFETs (threshold |VTO| for both models).
__global__ void k_param_grad(DCircuit C, const double* __restrict__ x, int xlen,
                             const double* __restrict__ lam, double* grad) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= C.ndev) return;
  const int* nd = C.nodes + 4 * d;
  const double* p = C.p + 6 * d;
  auto xg = [&](int i) { return (i >= 0 && i < xlen) ? x[i] : 0.0; };
  auto lg = [&](int i) { return (i >= 0 && i < C.n) ? lam[i] : 0.0; };
  double gr = 0.0;
  switch (C.type[d]) {
    case 0: {  // F_a += (va - vb)/R
      const double v = xg(nd[0]) - xg(nd[1]);
      gr = (lg(nd[0]) - lg(nd[1])) * v / (p[0] * p[0]);
      break;
    }
    case 1:  // aux row: va - vb - V
      gr = lg(nd[2]);
      break;
    case 2:  // F_a += I, F_b -= I
      gr = -(lg(nd[0]) - lg(nd[1]));
      break;
    case 3: {  // F_a += Is (exp(vd/vt) - 1)
      const double vt = 0.02585 * p[1];
      const double e = exp((xg(nd[0]) - xg(nd[1])) / vt);
      gr = -(lg(nd[0]) - lg(nd[1])) * (e - 1.0);
      break;
    }
    case 4:
    case 6: {  // F_d += id, F_s -= id; d id / d vth = -(frame sign) * gm
      const bool pm = p[0] != 0.0;
      const double vd = xg(nd[0]), vg = xg(nd[1]), vs = xg(nd[2]);
      const double beff = p[2] * 1e-4 * ((3.9 * 8.854e-12) / p[3]) * p[4] / p[5];
      double vgs, vds, vth, sgn;
      if (C.type[d] == 6) {
        const double pol = pm ? -1.0 : 1.0;
        vgs = pol * (vg - vs);
        vds = pol * (vd - vs);
        const bool rev = vds < 0.0;
        if (rev) {
          vgs = vgs - vds;
          vds = -vds;
        }
        vth = fabs(p[1]);
        sgn = rev ? -pol : pol;
      } else {  // the reference's frame (evaluate.rs:299-316)
        double vdi = pm ? -vs : vd, vgi = pm ? -vg : vg, vsi = pm ? -vd : vs;
        vgs = vgi - vsi;
        vds = vdi - vsi;
        if (vds < 0.0) {
          vds = -vds;
          vgs = vgi - vdi;
        }
        vth = pm ? -fabs(p[1]) : fabs(p[1]);
        sgn = pm ? -1.0 : 1.0;
      }
      double gm = 0.0;
      if (vgs > vth)
        gm = vds < vgs - vth ? beff * vds * (C.type[d] == 6 ? 1.0 + 0.02 * vds : 1.0)
                             : beff * (vgs - vth) * (1.0 + 0.02 * vds);
      // dvth/dVTO: |VTO| -> sign(VTO); the reference's PMOS uses -|VTO|
      double dvth = p[1] >= 0.0 ? 1.0 : -1.0;
      if (C.type[d] == 4 && pm) dvth = -dvth;
      const double did = sgn * (-gm) * dvth;
      gr = -(lg(nd[0]) - lg(nd[2])) * did;
      break;
    }
    default:
      break;
  }
  grad[d] = gr;
}

__global__ void k_rhs_sum(DCircuit C, const double* __restrict__ rhs_c, double* rhs) {
  if (C.skip != nullptr && __ldcg(C.skip) != 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C.n) return;
  double v = 0.0;
  for (int t = C.rhs_ptr[i]; t < C.rhs_ptr[i + 1]; ++t) v += rhs_c[C.rhs_src[t]];
  rhs[i] = v;
}

// --------------------------------------------------------------- Newton
// One thread's part of the update's norm and tests: elements tid, tid + 1024, ...
__device__ __forceinline__ void newton_part(int m, const double* x, const double* xn, NewtonCfg cfg,
                                            int tid, double& acc, int& conv, int& fin) {
  acc = 0.0;
  conv = fin = 1;
#pragma unroll 4
  for (int i = tid; i < m; i += 1024) {
    const double a = xn[i], dx = a - x[i];
    acc += dx * dx;
    if (!(fabs(dx) <= cfg.abs_tol + cfg.rel_tol * fabs(a))) conv = 0;
    if (((unsigned)__double2hiint(a) & 0x7ff00000u) == 0x7ff00000u) fin = 0;
  }
}
__device__ __forceinline__ void newton_reduce(double& acc, int& conv, int& fin) {
  for (int off = 16; off > 0; off >>= 1) {
    acc += __shfl_down_sync(FULL, acc, off);
    conv &= __shfl_down_sync(FULL, conv, off);
    fin &= __shfl_down_sync(FULL, fin, off);
  }
}
// The state after an update of norm sqrt(acc).
__device__ __forceinline__ void newton_step(NewtonState* st, const NewtonCfg& cfg, double acc,
                                            int conv, int fin, const int* status) {
  const double dxn = sqrt(acc);
  st->iter += 1;
  st->converged = conv;
  if (!conv) {
    if (dxn > st->prev_dx_norm && st->damping > cfg.damping_min)
      st->damping = fmax(st->damping * 0.5, cfg.damping_min);
    st->prev_dx_norm = dxn;
  }
  const int code = *(volatile const int*)status;
  st->nonfinite = !fin;
  st->status = code;
  st->stop = conv || code != DS_OK || (!fin && cfg.stop_nonfinite);
}

__global__ void __launch_bounds__(1024) k_newton_update(int m, int n, double* x,
                                                        const double* __restrict__ xn,
                                                        NewtonState* st, NewtonCfg cfg,
                                                        const int* status) {
  if (st->stop) return;  // launched before the last iteration was known to be that
  __shared__ double ssum[32];
  __shared__ int sconv[32], sfin[32];
  const int tid = threadIdx.x;
  double acc;
  int conv, fin;
  newton_part(m, x, xn, cfg, tid, acc, conv, fin);
  newton_reduce(acc, conv, fin);
  if ((tid & 31) == 0) {
    ssum[tid >> 5] = acc;
    sconv[tid >> 5] = conv;
    sfin[tid >> 5] = fin;
  }
  __syncthreads();
  if (tid < 32) {
    acc = ssum[tid];
    conv = sconv[tid];
    fin = sfin[tid];
    newton_reduce(acc, conv, fin);
    if (tid == 0) {
      newton_step(st, cfg, acc, conv, fin, status);
      ssum[0] = st->damping;
      sconv[0] = conv;
    }
  }
  __syncthreads();
  const double damp = ssum[0];
  if (sconv[0]) {
    for (int i = tid; i < n; i += blockDim.x) x[i] = xn[i];
  } else {
    for (int i = tid; i < m; i += blockDim.x) x[i] = x[i] + damp * (xn[i] - x[i]);
  }
}

// The same over the grid, for systems whose FP64 work one SM's pipes draw out:
// block w is the single block's warp w, the last one to finish adds the 32 sums
// in the same order (the state bit for bit), k_newton_apply updates the iterate.
// Measured, 102,065 unknowns: 290 us in one block, 41 us so; 15,403:
// 47 us and 13 us.
__global__ void __launch_bounds__(32) k_newton_norm(int m, const double* x,
                                                    const double* __restrict__ xn, NewtonState* st,
                                                    NewtonCfg cfg, const int* status) {
  const int lane = threadIdx.x;
  if (__ldcg(&st->stop)) {
    if (blockIdx.x == 0 && lane == 0) st->apply = 0;
    return;
  }
  double acc;
  int conv, fin;
  newton_part(m, x, xn, cfg, blockIdx.x * 32 + lane, acc, conv, fin);
  newton_reduce(acc, conv, fin);
  int last = 0;
  if (lane == 0) {
    st->part[blockIdx.x] = acc;
    st->pflag[blockIdx.x] = conv | fin << 1;
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  if (!__shfl_sync(FULL, last, 0)) return;
  __threadfence();
  acc = __ldcg(&st->part[lane]);
  const int f = __ldcg(&st->pflag[lane]);
  conv = f & 1;
  fin = f >> 1;
  newton_reduce(acc, conv, fin);
  if (lane == 0) {
    newton_step(st, cfg, acc, conv, fin, status);
    st->apply = 1;
    st->ticket = 0;
  }
}
__global__ void k_newton_apply(int m, int n, double* x, const double* __restrict__ xn,
                               const NewtonState* st) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (!st->apply) return;
  if (st->converged) {
    if (i < n) x[i] = xn[i];
  } else if (i < m) {
    x[i] = x[i] + st->damping * (xn[i] - x[i]);
  }
}

// FP64 pipe throughput probe: every thread runs 8 independent chains of
// fused multiply-adds (explicit fma, 2 flops each); the result is stored so
// the work cannot be removed.
__global__ void k_dfma_peak(double* out, int iters, double a, double b) {
  double v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = threadIdx.x * 1e-7 + k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = fma(v[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += v[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

__global__ void k_rcond(DPlan P, const double* __restrict__ lu, double* out) {
  __shared__ double smin[32], smax[32];
  const int tid = threadIdx.x;
  double mn = 1.7976931348623157e308, mx = 0.0;
  for (int k = tid; k < P.n; k += blockDim.x) {
    const double a = fabs(lu[P.dslot[k]]);
    mn = fmin(mn, a);
    mx = fmax(mx, a);
  }
  for (int off = 16; off > 0; off >>= 1) {
    mn = fmin(mn, __shfl_down_sync(FULL, mn, off));
    mx = fmax(mx, __shfl_down_sync(FULL, mx, off));
  }
  if ((tid & 31) == 0) {
    smin[tid >> 5] = mn;
    smax[tid >> 5] = mx;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      mn = fmin(mn, smin[w]);
      mx = fmax(mx, smax[w]);
    }
    out[0] = fmin(mn, smin[0]);
    out[1] = fmax(mx, smax[0]);
  }
}

// Pivot growth after a refactorization with kept pivots: one thread per
// column scans its multipliers (L slots after the pivot); a block with one
// above lim - the kept pivot is below 1/lim of the largest entry under it,
// the rule the first factorization swaps on - is marked.
__global__ void k_growth(DPlan P, const double* __restrict__ lu, double lim, int* grow) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.n) return;
  const int s1 = P.col_ptr[k + 1];
  for (int s = P.dslot[k] + 1; s < s1; ++s)
    if (!(fabs(lu[s]) <= lim)) {
      grow[P.pos_block[k]] = 1;
      return;
    }
}

// --------------------------------------------------------------- batched
// One warp owns M instances of one circuit program at a time and keeps all
// of their state in shared memory (batch_common.cuh); each Newton iteration
// touches global memory only for the program and the circuit constants.
//   stamp     - lanes evaluate devices (strided) into their value records
//   assemble  - lanes sum each LU slot's and each rhs row's contributions in
//               stamping order (bit-identical to the reference's scatter)
//   factor    - left-looking, column by column; a column's U entries in
//               order, each applying L(:,j) across lanes; the forward
//               substitution of the right-hand side is fused in
//   backward  - U sweep, lanes over a column's U entries
//   update    - convergence test, damping and iterate update
// M instances per warp, 32/M lanes each; the M instances run the same
// program (one group), so the warp's control flow is shared and every FP64
// warp instruction of the sequential factor and solve serves M instances.
// SHARED: the warps of a block work on one group at a time and share one
// staged program (more instances per SM when the program is large); the
// block moves to its next tile when every warp has run out of instances.
// The block's shared memory is carved per group: as many warps as the
// group's own program and instance regions fit take instances, the others
// sit the tile out, so groups smaller than the largest of their class keep
// more instances resident.
template <int M, bool SHARED>
__global__ void k_batch_newton(BatchArgs A) {
  constexpr int LPI = 32 / M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / LPI, sl = lane % LPI, lead = sub * LPI;
  const unsigned leaders =
      M == 1 ? 1u : (M == 2 ? 0x00010001u : (M == 4 ? 0x01010101u : 0x11111111u));
  // per-warp slice (the staged program, then M instance regions), or one
  // program for the block followed by every warp's regions
  unsigned char* const slice =
      SHARED ? smem_raw
             : smem_raw + (size_t)warp * ((size_t)A.prog_ints * 4 + (size_t)M * A.region * 8);
  int* const prog = reinterpret_cast<int*>(slice);
  const NewtonCfg cfg = A.cfg;
  const double gstart = fmax(cfg.gmin * 1e3, 1e-6);
  while (true) {
    int ti = 0;
    if (SHARED) {
      // a continuation tile whose group has no parked instance left is
      // skipped before its program is staged: most groups park none
      if (threadIdx.x == 0) {
        int t = (int)atomicAdd(A.counter, 1u);
        while (A.cont_mode && t < A.ntiles) {
          const int gg = A.tile_group[t];
          if (*(volatile unsigned*)&A.gnext2[gg] < *(volatile unsigned*)&A.cont_count[gg])
            break;
          t = (int)atomicAdd(A.counter, 1u);
        }
        s_tile = t;
      }
      __syncthreads();
      ti = s_tile;
    } else {
      if (lane == 0) ti = (int)atomicAdd(A.counter, 1u);
      ti = __shfl_sync(FULL, ti, 0);
    }
    if (ti >= A.ntiles) return;
    const int g = A.tile_group[ti];
    const GroupHdr G = A.groups[g];
    const int pg = SHARED ? G.prog : A.prog_ints;
    const int rg = SHARED ? G.region : A.region;
    const int active =
        SHARED ? min((int)(blockDim.x >> 5), (A.shared_bytes - pg * 4) / (rg * 8 * M)) : 1;
    double* const region = reinterpret_cast<double*>(slice + (size_t)pg * 4) +
                           (size_t)((SHARED ? warp * M : 0) + sub) * rg;
    bt::Prog P = SHARED ? bt::stage_program(A, G, prog, threadIdx.x, blockDim.x, true, true)
                        : bt::stage_program(A, G, prog, lane, 32, false, true);
    const int n = P.n, nc = P.nc;
    // region: X[nc] T[n] V[nslots + noffd] DV[ndv], then the row -> slot map
    // (the step program addresses X, T and V from the region's start)
    double* const X = region;
    double* const T = X + nc;
    double* const V = T + n;
    double* const DV = V + G.nslots + G.noffd;
    P.map = reinterpret_cast<int*>(DV + G.ndv);

    int inst = -1, it = 0, total = 0, gstep = 0, ov_dev = -1;
    bool exhausted = warp >= active;  // no room for this warp's instances in this group
    double damp = 0.0, prev = 0.0, gmin = 0.0, ov_val = 0.0;
    const double* dparams = nullptr;
    while (true) {
      // ---- idle sub-groups take the group's next instances (one atomic per warp)
      const bool need = inst < 0 && !exhausted;
      const unsigned want = __ballot_sync(FULL, need) & leaders;
      if (want) {
        const int first_lane = __ffs(want) - 1;
        unsigned* const ctr = A.cont_mode ? &A.gnext2[g] : &A.gnext[g];
        int base = 0;
        if (lane == first_lane) base = (int)atomicAdd(ctr, (unsigned)__popc(want));
        base = __shfl_sync(FULL, base, first_lane);
        if (need) {
          const int k = base + __popc(want & ((1u << lead) - 1));
          const int count = A.cont_mode ? (int)A.cont_count[g] : G.inst_count;
          if (k < count) {
            inst = A.cont_mode ? A.cont_list[G.inst_begin + k] : A.order[G.inst_begin + k];
            dparams = A.dparams + A.inst_p_off[inst];
            ov_dev = A.inst_ov_dev[inst];
            ov_val = A.inst_ov_val[inst];
            if (A.cont_mode) {  // resume where the lane phase parked it
              const long long xo = A.inst_x_off[inst];
              for (int i = sl; i < nc; i += LPI) X[i] = A.x_out[xo + i];
              it = A.cont_it[inst];
              total = A.cont_total[inst];
              gstep = A.cont_gstep[inst];
              damp = A.cont_damp[inst];
              prev = A.cont_prev[inst];
              gmin = cfg.gmin_steps == 0
                         ? cfg.gmin
                         : gstart + (cfg.gmin - gstart) * ((double)gstep / (double)cfg.gmin_steps);
            } else {
              const long long xo = A.inst_x0_off[inst];
              for (int i = sl; i < nc; i += LPI) X[i] = xo >= 0 ? A.x0[xo + i] : 0.0;
              it = total = gstep = 0;
              damp = cfg.damping;
              prev = 1.7976931348623157e308;
              gmin = cfg.gmin_steps == 0 ? cfg.gmin : gstart;
            }
          } else {
            exhausted = true;
          }
        }
      }
      if (!__any_sync(FULL, inst >= 0)) break;
      __syncwarp();
      const bool live = inst >= 0;
      if (live) bt::stamp_devices<LPI>(P, dparams, ov_dev, ov_val, X, X, gmin, 1e-12, false, DV, sl);
      __syncwarp();
      bt::assemble<LPI>(P, DV, V, T, sl);
      __syncwarp();
      if (P.nsteps > 0)
        bt::run_steps<LPI>(P, X, sl);
      else
        bt::factor_solve<LPI>(P, V, T, sl);
      // ---- Newton update (crates/sim-core/src/newton.rs:93-107)
      bool conv = true, fin = true;
      for (int c = sl; c < nc; c += LPI) {
        const double a = T[P.out_pos[c]];
        const double dx = a - X[c];
        DV[c] = dx * dx;
        if (!(fabs(dx) <= cfg.abs_tol + cfg.rel_tol * fabs(a))) conv = false;
        if (!isfinite(a)) fin = false;
      }
      const unsigned smask = (LPI == 32 ? FULL : (((1u << LPI) - 1u) << lead));
      const unsigned nconv = __ballot_sync(FULL, !conv) & smask;
      const unsigned nfin = __ballot_sync(FULL, !fin) & smask;
      __syncwarp();
      if (live) {
        ++it;
        ++total;
        int rsn = -1;
        if (!nconv) {
          rsn = 0;
          const long long xo = A.inst_x_off[inst];
          if (xo >= 0)
            for (int c = sl; c < n; c += LPI) A.x_out[xo + c] = T[P.out_pos[c]];
        } else {
          double ss = 0.0;  // norm2 of dx, reduced across the instance's lanes
          for (int c = sl; c < nc; c += LPI) ss += DV[c];
#pragma unroll
          for (int o = LPI / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(smask, ss, o);
          const double dxn = sqrt(ss);
          if (dxn > prev && damp > cfg.damping_min) damp = fmax(damp * 0.5, cfg.damping_min);
          prev = dxn;
          for (int c = sl; c < nc; c += LPI) X[c] = fma(damp, T[P.out_pos[c]] - X[c], X[c]);
          if (nfin) {
            rsn = 1;
          } else if (it >= cfg.max_iters) {
            if (gstep < cfg.gmin_steps) {  // next gmin step, fresh damping state
              ++gstep;
              gmin = gstart + (cfg.gmin - gstart) * ((double)gstep / (double)cfg.gmin_steps);
              it = 0;
              damp = cfg.damping;
              prev = 1.7976931348623157e308;
            } else {
              rsn = 1;
            }
          }
          if (rsn == 1) {
            const long long xo = A.inst_x_off[inst];
            if (xo >= 0)
              for (int c = sl; c < n; c += LPI) A.x_out[xo + c] = c < nc ? X[c] : 0.0;
          }
        }
        if (rsn >= 0) {
          if (sl == 0) {  // non-finite: the reference's run ends at the cap
            A.iters[inst] = (rsn == 1 && nfin) ? cfg.max_iters : it;
            A.iters_total[inst] = total;
            A.reason[inst] = rsn;
          }
          inst = -1;
        }
      }
      __syncwarp();
    }
    if (SHARED)
      __syncthreads();  // every warp is done with the block's staged program
    else
      __syncwarp();  // done with this group's staged program
  }
}

}  // namespace

// ------------------------------------------------------------------ launches
void launch_first_factor(const DPlan& P, int maxblk, const double* ax, double* lu,
                         double* work, int* rperm, int* rinv, double tol, int* status,
                         cudaStream_t s) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t fixed = (size_t)12 * maxblk + 4 * (size_t)(kPatCap + 33 + 32 + 32) + 16;
  int cap = 4096;
  while (cap > 256 && fixed + (size_t)12 * cap > (size_t)optin) cap >>= 1;
  const size_t bytes = fixed + (size_t)12 * cap;
  if (maxblk > 0 && bytes <= (size_t)optin) {
    raise_smem_limit<k_first_factor_s>(bytes);
    k_first_factor_s<<<1, 32, bytes, s>>>(P, ax, lu, rperm, rinv, tol, maxblk, cap);
    return;
  }
  k_first_factor<<<1, 32, 0, s>>>(P, ax, lu, work, rperm, rinv, tol, status);
}

void launch_refactor(const DPlan& P, const double* ax, double* lu, double* big, int* status,
                     int grid, cudaStream_t s, const PivotCheck& pc) {
  const long long words = (long long)P.nslots + kLuPad;
  if (P.skip != nullptr)
    k_preset<<<(int)std::min<long long>((words + 1023) / 1024, 4096), 256, 0, s>>>(lu, words, P.skip);
  else
    cudaMemsetAsync(lu, 0xff, (size_t)words * sizeof(double), s);
  const int colcap = std::min((P.max_col + 1) & ~1, kColCap);
  const int bytes = kPairs * (kGridRing * kGridStage + 8 * colcap);
  raise_smem_limit<k_refactor>(bytes);
  k_refactor<<<grid, 64 * kPairs, bytes, s>>>(P, ax, lu, big, colcap, status, pc);
}
bool refactor_needs_big(const DPlan& P) { return P.max_col > kColCap; }

namespace {
size_t refactor_cta_bytes(const DPlan& P) {
  return (((size_t)8 * P.nslots + 15) & ~(size_t)15) + (size_t)32 * kCtaRing * kCtaStage +
         (size_t)4 * P.n + 16;
}
int smem_optin() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin;
}
}  // namespace

bool refactor_cta_fits(const DPlan& P) {
  return P.n > 0 && refactor_cta_bytes(P) + 64 <= (size_t)smem_optin();
}

void launch_refactor_cta(const DPlan& P, const double* ax, double* lu, int* status,
                         cudaStream_t s, const PivotCheck& pc) {
  const size_t bytes = refactor_cta_bytes(P);
  raise_smem_limit<k_refactor_cta>(bytes);
  k_refactor_cta<<<1, 1024, bytes, s>>>(P, ax, lu, status, pc);
}

namespace {
size_t solve_cta_bytes(const DPlan& P, int rows) {
  return (size_t)8 * rows + (size_t)24 * kSolveChunk + (size_t)4 * (2 * (size_t)rows + 1) +
         (P.noffd > 0 ? (size_t)4 * (rows + 1) : 0) + 16;
}
size_t solve_cta_bytes(const DPlan& P) { return solve_cta_bytes(P, P.n); }
}  // namespace

bool solve_cta_fits(const DPlan& P) {
  return P.n > 0 && solve_cta_bytes(P) <= (size_t)smem_optin();
}

void launch_solve_cta(const DPlan& P, const double* rhs, const double* ax, const double* lu,
                      double* out, cudaStream_t s) {
  const size_t bytes = solve_cta_bytes(P);
  raise_smem_limit<k_solve_cta>(bytes);
  k_solve_cta<<<1, 256, bytes, s>>>(P, rhs, ax, lu, out, kSolveChunk, 0);
}

bool solve_steps_fits(const DPlan& P) {
  if (P.n > 0 && P.ss.nsteps > 0) return (size_t)8 * P.n + 16 <= (size_t)smem_optin();
  return P.n > 0 && P.ss.nchunks > 0 &&
         solve_steps_bytes(P.n, P.ss.chunk) + 64 <= (size_t)smem_optin();
}

void launch_solve_steps(const DPlan& P, bool transpose, const double* rhs, const double* ax,
                        const double* lu, double* rec, double* out, int* status, cudaStream_t s) {
  const int *const in = transpose ? P.out_col : P.in_row, *const outp = transpose ? P.in_row : P.out_col;
  if (P.ss.nsteps > 0) {
    const size_t bytes = (size_t)8 * P.n;
    raise_smem_limit<k_solve_list>(bytes);
    k_solve_list<<<1, kSolveListThreads, bytes, s>>>(P.ss, P.n, in, outp, P.dslot, rhs, ax, lu, rec,
                                                     out, P.skip);
    return;
  }
  const size_t bytes = solve_steps_bytes(P.n, P.ss.chunk);
  const bool staged = P.ss.vc != nullptr;
  const auto kernel = staged ? k_solve_steps<true> : k_solve_steps<false>;
  if (staged)
    raise_smem_limit<k_solve_steps<true>>(bytes);
  else
    raise_smem_limit<k_solve_steps<false>>(bytes);
  if (staged)
    k_solve_slots<<<(P.ss.nslots + 255) / 256, 256, 0, s>>>(P.ss, P.n, ax, lu, P.skip);
  // a program of one short chunk has nothing for the loader warps to fetch (two
  // rows, a call: 29.1 us without them, 30.0 with)
  const int loaded = P.ss.nchunks == 1 && P.ss.nslots <= kSolveRow * kLoadBatch ? kSolveRow
                                                                                : kSolveStepsThreads;
  kernel<<<1, staged ? kSolveRow + 32 : loaded, bytes, s>>>(
      P.ss, P.n, in, outp, P.dslot, rhs, ax, lu, rec, out, P.skip, status, P.pair_limit);
}

bool solve_groups_fit(const DPlan& P) {
  return P.cs_ngrp > 0 && P.noffd == 0 &&
         solve_cta_bytes(P, P.cs_grp_rows) <= (size_t)smem_optin();
}

void launch_solve_groups(const DPlan& P, const double* rhs, const double* ax, const double* lu,
                         double* out, cudaStream_t s) {
  const size_t bytes = solve_cta_bytes(P, P.cs_grp_rows);
  raise_smem_limit<k_solve_cta>(bytes);
  k_solve_cta<<<P.cs_ngrp, 256, bytes, s>>>(P, rhs, ax, lu, out, kSolveChunk, 1);
}

void launch_solve(const DPlan& P, const double* rhs, const double* ax, const double* lu,
                  double* z, double* x, double* out, unsigned* zflag, unsigned* xflag,
                  unsigned epoch, unsigned* counter, int* status, int grid, bool transpose,
                  cudaStream_t s) {
  cudaMemsetAsync(counter, 0, sizeof(unsigned), s);
  if (transpose)
    k_tsolve<<<grid, 128, 0, s>>>(P, rhs, ax, lu, z, x, out, zflag, xflag, epoch, counter,
                                  status);
  else
    k_solve<<<grid, 128, 0, s>>>(P, rhs, ax, lu, z, x, out, zflag, xflag, epoch, counter,
                                 status);
}

// Devices and rows of a circuit stamped in one block (two passes of its threads).
constexpr int kStampBlock = 1024;
void launch_stamp(const DCircuit& C, const double* x, int xlen, double gmin, double scale,
                  double dt, const double* cap_v, double be_sign, double* ax, double* rhs_c,
                  double* rhs, cudaStream_t s, double gdev) {
  if (C.ndev <= kStampBlock && C.n <= kStampBlock) {
    k_stamp_block<<<1, 512, 0, s>>>(C, x, xlen, gmin, scale, dt, cap_v, be_sign, ax, rhs_c, rhs,
                                    gdev);
    return;
  }
  const int nb = (C.ndev + 255) / 256;
  k_stamp<<<nb > 0 ? nb : 1, 256, 0, s>>>(C, x, xlen, gmin, scale, dt, cap_v, be_sign, ax,
                                          rhs_c, gdev);
  k_rhs_sum<<<(C.n + 255) / 256, 256, 0, s>>>(C, rhs_c, rhs);
}

void launch_param_grad(const DCircuit& C, const double* x, int xlen, const double* lam,
                       double* grad, cudaStream_t s) {
  k_param_grad<<<(C.ndev + 255) / 256 > 0 ? (C.ndev + 255) / 256 : 1, 256, 0, s>>>(C, x, xlen, lam,
                                                                                  grad);
}

// Unknowns from which the update runs over the grid: the second launch costs
// about 2 us, one block 3 us per 1024 unknowns.
constexpr int kNewtonGrid = 4096;
void launch_newton_update(int m, int n, double* x, const double* xnew, NewtonState* st,
                          NewtonCfg cfg, int* status, cudaStream_t s) {
  if (n < kNewtonGrid) {
    k_newton_update<<<1, 1024, 0, s>>>(m, n, x, xnew, st, cfg, status);
    return;
  }
  k_newton_norm<<<32, 32, 0, s>>>(m, x, xnew, st, cfg, status);
  k_newton_apply<<<(n + 255) / 256, 256, 0, s>>>(m, n, x, xnew, st);
}

void launch_growth(const DPlan& P, const double* lu, double lim, int* grow, cudaStream_t s) {
  if (P.n <= 0) return;
  k_growth<<<(P.n + 255) / 256, 256, 0, s>>>(P, lu, lim, grow);
}

void launch_rcond(const DPlan& P, const double* lu, double* out2, cudaStream_t s) {
  k_rcond<<<1, 1024, 0, s>>>(P, lu, out2);
}

double fp64_peak_tflops() {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = sms * 8, block = 256, iters = 4096;
  double* out = nullptr;
  if (cudaMalloc(&out, (size_t)grid * block * sizeof(double)) != cudaSuccess) return 0.0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_dfma_peak<<<grid, block>>>(out, 64, 0.999999, 1e-9);  // warm-up
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    cudaEventRecord(e0);
    k_dfma_peak<<<grid, block>>>(out, iters, 0.999999, 1e-9);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    best = ms < best ? ms : best;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  const double flops = 2.0 * 8.0 * iters * (double)grid * block;
  return flops / (best * 1e-3) / 1e12;
}

template <int M, bool SHARED>
static size_t smem_bytes(const BatchArgs& a, int warps_per_block) {
  if (SHARED) return (size_t)a.shared_bytes;
  return ((size_t)a.prog_ints * 4 + (size_t)a.region * M * sizeof(double)) * warps_per_block;
}

template <int M, bool SHARED>
static void launch_m(const BatchArgs& a, int grid, int warps_per_block, cudaStream_t s) {
  const size_t sm = smem_bytes<M, SHARED>(a, warps_per_block);
  raise_smem_limit<k_batch_newton<M, SHARED>>(sm);
  k_batch_newton<M, SHARED><<<grid, 32 * warps_per_block, sm, s>>>(a);
}

// The tile counter and the per-group instance counters are reset by the
// caller before the classes start (the classes share the group counter
// array and run concurrently).
void launch_batch_newton(const BatchArgs& a, int m, int grid, int warps_per_block,
                         cudaStream_t s, bool shared) {
  if (shared) {
    switch (m) {
      case 8: launch_m<8, true>(a, grid, warps_per_block, s); break;
      case 4: launch_m<4, true>(a, grid, warps_per_block, s); break;
      case 2: launch_m<2, true>(a, grid, warps_per_block, s); break;
      default: launch_m<1, true>(a, grid, warps_per_block, s); break;
    }
    return;
  }
  switch (m) {
    case 8: launch_m<8, false>(a, grid, warps_per_block, s); break;
    case 4: launch_m<4, false>(a, grid, warps_per_block, s); break;
    case 2: launch_m<2, false>(a, grid, warps_per_block, s); break;
    default: launch_m<1, false>(a, grid, warps_per_block, s); break;
  }
}

template <int M, bool SHARED>
static void info_m(int warps_per_block, int region, int prog_ints, int* regs,
                   int* blocks_per_sm, size_t shared_bytes) {
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, k_batch_newton<M, SHARED>);
  *regs = fa.numRegs;
  const size_t per = (size_t)region * M * sizeof(double);
  const size_t sm = SHARED ? shared_bytes : ((size_t)prog_ints * 4 + per) * warps_per_block;
  raise_smem_limit<k_batch_newton<M, SHARED>>(sm);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_batch_newton<M, SHARED>,
                                                32 * warps_per_block, sm);
  cudaGetLastError();  // more than a block may have: answered by *blocks_per_sm
}

void batch_kernel_info(int m, int warps_per_block, int region, int prog_ints, int* regs,
                       int* blocks_per_sm, bool shared, size_t shared_bytes) {
  auto run = [&](auto fn) {
    fn(warps_per_block, region, prog_ints, regs, blocks_per_sm, shared_bytes);
  };
  if (shared) {
    switch (m) {
      case 8: run(info_m<8, true>); break;
      case 4: run(info_m<4, true>); break;
      case 2: run(info_m<2, true>); break;
      default: run(info_m<1, true>); break;
    }
    return;
  }
  switch (m) {
    case 8: run(info_m<8, false>); break;
    case 4: run(info_m<4, false>); break;
    case 2: run(info_m<2, false>); break;
    default: run(info_m<1, false>); break;
  }
}

}  // namespace gk
