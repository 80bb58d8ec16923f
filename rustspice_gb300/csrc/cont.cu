// Batched DC operating points, one instance per warp or two (16 lanes each).
//
// Each warp takes instances from a queue over every program (most expensive
// programs first) and runs their Newton loops to the end, from the start or
// from where the lane kernel (lanes.cu) parked them: the permuted
// right-hand side and the LU values in the warp's slice of shared memory, the
// device records and the iterate in its slice of a global scratch (written
// and read by the warp's own lanes, L2 resident), the factorization and
// substitutions as the program's row stream (bt::run_stream). A warp that
// finishes an instance takes the next one at once: no warp waits for the
// others of its block, and no block stages a program.
//
// What bounds it: FP64 issue, one warp instruction per 64 cycles and SM
// sub-partition whatever its active lanes, and for the instances that run to
// the iteration cap the latency of their rows. Measured against the lane
// kernel's six iterations and a kernel that loads its steps from global
// memory behind it: 976 instances (16 chains of 8-256 stages) 38.9 -> 9.8 ms,
// 249,856 instances 71.7 -> 65.2 ms.
#include <cfloat>

#include "batch_common.cuh"
#include "kernels.cuh"

namespace gk {
namespace {

constexpr unsigned kFullMask = 0xffffffffu;

// The lane kernel (lanes.cu) sums every list and the update's norm in order,
// one instance per lane. The first `cap` iterations of an instance keep that
// order of additions here, so the iterates are the lane kernel's bit for bit;
// the lists are then gathered by all lanes into the slice (T and the LU
// values are not yet in use) and each summed by one lane, 64 cycles a term,
// the norm likewise from its differences.
//
// Sum of this lane's list (lane sl < nheavy <= LPI) in order, from 0.
template <int LPI>
__device__ __forceinline__ double ordered_lists(const bt::Prog& P, const double* DV, double* S,
                                                int room, int sl) {
  const int G = P.nheavy;
  int len = 0;
  const int* cds = sl < G ? bt::list_codes(P, P.heavy[sl], len) : nullptr;
  int longest = len;
#pragma unroll
  for (int o = LPI / 2; o > 0; o >>= 1)
    longest = max(longest, __shfl_xor_sync(kFullMask, longest, o));
  int chunk = room / G;  // an odd stride: the lanes read different banks
  if (chunk > 1 && chunk % 2 == 0) --chunk;
  double acc = 0.0;
  for (int base = 0; base < longest; base += chunk) {
    for (int g = 0; g < G; ++g) {
      const int n = min(chunk, __shfl_sync(kFullMask, len, g, LPI) - base);
      const int* const cg = reinterpret_cast<const int*>(
                                __shfl_sync(kFullMask, (unsigned long long)cds, g, LPI)) + base;
      for (int t0 = sl; t0 < n; t0 += 8 * LPI) {
        int cd[8];
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          cd[u] = t0 + u * LPI < n ? __ldg(cg + t0 + u * LPI) : bt::kPadCode;
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = bt::contrib_load(DV, cd[u]);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (t0 + u * LPI < n) S[g * chunk + t0 + u * LPI] = bt::contrib_value(v[u], cd[u]);
      }
    }
    __syncwarp();
    const int n = min(chunk, len - base);
    const double* const mine = S + sl * chunk;
#pragma unroll 4
    for (int t = 0; t < n; ++t) acc += mine[t];
    __syncwarp();
  }
  return acc;
}

// M instances of one program per warp (32 / M lanes each, in step: one FP64
// instruction of a row serves all M); a sub-warp whose instance ends takes
// the program's next instance, and the warp moves to the next program when
// every sub-warp has run out.
template <int M>
__global__ void __launch_bounds__(32, kContWarps) k_batch_cont(BatchArgs A) {
  constexpr int LPI = 32 / M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  const int sub = lane / LPI, sl = lane % LPI;
  const unsigned smask = M == 1 ? kFullMask : (((1u << LPI) - 1u) << (sub * LPI));
  int2* const ring = reinterpret_cast<int2*>(smem_raw);
  double* const S = reinterpret_cast<double*>(smem_raw + kStreamRing) + (size_t)sub * A.slice;
  double* const DV = A.dv_scratch + ((long long)blockIdx.x * M + sub) * A.dv_stride;
  const NewtonCfg cfg = A.cfg;
  const double gstart = fmax(cfg.gmin * 1e3, 1e-6);
  while (true) {
    // ---- the next program with instances left, and up to M of them
    // (every pass either takes instances or moves the cursor on, so the
    // loop ends)
    // Every lane takes the same turns; lane 0 alone in the loop would leave the
    // warp diverged, lane 0 behind the others, for all that follows (measured:
    // an iteration of a 210-stage chain 750 k cycles instead of 190 k).
    int g = -1;
    unsigned k0 = 0, cnt = 0;
    while (true) {
      unsigned c = 0;
      if (lane == 0) c = *(volatile unsigned*)A.cont_cursor;
      c = __shfl_sync(kFullMask, c, 0);
      if (c >= (unsigned)A.cont_ngroups) return;
      g = A.cont_groups[c];
      if (lane == 0) k0 = atomicAdd(&A.gnext2[g], (unsigned)M);
      k0 = __shfl_sync(kFullMask, k0, 0);
      cnt = A.cont_parked ? A.cont_count[g] : (unsigned)A.groups[g].inst_count;
      if (k0 < cnt) break;
      if (lane == 0) atomicCAS(A.cont_cursor, c, c + 1);
    }
    const GroupHdr G = A.groups[g];
    const bt::Prog P = bt::global_view(A, G);
    const int n = P.n, nc = P.nc;
    // shared: T, V, the row stream's constants; global (L2): the records and
    // the iterate. The row stream addresses T at nc and V at nc + n from a
    // base nc doubles before the slice (it touches no X entry).
    double* const X = DV + A.dv_x;
    double* const D = X + nc;  // the last ordered iteration's differences
    double* const T = S;
    double* const V = T + n;
    double* const R = S - nc;
    if (sl == 0) {
      V[P.nv] = 1.0;
      V[P.nv + 1] = 0.0;
    }
    const bool lists_fit = P.nheavy > 0 && P.nheavy <= LPI;
    const int* const list = (A.cont_parked ? A.cont_list : A.order) + G.inst_begin;
    int inst = k0 + sub < cnt ? list[k0 + sub] : -1;
    bool exhausted = inst < 0;
    int it = 0, total = 0, gstep = 0, ov_dev = -1;
    long long xo = 0;
    double damp = 0.0, prev = 0.0, gmin = 0.0, ov_val = 0.0;
    bool prev_exact = true;
    const double* dparams = nullptr;
    auto start = [&]() {  // or where the lane kernel parked it, with its own sums
      dparams = A.dparams + A.inst_p_off[inst];
      ov_dev = A.inst_ov_dev[inst];
      ov_val = A.inst_ov_val[inst];
      xo = A.inst_x_off[inst];
      prev_exact = true;
      if (A.cont_parked) {
        for (int i = sl; i < nc; i += LPI) X[i] = A.x_out[xo + i];
        it = A.cont_it[inst];
        total = A.cont_total[inst];
        gstep = A.cont_gstep[inst];
        damp = A.cont_damp[inst];
        prev = A.cont_prev[inst];
        gmin = cfg.gmin_steps == 0
                   ? cfg.gmin
                   : gstart + (cfg.gmin - gstart) * ((double)gstep / (double)cfg.gmin_steps);
        return;
      }
      const long long x0o = A.inst_x0_off[inst];
      for (int i = sl; i < nc; i += LPI) X[i] = x0o >= 0 ? A.x0[x0o + i] : 0.0;
      it = total = gstep = 0;
      damp = cfg.damping;
      prev = DBL_MAX;
      gmin = cfg.gmin_steps == 0 ? cfg.gmin : gstart;
    };
    if (inst >= 0) start();
    while (true) {
      if (M > 1) {  // idle sub-warps take the program's next instances
        const bool need = inst < 0 && !exhausted;
        const unsigned want = __ballot_sync(kFullMask, need && sl == 0);
        if (want) {
          const int first = __ffs(want) - 1;
          unsigned base = 0;
          if (lane == first) base = atomicAdd(&A.gnext2[g], (unsigned)__popc(want));
          base = __shfl_sync(kFullMask, base, first);
          if (need) {
            const unsigned kk = base + __popc(want & ((1u << (sub * LPI)) - 1u));
            if (kk < cnt) {
              inst = list[kk];
              start();
            } else {
              exhausted = true;
            }
          }
        }
      }
      if (!__any_sync(kFullMask, inst >= 0)) break;
      __syncwarp();
      const bool live = inst >= 0;
      // this iteration with the lane kernel's order of additions
      const bool ordered = total < A.cap;
      const bool any_ordered = __any_sync(kFullMask, live && ordered);
      if (live) bt::stamp_devices<LPI>(P, dparams, ov_dev, ov_val, X, X, gmin, 1e-12, false, DV, sl);
      __syncwarp();
      double lsum = 0.0;
      if (any_ordered && lists_fit) lsum = ordered_lists<LPI>(P, DV, S, n + P.nv, sl);
      bt::assemble<LPI>(P, DV, V, T, sl);
      if (any_ordered && P.nheavy > 0) {
        __syncwarp();
        if (ordered) {
          if (lists_fit) {
            if (sl < P.nheavy) bt::put_list(P, P.heavy[sl], lsum, V, T);
          } else {
            for (int h = sl; h < P.nheavy; h += LPI) {
              int len;
              const int* const cds = bt::list_codes(P, P.heavy[h], len);
              double acc = 0.0;
              for (int t = 0; t < len; ++t) acc += bt::contrib(DV, cds[t]);
              bt::put_list(P, P.heavy[h], acc, V, T);
            }
          }
        }
      }
      bt::run_stream<LPI>(P.stream, ring, R, sl, nc + n + P.nv + 1);
      // ---- Newton update (crates/sim-core/src/newton.rs:93-107)
      bool conv = true, fin = true;
      double ss = 0.0, hi = 0.0;  // hi: the terms of lane sl + 16 when a sub-warp has 16
      for (int c0 = sl; c0 < nc; c0 += 4 * LPI) {
        double xo4[4];
        int p4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * LPI;
          p4[u] = c < nc ? __ldg(P.out_pos + c) : 0;
          xo4[u] = c < nc ? X[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * LPI;
          if (c >= nc) break;
          const double a = T[p4[u]];
          const double dx = a - xo4[u];
          const double sq = dx * dx;
          if (LPI == 16 && (u & 1))
            hi += sq;
          else
            ss += sq;
          V[c] = dx;  // the factors are done with; the ordered norm and the update
          if (!(fabs(dx) <= cfg.abs_tol + cfg.rel_tol * fabs(a))) conv = false;
          if (!isfinite(a)) fin = false;
        }
      }
      if (LPI == 16) ss += hi;
      const unsigned nconv = __ballot_sync(kFullMask, !conv) & smask;
      const unsigned nfin = __ballot_sync(kFullMask, !fin) & smask;
#pragma unroll
      for (int o = (LPI == 16 ? 8 : LPI / 2); o > 0; o >>= 1)
        ss += __shfl_xor_sync(kFullMask, ss, o);
      __syncwarp();
      // The norm decides the damping by comparison with the one before, and
      // an ordered iteration's norm is the ordered sum. Summed across the lanes it
      // is within n 2^-53 of that (its terms are positive): unless the two
      // norms are within 1e-9 of each other, or so small or large that
      // squares leave the exponent range, that decides as well.
      double dxn = sqrt(ss);
      bool larger = dxn > prev;
      const bool near = !(dxn < prev * (1.0 - 1e-9)) && !(dxn > prev * (1.0 + 1e-9));
      const bool exact = live && nconv && (ordered || !prev_exact) &&
                         (near || !(dxn > 1e-140) || !(dxn < 1e140));
      if (__any_sync(kFullMask, exact)) {
        double os = 0.0, op = 0.0;
#pragma unroll 4
        for (int c = 0; c < nc; ++c) os = fma(V[c], V[c], os);
        if (__any_sync(kFullMask, exact && !prev_exact))
#pragma unroll 4
          for (int c = 0; c < nc; ++c) op = fma(D[c], D[c], op);
        if (exact) {
          if (ordered) dxn = sqrt(os);
          if (!prev_exact) prev = sqrt(op);
          larger = dxn > prev;
        }
      }
      __syncwarp();
      if (live) {
        ++it;
        ++total;
        int rsn = -1;
        if (!nconv) {
          rsn = 0;
          if (xo >= 0)
            for (int c = sl; c < n; c += LPI) A.x_out[xo + c] = T[P.out_pos[c]];
        } else {
          if (larger && damp > cfg.damping_min) damp = fmax(damp * 0.5, cfg.damping_min);
          prev = dxn;
          prev_exact = exact || !ordered;
          if (!prev_exact)
            for (int c = sl; c < nc; c += LPI) D[c] = V[c];
#pragma unroll 4
          for (int c = sl; c < nc; c += LPI) X[c] = fma(damp, V[c], X[c]);
          if (nfin) {
            rsn = 1;
          } else if (it >= cfg.max_iters) {
            if (gstep < cfg.gmin_steps) {  // next gmin step, fresh damping state
              ++gstep;
              gmin = gstart + (cfg.gmin - gstart) * ((double)gstep / (double)cfg.gmin_steps);
              it = 0;
              damp = cfg.damping;
              prev = DBL_MAX;
              prev_exact = true;
            } else {
              rsn = 1;
            }
          }
          if (rsn == 1 && xo >= 0)
            for (int c = sl; c < n; c += LPI) A.x_out[xo + c] = c < nc ? X[c] : 0.0;
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
  }
}

size_t cont_bytes(int m, int slice) { return (size_t)m * slice * sizeof(double) + kStreamRing; }

template <int M>
void launch_m(const BatchArgs& a, int grid, cudaStream_t s) {
  // The same limit and shared-memory carve-out for every class: the attributes
  // belong to the kernel, and blocks of launches that asked for different
  // carve-outs would not share an SM.
  cudaFuncSetAttribute(k_batch_cont<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  cudaFuncSetAttribute(k_batch_cont<M>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       cudaSharedmemCarveoutMaxShared);
  k_batch_cont<M><<<grid, 32, cont_bytes(M, a.slice), s>>>(a);
}

template <int M>
void info_m(int slice, int* regs, int* blocks_per_sm) {
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, k_batch_cont<M>);
  *regs = fa.numRegs;
  *blocks_per_sm = 0;
  if (cont_bytes(M, slice) > 227 * 1024) return;
  cudaFuncSetAttribute(k_batch_cont<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_batch_cont<M>, 32,
                                                cont_bytes(M, slice));
}

}  // namespace

void launch_batch_cont(const BatchArgs& a, int m, int grid, cudaStream_t s) {
  if (m == 2)
    launch_m<2>(a, grid, s);
  else
    launch_m<1>(a, grid, s);
}

void cont_kernel_info(int m, int slice, int* regs, int* blocks_per_sm) {
  if (m == 2)
    info_m<2>(slice, regs, blocks_per_sm);
  else
    info_m<1>(slice, regs, blocks_per_sm);
}

}  // namespace gk
