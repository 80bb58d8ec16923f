// Batched fixed-step backward-Euler transient and its checkpointed adjoint.
//
// One warp owns one instance (a circuit with its own constants) for the whole
// run and keeps its state in shared memory (layout in batch_common.cuh).
//
//  * k_tran_fwd - time steps t = 1..steps, each a Newton solve from the
//    previous time point with the capacitor companions built from it; the
//    loss sum_t (x_t[probe] - target)^2 accumulates on the fly and the state
//    is written every ckpt_every steps.
//  * k_tran_bwd - segments in reverse: the states of a segment are recomputed
//    from its checkpoint with the same Newton iterations (so they are the
//    forward's states bit for bit), then for t descending the exact Jacobian
//    J_t (level-1 floor 0) is stamped and factored and
//        J_t^T lambda_t = dL/dx_t + G_C lambda_{t+1}
//    is solved with the factors; dL/dC_d = -sum_t (lambda_t[a] -
//    lambda_t[b]) (dv_t - dv_{t-1}) / dt accumulates per capacitor.
//
// The factorization and substitutions of a step are the program's row stream
// (bt::run_stream), the adjoint's transpose solve a second one. Measured, 1024
// rings of 11-101 stages, 250 steps: forward 86.8 -> 34.9 ms, adjoint 176.9 ->
// 55.3 ms against the columns one after another and the adjoint's right-hand
// side summed by one lane.
#include <cfloat>

#include "batch_common.cuh"
#include "kernels.cuh"

namespace gk {
namespace {

constexpr int LPI = 32;

// One Newton solve of the time step (crates/sim-core/src/newton.rs:65-117):
// X holds the initial iterate on entry and the solution on exit (node
// voltages). Returns 0 when converged, 1 otherwise.
__device__ int newton_step(const BatchArgs& A, const bt::Prog& P, const double* dparams,
                           double* X, const double* XP, double* T, double* DV, double* V,
                           int2* ring, int sl, int& iters) {
  const NewtonCfg& cfg = A.cfg;
  const int nc = P.nc;
  double damp = cfg.damping, prev = DBL_MAX;
  for (int it = 0; it < cfg.max_iters; ++it) {
    bt::stamp_devices<LPI>(P, dparams, -1, 0.0, X, XP, cfg.gmin, 1e-12, true, DV, sl);
    __syncwarp();
    bt::assemble<LPI>(P, DV, V, T, sl);
    bt::run_stream<LPI>(P.stream, ring, T - nc, sl, nc + P.n + P.nv + 1);
    bool conv = true, fin = true;
    double ss = 0.0;
    for (int c = sl; c < nc; c += LPI) {
      const double a = T[P.out_pos[c]];
      const double dx = a - X[c];
      ss = fma(dx, dx, ss);
      if (!(fabs(dx) <= cfg.abs_tol + cfg.rel_tol * fabs(a))) conv = false;
      if (!isfinite(a)) fin = false;
    }
    conv = __all_sync(bt::kFull, conv);
    fin = __all_sync(bt::kFull, fin);
    ++iters;
    if (conv) {
      for (int c = sl; c < nc; c += LPI) X[c] = T[P.out_pos[c]];
      __syncwarp();
      return 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(bt::kFull, ss, o);
    const double dxn = sqrt(ss);
    if (dxn > prev && damp > cfg.damping_min) damp = fmax(damp * 0.5, cfg.damping_min);
    prev = dxn;
    for (int c = sl; c < nc; c += LPI) X[c] = fma(damp, T[P.out_pos[c]] - X[c], X[c]);
    __syncwarp();
    if (!fin) return 1;
  }
  return 1;
}

__device__ __forceinline__ void copy_vec(double* dst, const double* src, int n, int sl) {
  for (int i = sl; i < n; i += LPI) dst[i] = src[i];
}

struct Slice {
  int2* ring;  // of the row streams
  double* region;
};

__device__ __forceinline__ Slice warp_slice(const BatchArgs& A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* const s =
      smem_raw + (size_t)(threadIdx.x >> 5) * ((size_t)A.prog_ints * 4 + (size_t)A.region * 8);
  return {reinterpret_cast<int2*>(s), reinterpret_cast<double*>(s + (size_t)A.prog_ints * 4)};
}

// The row stream's entries behind V: 1.0, and the idle lanes' own.
__device__ __forceinline__ void stream_constants(double* c, int sl) {
  if (sl == 0) {
    c[0] = 1.0;
    c[1] = 0.0;
  }
}

__device__ __forceinline__ int next_instance(const BatchArgs& A, int lane) {
  int i = 0;
  if (lane == 0) i = (int)atomicAdd(A.counter, 1u);
  return __shfl_sync(bt::kFull, i, 0);
}

__global__ void k_tran_fwd(BatchArgs A) {
  const int lane = threadIdx.x & 31, sl = lane;
  const Slice S = warp_slice(A);
  while (true) {
    const int inst = next_instance(A, lane);
    if (inst >= A.ninst) return;
    const GroupHdr G = A.groups[A.inst_group[inst]];
    const bt::Prog P = bt::global_view(A, G);
    const int nc = P.nc, n = P.n;
    double* const X = S.region;
    double* const XP = X + nc;
    double* const T = XP + nc;  // T, V and two constants: the row stream's entries
    double* const V = T + n;
    double* const DV = V + P.nv + 2;
    stream_constants(V + P.nv, sl);
    const double* dparams = A.dparams + A.inst_p_off[inst];
    copy_vec(X, A.x0 + A.inst_x0_off[inst], nc, sl);
    double* ck = A.ckpt + A.ckpt_off[inst];
    __syncwarp();
    copy_vec(ck, X, nc, sl);
    const int probe = A.probe[inst];
    double loss = 0.0;
    int iters = 0, reason = 0;
    for (int t = 1; t <= A.steps; ++t) {
      copy_vec(XP, X, nc, sl);
      __syncwarp();
      if (newton_step(A, P, dparams, X, XP, T, DV, V, S.ring, sl, iters)) {
        reason = 1;
        break;
      }
      const double v = X[probe];
      loss = fma(v - A.target, v - A.target, loss);
      if (A.wave && sl == 0) A.wave[(long long)inst * A.steps + (t - 1)] = v;
      if (t % A.ckpt_every == 0) copy_vec(ck + (long long)(t / A.ckpt_every) * nc, X, nc, sl);
      __syncwarp();
    }
    if (sl == 0) {
      A.loss[inst] = reason ? __longlong_as_double(0x7ff8000000000000ll) : loss;
      A.iters_total[inst] = iters;
      A.reason[inst] = reason;
    }
    const long long xo = A.inst_x_off[inst];
    for (int c = sl; c < n; c += LPI) A.x_out[xo + c] = c < nc ? X[c] : 0.0;
    __syncwarp();
  }
}

__global__ void k_tran_bwd(BatchArgs A) {
  const int lane = threadIdx.x & 31, sl = lane;
  const Slice S = warp_slice(A);
  while (true) {
    const int inst = next_instance(A, lane);
    if (inst >= A.ninst) return;
    const GroupHdr G = A.groups[A.inst_group[inst]];
    const bt::Prog P = bt::global_view(A, G);
    const int nc = P.nc, n = P.n, ndev = P.ndev;
    double* const X = S.region;
    double* const XP = X + nc;
    double* const T = XP + nc;  // T, V and two constants: the row streams' entries
    double* const V = T + n;
    double* const DV = V + P.nv + 2;
    double* const LAM = DV + G.ndv;  // lambda_{t+1}, original row order
    double* const GR = LAM + n;      // dL/dC per device
    stream_constants(V + P.nv, sl);
    const double* dparams = A.dparams + A.inst_p_off[inst];
    const double* ck = A.ckpt + A.ckpt_off[inst];
    double* const seg = A.seg + A.seg_off[inst];
    const int probe = A.probe[inst];
    const int K = A.ckpt_every;
    for (int i = sl; i < n; i += LPI) LAM[i] = 0.0;
    for (int d = sl; d < ndev; d += LPI) GR[d] = 0.0;
    int iters = 0, failed = A.reason[inst];
    const int nseg = (A.steps + K - 1) / K;
    for (int s = nseg - 1; s >= 0 && !failed; --s) {
      const int t0 = s * K, t1 = min((s + 1) * K, A.steps);
      // recompute the segment's states from its checkpoint
      copy_vec(X, ck + (long long)s * nc, nc, sl);
      __syncwarp();
      copy_vec(seg, X, nc, sl);
      for (int t = t0 + 1; t <= t1; ++t) {
        copy_vec(XP, X, nc, sl);
        __syncwarp();
        if (newton_step(A, P, dparams, X, XP, T, DV, V, S.ring, sl, iters)) {
          failed = 1;
          break;
        }
        copy_vec(seg + (long long)(t - t0) * nc, X, nc, sl);
        __syncwarp();
      }
      if (failed) break;
      for (int t = t1; t > t0; --t) {
        copy_vec(X, seg + (long long)(t - t0) * nc, nc, sl);
        copy_vec(XP, seg + (long long)(t - 1 - t0) * nc, nc, sl);
        __syncwarp();
        bt::stamp_devices<LPI>(P, dparams, -1, 0.0, X, XP, A.cfg.gmin, 0.0, true, DV, sl);
        __syncwarp();
        bt::assemble<LPI>(P, DV, V, T, sl);
        bt::run_stream<LPI>(P.stream, S.ring, T - nc, sl, nc + n + P.nv + 1);
        // right-hand side dL/dx_t + G_C lambda_{t+1}, in permuted column
        // order: every capacitor's C/dt (lambda_a - lambda_b) as its record's
        // current, the other currents zero, summed by node as the assembly
        // sums a row's currents
        for (int q = sl; q < P.nev; q += LPI) {
          const int4 e = __ldg(P.ev + q);
          const int type = e.z >> 16;
          if (type == 5) {
            const int a = e.y & 0xffff, b = (e.y >> 16) & 0xffff;
            DV[e.w + 1] = __ldg(dparams + 4 * e.x + 1) * (LAM[a] - LAM[b]);
          } else if (type != 0) {  // I, V: the value; D, M, MC: the last of the record
            DV[e.w + bt::record_len(type, true) - 1] = 0.0;
          }
        }
        for (int i = sl; i < n; i += LPI) T[i] = 0.0;
        __syncwarp();
        for (int c = sl; c < nc; c += LPI) {
          const int t0 = P.rmap_ptr[c], t1 = P.rmap_ptr[c + 1];
          if (t1 - t0 > bt::kHeavy) continue;
          double acc = 0.0;
          for (int t = t0; t < t1; ++t) acc += bt::contrib(DV, P.rmap_code[t]);
          T[P.out_pos[c]] = acc;
        }
        for (int h = 0; h < P.nheavy; ++h) {  // the ground and supply rows
          const int code = P.heavy[h];
          if (!(code & 1)) continue;
          int len;
          const int* const cds = bt::list_codes(P, code, len);
          double acc = 0.0;
          for (int t = sl; t < len; t += LPI) acc += bt::contrib(DV, cds[t]);
#pragma unroll
          for (int o = LPI / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(bt::kFull, acc, o);
          if (sl == 0) T[P.out_pos[P.in_row[code >> 1]]] = acc;
        }
        __syncwarp();
        if (sl == 0) T[P.out_pos[probe]] += 2.0 * (X[probe] - A.target);
        bt::run_stream<LPI>(P.tstream, S.ring, T - nc, sl, nc + n + P.nv + 1);
        for (int i = sl; i < n; i += LPI) LAM[P.in_row[i]] = T[i];
        __syncwarp();
        for (int q = P.nev - P.ncap + sl; q < P.nev; q += LPI) {
          const int4 e = __ldg(P.ev + q);
          const int a = e.y & 0xffff, b = (e.y >> 16) & 0xffff;
          const double dv = (X[a] - X[b]) - (XP[a] - XP[b]);
          GR[e.x] = fma(-(LAM[a] - LAM[b]) * dv, A.inv_dt, GR[e.x]);
        }
        __syncwarp();
      }
    }
    double* const go = A.grad + A.grad_off[inst];
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (int d = sl; d < ndev; d += LPI) go[d] = failed ? nan : GR[d];
    if (sl == 0) A.iters[inst] = iters;
    __syncwarp();
  }
}

size_t tran_smem(const BatchArgs& a, int warps_per_block) {
  return (size_t)warps_per_block * ((size_t)a.prog_ints * 4 + (size_t)a.region * 8);
}

}  // namespace

void launch_tran_forward(const BatchArgs& a, int grid, int warps_per_block, cudaStream_t s) {
  k_tran_fwd<<<grid, 32 * warps_per_block, tran_smem(a, warps_per_block), s>>>(a);
}

void launch_tran_backward(const BatchArgs& a, int grid, int warps_per_block, cudaStream_t s) {
  k_tran_bwd<<<grid, 32 * warps_per_block, tran_smem(a, warps_per_block), s>>>(a);
}

void tran_kernel_info(bool backward, int warps_per_block, int region, int prog_ints, int* regs,
                      int* blocks_per_sm) {
  const void* fn = backward ? (const void*)k_tran_bwd : (const void*)k_tran_fwd;
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, fn);
  *regs = fa.numRegs;
  const size_t sm = (size_t)warps_per_block * ((size_t)prog_ints * 4 + (size_t)region * 8);
  if (backward)
    raise_smem_limit<k_tran_bwd>(sm);
  else
    raise_smem_limit<k_tran_fwd>(sm);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, 32 * warps_per_block, sm);
  cudaGetLastError();  // more than a block may have: answered by *blocks_per_sm
}

}  // namespace gk
