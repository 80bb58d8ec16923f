// Kernels of the bordered-block-diagonal (BBD) solver
// (crates/sim-core/src/bbd_solver.rs:633-979, restated for the GPU).
//
// The diagonal blocks form one block-diagonal matrix M that the regular
// factor kernels handle (its BTF finds the blocks). Around them:
//  * reach   - S = B_T - sum_k C_k B_k^-1 R_k through the two sparse halves
//              W = L^-1 P R and Z = U^-T Q^T C^T: one warp per border column
//              (row) of a block, over the elimination path of its entries only;
//              the column's warp then takes the products with the block's Z.
//  * schur   - S = B_T - sum_k Z_k^T W_k, a thread block per border column, the
//              blocks in order (deterministic).
//  * dense LU of S without pivoting, rows and columns in the AMD order of
//              S's structural pattern (the reference factors S with its
//              no-pivot, AMD-ordered SparseLU), in 32-wide panels: panel
//              factor, row-block triangular solve, trailing update in 64x64
//              shared-memory tiles.
//  * the border right-hand side, the R x_T product and the recombination.
#include "kernels.cuh"

namespace gk {
namespace {

__device__ __forceinline__ double perturb_tiny(double d) {  // sparse_lu.rs no-pivot rule
  if (fabs(d) < 1e-14) return d >= 0.0 ? 1e-14 : -1e-14;
  return d;
}

// L and U by rows in the sweeps' order and the pivots' reciprocals.
__global__ void k_bbd_rows(DPlan P, const double* __restrict__ lu, BbdArgs B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.l.nnz) B.l.val[i] = lu[B.l.slot[i]];
  if (i < B.u.nnz) B.u.val[i] = lu[B.u.slot[i]];
  if (i < P.n) B.rec[i] = 1.0 / lu[P.dslot[i]];
}

constexpr int kSweepThreads = 512;

// One block's triangular sweep on v, level by level: a warp per row where the
// level has no more rows than warps, eight lanes per row else. The levels, rows
// and ranges are copied to shared memory first; the next level's entries (four a
// lane) are read while this one's are at work.
__device__ __forceinline__ void sweep_block(const BbdSweep& S, int blk, int sz, const double* rec,
                                            double* v) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kAhead = 4;
  int* const lv = reinterpret_cast<int*>(v + sz);  // at most sz + 1 bounds
  int* const ptr = lv + sz + 1;
  int* const row = ptr + sz + 1;
  const int tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
  const int l0 = S.lvl_ptr[blk], nl = S.lvl_ptr[blk + 1] - l0 - 1;
  const int first = S.lv[l0], rows = S.lv[l0 + nl] - first;
  __syncthreads();  // the sweep before has read its lists
  for (int i = tid; i <= nl; i += blockDim.x) lv[i] = S.lv[l0 + i] - first;
  for (int i = tid; i <= rows; i += blockDim.x) ptr[i] = S.ptr[first + i];
  for (int i = tid; i < rows; i += blockDim.x) row[i] = S.row[first + i];
  __syncthreads();
  int w, i, e, end, c[kAhead];
  double l[kAhead];
  auto fetch = [&](int at, int b) {  // row `at` of the level that ends at row b
    i = at < b ? at : -1;
    e = end = 0;
    if (i >= 0) {
      e = ptr[i] + (lane & (w - 1));
      end = ptr[i + 1];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (e + q * w < end) {
          c[q] = S.col[e + q * w];
          l[q] = S.val[e + q * w];
        }
    }
  };
  auto level = [&](int q, int& a, int& b) {
    a = q < nl ? lv[q] : 0;
    b = q < nl ? lv[q + 1] : 0;
    w = b - a <= nw ? 32 : 8;
  };
  int a, b;
  level(0, a, b);
  fetch(a + tid / w, b);
  for (int q = 0; q < nl; ++q) {
    for (bool more = true; more;) {
      const int ci = i, cw = w, ce = e, cend = end;
      int cc[kAhead];
      double cl[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        cc[u] = c[u];
        cl[u] = l[u];
      }
      const int at = a + tid / w + (nw * 32) / w;  // this level's next rows, or the next level
      more = at - tid / w < b;
      if (more) {
        a += (nw * 32) / w;
        fetch(at, b);
      } else {
        level(q + 1, a, b);
        fetch(a + tid / w, b);
      }
      if (!__any_sync(FULL, ci >= 0)) continue;  // no FP64 from idle warps
      double acc = 0.0;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (ce + u * cw < cend) acc = fma(cl[u], v[cc[u]], acc);
      for (int x = ce + kAhead * cw; x < cend; x += cw) acc = fma(S.val[x], v[S.col[x]], acc);
      if (cw == 32) {
        acc += __shfl_xor_sync(FULL, acc, 16);
        acc += __shfl_xor_sync(FULL, acc, 8);
      }
      acc += __shfl_xor_sync(FULL, acc, 4);
      acc += __shfl_xor_sync(FULL, acc, 2);
      acc += __shfl_xor_sync(FULL, acc, 1);
      if (ci >= 0 && (lane & (cw - 1)) == 0) {
        const int r = row[ci];
        const double x = v[r] - acc;
        v[r] = rec != nullptr ? x * rec[r] : x;
      }
    }
    __syncthreads();
  }
}

// A thread block per block of M. With W and Z of the factorization at hand a solve
// takes each triangle once: forward y = L^-1 P b and Z^T y = C M^-1 b, and when the
// border's solution x is known, backward U^-1 (y - W x). Bounded by the levels'
// latency (the entries' products, the sum across the warp and a barrier). Measured,
// 64 meshes of 30-50 a side: 0.34 and 0.39 ms against 0.61 ms for both triangles at once,
// twice per solve, and 1.43 ms for a warp per block that takes the columns one after
// another, twice.
__global__ void __launch_bounds__(kSweepThreads) k_bbd_forward(DPlan P, BbdArgs B,
                                                               const double* __restrict__ rhs) {
  extern __shared__ double v[];
  const int blk = blockIdx.x, p0 = P.block_ptr[blk], sz = P.block_ptr[blk + 1] - p0;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < sz; i += blockDim.x) v[i] = rhs[B.perm[P.in_row[p0 + i]]];
  sweep_block(B.l, blk, sz, nullptr, v);
  __syncthreads();
  for (int i = tid; i < sz; i += blockDim.x) B.y[p0 + i] = v[i];
  const int r0 = B.row_ptr[blk], nrow = B.row_ptr[blk + 1] - r0;
  const int g0 = B.grp_ptr[blk], g1 = B.grp_ptr[blk + 1];
  for (int g = g0 + (tid >> 5); g < g1; g += blockDim.x >> 5) {
    const int* const zi = B.zpos + B.grp_base[g] + lane;
    const double* const zv = B.zval + B.grp_base[g] + lane;
    double acc = 0.0;
    for (int k = 0; k < B.grp_len[g]; k += 8) {  // a multiple of 8
      int ix[8];
      double zz[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        ix[u] = zi[(k + u) * 32];
        zz[u] = zv[(k + u) * 32];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (ix[u] < sz) acc = fma(zz[u], v[ix[u]], acc);  // (the padding's position is sz)
    }
    const int r = (g - g0) * 32 + lane;
    if (r < nrow) B.zdot[r0 + r] = acc;
  }
}

// bb[j] = rhs[border row j] - the blocks' parts of C M^-1 b, in block order.
__global__ void k_bbd_border(BbdArgs B, const double* __restrict__ rhs, double* bb) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B.bs) return;
  double v = rhs[B.bperm[j]];
  for (int e = B.zref_ptr[j]; e < B.zref_ptr[j + 1]; ++e) v -= B.zdot[B.zref[e]];
  bb[j] = v;
}

__global__ void __launch_bounds__(kSweepThreads) k_bbd_backward(DPlan P, BbdArgs B,
                                                                const double* __restrict__ xT,
                                                                double* x) {
  extern __shared__ double v[];
  const int blk = blockIdx.x, p0 = P.block_ptr[blk], sz = P.block_ptr[blk + 1] - p0;
  const int tid = threadIdx.x;
  for (int i = tid; i < sz; i += blockDim.x) v[i] = B.y[p0 + i];
  __syncthreads();
  // v -= W x, a border column after the other; the next one's first entries are
  // read while this one is subtracted
  const int q1 = B.bw_ptr[blk + 1];
  int nc = -1;
  double nw = 0.0, nx = 0.0;
  long long na = 0;
  int nlen = 0;
  auto ahead = [&](int q) {
    nc = -1;
    if (q >= q1) return;
    const int t = B.bw[q];
    na = B.w.ptr[t];
    nlen = (int)(B.w.ptr[t + 1] - na);
    nx = xT[B.wcol[t]];
    if (tid < nlen) {
      nc = B.w.reach[na + tid] - p0;
      nw = B.wval[na + tid];
    }
  };
  ahead(B.bw_ptr[blk]);
  for (int q = B.bw_ptr[blk]; q < q1; ++q) {
    const int c = nc, len = nlen;
    const double w = nw, xj = nx;
    const long long a = na;
    ahead(q + 1);
    if (c >= 0) v[c] = fma(-w, xj, v[c]);
    for (int i = tid + blockDim.x; i < len; i += blockDim.x) {
      const int r = B.w.reach[a + i] - p0;
      v[r] = fma(-B.wval[a + i], xj, v[r]);
    }
    __syncthreads();
  }
  sweep_block(B.u, blk, sz, B.rec + p0, v);
  __syncthreads();
  for (int i = tid; i < sz; i += blockDim.x) x[B.perm[P.out_col[p0 + i]]] = v[i];
  for (int i = blk * blockDim.x + tid; i < B.bs; i += gridDim.x * blockDim.x)
    x[B.bperm[i]] = xT[i];
}

// kRows: Z, by rows of U; else W, by columns of L, and its products with Z.
// The block's vector v sits in shared memory (kShared) or in scratch. Measured,
// 64 meshes of 30-50 a side and 1025 border nodes (5.9 k columns and rows, 130
// steps each): 0.72 ms against 14.7 ms for Y = B^-1 R on dense tiles of 32
// columns and C Y by one lane per column.
template <bool kRows, bool kShared>
__global__ void k_bbd_reach(DPlan P, const double* __restrict__ lu,
                            const double* __restrict__ ax, BbdArgs B, int stride, int t0, int t1) {
  extern __shared__ double vmem[];
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int gw = blockIdx.x * wpb + w;
  double* const v = kShared ? vmem + (size_t)w * stride : B.scratch + (size_t)gw * stride;
  const BbdTasks& T = kRows ? B.z : B.w;
  const double* const val = kRows ? B.u.val : lu;
  const int* const row = kRows ? B.u.col : P.slot_row;
  for (int q = t0 + gw; q < t1; q += gridDim.x * wpb) {
    const int t = T.order[q];
    const int blk = T.blk[t], p0 = P.block_ptr[blk], sz = P.block_ptr[blk + 1] - p0;
    const int rb = kRows ? 0 : p0;  // U's columns count from the block's first
    for (int i = lane; i <= sz; i += 32) v[i] = 0.0;  // v[sz] pads the products
    __syncwarp();
    if (lane == 0)  // in CSC order (duplicates add in that order)
      for (int e = T.init_ptr[t]; e < T.init_ptr[t + 1]; ++e) v[T.init_pos[e]] += ax[T.init_raw[e]];
    __syncwarp();
    const int* const reach = T.reach + T.ptr[t];
    const int len = (int)(T.ptr[t + 1] - T.ptr[t]);
    double* const out = kRows ? B.zval + B.zout[t] : B.wval + T.ptr[t];
    for (int c0 = 0; c0 < len; c0 += 32) {  // the ranges of 32 steps, one per lane
      int c = 0, qa = 0, qb = 0;
      double rc = 1.0;
      if (c0 + lane < len) {
        c = reach[c0 + lane];
        const int i = kRows ? B.u.at[c] : 0;
        qa = kRows ? B.u.ptr[i] : P.dslot[c] + 1;
        qb = kRows ? B.u.ptr[i + 1] : P.col_ptr[c + 1];
        if (kRows) rc = B.rec[c];
      }
      const int cnt = min(32, len - c0);
      int na, nb, n0, n1;  // the next step's range, first 64 rows and values
      double m0, m1;
      auto fetch = [&](int i) {
        na = __shfl_sync(FULL, qa, i);
        nb = __shfl_sync(FULL, qb, i);
        n0 = n1 = 0;
        m0 = m1 = 0.0;
        if (na + lane < nb) {
          n0 = row[na + lane] - rb;
          m0 = val[na + lane];
        }
        if (na + 32 + lane < nb) {
          n1 = row[na + 32 + lane] - rb;
          m1 = val[na + 32 + lane];
        }
      };
      fetch(0);
      for (int i = 0; i < cnt; ++i) {
        const int a = na, b = nb, i0 = n0, i1 = n1;
        const double l0 = m0, l1 = m1;
        if (i + 1 < cnt) fetch(i + 1);
        double x = v[__shfl_sync(FULL, c, i) - p0];
        if (kRows) x *= __shfl_sync(FULL, rc, i);
        if (lane == 0) out[(long long)(c0 + i) * (kRows ? 32 : 1)] = x;
        if (a + lane < b) v[i0] = fma(-l0, x, v[i0]);
        if (a + 32 + lane < b) v[i1] = fma(-l1, x, v[i1]);
        for (int q = a + 64 + lane; q < b; q += 32) {
          const int r = row[q] - rb;
          v[r] = fma(-val[q], x, v[r]);
        }
        __syncwarp();
      }
    }
    if (kRows) continue;
    const int nrow = B.row_ptr[blk + 1] - B.row_ptr[blk];
    double* const prod = B.gbuf + (B.goff[t] - B.goff[t0]);
    const int g0 = B.grp_ptr[blk], g1 = B.grp_ptr[blk + 1];
    for (int g = g0; g < g1; ++g) {
      const int* const zi = B.zpos + B.grp_base[g] + lane;
      const double* const zv = B.zval + B.grp_base[g] + lane;
      const int glen = B.grp_len[g];  // a multiple of 8
      double s0 = 0.0, s1 = 0.0;
      for (int k = 0; k < glen; k += 8) {
        int ix[8];
        double zz[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          ix[u] = zi[(k + u) * 32];
          zz[u] = zv[(k + u) * 32];
        }
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          s0 = fma(zz[u], v[ix[u]], s0);
          s1 = fma(zz[u + 1], v[ix[u + 1]], s1);
        }
      }
      const int r = (g - g0) * 32 + lane;
      if (r < nrow) prod[r] = s0 + s1;
    }
    __syncwarp();
  }
}

// S column j (column-major, leading dimension bs): B_T entries, then minus the
// products of every block that touches border column j. Warp w sums its blocks
// (every warps-th) in a column of its own, the columns are added in order.
__global__ void k_bbd_schur(const double* __restrict__ ax, BbdArgs B, int j0, double* S) {
  extern __shared__ double scol[];
  const int j = j0 + blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int w = tid >> 5, nw = blockDim.x >> 5;
  double* const col = scol + (size_t)w * B.bs;
  for (int r = tid; r < nw * B.bs; r += blockDim.x) scol[r] = 0.0;
  __syncthreads();
  // B_T, the entries of a row by one warp (the ground's diagonal has thousands)
  for (int q = B.bt_ptr[j] + w; q < B.bt_ptr[j + 1]; q += nw) {
    double v = 0.0;
    for (int e = B.bt_ent[q] + lane; e < B.bt_ent[q + 1]; e += 32) v += ax[B.bt_raw[e]];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) col[B.bt_row[q]] = v;
  }
  __syncwarp();
  const long long g0 = B.goff[B.wref_ptr[j0]];
  for (int t = B.wref_ptr[j] + w; t < B.wref_ptr[j + 1]; t += nw) {
    const int blk = B.w.blk[t], r0 = B.row_ptr[blk];
    const int nrow = B.row_ptr[blk + 1] - r0;
    const double* const g = B.gbuf + (B.goff[t] - g0);
    for (int r = lane; r < nrow; r += 32) col[B.row[r0 + r]] -= g[r];
    __syncwarp();
  }
  __syncthreads();
  for (int r = tid; r < B.bs; r += blockDim.x) {
    double v = scol[r];
    for (int q = 1; q < nw; ++q) v += scol[(size_t)q * B.bs + r];
    S[(long long)j * B.bs + r] = v;
  }
}

// Panel factorisation of columns [k0, k0+nb) over rows k0..bs-1.
// Panel factorization of columns [k0, k0+nb) in two launches: k_dlu_diag
// factors the nb x nb diagonal block in place (shared memory, one lane per
// row, columns in order); k_dlu_panel then eliminates every row below it
// against that block's U, one thread per row, column by column. Every element
// sees the operations of a column-by-column panel in the same order, so the
// factor is the same bit for bit.
__global__ void k_dlu_diag(double* S, int bs, int k0, int nb) {
  __shared__ double D[32][33];  // D[r][c] = S(k0 + r, k0 + c)
  const int r = threadIdx.x;
  for (int c = 0; c < nb; ++c)
    if (r < nb) D[r][c] = S[(long long)(k0 + c) * bs + k0 + r];
  __syncwarp();
  for (int c = 0; c < nb; ++c) {
    const double d = perturb_tiny(D[c][c]);
    __syncwarp();
    if (r == c) D[c][c] = d;
    if (r > c && r < nb) {
      const double l = D[r][c] / d;
      D[r][c] = l;
      for (int c2 = c + 1; c2 < nb; ++c2) D[r][c2] = fma(-l, D[c][c2], D[r][c2]);
    }
    __syncwarp();
  }
  for (int c = 0; c < nb; ++c)
    if (r < nb) S[(long long)(k0 + c) * bs + k0 + r] = D[r][c];
}

__global__ void __launch_bounds__(256) k_dlu_panel(double* S, int bs, int k0, int nb) {
  __shared__ double D[32][33];  // the factored diagonal block
  for (int q = threadIdx.x; q < nb * nb; q += blockDim.x) {
    const int c = q / nb, r = q % nb;
    D[r][c] = S[(long long)(k0 + c) * bs + k0 + r];
  }
  __syncthreads();
  const int r = k0 + nb + blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= bs) return;
  double a[32];
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c < nb) a[c] = S[(long long)(k0 + c) * bs + r];
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    if (c < nb) {
      const double l = a[c] / D[c][c];
      a[c] = l;
#pragma unroll
      for (int c2 = c + 1; c2 < 32; ++c2)
        if (c2 < nb) a[c2] = fma(-l, D[c][c2], a[c2]);
    }
  }
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c < nb) S[(long long)(k0 + c) * bs + r] = a[c];
}

// U12 = L11^-1 A12 for the rows of the panel, one thread per column, L11 in
// shared memory.
__global__ void k_dlu_trsm(double* S, int bs, int k0, int nb) {
  __shared__ double L[32][33];  // L[i][m] = S(k0 + i, k0 + m)
  for (int q = threadIdx.x; q < nb * nb; q += blockDim.x) {
    const int m = q / nb, i = q % nb;
    L[i][m] = S[(long long)(k0 + m) * bs + k0 + i];
  }
  __syncthreads();
  const int j = k0 + nb + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= bs) return;
  double* const col = S + (long long)j * bs;
  for (int i = 1; i < nb; ++i) {
    double v = col[k0 + i];
    for (int m = 0; m < i; ++m) v = fma(-L[i][m], col[k0 + m], v);
    col[k0 + i] = v;
  }
}

// A22 -= L21 U12 on 64x64 tiles; 256 threads, 4x4 outputs each.
__global__ void k_dlu_update(double* S, int bs, int k0, int nb) {
  __shared__ double Ls[32][65], Us[32][65];
  const int r0 = k0 + nb + blockIdx.y * 64, c0 = k0 + nb + blockIdx.x * 64;
  const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16;
  for (int q = tid; q < 64 * nb; q += 256) {
    const int m = q / 64, i = q % 64;
    const int r = r0 + i, c = c0 + i;
    Ls[m][i] = r < bs ? S[(long long)(k0 + m) * bs + r] : 0.0;
    Us[m][i] = c < bs ? S[(long long)c * bs + k0 + m] : 0.0;
  }
  __syncthreads();
  double acc[4][4] = {};
  for (int m = 0; m < nb; ++m) {
    double a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a[u] = Ls[m][tr * 4 + u];
      b[u] = Us[m][tc * 4 + u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = r0 + tr * 4 + u, c = c0 + tc * 4 + v;
      if (r < bs && c < bs) S[(long long)c * bs + r] -= acc[u][v];
    }
}

// x <- S^-1 x with the unit-lower / upper factors, one block, in panels of 32
// columns. While the other warps subtract a finished panel from the rows beyond,
// the first warp subtracts it from the next panel's 32 rows (one per lane) and
// solves that panel's triangle, its values shuffled. Bounded by FP64 issue on one
// SM (a million multiply-adds for 1025 rows: 250 us); 0.47 ms against 1.4 ms
// with two barriers per column.
constexpr int kDluThreads = 512;
__global__ void __launch_bounds__(kDluThreads) k_dlu_solve(const double* __restrict__ S, int bs,
                                                           double* x) {
  extern __shared__ double xs[];  // x[bs]
  constexpr unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int r = tid; r < bs; r += blockDim.x) xs[r] = x[r];
  __syncthreads();
  const int np = (bs + 31) / 32;
  // row r less panel p's columns
  auto update = [&](int r, int p) {
    const int k0 = 32 * p, nb = min(32, bs - k0);
    const double* const col = S + (long long)k0 * bs + r;
    double v = xs[r];
    if (nb == 32) {
#pragma unroll 16
      for (int c = 0; c < 32; ++c) v = fma(-col[(long long)c * bs], xs[k0 + c], v);
    } else {
      for (int c = 0; c < nb; ++c) v = fma(-col[(long long)c * bs], xs[k0 + c], v);
    }
    return v;
  };
  for (int p = -1; p < np - 1; ++p) {  // panel p is final
    const int n0 = 32 * (p + 1);
    if (tid < 32) {
      const int r = n0 + lane;
      double l[32];
#pragma unroll
      for (int c = 0; c < 32; ++c)
        l[c] = c < lane && r < bs ? S[(long long)(n0 + c) * bs + r] : 0.0;
      double v = r >= bs ? 0.0 : p >= 0 ? update(r, p) : xs[r];
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const double t = fma(-l[c], __shfl_sync(FULL, v, c), v);
        if (lane > c) v = t;
      }
      if (r < bs) xs[r] = v;
    } else if (p >= 0) {
      for (int r = n0 + tid; r < bs; r += blockDim.x - 32) xs[r] = update(r, p);
    }
    __syncthreads();
  }
  for (int p = np; p > 0; --p) {
    const int n0 = 32 * (p - 1);
    if (tid < 32) {
      const int r = n0 + lane;
      double u[32];
#pragma unroll
      for (int c = 0; c < 32; ++c)
        u[c] = lane < c && n0 + c < bs ? S[(long long)(n0 + c) * bs + r] : 0.0;
      const double rc = r < bs ? 1.0 / S[(long long)r * bs + r] : 0.0;
      double v = r >= bs ? 0.0 : p < np ? update(r, p) : xs[r];
#pragma unroll
      for (int c = 31; c >= 0; --c) {
        if (lane == c) v *= rc;
        const double t = fma(-u[c], __shfl_sync(FULL, v, c), v);
        if (lane < c) v = t;
      }
      if (r < bs) xs[r] = v;
    } else if (p < np) {
      for (int r = tid - 32; r < n0; r += blockDim.x - 32) xs[r] = update(r, p);
    }
    __syncthreads();
  }
  for (int r = tid; r < bs; r += blockDim.x) x[r] = xs[r];
}

// bb[j] = rhs[border row j] - sum_c C[j][c] z[c], a warp per border row (the
// ground row has thousands of entries).
__global__ void k_bbd_border_rhs(const double* __restrict__ ax, const double* __restrict__ rhs,
                                 const double* __restrict__ z, BbdArgs B, double* bb) {
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= B.bs) return;
  double v = 0.0;
  for (int e = B.crow_ptr[j] + lane; e < B.crow_ptr[j + 1]; e += 32)
    v = fma(ax[B.crow_raw[e]], z[B.crow_col[e]], v);
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  if (lane == 0) bb[j] = rhs[B.bperm[j]] - v;
}

// w[m] = sum_j R[m][j] xT[j] over the rows of M
__global__ void k_bbd_rmatvec(const double* __restrict__ ax, const double* __restrict__ xT,
                              BbdArgs B, double* w) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= B.border_start) return;
  double v = 0.0;
  for (int e = B.rrow_ptr[m]; e < B.rrow_ptr[m + 1]; ++e)
    v = fma(ax[B.rrow_raw[e]], xT[B.rrow_col[e]], v);
  w[m] = v;
}

__global__ void k_gather(double* dst, const double* __restrict__ src,
                         const int* __restrict__ idx, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

__global__ void k_bbd_combine(const double* __restrict__ z, const double* __restrict__ w2,
                              const double* __restrict__ xT, BbdArgs B, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.border_start)
    x[B.perm[i]] = z[i] - w2[i];
  else if (i < B.border_start + B.bs)
    x[B.bperm[i - B.border_start]] = xT[i - B.border_start];
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace

namespace {
// Warps per block of the reach kernels with their vectors in shared memory: two
// (five blocks of 50 x 50 meshes share an SM), one, or none.
int reach_warps(int max_block) {
  const size_t one = (size_t)8 * ((max_block + 2) & ~1);
  return 2 * one <= (size_t)(226 * 1024) ? 2 : one <= (size_t)(226 * 1024) ? 1 : 0;
}
template <bool kRows>
void launch_reach(const DPlan& P, const double* lu, const double* ax, const BbdArgs& B, int t0,
                  int t1, cudaStream_t s) {
  if (t1 <= t0) return;
  const int stride = (B.max_block + 2) & ~1, wpb = reach_warps(B.max_block);
  if (wpb > 0) {
    const int bytes = wpb * stride * 8;
    raise_smem_limit<k_bbd_reach<kRows, true>>(bytes);
    k_bbd_reach<kRows, true>
        <<<cdiv(t1 - t0, wpb), 32 * wpb, bytes, s>>>(P, lu, ax, B, stride, t0, t1);
  } else {
    k_bbd_reach<kRows, false>
        <<<bbd_scratch_warps() / 4, 128, 0, s>>>(P, lu, ax, B, stride, t0, t1);
  }
}
}  // namespace

bool bbd_shared_fits(int max_block) { return reach_warps(max_block) > 0; }
namespace {
size_t bbd_solve_bytes(int max_block) { return (size_t)20 * max_block + 16; }
}  // namespace
bool bbd_solve_fits(int max_block) { return bbd_solve_bytes(max_block) <= (size_t)(226 * 1024); }
int bbd_scratch_warps() { return 1024; }

void launch_bbd_z(const DPlan& P, const double* lu, const double* ax, const BbdArgs& B,
                  cudaStream_t s) {
  int m = P.n;
  if (B.l.nnz > m) m = B.l.nnz;
  if (B.u.nnz > m) m = B.u.nnz;
  if (m > 0) k_bbd_rows<<<cdiv(m, 256), 256, 0, s>>>(P, lu, B);
  launch_reach<true>(P, lu, ax, B, 0, B.z.n, s);
}

void launch_bbd_forward(const DPlan& P, const BbdArgs& B, const double* rhs, double* bb,
                        cudaStream_t s) {
  const int bytes = (int)bbd_solve_bytes(B.max_block);
  raise_smem_limit<k_bbd_forward>(bytes);
  k_bbd_forward<<<P.nblocks, kSweepThreads, bytes, s>>>(P, B, rhs);
  k_bbd_border<<<cdiv(B.bs, 128), 128, 0, s>>>(B, rhs, bb);
}

void launch_bbd_backward(const DPlan& P, const BbdArgs& B, const double* xT, double* x,
                         cudaStream_t s) {
  const int bytes = (int)bbd_solve_bytes(B.max_block);
  raise_smem_limit<k_bbd_backward>(bytes);
  k_bbd_backward<<<P.nblocks, kSweepThreads, bytes, s>>>(P, B, xT, x);
}

void launch_bbd_schur(const DPlan& P, const double* lu, const double* ax, const BbdArgs& B, int j0,
                      int j1, int t0, int t1, double* S, cudaStream_t s) {
  launch_reach<false>(P, lu, ax, B, t0, t1, s);
  int nw = 8;  // warps, a column of S each
  while (nw > 1 && nw * B.bs * 8 > 100 * 1024) nw >>= 1;
  const int bytes = nw * B.bs * 8;
  raise_smem_limit<k_bbd_schur>(bytes);
  k_bbd_schur<<<j1 - j0, 32 * nw, bytes, s>>>(ax, B, j0, S);
}

void launch_dense_lu(double* S, int bs, cudaStream_t s) {
  const int nb = 32;
  for (int k0 = 0; k0 < bs; k0 += nb) {
    const int w = bs - k0 < nb ? bs - k0 : nb;
    const int rest = bs - k0 - w;
    k_dlu_diag<<<1, 32, 0, s>>>(S, bs, k0, w);
    if (rest <= 0) break;
    k_dlu_panel<<<cdiv(rest, 256), 256, 0, s>>>(S, bs, k0, w);
    k_dlu_trsm<<<cdiv(rest, 128), 128, 0, s>>>(S, bs, k0, w);
    dim3 g(cdiv(rest, 64), cdiv(rest, 64));
    k_dlu_update<<<g, 256, 0, s>>>(S, bs, k0, w);
  }
}

void launch_dense_lu_solve(const double* S, int bs, double* x, cudaStream_t s) {
  raise_smem_limit<k_dlu_solve>((size_t)bs * 8);
  k_dlu_solve<<<1, kDluThreads, bs * 8, s>>>(S, bs, x);
}

void launch_bbd_border_rhs(const double* ax, const double* rhs, const double* z,
                           const BbdArgs& B, double* bb, cudaStream_t s) {
  k_bbd_border_rhs<<<cdiv(B.bs, 4), 128, 0, s>>>(ax, rhs, z, B, bb);
}

void launch_bbd_rmatvec(const double* ax, const double* xT, const BbdArgs& B, double* w,
                        cudaStream_t s) {
  if (B.border_start > 0) k_bbd_rmatvec<<<cdiv(B.border_start, 128), 128, 0, s>>>(ax, xT, B, w);
}

void launch_gather(double* dst, const double* src, const int* idx, int n, cudaStream_t s) {
  if (n > 0) k_gather<<<cdiv(n, 256), 256, 0, s>>>(dst, src, idx, n);
}

void launch_bbd_combine(const double* z, const double* w2, const double* xT, const BbdArgs& B,
                        double* x, cudaStream_t s) {
  const int n = B.border_start + B.bs;
  k_bbd_combine<<<cdiv(n, 256), 256, 0, s>>>(z, w2, xT, B, x);
}

}  // namespace gk
