// AC small-signal sweep over many frequencies at once (the reference's .ac:
// crates/sim-core/src/engine.rs:829-930, complex_solver.rs:28-144).
//
// Y(w) = G + jwC is filled cell by cell (G from the DC stamp at the operating
// point, the capacitor terms +-w*C in insertion order), then the reference's
// dense LU with partial pivoting and its back substitution run on it. Complex
// arithmetic is num-complex's (0.4.6): a*b = (ar br - ai bi, ar bi + ai br),
// a/b = ((ar br + ai bi)/n, (ai br - ar bi)/n) with n = br^2 + bi^2, |a| =
// hypot(ar, ai). Compiled without contraction, so the solutions match a scalar
// evaluation of the dense algorithm bit for bit wherever the magnitudes that
// pick the pivots agree.
//
// k_ac_sparse does only the operations of that dense LU that can change a
// value. An entry nothing has been added to is +0.0, and subtracting a
// product with such an entry leaves a finite operand as it is (a zero's sign
// aside), so per column k only the rows with an entry in it and the columns
// of the pivot row are touched. Which they are depends on the pivots, so the
// structure is kept at run time: one bit per entry by rows and one by
// columns. A frequency whose factors, pivot rows, right-hand side or solution
// hold an infinity or NaN (0 * inf is NaN, so a skipped product would have
// mattered) is done again by ac_point, the dense algorithm as it stands.
// Rows are not moved: pos / phys carry the exchanges.
//
// What bounds it: FP64 issue (a warp instruction per 64 cycles and SM
// sub-partition, whatever the active lanes) - about 25 for the candidates'
// hypot, 27 for the multipliers' division, 8 per 32 updated entries - so a
// frequency gets one warp where there are frequencies enough to fill the SMs,
// more where there are few. Candidates within a factor two of the largest
// component alone are contenders for the pivot (hypot is at most sqrt(2)
// times the larger component), and only two or more of them need a hypot.
// Measured against the dense sweep this replaces (every entry, one block per
// frequency): 4501 frequencies of the 103-node ladder 70.7 -> 2.7 ms, 226 of
// the 326-node grid 70.5 -> 3.0 ms.
#include <algorithm>

#include "kernels.cuh"

namespace gk {
namespace {

struct Cx {
  double re, im;
};
__device__ __forceinline__ Cx csub(Cx a, Cx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ Cx cmul(Cx a, Cx b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ Cx cdiv(Cx a, Cx b) {
  const double n = b.re * b.re + b.im * b.im;
  const double re = a.re * b.re + a.im * b.im;
  const double im = a.im * b.re - a.re * b.im;
  return {re / n, im / n};
}

// One frequency by the dense algorithm: M the n x n system (row-major, in
// global memory), x, pr, bv, bi in shared memory.
__device__ void ac_point(const AcArgs& A, long long f, Cx* M, Cx* x, Cx* pr, double* bv,
                         int* bi, int& s_fail) {
  const int n = A.n, tid = threadIdx.x, nt = blockDim.x;
  const double omega = 2.0 * 3.141592653589793 * A.freqs[f];
  for (int q = tid; q < n * n; q += nt) M[q] = Cx{0.0, 0.0};
  if (tid == 0) s_fail = 0;
  __syncthreads();
  for (int c = tid; c < A.ncell; c += nt) {  // each cell's terms in insertion order
    double re = 0.0, im = 0.0;
    for (int t = A.re_ptr[c]; t < A.re_ptr[c + 1]; ++t) re = re + A.ax[A.re_idx[t]];
    for (int t = A.im_ptr[c]; t < A.im_ptr[c + 1]; ++t) {
      const int code = A.im_code[t];
      const double y = omega * A.cap[code >> 1];
      im = im + ((code & 1) ? -y : y);
    }
    M[(size_t)A.cell_row[c] * n + A.cell_col[c]] = Cx{re, im};
  }
  if (tid == 0) M[0] = Cx{1.0, 0.0};  // ground row: 1 on the diagonal
  for (int i = tid; i < n; i += nt) x[i] = i == 0 ? Cx{0.0, 0.0} : Cx{A.rhs[2 * i], A.rhs[2 * i + 1]};
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    // the first row of largest magnitude in column k, from row k down: row k's
    // own unless another beats it (nothing beats a NaN)
    const Cx v0 = M[(size_t)k * n + k];
    double best = hypot(v0.re, v0.im);
    int brow = k;
    for (int i = k + 1 + tid; i < n; i += nt) {
      const Cx v = M[(size_t)i * n + k];
      const double m = hypot(v.re, v.im);
      if (m > best) {
        best = m;
        brow = i;
      }
    }
    bv[tid] = best;
    bi[tid] = brow;
    __syncthreads();
    for (int s = nt / 2; s > 0; s >>= 1) {
      if (tid < s) {
        const double ov = bv[tid + s];
        const int oi = bi[tid + s];
        if (ov > bv[tid] || (ov == bv[tid] && oi < bi[tid])) {
          bv[tid] = ov;
          bi[tid] = oi;
        }
      }
      __syncthreads();
    }
    const int mr = bi[0];
    __syncthreads();
    if (mr != k) {
      for (int j = tid; j < n; j += nt) {
        const Cx t = M[(size_t)k * n + j];
        M[(size_t)k * n + j] = M[(size_t)mr * n + j];
        M[(size_t)mr * n + j] = t;
      }
      if (tid == 0) {
        const Cx t = x[k];
        x[k] = x[mr];
        x[mr] = t;
      }
      __syncthreads();
    }
    const Cx piv = M[(size_t)k * n + k];
    if (hypot(piv.re, piv.im) < 1e-30) {
      if (tid == 0) s_fail = 1;
      break;
    }
    for (int i = k + 1 + tid; i < n; i += nt) M[(size_t)i * n + k] = cdiv(M[(size_t)i * n + k], piv);
    __syncthreads();
    const int w = n - k - 1;
    for (int q = tid; q < w * (w + 1); q += nt) {  // (w rows) x (w columns + the rhs)
      const int i = k + 1 + q / (w + 1), jj = q % (w + 1);
      const Cx fct = M[(size_t)i * n + k];
      if (jj < w) {
        const int j = k + 1 + jj;
        M[(size_t)i * n + j] = csub(M[(size_t)i * n + j], cmul(fct, M[(size_t)k * n + j]));
      } else {
        x[i] = csub(x[i], cmul(fct, x[k]));
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (!s_fail) {
    for (int i = n - 1; i >= 0; --i) {  // back substitution, terms in ascending order
      for (int j = i + 1 + tid; j < n; j += nt) pr[j] = cmul(M[(size_t)i * n + j], x[j]);
      __syncthreads();
      if (tid == 0) {
        Cx v = x[i];
        for (int j = i + 1; j < n; ++j) v = csub(v, pr[j]);
        const Cx piv = M[(size_t)i * n + i];
        if (hypot(piv.re, piv.im) < 1e-30)
          s_fail = 1;
        else
          x[i] = cdiv(v, piv);
      }
      __syncthreads();
      if (s_fail) break;
    }
  }
  if (s_fail) {
    if (tid == 0) atomicExch(A.status, 1);
    __syncthreads();
    return;
  }
  for (int i = tid; i < n; i += nt) {
    A.out_re[f * n + i] = x[i].re;
    A.out_im[f * n + i] = x[i].im;
  }
  __syncthreads();
}

__device__ __forceinline__ unsigned abs_hi(double v) {
  return (unsigned)__double2hiint(v) & 0x7fffffffu;
}
__device__ __forceinline__ unsigned mag_hi(double2 v) { return max(abs_hi(v.x), abs_hi(v.y)); }
constexpr unsigned kInfHi = 0x7ff00000u;  // high word of an infinity; NaNs are above
__device__ __forceinline__ bool finite2(double2 v) { return mag_hi(v) < kInfHi; }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) {
  const Cx r = cmul(Cx{a.x, a.y}, Cx{b.x, b.y});
  return make_double2(r.re, r.im);
}

// Indices of the set bits of word(w), w in [w0, nw), into list, by one warp;
// returns how many.
template <class Word>
__device__ __forceinline__ int list_bits(int w0, int nw, unsigned short* list, Word word) {
  const int lane = threadIdx.x & 31;
  int cnt = 0;
  for (int w = w0; w < nw; ++w) {
    const unsigned v = word(w);
    if ((v >> lane) & 1u)
      list[cnt + __popc(v & ((1u << lane) - 1u))] = (unsigned short)(w * 32 + lane);
    cnt += __popc(v);
  }
  __syncwarp();
  return cnt;
}

struct AcStep {     // what warp 0 finds for column k
  double2 piv;
  int row, nr, nc;  // the pivot's row, the other rows with an entry, the pivot row's columns
  int stop;         // 1: pivot below 1e-30, 2: a non-finite value
};

// One frequency per pass of the block (blockDim.x = 32 * warps). Shared: x
// (right-hand side by row), f (column k, then the multipliers; at the end the
// solution), u (the pivot row's values / products) [n] double2 each; pos,
// phys, rl, cl [n] u16 each; act [nw]; and the bit masks rm, cm [n][nw] where
// masks_shared, else they sit in the block's slice of A.masks.
__global__ void __launch_bounds__(256) k_ac_sparse(AcArgs A, int nf, int masks_shared) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = A.n, nw = (n + 31) >> 5, tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  double2* const x = reinterpret_cast<double2*>(smem_raw);
  double2* const f = x + n;
  double2* const u = f + n;
  unsigned short* const pos = reinterpret_cast<unsigned short*>(u + n);
  unsigned short* const phys = pos + n;
  unsigned short* const rl = phys + n;
  unsigned short* const cl = rl + n;
  unsigned* const act = reinterpret_cast<unsigned*>(cl + n);
  unsigned* const rm = masks_shared ? act + nw : A.masks + (size_t)blockIdx.x * 2 * n * nw;
  unsigned* const cm = rm + (size_t)n * nw;
  double2* const M = reinterpret_cast<double2*>(A.scratch) + (size_t)blockIdx.x * n * n;
  __shared__ AcStep S;
  __shared__ int s_bad, s_fail;
  for (long long fq = blockIdx.x; fq < nf; fq += gridDim.x) {
    const double omega = 2.0 * 3.141592653589793 * A.freqs[fq];
    for (int q = tid; q < 2 * n * nw; q += nt) rm[q] = A.masks0[q];
    for (int w = tid; w < nw; w += nt)
      act[w] = w + 1 < nw || (n & 31) == 0 ? 0xffffffffu : (1u << (n & 31)) - 1u;
    for (int i = tid; i < n; i += nt) {
      pos[i] = phys[i] = (unsigned short)i;
      x[i] = i == 0 ? make_double2(0.0, 0.0) : make_double2(A.rhs[2 * i], A.rhs[2 * i + 1]);
    }
    for (int c = tid; c < A.ncell; c += nt) {  // each cell's terms in insertion order
      double re = 0.0, im = 0.0;
      for (int t = A.re_ptr[c]; t < A.re_ptr[c + 1]; ++t) re = re + A.ax[A.re_idx[t]];
      for (int t = A.im_ptr[c]; t < A.im_ptr[c + 1]; ++t) {
        const int code = A.im_code[t];
        const double y = omega * A.cap[code >> 1];
        im = im + ((code & 1) ? -y : y);
      }
      M[(size_t)A.cell_row[c] * n + A.cell_col[c]] = make_double2(re, im);
    }
    if (tid == 0) {
      M[0] = make_double2(1.0, 0.0);  // ground row: 1 on the diagonal
      s_bad = 0;
    }
    __syncthreads();
    int stop = 0;
    for (int k = 0; k < n; ++k) {
      if (warp == 0) {
        int nr = list_bits(0, nw, rl, [&](int w) { return cm[(size_t)k * nw + w] & act[w]; });
        unsigned big = 0;
        for (int t = lane; t < nr; t += 32) {
          const double2 v = M[(size_t)rl[t] * n + k];
          f[t] = v;
          big = max(big, mag_hi(v));
        }
        big = __reduce_max_sync(0xffffffffu, big);
        int st = 0, tp = -1;
        if (big >= kInfHi) {
          st = 2;
        } else if (nr == 0) {
          st = 1;
        } else {
          // 0x39d00000 is the high word of a value above 4e-30: below it a
          // pivot may fail the 1e-30 test, so every magnitude is computed
          const bool all = big < 0x39d00000u;
          int cnt = 0;
          for (int t0 = 0; t0 < nr; t0 += 32) {
            const int t = t0 + lane;
            const unsigned b = __ballot_sync(
                0xffffffffu, t < nr && (all || mag_hi(f[t < nr ? t : 0]) + 0x00100000u >= big));
            if (b && tp < 0) tp = t0 + __ffs(b) - 1;
            cnt += __popc(b);
          }
          if (cnt > 1 || all) {  // the first row (by position) of largest magnitude
            unsigned long long best = 0;
            unsigned bp = 0xffffffffu;
            for (int t = lane; t < nr; t += 32) {
              const double2 v = f[t];
              if (!all && mag_hi(v) + 0x00100000u < big) continue;
              const unsigned long long m = (unsigned long long)__double_as_longlong(hypot(v.x, v.y));
              const unsigned p = pos[rl[t]];
              if (bp == 0xffffffffu || m > best || (m == best && p < bp)) {
                best = m;
                bp = p;
              }
            }
            const bool has = bp != 0xffffffffu;
            const unsigned hi = __reduce_max_sync(0xffffffffu, has ? (unsigned)(best >> 32) : 0u);
            const bool e1 = has && (unsigned)(best >> 32) == hi;
            const unsigned lo = __reduce_max_sync(0xffffffffu, e1 ? (unsigned)best : 0u);
            const bool e2 = e1 && (unsigned)best == lo;
            bp = __reduce_min_sync(0xffffffffu, e2 ? bp : 0xffffffffu);
            const double m = __hiloint2double((int)hi, (int)lo);
            if (m < 1e-30) st = 1;
            for (int t0 = 0; t0 < nr; t0 += 32) {
              const int t = t0 + lane;
              const unsigned b = __ballot_sync(0xffffffffu, t < nr && pos[rl[t < nr ? t : 0]] == bp);
              if (b) tp = t0 + __ffs(b) - 1;
            }
          }
        }
        int nc = 0, row = 0;
        if (st == 0) {
          row = rl[tp];
          const double2 piv = f[tp];
          __syncwarp();
          if (lane == 0) {
            rl[tp] = rl[nr - 1];  // the pivot leaves the list
            f[tp] = f[nr - 1];
            const int at = pos[row], old = phys[k];
            phys[at] = (unsigned short)old;
            pos[old] = (unsigned short)at;
            phys[k] = (unsigned short)row;
            pos[row] = (unsigned short)k;
            act[row >> 5] &= ~(1u << (row & 31));
            S.piv = piv;
            S.row = row;
            S.nr = nr - 1;
          }
          const int wk = (k + 1) >> 5;
          nc = list_bits(wk, nw, cl, [&](int w) {
            const unsigned v = rm[(size_t)row * nw + w];
            return w == wk ? v & (0xffffffffu << ((k + 1) & 31)) : v;
          });
        }
        if (lane == 0) {
          S.nc = nc;
          S.stop = st;
        }
      }
      __syncthreads();
      stop = S.stop;
      if (stop) break;
      const int nr = S.nr, nc = S.nc, row = S.row;
      const double2 piv = S.piv;
      bool bad = false;
      for (int t = tid; t < nr; t += nt) {
        const double2 v = f[t];
        const Cx q = cdiv(Cx{v.x, v.y}, Cx{piv.x, piv.y});
        f[t] = make_double2(q.re, q.im);
        bad |= !finite2(f[t]);
      }
      for (int j = tid; j < nc; j += nt) {
        u[j] = M[(size_t)row * n + cl[j]];
        bad |= !finite2(u[j]);
      }
      if (tid == 0) bad |= !finite2(x[row]);
      if (bad) s_bad = 1;
      __syncthreads();
      if (s_bad) break;
      // rows x (the pivot row's columns and the right-hand side): L lanes of
      // a warp take a row's columns, so few columns leave no lane idle
      int sh = 0;
      while (sh < 5 && (1 << sh) < nc + 1) ++sh;
      const double2 xk = x[row];
      for (int t = tid >> sh; t < nr; t += nt >> sh) {
        const int i = rl[t];
        const double2 ft = f[t];
        for (int j = tid & ((1 << sh) - 1); j <= nc; j += 1 << sh) {
          const bool rhs = j == nc;
          const int c = rhs ? 0 : cl[j];
          double2* const p = rhs ? x + i : M + (size_t)i * n + c;
          const bool has = rhs || ((rm[(size_t)i * nw + (c >> 5)] >> (c & 31)) & 1u);
          const double2 old = has ? *p : make_double2(0.0, 0.0);
          const double2 m = mul2(ft, rhs ? xk : u[j]);
          *p = make_double2(old.x - m.x, old.y - m.y);
        }
      }
      __syncthreads();
      // the rows' new entries
      const int wk = (k + 1) >> 5, words = nw - wk;
      for (int q = tid; q < nr * words; q += nt) {
        const int t = q / words, w = wk + q % words;
        const unsigned v = rm[(size_t)row * nw + w];
        rm[(size_t)rl[t] * nw + w] |= w == wk ? v & (0xffffffffu << ((k + 1) & 31)) : v;
      }
      for (int q = tid; q < nc * nw; q += nt) {
        const int j = q / nw, w = q % nw;
        cm[(size_t)cl[j] * nw + w] |= cm[(size_t)k * nw + w] & act[w];
      }
      __syncthreads();
    }
    if (warp == 0 && !stop && !s_bad) {
      // back substitution, terms in ascending order: the products of a row by
      // the lanes, the differences one after another (lane 0 the real parts,
      // lane 1 the imaginary ones), f the solution by column. The row's
      // columns and values are fetched one row ahead.
      bool bad = false;
      auto columns = [&](int i) {
        const int r = phys[i], wi = (i + 1) >> 5;
        return list_bits(wi, nw, rl, [&](int w) {
          const unsigned v = rm[(size_t)r * nw + w];
          return w == wi ? v & (0xffffffffu << ((i + 1) & 31)) : v;
        });
      };
      int cnt = columns(n - 1), c0 = 0, c1 = 0;
      double2 m0, m1, dg, xr;
      auto fetch = [&](int i) {
        const double2* const row = M + (size_t)phys[i] * n;
        c0 = lane < cnt ? rl[lane] : 0;
        c1 = lane + 32 < cnt ? rl[lane + 32] : 0;
        m0 = lane < cnt ? row[c0] : make_double2(0.0, 0.0);
        m1 = lane + 32 < cnt ? row[c1] : make_double2(0.0, 0.0);
        dg = row[i];
        xr = x[phys[i]];
      };
      fetch(n - 1);
      for (int i = n - 1; i >= 0; --i) {
        const int ccnt = cnt;
        const double2 cdg = dg, cx = xr;
        if (lane < cnt) u[lane] = mul2(m0, f[c0]);
        if (lane + 32 < cnt) u[lane + 32] = mul2(m1, f[c1]);
        for (int t = lane + 64; t < cnt; t += 32)
          u[t] = mul2(M[(size_t)phys[i] * n + rl[t]], f[rl[t]]);
        __syncwarp();
        if (i > 0) {
          cnt = columns(i - 1);
          fetch(i - 1);
        }
        const int h = lane & 1;
        double v = h ? cx.y : cx.x;
        const double* const pr = reinterpret_cast<const double*>(u) + h;
#pragma unroll 4
        for (int t = 0; t < ccnt; ++t) v = v - pr[2 * t];
        const double o = __shfl_xor_sync(0xffffffffu, v, 1);
        const double nn = cdg.x * cdg.x + cdg.y * cdg.y;
        const double p = v * cdg.x, q = o * cdg.y;
        const double s = (h ? p - q : p + q) / nn;
        bad |= abs_hi(s) >= kInfHi;
        if (lane < 2) reinterpret_cast<double*>(f + i)[h] = s;
        __syncwarp();
      }
      if (__any_sync(0xffffffffu, bad) && lane == 0) s_bad = 1;
    }
    __syncthreads();
    if (s_bad || stop == 2) {  // as the dense algorithm has it, from the start
      double* const bv = reinterpret_cast<double*>(u);
      ac_point(A, fq, reinterpret_cast<Cx*>(M), reinterpret_cast<Cx*>(x),
               reinterpret_cast<Cx*>(f), bv, reinterpret_cast<int*>(bv + nt), s_fail);
      __syncthreads();
      continue;
    }
    if (stop) {
      if (tid == 0) atomicExch(A.status, 1);
    } else {
      for (int i = tid; i < n; i += nt) {
        A.out_re[fq * n + i] = f[i].x;
        A.out_im[fq * n + i] = f[i].y;
      }
    }
    __syncthreads();
  }
}

size_t sparse_smem(int n, int warps, bool masks) {
  const size_t nw = (n + 31) / 32;
  // u also holds ac_point's pivot search (12 bytes a thread) when n is small
  const size_t lists = (size_t)56 * n + 4 * nw;
  const size_t need = std::max(lists, (size_t)32 * n + (size_t)12 * 32 * warps);
  return ((need + (masks ? 8 * n * nw : 0)) + 31) & ~(size_t)15;
}

}  // namespace

AcShape ac_shape(int n, int nf, int sms, size_t limit) {
  AcShape s;
  // One warp per frequency from eight frequencies an SM on, else as many as
  // keep eight warps an SM busy, a column's updates and the masks spread over
  // them, in small systems too (full ones have n^2 updates a column). Measured:
  // 326-node grid, 226 frequencies, 1 / 2 / 4 / 8 warps 5.4 / 4.0 / 3.3 / 3.1 ms;
  // 103-node ladder, 4501 frequencies, 2.7 / 5.1 / 7.9 / 12 ms, 46 frequencies
  // 0.72 / 0.65 / 0.64 / 0.64 ms; full system of 62 unknowns, 20 frequencies, 2
  // warps 1.46, 4 1.10, 8 0.97 ms, of 32, 1 warp 0.56, 8 0.33 ms. 16 resident warps
  // an SM: 1351 ladder frequencies take 0.86 ms against 1.43 ms with eight.
  s.warps = 1;
  while (s.warps < 8 && (long long)s.warps * nf < 8LL * sms) s.warps *= 2;
  s.masks_shared = sparse_smem(n, s.warps, true) <= 100 * 1024;
  s.smem = sparse_smem(n, s.warps, s.masks_shared);
  const long long per_sm =
      std::max<long long>(1, std::min<long long>(16 / s.warps, (long long)(220 * 1024 / s.smem)));
  const size_t slot = (size_t)16 * n * n;
  s.blocks = (int)std::min<long long>(
      std::min<long long>(nf, per_sm * sms),
      (long long)std::max<size_t>(1, limit / slot));
  s.scratch_bytes = slot * s.blocks;
  s.mask_words = (size_t)2 * n * ((n + 31) / 32);
  return s;
}

void launch_ac_sparse(const AcArgs& a, int nf, const AcShape& s, cudaStream_t st) {
  raise_smem_limit<k_ac_sparse>(s.smem);
  k_ac_sparse<<<s.blocks, 32 * s.warps, s.smem, st>>>(a, nf, s.masks_shared ? 1 : 0);
}

}  // namespace gk
