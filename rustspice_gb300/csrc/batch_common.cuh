// Building blocks of the batched kernels (DC Newton, transient forward and
// transient adjoint). One warp works on M instances of one circuit program
// at a time, LPI = 32/M lanes per instance, with every value of an instance
// in shared memory:
//   X[nc]   iterate (node voltages)      XP[nc] previous time point
//   T[n]    permuted right-hand side / solution
//   DV[ndv] device value records         V[nv]  LU values + BTF coupling
// The factorization and substitutions are a row stream (run_stream) that the
// warp copies through a small ring in shared memory; k_batch_newton stages a
// step program or the column records instead. Everything else of the program
// is read through the read-only path.
#pragma once

#include "kernels.cuh"

namespace gk {
namespace bt {

constexpr unsigned kFull = 0xffffffffu;

// Contribution lists longer than this are summed across the instance's
// lanes instead of by one lane.
constexpr int kHeavy = 12;

// S: element stride of dv (1 in shared memory; 32 in a lane-interleaved
// scratch, where element i of a lane's array sits at [i * 32])
template <int S = 1>
__device__ __forceinline__ double contrib(const double* dv, int code) {
  const int kind = code & 7, idx = code >> 3;
  switch (kind) {
    case 0: return dv[idx * S];
    case 1: return -dv[idx * S];
    case 2: return 1.0;
    case 3: return -1.0;
    default: return 0.0;
  }
}

// x with its sign bit flipped where m has it (m: 0 or the sign bit); on the
// integer pipe.
__device__ __forceinline__ double flip_sign(double x, unsigned long long m) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)m);
}

// Device value record: R [g]; V [value]; I [value]; D [g, ieq];
// M [gds, gm, ieq]; MC [ddd, dds, ddg, ieq]; C (transient) [g, ieq].
// Circuit constants per device: R [1/R]; V, I [value]; D [Is, vt, Is/vt];
// M [is_pmos, vth0, beff]; MC [polarity, |vth0|, beff]; C [C, C/dt].
// gdev is the level-1 conductance floor (1e-12 as the reference has it; 0
// for the exact Jacobian of the adjoint).
// v0, v1, v2: the voltages at the device's first three nodes (a capacitor's at
// the previous time point).
__device__ __forceinline__ void eval_values(int type, const double* dp, double v0, double v1,
                                            double v2, double gmin, double gdev, double* rec) {
  switch (type) {
    case 0:
    case 1:
    case 2:
      rec[0] = dp[0];
      break;
    case 3: {  // crates/sim-core/src/stamp.rs:351-387
      const double gf = gmin > 0.0 ? gmin : 1e-12;
      const double vd = v0 - v1;
      const double e = exp(vd / dp[1]);
      const double id = dp[0] * (e - 1.0);
      const double gd = dp[2] * e;
      rec[0] = fmax(gd, gf);
      rec[1] = id - gd * vd;
      break;
    }
    case 4: {  // level 1 as the reference evaluates it (evaluate.rs:285-356)
      const double lambda = 0.02;
      const double gf = gmin > 0.0 ? gmin : 1e-12;
      const bool pm = dp[0] != 0.0;
      const double vd = v0, vg = v1, vs = v2;
      double vdi = pm ? -vs : vd, vgi = pm ? -vg : vg, vsi = pm ? -vd : vs;
      double vgs = vgi - vsi, vds = vdi - vsi;
      if (vds < 0.0) {
        vds = -vds;
        vgs = vgi - vdi;
      }
      const double vth = pm ? -fabs(dp[1]) : fabs(dp[1]);
      const double beff = dp[2];
      double ids, gm, gds;
      if (vgs <= vth) {
        ids = 0.0;
        gm = 0.0;
        gds = gdev;
      } else if (vds < vgs - vth) {
        ids = beff * ((vgs - vth) * vds - 0.5 * vds * vds);
        gm = beff * vds;
        gds = fmax(beff * ((vgs - vth) - vds), gdev);
      } else {
        const double t = vgs - vth;
        ids = 0.5 * beff * (t * t) * (1.0 + lambda * vds);
        gm = beff * (vgs - vth) * (1.0 + lambda * vds);
        gds = fmax(0.5 * beff * (t * t) * lambda, gdev);
      }
      const double ids_s = pm ? -ids : ids;
      rec[0] = fmax(gds, gf);
      rec[1] = gm;
      rec[2] = ids_s - gm * (vg - vs) - gds * (vd - vs);
      break;
    }
    case 5: {  // backward-Euler capacitor companion, physical sign
      const double g = dp[1];
      const double vp = v0 - v1;
      rec[0] = g;
      rec[1] = g * vp;
      break;
    }
    case 6: {  // consistent level 1, Shichman-Hodges form
      // One formula for the three regions, with the region tests, signs,
      // absolute values and maxima on the integer pipe (on this part an FP64
      // warp instruction costs the SM sub-partition's FP64 unit 64 cycles,
      // and lanes of a warp evaluate devices in different regions): with
      // vde = 0 (cutoff), vds_eff (linear) or vgs_eff - vth (saturation),
      //   q = vde (vov - vde / 2), ids = beff q (1 + lambda vds_eff),
      //   gm = beff (1 + lambda vds_eff) vde,
      //   gds = max(beff (1 + lambda vds_eff) (vov - vde) + lambda beff q, gdev),
      // which are the Shichman-Hodges current and its partials in each
      // region (in cutoff gds comes out as the floor gdev).
      const unsigned long long sg = 0x8000000000000000ull;
      const double lambda = 0.02;
      const double vd = v0, vg = v1, vs = v2;
      const unsigned long long fm = (unsigned long long)__double_as_longlong(dp[0]) & sg;
      const double vgs = flip_sign(vg - vs, fm), vds = flip_sign(vd - vs, fm);
      const unsigned long long bds = (unsigned long long)__double_as_longlong(vds);
      const bool rev = (bds & sg) != 0 && (bds << 1) != 0;  // vds < 0
      const double vgse = vgs - (rev ? vds : 0.0);
      const long long bdse = (long long)(bds & ~sg);
      const double vdse = __longlong_as_double(bdse);
      const double vth = dp[1], beff = dp[2];
      const double vov = vgse - vth;
      const long long bov = __double_as_longlong(vov);
      // non-negative doubles order as their bit patterns
      const double vde = bov <= 0 ? 0.0 : (bdse < bov ? vdse : vov);
      const double k = fma(lambda, vdse, 1.0);
      const double q = vde * fma(-0.5, vde, vov);
      const double bq = beff * q, bk = beff * k;
      const double ids = bq * k, gm = bk * vde;
      const double g0 = fma(lambda, bq, bk * (vov - vde));
      const long long b0 = __double_as_longlong(g0);
      const double gds = (b0 < 0 || b0 < __double_as_longlong(gdev)) ? gdev : g0;
      const unsigned long long rm = rev ? sg : 0ull;
      const double sum = gm + gds;
      rec[0] = rev ? sum : gds;                  // ddd
      rec[1] = flip_sign(rev ? gds : sum, sg);   // dds
      rec[2] = flip_sign(gm, rm);                // ddg
      rec[3] = flip_sign(ids, fm ^ rm) - fma(rec[2], vg, fma(rec[0], vd, rec[1] * vs));
      break;
    }
    default:
      break;
  }
}

// The same at an iterate X (S: element stride), the previous point XP.
template <int S = 1>
__device__ __forceinline__ void eval_record(int type, const int* nd, const double* dp,
                                            const double* X, const double* XP, int nc,
                                            double gmin, double gdev, double* rec) {
  const double* const Y = type == 5 ? XP : X;
  auto at = [&](int i) { return (i >= 0 && i < nc) ? Y[i * S] : 0.0; };
  const bool three = type == 4 || type == 6, two = three || type == 3 || type == 5;
  eval_values(type, dp, two ? at(nd[0]) : 0.0, two ? at(nd[1]) : 0.0, three ? at(nd[2]) : 0.0,
              gmin, gdev, rec);
}

__device__ __forceinline__ int record_len(int type, bool transient) {
  return type == 6 ? 4 : type == 4 ? 3 : type == 3 ? 2 : type == 5 ? (transient ? 2 : 0) : 1;
}

// 1/d for the batched factorization: a single-precision seed built from d's
// bits on the integer pipe, the hardware float reciprocal, and one FP64
// Newton step (relative error about 1e-14). FP64 operations have a 64-cycle
// dependent latency on this part, so this is about half the latency of the
// correctly rounded reciprocal, which serves magnitudes outside the
// single-precision range.
__device__ __forceinline__ double fast_rcp(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ff);
  if (e < 1023 - 120 || e > 1023 + 120) return __drcp_rn(d);
  const unsigned fb = (unsigned)((b >> 32) & 0x80000000u) | ((unsigned)(e - 1023 + 127) << 23) |
                      (unsigned)((b >> 29) & 0x7fffffu);
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(fb)));
  const unsigned rb = __float_as_uint(rf);
  const unsigned long long r64 =
      ((unsigned long long)(rb & 0x80000000u) << 32) |
      ((unsigned long long)(((rb >> 23) & 0xff) - 127 + 1023) << 52) |
      ((unsigned long long)(rb & 0x7fffffu) << 29);
  const double r = __longlong_as_double((long long)r64);
  return fma(r, fma(-d, r, 1.0), r);
}

__device__ __forceinline__ bool nonzero(double u) {
  return (__double_as_longlong(u) << 1) != 0;
}

// The reference's pivot perturbation (native_klu.rs:1229-1231, :1345-1348)
// on the bit pattern: integer compares instead of FP64 pipe compares.
__device__ __forceinline__ double perturb_bits(double d, bool singleton) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned long long a = b & 0x7fffffffffffffffull;
  if (singleton)
    return a < (unsigned long long)__double_as_longlong(1e-300) ? 1e-14 : d;
  if (a < (unsigned long long)__double_as_longlong(1e-14))
    return (a == 0 || (b >> 63) == 0) ? 1e-14 : -1e-14;
  return d;
}

// One group's program as the phases below read it.
struct Prog {
  const int4* colrec;  // staged: (s0, dslot, s1, singleton) per column
  const int* srow;     // staged: slot rows
  const int* uptr;     // update-list offsets per slot (staged when leveled)
  const int* udst;     // update destinations (staged when leveled)
  int* map;            // per instance: row -> slot of the column being factored
  const int *dev_type, *dev_nodes, *dev_dv, *amap_ptr, *amap_code, *rmap_ptr, *rmap_code,
      *in_row, *out_pos, *offd_ptr, *offd_col, *bptr, *heavy;
  const int *lvl_col, *lseg_ptr, *lseg;  // level schedule of the factorization
  const int4 *amap4, *rmap4;             // four padded codes per slot / permuted row
  const int* lng;                        // slots and rows with more: (index << 1) | is_row
  int nlng;
  const int4* ev;                        // devices to evaluate, by type (capacitors last)
  RowStream stream;                      // factor and solve (run_stream)
  RowStream tstream;                     // transpose solve (transient adjoint)
  const int4* asm4;                      // records of up to four codes, longest first,
  const int* asm_dst;                    //   and where each goes: T at 0, V at n
  const int2* ops;                       // staged step program (or null)
  const int* sp;                         //   and its step pointers
  int n, nc, nv, nslots, ndev, nblocks, nheavy, nsteps, nev, ncap;
};

// The program view of a group without staging (global arrays only).
__device__ __forceinline__ Prog global_view(const BatchArgs& A, const GroupHdr& G) {
  Prog P;
  P.colrec = nullptr;
  P.srow = nullptr;
  P.uptr = A.upd_ptr + G.slot_off;
  P.udst = A.upd_dst + G.upd_off;
  P.map = nullptr;
  P.dev_type = A.dev_type + G.dev_off;
  P.dev_nodes = A.dev_nodes + 4 * G.dev_off;
  P.dev_dv = A.dev_dv + G.dev_off;
  P.amap_ptr = A.amap_ptr + G.amap_off;
  P.amap_code = A.amap_code + G.amap_code_off;
  P.rmap_ptr = A.rmap_ptr + G.rmap_off;
  P.rmap_code = A.rmap_code + G.rmap_code_off;
  P.in_row = A.in_row + G.col_off;
  P.out_pos = A.out_pos + G.col_off;
  P.offd_ptr = A.offd_ptr + G.col_off;
  P.offd_col = A.offd_col + G.offd_off;
  P.bptr = A.block_ptr + G.blk_off;
  P.heavy = A.heavy + G.heavy_off;
  P.lvl_col = A.lvl_col + G.col_off;
  P.lseg_ptr = A.lseg_ptr + G.blk_off;
  P.lseg = A.lseg + 3 * G.seg_off;
  P.amap4 = reinterpret_cast<const int4*>(A.amap4 + G.amap4_off);
  P.rmap4 = reinterpret_cast<const int4*>(A.rmap4 + G.rmap4_off);
  P.lng = A.lng + G.lng_off;
  P.nlng = G.nlng;
  P.ev = A.ev + G.ev_off;
  P.nev = G.nev;
  P.ncap = G.ncap;
  P.stream = {A.recs + (long long)G.stream_off * kStreamChunk, A.segs + G.sseg_off, G.nchunk,
              G.nsseg};
  P.tstream = {A.recs + (long long)G.tstream_off * kStreamChunk, A.segs + G.tsseg_off, G.ntchunk,
               G.ntsseg};
  P.asm4 = reinterpret_cast<const int4*>(A.asm4 + G.asm_off * 4);
  P.asm_dst = A.asm_dst + G.asm_off;
  P.ops = nullptr;
  P.sp = nullptr;
  P.n = G.n;
  P.nc = G.node_count;
  P.nslots = G.nslots;
  P.nv = G.nslots + G.noffd;
  P.ndev = G.ndev;
  P.nblocks = G.nblocks;
  P.nheavy = G.nheavy;
  P.nsteps = 0;
  return P;
}

// Stages the group's factor and solve structure into shared memory and
// returns the program view: by one warp (tid = lane, nthr = 32) or by the
// whole block (block = true; every thread of the block calls it). steps:
// a group with a step program stages that instead of the column records.
__device__ __forceinline__ Prog stage_program(const BatchArgs& A, const GroupHdr& G, int* prog,
                                              int lane, int nthr = 32, bool block = false,
                                              bool steps = false) {
  Prog P = global_view(A, G);
  const int n = G.n;
  int4* const colrec = reinterpret_cast<int4*>(prog);
  int* const srow = prog + 4 * n;
  if (steps && G.nsteps > 0) {
    int2* const ops = reinterpret_cast<int2*>(prog);
    int* const sp = prog + 2 * G.nops;
    const int2* gops = A.ops + G.ops_off;
    const int* gsp = A.step_ptr + G.step_off;
    for (int q = lane; q < G.nops; q += nthr) ops[q] = gops[q];
    for (int q = lane; q <= G.nsteps; q += nthr) sp[q] = gsp[q];
    P.ops = ops;
    P.sp = sp;
    P.nsteps = G.nsteps;
  } else {
    const int* cp = A.col_ptr + G.col_off;
    const int* dsl = A.dslot + G.col_off;
    const int* cs = A.col_single + G.col_off;
    for (int k = lane; k < n; k += nthr) colrec[k] = make_int4(cp[k], dsl[k], cp[k + 1], cs[k]);
    const int* sr = A.slot_row + G.slot_off;
    for (int q = lane; q < G.nslots; q += nthr) srow[q] = sr[q];
    if (G.nseg > 0) {  // the level path reads the update lists per lane: stage them too
      int* const uptr = srow + G.nslots;
      int* const udst = uptr + G.nslots;
      const int* up = A.upd_ptr + G.slot_off;
      for (int q = lane; q < G.nslots; q += nthr) uptr[q] = up[q];
      const int* ud = A.upd_dst + G.upd_off;
      for (int q = lane; q < G.nupd; q += nthr) udst[q] = ud[q];
    }
  }
  if (block)
    __syncthreads();
  else
    __syncwarp();
  if (P.nsteps == 0) {
    P.colrec = colrec;
    P.srow = srow;
    if (G.nseg > 0) {
      P.uptr = srow + G.nslots;
      P.udst = srow + 2 * G.nslots;
    }
  }
  return P;
}

// Device evaluation of one instance into its value records (lanes over the
// devices, sorted by type so that a warp's lanes take the same branch; two
// devices per lane at a time, the next two's references read meanwhile).
// ov_dev/ov_val override the first constant of one device.
template <int LPI>
__device__ __forceinline__ void stamp_devices(const Prog& P, const double* dparams, int ov_dev,
                                              double ov_val, const double* X, const double* XP,
                                              double gmin, double gdev, bool transient,
                                              double* DV, int sl) {
  constexpr int U = 2;
  const int4 no_dev = make_int4(-1, 0, 0, 0);
  auto ref = [&](int q) { return q < P.nev ? __ldg(P.ev + q) : no_dev; };
  int4 n0 = ref(sl), n1 = ref(sl + LPI);
  for (int q0 = sl; q0 < P.nev; q0 += U * LPI) {
    const int4 e[U] = {n0, n1};
    n0 = ref(q0 + 2 * LPI);
    n1 = ref(q0 + 3 * LPI);
    double2 pa[U], pb[U];
    double x[U][3];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e[u].x >= 0) {
        const double2* const src = reinterpret_cast<const double2*>(dparams + 4 * e[u].x);
        pa[u] = __ldg(src);
        pb[u] = __ldg(src + 1);
        const double* const Y = (e[u].z >> 16) == 5 ? XP : X;
        const int i0 = e[u].y & 0xffff, i1 = (e[u].y >> 16) & 0xffff, i2 = e[u].z & 0xffff;
        x[u][0] = i0 < P.nc ? Y[i0] : 0.0;
        x[u][1] = i1 < P.nc ? Y[i1] : 0.0;
        x[u][2] = i2 < P.nc ? Y[i2] : 0.0;
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e[u].x >= 0) {
        const int type = e[u].z >> 16;
        const double dp[4] = {e[u].x == ov_dev ? ov_val : pa[u].x, pa[u].y, pb[u].x, pb[u].y};
        double rec[4];
        eval_values(type, dp, x[u][0], x[u][1], x[u][2], gmin, gdev, rec);
        const int nrec = record_len(type, transient);
        for (int k = 0; k < nrec; ++k) DV[e[u].w + k] = rec[k];
      }
  }
}

// LU slot values and the permuted right-hand side from the value records,
// each the sum of its contributions in stamping order: lists of up to four
// as one padded 16-byte record (code 4 pads, never added), the longest first
// so that a warp's lanes add about as often, the values of several records in
// flight together; longer lists afterwards, one lane each, and the longest
// (the ground and supply rows and columns) reduced across 32 lanes (with 16
// lanes, each keeps the two sums of a pair 16 apart: the same additions).
constexpr int kPadCode = 4;

// contrib without a branch: the value loads, whatever the code's kind.
__device__ __forceinline__ double contrib_load(const double* dv, int code) {
  return dv[(code & 6) == 0 ? code >> 3 : 0];
}
__device__ __forceinline__ double contrib_value(double v, int code) {
  const int kind = code & 7;
  int hi = __double2hiint(v), lo = __double2loint(v);
  if (kind >= 2) {
    hi = kind == 4 ? 0 : 0x3ff00000;
    lo = 0;
  }
  if (kind & 1) hi ^= (int)0x80000000;
  return __hiloint2double(hi, lo);
}

// TV: T, then V.
template <int LPI>
__device__ __forceinline__ void assemble4(const Prog& P, const double* DV, double* TV, int sl) {
  constexpr int U = 4;
  const int count = P.n + P.nv;
  const int4 pad = make_int4(kPadCode, kPadCode, kPadCode, kPadCode);
  int4 nx[U];
  int nd[U];
  auto fetch = [&](int v0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = v0 + u * LPI < count;
      nx[u] = in ? __ldg(P.asm4 + v0 + u * LPI) : pad;
      nd[u] = in ? __ldg(P.asm_dst + v0 + u * LPI) : -1;
    }
  };
  fetch(sl);
  for (int v0 = sl; v0 < count; v0 += U * LPI) {
    int4 c[U];
    int d[U];
    double a[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      c[u] = nx[u];
      d[u] = nd[u];
      a[u][0] = contrib_load(DV, c[u].x);
      a[u][1] = contrib_load(DV, c[u].y);
      a[u][2] = contrib_load(DV, c[u].z);
      a[u][3] = contrib_load(DV, c[u].w);
    }
    fetch(v0 + U * LPI);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      double acc = contrib_value(a[u][0], c[u].x);
      if (c[u].y != kPadCode) {
        acc += contrib_value(a[u][1], c[u].y);
        if (c[u].z != kPadCode) {
          acc += contrib_value(a[u][2], c[u].z);
          if (c[u].w != kPadCode) acc += contrib_value(a[u][3], c[u].w);
        }
      }
      if (d[u] >= 0) TV[d[u]] = acc;
    }
  }
}

// A longer list: its codes' bounds, from (index << 1) | is_row.
__device__ __forceinline__ const int* list_codes(const Prog& P, int code, int& len) {
  const bool row = code & 1;
  const int key = row ? P.in_row[code >> 1] : code >> 1;
  const int* const ptr = row ? P.rmap_ptr : P.amap_ptr;
  const int t0 = ptr[key];
  len = ptr[key + 1] - t0;
  return (row ? P.rmap_code : P.amap_code) + t0;
}

__device__ __forceinline__ void put_list(const Prog& P, int code, double v, double* V, double* T) {
  if (code & 1)
    T[code >> 1] = v;
  else
    V[code >> 1] = v;
}

// All but the longest lists.
template <int LPI>
__device__ __forceinline__ void assemble_short(const Prog& P, const double* DV, double* V,
                                               double* T, int sl) {
  assemble4<LPI>(P, DV, T, sl);
  __syncwarp();  // the longer lists below overwrite their all-pad records' zeros
  for (int h = sl; h < P.nlng; h += LPI) {
    const int code = P.lng[h];  // (index << 1) | is_row
    int len;
    const int* const cds = list_codes(P, code, len);
    if (len > kHeavy) continue;
    double v[kHeavy], acc = 0.0;
    int cd[kHeavy];
#pragma unroll
    for (int t = 0; t < kHeavy; ++t) cd[t] = t < len ? cds[t] : kPadCode;
#pragma unroll
    for (int t = 0; t < kHeavy; ++t) v[t] = contrib_load(DV, cd[t]);
#pragma unroll
    for (int t = 0; t < kHeavy; ++t)
      if (t < len) acc = t == 0 ? contrib_value(v[0], cd[0]) : acc + contrib_value(v[t], cd[t]);
    put_list(P, code, acc, V, T);
  }
}

template <int LPI>
__device__ __forceinline__ void assemble(const Prog& P, const double* DV, double* V, double* T,
                                         int sl) {
  assemble_short<LPI>(P, DV, V, T, sl);
  for (int h = 0; h < P.nheavy; ++h) {
    const int code = P.heavy[h];
    int len;
    const int* const cds = list_codes(P, code, len);
    // lane sl's positions sl, sl + 32, ... (and with 16 lanes those of lane
    // sl + 16), eight of them in flight
    double acc = 0.0, hi = 0.0;
    for (int t0 = sl; t0 < len; t0 += 8 * LPI) {
      int cd[8];
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) cd[u] = t0 + u * LPI < len ? __ldg(cds + t0 + u * LPI) : kPadCode;
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = contrib_load(DV, cd[u]);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t0 + u * LPI < len) {
          if (LPI == 16 && (u & 1))
            hi += contrib_value(v[u], cd[u]);
          else
            acc += contrib_value(v[u], cd[u]);
        }
    }
    if (LPI == 16) acc += hi;
#pragma unroll
    for (int o = (LPI == 16 ? 8 : LPI / 2); o > 0; o >>= 1)
      acc += __shfl_xor_sync(kFull, acc, o);
    if (sl == 0) put_list(P, code, acc, V, T);
  }
}

// Factor, forward substitution, backward substitution, block by block
// (blocks in order; the BTF coupling lies below the diagonal blocks).
// The factorization follows the program's level schedule: in a parallel
// segment every lane factors whole columns of one level (each column reads
// only finished columns and writes only its own slots, its U entries in
// order), in a sequential segment (the rails) the lanes share each update.
// Afterwards V[dslot] holds the reciprocal of the (perturbed) pivot and T
// the permuted solution.
__device__ __forceinline__ void factor_column(const Prog& P, double* V, int k) {
  const int4 ck = P.colrec[k];
  for (int s = ck.x; s < ck.y; ++s) {
    const double u = V[s];
    if (nonzero(u)) {
      const int4 cj = P.colrec[P.srow[s]];
      const int q0 = cj.y + 1;
      const int* dst = P.udst + P.uptr[s] - q0;
      for (int qq = q0; qq < cj.z; ++qq) {
        const int dd = dst[qq];
        V[dd] = fma(-V[qq], u, V[dd]);
      }
    }
  }
  const double r = fast_rcp(perturb_bits(V[ck.y], ck.w != 0));
  for (int qq = ck.y + 1; qq < ck.z; ++qq) V[qq] = V[qq] * r;
  V[ck.y] = r;
}

// Column by column, lanes over each update, forward substitution fused.
template <int LPI>
__device__ __forceinline__ void factor_solve_columns(const Prog& P, double* V, double* T,
                                                     int sl) {
  for (int b = 0; b < P.nblocks; ++b) {
    const int b0 = P.bptr[b], b1 = P.bptr[b + 1];
    for (int i = b0 + sl; i < b1; i += LPI)
      for (int e = P.offd_ptr[i]; e < P.offd_ptr[i + 1]; ++e)
        T[i] = fma(-V[P.nslots + e], T[P.offd_col[e]], T[i]);
    __syncwarp();
    int* const map = P.map;
    for (int k = b0; k < b1; ++k) {
      const int4 ck = P.colrec[k];
      // destination slots of this column's updates: row -> slot
      for (int q = ck.x + sl; q < ck.z; q += LPI) map[P.srow[q]] = q;
      __syncwarp();
      // The update structure of U entry s (its L column, this lane's first
      // destination) does not depend on values: it is loaded one entry
      // ahead, so its latency overlaps the previous update and its warp
      // synchronisation.
      int4 cj = make_int4(0, 0, 0, 0);
      int dd0 = 0;
      if (ck.x < ck.y) {
        cj = P.colrec[P.srow[ck.x]];
        if (cj.y + 1 + sl < cj.z) dd0 = map[P.srow[cj.y + 1 + sl]];
      }
      for (int s = ck.x; s < ck.y; ++s) {
        const int4 cur = cj;
        const int cdd0 = dd0;
        if (s + 1 < ck.y) {
          cj = P.colrec[P.srow[s + 1]];
          if (cj.y + 1 + sl < cj.z) dd0 = map[P.srow[cj.y + 1 + sl]];
        }
        const double u = V[s];
        if (nonzero(u)) {
          const int q0 = cur.y + 1;
          int qq = q0 + sl;
          if (qq < cur.z) {
            V[cdd0] = fma(-V[qq], u, V[cdd0]);
            for (qq += LPI; qq < cur.z; qq += LPI) {
              const int dd = map[P.srow[qq]];
              V[dd] = fma(-V[qq], u, V[dd]);
            }
          }
        }
        __syncwarp();
      }
      const double r = fast_rcp(perturb_bits(V[ck.y], ck.w != 0));
      const double zk = T[k];
      for (int qq = ck.y + 1 + sl; qq < ck.z; qq += LPI) {
        const double l = V[qq] * r;
        V[qq] = l;
        const int row = P.srow[qq];
        T[row] = fma(-l, zk, T[row]);
      }
      if (sl == 0) V[ck.y] = r;
      __syncwarp();
    }
    for (int k = b1 - 1; k >= b0; --k) {
      const int4 ck = P.colrec[k];
      const double xk = T[k] * V[ck.y];
      for (int s = ck.x + sl; s < ck.y; s += LPI) {
        const int row = P.srow[s];
        T[row] = fma(-V[s], xk, T[row]);
      }
      __syncwarp();
      if (sl == 0) T[k] = xk;
      __syncwarp();
    }
  }
}

template <int LPI>
__device__ __forceinline__ void factor_solve(const Prog& P, double* V, double* T, int sl) {
  if (P.lseg_ptr[P.nblocks] == 0) {  // no level schedule for this program
    factor_solve_columns<LPI>(P, V, T, sl);
    return;
  }
  for (int b = 0; b < P.nblocks; ++b) {
    const int b0 = P.bptr[b], b1 = P.bptr[b + 1];
    for (int i = b0 + sl; i < b1; i += LPI)
      for (int e = P.offd_ptr[i]; e < P.offd_ptr[i + 1]; ++e)
        T[i] = fma(-V[P.nslots + e], T[P.offd_col[e]], T[i]);
    for (int g = P.lseg_ptr[b]; g < P.lseg_ptr[b + 1]; ++g) {
      const int start = P.lseg[3 * g], end = P.lseg[3 * g + 1];
      if (P.lseg[3 * g + 2] == 0) {
        for (int idx = start + sl; idx < end; idx += LPI) factor_column(P, V, P.lvl_col[idx]);
        __syncwarp();
        continue;
      }
      for (int idx = start; idx < end; ++idx) {
        const int k = P.lvl_col[idx];
        const int4 ck = P.colrec[k];
        for (int s = ck.x; s < ck.y; ++s) {
          const double u = V[s];
          if (nonzero(u)) {
            const int4 cj = P.colrec[P.srow[s]];
            const int q0 = cj.y + 1;
            const int* dst = P.udst + P.uptr[s] - q0;
            for (int qq = q0 + sl; qq < cj.z; qq += LPI) {
              const int dd = dst[qq];
              V[dd] = fma(-V[qq], u, V[dd]);
            }
          }
          __syncwarp();
        }
        const double r = fast_rcp(perturb_bits(V[ck.y], ck.w != 0));
        for (int qq = ck.y + 1 + sl; qq < ck.z; qq += LPI) V[qq] = V[qq] * r;
        __syncwarp();
        if (sl == 0) V[ck.y] = r;
        __syncwarp();
      }
    }
    for (int k = b0; k < b1; ++k) {  // L z = b, column order
      const int4 ck = P.colrec[k];
      const double zk = T[k];
      for (int qq = ck.y + 1 + sl; qq < ck.z; qq += LPI) {
        const int row = P.srow[qq];
        T[row] = fma(-V[qq], zk, T[row]);
      }
      __syncwarp();
    }
    for (int k = b1 - 1; k >= b0; --k) {
      const int4 ck = P.colrec[k];
      const double xk = T[k] * V[ck.y];
      for (int s = ck.x + sl; s < ck.y; s += LPI) {
        const int row = P.srow[s];
        T[row] = fma(-V[s], xk, T[row]);
      }
      __syncwarp();
      if (sl == 0) T[k] = xk;
      __syncwarp();
    }
  }
}

// One operation of a step program on an instance region R (X, T, V), two
// 32-bit words: d | a << 15 | kind bits 0-1 << 30 and b | c << 15 | kind
// bits 2-3 << 30. Kinds: 0 R[d] -= R[a] R[b] (one fma); 4 the same unless
// R[b] is zero (a factor update by a zero U entry is skipped); 2 R[d] =
// R[a] R[b]; 1 R[d] = 1 / perturbed R[d] (a: the column is a singleton); 5
// kind 4 then R[d] *= R[c] (an L entry's last update and its scaling); 6
// kind 0 then R[d] *= R[c] (a row's last backward update and its pivot);
// 3 nothing.
__device__ __forceinline__ void exec_op(int2 o, double* R) {
  const unsigned x = (unsigned)o.x, y = (unsigned)o.y;
  const int d = x & 0x7fff, a = (x >> 15) & 0x7fff, b = y & 0x7fff, c = (y >> 15) & 0x7fff;
  const int k = (int)((x >> 30) | ((y >> 30) << 2));
  if (k == 1) {
    R[d] = fast_rcp(perturb_bits(R[d], a != 0));
    return;
  }
  // The other kinds as one fma, so that lanes of a step that mix them issue
  // one FP64 instruction (and the product only where a lane needs it): kind 2
  // is fma(a, b, -0), which rounds like a b; kinds 0, 4, 5 and 6 are fma(-a,
  // b, d), with d kept where kind 4 or 5 skips a zero b. The signs and the
  // selections are integer operations.
  const bool mul = k == 2, fused = k >= 5;
  const double va = R[a], vb = R[b], vd = R[d];
  const double na = flip_sign(va, mul ? 0ull : 0x8000000000000000ull);
  const double t = fma(na, vb, mul ? -0.0 : vd);
  const bool skip = (k == 4 || k == 5) && !nonzero(vb);
  double r = skip ? vd : t;
  if (fused) r = r * R[c];
  if (k != 3) R[d] = r;
}

// The factorization, forward and backward substitution as the group's step
// program: the host lists every operation of factor_solve_columns in its
// order and places each in the first step after the steps that write its
// operands or read its destination, so the operations of one step are
// independent and every value sees the same operations in the same order
// as in the column-by-column path (the same results; fused pairs keep both
// roundings). The instance's lanes take a step's operations in parallel;
// the next step's operations are loaded while the current one runs. The
// warp's instances run the same program in step.
template <int LPI>
__device__ __forceinline__ void run_steps(const Prog& P, double* R, int sl) {
  const int2 nop = make_int2((int)(3u << 30), 0);  // kind 3: nothing
  const int2* const ops = P.ops;
  const int* const sp = P.sp;
  const int ns = P.nsteps;
  const int nops = sp[ns];
  // a step's operation and pointer load independently, a step ahead
  int s0 = sp[0], s1 = sp[1], s2 = ns >= 2 ? sp[2] : s1;
  int2 o0 = s0 + sl < nops ? ops[s0 + sl] : nop;
  for (int t = 0; t < ns; ++t) {
    const int2 o1 = s1 + sl < nops ? ops[s1 + sl] : nop;
    const int s3 = t + 3 <= ns ? sp[t + 3] : s2;
    if (s0 + sl < s1) exec_op(o0, R);
    for (int p = s0 + sl + LPI; p < s1; p += LPI) exec_op(ops[p], R);
    __syncwarp();
    s0 = s1;
    s1 = s2;
    s2 = s3;
    o0 = o1;
  }
}

// The factorization and substitutions (or the transpose solve) as a row
// stream: the step program's operations in 8-byte records, in segments
// (capi.cu::make_stream). The warp keeps kRing chunks of records in shared
// memory, filled by cp.async two chunks ahead (copies in flight hold no
// register and no scoreboard of the warp, which FP64 results and loads would
// otherwise wait behind); a row's records are read one row ahead. Segments:
//   plain    rows of W records: R[d] = t = fma(-R[a], R[b], R[d])
//   fused    ... R[d] = t R[c] (R[c] = 1 where an operation has no product)
//   rcp      R[d] = 1 / perturbed R[d]
//   serial   operation i's b is operation i-1's d, all fused: every lane runs
//            them on values the lanes loaded together
//   sum      one d: t = fma(-R[a_i], R[b_i], t)
// The signs and selections of an operation are integer operations on values
// still on their way to the FP64 unit, and its fma is one instruction for
// every kind (kind 2 a product: fma(a, b, -0); kinds 4 and 5 skip a zero b: a
// zero of the opposite sign takes a's place, and fma(-+0, +-0, d) = d), so a
// row costs the pipe one FP64 instruction, or two when fused.
// Measured, one warp, cycles: a plain row 157, a fused one 243, a serial
// operation 164, a sum operation 94. An FP64 result is 64 cycles away from
// another FP64 instruction and 114 from anything else, which is why the
// shuffles of a serial or sum segment come eight operations at a time, and
// why nothing but the fma waits for a row's values; a header per row, read
// with it, cost another 250 cycles.
constexpr int kRing = 4;  // chunks of kStreamChunk records per warp

__device__ __forceinline__ double fma_asm(double a, double b, double c) {
  double r;
  asm("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(a), "d"(b), "d"(c));
  return r;
}
__device__ __forceinline__ bool zero_bits(double v) {
  return (((unsigned)__double2hiint(v) << 1) | (unsigned)__double2loint(v)) == 0u;
}
__device__ __forceinline__ bool skips_zero(int2 o) {  // kinds 4 and 5
  return ((unsigned)o.y >> 30) == 1u && ((unsigned)o.x >> 30) <= 1u;
}

// Shared-memory accesses by 32-bit address. The loads and stores of a row are
// issued in program order.
__device__ __forceinline__ double lds64(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ int2 lds_rec(unsigned a) {
  int2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts64(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// The operands' addresses of a record (build_steps packs it), R the region's.
__device__ __forceinline__ unsigned rec_d(int2 o, unsigned R) { return R + (((unsigned)o.x << 3) & 0x3fff8u); }
__device__ __forceinline__ unsigned rec_a(int2 o, unsigned R) { return R + (((unsigned)o.x >> 12) & 0x3fff8u); }
__device__ __forceinline__ unsigned rec_b(int2 o, unsigned R) { return R + (((unsigned)o.y << 3) & 0x3fff8u); }
__device__ __forceinline__ unsigned rec_c(int2 o, unsigned R) { return R + (((unsigned)o.y >> 12) & 0x3fff8u); }

// One operation up to its fma.
__device__ __forceinline__ double row_fma(int2 o, unsigned R) {
  const unsigned x = (unsigned)o.x, y = (unsigned)o.y;
  const double vb = lds64(rec_b(o, R)), va = lds64(rec_a(o, R)), vd = lds64(rec_d(o, R));
  const bool prod = (x >> 30) == 2u && (y >> 30) == 0u;  // kind 2
  int ah = __double2hiint(va) ^ (prod ? 0 : (int)0x80000000);
  int al = __double2loint(va);
  if (skips_zero(o) && zero_bits(vb)) {
    ah = ~__double2hiint(vb) & (int)0x80000000;
    al = 0;
  }
  const int dh = prod ? (int)0x80000000 : __double2hiint(vd);
  const int dl = prod ? 0 : __double2loint(vd);
  return fma_asm(__hiloint2double(ah, al), vb, __hiloint2double(dh, dl));
}

// Not inlined: the kernels' other phases are long, and a row's loop should
// stay in the instruction cache.
template <int LPI>
__device__ __noinline__ void run_rows(RowStream S, unsigned ring, unsigned R, int sl, int dummy) {
  const int lane = threadIdx.x & 31;
  constexpr int RM = kRing * kStreamChunk - 1, B = 8;
  auto rec = [&](int p) { return lds_rec(ring + 8u * (unsigned)(p & RM)); };
  auto issue = [&](int c) {  // a chunk: 1 KB, twice 16 bytes per lane
    if (c < S.nchunk) {
#pragma unroll
      for (int u = 0; u < kStreamChunk / 64; ++u) {
        const int at = u * 64 + 2 * lane;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         ring + 8u * (unsigned)((c & (kRing - 1)) * kStreamChunk + at)),
                     "l"(S.recs + (long long)c * kStreamChunk + at)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int cc = 0;  // chunks cc and cc + 1 are here, cc + 2 is on its way
  auto reach = [&](int p) {
    while (p / kStreamChunk > cc) {
      ++cc;
      issue(cc + 2);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
    }
  };
  __syncwarp();  // the ring's last readers are done
  issue(0);
  issue(1);
  issue(2);
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncwarp();
  const int2 none = make_int2(dummy | dummy << 15, dummy | dummy << 15);
  int p = 0;
  int2 next = __ldg(S.segs);
  for (int sgi = 0; sgi < S.nseg; ++sgi) {
    const int2 sg = next;
    next = __ldg(S.segs + sgi + 1);  // the list ends with one more
    const int kind = sg.x & 7, cnt = sg.y;
    reach(p);
    if (kind <= kRowFused) {
      // by chunk: the rows of one, then the next (whose first row the last
      // iteration reads ahead)
      const int lw = sg.x >> 3, W = 1 << lw;
      const bool on = sl < W;
      int2 o = rec(p + sl);
      for (int left = cnt; left > 0;) {
        reach(p);
        const int m = min(left, (kStreamChunk - p % kStreamChunk) >> lw);
        left -= m;
        if (LPI < 32 && W > LPI) {  // two passes: a row's operations are independent
          for (int r = 0; r < m; ++r) {
            for (int u = 0; u < 2; ++u) {
              const int2 q = rec(p + u * LPI + sl);
              const double vc = lds64(rec_c(q, R));
              double t = row_fma(q, R);
              if (kind == kRowFused) t = t * vc;
              sts64(rec_d(q, R), t);
            }
            p += W;
            __syncwarp();
          }
          o = rec(p + sl);
        } else if (kind == kRowPlain) {
          for (int r = 0; r < m; ++r) {
            const int2 op = on ? o : none;
            p += W;
            const double t = row_fma(op, R);
            o = rec(p + sl);
            sts64(rec_d(op, R), t);
            __syncwarp();
          }
        } else {
          for (int r = 0; r < m; ++r) {
            const int2 op = on ? o : none;
            p += W;
            const double t = row_fma(op, R);
            const double vc = lds64(rec_c(op, R));
            o = rec(p + sl);
            sts64(rec_d(op, R), t * vc);
            __syncwarp();
          }
        }
      }
    } else if (kind == kRowSerial) {
      for (int p0 = 0; p0 < cnt; p0 += LPI) {
        reach(p + p0 + LPI - 1);
        const int2 q = p0 + sl < cnt ? rec(p + p0 + sl) : none;
        const double na = flip_sign(lds64(rec_a(q, R)), 0x8000000000000000ull);
        const double td = lds64(rec_d(q, R)), vc = lds64(rec_c(q, R)), vb = lds64(rec_b(q, R));
        const int m = min(LPI, cnt - p0);
        // operands B operations ahead, by shuffles placed between the two FP64
        // instructions of an operation; a result is kept by its lane one
        // operation later, when it has left the FP64 unit
        double xv = __shfl_sync(kFull, vb, 0, LPI), mine = 0.0;
        double ba[B], bd[B], bc[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          ba[j] = __shfl_sync(kFull, na, j, LPI);
          bd[j] = __shfl_sync(kFull, td, j, LPI);
          bc[j] = __shfl_sync(kFull, vc, j, LPI);
        }
        int i0 = 0;
        for (; i0 + B <= m; i0 += B) {
#pragma unroll
          for (int j = 0; j < B; ++j) {
            const double t = fma_asm(ba[j], xv, bd[j]), c = bc[j];
            if (sl == i0 + j - 1) mine = xv;
            ba[j] = __shfl_sync(kFull, na, i0 + B + j, LPI);
            bd[j] = __shfl_sync(kFull, td, i0 + B + j, LPI);
            bc[j] = __shfl_sync(kFull, vc, i0 + B + j, LPI);
            xv = t * c;
          }
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
          if (i0 + j >= m) break;
          const double t = fma_asm(ba[j], xv, bd[j]);
          if (sl == i0 + j - 1) mine = xv;
          xv = t * bc[j];
        }
        if (sl == m - 1) mine = xv;
        if (p0 + sl < cnt) sts64(rec_d(q, R), mine);
        __syncwarp();
      }
      p += cnt;
    } else if (kind == kRowSum) {
      double t = 0.0;
      for (int p0 = 0; p0 < cnt; p0 += LPI) {
        reach(p + p0 + LPI - 1);
        const int2 q = p0 + sl < cnt ? rec(p + p0 + sl) : none;
        const double va = lds64(rec_a(q, R)), vb = lds64(rec_b(q, R)), vc = lds64(rec_c(q, R));
        int ah = __double2hiint(va) ^ (int)0x80000000, al = __double2loint(va);
        if (skips_zero(q) && zero_bits(vb)) {
          ah = ~__double2hiint(vb) & (int)0x80000000;
          al = 0;
        }
        const double na = __hiloint2double(ah, al);
        if (p0 == 0) t = __shfl_sync(kFull, lds64(rec_d(q, R)), 0, LPI);
        const int m = min(LPI, cnt - p0);
        for (int i0 = 0; i0 < m; i0 += B) {
          double ba[B], bb[B];
#pragma unroll
          for (int j = 0; j < B; ++j) {
            ba[j] = __shfl_sync(kFull, na, i0 + j, LPI);
            bb[j] = __shfl_sync(kFull, vb, i0 + j, LPI);
          }
          if (i0 + B <= m) {  // no selection between one operation and the next
#pragma unroll
            for (int j = 0; j < B; ++j) t = fma_asm(ba[j], bb[j], t);
          } else {
#pragma unroll
            for (int j = 0; j < B; ++j)
              if (i0 + j < m) t = fma_asm(ba[j], bb[j], t);
          }
        }
        if (sl == m - 1 && p0 + LPI >= cnt) {  // the last operation's lane
          const unsigned x = (unsigned)q.x, y = (unsigned)q.y;
          if ((y >> 30) == 1u && (x >> 30) >= 1u) t = t * vc;  // kinds 5 and 6
          sts64(rec_d(q, R), t);
        }
      }
      __syncwarp();
      p += cnt;
    } else {  // kRowRcp
      for (int p0 = 0; p0 < cnt; p0 += LPI) {
        reach(p + p0 + LPI - 1);
        if (p0 + sl < cnt) {
          const int2 q = rec(p + p0 + sl);
          const unsigned at = rec_d(q, R);
          sts64(at, fast_rcp(perturb_bits(lds64(at), (((unsigned)q.x >> 15) & 0x7fffu) != 0)));
        }
      }
      __syncwarp();
      p += cnt;
    }
    p = (p + kStreamAlign - 1) & ~(kStreamAlign - 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
}

// R: the region (T at nc, V behind it) in shared memory, sl the lane within
// the instance, dummy the region's entry for idle lanes.
template <int LPI>
__device__ __forceinline__ void run_stream(const RowStream& S, int2* ring, double* R, int sl,
                                           int dummy) {
  run_rows<LPI>(S, (unsigned)__cvta_generic_to_shared(ring),
                (unsigned)__cvta_generic_to_shared(R), sl, dummy);
}

}  // namespace bt
}  // namespace gk
