// kern_force64.cu -- the plain FP64 force kernel (acc, jerk, pot, nearest
// neighbour): G6_PREC_FP64, and the GPU-side oracle at N = 2^20.
//
// The pair formula is ph4's (src/amuse_ph4/src/idata.cc:188-226), as in
// kern_force.cu, all in FP64.
//
// What bounds it: GB300 issues FP64 at 2 lanes per SM and cycle, so an FP64
// warp instruction costs 16 cycles of its SM whether one lane or 32 have work,
// and the 64 B of a j record are nothing beside the ~32 instructions spent on
// it.  Hence:
//   * one warp per CTA and no shared memory: records are read from L2 / L1
//     with the next one already in flight, and the work spreads over the SMs
//     in units of a warp (four-warp CTAs with four i per thread left SMs idle
//     and computed padding: 44 us for one i against 1024 j, 107 us for 356 i;
//     this shape 13 and 33 us);
//   * a warp holds IL i-lanes x 32/IL j-lanes of one i each, IL the width
//     that pads the block least; the j range is cut into nsplit chunks of any
//     length (no tiles), so that every SM has warps to switch between;
//   * few FP64 instructions per pair: 1/sqrt from the FP64 MUFU seed (no
//     conversions) and one third-order step, the nearest neighbour kept with
//     integer compares, the self pair masked by a select;
//   * the warp whose ticket completes an i-group adds the chunks' partial
//     sums in chunk order (no second launch; deterministic).
#include "pdl.cuh"
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "fp64_approx.cuh"
#include "g6_dev.h"

namespace {

struct __align__(16) Rec64 {  // the predictor's FP64 record, 64 B
  double x, y, z, m, vx, vy, vz, pad;
};
static_assert(sizeof(Rec64) == 64, "fp64 record");

struct Sum64 {  // partial record of one i and one chunk, 72 B
  double a[3], j[3], p;
  unsigned long long key;  // bits of ph4's r^2 of the nearest j so far
  int nn, pad;
};
static_assert(sizeof(Sum64) == 72, "partial record");

struct K64 {
  int ni, nj, nsplit, chunk;  // chunk: j per split
  double eps2;
  const double *ipos, *ivel;
  const int *ilist, *iself;
  const Rec64 *rec;
  double *acc, *jerk, *pot;
  int *nn;
  float *nn_r2;
  Sum64 *part;      // [nsplit][ni] when nsplit > 1
  unsigned *ticket;  // per i-group, zero between launches
};

constexpr unsigned long long INF_BITS = 0x7ff0000000000000ull;
constexpr unsigned FULL = 0xffffffffu;
constexpr int FOLD = 64;  // records per lane between folds

__device__ __forceinline__ Rec64 load_rec(const Rec64 *p) {
  const double2 *q = reinterpret_cast<const double2 *>(p);
  const double2 a = q[0], b = q[1], c = q[2], d = q[3];
  Rec64 r;
  r.x = a.x; r.y = a.y; r.z = b.x; r.m = b.y;
  r.vx = c.x; r.vy = c.y; r.vz = d.x; r.pad = 0.0;
  return r;
}

// The nearer of two candidates; the smaller slot on equal keys (keys are
// bits of values >= +0, which order like the values).
__device__ __forceinline__ void nn_take(unsigned long long &k, int &n, unsigned long long ok,
                                        int on) {
  if (ok < k || (ok == k && (unsigned)on < (unsigned)n)) {
    k = ok;
    n = on;
  }
}

// FOLDS: a lane has more than FOLD records of its chunk and adds them up FOLD at a
// time.  One running sum over all of them had up to four times the rounding error
// (and unfolded below 128 still a tenth more: rms of the jerk for 501 i, 16384 j,
// 114 records a lane, against 128-bit sums 6.1e-16, folded 4.8e-16).  The totals take 14 registers and 8 of 28 warps off an SM, which shape64
// allows for.  Tried for them: shared memory (an SM takes no CTA of this kernel
// before its last one of the predictor has ended and its L1 is divided anew, and
// the CTAs crowd on the SMs that are through: 501 i, 16384 j 576 -> 1015 us) and
// local memory (570 us, but 675 for 605 on a call after other work).
template <bool NN, bool HJ, bool FOLDS>
__global__ void __launch_bounds__(32) force64_kernel(K64 kp, int il_log2) {
  pdl_wait();  // the predictor's records and the block list are complete
  const int lane = threadIdx.x;
  const int IL = 1 << il_log2, JL = 32 >> il_log2;
  const int i = blockIdx.x * IL + (lane & (IL - 1));
  const int jl = lane >> il_log2;
  const bool valid = i < kp.ni;
  const int ii = valid ? i : 0;
  double x, y, z, vx, vy, vz;
  int self;
  if (kp.ilist) {
    const int slot = kp.ilist[ii];
    const Rec64 r = load_rec(kp.rec + slot);
    x = r.x; y = r.y; z = r.z;
    vx = r.vx; vy = r.vy; vz = r.vz;
    self = kp.iself ? kp.iself[ii] : slot;
  } else {
    x = kp.ipos[3 * ii]; y = kp.ipos[3 * ii + 1]; z = kp.ipos[3 * ii + 2];
    vx = kp.ivel[3 * ii]; vy = kp.ivel[3 * ii + 1]; vz = kp.ivel[3 * ii + 2];
    self = kp.iself ? kp.iself[ii] : -1;
  }
  Sum64 s;
#pragma unroll
  for (int k = 0; k < 3; k++) s.a[k] = s.j[k] = 0.0;
  s.p = 0.0;
  s.key = INF_BITS;
  s.nn = -1;
  s.pad = 0;
  const double eps2 = kp.eps2 + 1.0 / 4503599627370496.0;  // eps^2 + 2^-52 (ph4)
  const int j0 = blockIdx.y * kp.chunk;
  const int j1 = min(kp.nj, j0 + kp.chunk);
  const int last = kp.nj - 1;
  Rec64 nxt = load_rec(kp.rec + min(j0 + jl, last));
  double ta[3] = {0.0, 0.0, 0.0}, tj[3] = {0.0, 0.0, 0.0}, tp = 0.0;
  for (int jb = j0 + jl;;) {
    const int je = FOLDS ? min(j1, jb + FOLD * JL) : j1;
#pragma unroll 2
    for (int j = jb; j < je; j += JL) {
      const Rec64 r = nxt;
      nxt = load_rec(kp.rec + min(j + JL, last));
      const double dx = r.x - x, dy = r.y - y, dz = r.z - z;
      double r2;
      if (NN) {
        // ph4's key: the unsoftened r^2 summed in component order without
        // contraction (idata.cc:200-205,214-218), so the argmin (first slot on
        // equal keys) is ph4's neighbour bit for bit
        const double key = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                     __dmul_rn(dz, dz));
        const unsigned long long kb = (unsigned long long)__double_as_longlong(key);
        if (j != self && kb < s.key) {
          s.key = kb;
          s.nn = j;
        }
        r2 = key + eps2;
      } else {
        r2 = __fma_rn(dz, dz, __fma_rn(dy, dy, __fma_rn(dx, dx, eps2)));
      }
      double rinv = fp64::rsqrt64_normal(r2);
      rinv = j == self ? 0.0 : rinv;
      const double dvx = r.vx - vx, dvy = r.vy - vy, dvz = r.vz - vz;
      const double rv = __fma_rn(dz, dvz, __fma_rn(dy, dvy, dx * dvx));
      const double rinv2 = rinv * rinv;
      const double mri = r.m * rinv;
      const double mr3i = mri * rinv2;
      double a3;
      if (HJ) {  // the hermite code's jerk (src/amuse_hermite/interface.cc:440-449,486)
        const double q = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
        a3 = j == self ? 0.0 : -3.0 * (rv * fp64::rcp64(q));
      } else {
        a3 = -3.0 * (rv * rinv2);
      }
      s.a[0] = __fma_rn(mr3i, dx, s.a[0]);
      s.a[1] = __fma_rn(mr3i, dy, s.a[1]);
      s.a[2] = __fma_rn(mr3i, dz, s.a[2]);
      s.j[0] = __fma_rn(mr3i, __fma_rn(a3, dx, dvx), s.j[0]);
      s.j[1] = __fma_rn(mr3i, __fma_rn(a3, dy, dvy), s.j[1]);
      s.j[2] = __fma_rn(mr3i, __fma_rn(a3, dz, dvz), s.j[2]);
      s.p += mri;
    }
    jb += FOLD * JL;
    if (!FOLDS || jb >= j1) break;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ta[k] += s.a[k];
      tj[k] += s.j[k];
      s.a[k] = s.j[k] = 0.0;
    }
    tp += s.p;
    s.p = 0.0;
  }
  if (FOLDS) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      s.a[k] += ta[k];
      s.j[k] += tj[k];
    }
    s.p += tp;
  }
  pdl_trigger();  // j loop done: the next kernel of the chain may be scheduled

  auto merge_lanes = [&](Sum64 &v) {
    for (int o = 16; o >= IL; o >>= 1) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        v.a[k] += __shfl_down_sync(FULL, v.a[k], o);
        v.j[k] += __shfl_down_sync(FULL, v.j[k], o);
      }
      v.p += __shfl_down_sync(FULL, v.p, o);
      if (NN) {
        const unsigned long long ok = __shfl_down_sync(FULL, v.key, o);
        const int on = __shfl_down_sync(FULL, v.nn, o);
        nn_take(v.key, v.nn, ok, on);
      }
    }
  };
  auto finish = [&](const Sum64 &v) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      kp.acc[3 * i + k] = v.a[k];
      kp.jerk[3 * i + k] = v.j[k];
    }
    kp.pot[i] = -v.p;
    if (kp.nn) kp.nn[i] = NN ? v.nn : -1;
    if (kp.nn_r2)
      kp.nn_r2[i] = NN && v.nn >= 0 ? (float)__longlong_as_double((long long)v.key)
                                    : __int_as_float(0x7f800000);
  };

  merge_lanes(s);  // lanes 0 .. IL-1 now hold their i's sums of this chunk
  if (kp.nsplit == 1) {
    if (valid && jl == 0) finish(s);
    return;
  }
  if (valid && jl == 0) kp.part[(size_t)blockIdx.y * kp.ni + i] = s;
  __threadfence();
  __syncwarp();
  unsigned t = 0;
  if (lane == 0) t = atomicAdd(&kp.ticket[blockIdx.x], 1u);
  t = __shfl_sync(FULL, t, 0);
  if (t != (unsigned)(kp.nsplit - 1)) return;
  __threadfence();
  // the group's last warp: j-lane l adds chunks l, l + JL, ... in order, then
  // the lanes merge as above (the order depends on the shape alone)
  Sum64 v;
#pragma unroll
  for (int k = 0; k < 3; k++) v.a[k] = v.j[k] = 0.0;
  v.p = 0.0;
  v.key = INF_BITS;
  v.nn = -1;
  if (valid) {
#pragma unroll 4
    for (int sp = jl; sp < kp.nsplit; sp += JL) {
      const Sum64 *q = kp.part + (size_t)sp * kp.ni + i;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        v.a[k] += __ldcg(&q->a[k]);
        v.j[k] += __ldcg(&q->j[k]);
      }
      v.p += __ldcg(&q->p);
      if (NN) nn_take(v.key, v.nn, __ldcg(&q->key), __ldcg(&q->nn));
    }
  }
  merge_lanes(v);
  if (valid && jl == 0) finish(v);
  if (lane == 0) kp.ticket[blockIdx.x] = 0u;
}

// Launch shape: the i-lanes per warp and the number of j chunks with the
// smallest estimated time.  Per warp, an FP64 instruction takes 16 cycles of
// its SM: PAIR of them per j record and lane group, LVL per shuffle level,
// FIX for the rest; the warps of an SM share its FP64 unit.  A warp by itself
// takes STEP cycles per record (dependent chain, load); 1.2 of that over the
// number of warps per SM is added: about five keep the unit busy (89 i
// against 1024 j: 24 us at two warps per SM, 18 at five; 33 against 16384: 74
// and 45).  Chunks are merged by one warp per i-group, ADD cycles each.
struct Shape64 {
  int il_log2, nsplit, chunk;
};
struct Cached64 {
  int ni, nj, nn, fjl, fns, groups_max;
  Shape64 s;
};
Cached64 g_cache[256];

Shape64 shape64(int ni, int nj, int nn, int force_jl, int force_ns, int groups_max) {
  const unsigned h = ((unsigned)ni * 2654435761u ^ (unsigned)nj * 40503u ^ (unsigned)nn) >> 7 & 255u;
  Cached64 &c = g_cache[h];
  if (c.ni == ni && c.nj == nj && c.nn == nn && c.fjl == force_jl && c.fns == force_ns &&
      c.groups_max == groups_max && c.s.nsplit > 0)
    return c.s;
  const double PAIR = nn ? 36.0 : 33.0, LVL = 9.0, FIX = 120.0, STEP = 2000.0, ADD = 300.0;
  const double C = 16.0;  // cycles of an FP64 warp instruction
  const int sms = g6k_sm_count();
  int lo = 0, hi = 5;
  while (hi > 0 && (1 << (hi - 1)) >= ni) hi--;
  if (force_jl > 0) {
    int l = 0;
    while ((1 << l) < 32 && (32 >> l) > force_jl) l++;
    lo = hi = l;
  }
  Shape64 best = {hi, 1, nj};
  double bc = 1e300;
  for (int l = lo; l <= hi; l++) {
    const int IL = 1 << l, JL = 32 >> l;
    const long long G = (ni + IL - 1) / IL;
    // more chunks than this would not fit what a caller without allocations
    // has (16 MiB), the ticket array or a useful chunk length
    long long smax = (16ll << 20) / ((long long)ni * (long long)sizeof(Sum64));
    if (G > groups_max) smax = 1;
    if (smax > 96) smax = 96;
    if (smax > nj) smax = nj;
    if (smax < 1) smax = 1;
    for (int ns0 = 1; ns0 <= smax; ns0 += ns0 < 32 ? 1 : 4) {
      int ns = force_ns > 0 ? (int)(force_ns < smax ? force_ns : smax) : ns0;
      const int chunk = (nj + ns - 1) / ns;
      ns = (nj + chunk - 1) / chunk;
      const double it = (double)((chunk + JL - 1) / JL);
      const double instr = it * PAIR + (5 - l) * LVL + FIX;
      const double per_sm = (double)((G * ns + sms - 1) / sms);
      double cost = per_sm * instr * C + 1.2 / (per_sm > 1.2 ? per_sm : 1.2) * (it * STEP + (5 - l) * 300.0);
      if (it > FOLD) {
        // 20 warps per SM hold the totals, for 28: where that takes a second
        // wave, the part of a warp's time by which it ends later
        const int tail = ((int)per_sm - 1) % 20 + 1;
        if (per_sm > 20 && per_sm <= 28) cost += (tail < 4 ? 0.5 * (5 - tail) : 0.8) * instr * C;
        cost *= 1.004;
      }
      if (ns > 1) cost += 2000.0 + ((ns + JL - 1) / JL) * ADD + (5 - l) * 300.0;
      if (cost < bc * 0.999) {
        bc = cost;
        best.il_log2 = l;
        best.nsplit = ns;
        best.chunk = chunk;
      }
      if (force_ns > 0) break;
    }
  }
  c.ni = ni;
  c.nj = nj;
  c.nn = nn;
  c.fjl = force_jl;
  c.fns = force_ns;
  c.groups_max = groups_max;
  c.s = best;
  return best;
}

}  // namespace

// Bytes of partial sums that g6k_force64 needs for this call.
extern "C" size_t g6k_force64_scratch(int ni, int nj, int nn, int force_jl, int force_nsplit,
                                      int groups_max) {
  if (ni <= 0 || nj <= 0) return 0;
  const Shape64 s = shape64(ni, nj, nn ? 1 : 0, force_jl, force_nsplit, groups_max);
  return s.nsplit > 1 ? (size_t)s.nsplit * (size_t)ni * sizeof(Sum64) : 0;
}

// ticket: groups_max zeroed counters (left zero), or NULL with groups_max 0
// (no j chunks then).
extern "C" int g6k_force64(const g6_force_args *a, unsigned *ticket, int groups_max,
                           g6_shape *shape, cudaStream_t st) {
  const Shape64 s = shape64(a->ni, a->nj, a->want_nn ? 1 : 0, a->hjerk ? 1 : a->force_jl,
                            a->force_nsplit, groups_max);
  const int IL = 1 << s.il_log2;
  const int gx = (a->ni + IL - 1) / IL;
  K64 k;
  k.ni = a->ni;
  k.nj = a->nj;
  k.nsplit = s.nsplit;
  k.chunk = s.chunk;
  k.eps2 = a->eps2;
  k.ipos = a->ipos;
  k.ivel = a->ivel;
  k.ilist = a->ilist;
  k.iself = a->iself;
  k.rec = reinterpret_cast<const Rec64 *>(a->js->jp_f64);
  k.acc = a->acc;
  k.jerk = a->jerk;
  k.pot = a->pot;
  k.nn = a->nn;
  k.nn_r2 = a->nn_r2;
  k.part = reinterpret_cast<Sum64 *>(a->scratch);
  k.ticket = ticket;
  if (s.nsplit > 1 && (size_t)s.nsplit * (size_t)a->ni * sizeof(Sum64) > a->scratch_bytes)
    return -4;
  if (shape) {
    shape->jl = 32 / IL;
    shape->nsplit = s.nsplit;
    shape->grid_x = gx;
    shape->grid_y = s.nsplit;
    shape->threads = 32;
  }
  const dim3 grid(gx, s.nsplit), block(32);
  const bool fold = (s.chunk + 32 / IL - 1) / (32 / IL) > FOLD;
  auto kern = a->hjerk     ? (fold ? force64_kernel<false, true, true>
                                    : force64_kernel<false, true, false>)
              : a->want_nn ? (fold ? force64_kernel<true, false, true>
                                    : force64_kernel<true, false, false>)
                           : (fold ? force64_kernel<false, false, true>
                                    : force64_kernel<false, false, false>);
  launch_pdl(kern, grid, block, 0, st, k, s.il_log2);
  if (a->ev_mid) cudaEventRecord(a->ev_mid, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
