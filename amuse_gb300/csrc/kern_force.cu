// kern_force.cu -- the i-block Hermite force kernel (acc, jerk, pot, nearest
// neighbour) for sm_103a in split precision (the plain FP64 kernel is
// kern_force64.cu):
//
//   split: positions as double-single (hi+lo float pairs), relative
//          position formed by (xj_hi - xi_hi) + (xj_lo - xi_lo), all pair
//          arithmetic in FP32 (one MUFU rsqrt per pair), per-tile FP32
//          partial sums folded into compensated (TwoSum) hi/lo totals.
//          The j records are stored in pairs (every field a float2 of two
//          consecutive j), so each packed f32x2 instruction (add/sub/mul/fma
//          .rn.f32x2) evaluates one i against two j: half the issue slots of
//          scalar code for the same FP32 work.
//
// The pair formula is ph4's (src/amuse_ph4/src/idata.cc:188-226):
//   dx = xj - xi, dv = vj - vi, r2 = |dx|^2 + eps2 (+2^-52 as ph4),
//   rinv = r2^-1/2, mr3i = m rinv^3,
//   acc += mr3i dx, jerk += mr3i (dv - 3 (dx.dv)/r2 dx), pot -= m rinv,
//   nn = argmin r2 over j != self (first j on ties).
// The GRAPE-6 semantics of the g6 API excludes the i-particle itself by
// identity (lib/sapporo_light/dev_evaluate_gravity.cu:80-84 compares ids);
// here the host resolves id -> j slot once per call and the kernel skips
// that slot.
//
// Structure (one CTA = 128 threads = 4 warps; 2 i-particles per thread, 3
// CTAs per SM):
//   * j-tiles of 256 records are streamed HBM/L2 -> shared memory with
//     cp.async.bulk (TMA, non-tensor) completing on an mbarrier; warps
//     consume the ring independently (no CTA barrier in the loop).
//   * JL j-lanes share each i-particle (JL = 1 for large i-blocks, up to
//     128 for tiny ones); j is also split across CTAs (grid.y) so that small
//     active blocks still fill all 152 SMs.
//   * Lanes of one i merge with warp shuffles, for JL >= 16 through a table
//     in shared memory; CTAs of one i merge in the last CTA of the group (one
//     or two i per group) or in a second kernel, in fixed order, with
//     float-float adds: deterministic.
//   * Nearest neighbour (optional, a template flag): the hot loop keeps only
//     a running min of r2 (one FMNMX per pair) and the tile where it last
//     improved; after the loop that tile is re-read from L2 and re-scanned
//     with bit-identical arithmetic to find the index.
//   * A tile that holds the self slot of one of the warp's i-particles takes
//     a checked copy of the loop (rinv = 0, r2 -> +inf for self).
#include "pdl.cuh"
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "fp64_approx.cuh"
#include "g6_dev.h"

namespace {

// Tuning constants (compile-time; the defaults are the measured best).
#ifndef G6_NT
#define G6_NT 128
#endif
#ifndef G6_IPT
#define G6_IPT 2
#endif
#ifndef G6_UNROLL_NN
#define G6_UNROLL_NN 4  // j-loop unroll factor of the nearest-neighbour variant
#endif
#ifndef G6_UNROLL
#define G6_UNROLL 8
#endif
#ifndef G6_MINB
#define G6_MINB 3
#endif
#ifndef G6_XMERGE_MAX
#define G6_XMERGE_MAX 2  // split merge in the force kernel at most for so many i per group
#endif
#ifndef G6_JCHUNK
#define G6_JCHUNK 32  // split: records per jerk fold
#endif
#ifndef G6_TOT_SMEM
#define G6_TOT_SMEM 2  // split: compensated totals in shared memory (2: with NN only)
#endif
constexpr int NT = G6_NT;    // threads per CTA
constexpr int TJ = G6_TILE;  // j records per tile
constexpr int IPT_SPLIT = G6_IPT;  // i-particles per thread
constexpr int UNROLL = G6_UNROLL;  // j-loop unroll factor (the best measured: 8
                                    // plain, 4 with the nearest neighbour, 16
                                    // with the hermite jerk: 131072 bodies
                                    // 19.09 -> 18.90 ms)
constexpr int JLMAX = TJ < NT ? TJ : NT;  // j-lanes per i at most
constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s bound per wait
constexpr unsigned long long STALL_TEST_NS = 20000000ull;  // 20 ms under the test hook

enum { ERR_TMA_TIMEOUT = 1, ERR_SHAPE = 2 };

// Split records come in pairs of consecutive j slots, every field a float2
// {j even, j odd} (the global layout the predictor writes, g6_dev.h), so a
// packed f32x2 instruction evaluates two j at once.
struct __align__(16) RecS {
  float2 xh, yh, zh, m, xl, yl, zl, ml, vx, vy, vz, pad1;  // ml: the mass's low part
};
static_assert(sizeof(RecS) == 96, "split record pair");

// ---------------------------------------------------------------- PTX ---
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile(
      "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void tma_load_1d(void *dst, const void *src, uint32_t bytes,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
      "[%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait that also gives up when another warp of the CTA raised
// *abort (false in both cases, or after limit_ns of global time).
__device__ __forceinline__ bool mbar_wait_abortable(uint64_t *bar, uint32_t parity,
                                                    volatile int *abort,
                                                    unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort) return false;
    if (gtimer() - t0 > limit_ns) return false;
  }
}
// Bounded wait: false after limit_ns of global time.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (gtimer() - t0 > limit_ns) return false;
  }
}

// One MUFU.RSQ, flush-to-zero (r2 >= eps2 + 2^-52 is never subnormal).
// (A Newton step after it costs 13% and does not change the block-step
// behaviour measured at eta = 0.01..0.14, so there is none.)
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One MUFU.RCP, flush-to-zero.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// max(a, b, c) and min(a, b, c) in one ALU instruction each (3-input
// max.f32 / min.f32).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// ------------------------------------------------------- float-float ---
// Knuth TwoSum folded into a (hi, lo) accumulator.
__device__ __forceinline__ void ff_acc(float &hi, float &lo, float p) {
  const float s = __fadd_rn(hi, p);
  const float bb = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  hi = s;
  lo = __fadd_rn(lo, e);
}
// (ah, al) += (bh, bl), renormalised.
__device__ __forceinline__ void ff_add(float &ah, float &al, float bh, float bl) {
  const float s = __fadd_rn(ah, bh);
  const float bb = __fsub_rn(s, ah);
  float e = __fadd_rn(__fsub_rn(ah, __fsub_rn(s, bb)), __fsub_rn(bh, bb));
  e = __fadd_rn(e, __fadd_rn(al, bl));
  ah = __fadd_rn(s, e);
  al = __fsub_rn(e, __fsub_rn(ah, s));
}

struct KParams;

// ------------------------------------------------------------ policies ---
struct SplitP {
  using Rec = RecS;
  using R = float;
  static constexpr int JPR = 2;     // j per record (packed pair)
  static constexpr int IPT = IPT_SPLIT;
  static constexpr int NSTAGE = 3;  // TMA ring depth (3 x 12 KB)
  static constexpr int MINB = G6_MINB;  // resident CTAs per SM
  struct I {  // i values duplicated into both halves
    f2x xh, yh, zh, xl, yl, zl, vx, vy, vz;
  };
  struct Part {  // per-fold-period partial sums, one per half
    f2x a[3], j[3], p, s;
  };
  struct Tot {  // compensated totals (s: plain sum, an estimate), largest chunk of s
    float ah[3], al[3], jh[3], jl[3], ph, pl, s, mt, pad;  // 17 words: odd stride
  };
  struct __align__(16) Out {  // partial record exchanged between CTAs, 80 B
    float2 a[3], j[3], p;
    float nnr2;   // smallest nearest-neighbour key (r^2 + eps^2, FP32)
    float nnr2b;  // second smallest key over the other j
    float s1;     // sum of m / (r^2 + eps^2): the condition number's numerator
    float mt;     // largest partial sum of s over 32 j: bounds the largest term
    int nn;
    int pad;
  };
  __device__ static void split(double d, float &h, float &l) {
    h = __double2float_rn(d);
    l = __double2float_rn(d - (double)h);
  }
  __device__ static I dup(float xh, float yh, float zh, float xl, float yl, float zl, float vx,
                          float vy, float vz) {
    I s;
    s.xh = f2_pack(xh, xh); s.yh = f2_pack(yh, yh); s.zh = f2_pack(zh, zh);
    s.xl = f2_pack(xl, xl); s.yl = f2_pack(yl, yl); s.zl = f2_pack(zl, zl);
    s.vx = f2_pack(vx, vx); s.vy = f2_pack(vy, vy); s.vz = f2_pack(vz, vz);
    return s;
  }
  __device__ static I load_i_explicit(const double *p, const double *v) {
    float xh, yh, zh, xl, yl, zl;
    split(p[0], xh, xl);
    split(p[1], yh, yl);
    split(p[2], zh, zl);
    return dup(xh, yh, zh, xl, yl, zl, __double2float_rn(v[0]), __double2float_rn(v[1]),
               __double2float_rn(v[2]));
  }
  __device__ static I load_i_slot(const void *recs, int slot) {
    return dup(g6_split_get(recs, slot, 0), g6_split_get(recs, slot, 1),
               g6_split_get(recs, slot, 2), g6_split_get(recs, slot, 4),
               g6_split_get(recs, slot, 5), g6_split_get(recs, slot, 6),
               g6_split_get(recs, slot, 8), g6_split_get(recs, slot, 9),
               g6_split_get(recs, slot, 10));
  }
  __device__ static void zero(Part &q) {
#pragma unroll
    for (int k = 0; k < 3; k++) q.a[k] = q.j[k] = 0ull;
    q.p = 0ull;
    q.s = 0ull;
  }
  __device__ static void zero(Tot &t) {
#pragma unroll
    for (int k = 0; k < 3; k++) t.ah[k] = t.al[k] = t.jh[k] = t.jl[k] = 0.f;
    t.ph = t.pl = 0.f;
    t.s = t.mt = 0.f;
  }
  __device__ static void fold(Tot &t, const Part &q) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ff_acc(t.ah[k], t.al[k], f2_lo(q.a[k]));
      ff_acc(t.ah[k], t.al[k], f2_hi(q.a[k]));
      ff_acc(t.jh[k], t.jl[k], f2_lo(q.j[k]));
      ff_acc(t.jh[k], t.jl[k], f2_hi(q.j[k]));
    }
    ff_acc(t.ph, t.pl, f2_lo(q.p));
    ff_acc(t.ph, t.pl, f2_hi(q.p));
    fold_s(t, q);
  }
  // The condition number's sum arrives in chunks of at most 32 j per half
  // (the jerk fold period): the largest chunk bounds the largest single term
  // m / (r^2 + eps^2) from above, for the price of one 3-input maximum per
  // chunk rather than per pair.
  __device__ static __forceinline__ void fold_s(Tot &t, const Part &q) {
    t.s += f2_lo(q.s) + f2_hi(q.s);
    t.mt = fmax3(t.mt, f2_lo(q.s), f2_hi(q.s));
  }
  // r^2 + eps^2 of both j of a record (the nearest-neighbour key): the main
  // loop and the re-scan use this same arithmetic, so the keys are
  // bit-identical.
  __device__ static __forceinline__ f2x r2e(const I &s, const Rec &r, f2x eps2, f2x &dx, f2x &dy,
                                            f2x &dz) {
    dx = f2_add(f2_sub(f2_of(r.xh), s.xh), f2_sub(f2_of(r.xl), s.xl));
    dy = f2_add(f2_sub(f2_of(r.yh), s.yh), f2_sub(f2_of(r.yl), s.yl));
    dz = f2_add(f2_sub(f2_of(r.zh), s.zh), f2_sub(f2_of(r.zl), s.zl));
    return f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, eps2)));
  }
  // Both j of record r on one i.  selfrel = (self slot) - (slot of the
  // record's first j): half h is the i itself when selfrel == h (CHECK only).
  // HJ: the jerk as the hermite code forms it (src/amuse_hermite/
  // interface.cc:440-449,469-486): the (r.v) factor divided by the
  // UNsoftened r^2.
  //
  // NN keeps the smallest key of the tile (nnmin, one 3-input minimum per j pair); the
  // kernel turns the tile minima into the smallest and second smallest key
  // over all j, whose gap decides whether the FP32 argmin is provably ph4's
  // FP64 nearest neighbour (finish() below).  Without HJ the sum of
  // m / (r^2 + eps^2) (Part::s) is kept for the condition number of the
  // acceleration sum.
  template <bool CHECK, bool NN, bool HJ = false>
  __device__ static __forceinline__ void pair(const I &s, const Rec &r, f2x eps2, Part &q,
                                              float &nnmin, int selfrel) {
    f2x dx, dy, dz;
    const f2x r2 = r2e(s, r, eps2, dx, dy, dz);
    const float r2a = f2_lo(r2), r2b = f2_hi(r2);
    float ra = rsqrt_approx(r2a), rb = rsqrt_approx(r2b);
    if (CHECK) {
      ra = selfrel == 0 ? 0.f : ra;
      rb = selfrel == 1 ? 0.f : rb;
      if (NN) {
        const float inf = __int_as_float(0x7f800000);
        nnmin = fmin3(nnmin, selfrel == 0 ? inf : r2a, selfrel == 1 ? inf : r2b);
      }
    } else if (NN) {
      nnmin = fmin3(nnmin, r2a, r2b);
    }
    const f2x rinv = f2_pack(ra, rb);
    const f2x dvx = f2_sub(f2_of(r.vx), s.vx);
    const f2x dvy = f2_sub(f2_of(r.vy), s.vy);
    const f2x dvz = f2_sub(f2_of(r.vz), s.vz);
    const f2x rv = f2_fma(dz, dvz, f2_fma(dy, dvy, f2_mul(dx, dvx)));
    const f2x rinv2 = f2_mul(rinv, rinv);
    const f2x mri = f2_mul(f2_of(r.m), rinv);
    const f2x mr3i = f2_mul(mri, rinv2);
    const f2x m3 = f2_pack(-3.0f, -3.0f);
    f2x a3;
    if (HJ) {
      const f2x r2u = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
      float ia = rcp_approx(f2_lo(r2u)), ib = rcp_approx(f2_hi(r2u));
      if (CHECK) {
        ia = selfrel == 0 ? 0.f : ia;
        ib = selfrel == 1 ? 0.f : ib;
      }
      a3 = f2_mul(m3, f2_mul(rv, f2_pack(ia, ib)));
    } else {
      a3 = f2_mul(m3, f2_mul(rv, rinv2));
    }
    q.a[0] = f2_fma(mr3i, dx, q.a[0]);
    q.a[1] = f2_fma(mr3i, dy, q.a[1]);
    q.a[2] = f2_fma(mr3i, dz, q.a[2]);
    q.j[0] = f2_fma(mr3i, f2_fma(a3, dx, dvx), q.j[0]);
    q.j[1] = f2_fma(mr3i, f2_fma(a3, dy, dvy), q.j[1]);
    q.j[2] = f2_fma(mr3i, f2_fma(a3, dz, dvz), q.j[2]);
    q.p = f2_add(q.p, mri);
    if (!HJ) q.s = f2_fma(mri, rinv, q.s);  // the condition number's sum
  }
  // Nearest-neighbour re-scan of one record of the best tile: the first j
  // (in slot order) whose key equals best and that is not the i itself
  // becomes idx; every other key lowers m2 (the second smallest key).
  __device__ static __forceinline__ void rescan(const I &s, const Rec &r, f2x eps2, float best,
                                                int slot0, int self, int &idx, float &m2) {
    f2x dx, dy, dz;
    const f2x r2 = r2e(s, r, eps2, dx, dy, dz);
    const float kk[2] = {f2_lo(r2), f2_hi(r2)};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (slot0 + h == self) continue;
      if (idx < 0 && kk[h] == best)
        idx = slot0 + h;
      else
        m2 = fminf(m2, kk[h]);
    }
  }
  // Mid-tile fold of the jerk partial sums (and of the condition number's
  // chunk): the jerk sum cancels more than the others, so it is folded every
  // JCHUNK records.
  static constexpr bool JFOLD = true;
  // shared-memory totals free registers: they pay off in the nearest-
  // neighbour variant, not in the plain one (measured)
  template <bool NN>
  __host__ __device__ static constexpr bool tot_shared() {
    return G6_TOT_SMEM == 1 || (G6_TOT_SMEM == 2 && NN);
  }
  __device__ static void fold_jerk(Tot &t, Part &q) {
    fold_s(t, q);
    q.s = 0ull;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ff_acc(t.jh[k], t.jl[k], f2_lo(q.j[k]));
      ff_acc(t.jh[k], t.jl[k], f2_hi(q.j[k]));
      q.j[k] = 0ull;
    }
  }
  __device__ static f2x eps(double eps2) {
    const float e = (float)eps2 + (float)(1.0 / 4503599627370496.0);  // + 2^-52 (ph4)
    return f2_pack(e, e);
  }
  __device__ static void to_out(const Tot &t, float nnr2, float nnr2b, int nn, Out &o) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      o.a[k] = make_float2(t.ah[k], t.al[k]);
      o.j[k] = make_float2(t.jh[k], t.jl[k]);
    }
    o.p = make_float2(t.ph, t.pl);
    o.nnr2 = nnr2;
    o.nnr2b = nnr2b;
    o.s1 = t.s;
    o.mt = t.mt;
    o.nn = nn;
    o.pad = 0;
  }
  __device__ static void to_out_zero(Out &o) {  // merge's neutral element
#pragma unroll
    for (int k = 0; k < 3; k++) o.a[k] = o.j[k] = make_float2(0.f, 0.f);
    o.p = make_float2(0.f, 0.f);
    o.nnr2 = o.nnr2b = __int_as_float(0x7f800000);
    o.s1 = o.mt = 0.f;
    o.nn = 0x7fffffff;
    o.pad = 0;
  }
  __device__ static void merge(Out &a, const Out &b) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ff_add(a.a[k].x, a.a[k].y, b.a[k].x, b.a[k].y);
      ff_add(a.j[k].x, a.j[k].y, b.j[k].x, b.j[k].y);
    }
    ff_add(a.p.x, a.p.y, b.p.x, b.p.y);
    a.s1 += b.s1;
    a.mt = fmaxf(a.mt, b.mt);
    // second smallest of the four keys: min(max of the minima, min of the seconds)
    const float m2 = fminf(fmaxf(a.nnr2, b.nnr2), fminf(a.nnr2b, b.nnr2b));
    if (b.nnr2 < a.nnr2 || (b.nnr2 == a.nnr2 && b.nn < a.nn)) {
      a.nnr2 = b.nnr2;
      a.nn = b.nn;
    }
    a.nnr2b = m2;
  }
  __device__ static void write_final(const Out &o, int i, double *acc, double *jerk,
                                     double *pot) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      acc[3 * i + k] = (double)o.a[k].x + (double)o.a[k].y;
      jerk[3 * i + k] = (double)o.j[k].x + (double)o.j[k].y;
    }
    pot[i] = -((double)o.p.x + (double)o.p.y);
  }
  __device__ static void finish(const Out &o, int i, const KParams &kp);
};

// A partial record written by another CTA of this launch: read around L1.
template <class O>
__device__ __forceinline__ O load_out_cg(const O *p) {
  O r;
  const int *src = reinterpret_cast<const int *>(p);
  int *dst = reinterpret_cast<int *>(&r);
#pragma unroll
  for (int w = 0; w < (int)(sizeof(O) / 4); w++) dst[w] = __ldcg(src + w);
  return r;
}

// Shuffle helpers for Out (field by field).
template <class O>
__device__ __forceinline__ O shfl_xor_out(const O &o, int m) {
  O r;
  const int *src = reinterpret_cast<const int *>(&o);
  int *dst = reinterpret_cast<int *>(&r);
#pragma unroll
  for (int w = 0; w < (int)(sizeof(O) / 4); w++) dst[w] = __shfl_xor_sync(0xffffffffu, src[w], m);
  return r;
}

struct KParams {
  int ni, nj, nsplit, jsplit;  // jsplit: j per CTA-split (multiple of TJ)
  double eps2;
  const double *ipos, *ivel;
  const int *ilist, *iself;
  const void *jrec;
  double *acc, *jerk, *pot;
  int *nn;
  float *nn_r2;
  void *part;  // [nsplit][ni_pad] Out records when nsplit > 1
  int ni_pad;
  int *err;
  int want_nn;
  int hjerk;  // the hermite code's jerk form (JL = 1, no nn only)
  // nearest-neighbour proof and refinement queue (split precision)
  g6_jstate js;   // FP64 state: ph4-predicted positions of i and nn
  double ti;      // prediction time of the records
  void *refine;   // refinement buffer (NULL: none)
  double kappa2;  // squared condition-number limit (0: no FP64 redo)
  // bounded waits: limit per wait; stall (test hook) makes CTA (0, 0) wait
  // for its first tile on a barrier that nothing arrives on
  unsigned long long wait_ns;
  int stall;
  unsigned *xtick;  // per-i-group tickets for the in-kernel split merge (NULL: second pass)
};

// ------------------------------------------------ nearest neighbour proof ---
//
// ph4's nearest neighbour (idata.cc:200-226) is the j with the smallest FP64
// r^2 = (dx^2 + dy^2) + dz^2 of the ph4-predicted positions, the first j on
// equal values.  The split kernel ranks j by the FP32 key k = r^2 + eps^2
// of the double-single records.  Bound (the argument of kern_knn.cu, with
// the softening added first in the FMA chain): with X >= |coordinate| of i
// and of every j within distance sqrt(D) of i, E = 2^-30 X and e the FP32
// softening, any j with ph4 r^2 <= D has
//     k <= Tk(D) = (1 + 2^-16)(D + e) + 4 E sqrt(D) + 4 E^2.
// So if the second smallest key m2 exceeds Tk(D_f), D_f the FP64 r^2 of the
// FP32 argmin j_f, every other j has ph4 r^2 > D_f and j_f is ph4's nearest
// neighbour.  X = max |x_i| + sqrt(D_f) covers every j that could beat it.
// Otherwise (near-equal keys, e.g. distance ties) the i-particle is queued
// and refine_kernel ranks every j with k <= Tk(D_f) in FP64.
//
// ---------------------------------------------- condition-number refinement
//
// The FP32 pair terms carry a few ulps each, so the relative error of the
// acceleration grows with the condition number of its sum,
// kappa = sum m / (r^2 + eps^2) / |a| (about 1e-8 kappa at N = 2^20; the
// particles near the centre of a cluster, where the pulls cancel, reach
// kappa ~ 100-300), and with the largest single term over |a|, whose own
// error does not average out (a massive neighbour pulling against the rest
// of the cluster).  i-particles with kappa above the caller's limit are
// queued (REF_ACC), and refine_kernel recomputes their acceleration and
// potential in FP64 from the same records (double-single positions exact in
// FP64).  Those with kappa below it but a largest term (bounded by the
// largest partial sum over 32 j of one thread) above MU0 |a| are queued for
// the cheaper REF_MT pass: the sum redone with the kernel's FP32 pair terms
// but compensated (TwoSum) accumulation, every term above TAU |a| replaced
// by its float-float value.  That removes the dominant terms' own errors and the
// FP32 partial sums' roundings relative to them, which are what does not
// average out there; the remaining terms are each below TAU |a|, so their
// random errors add up to ~1e-7 sqrt(TAU kappa) |a|.  Common in clusters
// with a mass spectrum (a massive star near the i), REF_MT costs ~50 FP32
// operations per pair where REF_ACC costs ~20 FP64 ones (each 1/64 the
// FP32 rate).  In both the jerk keeps its split value.
//
// Refinement buffer (g6k_refine_bytes, zeroed once): a header, the queue
// (i, reason, key bound), per-entry tickets, per-(entry, chunk) partial
// records, and the force kernel's per-i-group tickets for its in-kernel
// split merge.  refine_kernel leaves the header's count at zero.
constexpr int RCAP = 16384;    // queue entries
constexpr int RPCAP = 32768;   // partial records (entries x chunks)
constexpr int RCHMAX = 64;     // j-chunks per entry at most
constexpr int RNT = 256;       // refine_kernel threads per CTA
constexpr int XTMAX = 8192;    // i-groups (grid.x) whose split merge runs in the force kernel
enum { REF_ACC = 1, REF_NN = 2, REF_MT = 4 };
// Largest single term over |a| above which the sum is redone (REF_MT): a
// term carries up to ~7e-7 relative error (three times the 1.25e-7 of the
// MUFU reciprocal square root, measured over all FP32 inputs in [1, 4), plus
// the roundings of r^2, the differences and the products), and a partial
// sum holding it rounds every later term to its own ulp.  At 1.5 a particle
// with a term of 1.4 |a| reached 1.23e-6 (a star pulling against a cluster,
// 6000 bodies); at 1.0 the worst left unrefined is one term's error.
constexpr double MU0 = 1.0;
// Terms above TAU |a| are evaluated in float-float in the REF_MT pass: at
// 0.02 the remaining terms' random errors stay below ~1e-7 sqrt(0.02 kappa)
// |a| (C2 at 65536 Salpeter: the same largest error as at 0.005).
#ifndef G6_REF_CTAS
#define G6_REF_CTAS 4  // refine_kernel: CTAs per SM (62 registers, 256 threads)
#endif
#ifndef G6_REF_UNITS
#define G6_REF_UNITS 2  // refine_kernel: (entry, j-chunk) units per CTA to aim for
#endif
#ifndef G6_TAU
#define G6_TAU 0.02f
#endif
constexpr float TAU = G6_TAU;

struct RefHdr {
  unsigned count;     // entries queued by this call (reset by refine_kernel)
  unsigned done;      // refine_kernel CTAs finished
  unsigned overflow;  // largest count that exceeded RCAP (sticky until read)
  unsigned last;      // count of the last refinement
  unsigned last_acc;  // of which queued for the condition number
  unsigned nacc;      // REF_ACC entries queued by this call
  unsigned nmt;       // REF_MT entries queued by this call
  unsigned last_mt;   // of the last refinement
  unsigned cmt;       // entries queued for REF_MT alone
};
struct RefPart {  // one j-chunk of one entry, FP64
  double a[3], p, r2;
  int slot, pad;
};
struct RefBuf {
  RefHdr h;
  int list[RCAP];
  int mode[RCAP];
  float thr[RCAP];     // REF_NN: the FP32 key bound
  float thr_mt[RCAP];  // REF_MT: TAU |a|
  unsigned ticket[RCAP];
  RefPart part[RPCAP];
  unsigned xtick[XTMAX];  // force kernel: CTAs of an i-group done (reset by the last)
  // REF_MT alone, nearly all entries of a cluster with a mass spectrum
  int mt_list[RCAP];
  float mt_thr[RCAP];
  unsigned mt_ticket[RCAP];   // per group of entries
  float2 mt_part[RPCAP][4];   // [group][chunk][entry] sums, float-float
};

__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// FP64 position of j slot s predicted to ti with ph4's expression.
__device__ __forceinline__ void jpos64(const g6_jstate &js, double ti, int s, double x[3]) {
  const int cap = js.cap;
  const double dt = dsub(ti, js.t[s]);
#pragma unroll
  for (int k = 0; k < 3; k++)
    x[k] = g6_predict_x(js.x[k * cap + s], js.v[k * cap + s], js.a[k * cap + s],
                        js.j[k * cap + s], dt);
}
// FP64 position of i-particle i as ph4 holds it: the caller's point, or the
// listed slot predicted to ti.
__device__ __forceinline__ void ipos64(const KParams &kp, int i, double x[3]) {
  if (kp.ilist) {
    jpos64(kp.js, kp.ti, kp.ilist[i], x);
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++) x[k] = kp.ipos[3 * i + k];
  }
}
// ph4's r^2 of j relative to i (dx = x_j - x_i), component order, no FMA.
__device__ __forceinline__ double ph4_r2(const double xi[3], const double xj[3]) {
  const double d0 = dsub(xj[0], xi[0]), d1 = dsub(xj[1], xi[1]), d2 = dsub(xj[2], xi[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
}
// An FP32 upper bound of Tk(D): every factor is rounded up or padded by more
// than the roundings of the FP32 evaluation (a larger bound only queues a
// few more particles, whose neighbour the redo finds either way).
__device__ __forceinline__ float nn_bound(double D, float e, const double xi[3]) {
  const float d = __double2float_ru(D);
  const float sD = __fsqrt_ru(d);
  const float X = __fadd_ru(fmaxf(fabsf(__double2float_rn(xi[0])),
                                  fmaxf(fabsf(__double2float_rn(xi[1])),
                                        fabsf(__double2float_rn(xi[2])))),
                            sD);
  const float E = __fmul_ru(X, (1.0f + 1.0f / 524288.0f) * (1.0f / 1073741824.0f));
  const float t = __fmul_ru(1.0f + 1.0f / 65536.0f, __fadd_ru(d, e));
  return __fmaf_ru(4.0f, __fmul_ru(E, __fadd_ru(sD, E)), t);
}
// The FP32 softening of the split key (SplitP::eps).
__device__ __forceinline__ float split_eps(double eps2) {
  return (float)eps2 + (float)(1.0 / 4503599627370496.0);
}

__device__ __forceinline__ void ref_enqueue(void *buf, int i, int mode, float thr,
                                            float thr_mt) {
  RefBuf *b = reinterpret_cast<RefBuf *>(buf);
  if (mode == REF_MT) {
    const unsigned e = atomicAdd(&b->h.cmt, 1u);
    if (e < (unsigned)RCAP) {
      b->mt_list[e] = i;
      b->mt_thr[e] = thr_mt;
    }
    return;
  }
  const unsigned e = atomicAdd(&b->h.count, 1u);
  if (mode & REF_ACC) atomicAdd(&b->h.nacc, 1u);
  if (mode & REF_MT) atomicAdd(&b->h.nmt, 1u);
  if (e < (unsigned)RCAP) {
    b->list[e] = i;
    b->mode[e] = mode;
    b->thr[e] = thr;
    b->thr_mt[e] = thr_mt;
  }
}

__device__ __noinline__ void SplitP::finish(const Out &o, int i, const KParams &kp) {
  write_final(o, i, kp.acc, kp.jerk, kp.pot);
  int mode = 0;
  float thr = 0.f, thr_mt = 0.f;
  // Most sums are far from both limits: an FP32 test with a margin of 1e-3
  // settles those, the FP64 one (16 cycles of the SM per instruction)
  // decides the rest.
  const float a2f = __fmaf_rn(o.a[0].x, o.a[0].x,
                              __fmaf_rn(o.a[1].x, o.a[1].x, __fmul_rn(o.a[2].x, o.a[2].x)));
  const float lim = 0.999f * (float)kp.kappa2 * a2f;
  const bool clear = a2f > 1e-30f && lim < 1e37f && __fmul_rn(o.s1, o.s1) < lim &&
                     __fmul_rn(o.mt, o.mt) < 0.999f * (float)(MU0 * MU0) * a2f;
  if (kp.refine && kp.kappa2 > 0.0 && !clear) {
    double a2 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double a = (double)o.a[k].x + (double)o.a[k].y;
      a2 += a * a;
    }
    const double s1 = (double)o.s1, mt = (double)o.mt;
    if (s1 * s1 > kp.kappa2 * a2) {
      mode |= REF_ACC;
    } else if (mt * mt > MU0 * MU0 * a2) {
      mode |= REF_MT;
      thr_mt = (float)((double)TAU * sqrt(a2));
    }
  }
  const int nn = (o.nn >= 0 && o.nn < kp.nj) ? o.nn : -1;
  if (kp.want_nn) {
    float r2out = __int_as_float(0x7f800000);
    if (nn >= 0) {
      double xi[3], xj[3];
      ipos64(kp, i, xi);
      jpos64(kp.js, kp.ti, nn, xj);
      const double D = ph4_r2(xi, xj);
      r2out = (float)D;
      const float T = nn_bound(D, split_eps(kp.eps2), xi);
      if (kp.refine && !(o.nnr2b > T)) {
        mode |= REF_NN;
        thr = T;
      }
    }
    if (kp.nn) kp.nn[i] = nn;
    if (kp.nn_r2) kp.nn_r2[i] = r2out;
  } else if (kp.nn) {
    kp.nn[i] = -1;
  }
  if (mode) ref_enqueue(kp.refine, i, mode, thr, thr_mt);
}

// ---------------------------------------------------------- lane table ---
//
// The sums of one i over its NL lanes (j-lanes of a CTA, or splits) by way
// of shared memory.  A shuffle tree makes every lane carry all 20 words of
// the record through every level (1250 instructions per warp at JL = 128,
// five times the pair work of one tile).  Here each lane stores its words,
// NT / NI threads per i then take one float-float quantity per eighth of
// them: PARTS threads add NL / PARTS lanes each (independent TwoSums, the
// dependent chain is one addition per lane) and merge by shuffle; the last
// eighth does the condition sum, the largest chunk and the neighbour keys.
// Row pitch NI * NL + 8 words: the eight rows a warp reads start in
// different banks.  The results go to column 0 of the i's first lane.
// For NL >= TAB_JL, where NT / NI >= 8.
constexpr int TAB_JL = 16;
constexpr int TAB_ROWS = 19;  // 7 x (hi, lo), key, second key, s, mt, slot
template <int NL, int NI>
__host__ __device__ constexpr int lane_table_pitch() {
  return NI * NL + 8;
}
template <int NL, int NI>
__host__ __device__ constexpr int lane_table_words() {
  return TAB_ROWS * lane_table_pitch<NL, NI>();
}
template <int NL, int NI>
__device__ __forceinline__ void lane_table_put(float *tab, int i, int l, const SplitP::Out &o) {
  constexpr int P = lane_table_pitch<NL, NI>();
  float *t = tab + i * NL + l;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    t[(2 * k) * P] = o.a[k].x;
    t[(2 * k + 1) * P] = o.a[k].y;
    t[(6 + 2 * k) * P] = o.j[k].x;
    t[(7 + 2 * k) * P] = o.j[k].y;
  }
  t[12 * P] = o.p.x;
  t[13 * P] = o.p.y;
  t[14 * P] = o.nnr2;
  t[15 * P] = o.nnr2b;
  t[16 * P] = o.s1;
  t[17 * P] = o.mt;
  t[18 * P] = __int_as_float(o.nn);
}
template <int NL, int NI>
__device__ __forceinline__ SplitP::Out lane_table_get(const float *tab, int i) {
  constexpr int P = lane_table_pitch<NL, NI>();
  const float *t = tab + i * NL;
  SplitP::Out o;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    o.a[k] = make_float2(t[(2 * k) * P], t[(2 * k + 1) * P]);
    o.j[k] = make_float2(t[(6 + 2 * k) * P], t[(7 + 2 * k) * P]);
  }
  o.p = make_float2(t[12 * P], t[13 * P]);
  o.nnr2 = t[14 * P];
  o.nnr2b = t[15 * P];
  o.s1 = t[16 * P];
  o.mt = t[17 * P];
  o.nn = __float_as_int(t[18 * P]);
  o.pad = 0;
  return o;
}
template <int NL, int NI>
__device__ __forceinline__ void lane_table_sum(float *tab) {
  constexpr int P = lane_table_pitch<NL, NI>();
  constexpr int TPI = NT / NI;       // threads per i
  constexpr int PARTS = TPI / 8;     // threads per quantity
  static_assert(TPI >= 8 && NL % PARTS == 0 && PARTS <= 32, "table");
  const int i = threadIdx.x / TPI, r = threadIdx.x % TPI;
  const int c = r / PARTS, part = r % PARTS;
  float *t = tab + i * NL;
  SplitP::Out o;
  SplitP::to_out_zero(o);
  float h = 0.f, l = 0.f;
  if (c < 7) {
    const float *th = t + 2 * c * P + part, *tl = th + P;
#pragma unroll 4
    for (int q = 0; q < NL / PARTS; q++) {
      ff_acc(h, l, th[q * PARTS]);
      l = __fadd_rn(l, tl[q * PARTS]);
    }
  } else {
    for (int q = 0; q < NL / PARTS; q++) {
      const float *u = t + 14 * P + part + q * PARTS;
      const float k1 = u[0], k2 = u[P];
      const int s = __float_as_int(u[4 * P]);
      o.nnr2b = fminf(fmaxf(o.nnr2, k1), fminf(o.nnr2b, k2));
      if (k1 < o.nnr2 || (k1 == o.nnr2 && s < o.nn)) {
        o.nnr2 = k1;
        o.nn = s;
      }
      o.s1 += u[2 * P];
      o.mt = fmaxf(o.mt, u[3 * P]);
    }
  }
#pragma unroll
  for (int m = 1; m < PARTS; m <<= 1) {
    ff_add(h, l, __shfl_down_sync(0xffffffffu, h, m), __shfl_down_sync(0xffffffffu, l, m));
    const float k1 = __shfl_down_sync(0xffffffffu, o.nnr2, m);
    const float k2 = __shfl_down_sync(0xffffffffu, o.nnr2b, m);
    const float s1 = __shfl_down_sync(0xffffffffu, o.s1, m);
    const float mt = __shfl_down_sync(0xffffffffu, o.mt, m);
    const int s = __shfl_down_sync(0xffffffffu, o.nn, m);
    o.nnr2b = fminf(fmaxf(o.nnr2, k1), fminf(o.nnr2b, k2));
    if (k1 < o.nnr2 || (k1 == o.nnr2 && s < o.nn)) {
      o.nnr2 = k1;
      o.nn = s;
    }
    o.s1 += s1;
    o.mt = fmaxf(o.mt, mt);
  }
  __syncthreads();  // every lane's words are read before column 0 is written
  if (part == 0) {
    if (c < 7) {
      t[2 * c * P] = h;
      t[(2 * c + 1) * P] = l;
    } else {
      t[14 * P] = o.nnr2;
      t[15 * P] = o.nnr2b;
      t[16 * P] = o.s1;
      t[17 * P] = o.mt;
      t[18 * P] = __int_as_float(o.nn);
    }
  }
}

// Number of j per thread between compensated folds.
constexpr int FOLD_J = 64;

template <class P, int JL, bool NN, bool HJ = false>
__global__ void __launch_bounds__(NT, P::MINB) force_kernel(KParams kp) {
  constexpr int NSTAGE = P::NSTAGE;
  using Rec = typename P::Rec;
  using R = typename P::R;
  constexpr int JPR = P::JPR;            // j per record
  constexpr int IPT = P::IPT;            // i-particles per thread
  constexpr int RPT = TJ / JPR;          // records per tile
  constexpr int NIL = NT / JL;           // i-lanes per CTA
  constexpr int ISLOTS = NIL * IPT;      // i-particles per CTA
  constexpr int JPT = RPT / JL;          // records per thread per tile
  constexpr int FOLD_TILES = (FOLD_J / (JPT * JPR)) > 0 ? (FOLD_J / (JPT * JPR)) : 1;
  constexpr int JCHUNK = JPT < G6_JCHUNK ? JPT : G6_JCHUNK;  // records per jerk fold (split)
  static_assert(JL >= 1 && JL <= JLMAX && JL <= RPT && (RPT % JL) == 0, "JL");

  __shared__ __align__(128) Rec tiles[NSTAGE][RPT];
  __shared__ __align__(8) uint64_t full[NSTAGE];
  __shared__ __align__(8) uint64_t never;  // test hook: no arrival ever
  __shared__ int released[NSTAGE];
  __shared__ int issued_s;
  __shared__ volatile int abort_s;

  const int tid = threadIdx.x;
  const int jl = tid % JL;
  const int il = tid / JL;
  const int lane = tid & 31;
  pdl_wait();  // the predictor's records and the block list are complete

  // ---- j-range of this CTA ----
  // Where every tile is folded by itself (JL <= 4) the splits differ by one
  // tile at most; with more j-lanes a fold covers several tiles, counted from
  // the split's first, and the splits keep equal lengths.
  const int all = (kp.nj + TJ - 1) / TJ;
  int t0, t1;
  if (FOLD_TILES == 1) {
    t0 = (int)((long long)all * blockIdx.y / kp.nsplit);
    t1 = (int)((long long)all * (blockIdx.y + 1) / kp.nsplit);
  } else {
    t0 = min(all, (int)blockIdx.y * (kp.jsplit / TJ));
    t1 = min(all, t0 + kp.jsplit / TJ);
  }
  const int js = t0 * TJ;
  const int ntiles = t1 - t0;
  const Rec *gj = reinterpret_cast<const Rec *>(kp.jrec) + js / JPR;

  constexpr int NWARP = NT / 32;
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < NSTAGE; s++) {
      mbar_init(&full[s], 1);
      released[s] = 0;
    }
    mbar_init(&never, 1);
    issued_s = ntiles < NSTAGE ? ntiles : NSTAGE;
    abort_s = 0;
    fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    for (int s = 0; s < NSTAGE && s < ntiles; s++) {
      mbar_expect_tx(&full[s], RPT * sizeof(Rec));
      tma_load_1d(&tiles[s][0], gj + s * RPT, RPT * sizeof(Rec), &full[s]);
    }
  }

  // ---- i-particles of this thread ----
  typename P::I I[IPT];
  int self[IPT];
  bool valid[IPT];
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    const int i = blockIdx.x * ISLOTS + k * NIL + il;
    valid[k] = i < kp.ni;
    const int ii = valid[k] ? i : 0;
    if (kp.ilist) {
      const int slot = kp.ilist[ii];
      I[k] = P::load_i_slot(kp.jrec, slot);
      self[k] = valid[k] ? (kp.iself ? kp.iself[ii] : slot) : -1;
    } else {
      I[k] = P::load_i_explicit(kp.ipos + 3 * ii, kp.ivel + 3 * ii);
      self[k] = valid[k] && kp.iself ? kp.iself[ii] : -1;
    }
  }

  const auto eps2 = P::eps(kp.eps2);  // eps^2 + 2^-52 (ph4)
  typename P::Part q[IPT];
  // Compensated totals: in shared memory for the split nearest-neighbour
  // variant (touched once per fold; it frees registers for the pair loop),
  // in registers otherwise.  Layout [k][thread]: 17-word records,
  // conflict-free.
  constexpr bool TSH = P::template tot_shared<NN>();
  __shared__ typename P::Tot tot_sh[TSH ? IPT * NT : 1];
  typename P::Tot tot_reg[TSH ? 1 : IPT];
  auto T = [&](int k) -> typename P::Tot & {
    if constexpr (TSH)
      return tot_sh[k * NT + threadIdx.x];
    else
      return tot_reg[k];
  };
  R nnmin[IPT], nnbest[IPT], nnm2[IPT];
  int nnidx[IPT], besttile[IPT];
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    P::zero(q[k]);
    P::zero(T(k));
    nnmin[k] = nnbest[k] = nnm2[k] = (R)__int_as_float(0x7f800000);
    nnidx[k] = -1;
    besttile[k] = -1;
  }

  // Warps consume tiles independently: no CTA barrier in the loop.  Each
  // warp releases a stage after reading it; the warp whose release completes
  // a use of the stage (all NWARP warps done) refills it with tile t+NSTAGE.
  // The per-stage release counter only grows: use k of stage s ends when it
  // reaches (k+1)*NWARP.
  bool failed = false;
  for (int t = 0; t < ntiles; t++) {
    const int s = t % NSTAGE;
    const bool stall = kp.stall && t == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    const bool ok = stall ? mbar_wait_abortable(&never, 0, &abort_s, kp.wait_ns)
                          : mbar_wait_abortable(&full[s], (t / NSTAGE) & 1, &abort_s, kp.wait_ns);
    if (!__all_sync(0xffffffffu, ok)) {
      failed = true;
      if (lane == 0) abort_s = 1;
      break;
    }
    const Rec *tile = &tiles[s][0];
    const int tj0 = js + t * TJ;

    // Does this tile hold the self slot of any i of this warp?
    bool mine = false;
#pragma unroll
    for (int k = 0; k < IPT; k++) mine |= (unsigned)(self[k] - tj0) < (unsigned)TJ;
    const bool slow = __any_sync(0xffffffffu, mine);

    // JCHUNK records between jerk folds (split: the jerk partials are
    // folded more often than the rest; the last chunk folds with the tile).
    if (!slow) {
#pragma unroll 1
      for (int ub = 0; ub < JPT; ub += JCHUNK) {
        constexpr int UNR = NN ? G6_UNROLL_NN : HJ ? 2 * UNROLL : UNROLL;
#pragma unroll UNR
        for (int u = ub; u < ub + JCHUNK; u++) {
          const Rec r = tile[jl + JL * u];
#pragma unroll
          for (int k = 0; k < IPT; k++)
            P::template pair<false, NN, HJ>(I[k], r, eps2, q[k], nnmin[k], 0);
        }
        if (P::JFOLD && ub + JCHUNK < JPT) {
#pragma unroll
          for (int k = 0; k < IPT; k++) P::fold_jerk(T(k), q[k]);
        }
      }
    } else {
      for (int u = 0; u < JPT; u++) {
        const int jj = jl + JL * u;
        const Rec r = tile[jj];
#pragma unroll
        for (int k = 0; k < IPT; k++)
          P::template pair<true, NN, HJ>(I[k], r, eps2, q[k], nnmin[k],
                                         self[k] - (tj0 + JPR * jj));
        if (P::JFOLD && (u + 1) % JCHUNK == 0 && u + 1 < JPT) {
#pragma unroll
          for (int k = 0; k < IPT; k++) P::fold_jerk(T(k), q[k]);
        }
      }
    }

    // Nearest neighbour: nnmin holds this tile's smallest key.  Keep the
    // smallest over the tiles (nnbest) and the tile where it occurs (strict
    // <, so the earliest tile wins ties; the index within the tile is
    // recovered once, after the loop), and fold the larger of the tile's
    // and the running minimum into the second smallest key (nnm2).
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      if (!NN) break;
      const R tmin = nnmin[k];
      nnm2[k] = fmin(nnm2[k], fmax(tmin, nnbest[k]));
      const bool imp = tmin < nnbest[k];
      nnbest[k] = imp ? tmin : nnbest[k];
      besttile[k] = imp ? t : besttile[k];
      nnmin[k] = (R)__int_as_float(0x7f800000);
    }

    if ((t + 1) % FOLD_TILES == 0) {
#pragma unroll
      for (int k = 0; k < IPT; k++) {
        P::fold(T(k), q[k]);
        P::zero(q[k]);
      }
    }

    // Release stage s; the last releaser refills it.
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      const int c = atomicAdd(&released[s], 1);
      if (c == (t / NSTAGE + 1) * NWARP - 1 && t + NSTAGE < ntiles) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&full[s], RPT * sizeof(Rec));
        tma_load_1d(&tiles[s][0], gj + (t + NSTAGE) * RPT, RPT * sizeof(Rec), &full[s]);
        atomicMax(&issued_s, t + NSTAGE + 1);
      }
    }
  }

  pdl_trigger();  // j loop done: the next kernel of the chain may be scheduled
  if (__syncthreads_or(failed)) {
    // Drain the copies still in flight (bounded) before the CTA leaves.
    if (tid == 0) {
      atomicOr(kp.err, ERR_TMA_TIMEOUT);
      const int hi = issued_s;
      for (int u = hi - NSTAGE > 0 ? hi - NSTAGE : 0; u < hi; u++)
        (void)mbar_wait_bounded(&full[u % NSTAGE], (u / NSTAGE) & 1, kp.wait_ns);
      // Still count this CTA in its i-group, so that the group's ticket
      // returns to zero for the next launch (the results are void: the
      // error word is set).
      if (kp.nsplit > 1 && kp.xtick &&
          atomicAdd(&kp.xtick[blockIdx.x], 1u) == (unsigned)(kp.nsplit - 1))
        kp.xtick[blockIdx.x] = 0u;
    }
    return;
  }

  // ---- nearest neighbour: find the first j of the best tile (this lane's
  // j subset) whose r^2 equals the running min, with the same arithmetic,
  // reading the records back from global memory (L2). ----
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    if (!NN || besttile[k] < 0) continue;
    const Rec *g = gj + besttile[k] * RPT;
    const int tj0 = js + besttile[k] * TJ;
    for (int u = 0; u < JPT; u++) {
      const int jj = jl + JL * u;
      P::rescan(I[k], g[jj], eps2, nnbest[k], tj0 + JPR * jj, self[k], nnidx[k], nnm2[k]);
    }
  }

  // ---- merge: fold remainders, then j-lanes, then (maybe) CTAs ----
  typename P::Out o[IPT];
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    P::fold(T(k), q[k]);
    P::to_out(T(k), nnbest[k], nnm2[k], nnidx[k], o[k]);
  }
  if constexpr (JL >= TAB_JL) {
    // many lanes per i: through a shared-memory table (see lane_table)
    float *tab = reinterpret_cast<float *>(&tiles[0][0]);
    static_assert(lane_table_words<JL, ISLOTS>() * 4 <= sizeof(Rec) * RPT * NSTAGE, "table");
    __syncthreads();  // the tiles are read
#pragma unroll
    for (int k = 0; k < IPT; k++) lane_table_put<JL, ISLOTS>(tab, k * NIL + il, jl, o[k]);
    __syncthreads();
    lane_table_sum<JL, ISLOTS>(tab);
    __syncthreads();
    if (tid < ISLOTS) {
      const int i = blockIdx.x * ISLOTS + tid;
      const typename P::Out m = lane_table_get<JL, ISLOTS>(tab, tid);
      if (i < kp.ni) {
        if (kp.nsplit == 1)
          P::finish(m, i, kp);
        else
          reinterpret_cast<typename P::Out *>(kp.part)[(size_t)blockIdx.y * kp.ni_pad + i] = m;
      }
    }
  } else {
#pragma unroll
    for (int m = 1; m < JL; m <<= 1) {
#pragma unroll
      for (int k = 0; k < IPT; k++) {
        typename P::Out other = shfl_xor_out(o[k], m);
        // Lower lane first keeps the order fixed.
        if (lane & m) {
          P::merge(other, o[k]);
          o[k] = other;
        } else {
          P::merge(o[k], other);
        }
      }
    }
    if (jl == 0) {
#pragma unroll
      for (int k = 0; k < IPT; k++) {
        if (!valid[k]) continue;
        const int i = blockIdx.x * ISLOTS + k * NIL + il;
        if (kp.nsplit == 1)
          P::finish(o[k], i, kp);
        else
          reinterpret_cast<typename P::Out *>(kp.part)[(size_t)blockIdx.y * kp.ni_pad + i] = o[k];
      }
    }
  }
  if constexpr (ISLOTS > G6_XMERGE_MAX) return;
  if (kp.nsplit == 1 || !kp.xtick) return;

  // ---- split merge in the last CTA of the i-group (no second launch): NT /
  // ISLOTS threads per i, thread l taking splits l, l + ML, ... in order,
  // then the table sums them as it sums the lanes.  The ticket is reset for
  // the next launch. ----
  if constexpr (ISLOTS <= G6_XMERGE_MAX) {
    constexpr int ML = NT / ISLOTS;
    __shared__ int last_s;
    __threadfence();
    __syncthreads();
    if (tid == 0) last_s = atomicAdd(&kp.xtick[blockIdx.x], 1u) == (unsigned)(kp.nsplit - 1);
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    using Out = typename P::Out;
    float *tab = reinterpret_cast<float *>(&tiles[0][0]);
    const int q = tid / ML, l = tid % ML;
    const int i = blockIdx.x * ISLOTS + q;
    const Out *part = reinterpret_cast<const Out *>(kp.part) + (i < kp.ni ? i : 0);
    Out m;
    P::to_out_zero(m);
    if (l < kp.nsplit) {
      m = load_out_cg(part + (size_t)l * kp.ni_pad);
      for (int sp = l + ML; sp < kp.nsplit; sp += ML)
        P::merge(m, load_out_cg(part + (size_t)sp * kp.ni_pad));
    }
    lane_table_put<ML, ISLOTS>(tab, q, l, m);
    __syncthreads();
    lane_table_sum<ML, ISLOTS>(tab);
    __syncthreads();
    if (tid < ISLOTS && blockIdx.x * ISLOTS + tid < kp.ni)
      P::finish(lane_table_get<ML, ISLOTS>(tab, tid), blockIdx.x * ISLOTS + tid, kp);
    if (tid == 0) kp.xtick[blockIdx.x] = 0u;
  }
}

// Second pass: merge the nsplit partial records of each i.  A CTA takes IPB
// i; thread (l, i) merges splits l, l + 128/IPB, ... in order, the 128/IPB
// threads of an i merge in a fixed tree through shared memory, and the first
// IPB threads finish their i together (finish's FP64 instructions cost 16
// cycles of the SM each, whether one lane or 32 have an i: with a warp per i
// they were most of this pass).  Deterministic for a given (ni, nsplit).
// IPB = 8 while that gives every SM at most one CTA (splits in parallel), 32
// above (dense finish).  8.5 -> 7.9 us at 651 i x 11 splits, 18 -> 11 us at
// 4004 x 13, 16 -> 14 us at 722 x 37 with neighbours (a warp per i before).
template <class P, int IPB>
__global__ void __launch_bounds__(128) reduce_kernel(KParams kp) {
  constexpr int SL = 128 / IPB;
  using Out = typename P::Out;
  __shared__ Out sh[SL / 2][IPB];
  pdl_wait();
  pdl_trigger();
  const int il = threadIdx.x % IPB, l = threadIdx.x / IPB;
  const int i = blockIdx.x * IPB + il;
  const Out *part = reinterpret_cast<const Out *>(kp.part) + (i < kp.ni ? i : 0);
  Out o;
  P::to_out_zero(o);
  if (l < kp.nsplit) {
    o = part[(size_t)l * kp.ni_pad];
#pragma unroll 2
    for (int s = l + SL; s < kp.nsplit; s += SL) P::merge(o, part[(size_t)s * kp.ni_pad]);
  }
#pragma unroll
  for (int h = SL / 2; h > 0; h >>= 1) {
    if (l >= h && l < 2 * h) sh[l - h][il] = o;
    __syncthreads();
    if (l < h) P::merge(o, sh[l][il]);
    __syncthreads();
  }
  if (l == 0 && i < kp.ni) P::finish(o, i, kp);
}

// FP64 redo of the queued i-particles (see "nearest neighbour proof" and
// "condition-number refinement" above).  A persistent grid walks the
// (entry, j-chunk) units; each CTA reduces its unit in a fixed order and the
// CTA that completes an entry's last chunk (atomic ticket) merges the chunks
// in chunk order and overwrites that particle's results.  The chunk count
// depends only on the number of queued entries, so results are
// deterministic.  The last CTA to finish resets the queue.
//
// What bounds it: FP64 issues at 2 lanes per SM and cycle (16 cycles per warp
// instruction, however many lanes have work), so REF_MT entries, nearly all
// of them, use none inside a unit: the terms that need more than FP32 are
// evaluated in float-float (about 150 FP32 instructions, relative error
// ~1e-12, where FP64 took 30 at 16 cycles) and, because few lanes meet one at
// a time, listed per warp in shared memory and evaluated 32 at a time; lane
// sums merge in float-float.  REF_ACC entries exchange halves of their four
// FP64 quantities across lanes (6 additions for 20).

// FP64 term of j on the i at xi, added to sa and sp.
__device__ __forceinline__ void f64_term(const void *rec, int j, const double xi[3], double eps2,
                                         double sa[3], double &sp) {
  double dx[3];
#pragma unroll
  for (int k = 0; k < 3; k++)
    dx[k] = ((double)g6_split_get(rec, j, k) + (double)g6_split_get(rec, j, 4 + k)) - xi[k];
  const double m = (double)g6_split_get(rec, j, 3) + (double)g6_split_get(rec, j, 7);
  const double r2 = __fma_rn(dx[2], dx[2], __fma_rn(dx[1], dx[1], __fma_rn(dx[0], dx[0], eps2)));
  const double rinv = fp64::rsqrt64_normal(r2);
  const double mri = m * rinv;
  const double mr3i = mri * (rinv * rinv);
#pragma unroll
  for (int k = 0; k < 3; k++) sa[k] = __fma_rn(mr3i, dx[k], sa[k]);
  sp += mri;
}

// One j of a REF_MT entry: the force kernel's FP32 term (same operations,
// so the same value up to the final product's rounding) into compensated
// FP32 sums; true (and nothing added) above thr = TAU |a|, where the term is
// due in float-float.
__device__ __forceinline__ bool mt_term(float xh, float yh, float zh, float m, float ml, float xl,
                                        float yl, float zl, const float ih[3], const float il[3],
                                        float e32, float thr, bool skip, float ah[3], float al[3],
                                        float &ph, float &pl) {
  const float jh[3] = {xh, yh, zh}, jl[3] = {xl, yl, zl};
  float d[3];
#pragma unroll
  for (int k = 0; k < 3; k++) d[k] = __fadd_rn(__fsub_rn(jh[k], ih[k]), __fsub_rn(jl[k], il[k]));
  const float r2f = __fmaf_rn(d[2], d[2], __fmaf_rn(d[1], d[1], __fmaf_rn(d[0], d[0], e32)));
  const float rinv = rsqrt_approx(r2f);
  const float mri = __fmul_rn(m, rinv);
  if (skip) return false;
  if (__fmul_rn(mri, rinv) > thr) return true;
  // the FP32 term with the mass's high part, compensated; its low part
  // (2^-24 of the term) goes straight into the low words
  const float r3 = __fmul_rn(rinv, __fmul_rn(rinv, rinv));
  const float mr3i = __fmul_rn(mri, __fmul_rn(rinv, rinv));
  const float lr3 = __fmul_rn(ml, r3);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    ff_acc(ah[k], al[k], __fmul_rn(mr3i, d[k]));
    al[k] = __fmaf_rn(lr3, d[k], al[k]);
  }
  ff_acc(ph, pl, mri);
  pl = __fmaf_rn(ml, rinv, pl);
  return false;
}

__device__ __forceinline__ float2 ff_mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = __fmaf_rn(a.x, b.x, -p);
  e = __fmaf_rn(a.x, b.y, e);
  e = __fmaf_rn(a.y, b.x, e);
  const float h = __fadd_rn(p, e);
  return make_float2(h, __fsub_rn(e, __fsub_rn(h, p)));
}

// The term of j in float-float, added to the compensated sums.
__device__ __forceinline__ void ff_term(const void *rec, int j, const float ih[3],
                                        const float il[3], float2 eps2, float ah[3], float al[3],
                                        float &ph, float &pl) {
  float2 d[3], r2 = eps2;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    // (xh_j - xh_i) exactly as s + e (TwoSum), then the low words
    const float a = g6_split_get(rec, j, k), b = -ih[k];
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    const float t = __fadd_rn(e, __fsub_rn(g6_split_get(rec, j, 4 + k), il[k]));
    d[k].x = __fadd_rn(s, t);
    const float tt = __fsub_rn(d[k].x, s);
    d[k].y = __fadd_rn(__fsub_rn(s, __fsub_rn(d[k].x, tt)), __fsub_rn(t, tt));
    const float q = __fmul_rn(d[k].x, d[k].x);
    const float ql = __fmaf_rn(2.0f * d[k].x, d[k].y, __fmaf_rn(d[k].x, d[k].x, -q));
    ff_add(r2.x, r2.y, q, ql);
  }
  // 1/sqrt: y + y h (1/2 + 3/8 h), h = 1 - r2 y^2 from exact products (1 - u
  // is exact, u being near 1)
  const float y = rsqrt_approx(r2.x);
  const float t = __fmul_rn(y, y), te = __fmaf_rn(y, y, -t);
  const float u = __fmul_rn(t, r2.x), ue = __fmaf_rn(t, r2.x, -u);
  const float h = __fsub_rn(__fsub_rn(1.0f, u), __fmaf_rn(t, r2.y, __fmaf_rn(te, r2.x, ue)));
  float2 ri;
  const float c = __fmul_rn(y, __fmaf_rn(__fmul_rn(0.375f, h), h, __fmul_rn(0.5f, h)));
  ri.x = __fadd_rn(y, c);
  ri.y = __fsub_rn(c, __fsub_rn(ri.x, y));
  const float2 mr = ff_mul(make_float2(g6_split_get(rec, j, 3), g6_split_get(rec, j, 7)), ri);
  const float2 mr3 = ff_mul(mr, ff_mul(ri, ri));
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float2 f = ff_mul(mr3, d[k]);
    ff_acc(ah[k], al[k], f.x);
    al[k] = __fadd_rn(al[k], f.y);
  }
  ff_acc(ph, pl, mr.x);
  pl = __fadd_rn(pl, mr.y);
}

// Warp sums of four FP64 quantities: halves of them change lanes first, so
// every lane of group lane >> 3 ends with the sum of v[lane >> 3].
__device__ __forceinline__ double warp_sum4(const double v[4], int lane) {
  const bool hi = lane & 16, h2 = lane & 8;
  double a = hi ? v[2] : v[0], b = hi ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
  b += __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
  double c = h2 ? b : a;
  c += __shfl_xor_sync(0xffffffffu, h2 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}

// The nearer of two neighbour candidates, the smaller slot on equal r^2
// (slot < 0: none).  r^2 >= +0, so the bits order like the values.
__device__ __forceinline__ void ref_nn_take(double &r2, int &slot, double or2, int os) {
  const long long a = __double_as_longlong(r2), b = __double_as_longlong(or2);
  if (os >= 0 && (slot < 0 || b < a || (b == a && os < slot))) {
    r2 = or2;
    slot = os;
  }
}

// The entries queued for REF_MT alone.  A warp holds EL of them in its lanes
// (and 32 / EL j-lanes where they are few), so that a record loaded serves all
// of them and nothing is reduced across lanes for EL = 32; a CTA's eight warps
// share a chunk of the j, and the CTA that completes a group of entries adds
// the chunks' sums in order.  A unit of one entry per CTA, as below, spent
// most of its time on its own start and reduction: Salpeter cluster, N =
// 16384, 165 entries 62 us that way and 33 this, 92 entries 42 and 33, 24
// entries 18 and 16, 2 entries 14 and 12.
constexpr int MT_WARPS = RNT / 32;
__device__ __forceinline__ void refine_mt(const KParams &kp, RefBuf *b, int ne,
                                          float2 (*s_sum)[32][4], int *s_flag) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // log2 EL: as many entries per warp as still leave two CTAs for every SM when
  // a group's merge, RNT / (4 EL) threads per quantity, is kept to 16 chunks
  // per thread: about 1024 ne / 4^el CTAs (24 entries at EL = 32 and 512 chunks
  // took 41 us).
  int el = 0;
  while (el < 5 && (1 << el) < ne && (4 << (2 * el)) * 304LL <= 1024LL * ne) el++;
  const int EL = 1 << el, JL = 32 >> el;
  const int groups = (ne + EL - 1) >> el;
  const int npair = (kp.nj + 1) >> 1;
  const int TP = min(32, RNT >> (el + 2));  // threads per quantity in the merge
  int nch = min((int)gridDim.x / groups, 16 * TP);
  nch = min(nch, RPCAP / (groups << el));
  nch = min(nch, npair / (MT_WARPS * JL * 2));
  nch = max(nch, 1);
  const float e32 = split_eps(kp.eps2);
  const double eps2 = kp.eps2 + 1.0 / 4503599627370496.0;  // ph4's + 2^-52
  const float2 eps2f = make_float2((float)eps2, (float)(eps2 - (double)(float)eps2));
  const void *rec = kp.jrec;
  const float4 *q4 = reinterpret_cast<const float4 *>(rec);
  for (int u = blockIdx.x; u < groups * nch; u += gridDim.x) {
    const int g = u / nch, c = u - g * nch;
    const int e = (g << el) + (lane & (EL - 1));
    const bool valid = e < ne;
    const int i = b->mt_list[valid ? e : 0];
    const float thr = b->mt_thr[valid ? e : 0];
    int self;
    float ih[3], il[3];
    if (kp.ilist) {
      const int slot = kp.ilist[i];
      self = kp.iself ? kp.iself[i] : slot;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        ih[k] = g6_split_get(rec, slot, k);
        il[k] = g6_split_get(rec, slot, 4 + k);
      }
    } else {
      self = kp.iself ? kp.iself[i] : -1;
#pragma unroll
      for (int k = 0; k < 3; k++) SplitP::split(kp.ipos[3 * i + k], ih[k], il[k]);
    }
    const int p0 = (int)((long long)npair * c / nch);
    const int p1 = (int)((long long)npair * (c + 1) / nch);
    float ah[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f}, ph = 0.f, pl = 0.f;
#pragma unroll 2
    for (int rp = p0 + warp * JL + (lane >> el); rp < p1; rp += MT_WARPS * JL) {
      const float4 A = __ldg(q4 + 6 * rp), B = __ldg(q4 + 6 * rp + 1);
      const float4 C = __ldg(q4 + 6 * rp + 2), D = __ldg(q4 + 6 * rp + 3);
      const int j = 2 * rp;
      if (mt_term(A.x, A.z, B.x, B.z, D.z, C.x, C.z, D.x, ih, il, e32, thr,
                  j == self || j >= kp.nj, ah, al, ph, pl))
        ff_term(rec, j, ih, il, eps2f, ah, al, ph, pl);
      if (mt_term(A.y, A.w, B.y, B.w, D.w, C.y, C.w, D.y, ih, il, e32, thr,
                  j + 1 == self || j + 1 >= kp.nj, ah, al, ph, pl))
        ff_term(rec, j + 1, ih, il, eps2f, ah, al, ph, pl);
    }
    for (int off = 16; off >= EL; off >>= 1) {
#pragma unroll
      for (int k = 0; k < 3; k++)
        ff_add(ah[k], al[k], __shfl_xor_sync(0xffffffffu, ah[k], off),
               __shfl_xor_sync(0xffffffffu, al[k], off));
      ff_add(ph, pl, __shfl_xor_sync(0xffffffffu, ph, off), __shfl_xor_sync(0xffffffffu, pl, off));
    }
    if (lane < EL) {
#pragma unroll
      for (int k = 0; k < 3; k++) s_sum[warp][lane][k] = make_float2(ah[k], al[k]);
      s_sum[warp][lane][3] = make_float2(ph, pl);
    }
    __syncthreads();
    // four quantities of EL entries: the warps in order
    float2 *part = &b->mt_part[0][0] + (((size_t)g * nch) << el) * 4;
    if (tid < 4 * EL) {
      float2 q = s_sum[0][tid >> 2][tid & 3];
      for (int w = 1; w < MT_WARPS; w++) {
        const float2 o = s_sum[w][tid >> 2][tid & 3];
        ff_add(q.x, q.y, o.x, o.y);
      }
      part[((size_t)c << el) * 4 + tid] = q;
      __threadfence();
    }
    __syncthreads();
    if (tid == 0) *s_flag = atomicAdd(&b->mt_ticket[g], 1u) == (unsigned)(nch - 1);
    __syncthreads();
    if (*s_flag) {
      // the group's last CTA: TP threads per quantity (a power of two, in one
      // warp), each adding chunks t, t + TP, ... in order, then a fixed tree
      __threadfence();
      const int t = tid & (TP - 1), x = tid / TP;
      float2 q = make_float2(0.f, 0.f);
      if (x < 4 * EL) {
#pragma unroll 4
        for (int cc = t; cc < nch; cc += TP) {
          const float2 o = __ldcg(part + ((size_t)cc << el) * 4 + x);
          ff_add(q.x, q.y, o.x, o.y);
        }
      }
      for (int off = TP >> 1; off > 0; off >>= 1) {
        const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, q.x, off),
                                     __shfl_xor_sync(0xffffffffu, q.y, off));
        // (the lower lane first, so that both ends hold the same sum)
        float2 lo = (tid & off) ? o : q, hi = (tid & off) ? q : o;
        ff_add(lo.x, lo.y, hi.x, hi.y);
        q = lo;
      }
      const int ee = (g << el) + (x >> 2);
      if (t == 0 && x < 4 * EL && ee < ne) {
        const int ii = b->mt_list[ee];
        const double v = (double)q.x + (double)q.y;
        if ((x & 3) < 3)
          kp.acc[3 * ii + (x & 3)] = v;
        else
          kp.pot[ii] = -v;
      }
      if (tid == 0) b->mt_ticket[g] = 0u;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(RNT) refine_kernel(KParams kp) {
  pdl_wait();
  pdl_trigger();
  RefBuf *b = reinterpret_cast<RefBuf *>(kp.refine);
  __shared__ unsigned s_cnt, s_cmt;
  __shared__ float2 s_mt[MT_WARPS][32][4];
  __shared__ double s_sum[RNT / 32][4], s_r2[RNT / 32];
  __shared__ int s_slot[RNT / 32];
  __shared__ int s_last;
  __shared__ int s_due[RNT / 32][96];  // per warp: j whose REF_MT term is due in float-float
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_cnt = *reinterpret_cast<volatile unsigned *>(&b->h.count);
    s_cmt = *reinterpret_cast<volatile unsigned *>(&b->h.cmt);
  }
  __syncthreads();
  const unsigned cnt = s_cnt, cmt = s_cmt;
  if (cnt == 0 && cmt == 0) {  // nothing queued (most calls): record that and leave
    if (blockIdx.x == 0 && tid == 0) b->h.last = b->h.last_acc = b->h.last_mt = 0u;
    return;
  }
  const int ne = cnt > (unsigned)RCAP ? 0 : (int)cnt;
  if (max(cnt, cmt) > (unsigned)RCAP && blockIdx.x == 0 && tid == 0)
    atomicMax(&b->h.overflow, max(cnt, cmt));
  if (cmt > 0 && cmt <= (unsigned)RCAP) refine_mt(kp, b, (int)cmt, s_mt, &s_last);
  int nch = 1;
  if (ne > 0) {
    // One unit per CTA while the entries are few (the CTA reduces once), two
    // once they are many, for balance.  Salpeter cluster, N = 16384, 4 CTAs
    // per SM, at one, two and four: 67 entries for kappa (and 155 in refine_mt)
    // 109, 108 and 108 us, 12 of them 34 at each; at 2 CTAs per SM an earlier
    // build took a quarter more.
    const int upc = ne * 4 > (int)gridDim.x ? G6_REF_UNITS : 1;
    nch = (upc * (int)gridDim.x + ne - 1) / ne;
    nch = min(nch, RCHMAX);
    nch = min(nch, RPCAP / ne);
    nch = min(nch, max(1, kp.nj / 1024));
    nch = max(nch, 1);
  }
  const int units = ne * nch;
  const double eps2 = kp.eps2 + 1.0 / 4503599627370496.0;  // ph4's + 2^-52
  const float e32 = split_eps(kp.eps2);
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const void *rec = kp.jrec;
  // (from the last CTA down: the first ones hold the units of refine_mt)
  for (int u = gridDim.x - 1 - blockIdx.x; u < units; u += gridDim.x) {
    const int e = u / nch, c = u - e * nch;
    const int i = b->list[e];
    const int mode = b->mode[e];
    const float thr = b->thr[e], thr_mt = b->thr_mt[e];
    // chunk c: record pairs [p0, p1) (j from 2 p0 to 2 p1, nj at most)
    const int npair = (kp.nj + 1) >> 1;
    const int p0 = (int)((long long)npair * c / nch);
    const int p1 = (int)((long long)npair * (c + 1) / nch);
    const int j0 = 2 * p0;
    const int j1 = 2 * p1 < kp.nj ? 2 * p1 : kp.nj;
    // The i-particle in the split kernel's own representation (double-single
    // position), so that an i and a j copy of it at the same place give
    // dx = 0 exactly, as there.
    int self;
    double xi[3], xi64[3];
    float ih[3], il[3];
    if (kp.ilist) {
      const int slot = kp.ilist[i];
      self = kp.iself ? kp.iself[i] : slot;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        ih[k] = g6_split_get(rec, slot, k);
        il[k] = g6_split_get(rec, slot, 4 + k);
      }
    } else {
      self = kp.iself ? kp.iself[i] : -1;
#pragma unroll
      for (int k = 0; k < 3; k++) SplitP::split(kp.ipos[3 * i + k], ih[k], il[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) xi[k] = (double)ih[k] + (double)il[k];
    if (mode & REF_NN) ipos64(kp, i, xi64);
    double br2 = inf;
    int bslot = -1;
    double sum4 = 0.0;  // this lane group's quantity (warp_sum4's order)
    if (mode & REF_MT) {
      // whole record pairs in four 16-byte loads, two pairs in flight per
      // thread; all lanes of a warp take the same number of steps
      float ah[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f}, ph = 0.f, pl = 0.f;
      const float4 *q4 = reinterpret_cast<const float4 *>(rec);
      int *due = s_due[warp];
      int nd = 0;  // listed and not yet evaluated (the same in every lane)
      const float2 eps2f = make_float2((float)eps2, (float)(eps2 - (double)(float)eps2));
      const unsigned below = (1u << lane) - 1u;
      const int steps = (p1 - p0 - 32 * warp + RNT - 1) / RNT;
#pragma unroll 2
      for (int st = 0; st < steps; st++) {
        const int rp = p0 + 32 * warp + lane + st * RNT;
        const int rq = rp < p1 ? rp : p1 - 1;
        const float4 A = __ldg(q4 + 6 * rq), B = __ldg(q4 + 6 * rq + 1);
        const float4 C = __ldg(q4 + 6 * rq + 2), D = __ldg(q4 + 6 * rq + 3);
        const int j = 2 * rp;
        const bool d0 = mt_term(A.x, A.z, B.x, B.z, D.z, C.x, C.z, D.x, ih, il, e32, thr_mt,
                                rp >= p1 || j == self || j >= kp.nj, ah, al, ph, pl);
        const bool d1 = mt_term(A.y, A.w, B.y, B.w, D.w, C.y, C.w, D.y, ih, il, e32, thr_mt,
                                rp >= p1 || j + 1 == self || j + 1 >= kp.nj, ah, al, ph, pl);
        const unsigned m0 = __ballot_sync(0xffffffffu, d0), m1 = __ballot_sync(0xffffffffu, d1);
        if (m0 | m1) {
          if (d0) due[nd + __popc(m0 & below)] = j;
          nd += __popc(m0);
          if (d1) due[nd + __popc(m1 & below)] = j + 1;
          nd += __popc(m1);
          __syncwarp();
          while (nd >= 32) {
            nd -= 32;
            ff_term(rec, due[nd + lane], ih, il, eps2f, ah, al, ph, pl);
          }
          __syncwarp();
        }
      }
      if (nd > 0) {
        if (lane < nd) ff_term(rec, due[lane], ih, il, eps2f, ah, al, ph, pl);
        __syncwarp();
      }
      // FP32 sums: float-float over the warp
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; k++)
          ff_add(ah[k], al[k], __shfl_xor_sync(0xffffffffu, ah[k], off),
                 __shfl_xor_sync(0xffffffffu, al[k], off));
        ff_add(ph, pl, __shfl_xor_sync(0xffffffffu, ph, off),
               __shfl_xor_sync(0xffffffffu, pl, off));
      }
      const int c = lane >> 3;
      const float fh = c == 0 ? ah[0] : c == 1 ? ah[1] : c == 2 ? ah[2] : ph;
      const float fl = c == 0 ? al[0] : c == 1 ? al[1] : c == 2 ? al[2] : pl;
      sum4 = (double)fh + (double)fl;
    }
    if (mode & REF_ACC) {  // acceleration and potential; the jerk stays
      double sa[3] = {0.0, 0.0, 0.0}, sp = 0.0;
      for (int j = j0 + tid; j < j1; j += RNT)
        if (j != self) f64_term(rec, j, xi, eps2, sa, sp);
      const double v[4] = {sa[0], sa[1], sa[2], sp};
      sum4 = warp_sum4(v, lane);
    }
    if (mode & REF_NN) {
      for (int j = j0 + tid; j < j1; j += RNT) {
        if (j == self) continue;
        float d[3];
#pragma unroll
        for (int k = 0; k < 3; k++)
          d[k] = __fadd_rn(__fsub_rn(g6_split_get(rec, j, k), ih[k]),
                           __fsub_rn(g6_split_get(rec, j, 4 + k), il[k]));
        const float key = __fmaf_rn(d[2], d[2], __fmaf_rn(d[1], d[1], __fmaf_rn(d[0], d[0], e32)));
        if (key <= thr) {
          double xj[3];
          jpos64(kp.js, kp.ti, j, xj);
          ref_nn_take(br2, bslot, ph4_r2(xi64, xj), j);
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double or2 = __shfl_down_sync(0xffffffffu, br2, off);
        const int os = __shfl_down_sync(0xffffffffu, bslot, off);
        ref_nn_take(br2, bslot, or2, os);
      }
    }
    if ((lane & 7) == 0) s_sum[warp][lane >> 3] = sum4;
    if (lane == 0) {
      s_r2[warp] = br2;
      s_slot[warp] = bslot;
    }
    __syncthreads();
    // the warps in order: one lane per quantity
    RefPart *out = &b->part[e * nch + c];
    if (tid < 4) {
      double q = s_sum[0][tid];
      for (int w = 1; w < RNT / 32; w++) q += s_sum[w][tid];
      if (tid < 3)
        out->a[tid] = q;
      else
        out->p = q;
    } else if (tid == 4) {
      double r2 = inf;
      int sl = -1;
      for (int w = 0; w < RNT / 32; w++) ref_nn_take(r2, sl, s_r2[w], s_slot[w]);
      out->r2 = r2;
      out->slot = sl;
      out->pad = 0;
    }
    if (warp == 0) {
      __threadfence();
      __syncwarp();
      if (lane == 0) s_last = atomicAdd(&b->ticket[e], 1u) == (unsigned)(nch - 1);
    }
    __syncthreads();
    // The CTA that completed the entry merges its chunks: warp 0, lane l
    // taking chunks l and l + 32, then a fixed shuffle tree (the result does
    // not depend on which CTA finished last).
    if (s_last && warp == 0) {
      __threadfence();
      const volatile RefPart *vp = b->part + (size_t)e * nch;
      double f[4] = {0.0, 0.0, 0.0, 0.0}, fr2 = inf;
      int fs = -1;
      for (int cc = lane; cc < nch; cc += 32) {
        for (int k = 0; k < 3; k++) f[k] += vp[cc].a[k];
        f[3] += vp[cc].p;
        if (mode & REF_NN) ref_nn_take(fr2, fs, vp[cc].r2, vp[cc].slot);
      }
      const double q = warp_sum4(f, lane);
      if ((mode & (REF_ACC | REF_MT)) && (lane & 7) == 0) {
        if (lane < 24)
          kp.acc[3 * i + (lane >> 3)] = q;
        else
          kp.pot[i] = -q;
      }
      if (mode & REF_NN) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const double or2 = __shfl_down_sync(0xffffffffu, fr2, off);
          const int os = __shfl_down_sync(0xffffffffu, fs, off);
          ref_nn_take(fr2, fs, or2, os);
        }
      }
      if (lane == 0) {
        if ((mode & REF_NN) && fs >= 0) {
          if (kp.nn) kp.nn[i] = fs;
          if (kp.nn_r2) kp.nn_r2[i] = (float)fr2;
        }
        b->ticket[e] = 0u;
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned d = atomicAdd(&b->h.done, 1u);
    if (d == gridDim.x - 1) {
      b->h.last = cnt + cmt;
      b->h.last_acc = b->h.nacc;
      b->h.last_mt = b->h.nmt + cmt;
      b->h.count = 0u;
      b->h.cmt = 0u;
      b->h.nacc = 0u;
      b->h.nmt = 0u;
      b->h.done = 0u;
      __threadfence();
    }
  }
}

// The wait-expiry hook in FP64, whose kernel has no wait of its own: the same
// bounded wait on a barrier that nothing arrives on, then the error word.
__global__ void expiry_kernel(int *err, unsigned long long wait_ns) {
  __shared__ __align__(8) uint64_t never;
  mbar_init(&never, 1);
  fence_barrier_init();
  if (!mbar_wait_bounded(&never, 0, wait_ns)) atomicOr(err, ERR_TMA_TIMEOUT);
}

int g_sms = 0;

int sm_count() {
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 152;
  }
  return g_sms;
}

// Launch shape from a small cost model.  A CTA streams tiles_per tiles of
// its j-range; per tile each thread spends ~A issue slots of fixed work
// (wait, release, bookkeeping) plus B per j-record for its IPT i-particles
// (JPT = 256/JL records), plus F per CTA (i-loads, lane merges, output).
// Resident CTAs run in waves of MINB per SM, so
//   cost = waves * (tiles_per * (A + B * JPT) + F) * (1 + 0.002 * nsplit)
// (the last factor charges the partial-sum traffic of the second pass).
// Candidates: JL from the smallest that does not waste CTA i-slots up to
// 256 (more j-lanes = more CTAs for small blocks), and every distinct split
// count up to 4 resident waves' worth.  Large blocks (a full wave of CTAs at
// JL = 1) stay at JL = 1; balanced_splits below has the last word on the
// splits for JL <= 4.  The last few shapes are cached (block steps repeat the
// same ni).
struct ShapeKey {
  int ni, nj, nn, fjl, fns;
  int jl, nsplit, jsplit;
};
ShapeKey g_shape_cache[256];

// The number of splits where their lengths may differ by a tile (JL <= 4): what
// counts is the tiles of the busiest SM.  In units of one tile's time there: up
// to three CTAs per SM run at once, fewer leave a fifth of the FP32 cycles
// unused; beyond three slots refill as CTAs end, and the longer splits cost half
// of their tile.  OV is a CTA's start and end, with the nearest neighbour the
// re-scan of its best tile too (the dearer the farther apart the tiles lie, up to
// 65536 j): counted once, and in part for each CTA that waits for a slot.  Another
// count than ns0 (choose_shape's, equal lengths) is taken where it should gain half
// a per cent.  Fitted to 3800 forced counts of 211 sizes: 0.6 % behind the best
// count on average, ns0 2.1 %.  At 190 other sizes where the count is not ns0 it
// gains 3.0 %; seven of them lose 2 to 7 %.  8192 x 8192 121 -> 103 us (11 -> 32
// splits), 11719 x 2^20 13.20 -> 13.10 ms, 11850 x 11850 with neighbours 312 -> 256
// us (8 -> 16); 1000 x 2^18 with neighbours stays at 57 (390 us; 408 at 76).
int balanced_splits(int ni, int ntiles, int jl, int nn, int ns0, int force_nsplit) {
  if (force_nsplit > 0) return force_nsplit < ntiles ? force_nsplit : ntiles;
  const int sms = sm_count(), islots = (NT / jl) * IPT_SPLIT;
  const long long gx = (ni + islots - 1) / islots;
  const double rescan = nn ? (1.5 + 7.0 / jl) * (ntiles < 256 ? ntiles / 256.0 : 1.0) : 0.0;
  const double OV = 0.8 * jl + rescan, WAIT = nn ? 0.28 : 0.1;
  auto cost = [&](int ns) {
    const long long c = (gx * ns + sms - 1) / sms;  // CTAs of the busiest SM
    const double mean = (double)ntiles / ns, most = (ntiles + ns - 1) / ns;
    if (c <= 3) return (double)c * most / (c < 3 ? 0.8 : 1.0) + OV;
    return (double)c * (mean + 0.45 * (most - mean)) + OV * (1.0 + WAIT * (double)(c - 3));
  };
  // The partial records stay within the fixed scratch array where those of
  // the count before do (one split needs none); else within what the L2 holds,
  // or the count before took: without a limit 273408 i against 2^20 j took 831
  // MB instead of 175 for a gain of 1 %.
  const size_t room = (size_t)16 << 20, l2 = (size_t)128 << 20;
  const size_t rec = (size_t)ni * sizeof(SplitP::Out), was = ns0 > 1 ? (size_t)ns0 * rec : 0;
  const size_t limit = was <= room ? room : was > l2 ? was : l2;
  int best = ns0;
  double bc = cost(ns0) * 0.995;
  const int most = ntiles < 128 ? ntiles : 128;
  for (int ns = 1; ns <= most; ns++) {
    if (ns > ns0 && (size_t)ns * rec > limit) break;
    const double c = cost(ns);
    if (c < bc) {
      bc = c;
      best = ns;
    }
  }
  return best;
}

void choose_shape(int ni, int nj, int nn, int force_jl, int force_nsplit, int *jl_out,
                  int *nsplit_out, int *jsplit_out) {
  nn = nn ? 1 : 0;
  const unsigned h =
      ((unsigned)ni * 2654435761u ^ (unsigned)nj * 40503u ^ (unsigned)nn * 97u) &
      255u;
  ShapeKey &c = g_shape_cache[h];
  if (c.ni == ni && c.nj == nj && c.nn == nn && c.fjl == force_jl &&
      c.fns == force_nsplit && c.jl > 0) {
    *jl_out = c.jl;
    *nsplit_out = c.nsplit;
    *jsplit_out = c.jsplit;
    return;
  }
  const int ntiles = nj > 0 ? (nj + TJ - 1) / TJ : 1;
  const int slots = SplitP::MINB * sm_count();
  const double A = 150.0, F = 3000.0;
  const int IPT = IPT_SPLIT;
  const double B = 20.0 * IPT;  // per j and i: ~20 issue slots (packed j pairs)
  int jl0 = 1;
  while (jl0 < JLMAX && (NT / (jl0 * 2)) * IPT >= ni && ni > 0) jl0 *= 2;
  int jl_lo = jl0, jl_hi = JLMAX;
  if (force_jl > 0) jl_lo = jl_hi = force_jl;
  else if (jl0 == 1 && (ni + (NT * IPT) - 1) / (NT * IPT) >= slots) jl_hi = 1;
  const int max_ns = ntiles < 4 * slots ? ntiles : 4 * slots;
  // Split counts: all small ones, then those from small tiles_per; each is
  // normalised to (tiles per split, splits), and repeats are dropped (a
  // repeat has the same cost and cannot win the strict comparison below).
  int cand_tp[512], cand_ns[512];
  int nc = 0;
  {
    int raw[512];
    int nr = 0;
    if (force_nsplit > 0) {
      raw[nr++] = force_nsplit;
    } else {
      for (int q = 1; q <= 128 && q <= max_ns; q++) raw[nr++] = q;
      for (int tp = 1; tp <= 256 && nr < 512; tp++) {
        const int q = (ntiles + tp - 1) / tp;
        if (q > 128 && q <= max_ns) raw[nr++] = q;
      }
    }
    for (int k = 0; k < nr; k++) {
      int ns = raw[k] < 1 ? 1 : raw[k];
      if (ns > ntiles) ns = ntiles;
      const int tp = (ntiles + ns - 1) / ns;
      if (nc > 0 && cand_tp[nc - 1] == tp) continue;
      cand_tp[nc] = tp;
      cand_ns[nc] = (ntiles + tp - 1) / tp;
      nc++;
    }
  }
  double best = 1e300;
  int bjl = jl_lo, bns = 1;
  for (int jl = jl_lo; jl <= jl_hi; jl *= 2) {
    const int islots = (NT / jl) * IPT;
    const long long gx = (ni + islots - 1) / islots;
    for (int k = 0; k < nc; k++) {
      const int tp = cand_tp[k], ns = cand_ns[k];
      const long long ctas = gx * ns;
      const long long waves = (ctas + slots - 1) / slots;
      // Where the i-groups alone do not fill the GPU, CTAs are kept to at
      // most 128 tiles (256 with the nearest neighbour, whose CTAs each
      // re-scan a best tile at the end): many short CTAs balance over the
      // SMs as slots free up, better than a few long ones in one wave
      // (measured, 16384 i against 2^20 j: 0.674 of peak at 7 splits of 586
      // tiles, 0.700 at 38 or 57 splits; the wave count does not capture
      // it; with nn at 65536 i: 0.690 at 16 splits, 0.685 at 32).
      if (gx < slots && tp > (nn ? 256 : 128) && k + 1 < nc) continue;
      // j-lanes (JL > 1) cost a few per cent per pair in large blocks
      // (measured at 65536 i: JL = 2 ran 3 % slower than JL = 1 without the
      // nearest neighbour and 6 % slower with it), where JL = 1 fills the
      // GPU by splitting j alone
      const double jl_pen = (jl > 1 && ni >= 16384) ? 1.05 : 1.0;
      // each split adds per-CTA start-up, a partial record per i to write
      // and merge, and (nearest neighbour) a re-scan of its best tile: 0.2 %
      // per split against j sets of up to 2048 tiles (measured: 65536 i
      // against 2^18 j ran 2 % slower at 16 splits than at 7), proportionally
      // less against larger ones (2^20 j: 16 splits beat 7 by 1.5 %)
      const double split_pen = 0.002 * ns * (ntiles > 2048 ? 2048.0 / ntiles : 1.0);
      const double cost = (double)waves * (tp * (A + B * (double)(TJ / jl)) + F) *
                          (1.0 + split_pen) * jl_pen;
      if (cost < best * 0.999) {
        best = cost;
        bjl = jl;
        bns = ns;
      }
    }
  }
  const int tp = (ntiles + bns - 1) / bns;
  *jl_out = bjl;
  *nsplit_out = (ntiles + tp - 1) / tp;
  *jsplit_out = tp * TJ;
  if (bjl <= 4) *nsplit_out = balanced_splits(ni, ntiles, bjl, nn, *nsplit_out, force_nsplit);
  c.ni = ni;
  c.nj = nj;
  c.nn = nn;
  c.fjl = force_jl;
  c.fns = force_nsplit;
  c.jl = *jl_out;
  c.nsplit = *nsplit_out;
  c.jsplit = *jsplit_out;
}

template <class P>
int launch(const KParams &kp, int jl, int gx, cudaStream_t st, cudaEvent_t ev_mid) {
  dim3 grid(gx, kp.nsplit), block(NT);
  // Without nearest neighbours only the large-block shape has its own
  // instantiation; small blocks are latency-bound and keep the nn code.
  if (kp.hjerk) {
    if (jl != 1 || kp.want_nn) return -2;
    launch_pdl(force_kernel<P, 1, false, true>, grid, block, 0, st, kp);
  } else switch (jl) {
#define G6_CASE(J)                                            \
  case J:                                                     \
    if (kp.want_nn)                                           \
      launch_pdl(force_kernel<P, J, true>, grid, block, 0, st, kp);  \
    else                                                      \
      launch_pdl(force_kernel<P, J, false>, grid, block, 0, st, kp); \
    break;
    G6_CASE(1)
    G6_CASE(2)
    G6_CASE(4)
    G6_CASE(8)
    G6_CASE(16)
    G6_CASE(32)
    G6_CASE(64)
    G6_CASE(128)
#if G6_NT >= 256
    G6_CASE(256)
#endif
#undef G6_CASE
    default:
      return -2;
  }
  if (kp.nsplit > 1 && !kp.xtick) {
    if (kp.ni <= 8 * sm_count())
      launch_pdl(reduce_kernel<P, 8>, dim3((kp.ni + 7) / 8), dim3(128), 0, st, kp);
    else
      launch_pdl(reduce_kernel<P, 32>, dim3((kp.ni + 31) / 32), dim3(128), 0, st, kp);
  }
  if (ev_mid) cudaEventRecord(ev_mid, st);
  // refine_kernel: units of (entry, j-chunk), at most RCHMAX chunks per
  // entry and ni entries, so small blocks get a small grid
  if (kp.refine) {
    const long long cap = (long long)kp.ni * RCHMAX;
    const int grid = cap < (long long)G6_REF_CTAS * sm_count() ? (int)cap : G6_REF_CTAS * sm_count();
    launch_pdl(refine_kernel, dim3(grid), dim3(RNT), 0, st, kp);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

extern "C" int g6k_sm_count(void) { return sm_count(); }

extern "C" size_t g6k_refine_bytes(void) { return sizeof(RefBuf); }

extern "C" int g6k_refine_read(const void *refine, int out[4], cudaStream_t st) {
  RefHdr h;
  if (cudaMemcpyAsync(&h, refine, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return -3;
  out[0] = (int)h.last;
  out[1] = (int)h.last_acc;
  out[2] = (int)h.overflow;
  out[3] = (int)h.last_mt;
  if (h.overflow) {
    const unsigned zero = 0;
    cudaMemcpyAsync(reinterpret_cast<char *>(const_cast<void *>(refine)) +
                        offsetof(RefHdr, overflow),
                    &zero, sizeof(zero), cudaMemcpyHostToDevice, st);
    cudaStreamSynchronize(st);
  }
  return 0;
}

extern "C" size_t g6k_scratch_bytes(int ni, int nj, int prec, int nn, int force_jl,
                                    int force_nsplit) {
  if (prec == G6_PREC_FP64) return g6k_force64_scratch(ni, nj, nn, force_jl, force_nsplit, XTMAX);
  int jl, nsplit, jsplit;
  choose_shape(ni, nj, nn, force_jl, force_nsplit, &jl, &nsplit, &jsplit);
  if (nsplit <= 1) return 0;
  return (size_t)nsplit * (size_t)ni * sizeof(SplitP::Out);
}

extern "C" int g6k_force(const g6_force_args *a, g6_shape *shape, cudaStream_t st) {
  if (a->ni <= 0) return 0;
  if (a->nj <= 0 || !a->acc || !a->jerk || !a->pot || !a->js || !a->err) return -1;
  if (!a->ilist && (!a->ipos || !a->ivel)) return -1;
  if (a->hjerk && (a->want_nn || (a->force_jl != 0 && a->force_jl != 1))) return -2;
  if (a->force_jl < 0 || a->force_jl > JLMAX || (a->force_jl & (a->force_jl - 1))) return -2;
  if (a->prec == G6_PREC_FP64 && a->stall_test)
    expiry_kernel<<<1, 1, 0, st>>>(a->err, STALL_TEST_NS);
  if (a->prec == G6_PREC_FP64)
    return g6k_force64(a, a->refine ? reinterpret_cast<RefBuf *>(a->refine)->xtick : nullptr,
                       a->refine ? XTMAX : 0, shape, st);
  int jl, nsplit, jsplit;
  choose_shape(a->ni, a->nj, a->want_nn, a->hjerk ? 1 : a->force_jl, a->force_nsplit, &jl,
               &nsplit, &jsplit);
  if (jl < 1 || jl > JLMAX || (jl & (jl - 1))) return -2;
  KParams kp;
  kp.ni = a->ni;
  kp.nj = a->nj;
  kp.nsplit = nsplit;
  kp.jsplit = jsplit;
  kp.eps2 = a->eps2;
  kp.ipos = a->ipos;
  kp.ivel = a->ivel;
  kp.ilist = a->ilist;
  kp.iself = a->iself;
  kp.acc = a->acc;
  kp.jerk = a->jerk;
  kp.pot = a->pot;
  kp.nn = a->nn;
  kp.nn_r2 = a->nn_r2;
  kp.part = a->scratch;
  kp.ni_pad = a->ni;
  kp.err = a->err;
  kp.want_nn = a->want_nn;
  kp.hjerk = a->hjerk;
  kp.js = *a->js;
  kp.ti = a->ti;
  // The refinement pass serves the split kernel's g6 results; the hermite
  // jerk form and callers passing kappa < 0 (the fixed-step path) keep plain
  // split arithmetic.
  kp.refine = !a->hjerk && a->kappa >= 0.0 ? a->refine : nullptr;
  kp.kappa2 = a->kappa > 0.0 ? a->kappa * a->kappa : 0.0;
  kp.stall = a->stall_test;
  kp.wait_ns = a->stall_test ? STALL_TEST_NS : WAIT_NS;
  const size_t need =
      nsplit > 1 ? g6k_scratch_bytes(a->ni, a->nj, a->prec, a->want_nn, jl, nsplit) : 0;
  if (need > a->scratch_bytes) return -4;
  const int islots = (NT / jl) * IPT_SPLIT;
  const int gx = (a->ni + islots - 1) / islots;
  if (shape) {
    shape->jl = jl;
    shape->nsplit = nsplit;
    shape->grid_x = gx;
    shape->grid_y = nsplit;
    shape->threads = NT;
  }
  // The in-kernel split merge runs in the one CTA that completes an i-group of
  // one or two i (JL = 128).  It saves a launch, but that CTA works alone at the
  // end, and the refinement pass, released meanwhile, crowds on the SMs that are
  // through.  It pays for many splits: 1 i, 205 splits 15.6 us against 17.9 with the
  // second launch, 86 splits 12.1 and 12.6, 8 i, 114 splits 20.0 and 20.8; but 8 i, 86
  // splits 17.2 and 15.6, 1 to 16 i, 2 to 16 splits 10.5 and 9.6, and 16 i, 32 splits
  // with one entry to refine 63.8 and 31.3.  (More i per group, JL = 64 and 32: 44.9 and 33.1, 25.0 and 22.6.)
  kp.xtick = (a->refine && nsplit >= (gx == 1 ? 64 : 96) && gx <= XTMAX && islots <= G6_XMERGE_MAX)
                 ? reinterpret_cast<RefBuf *>(a->refine)->xtick
                 : nullptr;
  kp.jrec = a->js->jp_split;
  return launch<SplitP>(kp, jl, gx, st, a->ev_mid);
}

// ---------------------------------------------------------------------------
// Fixed scratch for callers that cannot allocate device memory.
//
// The split-j partial sums normally live in a buffer that the host library
// grows with cudaMalloc on demand.  g6k_force_static instead places them in
// this file-scope array, which every GPU that loads the library holds (16 MiB)
// until the process exits.  Host code cannot use the array's name as a device
// address: g6k_static_scratch_addr looks the address up (cudaGetSymbolAddress)
// with the caller's device current; the host library does that once in
// g6_open and keeps it in its context until g6_close (a device reset needs
// g6_close + g6_open).  The lookup also loads this module, so the array is
// taken at g6_open, not at the first call.  Every call shares the array:
// nothing in it has to start at zero (each partial record is written by
// exactly one CTA before it is read), and calls that overlap on the GPU
// (different streams, or host threads) race on it.
#define G6_STATIC_SCRATCH_BYTES (16u << 20)
static __device__ __align__(256) unsigned char g6_static_scratch[G6_STATIC_SCRATCH_BYTES];

extern "C" size_t g6k_static_scratch_capacity(void) { return G6_STATIC_SCRATCH_BYTES; }

// 0 and the array's device address on the current device, or -5.
extern "C" int g6k_static_scratch_addr(void **out) {
  void *p = nullptr;
  if (cudaGetSymbolAddress(&p, g6_static_scratch) != cudaSuccess || p == nullptr) return -5;
  *out = p;
  return 0;
}

// Returns 0, -1/-2/-3 as g6k_force, -4 when the launch shape needs more than
// G6_STATIC_SCRATCH_BYTES of scratch (*need_out tells how much), -5 without
// the array's address (static_addr from g6k_static_scratch_addr).
extern "C" int g6k_force_static(const g6_force_args *a, void *static_addr, g6_shape *shape,
                                cudaStream_t st, size_t *need_out) {
  if (!static_addr) return -5;
  const size_t need = g6k_scratch_bytes(a->ni, a->nj, a->prec, a->want_nn,
                                        a->hjerk ? 1 : a->force_jl,
                                        a->force_nsplit);
  if (need_out) *need_out = need;
  if (need > G6_STATIC_SCRATCH_BYTES) return -4;
  g6_force_args b = *a;
  b.scratch = static_addr;
  b.scratch_bytes = G6_STATIC_SCRATCH_BYTES;
  return g6k_force(&b, shape, st);
}
