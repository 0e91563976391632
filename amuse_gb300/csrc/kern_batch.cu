// kern_batch.cu -- many independent few-body systems in one persistent
// launch (the encounters that AMUSE's multiples module hands to smallN).
//
// Each warp takes a system from a device work queue (an atomic counter over
// a host-chosen order, largest systems first), integrates it to its end
// time, writes it back and takes the next one, so uneven systems balance
// themselves.  The integrator is smallN's (src/amuse_ph4/src/smallN.cc):
// batch_exact_kernel without the unperturbed-binary tree (bit-identical to
// smallN with dt_crit = 0), batch_tree_kernel (the fast and split modes) with
// it or without -- a shared-step, time-symmetrised
// 4th-order Hermite scheme --
//   predict_loworder (hdyn.h:192-201) from the stored old acc/jerk,
//   n_iter + 1 force evaluations per step, each followed by
//   correct_acc_and_jerk / correct_pos_and_vel (smallN.cc:487-531) for the
//   iterated step new_dt (smallN.cc:617-660),
//   step from the Kepler criterion eta * sqrt(min over pairs of
//   min(0.5 r^3 / (m_i + m_j), r^2 / v^2)) (smallN.cc:85-116, :318-363).
// State is FP64.  n <= 64.
//
// The exact mode evaluates every expression with the same IEEE operations, in
// the same order, as smallN on the CPU (each pair in its (i < j) orientation,
// contributions accumulated in smallN's pair order, no fused multiply-adds,
// correctly rounded divides and square roots).
// MODE_FAST uses one reciprocal square root per pair and FMAs (results differ
// from smallN at the last-bit level, which chaotic systems amplify).
// MODE_SPLIT keeps the state, the predictor and the corrector in FP64 but
// evaluates the pair terms in FP32 from double-single positions (the
// relative position is exact to FP32 precision of |r|, as in the g6 force
// kernel) and FP32 velocities, with one rsqrt.approx per pair: GB300 runs
// FP32 at 64x its FP64 rate, and the pair terms are the O(n^2) part.
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "fp64_approx.cuh"
#include "g6_dev.h"

namespace {

using namespace fp64;

constexpr int MAXN = 64;
constexpr int WARPS_MAX = 8;
enum { MODE_FAST = 0, MODE_EXACT = 1, MODE_SPLIT = 2 };  // the ABI's G6_BATCH_*


__device__ __forceinline__ double ADD(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double SUB(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double MUL(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double DIV(double a, double b) { return __ddiv_rn(a, b); }

struct Body {
  double m, inv_m;
  double pos[3], vel[3], pp[3], pv[3], acc[3], jerk[3], oacc[3], ojerk[3];
};

struct alignas(16) double4_16 {
  double x, y, z, w;
};

struct WarpSmem {
  double pp[MAXN][3];
  double pv[MAXN][3];
  double m[MAXN];
};

// Contribution of the pair (a, b), a < b in smallN's orientation, to body
// `me` (me == a or me == b), plus the pair's Kepler time-step^2.
__device__ __forceinline__ double pair_term(const WarpSmem &S, int a, int b, bool me_is_a,
                                            double inv_me, double acc[3], double jerk[3]) {
  const double ma = S.m[a], mb = S.m[b];
  double dx[3], dv[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    dx[k] = SUB(S.pp[b][k], S.pp[a][k]);
    dv[k] = SUB(S.pv[b][k], S.pv[a][k]);
  }
  const double d2 = ADD(ADD(MUL(dx[0], dx[0]), MUL(dx[1], dx[1])), MUL(dx[2], dx[2]));
  const double d = __dsqrt_rn(d2);
  const double d3 = MUL(d2, d);
  const double xv = ADD(ADD(MUL(dx[0], dv[0]), MUL(dx[1], dv[1])), MUL(dx[2], dv[2]));
  const double d5 = MUL(d3, d2);
  const double y3 = __drcp_rn(d3), y5 = __drcp_rn(d5);
  const bool r3 = mid_range(d3), r5 = mid_range(d5);
  const double s = me_is_a ? inv_me : -inv_me;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double iforce = div_by(MUL(mb, dx[k]), d3, y3, r3);
    const double ijerk = MUL(mb, SUB(div_by(dv[k], d3, y3, r3),
                                     div_by(MUL(MUL(3.0, dx[k]), xv), d5, y5, r5)));
    const double force = MUL(ma, iforce);
    const double jk = MUL(ma, ijerk);
    acc[k] = ADD(acc[k], MUL(s, force));
    jerk[k] = ADD(jerk[k], MUL(s, jk));
  }
  const double mass = ADD(mb, ma);
  const double vel2 = ADD(ADD(MUL(dv[0], dv[0]), MUL(dv[1], dv[1])), MUL(dv[2], dv[2]));
  const double dtff2 = DIV(MUL(0.5, d3), mass);
  const double dtv2 = DIV(d2, fabs(vel2));
  return fmin(dtff2, dtv2);
}

// acc/jerk of the lane's bodies from the predicted state in S; returns the
// system's min Kepler step^2 (warp-uniform).
__device__ double forces(const WarpSmem &S, int n, int lane, Body B[2]) {
  double ts2 = __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int i = lane + 32 * q;
#pragma unroll
    for (int k = 0; k < 3; k++) B[q].acc[k] = B[q].jerk[k] = 0.0;
    if (i >= n) continue;
    // smallN's pair order: (j, i) for j < i first, then (i, j) for j > i,
    // each pair in its (i < j) orientation.
    for (int j = 0; j < i; j++)
      ts2 = fmin(ts2, pair_term(S, j, i, false, B[q].inv_m, B[q].acc, B[q].jerk));
    for (int j = i + 1; j < n; j++)
      ts2 = fmin(ts2, pair_term(S, i, j, true, B[q].inv_m, B[q].acc, B[q].jerk));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ts2 = fmin(ts2, __shfl_xor_sync(0xffffffffu, ts2, o));
  return ts2;
}

__device__ __forceinline__ void publish(WarpSmem &S, int n, int lane, const Body B[2]) {
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int i = lane + 32 * q;
    if (i < n) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        S.pp[i][k] = B[q].pp[k];
        S.pv[i][k] = B[q].pv[k];
      }
    }
  }
  __syncwarp();
}

// The queue: a warp's first system is its rank with the CTAs counted first,
// so that the first (largest) systems, or the only ones, go to different SMs
// (FP64 issues at 2 lanes per SM: four warps of one CTA at work beside idle
// SMs ran at a quarter of their speed); the others come from the counter.
__device__ __forceinline__ int first_system(int w) { return w * gridDim.x + blockIdx.x; }
__device__ __forceinline__ int next_system(int *queue, int lane) {
  int q = 0;
  if (lane == 0) q = atomicAdd(queue, 1);
  return (int)(gridDim.x * (blockDim.x >> 5)) + __shfl_sync(0xffffffffu, q, 0);
}

__global__ void batch_exact_kernel(const int *__restrict__ order, const int *__restrict__ off,
                                   const double *__restrict__ t_end_s,
                                   const double *__restrict__ mass, double *pos, double *vel,
                                   double eta, int n_iter, long long max_steps, int *queue,
                                   double *t_out, long long *steps_out,
                                   unsigned long long *wall_ns, int *status) {
  __shared__ WarpSmem smem[WARPS_MAX];
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  WarpSmem &S = smem[w];
  const int nsys = queue[1];  // written by the host before the launch
  for (int q = first_system(w); q < nsys; q = next_system(queue, lane)) {
    const int s = order[q];
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    const int base = off[s];
    const int n = off[s + 1] - base;
    const double t_end = t_end_s[s];
    if (n < 2 || n > MAXN) {
      if (lane == 0) {
        status[s] = 2;  // unsupported size (host also checks)
        steps_out[s] = 0;
        t_out[s] = 0.0;
      }
      continue;
    }
    const int nq = n > 32 ? 2 : 1;  // bodies per lane
    Body B[2];
#pragma unroll
    for (int qq = 0; qq < 2; qq++) {
      const int i = lane + 32 * qq;
      const int ii = i < n ? i : 0;
      B[qq].m = mass[base + ii];
      B[qq].inv_m = DIV(1.0, B[qq].m);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        B[qq].pos[k] = pos[3 * (base + ii) + k];
        B[qq].vel[k] = vel[3 * (base + ii) + k];
        B[qq].pp[k] = B[qq].pos[k];  // init_pred
        B[qq].pv[k] = B[qq].vel[k];
        B[qq].oacc[k] = B[qq].ojerk[k] = 0.0;  // hdyn() zeroes them
      }
      if (i < n) S.m[i] = B[qq].m;
    }
    publish(S, n, lane, B);
    double t = 0.0, t_pred = -1.0;
    double dt = MUL(eta, __dsqrt_rn(forces(S, n, lane, B)));
    long long nsteps = 0;
    int st = 0;
    while (t < t_end) {
      if (nsteps >= max_steps) {
        st = 1;  // step budget exhausted
        break;
      }
      const double tn = ADD(t, dt);
      if (tn != t_pred) {  // predict_loworder_all
        const double h = SUB(tn, t);
        const double h3 = DIV(h, 3.0);
        const double h2 = MUL(h, 0.5);  // halving rounds as the division by 2
#pragma unroll
        for (int qq = 0; qq < 2; qq++) {
          if (qq >= nq) break;
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const double oj = B[qq].ojerk[k], oa = B[qq].oacc[k];
            B[qq].pp[k] = ADD(MUL(ADD(MUL(ADD(MUL(oj, h3), oa), h2), B[qq].vel[k]), h), B[qq].pos[k]);
            B[qq].pv[k] = ADD(MUL(ADD(MUL(oj, h2), oa), h), B[qq].vel[k]);
          }
        }
        t_pred = tn;
      }
#pragma unroll
      for (int qq = 0; qq < 2; qq++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          B[qq].oacc[k] = B[qq].acc[k];
          B[qq].ojerk[k] = B[qq].jerk[k];
        }
      double new_dt = dt, end_dt = dt;
      for (int it = 0; it <= n_iter; it++) {
        const double prev = new_dt;
        publish(S, n, lane, B);
        const double ts2 = forces(S, n, lane, B);
        end_dt = MUL(eta, __dsqrt_rn(ts2));
        if (it < n_iter) {
          new_dt = MUL(0.5, ADD(dt, end_dt));
          new_dt = ADD(dt, MUL(MUL(0.5, SUB(end_dt, dt)), DIV(new_dt, prev)));
        }
        const bool cj = new_dt != prev;
        double tau = 0, tau2 = 0, tau3 = 0, theta = 0, inv_theta = 0;
        if (cj) {
          const double dt_off = SUB(new_dt, MUL(0.5, prev));
          theta = MUL(0.5, prev);
          tau = DIV(dt_off, theta);
          inv_theta = DIV(1.0, theta);
          tau2 = MUL(tau, tau);
          tau3 = MUL(tau2, tau);
        }
        const double nd2 = MUL(new_dt, new_dt);
#pragma unroll
        for (int qq = 0; qq < 2; qq++) {
          if (qq >= nq) break;  // an FP64 instruction costs the same without bodies
          Body &b = B[qq];
#pragma unroll
          for (int k = 0; k < 3; k++) {
            if (cj) {  // correct_acc_and_jerk(new_dt, prev)
              const double pa = b.acc[k], pj = b.jerk[k], oa = b.oacc[k], oj = b.ojerk[k];
              const double c1 = ADD(SUB(2.0, MUL(3.0, tau)), tau3);
              const double c2 = SUB(ADD(2.0, MUL(3.0, tau)), tau3);
              const double c3 = ADD(SUB(SUB(1.0, tau), tau2), tau3);
              const double c4 = ADD(ADD(SUB(-1.0, tau), tau2), tau3);
              b.acc[k] = MUL(0.25, ADD(ADD(ADD(MUL(oa, c1), MUL(pa, c2)), MUL(MUL(oj, theta), c3)),
                                       MUL(MUL(pj, theta), c4)));
              const double e1 = ADD(-1.0, tau2), e2 = SUB(1.0, tau2);
              const double e3 = ADD(SUB(-1.0, MUL(2.0, tau)), MUL(3.0, tau2));
              const double e4 = ADD(ADD(-1.0, MUL(2.0, tau)), MUL(3.0, tau2));
              b.jerk[k] = MUL(0.25, ADD(ADD(ADD(MUL(MUL(MUL(oa, inv_theta), 3.0), e1),
                                                MUL(MUL(MUL(pa, inv_theta), 3.0), e2)),
                                            MUL(oj, e3)),
                                        MUL(pj, e4)));
            }
            // correct_pos_and_vel(new_dt)
            b.pv[k] = SUB(ADD(b.vel[k], MUL(MUL(new_dt, ADD(b.acc[k], b.oacc[k])), 0.5)),
                          g6_div_const(MUL(nd2, SUB(b.jerk[k], b.ojerk[k])), 12.0, 1.0 / 12.0));
            b.pp[k] = SUB(ADD(b.pos[k], MUL(MUL(new_dt, ADD(b.pv[k], b.vel[k])), 0.5)),
                          g6_div_const(MUL(nd2, SUB(b.acc[k], b.oacc[k])), 12.0, 1.0 / 12.0));
          }
        }
      }
#pragma unroll
      for (int qq = 0; qq < 2; qq++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          B[qq].pos[k] = B[qq].pp[k];
          B[qq].vel[k] = B[qq].pv[k];
        }
      dt = end_dt;
      t = ADD(t, new_dt);
      nsteps++;
    }
#pragma unroll
    for (int qq = 0; qq < 2; qq++) {
      const int i = lane + 32 * qq;
      if (i < n) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
          pos[3 * (base + i) + k] = B[qq].pos[k];
          vel[3 * (base + i) + k] = B[qq].vel[k];
        }
      }
    }
    if (lane == 0) {
      unsigned long long t1;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      t_out[s] = t;
      steps_out[s] = nsteps;
      wall_ns[s] = t1 - t0;
      status[s] = st;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Unperturbed binaries (smallN's default treatment: src/amuse_ph4/src/
// smallN.cc:1022-1060 and smallN_unpert.cc): after each step the pair that
// set the time step becomes a binary node when it is approaching, closer
// than r_crit, its step is below dt_crit and the strongest perturber's
// tidal parameter gamma^2 = 4 (m_k/M)^2 (r^2/d_k^2)^3 is below gamma^2_unpert
// (smallN_unpert.cc:44-88).  Its centre of mass is integrated like a body;
// its components follow the two-body orbit (universal-variable Kepler
// propagation) and are resolved for every force evaluation (forces between
// top-level nodes are sums over their leaves, smallN.cc:127-240; the step
// criterion takes the closest leaf pair with the nodes' masses and
// velocities).  The unperturbed segment ends at the time the orbit returns
// to the same separation past pericentre (smallN_unpert.cc:252-266, 335);
// there the change of the tidal potential is absorbed into the relative
// velocity, and the binary is either extended by whole periods (frozen
// components) while no perturber can arrive (dt_perturbers,
// smallN_unpert.cc:402-460, 682-704) or dissolved.  The same algorithm, with
// the same stated differences from smallN, is the oracle's
// orc_smalln_unpert.  FAST (FP64 pair terms) and SPLIT (FP32 pair terms)
// modes; all tree decisions are taken redundantly by every lane of the
// warp from shared data, so they are warp-uniform.
//
// What bounds it: FP64 issues at 2 lanes per SM and cycle, half a lane per
// scheduler, so an FP64 instruction holds a warp's scheduler for 64 cycles
// however few lanes need it.  So the per-body work is laid out by component:
// lane l holds components l, l + 32, ... of the system's 3n (a 3-body system
// has 9 lanes at work in one pass, where a lane per body took three passes of
// three lanes, and two more for bodies 33 .. 64 that were not there); the
// corrector's eight coefficients are evaluated by eight lanes at once;
// quotients and square roots are fp64_approx.cuh's; and comparisons of non-negative
// values are integer compares.  4096 scatterings 20.4 -> 5.4 ms, 1024 systems
// of 3 to 64 bodies over 0.05 crossing times 10.3 -> 6.1 ms (one draw; its longest
// system sets the time, and other draws take 5 to 31).  A lone warp is
// bound by instruction latency (6 to 7 cycles per instruction of 32,000 a step
// at n = 52), so the split mode's pair loop reads a body in three or four
// 16-byte loads and evaluates two pairs per packed f32x2 instruction.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr int NB = 8;  // binaries per system at most

struct BinRec {
  int li, lj, full, pad;
  double mi, mj, r0[3], v0[3], t0, tpred, tidal;
  // the last Kepler solution (universal anomaly, its dt, the separation):
  // the next solve starts from it (dtw = 0: none yet)
  double xw, dtw, rw;
};

struct UnpParams {
  double dt_crit, r2_crit, gamma2, gamma_inv3;
  int allow_full;
  int on;  // 0: no binaries are made
};

struct alignas(16) UnpSmem {
  // leaves for the force loop; in split mode d holds the nodes for the tree
  struct {
    double4_16 pp[MAXN];  // x, y, z, leaf mass
    double4_16 pv[MAXN];  // velocity, mass of the leaf's node
  } d;
  struct {
    float4 hi[MAXN];  // x, y, z (high words), leaf mass
    float4 lo[MAXN];  // x, y, z (low words), -
    float4 vf[MAXN];  // velocity, mass of the leaf's node
    float4 cv[MAXN];  // velocity of the leaf's node
  } f;
  double4_16 cv[MAXN];  // fast mode: velocity of the leaf's node
  double la[MAXN][3], lj[MAXN][3];  // leaf forces, then node accelerations
  double nm[MAXN];                   // node masses (at node slots)
  double kr[NB][6];                  // binaries' relative position and velocity
  int nd[MAXN];                      // node (leader slot) of every leaf slot
  int bi[MAXN];                      // binary of a node slot, -1: a single leaf
  BinRec bin[NB];
  int nb;
};

// a b + c d and a . b with the order of their roundings fixed (left to the
// compiler, it varies with the surroundings): the split mode's FP32 pair terms
// turn a last bit of the FP64 state into 6e-8 of a term now and then, and a
// hard binary amplifies that to 1e-6 of a position within 0.05 crossing times.
__device__ __forceinline__ double two(double a, double b, double c, double d) {
  return __fma_rn(a, b, __dmul_rn(c, d));
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return __fma_rn(a[2], b[2], two(a[0], b[0], a[1], b[1]));
}
// Stumpff functions C(z) = (1 - cos sqrt z) / z, S(z) = (sqrt z - sin sqrt z)
// / z^(3/2) (cosh, sinh for z < 0), both from one sincos (one exp) of
// sqrt(|z|) / 2: 1 - cos s = 2 sin^2(s/2) (no cancellation), sin s = 2
// sin(s/2) cos(s/2).  Taylor series to z^6 for |z| < 0.1 (below 1e-17
// relative).  FP64 transcendentals run at the FP64 rate, so one call per
// Newton step rather than two.
__device__ __forceinline__ void kst_cs(double z, double &C, double &S) {
  if (z > 0.1) {
    const double s = sqrt64(z);
    double sh, ch;
    sincos(0.5 * s, &sh, &ch);
    C = div64(2.0 * sh * sh, z);
    S = div64(s - 2.0 * sh * ch, s * z);
  } else if (z < -0.1) {
    const double s = sqrt64(-z), e = exp(0.5 * s), ei = Div(e).inv();
    const double sh = 0.5 * (e - ei), ch = 0.5 * (e + ei);
    C = div64(2.0 * sh * sh, -z);
    S = div64(2.0 * sh * ch - s, s * -z);
  } else {
    C = 1.0 / 2 +
        z * (-1.0 / 24 +
             z * (1.0 / 720 +
                  z * (-1.0 / 40320 +
                       z * (1.0 / 3628800 + z * (-1.0 / 479001600 + z / 87178291200.0)))));
    S = 1.0 / 6 +
        z * (-1.0 / 120 +
             z * (1.0 / 5040 +
                  z * (-1.0 / 362880 +
                       z * (1.0 / 39916800 + z * (-1.0 / 6227020800.0 + z / 1307674368000.0)))));
  }
}

// Two-body relative motion over dt (mu = G M), universal variables: the
// universal anomaly x solves
//   F(x) = (r0.v0 / sqrt(mu)) x^2 C(z) + (1 - alpha r0) x^3 S(z) + r0 x - sqrt(mu) dt = 0,
// z = alpha x^2, whose derivative is the separation r(x) > 0.  F being
// monotonic, the root is bracketed and found by Newton steps that fall back
// to bisection when a step leaves the bracket or does not halve the one
// before last (a plain Newton iteration diverges on eccentric orbits near
// pericentre).  The first guess is the mean-motion one, or, with a warm
// start (*dtw > 0: the solution xw at dtw, separation rw, of the same
// orbit), xw + sqrt(mu) (dt - dtw) / rw (dx/dt = sqrt(mu) / r); x grows with
// dt, so xw then also bounds the root from one side.  The C and S of the
// step whose correction is below 1e-15 x give the f and g functions.
// LAST: which of F's first two terms is added last (the force evaluations
// round one way, the tree's decisions the other).
template <bool LAST>
__device__ __noinline__ void kep_prop(double mu, const double r0[3], const double v0[3], double dt,
                         double r[3], double v[3], double *xw = nullptr, double *dtw = nullptr,
                         double *rw = nullptr) {
  const double rn = sqrt64(dot3(r0, r0));
  const double v2 = dot3(v0, v0), rv = dot3(r0, v0);
  const double smu = sqrt64(mu);
  const Div by_rn(rn), by_smu(smu);
  const double alpha = by_rn(2.0) - div64(v2, mu);
  const double c1 = by_smu(rv), c2 = 1.0 - alpha * rn;
  if (dt == 0.0) {
    for (int k = 0; k < 3; k++) r[k] = r0[k], v[k] = v0[k];
    return;
  }
  const double sd = __dmul_rn(smu, dt);
  auto Fcs = [&](double x, double C, double S) {
    const double a = c1 * x * x, b = c2 * x * x * x;
    return __dsub_rn(__fma_rn(rn, x, LAST ? two(b, S, a, C) : two(a, C, b, S)), sd);
  };
  auto Fx = [&](double x) {
    double C, S;
    kst_cs(alpha * x * x, C, S);
    return Fcs(x, C, S);
  };
  const bool warm = xw && *dtw > 0.0 && dt > 0.0;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  double x0 = alpha > 0.0 ? smu * dt * alpha : by_rn(smu * dt);  // sign of dt
  double lo, hi;
  if (warm) {
    // The root lies above xw when dt >= dtw (F(xw) <= 0), else in (0, xw).
    // No evaluation before the first Newton step: with hi = +inf, steps from
    // below (F < 0, dF > 0) only move up, until one lands above the root and
    // bounds it.
    x0 = *xw + div64(smu * (dt - *dtw), *rw);
    lo = dt >= *dtw ? *xw : 0.0;
    hi = dt >= *dtw ? inf : *xw;
    if (!(x0 > lo && x0 < hi)) x0 = hi < inf ? 0.5 * (lo + hi) : lo + fabs(lo) + 1e-300;
  } else if (dt > 0.0) {
    lo = 0.0, hi = x0;
    for (int k = 0; k < 200 && Fx(hi) < 0.0; k++) lo = hi, hi *= 2.0;
  } else {
    hi = 0.0, lo = x0;
    for (int k = 0; k < 200 && Fx(lo) > 0.0; k++) hi = lo, lo *= 2.0;
  }
  double x = x0 > lo && x0 < hi ? x0 : 0.5 * (lo + hi);
  double step_old = hi - lo, step = step_old, C = 0.5, S = 1.0 / 6;
  for (int it = 0; it < 200; it++) {
    const double z = alpha * x * x;
    kst_cs(z, C, S);
    const double F = Fcs(x, C, S);
    const double dF = __dadd_rn(two(c2 * x * x, C, c1 * x, __fma_rn(-z, S, 1.0)), rn);
    if (F == 0.0 || fabs(F) <= 1e-15 * fabs(x * dF)) break;  // x is the root: C, S belong to it
    if (F < 0.0)
      lo = x;
    else
      hi = x;
    const double newton = div64(F, dF);
    double xn = x - newton;
    if (hi < inf && (!(xn > lo && xn < hi) || fabs(2.0 * F) > fabs(step_old * dF))) {
      step_old = step;
      step = 0.5 * (hi - lo);
      xn = lo + step;
    } else {
      step_old = step;
      step = newton;
    }
    if (xn == x) break;
    x = xn;
  }
  const double f = 1.0 - by_rn(x * x * C), g = dt - by_smu(x * x * x * S);
  for (int k = 0; k < 3; k++) r[k] = two(f, r0[k], g, v0[k]);
  const double rr = sqrt64(dot3(r, r));
  const double fd = div64(smu, rr * rn) * (alpha * x * x * x * S - x);
  const double gd = 1.0 - div64(x * x * C, rr);
  for (int k = 0; k < 3; k++) v[k] = two(fd, r0[k], gd, v0[k]);
  if (xw && dt > 0.0) {
    *xw = x;
    *dtw = dt;
    *rw = rr;
  }
}

// Time to the next pericentre (0: not approaching it) and the period (inf
// unless bound): mean anomaly from the eccentric (hyperbolic) anomaly;
// Barker's equation near e = 1.
__device__ __noinline__ int kep_peri(double mu, const double r[3], const double v[3], double *dt_peri,
                        double *period) {
  const double rn = sqrt(dot3(r, r));
  const double v2 = dot3(v, v);
  const double rv = dot3(r, v);
  *period = __longlong_as_double(0x7ff0000000000000ll);
  if (rv >= 0.0) return 0;
  const double alpha = 2.0 / rn - v2 / mu;
  const double h[3] = {two(r[1], v[2], -r[2], v[1]), two(r[2], v[0], -r[0], v[2]),
                       two(r[0], v[1], -r[1], v[0])};
  const double p = dot3(h, h) / mu;
  const double e = sqrt(fmax(0.0, 1.0 - p * alpha));
  if (fabs(alpha) * rn < 1e-8 || e < 1e-12) {
    const double D = rv / sqrt(mu * p);
    *dt_peri = -0.5 * sqrt(p * p * p / mu) * (D + D * D * D / 3.0);
    if (alpha > 0.0) *period = 2.0 * M_PI / sqrt(mu * alpha * alpha * alpha);
    return *dt_peri > 0.0;
  }
  double M, n;
  if (alpha > 0.0) {
    const double a = 1.0 / alpha;
    const double E = atan2(rv / (e * sqrt(mu * a)), (1.0 - rn * alpha) / e);
    M = E - e * sin(E);
    n = sqrt(mu * alpha * alpha * alpha);
    *period = 2.0 * M_PI / n;
  } else {
    const double sF = rv / (e * sqrt(-mu / alpha));
    M = e * sF - asinh(sF);
    n = sqrt(-mu * alpha * alpha * alpha);
  }
  if (M >= 0.0) return 0;
  *dt_peri = -M / n;
  return 1;
}

__device__ __forceinline__ double dist3(const double a[3], const double4_16 &b) {
  const double d[3] = {a[0] - b.x, a[1] - b.y, a[2] - b.z};
  return sqrt64(dot3(d, d));
}

// The relative state of a binary at time t (frozen when fully unperturbed).
__device__ __forceinline__ void bin_rel(const BinRec &b, double t, double r[3], double v[3]) {
  if (b.full) {
    for (int k = 0; k < 3; k++) r[k] = b.r0[k], v[k] = b.v0[k];
  } else {
    kep_prop<false>(b.mi + b.mj, b.r0, b.v0, t - b.t0, r, v);
  }
}
// The same, starting the Kepler solve from the binary's last solution and
// keeping this one (the force evaluations: a few per step, at nearby times).
template <bool LAST>
__device__ __forceinline__ void bin_rel_warm(BinRec &b, double t, double r[3], double v[3]) {
  if (b.full) {
    for (int k = 0; k < 3; k++) r[k] = b.r0[k], v[k] = b.v0[k];
  } else {
    kep_prop<LAST>(b.mi + b.mj, b.r0, b.v0, t - b.t0, r, v, &b.xw, &b.dtw, &b.rw);
  }
}

// Warp-wide sum and minimum (xor butterfly: every lane ends with the same
// value, a + b being b + a).
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ double warp_min(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmin(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Tidal potential of the other top-level nodes on leaves (xi, xj) around
// the centre of mass xc (smallN_unpert.cc:17-40); node positions in S.d.
// The whole warp calls it (uniform arguments); each lane sums its two node
// slots (the tree's loops over nodes run at 1/32 of the FP64 work per lane).
__device__ __noinline__ double tidal_pot(const UnpSmem &S, int n, int lane, int li, int lj, double mi,
                            double mj, const double xi[3], const double xj[3],
                            const double xc[3]) {
  double phi = 0.0;
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int k = lane + 32 * q;
    if (k >= n || S.nd[k] != k || k == li || k == lj) continue;
    phi += S.nm[k] * (div64(-mi, dist3(xi, S.d.pp[k])) - div64(mj, dist3(xj, S.d.pp[k])) +
                      div64(mi + mj, dist3(xc, S.d.pp[k])));
  }
  return warp_sum(phi);
}

// What every lane keeps of the components c = lane + 32 r of the 3n: body
// c / 3, coordinate c % 3.  NS slots, a template parameter of all that
// follows: slots a system does not have would be predicated off, and an FP64
// instruction costs its time all the same (a 3-body step issued 813 of them
// with six slots).
template <int NS>
struct Comp {
  double pos[NS], vel[NS], pp[NS], pv[NS], acc[NS], jerk[NS], oacc[NS], ojerk[NS];
};

#define FOR_COMP(r, c, n)                          \
  _Pragma("unroll") for (int r = 0; r < NS; r++) \
    if (const int c = lane + 32 * r; c < 3 * (n))

__device__ __forceinline__ double &elem(double4_16 &v, int k) { return (&v.x)[k]; }
__device__ __forceinline__ float &elem(float4 &v, int k) { return (&v.x)[k]; }

// One component of a leaf's predicted state, and (TREE) of its node's
// velocity.
template <int MODE, bool TREE>
__device__ __forceinline__ void store_leaf(UnpSmem &S, int s, int k, double x, double v,
                                           double cv) {
  if (MODE == MODE_SPLIT) {
    const float h = __double2float_rn(x);
    elem(S.f.hi[s], k) = h;
    elem(S.f.lo[s], k) = __double2float_rn(x - (double)h);
    elem(S.f.vf[s], k) = __double2float_rn(v);
    if (TREE) elem(S.f.cv[s], k) = __double2float_rn(cv);
  } else {
    elem(S.d.pp[s], k) = x;
    elem(S.d.pv[s], k) = v;
    if (TREE) elem(S.cv[s], k) = cv;
  }
}

// The masses beside the leaves (their own and their node's), and the binary
// of every node slot: after the tree changed.
template <int MODE>
__device__ void tree_masses(UnpSmem &S, int n, int lane) {
  __syncwarp();
  for (int s = lane; s < n; s += 32) {
    int b = -1;
    for (int q = 0; q < S.nb; q++)
      if (S.bin[q].li == s) b = q;
    S.bi[s] = b;
    const double nm = S.nm[S.nd[s]];
    if (MODE == MODE_SPLIT)
      S.f.vf[s].w = __double2float_rn(nm);
    else
      S.d.pv[s].w = nm;
  }
  __syncwarp();
}

// MODE_SPLIT pair loop for the lane's leaves i = lane (and lane + 32): sums
// over all leaves of other nodes, the smallest step^2 and its node pair, two
// pairs per packed instruction: both leaves of the lane with one j (NQ = 2),
// or one leaf with two j, whose terms are then added one after the other, so
// the sums run over j in order either way.  Pairs within one node (the leaf
// itself among them) are evaluated with rinv = 0, so the loop does not
// diverge.  The pair that sets the step is the one with the largest max(2 M /
// r^3, v^2 / r^2); its step^2 is then taken from the quotients (approximate
// division), or the smallest of all pairs' where a second one is as large to
// within the measures' errors (2^-17).  FP32 unless a pair is closer than 1e-9
// (d^2 < 1e-18): there m / d^3 times a relative velocity ~ sqrt(M / d) can
// leave the FP32 range, so such (rare) pairs are left out of the loop and
// evaluated in FP64 after it.
// TREE false: no binaries, every leaf is its node.
struct Leaf {
  float4 h, l, v, c;  // position words (mass), velocity (node mass), node velocity
  int node;
};
template <bool TREE>
__device__ __forceinline__ Leaf get_leaf(const UnpSmem &S, int j) {
  Leaf b;
  b.h = S.f.hi[j];
  b.l = S.f.lo[j];
  b.v = S.f.vf[j];
  b.c = TREE ? S.f.cv[j] : b.v;
  b.node = TREE ? S.nd[j] : j;
  return b;
}
struct Pair2 {  // two leaves, one per half
  f2x hx, hy, hz, lx, ly, lz, vx, vy, vz, cx, cy, cz, m, nm;
};
__device__ __forceinline__ Pair2 pack_leaves(const Leaf &a, const Leaf &b) {
  Pair2 p;
  p.hx = f2_pack(a.h.x, b.h.x), p.hy = f2_pack(a.h.y, b.h.y), p.hz = f2_pack(a.h.z, b.h.z);
  p.lx = f2_pack(a.l.x, b.l.x), p.ly = f2_pack(a.l.y, b.l.y), p.lz = f2_pack(a.l.z, b.l.z);
  p.vx = f2_pack(a.v.x, b.v.x), p.vy = f2_pack(a.v.y, b.v.y), p.vz = f2_pack(a.v.z, b.v.z);
  p.cx = f2_pack(a.c.x, b.c.x), p.cy = f2_pack(a.c.y, b.c.y), p.cz = f2_pack(a.c.z, b.c.z);
  p.m = f2_pack(a.h.w, b.h.w), p.nm = f2_pack(a.v.w, b.v.w);
  return p;
}
// The terms of the pairs (i, j) of both halves: f dx is the acceleration, f u
// the jerk, w the step's measure; near is set where a pair is too close.
template <bool TREE>
__device__ __forceinline__ void pair_terms(const Pair2 &i, const Pair2 &j, bool same0, bool same1,
                                           f2x &f, f2x dx[3], f2x u[3], float &w0, float &w1,
                                           bool &near0, bool &near1) {
  dx[0] = f2_add(f2_sub(j.hx, i.hx), f2_sub(j.lx, i.lx));
  dx[1] = f2_add(f2_sub(j.hy, i.hy), f2_sub(j.ly, i.ly));
  dx[2] = f2_add(f2_sub(j.hz, i.hz), f2_sub(j.lz, i.lz));
  const f2x dv[3] = {f2_sub(j.vx, i.vx), f2_sub(j.vy, i.vy), f2_sub(j.vz, i.vz)};
  const f2x d2 = f2_fma(dx[2], dx[2], f2_fma(dx[1], dx[1], f2_mul(dx[0], dx[0])));
  f2x v2;
  if (TREE) {
    const f2x c0 = f2_sub(j.cx, i.cx), c1 = f2_sub(j.cy, i.cy), c2 = f2_sub(j.cz, i.cz);
    v2 = f2_fma(c2, c2, f2_fma(c1, c1, f2_mul(c0, c0)));
  } else {
    v2 = f2_fma(dv[2], dv[2], f2_fma(dv[1], dv[1], f2_mul(dv[0], dv[0])));
  }
  float a, b;
  f2_unpack(d2, a, b);
  const bool n0 = !(a >= 1e-18f), n1 = !(b >= 1e-18f);
  near0 |= n0 && !same0;
  near1 |= n1 && !same1;
  const f2x rinv = f2_pack(same0 || n0 ? 0.f : rsqrt_approx(a), same1 || n1 ? 0.f : rsqrt_approx(b));
  const f2x rinv2 = f2_mul(rinv, rinv);
  f = f2_mul(f2_mul(j.m, rinv), rinv2);
  const f2x xv = f2_fma(dx[2], dv[2], f2_fma(dx[1], dv[1], f2_mul(dx[0], dv[0])));
  const f2x a3 = f2_mul(f2_mul(f2_dup(-3.0f), xv), rinv2);
#pragma unroll
  for (int k = 0; k < 3; k++) u[k] = f2_fma(a3, dx[k], dv[k]);
  const f2x M = f2_add(i.nm, j.nm);
  const f2x wm = f2_mul(f2_mul(f2_add(M, M), rinv), rinv2), wv = f2_mul(v2, rinv2);
  w0 = fmaxf(f2_lo(wm), f2_lo(wv));
  w1 = fmaxf(f2_hi(wm), f2_hi(wv));
}

template <bool TREE, int NQ>
__device__ __forceinline__ void pairs_split(UnpSmem &S, int n, int lane, double la[2][3],
                                            double lj[2][3], float tsq[2], int pq[2]) {
  float a[NQ][3], jk[NQ][3], wb[NQ], ws[NQ];
  int jb[NQ], ni[NQ];
  bool near[2] = {false, false};
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    wb[q] = ws[q] = 0.f;
    jb[q] = -1;
    ni[q] = TREE ? S.nd[min(lane + 32 * q, n - 1)] : lane + 32 * q;
  }
  f2x f, dx[3], u[3];
  float w0, w1;
  if (NQ == 2) {
    const Pair2 I = pack_leaves(get_leaf<TREE>(S, lane), get_leaf<TREE>(S, min(lane + 32, n - 1)));
    f2x A[3] = {0ull, 0ull, 0ull}, J[3] = {0ull, 0ull, 0ull};
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      const Leaf b = get_leaf<TREE>(S, j);
      pair_terms<TREE>(I, pack_leaves(b, b), b.node == ni[0], b.node == ni[NQ - 1], f, dx, u, w0,
                       w1, near[0], near[1]);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        A[k] = f2_fma(f, dx[k], A[k]);
        J[k] = f2_fma(f, u[k], J[k]);
      }
      ws[0] = fmaxf(ws[0], fminf(w0, wb[0]));
      if (w0 > wb[0]) wb[0] = w0, jb[0] = j;
      ws[NQ - 1] = fmaxf(ws[NQ - 1], fminf(w1, wb[NQ - 1]));
      if (w1 > wb[NQ - 1]) wb[NQ - 1] = w1, jb[NQ - 1] = j;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      f2_unpack(A[k], a[0][k], a[NQ - 1][k]);
      f2_unpack(J[k], jk[0][k], jk[NQ - 1][k]);
    }
  } else {
    const Leaf me = get_leaf<TREE>(S, min(lane, n - 1));
    const Pair2 I = pack_leaves(me, me);
#pragma unroll
    for (int k = 0; k < 3; k++) a[0][k] = jk[0][k] = 0.f;
#pragma unroll 1
    for (int j = 0; j < n; j += 2) {
      const bool two = j + 1 < n;
      const Leaf b = get_leaf<TREE>(S, j), c = get_leaf<TREE>(S, two ? j + 1 : j);
      pair_terms<TREE>(I, pack_leaves(b, c), b.node == ni[0], !two || c.node == ni[0], f, dx, u,
                       w0, w1, near[0], near[1]);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        a[0][k] = fmaf(f2_hi(f), f2_hi(dx[k]), fmaf(f2_lo(f), f2_lo(dx[k]), a[0][k]));
        jk[0][k] = fmaf(f2_hi(f), f2_hi(u[k]), fmaf(f2_lo(f), f2_lo(u[k]), jk[0][k]));
      }
      ws[0] = fmaxf(ws[0], fminf(w0, wb[0]));
      if (w0 > wb[0]) wb[0] = w0, jb[0] = j;
      ws[0] = fmaxf(ws[0], fminf(w1, wb[0]));
      if (w1 > wb[0]) wb[0] = w1, jb[0] = j + 1;
    }
    near[0] |= near[1];
  }
#pragma unroll
  for (int q = 0; q < NQ; q++) {
#pragma unroll
    for (int k = 0; k < 3; k++) la[q][k] = (double)a[q][k], lj[q][k] = (double)jk[q][k];
    const int i = lane + 32 * q;
    tsq[q] = __int_as_float(0x7f800000);
    pq[q] = 0x7fffffff;
    if (i >= n) continue;
    const Leaf me = get_leaf<TREE>(S, i);
    // another pair's measure as large to within the measures' errors: the
    // quotients of all of them decide
    const bool all = ws[q] >= wb[q] * (1.0f - 0x1p-17f);
    for (int j = all ? 0 : jb[q]; j >= 0 && j < n; j++) {
      if (!all && j != jb[q]) break;
      const Leaf b = get_leaf<TREE>(S, j);
      if (b.node == ni[q]) continue;
      const float d0 = __fadd_rn(__fsub_rn(b.h.x, me.h.x), __fsub_rn(b.l.x, me.l.x));
      const float d1 = __fadd_rn(__fsub_rn(b.h.y, me.h.y), __fsub_rn(b.l.y, me.l.y));
      const float d2 = __fadd_rn(__fsub_rn(b.h.z, me.h.z), __fsub_rn(b.l.z, me.l.z));
      const float c0 = b.c.x - me.c.x, c1 = b.c.y - me.c.y, c2 = b.c.z - me.c.z;
      const float dd = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
      if (dd < 1e-18f) continue;
      const float v2 = fmaf(c2, c2, fmaf(c1, c1, c0 * c0));
      const float ts = fminf(__fdividef(0.5f * dd * (dd * rsqrt_approx(dd)), me.v.w + b.v.w),
                             __fdividef(dd, v2));
      const int pid = ni[q] < b.node ? ni[q] * MAXN + b.node : b.node * MAXN + ni[q];
      if (ts < tsq[q] || (ts == tsq[q] && pid < pq[q])) tsq[q] = ts, pq[q] = pid;
    }
    if (near[q]) {  // pairs too close for FP32: FP64, added up by themselves
      double na[3] = {0.0, 0.0, 0.0}, nj[3] = {0.0, 0.0, 0.0};
      for (int j = 0; j < n; j++) {
        const Leaf b = get_leaf<TREE>(S, j);
        if (b.node == ni[q]) continue;
        const float e0 = __fadd_rn(__fsub_rn(b.h.x, me.h.x), __fsub_rn(b.l.x, me.l.x));
        const float e1 = __fadd_rn(__fsub_rn(b.h.y, me.h.y), __fsub_rn(b.l.y, me.l.y));
        const float e2 = __fadd_rn(__fsub_rn(b.h.z, me.h.z), __fsub_rn(b.l.z, me.l.z));
        if (fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) >= 1e-18f) continue;
        const float c0 = b.c.x - me.c.x, c1 = b.c.y - me.c.y, c2 = b.c.z - me.c.z;
        const double v2 = (double)fmaf(c2, c2, fmaf(c1, c1, c0 * c0));
        const double X[3] = {(double)e0, (double)e1, (double)e2};
        const double U[3] = {(double)(b.v.x - me.v.x), (double)(b.v.y - me.v.y),
                             (double)(b.v.z - me.v.z)};
        const double dd2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
        const double d = sqrt(dd2), ri2 = 1.0 / dd2, fd = S.d.pp[j].w * ri2 / d;
        const double a3 = -3.0 * (X[0] * U[0] + X[1] * U[1] + X[2] * U[2]) * ri2;
        for (int k = 0; k < 3; k++) {
          na[k] += fd * X[k];
          nj[k] += fd * (a3 * X[k] + U[k]);
        }
        const float ts =
            (float)fmin(0.5 * dd2 * d / (double)(me.v.w + b.v.w), dd2 / v2);
        const int pid = ni[q] < b.node ? ni[q] * MAXN + b.node : b.node * MAXN + ni[q];
        if (ts < tsq[q] || (ts == tsq[q] && pid < pq[q])) tsq[q] = ts, pq[q] = pid;
      }
      for (int k = 0; k < 3; k++) la[q][k] += na[k], lj[q][k] += nj[k];
    }
  }
}

// MODE_FAST pair loop: FP64, with the largest 1 / step^2 = max(2 M / r^3,
// v^2 / r^2) in the place of the smallest step^2 (no divisions).  The pairs of
// one node are masked (rinv = 0).  Bound by FP64 issue: about 40 instructions
// per pair at 64 cycles (52 bodies: 150 us per evaluation, 240 before).
template <bool TREE, int NQ>
__device__ __forceinline__ void pairs_fast(UnpSmem &S, int n, int lane, double la[2][3],
                                           double lj[2][3], double &wmax, int &pmin) {
  double4_16 X[NQ], V[NQ], C[NQ];
  int ni[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int i = min(lane + 32 * q, n - 1);
    X[q] = S.d.pp[i];
    V[q] = S.d.pv[i];
    if (TREE) C[q] = S.cv[i];
    ni[q] = TREE ? S.nd[i] : i;
#pragma unroll
    for (int k = 0; k < 3; k++) la[q][k] = lj[q][k] = 0.0;
  }
  constexpr int UNR = NQ == 2 ? 1 : 2;
#pragma unroll UNR
  for (int j = 0; j < n; j++) {
    const int nj = TREE ? S.nd[j] : j;
    const double4_16 Y = S.d.pp[j], U = S.d.pv[j];
    double4_16 D;
    if (TREE) D = S.cv[j];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const bool same = nj == ni[q];
      const double dx = Y.x - X[q].x, dy = Y.y - X[q].y, dz = Y.z - X[q].z;
      const double du = U.x - V[q].x, dv = U.y - V[q].y, dw = U.z - V[q].z;
      const double d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
      const double rinv = same ? 0.0 : rsqrt64_normal(d2);
      const double rinv2 = rinv * rinv, rinv3 = rinv * rinv2;
      const double f = Y.w * rinv3;
      const double a3 = -3.0 * __fma_rn(dz, dw, __fma_rn(dy, dv, dx * du)) * rinv2;
      la[q][0] = __fma_rn(f, dx, la[q][0]);
      la[q][1] = __fma_rn(f, dy, la[q][1]);
      la[q][2] = __fma_rn(f, dz, la[q][2]);
      lj[q][0] = __fma_rn(f, __fma_rn(a3, dx, du), lj[q][0]);
      lj[q][1] = __fma_rn(f, __fma_rn(a3, dy, dv), lj[q][1]);
      lj[q][2] = __fma_rn(f, __fma_rn(a3, dz, dw), lj[q][2]);
      double c0 = du, c1 = dv, c2 = dw;
      if (TREE) c0 = D.x - C[q].x, c1 = D.y - C[q].y, c2 = D.z - C[q].z;
      const double v2 = __fma_rn(c2, c2, __fma_rn(c1, c1, c0 * c0));
      const double w1 = (V[q].w + U.w) * (rinv3 + rinv3), w2 = v2 * rinv2;
      // both are >= 0 (0 when masked): integer compares
      const long long b1 = __double_as_longlong(w1), b2 = __double_as_longlong(w2);
      const long long bw = b1 > b2 ? b1 : b2, b0 = __double_as_longlong(wmax);
      const int pid = ni[q] < nj ? ni[q] * MAXN + nj : nj * MAXN + ni[q];
      if (!same && (bw > b0 || (bw == b0 && pid < pmin))) {
        wmax = __longlong_as_double(bw);
        pmin = pid;
      }
    }
  }
}

// Resolved forces on the top-level nodes from the predicted components:
// returns the natural step (warp-uniform, eta sqrt(min step^2)) and the node
// pair setting it.
template <int MODE, int NS>
__device__ __forceinline__ double tree_forces(UnpSmem &S, int n, int lane, Comp<NS> &B, double t, double eta,
                              int *imin, int *jmin) {
  const unsigned FULL = 0xffffffffu;
  constexpr int NQ = NS > 3 ? 2 : 1;  // leaves per lane
  const int nb = S.nb;
  __syncwarp();
  if (nb > 0) {
    if (lane < nb) {  // a lane per binary: its components' relative state at t
      double r[3], v[3];
      bin_rel_warm<false>(S.bin[lane], t, r, v);
      for (int k = 0; k < 3; k++) S.kr[lane][k] = r[k], S.kr[lane][3 + k] = v[k];
    }
    __syncwarp();
  }
  FOR_COMP(r, c, n) {
    const int s = c / 3, k = c - 3 * s;
    if (nb == 0) {
      store_leaf<MODE, false>(S, s, k, B.pp[r], B.pv[r], B.pv[r]);
    } else if (S.nd[s] == s) {
      const int b = S.bi[s];
      if (b < 0) {
        store_leaf<MODE, true>(S, s, k, B.pp[r], B.pv[r], B.pv[r]);
      } else {
        const BinRec &bb = S.bin[b];
        const Div by_M(bb.mi + bb.mj);
        const double fi = by_M(bb.mj), fj = by_M(bb.mi);
        const double x = S.kr[b][k], v = S.kr[b][3 + k];
        store_leaf<MODE, true>(S, bb.li, k, B.pp[r] - fi * x, B.pv[r] - fi * v, B.pv[r]);
        store_leaf<MODE, true>(S, bb.lj, k, B.pp[r] + fj * x, B.pv[r] + fj * v, B.pv[r]);
      }
    }
  }
  __syncwarp();
  double dt;
  int pmin = 0x7fffffff;
  double la[2][3], lj[2][3];
  if (MODE == MODE_SPLIT) {
    float ts[2];
    int pq[2];
    ts[1] = __int_as_float(0x7f800000);
    pq[1] = 0x7fffffff;
    if (nb == 0)
      pairs_split<false, NQ>(S, n, lane, la, lj, ts, pq);
    else
      pairs_split<true, NQ>(S, n, lane, la, lj, ts, pq);
    if (ts[1] < ts[0] || (ts[1] == ts[0] && pq[1] < pq[0])) ts[0] = ts[1], pq[0] = pq[1];
    const unsigned u = __float_as_uint(ts[0]);  // >= +0, or +inf: ordered as its bits
    const unsigned m = __reduce_min_sync(FULL, u);
    pmin = (int)__reduce_min_sync(FULL, u == m ? (unsigned)pq[0] : 0x7fffffffu);
    dt = eta * sqrt64((double)(__uint_as_float(m)));
  } else {
    double w = 0.0;
    if (nb == 0)
      pairs_fast<false, NQ>(S, n, lane, la, lj, w, pmin);
    else
      pairs_fast<true, NQ>(S, n, lane, la, lj, w, pmin);
    long long b = __double_as_longlong(w);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long ob = __shfl_xor_sync(FULL, b, o);
      const int op = __shfl_xor_sync(FULL, pmin, o);
      if (ob > b || (ob == b && op < pmin)) {
        b = ob;
        pmin = op;
      }
    }
    dt = eta * rsqrt64(__longlong_as_double(b));
  }
  *imin = pmin == 0x7fffffff ? -1 : pmin / MAXN;
  *jmin = pmin == 0x7fffffff ? -1 : pmin % MAXN;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int i = lane + 32 * q;
    if (i < n)
      for (int k = 0; k < 3; k++) S.la[i][k] = la[q][k], S.lj[i][k] = lj[q][k];
  }
  __syncwarp();
  // node forces: mass-weighted leaf forces
  FOR_COMP(r, c, n) {
    const int s = c / 3, k = c - 3 * s;
    const int b = nb > 0 ? S.bi[s] : -1;
    if (b < 0) {
      const bool node = nb == 0 || S.nd[s] == s;
      B.acc[r] = node ? S.la[s][k] : 0.0;
      B.jerk[r] = node ? S.lj[s][k] : 0.0;
    } else {
      const BinRec &bb = S.bin[b];
      const Div by_M(bb.mi + bb.mj);
      B.acc[r] = by_M(two(bb.mi, S.la[bb.li][k], bb.mj, S.la[bb.lj][k]));
      B.jerk[r] = by_M(two(bb.mi, S.lj[bb.li][k], bb.mj, S.lj[bb.lj][k]));
    }
  }
  return dt;
}

// Node states (after a step) into shared memory for the tree logic: positions
// and velocities in d, accelerations in la.
template <int NS>
__device__ __forceinline__ void publish_nodes(UnpSmem &S, int n, int lane, const Comp<NS> &B) {
  __syncwarp();
  FOR_COMP(r, c, n) {
    const int s = c / 3, k = c - 3 * s;
    if (S.nd[s] == s) {
      elem(S.d.pp[s], k) = B.pos[r];
      elem(S.d.pv[s], k) = B.vel[r];
      S.la[s][k] = B.acc[r];
    }
  }
  __syncwarp();
}

// The components of node slot i after the tree made it anew.
template <int NS>
__device__ __forceinline__ void node_set(Comp<NS> &B, int n, int lane, int i, const double x[3],
                                         const double v[3]) {
  FOR_COMP(r, c, n) {
    const int s = c / 3, k = c - 3 * s;
    if (s == i) {
      B.pos[r] = B.pp[r] = k == 0 ? x[0] : k == 1 ? x[1] : x[2];
      B.vel[r] = B.pv[r] = k == 0 ? v[0] : k == 1 ? v[1] : v[2];
      B.oacc[r] = B.ojerk[r] = 0.0;
    }
  }
}

__device__ __forceinline__ void get3(const double4_16 &v, double x[3]) {
  x[0] = v.x, x[1] = v.y, x[2] = v.z;
}
__device__ __forceinline__ void put3(double4_16 &v, const double x[3]) {
  v.x = x[0], v.y = x[1], v.z = x[2];
}

// The tree changes after a step (smallN.cc:1022-1060): binary creation from
// the pair that set the step, then the end of every segment due now.  Every
// lane evaluates the same decisions from shared data; lane 0 writes the
// shared records, the owners of the components update theirs.  Returns 0
// (no change), 1 (changed), 3 (changed, a binary made).
template <int MODE, int NS>
__device__ __forceinline__ int tree_step(UnpSmem &S, int n, int lane, Comp<NS> &B, double t, double dt_nat, int bim,
                         int bjm, const UnpParams &P) {
  const bool create = bim >= 0 && S.nb < NB && dt_nat <= P.dt_crit;
  bool due = false;
  for (int b = 0; b < S.nb; b++) due |= !(S.bin[b].tpred > t);
  if (!create && !due) return 0;
  publish_nodes(S, n, lane, B);
  int changed = 0;
  // --- creation (is_unperturbed_and_approaching, create_binary)
  if (create) {
    bool leaves = true;
    for (int b = 0; b < S.nb; b++)
      if (S.bin[b].li == bim || S.bin[b].li == bjm) leaves = false;
    const int i = bim, j = bjm;
    double xi[3], xj[3], vi[3], vj[3];
    get3(S.d.pp[i], xi), get3(S.d.pp[j], xj), get3(S.d.pv[i], vi), get3(S.d.pv[j], vj);
    double r[3], v[3];
    for (int k = 0; k < 3; k++) r[k] = xj[k] - xi[k], v[k] = vj[k] - vi[k];
    const double d2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    const double rv = r[0] * v[0] + r[1] * v[1] + r[2] * v[2];
    if (leaves && d2 <= P.r2_crit && rv <= 0.0) {
      const double mi = S.nm[i], mj = S.nm[j], M = mi + mj;
      const Div by_M(M);
      double cm[3], cmv[3];
      for (int k = 0; k < 3; k++) {
        cm[k] = by_M(two(mi, xi[k], mj, xj[k]));
        cmv[k] = by_M(two(mi, vi[k], mj, vj[k]));
      }
      // the strongest perturber (largest m^2 / d^2 from the CM; the first
      // node on ties): each lane its two node slots, then a warp argmax
      double maxp = 0.0, nnd2 = 0.0, mk = 0.0;
      int kk = 0x7fffffff;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int k2 = lane + 32 * q;
        if (k2 >= n || S.nd[k2] != k2 || k2 == i || k2 == j) continue;
        const double4_16 y = S.d.pp[k2];
        const double e0 = y.x - cm[0], e1 = y.y - cm[1], e2 = y.z - cm[2];
        const double ee = fma(e2, e2, fma(e1, e1, e0 * e0));
        const double p2 = div64(S.nm[k2] * S.nm[k2], ee);
        if (p2 > maxp) maxp = p2, nnd2 = ee, mk = S.nm[k2], kk = k2;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double op = __shfl_xor_sync(0xffffffffu, maxp, o);
        const double od = __shfl_xor_sync(0xffffffffu, nnd2, o);
        const double om = __shfl_xor_sync(0xffffffffu, mk, o);
        const int ok = __shfl_xor_sync(0xffffffffu, kk, o);
        const long long bo = __double_as_longlong(op), bm = __double_as_longlong(maxp);
        if (bo > bm || (bo == bm && ok < kk)) maxp = op, nnd2 = od, mk = om, kk = ok;
      }
      bool unp = true;
      if (maxp > 0.0) {
        const double q = div64(d2, nnd2), mm = by_M(mk);
        unp = 4.0 * mm * mm * q * q * q < P.gamma2;
      }
      double dtp, per;
      if (unp && kep_peri(M, r, v, &dtp, &per)) {
        const double tid = tidal_pot(S, n, lane, i, j, mi, mj, xi, xj, cm);
        __syncwarp();
        if (lane == 0) {
          BinRec &b = S.bin[S.nb];
          b.li = i;
          b.lj = j;
          b.full = 0;
          b.mi = mi;
          b.mj = mj;
          for (int k = 0; k < 3; k++) b.r0[k] = r[k], b.v0[k] = v[k];
          b.t0 = t;
          b.dtw = 0.0;
          b.tpred = 2.0 * (t + dtp) - t;
          b.tidal = tid;
          S.nd[j] = i;
          S.nm[i] = M;
          put3(S.d.pp[i], cm);
          put3(S.d.pv[i], cmv);
          S.nb++;
        }
        node_set(B, n, lane, i, cm, cmv);
        __syncwarp();
        changed = 3;
      }
    }
  }
  // --- segments ending now (extend_or_end_binary)
  for (int qb = 0; qb < S.nb; qb++) {
    const BinRec bb = S.bin[qb];
    if (bb.tpred > t) continue;
    const int i = bb.li, j = bb.lj;
    const double M = bb.mi + bb.mj;
    const Div by_M(M);
    const double gi = by_M(bb.mj), gj = by_M(bb.mi);
    double r[3], v[3], xi[3], xj[3], xc[3], vc[3];
    BinRec bw = bb;  // warm-started solve on a copy (every lane, same values)
    bin_rel_warm<true>(bw, t, r, v);
    get3(S.d.pp[i], xc);
    get3(S.d.pv[i], vc);
    for (int k = 0; k < 3; k++) {
      xi[k] = xc[k] - gi * r[k];
      xj[k] = xc[k] + gj * r[k];
    }
    const double tid = tidal_pot(S, n, lane, i, j, bb.mi, bb.mj, xi, xj, xc);
    if (!bb.full) {
      const double mu = by_M(bb.mi * bb.mj), v2 = dot3(v, v);
      const double fac = 1.0 - 2.0 * (tid - bb.tidal) / (mu * v2);
      if (fac > 0.0) {
        const double sf = sqrt(fac);
        for (int k = 0; k < 3; k++) v[k] *= sf;
      }
    }
    const double rn = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const double alpha = 2.0 / rn - (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) / M;
    double dtp = -1.0, period = __longlong_as_double(0x7ff0000000000000ll);
    if (P.allow_full && alpha > 0.0) {
      const double a = 1.0 / alpha;
      period = 2.0 * M_PI / sqrt(M * alpha * alpha * alpha);
      // time for any other node to come within the perturbation radius
      // (dt_perturbers): each lane its two node slots, then a warp minimum
      dtp = __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int k2 = lane + 32 * q;
        if (k2 >= n || S.nd[k2] != k2 || k2 == i) continue;
        const double rp = P.gamma_inv3 * a * cbrt(2.0 * S.nm[k2] / M);
        double yp[3], yv[3], dp[3], dvl[3], da[3];
        get3(S.d.pp[k2], yp);
        get3(S.d.pv[k2], yv);
        for (int k = 0; k < 3; k++) {
          dp[k] = yp[k] - xc[k];
          dvl[k] = yv[k] - vc[k];
          da[k] = S.la[k2][k] - S.la[i][k];
        }
        const double dr = sqrt(dp[0] * dp[0] + dp[1] * dp[1] + dp[2] * dp[2]);
        const double vr = (dvl[0] * dp[0] + dvl[1] * dp[1] + dvl[2] * dp[2]) / dr;
        const double ar = (da[0] * dp[0] + da[1] * dp[1] + da[2] * dp[2]) / dr;
        const double dd = dr - rp;
        double tr = 0.0;  // time_to_radius (smallN_unpert.cc:367-392)
        if (dd > 0.0) {
          tr = __longlong_as_double(0x7ff0000000000000ll);
          if (vr < 0.0) tr = -dd / vr;
          if (ar < 0.0) tr = fmin(tr, sqrt(-2.0 * dd / ar));
        }
        if (tr < dtp) dtp = tr;
      }
      dtp = 0.5 * warp_min(dtp);
    }
    __syncwarp();
    if (dtp >= period) {  // extend by whole periods, components frozen
      if (lane == 0) {
        BinRec &b = S.bin[qb];
        b.tpred += floor(dtp / period) * period;
        b.full = 1;
        b.tidal = tid;
        for (int k = 0; k < 3; k++) b.r0[k] = r[k], b.v0[k] = v[k];
        b.t0 = t;
        b.dtw = 0.0;
      }
      __syncwarp();
      continue;
    }
    // dissolve: the components become top-level nodes again
    double yi[3], yj[3], wi[3], wj[3];
    for (int k = 0; k < 3; k++) {
      yi[k] = xc[k] - gi * r[k];
      yj[k] = xc[k] + gj * r[k];
      wi[k] = vc[k] - gi * v[k];
      wj[k] = vc[k] + gj * v[k];
    }
    node_set(B, n, lane, i, yi, wi);
    node_set(B, n, lane, j, yj, wj);
    __syncwarp();
    if (lane == 0) {
      put3(S.d.pp[i], yi);
      put3(S.d.pv[i], wi);
      put3(S.d.pp[j], yj);
      put3(S.d.pv[j], wj);
      S.nd[j] = j;
      S.nm[i] = bb.mi;
      S.nm[j] = bb.mj;
      S.bin[qb] = S.bin[S.nb - 1];
      S.nb--;
    }
    __syncwarp();
    qb--;
    changed |= 1;
  }
  if (changed) tree_masses<MODE>(S, n, lane);
  return changed;
}

struct TreeRun {  // one system's integration
  int n, n_iter;
  double t_end, eta;
  long long max_steps;
  double *pos, *vel;  // its first body
  const double *mass;
  // results
  double t;
  long long steps;
  int status, made;
};

template <int MODE, int NS>
__device__ __noinline__ void integrate(UnpSmem &S, int lane, TreeRun &run, const UnpParams &P) {
  const int n = run.n, n_iter = run.n_iter;
  const double t_end = run.t_end, eta = run.eta;
  const long long max_steps = run.max_steps;
  double *pos = run.pos, *vel = run.vel;
  const double *mass = run.mass;
  // lane & 7: one of the corrector's coefficients, a cubic in tau, a quarter
  // included: acc = c0 oa + c1 pa + theta (c2 oj + c3 pj),
  // jerk = (c4 oa + c5 pa) / theta + c6 oj + c7 pj (smallN.cc:487-510).  Only
  // the state of the next evaluation depends on it, not the step's result.
  double q0, q1, q2, q3;
  {
    const int l = lane & 7;
    q0 = l < 2 ? 0.5 : l == 2 ? 0.25 : l == 4 ? -0.75 : l == 5 ? 0.75 : -0.25;
    q1 = l == 0 ? -0.75 : l == 1 ? 0.75 : l == 2 || l == 3 ? -0.25 : l == 6 ? -0.5 : l == 7 ? 0.5 : 0.0;
    q2 = l < 2 ? 0.0 : l == 2 ? -0.25 : l == 3 ? 0.25 : l == 5 ? -0.75 : 0.75;
    q3 = l == 0 || l == 2 || l == 3 ? 0.25 : l == 1 ? -0.25 : 0.0;
  }
  Comp<NS> B;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NS; r++) {
    const int c = lane + 32 * r;
    B.pos[r] = B.pp[r] = c < 3 * n ? pos[c] : 0.0;
    B.vel[r] = B.pv[r] = c < 3 * n ? vel[c] : 0.0;
    B.acc[r] = B.jerk[r] = B.oacc[r] = B.ojerk[r] = 0.0;
  }
  for (int i = lane; i < n; i += 32) {
    const double m = mass[i];
    S.nd[i] = i;
    S.nm[i] = m;
    S.d.pp[i].w = m;
    if (MODE == MODE_SPLIT) S.f.hi[i].w = __double2float_rn(m);
  }
  if (lane == 0) S.nb = 0;
  tree_masses<MODE>(S, n, lane);
  int bim, bjm, made = 0;
  double t = 0.0;
  double dt = tree_forces<MODE, NS>(S, n, lane, B, t, eta, &bim, &bjm);
  long long nsteps = 0;
  int st = 0;
  while (t < t_end) {
    if (nsteps >= max_steps) {
      st = 1;  // step budget exhausted
      break;
    }
    double lim = __longlong_as_double(0x7ff0000000000000ll);
    for (int b = 0; b < S.nb; b++) lim = fmin(lim, S.bin[b].tpred - t);
    int nit = n_iter;
    if (dt >= lim) {
      dt = lim;
      nit = 0;
    }
    // predict_loworder (hdyn.h:192-201: with the stored old force)
    {
      const double h = P.on ? dt : (t + dt) - t;  // without the tree, as batch_exact_kernel's
      const double h3 = g6_div_const(h, 3.0, 1.0 / 3.0), h2 = h * 0.5;
      FOR_COMP(r, c, n) {
        const double oj = B.ojerk[r], oa = B.oacc[r];
        B.pp[r] = fma(fma(fma(oj, h3, oa), h2, B.vel[r]), h, B.pos[r]);
        B.pv[r] = fma(fma(oj, h2, oa), h, B.vel[r]);
        B.oacc[r] = B.acc[r];
        B.ojerk[r] = B.jerk[r];
      }
    }
    double new_dt = dt, end_dt = dt;
    for (int it = 0; it <= nit; it++) {
      const double prev = new_dt;
      end_dt = tree_forces<MODE, NS>(S, n, lane, B, t + new_dt, eta, &bim, &bjm);
      double iprev = 0.0;
      if (it < nit) {
        const Div by_prev(prev);
        iprev = by_prev.y;
        new_dt = 0.5 * (dt + end_dt);
        new_dt = dt + 0.5 * (end_dt - dt) * by_prev(new_dt);
        if (new_dt >= lim) {
          new_dt = lim;
          nit = 0;
        }
      }
      if (new_dt != prev) {  // correct_acc_and_jerk(new_dt, prev)
        const double theta = 0.5 * prev, itheta = 2.0 * iprev;
        const double tau = (new_dt - theta) * itheta;
        double cc = fma(fma(fma(q3, tau, q2), tau, q1), tau, q0);
        const int l = lane & 7;
        cc *= (l & 6) == 2 ? theta : (l & 6) == 4 ? itheta : 1.0;
        double k[8];
#pragma unroll
        for (int q = 0; q < 8; q++) k[q] = __shfl_sync(0xffffffffu, cc, q);
        FOR_COMP(r, c, n) {
          const double pa = B.acc[r], pj = B.jerk[r], oa = B.oacc[r], oj = B.ojerk[r];
          B.acc[r] = fma(k[3], pj, fma(k[2], oj, fma(k[1], pa, k[0] * oa)));
          B.jerk[r] = fma(k[7], pj, fma(k[6], oj, fma(k[5], pa, k[4] * oa)));
        }
      }
      // correct_pos_and_vel(new_dt)
      const double nd2 = new_dt * new_dt;
      if (it < nit) {  // only the next evaluation's state: two FP64 instructions fewer each
        const double hh = 0.5 * new_dt, h12 = nd2 * (1.0 / 12.0);
        FOR_COMP(r, c, n) {
          B.pv[r] = fma(-h12, B.jerk[r] - B.ojerk[r], fma(hh, B.acc[r] + B.oacc[r], B.vel[r]));
          B.pp[r] = fma(-h12, B.acc[r] - B.oacc[r], fma(hh, B.pv[r] + B.vel[r], B.pos[r]));
        }
      } else {
        FOR_COMP(r, c, n) {
          B.pv[r] = B.vel[r] + new_dt * (B.acc[r] + B.oacc[r]) * 0.5 -
                    nd2 * (B.jerk[r] - B.ojerk[r]) * (1.0 / 12.0);
          B.pp[r] = B.pos[r] + new_dt * (B.pv[r] + B.vel[r]) * 0.5 -
                    nd2 * (B.acc[r] - B.oacc[r]) * (1.0 / 12.0);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < NS; r++) B.pos[r] = B.pp[r], B.vel[r] = B.pv[r];
    dt = end_dt;
    t = t + new_dt;
    nsteps++;
    if (P.on) {
      const int tc = tree_step<MODE, NS>(S, n, lane, B, t, dt, bim, bjm, P);
      if (tc) {
        if (tc & 2) made++;
        dt = tree_forces<MODE, NS>(S, n, lane, B, t, eta, &bim, &bjm);
      }
    }
  }
  // resolve the binaries left at the end into their components
  __syncwarp();
  if (lane < S.nb) {
    double r[3], v[3];
    bin_rel(S.bin[lane], t, r, v);
    for (int k = 0; k < 3; k++) S.kr[lane][k] = r[k], S.kr[lane][3 + k] = v[k];
  }
  __syncwarp();
  FOR_COMP(r, c, n) {
    const int i = c / 3, k = c - 3 * i;
    const int b = S.bi[i];
    if (S.nd[i] == i && b < 0) {
      pos[c] = B.pos[r];
      vel[c] = B.vel[r];
    } else if (S.nd[i] == i) {
      const BinRec &bb = S.bin[b];
      const Div by_M(bb.mi + bb.mj);
      const double gi = by_M(bb.mj), gj = by_M(bb.mi), x = S.kr[b][k], v = S.kr[b][3 + k];
      pos[3 * bb.li + k] = B.pos[r] - gi * x;
      vel[3 * bb.li + k] = B.vel[r] - gi * v;
      pos[3 * bb.lj + k] = B.pos[r] + gj * x;
      vel[3 * bb.lj + k] = B.vel[r] + gj * v;
    }
  }
  run.t = t;
  run.steps = nsteps;
  run.status = st;
  run.made = made;
}
#undef FOR_COMP

template <int MODE>
__global__ void batch_tree_kernel(const int *__restrict__ order, const int *__restrict__ off,
                                  const double *__restrict__ t_end_s,
                                  const double *__restrict__ mass, double *pos, double *vel,
                                  double eta, int n_iter, long long max_steps, int *queue,
                                  double *t_out, long long *steps_out,
                                  unsigned long long *wall_ns, int *status, int *nbin_out,
                                  UnpParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  UnpSmem &S = reinterpret_cast<UnpSmem *>(smem_raw)[w];
  const int nsys = queue[1];  // written by the host before the launch
  for (int q = first_system(w); q < nsys; q = next_system(queue, lane)) {
    const int s = order[q];
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    const int base = off[s];
    const int n = off[s + 1] - base;
    if (n < 2 || n > MAXN) {
      if (lane == 0) {
        status[s] = 2;  // unsupported size (host also checks)
        steps_out[s] = 0;
        t_out[s] = 0.0;
        if (nbin_out) nbin_out[s] = 0;
      }
      continue;
    }
    TreeRun run;
    run.n = n;
    run.n_iter = n_iter;
    run.t_end = t_end_s[s];
    run.eta = eta;
    run.max_steps = max_steps;
    run.pos = pos + 3 * (size_t)base;
    run.vel = vel + 3 * (size_t)base;
    run.mass = mass + base;
    switch ((3 * n + 31) / 32) {
      case 1: integrate<MODE, 1>(S, lane, run, P); break;  // 2 to 10 bodies
      case 2: integrate<MODE, 2>(S, lane, run, P); break;  // to 21
      case 3: integrate<MODE, 3>(S, lane, run, P); break;  // to 32
      default: integrate<MODE, 6>(S, lane, run, P); break;
    }
    if (lane == 0) {
      unsigned long long t1;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      t_out[s] = run.t;
      steps_out[s] = run.steps;
      wall_ns[s] = t1 - t0;
      status[s] = run.status;
      if (nbin_out) nbin_out[s] = run.made;
    }
    __syncwarp();
  }
}


__global__ void queue_reset(int *queue) { queue[0] = 0; }

}  // namespace

extern "C" int g6k_batch_max_n(void) { return MAXN; }

// The CTAs of a launch: as asked for, but no more than are resident at once.
// first_system gives every warp of the grid a system, the largest first, and
// a CTA that must wait for another one to end would hold its own back until
// the queue has run out (three CTAs of four warps per SM asked for where two
// fit: 400 equal systems of 24 bodies took 375 us for 207 at two, 4096 uneven
// ones 11.0 ms for 9.6).
template <typename K>
static int resident_ctas(K kern, int threads, size_t smem, int ctas) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess ||
      per_sm < 1)
    return ctas;
  const int most = per_sm * g6k_sm_count();
  return ctas < most ? ctas : most;
}

// The fast and split modes: dynamic shared memory for warps_per_cta warps.
static int launch_tree(int mode, const int *order, const int *off, const double *t_end,
                       const double *mass, double *pos, double *vel, double eta, int n_iter,
                       long long max_steps, int warps_per_cta, int ctas, int *queue,
                       double *t_out, long long *steps_out, unsigned long long *wall_ns,
                       int *status, int *nbin_out, const UnpParams &P, cudaStream_t st) {
  const size_t sm = sizeof(UnpSmem) * (size_t)warps_per_cta;
  const int most = (int)(sizeof(UnpSmem) * WARPS_MAX);
  auto kern = mode == MODE_SPLIT ? batch_tree_kernel<MODE_SPLIT> : batch_tree_kernel<MODE_FAST>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most) !=
      cudaSuccess)
    return -3;
  ctas = resident_ctas(kern, 32 * warps_per_cta, sm, ctas);
  kern<<<ctas, 32 * warps_per_cta, sm, st>>>(order, off, t_end, mass, pos, vel, eta, n_iter,
                                             max_steps, queue, t_out, steps_out, wall_ns, status,
                                             nbin_out, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// One persistent launch: grid = ctas_per_sm * SMs, warps_per_cta warps each.
// Resets the queue counter first (same stream), so the pair can be captured
// in a CUDA graph and replayed.  queue[0] is the counter, queue[1] the number
// of systems, which the host writes before each replay (a graph then serves
// every batch size).
extern "C" int g6k_batch_launch(const int *order, const int *off, const double *t_end,
                                const double *mass, double *pos, double *vel, double eta,
                                int n_iter, long long max_steps, int exact, int warps_per_cta,
                                int ctas, int *queue, double *t_out, long long *steps_out,
                                unsigned long long *wall_ns, int *status, cudaStream_t st) {
  if (warps_per_cta < 1 || warps_per_cta > WARPS_MAX || ctas < 1) return -2;
  if (exact < MODE_FAST || exact > MODE_SPLIT) return -2;
  queue_reset<<<1, 1, 0, st>>>(queue);
  if (exact != MODE_EXACT) {
    UnpParams P = {};
    return launch_tree(exact, order, off, t_end, mass, pos, vel, eta, n_iter, max_steps,
                       warps_per_cta, ctas, queue, t_out, steps_out, wall_ns, status, nullptr, P,
                       st);
  }
  ctas = resident_ctas(batch_exact_kernel, 32 * warps_per_cta, 0, ctas);
  batch_exact_kernel<<<ctas, 32 * warps_per_cta, 0, st>>>(order, off, t_end, mass, pos, vel, eta,
                                                          n_iter, max_steps, queue, t_out,
                                                          steps_out, wall_ns, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// The fast or split mode with smallN's unperturbed binaries: dt_crit,
// r2_crit, gamma and allow_full as smallN's set_dt_crit, set_r2_crit,
// set_gamma, set_allow_full_unperturbed; nbin_out[s] counts the binaries made
// in system s.
extern "C" int g6k_batch_launch_unp(const int *order, const int *off,
                                    const double *t_end, const double *mass, double *pos,
                                    double *vel, double eta, int n_iter, long long max_steps,
                                    int mode, int warps_per_cta, int ctas, double dt_crit,
                                    double r2_crit, double gamma, int allow_full, int *queue,
                                    double *t_out, long long *steps_out,
                                    unsigned long long *wall_ns, int *status, int *nbin_out,
                                    cudaStream_t st) {
  if (warps_per_cta < 1 || warps_per_cta > 4 || ctas < 1) return -2;
  if (mode != MODE_FAST && mode != MODE_SPLIT) return -2;
  UnpParams P;
  P.dt_crit = dt_crit;
  P.r2_crit = r2_crit;
  P.gamma2 = gamma * gamma;
  P.gamma_inv3 = pow(fmax(P.gamma2, 1e-120), -1.0 / 6.0);
  P.allow_full = allow_full;
  P.on = 1;
  queue_reset<<<1, 1, 0, st>>>(queue);
  return launch_tree(mode, order, off, t_end, mass, pos, vel, eta, n_iter, max_steps,
                     warps_per_cta, ctas, queue, t_out, steps_out, wall_ns, status, nbin_out, P,
                     st);
}
