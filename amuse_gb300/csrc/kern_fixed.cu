// kern_fixed.cu -- fixed-step Hermite integration and its adjoint.
//
// Forward step (the hermite code's scheme, src/amuse_hermite/interface.cc:
// predict_step :266-281, correct_step :536-552), state (x, v, a, j), step h:
//   xp = x + v h + a h^2/2 + j h^3/6,   vp = v + a h + j h^2/2
//   (a1, j1) = F(xp, vp; m)              (the library's force kernel)
//   v' = v + (a + a1) h/2 + (j - j1) h^2/12
//   x' = x + (v + v') h/2 + (a - a1) h^2/12,   (a, j) <- (a1, j1)
// F is ph4's pair force: a_k = sum_j m_j r s^-3/2, j_k = sum_j m_j (v s^-3/2
// - 3 (r.v) r s^-5/2), r = x_j - x_k, v = v_j - v_k, s = r^2 + eps^2.
//
// Adjoint of one step, given the adjoints (Lx', Lv', La', Lj') of its
// outputs (exact-arithmetic derivative of the map above):
//   Lvt = Lv' + Lx' h/2
//   La1 = La' - Lx' h^2/12 + Lvt h/2,   Lj1 = Lj' - Lvt h^2/12
//   (gxp, gvp, gm) = VJP_F(xp, vp, m; La1, Lj1)
//   Lx = Lx' + gxp
//   Lv = Lx' h/2 + Lvt + gxp h + gvp
//   La = Lx' h^2/12 + Lvt h/2 + gxp h^2/2 + gvp h
//   Lj = Lvt h^2/12 + gxp h^3/6 + gvp h^2/2,     Lm += gm
// Force VJP for body k, from its side of each pair (r = x_j - x_k, ...):
//   c = m_k Lam_j - m_j Lam_k  (Lam = (La1, Lj1)),  lam = c_a, mu = c_j
//   gx_k += lam s^-3/2 - 3 (r.lam) r s^-5/2
//           - 3 [(mu.v) r + (mu.r) v + (r.v) mu] s^-5/2 + 15 (r.v)(mu.r) r s^-7/2
//   gv_k += mu s^-3/2 - 3 (r.mu) r s^-5/2
//   gm_k -= La1_j . r s^-3/2 + Lj1_j . (v s^-3/2 - 3 (r.v) r s^-5/2)
// (the pair Jacobians are even in (r, v), which gives the c combination).
// With the hermite code's jerk form (r.v divided by the unsoftened q = r^2,
// src/amuse_hermite/interface.cc:440-449,486) the jerk terms become
//   gx_k += -3 (mu.v) r s^-5/2 - 3 [(mu.r) v + (r.v) mu] q^-1 s^-3/2
//           + 3 (r.v)(mu.r) r (2 q^-2 s^-3/2 + 3 q^-1 s^-5/2)
//   gv_k += mu s^-3/2 - 3 (r.mu) r q^-1 s^-3/2
//   gm_k -= ... + Lj1_j . (v s^-3/2 - 3 (r.v) r q^-1 s^-3/2)
// (q = s recovers the softened form).
// The VJP runs in split precision (double-single r, FP32 pair math, per-tile
// FP32 partials folded into FP64 totals) or in FP64.
#include "pdl.cuh"
#include <cuda_runtime.h>

#include "f32x2.cuh"
#include "fp64_approx.cuh"
#include "g6_dev.h"

struct __align__(32) G6D4 {
  double x, y, z, w;
};

namespace {

constexpr int VT = 32;  // FP64 VJP threads per CTA
constexpr int VTILE = 128;

// One force record from a body's state (s >= n: padding, massless and far).
__device__ __forceinline__ void store_record(int s, int n, const double x[3], const double v[3],
                                             double m, int prec, void *jp_split, void *jp_f64) {
  double xp[3], vp[3];
  const double mm = s < n ? m : 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    xp[k] = s < n ? x[k] : 1.0e18;
    vp[k] = s < n ? v[k] : 0.0;
  }
  if (prec == G6_PREC_FP64) {
    G6D4 *r = reinterpret_cast<G6D4 *>(jp_f64) + 2 * (size_t)s;
    r[0] = G6D4{xp[0], xp[1], xp[2], mm};
    r[1] = G6D4{vp[0], vp[1], vp[2], 0.0};
  } else {
    float h[3], l[3];
    for (int k = 0; k < 3; k++) {
      h[k] = __double2float_rn(xp[k]);
      l[k] = __double2float_rn(xp[k] - (double)h[k]);
    }
    const float mh = __double2float_rn(mm);
    g6_split_store(jp_split, s, h[0], h[1], h[2], mh, __double2float_rn(mm - (double)mh), l[0],
                   l[1], l[2], __double2float_rn(vp[0]), __double2float_rn(vp[1]),
                   __double2float_rn(vp[2]));
  }
}

__global__ void records_kernel(int n, int n_pad, const double *__restrict__ x,
                               const double *__restrict__ v, const double *__restrict__ m,
                               int prec, void *jp_split, void *jp_f64) {
  pdl_wait();
  pdl_trigger();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_pad) return;
  double xs[3] = {0, 0, 0}, vs[3] = {0, 0, 0};
  if (s < n)
    for (int k = 0; k < 3; k++) xs[k] = x[3 * s + k], vs[k] = v[3 * s + k];
  store_record(s, n, xs, vs, s < n ? m[s] : 0.0, prec, jp_split, jp_f64);
}

// What lies between two force evaluations of a fixed-step run, a body per
// thread: the corrector of the step that ends (CORRECT) and the prediction
// and force records of the one that begins (PREDICT).  Three launches before,
// 4 us each at n = 8192; one warp per CTA, since the ~60 FP64 instructions of a
// warp take 64 cycles of its scheduler each.
template <bool CORRECT, bool PREDICT>
__global__ void __launch_bounds__(32) advance_kernel(int n, int n_pad, double h, double *x,
                                                     double *v, double *a, double *j,
                                                     const double *__restrict__ a1,
                                                     const double *__restrict__ j1,
                                                     const double *__restrict__ m, double *xp,
                                                     double *vp, int prec, void *jp_split,
                                                     void *jp_f64) {
  pdl_wait();
  pdl_trigger();
  const int s = blockIdx.x * 32 + threadIdx.x;
  if (s >= n_pad) return;
  double xs[3] = {0, 0, 0}, vs[3] = {0, 0, 0};
  if (s < n) {
    const double hh = 0.5 * h, h2 = h * h / 2, h12 = h * h / 12, h6 = h * h * h / 6;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int e = 3 * s + k;
      double X = x[e], V = v[e], A = a[e], J = j[e];
      if (CORRECT) {  // hermite correct_step
        const double an = a1[e], jn = j1[e];
        const double vn = V + (A + an) * hh + (J - jn) * h12;
        X = X + (V + vn) * hh + (A - an) * h12;
        V = vn;
        A = an;
        J = jn;
        x[e] = X;
        v[e] = V;
        a[e] = A;
        j[e] = J;
      }
      if (PREDICT) {  // predict_step: pos += vel*dt + acc*dt*dt/2 + jerk*dt*dt*dt/6
        xs[k] = X + (V * h + A * h2 + J * h6);
        vs[k] = V + (A * h + J * h2);
        xp[e] = xs[k];
        vp[e] = vs[k];
      }
    }
  }
  if (PREDICT) store_record(s, n, xs, vs, s < n ? m[s] : 0.0, prec, jp_split, jp_f64);
}

// ---- force VJP, FP64 ----
struct VRecD {
  double x[3], v[3], m, la[3], lj[3];
};

// One body k per thread, one warp per CTA (an FP64 instruction takes 64 cycles
// of the warp's scheduler: warps spread over the SMs), j in shared-memory
// tiles of VTD, the j range split over gridDim.y CTA rows.  Of n = 128 .. 1024
// bodies, four-warp CTAs with IEEE divisions and a square root per pair took 7
// to 15 times as long (8 steps with their adjoint, n = 1024: 39.9 -> 4.9 ms
// with the FP64 force's part).
constexpr int VTD = 32;
template <bool HJ>
__global__ void __launch_bounds__(VT) vjp_f64_kernel(int n, double eps2,
                                                     const double *__restrict__ x,
                                                     const double *__restrict__ v,
                                                     const double *__restrict__ m,
                                                     const double *__restrict__ la1,
                                                     const double *__restrict__ lj1, int jsplit,
                                                     double *part /* [nsplit][n][7] */) {
  __shared__ VRecD td[VTD];
  pdl_wait();
  pdl_trigger();
  eps2 += 1.0 / 4503599627370496.0;  // the force kernel's softening (+2^-52, as ph4)
  const int k = blockIdx.x * VT + threadIdx.x;
  const bool valid = k < n;
  const int kk = valid ? k : 0;
  const int j0 = blockIdx.y * jsplit;
  const int j1 = min(n, j0 + jsplit);
  const double xk[3] = {x[3 * kk], x[3 * kk + 1], x[3 * kk + 2]};
  const double vk[3] = {v[3 * kk], v[3 * kk + 1], v[3 * kk + 2]};
  const double mk = m[kk];
  const double lak[3] = {la1[3 * kk], la1[3 * kk + 1], la1[3 * kk + 2]};
  const double ljk[3] = {lj1[3 * kk], lj1[3 * kk + 1], lj1[3 * kk + 2]};
  // gx[3], gv[3], gm: the sums of up to four tiles and the totals of those
  // before them (one sum over all j of a split, 5461 at 16384 bodies, had ten
  // times the rounding error)
  double acc[7] = {0, 0, 0, 0, 0, 0, 0}, tot[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int t0 = j0; t0 < j1; t0 += VTD) {
    if (t0 != j0 && (t0 - j0) % (4 * VTD) == 0)
      for (int c = 0; c < 7; c++) tot[c] += acc[c], acc[c] = 0;
    __syncwarp();
    const int jj = min(t0 + (int)threadIdx.x, n - 1);
    VRecD &w = td[threadIdx.x];
    for (int c = 0; c < 3; c++) {
      w.x[c] = x[3 * jj + c];
      w.v[c] = v[3 * jj + c];
      w.la[c] = la1[3 * jj + c];
      w.lj[c] = lj1[3 * jj + c];
    }
    w.m = m[jj];
    __syncwarp();
    const int nq = min(VTD, j1 - t0);
    for (int q = 0; q < nq; q++) {
      const VRecD &r = td[q];
      if (t0 + q == k) continue;
      double R[3], V[3], lam[3], mu[3];
      for (int c = 0; c < 3; c++) {
        R[c] = r.x[c] - xk[c];
        V[c] = r.v[c] - vk[c];
        lam[c] = mk * r.la[c] - r.m * lak[c];
        mu[c] = mk * r.lj[c] - r.m * ljk[c];
      }
      const double r2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2];
      const double s1 = fp64::rsqrt64(r2 + eps2), si = s1 * s1;
      const double s3 = s1 * si, s5 = s3 * si;
      // lam.r + mu.v and the other dot products
      const double rlvm = R[0] * lam[0] + R[1] * lam[1] + R[2] * lam[2] + V[0] * mu[0] +
                          V[1] * mu[1] + V[2] * mu[2];
      const double rm = R[0] * mu[0] + R[1] * mu[1] + R[2] * mu[2];
      const double rv = R[0] * V[0] + R[1] * V[1] + R[2] * V[2];
      // q3 = -3 q^-1 s^-3/2 (-3 s^-5/2 in the softened form); the last term of
      // cr is 15 s^-7/2 resp. 3 (2 q^-2 s^-3/2 + 3 q^-1 s^-5/2) times rv rm
      double q3, d;
      if (HJ) {
        const double qi = fp64::rcp64(r2);
        q3 = -3.0 * (qi * s3);
        d = 2.0 * qi + 3.0 * si;
      } else {
        q3 = -3.0 * s5;
        d = 5.0 * si;
      }
      const double w5 = q3 * rm, y = q3 * rv;
      const double cr = -3.0 * (rlvm * s5) - (y * rm) * d;
      for (int c = 0; c < 3; c++) {
        acc[c] += lam[c] * s3 + cr * R[c] + w5 * V[c] + y * mu[c];
        acc[3 + c] += mu[c] * s3 + w5 * R[c];
      }
      const double g = r.la[0] * R[0] + r.la[1] * R[1] + r.la[2] * R[2] + r.lj[0] * V[0] +
                       r.lj[1] * V[1] + r.lj[2] * V[2];
      const double lr = r.lj[0] * R[0] + r.lj[1] * R[1] + r.lj[2] * R[2];
      acc[6] -= g * s3 + y * lr;
    }
  }
  if (valid) {
    double *p = part + ((size_t)blockIdx.y * n + k) * 7;
    for (int c = 0; c < 7; c++) p[c] = tot[c] + acc[c];
  }
}

// ---- split-precision force VJP, packed f32x2, register-blocked ----
// Records come in pairs of consecutive bodies, every field a float2 (body
// 2p, body 2p+1), 128 B per pair: xh yh zh m xl yl zl vx vy vz la0 la1 la2
// lj0 lj1 lj2.  Each add/sub/mul/fma.rn.f32x2 evaluates one body k against
// two bodies j; each thread owns VIPT bodies k (values duplicated into both
// halves), so every shared-memory record pair serves 2 x VIPT pairs.
// Padding records (zero mass and cotangents, far away) contribute exactly
// zero.  The self pair also contributes exactly zero: r = v = 0 and
// lam = m_k La_j - m_j La_k cancels bit for bit (two rounded products, no
// contraction); with the hermite jerk form the 1/r^2 factor is set to 0
// there.
constexpr int VF = 16;  // fields per body
struct __align__(16) VJPair {
  float2 f[VF];
};
constexpr int VIPT = 2;
constexpr int VT2 = 128;

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void store_vjp_record(int s, int n, const double x[3],
                                                 const double v[3], double m, const double la[3],
                                                 const double lj[3], VJPair *rec) {
  float f[VF];
  if (s < n) {
    for (int k = 0; k < 3; k++) {
      f[k] = __double2float_rn(x[k]);
      f[4 + k] = __double2float_rn(x[k] - (double)f[k]);
      f[7 + k] = __double2float_rn(v[k]);
      f[10 + k] = __double2float_rn(la[k]);
      f[13 + k] = __double2float_rn(lj[k]);
    }
    f[3] = __double2float_rn(m);
  } else {
    for (int k = 0; k < VF; k++) f[k] = 0.f;
    f[0] = f[1] = f[2] = 1.0e18f;
  }
  float *dst = reinterpret_cast<float *>(rec + (s >> 1)) + (s & 1);
  for (int k = 0; k < VF; k++) dst[2 * k] = f[k];
}

__global__ void vjp_records_kernel(int n, int n_pad, const double *__restrict__ x,
                                   const double *__restrict__ v, const double *__restrict__ m,
                                   const double *__restrict__ la1, const double *__restrict__ lj1,
                                   VJPair *rec) {
  pdl_wait();
  pdl_trigger();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_pad) return;
  const int e = 3 * (s < n ? s : 0);
  store_vjp_record(s, n, x + e, v + e, m[s < n ? s : 0], la1 + e, lj1 + e, rec);
}

// Between two force VJPs of the adjoint, a body per thread.  POST: the step
// whose VJP (gxp, gvp, gm) is done, the predictor's pull-back; lm (if not
// NULL) accumulates the mass cotangent.  PRE: the step before it, the
// corrector's transpose: step-output adjoints in (lx, lv, la, lj) become the
// corrector's input-adjoint contributions (in place), and the adjoints of the
// force outputs go into the VJP's records (split) or la1, lj1 (FP64).
template <bool POST, bool PRE>
__global__ void __launch_bounds__(32) adjoint_kernel(
    int n, int n_pad, double h, double *lx, double *lv, double *la, double *lj,
    const double *__restrict__ gxp, const double *__restrict__ gvp, double *lm,
    const double *__restrict__ gm, const double *__restrict__ x, const double *__restrict__ v,
    const double *__restrict__ m, double *la1, double *lj1, VJPair *rec) {
  pdl_wait();
  pdl_trigger();
  const int s = blockIdx.x * 32 + threadIdx.x;
  if (s >= n_pad) return;
  double ca[3] = {0, 0, 0}, cj[3] = {0, 0, 0};
  if (s < n) {
    const double hh = 0.5 * h, h2 = h * h / 2, h12 = h * h / 12, h6 = h * h * h / 6;
    if (POST && lm) lm[s] += gm[s];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int e = 3 * s + k;
      double Lx = lx[e], Lv = lv[e], La = la[e], Lj = lj[e];
      if (POST) {
        const double gx = gxp[e], gv = gvp[e];
        Lx += gx;
        Lv += gx * h + gv;
        La += gx * h2 + gv * h;
        Lj += gx * h6 + gv * h2;
      }
      if (PRE) {
        const double Lvt = Lv + Lx * hh;
        ca[k] = La - Lx * h12 + Lvt * hh;
        cj[k] = Lj - Lvt * h12;
        if (!rec) {
          la1[e] = ca[k];
          lj1[e] = cj[k];
        }
        Lv = Lx * hh + Lvt;
        La = Lx * h12 + Lvt * hh;
        Lj = Lvt * h12;
      }
      lx[e] = Lx;
      lv[e] = Lv;
      la[e] = La;
      lj[e] = Lj;
    }
  }
  if (PRE && rec) {
    const int e = 3 * (s < n ? s : 0);
    store_vjp_record(s, n, x + e, v + e, m[s < n ? s : 0], ca, cj, rec);
  }
}

template <bool HJ>
__global__ void __launch_bounds__(VT2) vjp_split_kernel(int n, float eps2, const VJPair *__restrict__ rec,
                                                        int jsplit, int n_pad,
                                                        double *part /* [nsplit][n][7] */) {
  __shared__ VJPair tile[VTILE / 2];
  pdl_wait();
  pdl_trigger();
  f2x xh[VIPT][3], xl[VIPT][3], vk[VIPT][3], mk[VIPT], lak[VIPT][3], ljk[VIPT][3];
  int kk[VIPT];
#pragma unroll
  for (int q = 0; q < VIPT; q++) {
    kk[q] = blockIdx.x * (VT2 * VIPT) + q * VT2 + threadIdx.x;
    const int k = kk[q] < n_pad ? kk[q] : 0;
    const float *src = reinterpret_cast<const float *>(rec + (k >> 1)) + (k & 1);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      xh[q][c] = f2_dup(src[2 * c]);
      xl[q][c] = f2_dup(src[2 * (4 + c)]);
      vk[q][c] = f2_dup(src[2 * (7 + c)]);
      lak[q][c] = f2_dup(src[2 * (10 + c)]);
      ljk[q][c] = f2_dup(src[2 * (13 + c)]);
    }
    mk[q] = f2_dup(src[2 * 3]);
  }
  double tot[VIPT][7];
#pragma unroll
  for (int q = 0; q < VIPT; q++)
#pragma unroll
    for (int c = 0; c < 7; c++) tot[q][c] = 0.0;
  const f2x e2 = f2_dup(eps2);
  const f2x m3 = f2_dup(-3.0f);
  const int j0 = blockIdx.y * jsplit;
  const int j1 = min(n_pad, j0 + jsplit);
  for (int t0 = j0; t0 < j1; t0 += VTILE) {
    __syncthreads();
    for (int q = threadIdx.x; q < VTILE / 2; q += VT2) tile[q] = rec[t0 / 2 + q];
    __syncthreads();
    f2x g[VIPT][7];
#pragma unroll
    for (int q = 0; q < VIPT; q++)
#pragma unroll
      for (int c = 0; c < 7; c++) g[q][c] = 0ull;
#pragma unroll 2
    for (int jj = 0; jj < VTILE / 2; jj++) {
      const VJPair &r = tile[jj];
      f2x xhj[3], xlj[3], vj[3], laj[3], ljj[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        xhj[c] = f2_of(r.f[c]);
        xlj[c] = f2_of(r.f[4 + c]);
        vj[c] = f2_of(r.f[7 + c]);
        laj[c] = f2_of(r.f[10 + c]);
        ljj[c] = f2_of(r.f[13 + c]);
      }
      const f2x mj = f2_of(r.f[3]);
#pragma unroll
      for (int q = 0; q < VIPT; q++) {
        f2x R[3], V[3], lam[3], mu[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          R[c] = f2_add(f2_sub(xhj[c], xh[q][c]), f2_sub(xlj[c], xl[q][c]));
          V[c] = f2_sub(vj[c], vk[q][c]);
          lam[c] = f2_sub(f2_mul(mk[q], laj[c]), f2_mul(mj, lak[q][c]));
          mu[c] = f2_sub(f2_mul(mk[q], ljj[c]), f2_mul(mj, ljk[q][c]));
        }
        const f2x s = f2_fma(R[2], R[2], f2_fma(R[1], R[1], f2_fma(R[0], R[0], e2)));
        float sa, sb;
        f2_unpack(s, sa, sb);
        const f2x s1 = f2_pack(rsqrt_approx(sa), rsqrt_approx(sb));
        const f2x si = f2_mul(s1, s1);
        const f2x s3 = f2_mul(s1, si), s5 = f2_mul(s3, si);
        const f2x rl = f2_fma(R[2], lam[2], f2_fma(R[1], lam[1], f2_mul(R[0], lam[0])));
        const f2x rm = f2_fma(R[2], mu[2], f2_fma(R[1], mu[1], f2_mul(R[0], mu[0])));
        const f2x vm = f2_fma(V[2], mu[2], f2_fma(V[1], mu[1], f2_mul(V[0], mu[0])));
        const f2x rv = f2_fma(R[2], V[2], f2_fma(R[1], V[1], f2_mul(R[0], V[0])));
        f2x qs, c7;
        if (HJ) {
          const f2x r2u = f2_fma(R[2], R[2], f2_fma(R[1], R[1], f2_mul(R[0], R[0])));
          float ua, ub;
          f2_unpack(r2u, ua, ub);
          const f2x qi = f2_pack(ua > 0.f ? rcp_approx(ua) : 0.f, ub > 0.f ? rcp_approx(ub) : 0.f);
          qs = f2_mul(qi, s3);
          c7 = f2_mul(qi, f2_fma(f2_dup(6.0f), qs, f2_mul(f2_dup(9.0f), s5)));
        } else {
          qs = s5;
          c7 = f2_mul(f2_dup(15.0f), f2_mul(s5, si));
        }
        const f2x q3 = f2_mul(m3, qs);
        const f2x cr = f2_fma(f2_mul(rv, rm), c7, f2_mul(m3, f2_mul(f2_add(rl, vm), s5)));
        const f2x w = f2_mul(q3, rm);
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const f2x u = f2_fma(rm, V[c], f2_mul(rv, mu[c]));
          g[q][c] = f2_fma(q3, u, f2_fma(cr, R[c], f2_fma(lam[c], s3, g[q][c])));
          g[q][3 + c] = f2_fma(w, R[c], f2_fma(mu[c], s3, g[q][3 + c]));
        }
        const f2x ga = f2_fma(laj[2], R[2], f2_fma(laj[1], R[1], f2_mul(laj[0], R[0])));
        const f2x lv = f2_fma(ljj[2], V[2], f2_fma(ljj[1], V[1], f2_mul(ljj[0], V[0])));
        const f2x lr = f2_fma(ljj[2], R[2], f2_fma(ljj[1], R[1], f2_mul(ljj[0], R[0])));
        g[q][6] = f2_sub(g[q][6], f2_fma(f2_add(ga, lv), s3, f2_mul(f2_mul(q3, rv), lr)));
      }
    }
#pragma unroll
    for (int q = 0; q < VIPT; q++)
#pragma unroll
      for (int c = 0; c < 7; c++) {
        float lo, hi;
        f2_unpack(g[q][c], lo, hi);
        tot[q][c] += (double)lo + (double)hi;
      }
  }
#pragma unroll
  for (int q = 0; q < VIPT; q++) {
    if (kk[q] < n) {
      double *p = part + ((size_t)blockIdx.y * n + kk[q]) * 7;
#pragma unroll
      for (int c = 0; c < 7; c++) p[c] = tot[q][c];
    }
  }
}

// One quantity of one body per thread: consecutive threads read consecutive
// doubles of every split, all splits in flight (a thread per body, walking its
// splits 56 bytes apart, took 15 us at n = 8192; this takes 4).
__global__ void vjp_reduce_kernel(int n, int nsplit, const double *__restrict__ part, double *gx,
                                  double *gv, double *gm) {
  pdl_wait();
  pdl_trigger();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 7 * n) return;
  double u[4] = {0, 0, 0, 0};
#pragma unroll 2
  for (int s = 0; s < nsplit; s += 4)
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (s + q < nsplit) u[q] += part[(size_t)(s + q) * n * 7 + e];
  const double t = (u[0] + u[1]) + (u[2] + u[3]);
  const int k = e / 7, c = e - 7 * k;
  if (c < 3)
    gx[3 * k + c] = t;
  else if (c < 6)
    gv[3 * k + c - 3] = t;
  else
    gm[k] = t;
}

}  // namespace

extern "C" int g6k_fixed_records(const g6_jstate *js, int n, const double *x, const double *v,
                                 const double *m, int prec, cudaStream_t st) {
  const int n_pad = (n + G6_TILE - 1) / G6_TILE * G6_TILE;
  if (n <= 0 || n_pad > js->cap) return -1;
  return launch_pdl(records_kernel, dim3((n_pad + 31) / 32), dim3(32), 0, st, n, n_pad, x, v, m,
                    prec, js->jp_split, js->jp_f64) == cudaSuccess
             ? 0
             : -3;
}

// correct: the corrector with (a1, j1); predict: the next step's prediction
// into xp, vp and the force records.
extern "C" int g6k_fixed_advance(const g6_jstate *js, int n, double h, int correct, int predict,
                                 double *x, double *v, double *a, double *j, const double *a1,
                                 const double *j1, const double *m, double *xp, double *vp,
                                 int prec, cudaStream_t st) {
  const int n_pad = (n + G6_TILE - 1) / G6_TILE * G6_TILE;
  if (n <= 0 || n_pad > js->cap || (!correct && !predict)) return -1;
  auto kern = correct ? (predict ? advance_kernel<true, true> : advance_kernel<true, false>)
                      : advance_kernel<false, true>;
  return launch_pdl(kern, dim3(((predict ? n_pad : n) + 31) / 32), dim3(32), 0, st, n, n_pad, h, x,
                    v, a, j, a1, j1, m, xp, vp, prec, js->jp_split, js->jp_f64) == cudaSuccess
             ? 0
             : -3;
}

// Launch shapes.  FP64: one body per thread, one warp per CTA.
// Split: VIPT bodies per thread, j split so that there are about 24 CTAs per SM
// (three at a time), so that the last ones to end leave few SMs idle: call of
// 8192 bodies 274 us at 16 splits, 241 at 64; 16384: 950 at 10, 813 at 64;
// 32768: 3.75 ms at 5, 3.09 at 32.
static void vjp_shape(int n, int prec, int *nsplit, int *jsplit, int *n_pad) {
  *n_pad = (n + VTILE - 1) / VTILE * VTILE;
  if (prec == G6_PREC_FP64) {
    // about eight warps for every SM, no split below 16 j; and eight splits of
    // a large system, whose sums are the more exact for it
    const int warps = (n + VT - 1) / VT, want = 8 * g6k_sm_count();
    int ns = (want + warps - 1) / warps;
    if (ns < 8) ns = 8;
    if (ns > n / 16) ns = n / 16;
    if (ns < 1) ns = 1;
    *jsplit = (n + ns - 1) / ns;
    *nsplit = (n + *jsplit - 1) / *jsplit;
    return;
  }
  static int sms = 0;  // SM count of the (single) device, looked up once
  if (sms <= 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        sms <= 0)
      sms = 152;
  }
  const int gx = (n + VT2 * VIPT - 1) / (VT2 * VIPT);
  const int tiles = *n_pad / VTILE;
  int ns = (24 * sms + gx - 1) / gx;
  if (ns > tiles) ns = tiles;
  if (ns < 1) ns = 1;
  const int tp = (tiles + ns - 1) / ns;  // tiles per split
  *jsplit = tp * VTILE;
  *nsplit = (tiles + tp - 1) / tp;
}

// Scratch: the split records (n_pad x 64 B), then the partials
// (nsplit x n x 7 doubles); the larger of the two precisions' needs.
extern "C" size_t g6k_vjp_scratch_bytes(int n) {
  size_t need = 0;
  for (int prec = 0; prec < 2; prec++) {
    int ns, js, np;
    vjp_shape(n, prec, &ns, &js, &np);
    const size_t b = (size_t)np * (sizeof(VJPair) / 2) + (size_t)ns * (size_t)n * 7 * sizeof(double);
    if (b > need) need = b;
  }
  return need;
}

// The VJP from records (split) or la1, lj1 (FP64) that are ready.
static int vjp_core(int n, double eps2, int prec, int hjerk, const double *x, const double *v,
                    const double *m, const double *la1, const double *lj1, double *gx, double *gv,
                    double *gm, void *scratch, cudaStream_t st) {
  int nsplit, jsplit, n_pad;
  vjp_shape(n, prec, &nsplit, &jsplit, &n_pad);
  const VJPair *rec = reinterpret_cast<const VJPair *>(scratch);
  double *part = reinterpret_cast<double *>(reinterpret_cast<char *>(scratch) +
                                            (size_t)n_pad * (sizeof(VJPair) / 2));
  if (prec == G6_PREC_FP64) {
    launch_pdl(hjerk ? vjp_f64_kernel<true> : vjp_f64_kernel<false>,
               dim3((n + VT - 1) / VT, nsplit), dim3(VT), 0, st, n, eps2, x, v, m, la1, lj1,
               jsplit, part);
  } else {
    const float e2 = (float)eps2 + (float)(1.0 / 4503599627370496.0);
    launch_pdl(hjerk ? vjp_split_kernel<true> : vjp_split_kernel<false>,
               dim3((n + VT2 * VIPT - 1) / (VT2 * VIPT), nsplit), dim3(VT2), 0, st, n, e2, rec,
               jsplit, n_pad, part);
  }
  launch_pdl(vjp_reduce_kernel, dim3((7 * n + 127) / 128), dim3(128), 0, st, n, nsplit,
             (const double *)part, gx, gv, gm);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// hjerk: differentiate the hermite code's jerk form instead of the softened
// one (must match the force the forward step used).
extern "C" int g6k_force_vjp(int n, double eps2, int prec, int hjerk, const double *x,
                             const double *v, const double *m, const double *la1,
                             const double *lj1, double *gx, double *gv, double *gm, void *scratch,
                             cudaStream_t st) {
  if (n <= 0) return 0;
  if (prec != G6_PREC_FP64) {
    int nsplit, jsplit, n_pad;
    vjp_shape(n, prec, &nsplit, &jsplit, &n_pad);
    launch_pdl(vjp_records_kernel, dim3((n_pad + 31) / 32), dim3(32), 0, st, n, n_pad, x, v, m, la1,
               lj1, reinterpret_cast<VJPair *>(scratch));
  }
  return vjp_core(n, eps2, prec, hjerk, x, v, m, la1, lj1, gx, gv, gm, scratch, st);
}

// The adjoints of nsteps consecutive fixed steps, last first, at the predicted
// states xp_all, vp_all ([nsteps][n][3]): per step the force VJP with its
// reduction, and one kernel that ends the step's adjoint and begins the next
// one's.
extern "C" int g6k_fixed_adjoint(int n, double h, double eps2, int nsteps, int prec, int hjerk,
                                 const double *xp_all, const double *vp_all, const double *m,
                                 double *lx, double *lv, double *la, double *lj, double *lm,
                                 double *la1, double *lj1, double *gxp, double *gvp, double *gm,
                                 void *scratch, cudaStream_t st) {
  if (n <= 0 || nsteps <= 0) return 0;
  int nsplit, jsplit, n_pad;
  vjp_shape(n, prec, &nsplit, &jsplit, &n_pad);
  VJPair *rec = prec == G6_PREC_FP64 ? nullptr : reinterpret_cast<VJPair *>(scratch);
  const dim3 grid(((rec ? n_pad : n) + 31) / 32), block(32);
  const size_t step = 3 * (size_t)n;
  for (int s = nsteps - 1; s >= -1; s--) {
    // before the VJP of step s: the end of step s + 1, the beginning of s
    const double *x = s >= 0 ? xp_all + step * s : nullptr, *v = s >= 0 ? vp_all + step * s : nullptr;
    auto kern = s == nsteps - 1 ? adjoint_kernel<false, true>
                : s >= 0        ? adjoint_kernel<true, true>
                                : adjoint_kernel<true, false>;
    if (launch_pdl(kern, grid, block, 0, st, n, n_pad, h, lx, lv, la, lj, (const double *)gxp,
                   (const double *)gvp, lm, (const double *)gm, x, v, m, la1, lj1,
                   rec) != cudaSuccess)
      return -3;
    if (s >= 0 && vjp_core(n, eps2, prec, hjerk, x, v, m, la1, lj1, gxp, gvp, gm, scratch, st))
      return -3;
  }
  return 0;
}
