// kern_knn.cu -- the k nearest neighbours of listed particles (extension
// call g6x_knn), exact in FP64.
//
// ph4's jdata::get_densities_on_gpu (src/amuse_ph4/src/gpu.cc:568-866)
// gathers, through the GRAPE neighbour-list calls and a retry loop on the
// search radii, the knn = 12 nearest neighbours of every particle:
// save_neighbors (gpu.cc:534-558) sorts all other particles by the squared
// distance sum_k (x_i,k - x_j,k)^2 and keeps the first knn.  Here:
//
//   knn_kernel     one thread per listed particle streams the split records
//                  (j split across CTAs when few particles are listed) and
//                  keeps, in shared memory, the k + KEXTRA smallest FP32
//                  double-single squared distances (two j per packed f32x2
//                  instruction; no FP64 in the loop), then writes the FP64
//                  squared distances of those candidates, summed in
//                  component order as save_neighbors sums them, from
//                  positions predicted with ph4's expression;
//   knn_cells_kernel  the same candidates where there are many pairs: the
//                  j-particles sorted into spatial cells and tiles of 64,
//                  and whole tiles skipped whose bounding box is provably
//                  farther than every kept key (below);
//   knn_merge      per particle: sorts each split's candidates by (d^2,
//                  slot), proves that no particle left out can be among the
//                  k nearest (gap test below), and merges the splits;
//   knn_exact      particles whose gap test failed (many FP32-equal
//                  distances at the cut, e.g. a lattice) are redone with an
//                  FP64 distance for every j that passes the filter bound.
//
// Filter bound.  With X >= max |coordinate| over the j-system, each FP32
// difference dx_f of the split records obeys |dx_f - dx| <= 2^-22 |dx| + E,
// E = 2^-30 X (double-single representation 2^-48 X per position, three
// FP32 roundings, and a few ulps between the split predictor's FMA form and
// ph4's expression).  The FMA chain for the square sum adds 3 roundings.  So
// d^2 <= D implies d_f^2 <= T(D) = (1 + 2^-16) D + 4 E sqrt(D) + 4 E^2.
// Gap test: the candidates are the particles with the smallest FP32 keys,
// every other j has d_f^2 >= F (the largest kept key); if T(d_k^2) < F for
// the k-th exact distance d_k^2 among the candidates, every other j has
// d^2 > d_k^2, so the candidates hold the exact k nearest.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include "f32x2.cuh"
#include "g6_dev.h"

namespace {

constexpr int KT = 128;            // threads per CTA, one listed particle each
constexpr int KTJ = G6_TILE;       // j per shared-memory tile
constexpr int KRPT = KTJ / 2;      // split record pairs per tile
constexpr int KMAXSPLIT = 64;      // j-splits at most
constexpr int KEXTRA = 8;          // candidates kept beyond k
constexpr int KPMAX = G6_KNN_MAX + KEXTRA;

// One pair of consecutive split records (the layout in g6_dev.h).
struct __align__(16) PairRec {
  float2 xh, yh, zh, m, xl, yl, zl, pad0, vx, vy, vz, pad1;
};
static_assert(sizeof(PairRec) == 96, "split record pair");

struct KArgs {
  g6_jstate js;
  int nj, ni, k, kp, nsplit, jsplit;
  const int *slots;      // [ni]
  const double *pos64;   // [nj][4]: ph4-predicted x, y, z
  const unsigned *xmax;  // FP32 bits of max |xh| over j < nj
  double *cand_d;        // [nsplit][ni][kp] exact d^2 of the candidates
  int *cand_s;           // [nsplit][ni][kp] their slots
  int *cand_n;           // [nsplit][ni] candidates kept
  float *cand_f;         // [nsplit][ni] largest FP32 key kept (+inf: all kept)
  int *flag;             // [ni] gap test failed
  int *ids;              // [ni][k] out
  double *d2;            // [ni][k] out
};

__global__ void knn_xmax_kernel(g6_jstate js, int nj, unsigned *xmax) {
  float m = 0.f;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nj; s += gridDim.x * blockDim.x) {
    m = fmaxf(m, fabsf(g6_split_get(js.jp_split, s, 0)));
    m = fmaxf(m, fabsf(g6_split_get(js.jp_split, s, 1)));
    m = fmaxf(m, fabsf(g6_split_get(js.jp_split, s, 2)));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(xmax, __float_as_uint(m));  // m >= 0: bits order
}

// ph4-predicted FP64 positions of all j (save_neighbors' coordinates).
__global__ void knn_pos_kernel(g6_jstate js, int nj, double t, double *pos64) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nj) return;
  const int cap = js.cap;
  const double dt = __dsub_rn(t, js.t[s]);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int a = k * cap + s;
    pos64[4 * (size_t)s + k] = g6_predict_x(js.x[a], js.v[a], js.a[a], js.j[a], dt);
  }
  pos64[4 * (size_t)s + 3] = 0.0;
}

// Squared distances are >= +0, so their IEEE bits order like the values:
// the sort keys compare as integers (FP64 compares issue at the FP64 rate).
__device__ __forceinline__ unsigned long long kbits(double d) {
  return (unsigned long long)__double_as_longlong(d);
}
__device__ __forceinline__ bool kless(unsigned long long a, int sa, unsigned long long b,
                                      int sb) {
  return a < b || (a == b && sa < sb);
}

__device__ __forceinline__ double knn_E(const unsigned *xmax) {
  return (double)__uint_as_float(*xmax) * (1.0 + 1.0 / 1048576.0) * (1.0 / 1073741824.0);
}

// T(D) of the header, rounded up to FP32.
__device__ __forceinline__ float knn_bound(double D, double E) {
  const double T = (1.0 + 1.0 / 65536.0) * D + 4.0 * E * sqrt(D) + 4.0 * E * E;
  return __double2float_ru(T);
}

// FP64 squared distance, summed in component order (save_neighbors).
__device__ __forceinline__ double knn_d2(const double *pos64, double x0, double x1, double x2,
                                         int j) {
  const double d0 = __dsub_rn(x0, pos64[4 * (size_t)j]);
  const double d1 = __dsub_rn(x1, pos64[4 * (size_t)j + 1]);
  const double d2 = __dsub_rn(x2, pos64[4 * (size_t)j + 2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
}

struct IPos {
  f2x xh, yh, zh, xl, yl, zl;
  double x0, x1, x2;
};

__device__ __forceinline__ IPos knn_ipos(const KArgs &ka, int self) {
  IPos p;
  const void *r = ka.js.jp_split;
  p.xh = f2_dup(g6_split_get(r, self, 0));
  p.yh = f2_dup(g6_split_get(r, self, 1));
  p.zh = f2_dup(g6_split_get(r, self, 2));
  p.xl = f2_dup(g6_split_get(r, self, 4));
  p.yl = f2_dup(g6_split_get(r, self, 5));
  p.zl = f2_dup(g6_split_get(r, self, 6));
  p.x0 = ka.pos64[4 * (size_t)self];
  p.x1 = ka.pos64[4 * (size_t)self + 1];
  p.x2 = ka.pos64[4 * (size_t)self + 2];
  return p;
}

// FP32 squared distances of one record pair (two j) to the particle.
__device__ __forceinline__ void knn_r2f(const PairRec &r, const IPos &p, float &ra, float &rb) {
  const f2x dx = f2_add(f2_sub(f2_of(r.xh), p.xh), f2_sub(f2_of(r.xl), p.xl));
  const f2x dy = f2_add(f2_sub(f2_of(r.yh), p.yh), f2_sub(f2_of(r.yl), p.yl));
  const f2x dz = f2_add(f2_sub(f2_of(r.zh), p.zh), f2_sub(f2_of(r.zl), p.zl));
  f2_unpack(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))), ra, rb);
}

__device__ __forceinline__ void knn_load_tile(PairRec *tile, const PairRec *gj, int tj) {
  const float4 *src = reinterpret_cast<const float4 *>(gj + tj / 2);
  float4 *dst = reinterpret_cast<float4 *>(tile);
  for (int q = threadIdx.x; q < KRPT * 6; q += KT) dst[q] = src[q];
}

// Candidate pass: the kp smallest FP32 keys (ties to the smaller slot) of
// this split's j range, then their exact FP64 squared distances.
__global__ void __launch_bounds__(KT) knn_kernel(KArgs ka) {
  extern __shared__ __align__(16) unsigned char smem[];
  PairRec *tile = reinterpret_cast<PairRec *>(smem);
  float *lf = reinterpret_cast<float *>(tile + KRPT);  // [kp][KT]
  int *ls = reinterpret_cast<int *>(lf + ka.kp * KT);   // [kp][KT]
  const int tid = threadIdx.x;
  const int i = blockIdx.x * KT + tid;
  const bool active = i < ka.ni;
  const int self = active ? ka.slots[i] : -1;
  const int KP = ka.kp;
  IPos ip;
  if (active) ip = knn_ipos(ka, self);
  int cnt = 0;
  float F = __int_as_float(0x7f800000);  // largest kept key once the list is full

  const int j0 = blockIdx.y * ka.jsplit;
  const int j1 = min(j0 + ka.jsplit, ka.nj);
  const PairRec *gj = reinterpret_cast<const PairRec *>(ka.js.jp_split);
  for (int tj = j0; tj < j1; tj += KTJ) {
    knn_load_tile(tile, gj, tj);
    __syncthreads();
    if (active) {
      // Two record pairs (four j) per step: two independent FP32 chains and
      // one early-out test.  The kept set does not depend on the order in
      // which candidates arrive.
      const int npair = min(KRPT, (j1 - tj + 1) / 2);
      for (int p = 0; p < npair; p += 2) {
        float rr[4];
        knn_r2f(tile[p], ip, rr[0], rr[1]);
        if (p + 1 < npair) {
          knn_r2f(tile[p + 1], ip, rr[2], rr[3]);
        } else {
          rr[2] = rr[3] = __int_as_float(0x7f800000);
        }
        if (fminf(fminf(rr[0], rr[1]), fminf(rr[2], rr[3])) > F) continue;
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int j = tj + 2 * p + h;
          const float r = rr[h];
          if ((h >= 2 && p + 1 >= npair) || r > F || j >= j1 || j == self) continue;
          if (cnt == KP) {
            const float lr = lf[(KP - 1) * KT + tid];
            if (!(r < lr || (r == lr && j < ls[(KP - 1) * KT + tid]))) continue;
          }
          int q = cnt < KP ? cnt : KP - 1;
          while (q > 0) {
            const float pr = lf[(q - 1) * KT + tid];
            const int ps = ls[(q - 1) * KT + tid];
            if (!(r < pr || (r == pr && j < ps))) break;
            lf[q * KT + tid] = pr;
            ls[q * KT + tid] = ps;
            q--;
          }
          lf[q * KT + tid] = r;
          ls[q * KT + tid] = j;
          if (cnt < KP) cnt++;
          if (cnt == KP) F = lf[(KP - 1) * KT + tid];
        }
      }
    }
    __syncthreads();
  }
  if (!active) return;
  const size_t o = (size_t)blockIdx.y * ka.ni + i;
  ka.cand_n[o] = cnt;
  ka.cand_f[o] = cnt == KP ? F : __int_as_float(0x7f800000);
  for (int q = 0; q < cnt; q++) {
    const int j = ls[q * KT + tid];
    ka.cand_d[o * KP + q] = knn_d2(ka.pos64, ip.x0, ip.x1, ip.x2, j);
    ka.cand_s[o * KP + q] = j;
  }
}

// Per listed particle: exact sort of each split's candidates, the gap test,
// and the merge of the splits' k nearest.
__global__ void knn_merge_kernel(KArgs ka) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ka.ni) return;
  const int K = ka.k, KP = ka.kp;
  const double E = knn_E(ka.xmax);
  unsigned long long ck[KPMAX], gk[G6_KNN_MAX], tk[G6_KNN_MAX];
  int cs[KPMAX], gs[G6_KNN_MAX], ts[G6_KNN_MAX];
  int gn = 0;
  bool ok = true;
  for (int sp = 0; sp < ka.nsplit; sp++) {
    const size_t o = (size_t)sp * ka.ni + i;
    const int n = ka.cand_n[o];
    for (int q = 0; q < n; q++) {  // insertion sort by (d^2, slot)
      const unsigned long long key = kbits(ka.cand_d[o * KP + q]);
      const int sl = ka.cand_s[o * KP + q];
      int r = q;
      while (r > 0 && kless(key, sl, ck[r - 1], cs[r - 1])) {
        ck[r] = ck[r - 1];
        cs[r] = cs[r - 1];
        r--;
      }
      ck[r] = key;
      cs[r] = sl;
    }
    const float F = ka.cand_f[o];
    if (n == KP && !(knn_bound(__longlong_as_double((long long)ck[K - 1]), E) < F)) ok = false;
    // merge the split's first min(K, n) into the running k nearest
    const int m = n < K ? n : K;
    int a = 0, b = 0, t = 0;
    while (t < K && (a < gn || b < m)) {
      if (b >= m || (a < gn && kless(gk[a], gs[a], ck[b], cs[b]))) {
        tk[t] = gk[a];
        ts[t++] = gs[a++];
      } else {
        tk[t] = ck[b];
        ts[t++] = cs[b++];
      }
    }
    for (int q = 0; q < t; q++) {
      gk[q] = tk[q];
      gs[q] = ts[q];
    }
    gn = t;
  }
  ka.flag[i] = ok ? 0 : 1;
  for (int q = 0; q < K; q++) {
    ka.ids[(size_t)i * K + q] = q < gn ? ka.js.id[gs[q]] : -1;
    ka.d2[(size_t)i * K + q] =
        q < gn ? __longlong_as_double((long long)gk[q]) : __longlong_as_double(0x7ff0000000000000ll);
  }
}

// Particles whose gap test failed: one pass over all j with an FP64
// distance for every j that passes the filter bound T(current k-th), and a
// sorted list of the k nearest in shared memory.  CTAs without such a
// particle return at once.
__global__ void __launch_bounds__(KT) knn_exact_kernel(KArgs ka) {
  extern __shared__ __align__(16) unsigned char smem[];
  PairRec *tile = reinterpret_cast<PairRec *>(smem);
  unsigned long long *lk = reinterpret_cast<unsigned long long *>(tile + KRPT);  // [k][KT]
  int *ls = reinterpret_cast<int *>(lk + ka.k * KT);                               // [k][KT]
  const int tid = threadIdx.x;
  const int i = blockIdx.x * KT + tid;
  const bool mine = i < ka.ni && ka.flag[i];
  if (!__syncthreads_or(mine)) return;
  const int self = mine ? ka.slots[i] : -1;
  const int K = ka.k;
  IPos ip;
  if (mine) ip = knn_ipos(ka, self);
  const double E = knn_E(ka.xmax);
  int cnt = 0;
  float T = __int_as_float(0x7f800000);
  const PairRec *gj = reinterpret_cast<const PairRec *>(ka.js.jp_split);
  for (int tj = 0; tj < ka.nj; tj += KTJ) {
    knn_load_tile(tile, gj, tj);
    __syncthreads();
    if (mine) {
      const int npair = min(KRPT, (ka.nj - tj + 1) / 2);
      for (int p = 0; p < npair; p++) {
        float ra, rb;
        knn_r2f(tile[p], ip, ra, rb);
        if (fminf(ra, rb) > T) continue;
        for (int h = 0; h < 2; h++) {
          const int j = tj + 2 * p + h;
          if ((h ? rb : ra) > T || j >= ka.nj || j == self) continue;
          const unsigned long long key = kbits(knn_d2(ka.pos64, ip.x0, ip.x1, ip.x2, j));
          if (cnt == K && !kless(key, j, lk[(K - 1) * KT + tid], ls[(K - 1) * KT + tid]))
            continue;
          int q = cnt < K ? cnt : K - 1;
          while (q > 0 && kless(key, j, lk[(q - 1) * KT + tid], ls[(q - 1) * KT + tid])) {
            lk[q * KT + tid] = lk[(q - 1) * KT + tid];
            ls[q * KT + tid] = ls[(q - 1) * KT + tid];
            q--;
          }
          lk[q * KT + tid] = key;
          ls[q * KT + tid] = j;
          if (cnt < K) cnt++;
          if (cnt == K)
            T = knn_bound(__longlong_as_double((long long)lk[(K - 1) * KT + tid]), E);
        }
      }
    }
    __syncthreads();
  }
  if (!mine) return;
  for (int q = 0; q < K; q++) {
    ka.ids[(size_t)i * K + q] = q < cnt ? ka.js.id[ls[q * KT + tid]] : -1;
    ka.d2[(size_t)i * K + q] = q < cnt ? __longlong_as_double((long long)lk[q * KT + tid])
                                       : __longlong_as_double(0x7ff0000000000000ll);
  }
}

// ------------------------------------------------------------ cell path ---
//
// Brute force looks at every pair and, while a particle's list settles, the
// lanes of a warp insert at different times (N = 65536: 8.3 ms, 5e11 pairs/s).
// Here the j-particles are put in the order of spatial cells (a counting
// sort: histogram, scan, placement), cut into tiles of 64 with bounding boxes
// and a second level of boxes of 32 tiles.  A warp takes 32 listed particles
// of neighbouring cells, fills its lists from the tiles around its own cell,
// and then skips every tile (and every group of 32) whose box cannot hold a
// candidate of any of its lanes.  What bounds it now is the issue of the
// distance and insertion instructions of the tiles left (N = 65536, all:
// 2.0e8 warp instructions in 0.72 ms, against 8.3 ms by brute force).
//
// Skip test.  B, the squared distance of the warp's box and the tile's, is at
// most D, the squared distance of any pair of them, and by the filter bound's
// argument (file header) the FP32 key of a pair is at least
// (1 - 2^-16) D - 4 E sqrt(D).  That grows with D where it is positive, so
// with every rounding taken down, (1 - 2^-16) B - 4 E sqrt(B) > F means that
// no key of the tile is at or below F: the kept set is the one that brute
// force keeps, ties included, whatever the cells look like.  Cells only
// decide how much is skipped: the map x -> (x - c) / (s + |x - c|), c and s
// the median and the quartile distance of 1024 sampled particles, gives a
// centrally concentrated system small cells in the middle and takes any
// outlier.
constexpr int CTJ = 64;          // j per tile
constexpr int CW = 4;            // warps per CTA
constexpr int CMAP = 1024;       // sampled particles
struct CBox {
  float lo[3], pad0, hi[3], pad1;
};

struct CArgs {
  int nj_pad, bits, ntile, nsuper;
  float *map;            // c[3], s[3]
  int *count;            // [cells] j: histogram, then first positions
  int *icount;           // [cells] the same for the listed particles
  int *cell, *rank;      // [nj]
  int *icell, *irank;    // [ni]
  float *rec;            // [nj_pad / 2][12] pairs, fields xh yh zh xl yl zl
  int *order;            // [nj_pad] slots in cell order, -1 padding
  int *iorder;           // [ni] listed indices in cell order
  CBox *box, *super;     // [ntile], [nsuper]
};

__global__ void __launch_bounds__(CMAP) knn_map_kernel(g6_jstate js, int nj, float *map) {
  __shared__ float v[CMAP];
  const int t = threadIdx.x;
  const int s = (int)((long long)t * nj / CMAP);
  for (int a = 0; a < 3; a++) {
    v[t] = g6_split_get(js.jp_split, s, a);
    __syncthreads();
    for (int k = 2; k <= CMAP; k <<= 1)  // bitonic sort
      for (int q = k >> 1; q > 0; q >>= 1) {
        const int o = t ^ q;
        if (o > t) {
          const float x = v[t], y = v[o];
          if ((x > y) == ((t & k) == 0)) {
            v[t] = y;
            v[o] = x;
          }
        }
        __syncthreads();
      }
    if (t == 0) {
      map[a] = v[CMAP / 2];
      map[3 + a] = fmaxf(v[3 * CMAP / 4] - v[CMAP / 4], 1e-30f);
    }
    __syncthreads();
  }
}

__device__ __forceinline__ int knn_cell(const void *rec, int s, const float *map, int bits) {
  int key = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float d = (g6_split_get(rec, s, a) - map[a]) / map[3 + a];
    const float u = 0.5f + 0.5f * (d / (1.0f + fabsf(d)));
    const int q = min(max((int)(u * (float)(1 << bits)), 0), (1 << bits) - 1);
    for (int b = 0; b < bits; b++) key |= ((q >> b) & 1) << (3 * b + a);
  }
  return key;
}

__global__ void knn_hist_kernel(const void *rec, const int *slots, int n, const float *map,
                                int bits, int *count, int *cell, int *rank) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int c = knn_cell(rec, slots ? slots[e] : e, map, bits);
  cell[e] = c;
  rank[e] = atomicAdd(count + c, 1);
}

// Exclusive prefix sums in place: one CTA per array of `cells` counts (a
// multiple of 1024); a warp takes a contiguous piece, 32 counts at a time.
__global__ void __launch_bounds__(1024) knn_scan_kernel(int *a0, int *a1, int cells) {
  __shared__ int w[32];
  const int t = threadIdx.x, lane = t & 31, per = cells / 1024;
  int *a = (blockIdx.x ? a1 : a0) + (t >> 5) * per * 32 + lane;
  int sum = 0;
#pragma unroll 8
  for (int k = 0; k < per; k++) sum += a[32 * k];
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) w[t >> 5] = sum;
  __syncthreads();
  int run = lane < (t >> 5) ? w[lane] : 0;  // counts before this warp's piece
  run = __reduce_add_sync(0xffffffffu, run);
#pragma unroll 4
  for (int k = 0; k < per; k++) {
    const int c = a[32 * k];
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    a[32 * k] = run + inc - c;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
}

__global__ void knn_place_kernel(KArgs ka, CArgs ca) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < ka.ni) ca.iorder[ca.icount[ca.icell[e]] + ca.irank[e]] = e;
  if (e >= ca.nj_pad) return;
  const int q = e < ka.nj ? ca.count[ca.cell[e]] + ca.rank[e] : e;
  float *r = ca.rec + (size_t)(q >> 1) * 12 + (q & 1);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    r[2 * a] = e < ka.nj ? g6_split_get(ka.js.jp_split, e, a) : 1.0e18f;
    r[6 + 2 * a] = e < ka.nj ? g6_split_get(ka.js.jp_split, e, 4 + a) : 0.f;
  }
  ca.order[q] = e < ka.nj ? e : -1;
}

__device__ __forceinline__ void box_warp(CBox &b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 3; a++) {
      b.lo[a] = fminf(b.lo[a], __shfl_xor_sync(0xffffffffu, b.lo[a], o));
      b.hi[a] = fmaxf(b.hi[a], __shfl_xor_sync(0xffffffffu, b.hi[a], o));
    }
}
__device__ __forceinline__ CBox box_empty() {
  CBox b;
  b.pad0 = b.pad1 = 0.f;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    b.lo[a] = __int_as_float(0x7f800000);
    b.hi[a] = __int_as_float(0xff800000);
  }
  return b;
}
__device__ __forceinline__ void box_add(CBox &b, int a, float xh, float xl) {
  b.lo[a] = fminf(b.lo[a], __fadd_rd(xh, xl));
  b.hi[a] = fmaxf(b.hi[a], __fadd_ru(xh, xl));
}

// A warp per tile (padding excluded), or per 32 tiles (level 1).
__global__ void knn_box_kernel(CArgs ca, int level) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= (level ? ca.nsuper : ca.ntile)) return;
  CBox b = box_empty();
  if (level == 0) {
    const float *r = ca.rec + ((size_t)w * (CTJ / 2) + lane) * 12;
    for (int h = 0; h < 2; h++)
      if (ca.order[w * CTJ + 2 * lane + h] >= 0)
        for (int a = 0; a < 3; a++) box_add(b, a, r[2 * a + h], r[6 + 2 * a + h]);
  } else if (32 * w + lane < ca.ntile) {
    b = ca.box[32 * w + lane];
  }
  box_warp(b);
  if (lane == 0) (level ? ca.super : ca.box)[w] = b;
}

// Lower bound of the FP32 key between boxes, or below zero.
__device__ __forceinline__ float box_bound(const CBox &p, const CBox &q, float E4) {
  float B = 0.f;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float g =
        fmaxf(0.f, fmaxf(__fsub_rd(q.lo[a], p.hi[a]), __fsub_rd(p.lo[a], q.hi[a])));
    B = __fmaf_rd(g, g, B);
  }
  return __fsub_rd(__fmul_rd(B, 1.0f - 1.0f / 65536.0f), __fmul_ru(E4, __fsqrt_ru(B)));
}

// KP: candidates kept, in registers as sorted (key bits, slot) words.  An
// insertion is branchless: position q takes its left neighbour, the new word
// or stays, all positions at once (about 6 KP instructions, for all lanes
// together).  Lists in shared memory, each lane shifting its own, made one
// warp take 0.8 ms.
template <int KP>
__global__ void __launch_bounds__(32 * CW) knn_cells_kernel(KArgs ka, CArgs ca) {
  __shared__ __align__(16) float s_tile[CW][CTJ / 2 * 12];
  __shared__ int s_sid[CW][CTJ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float *tile = s_tile[warp];
  int *sid = s_sid[warp];
  const float inf = __int_as_float(0x7f800000);
  const unsigned FULL = 0xffffffffu;
  const int w0 = (blockIdx.x * CW + warp) * 32;
  if (w0 >= ka.ni) return;  // whole warps; nothing below crosses warps
  const bool active = w0 + lane < ka.ni;
  const int li = ca.iorder[active ? w0 + lane : w0];
  const int self = ka.slots[li];
  const IPos ip = knn_ipos(ka, self);
  CBox own = box_empty();
#pragma unroll
  for (int a = 0; a < 3; a++)
    box_add(own, a, g6_split_get(ka.js.jp_split, self, a), g6_split_get(ka.js.jp_split, self, 4 + a));
  CBox ib = own;
  box_warp(ib);
  const float E4 = __double2float_ru(4.0 * knn_E(ka.xmax));
  constexpr unsigned long long NONE = 0x7f8000007fffffffull;  // key +inf, no slot
  unsigned long long kept[KP];
#pragma unroll
  for (int q = 0; q < KP; q++) kept[q] = NONE;
  float F = active ? inf : 0.f;  // largest kept key once the list is full
  float Fw = inf;                // the warp's largest

  auto process = [&](int t) {
    __syncwarp();
    const float4 *src = reinterpret_cast<const float4 *>(ca.rec + (size_t)t * (CTJ / 2) * 12);
    float4 *dst = reinterpret_cast<float4 *>(tile);
#pragma unroll
    for (int q = 0; q < 3; q++) dst[lane + 32 * q] = src[lane + 32 * q];
    sid[lane] = ca.order[t * CTJ + lane];
    sid[lane + 32] = ca.order[t * CTJ + 32 + lane];
    __syncwarp();
#pragma unroll 1
    for (int p = 0; p < CTJ / 2; p += 2) {
      float rr[4];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float4 *r = reinterpret_cast<const float4 *>(tile + (p + h) * 12);
        const float4 A = r[0], B = r[1], C = r[2];
        const f2x dx = f2_add(f2_sub(f2_pack(A.x, A.y), ip.xh), f2_sub(f2_pack(B.z, B.w), ip.xl));
        const f2x dy = f2_add(f2_sub(f2_pack(A.z, A.w), ip.yh), f2_sub(f2_pack(C.x, C.y), ip.yl));
        const f2x dz = f2_add(f2_sub(f2_pack(B.x, B.y), ip.zh), f2_sub(f2_pack(C.z, C.w), ip.zl));
        f2_unpack(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))), rr[2 * h], rr[2 * h + 1]);
      }
      if (!__any_sync(FULL, fminf(fminf(rr[0], rr[1]), fminf(rr[2], rr[3])) <= F)) continue;
#pragma unroll 1
      for (int h = 0; h < 4; h++) {
        const float r = h == 0 ? rr[0] : h == 1 ? rr[1] : h == 2 ? rr[2] : rr[3];
        const int j = sid[2 * p + h];
        unsigned long long key = ~0ull;
        // keys are >= +0, so their bits order like the values
        if (r <= F && j != self)
          key = (unsigned long long)__float_as_uint(r) << 32 | (unsigned)j;
        if (j < 0 || !__any_sync(FULL, key < kept[KP - 1])) continue;  // j < 0: padding
        bool lt = key < kept[KP - 1];
#pragma unroll
        for (int q = KP - 1; q > 0; q--) {
          const bool ltq = key < kept[q - 1];
          kept[q] = lt ? (ltq ? kept[q - 1] : key) : kept[q];
          lt = ltq;
        }
        kept[0] = lt ? key : kept[0];
        if (active) F = __uint_as_float((unsigned)(kept[KP - 1] >> 32));
      }
    }
    Fw = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(F)));
  };

  // does any lane's own particle want the box?  (The warp's box may be wide:
  // in a halo, or where the cell order jumps.)
  auto wanted = [&](const CBox &b) {
    return __any_sync(FULL, active && !(box_bound(own, b, E4) > F)) != 0;
  };

  // the tiles around the warp's own cell first
  int t0 = ca.count[ca.icell[__shfl_sync(0xffffffffu, li, 0)]] / CTJ;
  t0 = min(t0, ca.ntile - 1);
  process(t0);
  if (t0 + 1 < ca.ntile) process(t0 + 1);
  if (t0 > 0) process(t0 - 1);
  for (int sb = 0; sb < ca.nsuper; sb += 32) {
    const int su = sb + lane;
    unsigned sm = __ballot_sync(
        0xffffffffu, su < ca.nsuper && !(box_bound(ib, ca.super[min(su, ca.nsuper - 1)], E4) > Fw));
    while (sm) {
      const int sup = sb + __ffs(sm) - 1;
      sm &= sm - 1;
      if (!wanted(ca.super[sup])) continue;
      const int t = sup * 32 + lane;
      const float lb = t < ca.ntile ? box_bound(ib, ca.box[t], E4) : inf;
      const bool done = t == t0 || t == t0 + 1 || t == t0 - 1 || t >= ca.ntile;
      unsigned tm = __ballot_sync(0xffffffffu, !done && !(lb > Fw));
      while (tm) {
        const int l = __ffs(tm) - 1;
        tm &= tm - 1;
        if (!wanted(ca.box[sup * 32 + l])) continue;
        process(sup * 32 + l);
        tm &= __ballot_sync(0xffffffffu, !(lb > Fw));  // the lists got shorter keys
      }
    }
  }
  if (!active) return;
  ka.cand_f[li] = F;  // +inf: fewer than KP others
  int cnt = 0;
#pragma unroll
  for (int q = 0; q < KP; q++) {
    const int j = (int)(unsigned)kept[q];
    if (j == 0x7fffffff) continue;
    ka.cand_d[(size_t)li * KP + cnt] = knn_d2(ka.pos64, ip.x0, ip.x1, ip.x2, j);
    ka.cand_s[(size_t)li * KP + cnt] = j;
    cnt++;
  }
  ka.cand_n[li] = cnt;
}

// The cell path where it pays for its sort (about 60 us) and where the listed
// particles are dense enough for the 32 of a warp to want the same tiles.
// Whole call, cells against brute force: 4096 of 4096 393 and 503 us, 2048 of
// 8192 633 and 592, 4096 of 16384 527 and 685, 2048 of 16384 903 and 817, 8192
// of 65536 1.83 and 2.26 ms, 1024 of 65536 2.8 and 1.3 ms; all of 65536 0.98
// and 8.5 ms, all of 2^20 13.7 and 627 ms.
bool knn_use_cells(int ni, int nj) {
  const long long pairs = (long long)ni * nj, n = ni;
  return (pairs >= 1ll << 24 && 2 * n >= nj) || (pairs >= 1ll << 26 && 4 * n >= nj) ||
         (pairs >= 1ll << 29 && 8 * n >= nj);
}

// Candidates kept per particle: k + KEXTRA, on the cell path the next of its
// list lengths.
int knn_kept(int ni, int nj, int k) {
  if (!knn_use_cells(ni, nj)) return k + KEXTRA;
  return k <= 4 ? 12 : k <= 8 ? 16 : k <= 12 ? 20 : k <= 20 ? 28 : KPMAX;
}
// 2^15 cells up to 2^17 particles, 2^18 above.
int knn_bits(int nj) { return nj <= (1 << 17) ? 5 : 6; }

void knn_shape(int ni, int nj, int *nsplit, int *jsplit) {
  if (knn_use_cells(ni, nj)) {
    *nsplit = 1;
    *jsplit = nj;
    return;
  }
  const int ntiles = (nj + KTJ - 1) / KTJ;
  const int gx = (ni + KT - 1) / KT;
  const int want = 4 * g6k_sm_count();
  int ns = (want + gx - 1) / gx;
  if (ns > KMAXSPLIT) ns = KMAXSPLIT;
  if (ns > ntiles) ns = ntiles;
  if (ns < 1) ns = 1;
  const int tp = (ntiles + ns - 1) / ns;
  *jsplit = tp * KTJ;
  *nsplit = (ntiles + tp - 1) / tp;
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

struct Layout {
  size_t pos64, xmax, cand_d, cand_s, cand_n, cand_f, flag;
  size_t map, count, icount, cell, rank, icell, irank, rec, order, iorder, box, super;  // cell path
  size_t total;
};

Layout knn_layout(int nj, int ni, int k, int nsplit) {
  const size_t kp = (size_t)knn_kept(ni, nj, k), nc = (size_t)nsplit * ni;
  Layout L;
  L.pos64 = 0;
  L.xmax = L.pos64 + align256(sizeof(double) * 4 * (size_t)nj);
  L.cand_d = L.xmax + align256(sizeof(unsigned));
  L.cand_s = L.cand_d + align256(sizeof(double) * nc * kp);
  L.cand_n = L.cand_s + align256(sizeof(int) * nc * kp);
  L.cand_f = L.cand_n + align256(sizeof(int) * nc);
  L.flag = L.cand_f + align256(sizeof(float) * nc);
  size_t o = L.flag + align256(sizeof(int) * (size_t)ni);
  L.map = o;
  if (knn_use_cells(ni, nj)) {
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += align256(bytes);
      return at;
    };
    const size_t cells = (size_t)1 << (3 * knn_bits(nj));
    const size_t nt = ((size_t)nj + CTJ - 1) / CTJ;
    L.map = take(6 * sizeof(float));
    L.count = take(2 * cells * sizeof(int));
    L.icount = L.count + cells * sizeof(int);
    L.cell = take(sizeof(int) * (size_t)nj);
    L.rank = take(sizeof(int) * (size_t)nj);
    L.icell = take(sizeof(int) * (size_t)ni);
    L.irank = take(sizeof(int) * (size_t)ni);
    L.rec = take(nt * CTJ * 24);
    L.order = take(nt * CTJ * sizeof(int));
    L.iorder = take(sizeof(int) * (size_t)ni);
    L.box = take(nt * sizeof(CBox));
    L.super = take((nt + 31) / 32 * sizeof(CBox));
  }
  L.total = o;
  return L;
}

}  // namespace

extern "C" size_t g6k_knn_scratch_bytes(int nj, int ni, int k) {
  int nsplit, jsplit;
  knn_shape(ni, nj, &nsplit, &jsplit);
  return knn_layout(nj, ni, k, nsplit).total;
}

// The split records must hold the j-system predicted to t (g6k_predict,
// G6_PREC_SPLIT); slots, ids and d2 are device arrays.
extern "C" int g6k_knn(const g6_jstate *js, int nj, double t, int k, int ni, const int *slots,
                       int *ids, double *d2, void *scratch, size_t scratch_bytes,
                       cudaStream_t st) {
  if (ni <= 0) return 0;
  if (nj <= 0 || k < 1 || k > G6_KNN_MAX) return -2;
  if (scratch_bytes < g6k_knn_scratch_bytes(nj, ni, k)) return -4;
  int nsplit, jsplit;
  knn_shape(ni, nj, &nsplit, &jsplit);
  const Layout L = knn_layout(nj, ni, k, nsplit);
  char *p = static_cast<char *>(scratch);
  static bool attr = false;
  if (!attr) {
    const int fast = (int)(sizeof(PairRec) * KRPT + (sizeof(float) + sizeof(int)) * KPMAX * KT);
    const int exact =
        (int)(sizeof(PairRec) * KRPT + (sizeof(double) + sizeof(int)) * G6_KNN_MAX * KT);
    if (cudaFuncSetAttribute(knn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fast) !=
            cudaSuccess ||
        cudaFuncSetAttribute(knn_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             exact) != cudaSuccess)
      return -3;
    attr = true;
  }
  KArgs ka;
  ka.js = *js;
  ka.nj = nj;
  ka.ni = ni;
  ka.k = k;
  ka.kp = knn_kept(ni, nj, k);
  ka.nsplit = nsplit;
  ka.jsplit = jsplit;
  ka.slots = slots;
  ka.pos64 = reinterpret_cast<const double *>(p + L.pos64);
  ka.xmax = reinterpret_cast<const unsigned *>(p + L.xmax);
  ka.cand_d = reinterpret_cast<double *>(p + L.cand_d);
  ka.cand_s = reinterpret_cast<int *>(p + L.cand_s);
  ka.cand_n = reinterpret_cast<int *>(p + L.cand_n);
  ka.cand_f = reinterpret_cast<float *>(p + L.cand_f);
  ka.flag = reinterpret_cast<int *>(p + L.flag);
  ka.ids = ids;
  ka.d2 = d2;
  if (cudaMemsetAsync(p + L.xmax, 0, sizeof(unsigned), st) != cudaSuccess) return -3;
  knn_xmax_kernel<<<2 * g6k_sm_count(), 256, 0, st>>>(*js, nj,
                                                      reinterpret_cast<unsigned *>(p + L.xmax));
  knn_pos_kernel<<<(nj + 255) / 256, 256, 0, st>>>(*js, nj, t,
                                                   reinterpret_cast<double *>(p + L.pos64));
  const size_t smem_fast = sizeof(PairRec) * KRPT + (sizeof(float) + sizeof(int)) * ka.kp * KT;
  const size_t smem_exact = sizeof(PairRec) * KRPT + (sizeof(double) + sizeof(int)) * k * KT;
  const int gx = (ni + KT - 1) / KT;
  if (knn_use_cells(ni, nj)) {
    CArgs ca;
    ca.bits = knn_bits(nj);
    ca.ntile = (nj + CTJ - 1) / CTJ;
    ca.nj_pad = ca.ntile * CTJ;
    ca.nsuper = (ca.ntile + 31) / 32;
    ca.map = reinterpret_cast<float *>(p + L.map);
    ca.count = reinterpret_cast<int *>(p + L.count);
    ca.icount = reinterpret_cast<int *>(p + L.icount);
    ca.cell = reinterpret_cast<int *>(p + L.cell);
    ca.rank = reinterpret_cast<int *>(p + L.rank);
    ca.icell = reinterpret_cast<int *>(p + L.icell);
    ca.irank = reinterpret_cast<int *>(p + L.irank);
    ca.rec = reinterpret_cast<float *>(p + L.rec);
    ca.order = reinterpret_cast<int *>(p + L.order);
    ca.iorder = reinterpret_cast<int *>(p + L.iorder);
    ca.box = reinterpret_cast<CBox *>(p + L.box);
    ca.super = reinterpret_cast<CBox *>(p + L.super);
    const int cells = 1 << (3 * ca.bits);
    if (cudaMemsetAsync(ca.count, 0, 2 * (size_t)cells * sizeof(int), st) != cudaSuccess)
      return -3;
    knn_map_kernel<<<1, CMAP, 0, st>>>(*js, nj, ca.map);
    knn_hist_kernel<<<(nj + 255) / 256, 256, 0, st>>>(js->jp_split, nullptr, nj, ca.map, ca.bits,
                                                      ca.count, ca.cell, ca.rank);
    knn_hist_kernel<<<(ni + 255) / 256, 256, 0, st>>>(js->jp_split, slots, ni, ca.map, ca.bits,
                                                      ca.icount, ca.icell, ca.irank);
    knn_scan_kernel<<<2, 1024, 0, st>>>(ca.count, ca.icount, cells);
    const int np = ca.nj_pad > ni ? ca.nj_pad : ni;
    knn_place_kernel<<<(np + 255) / 256, 256, 0, st>>>(ka, ca);
    knn_box_kernel<<<(ca.ntile + 7) / 8, 256, 0, st>>>(ca, 0);
    knn_box_kernel<<<(ca.nsuper + 7) / 8, 256, 0, st>>>(ca, 1);
    const int grid = (ni + 32 * CW - 1) / (32 * CW);
    switch (ka.kp) {
      case 12: knn_cells_kernel<12><<<grid, 32 * CW, 0, st>>>(ka, ca); break;
      case 16: knn_cells_kernel<16><<<grid, 32 * CW, 0, st>>>(ka, ca); break;
      case 20: knn_cells_kernel<20><<<grid, 32 * CW, 0, st>>>(ka, ca); break;
      case 28: knn_cells_kernel<28><<<grid, 32 * CW, 0, st>>>(ka, ca); break;
      default: knn_cells_kernel<KPMAX><<<grid, 32 * CW, 0, st>>>(ka, ca); break;
    }
  } else {
    knn_kernel<<<dim3(gx, nsplit), KT, smem_fast, st>>>(ka);
  }
  knn_merge_kernel<<<(ni + 127) / 128, 128, 0, st>>>(ka);
  knn_exact_kernel<<<gx, KT, smem_exact, st>>>(ka);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
