// ob2_serve.cu -- the solve-serving engine (include/ops_b200_serve.h).
//
// Device state: an array of request slots (struct Req, FP64 CG scalars
// included) and a work list (struct Work) naming the active requests with
// prefix sums of their work units.  One call of ob2s_run is
//   pois_iterate  one cooperative launch that runs all the iterations of the
//                 Poisson and heat requests: every CTA owns a run of tiles of
//                 the work list; per iteration p' = r + beta p, w = A p' and
//                 per-tile (p', w), a grid barrier, x += alpha p', r -= alpha
//                 w and per-tile (r, r) (or the FP64 residual b - A x), a
//                 grid barrier.  Each CTA forms alpha, beta and the state
//                 changes of its own requests from all their tile partials,
//                 in a fixed order, so that all CTAs of a request agree;
//   adi_x/y/z     three launches per ADI step: right-hand side and x solve,
//                 y solve, z solve added into u (chunks in registers, PCR
//                 among the lanes of a line), then adi_count once.
// All kernels read the work list from device memory.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "../device/ob2_trid.cuh"
#include "ops_b200_serve.h"

namespace {

using namespace ob2t;

constexpr int TX = 32;       // CTA x extent (one warp per row of a tile)
constexpr int TXC = 2 * TX;  // columns per tile: two adjacent columns per thread
constexpr int C0 = 2;        // storage column of interior column 0 (even: 2-column
                             // accesses are 8- or 16-byte aligned)
constexpr int MAXA = OB2S_MAX_ACTIVE;
constexpr int ADI_MAX_N = 192;  // 32 lanes x 6 points
constexpr int ADI_CL = 6;       // points per chunk of a line
// (OB2S_HEAT2D is declared in ops_b200_serve.h)
constexpr double kHeatRho = 1.0;  // heat requests: dt / h^2 of the implicit step

struct Req {
  int kind, n, pitch, tiles_x, tiles;
  int ry;   // 2D: rows per thread of a tile (1, 2 or 4); ADI: lanes per line (8, 16 or 32)
  int phase, done, outer, inner_it, iters;
  int max_inner, max_outer, steps, step;
  int par;  // p buffer parity
  int newstep;  // heat: the next residual pass starts a time step (b = x)
  double tol, inner_tol;
  double alpha, beta, gamma, gamma_in0, rr0, rel;
  double diag, off;  // heat operator: diag x - off (sum of the 4 neighbours)
  double *x, *b, *part;
  void *r, *w, *p0, *p1;
  double *u, *du;
  double lambda;
};

struct Work {
  int npois, nadi;
  int pois_slot[MAXA];
  int adi_slot[MAXA];
  long long pois_pref[MAXA + 1];
  long long adi_pref[MAXA + 1];
};

__device__ __forceinline__ int find_req(const long long *pref, int n, long long u) {
  int lo = 0, hi = n;  // pref[lo] <= u < pref[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pref[mid] <= u)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ double hash_uniform(int seed, int i, int j, int k) {
  unsigned long long z = ((unsigned long long)(unsigned)seed << 42) ^
                         ((unsigned long long)(unsigned)i << 21) ^ (unsigned long long)(unsigned)j ^
                         ((unsigned long long)(unsigned)k << 52);
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  z = z ^ (z >> 31);
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// ---------------------------------------------------------------- Poisson
// Layout of a 2D request's arrays: rows -1 .. n (the zero halo rows) at
// storage rows 0 .. n+1, row pitch P even and at least n + 3, interior
// column i at storage column i + C0 (column -1, the left halo, at C0 - 1;
// column n, the right halo, at n + C0); every unused element is zero.
// A tile is worked on by a group of 32 x 8 threads; each thread handles two
// adjacent columns (one 8- or 16-byte access per array and row) and RY
// consecutive rows, so a tile is 64 x (8 RY) points.  Loads of out-of-range
// rows are clamped to the last interior row (always valid memory) and only
// the stores are guarded, so the loads of all RY rows are issued before any
// store.
//
// Poisson and heat requests: conjugate gradients (the standard
// two-reduction form) with the iterate x in FP64, the vectors r, w, p in TI
// (FP32 in the mixed mode, FP64 otherwise) and every dot product accumulated
// in FP64.  Poisson: A x = 4 x - (neighbours); heat (one backward-Euler step
// per solve, dt / h^2 = rho): A x = (1 + 4 rho) x - rho (neighbours), b the
// previous step's solution.  The recursive residual is replaced by the true
// one, b - A x computed in FP64, whenever it has dropped by inner_tol since
// the last true residual or meets the tolerance (reliable updates: the
// search direction is kept, so the Krylov convergence of FP64 CG is kept
// too; an FP32 iterate or an FP32 correction accumulated between
// replacements needs far more iterations on fine grids: 10575 instead of
// 5781 at 2048^2, measured).
// Phases:
//   0  start (and restart after a breakdown; for heat requests also the start
//      of each time step, which first sets b = x): r = b - A x in FP64
//   2  CG iteration: p' = r + beta p, w = A p', (p', w)   [pw_tile]
//                    alpha = gamma / (p', w)               [form_alpha]
//                    x += alpha p', r -= alpha w, (r, r)   [xr_tile]
//                    beta, gamma; replacement test         [advance]
//   3  replacement: r = b - A x in FP64, convergence test on it; beta from
//      the true (r, r), p kept
// p is double-buffered (p[par] read, p[par ^ 1] written by pw_tile), since
// pw_tile forms p' of the stencil neighbours itself: w = A p' needs p' at
// the neighbours, and recomputing r + beta p there avoids a separate pass.

constexpr int CTA_Y = 8;
// partial sums per tile: (p', w), (r, r) and, at a heat request's new time
// step, ||b||^2.  The last has a column of its own: it is read after the same
// barrier as (r, r), and a CTA that is done with it goes on to write (p', w)
// while the others still read.
constexpr int NPART = 3;

// two adjacent elements of type T
template <typename T> struct V2;
template <> struct V2<float> { typedef float2 type; };
template <> struct V2<double> { typedef double2 type; };
template <typename T>
__device__ __forceinline__ typename V2<T>::type ld2(const T *p) {
  return *(const typename V2<T>::type *)p;
}
template <typename T>
__device__ __forceinline__ void st2(T *p, T a, T b) {
  typename V2<T>::type v;
  v.x = a;
  v.y = b;
  *(typename V2<T>::type *)p = v;
}

// Groups of 256 threads per CTA, one CTA per SM: 4 for FP32 vectors (64
// registers a thread), 3 for FP64 ones, whose two columns of RY rows need
// more than 64
constexpr int GT = TX * CTA_Y;  // threads of a group
template <typename TI>
__host__ __device__ constexpr int pois_groups() {
  return sizeof(TI) == 8 ? 3 : 4;
}

// a group's own barrier (every group of the CTA takes its tiles at its pace)
__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(GT) : "memory");
}

// fixed-order sum over a group of NV values per thread; result in thread 0
template <int NV>
__device__ __forceinline__ void group_sum(double (&v)[NV], double (*sh)[CTA_Y], int g) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < NV; c++) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
  const int t = threadIdx.x % GT;
  if ((t & 31) == 0)
#pragma unroll
    for (int c = 0; c < NV; c++) sh[c][t >> 5] = v[c];
  group_sync(g);
  if (t == 0)
#pragma unroll
    for (int c = 0; c < NV; c++) {
      double a = 0.0;
      for (int k = 0; k < CTA_Y; k++) a += sh[c][k];
      v[c] = a;
    }
  group_sync(g);
}

// fixed-order CTA sum of NV values per thread; result in thread 0
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sh)[32]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < NV; c++) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
  const int t = threadIdx.x + blockDim.x * threadIdx.y;
  const int nw = (blockDim.x * blockDim.y + 31) >> 5;
  if ((t & 31) == 0)
#pragma unroll
    for (int c = 0; c < NV; c++) sh[c][t >> 5] = v[c];
  __syncthreads();
  if (t == 0)
#pragma unroll
    for (int c = 0; c < NV; c++) {
      double a = 0.0;
      for (int k = 0; k < nw; k++) a += sh[c][k];
      v[c] = a;
    }
  __syncthreads();
}

// What the CTAs that work on a request keep of it in shared memory: its
// arrays and operator (constant), and its CG state, which each of them
// advances by itself from the same partial sums.
struct Pois {
  int kind, n, pitch, tiles_x, tiles, ry;
  int phase, done, outer, iters, step, par, newstep;
  int max_inner, max_outer, steps;
  double tol, inner_tol, diag, off;
  double alpha, beta, gamma, gamma_in0, rr0, rel;
  double *x, *b, *part;
  void *r, *w, *p0, *p1;
};

// p' = r + beta p and w = A p' over tile t, (p', w) of the tile (phase 2)
template <typename TI, int RY>
__device__ __forceinline__ void pw_tile(const Pois &q, int t, int g, double (*sh)[CTA_Y]) {
  const int lane = threadIdx.x % TX, ty = threadIdx.x % GT / TX;
  const int n = q.n, P = q.pitch;
  const int i = (t % q.tiles_x) * TXC + 2 * lane;  // columns i, i + 1
  const int j0 = (t / q.tiles_x) * (CTA_Y * RY) + ty * RY;
  double v[1] = {0.0};
  if (j0 < n) {  // uniform over the warp (one row of a tile per warp)
    const TI *rr = (const TI *)q.r;
    const TI *pin = (const TI *)(q.par ? q.p1 : q.p0);
    TI *pout = (TI *)(q.par ? q.p0 : q.p1);
    TI *ww = (TI *)q.w;
    const TI beta = (TI)q.beta;
    const bool in0 = i < n, in1 = i + 1 < n;
    const int ic = in0 ? i : ((n - 1) & ~1);  // lanes past the edge load valid memory
    // p' = r + beta p on rows j0-1 .. j0+RY of columns i, i+1 (storage rows
    // clamped into the array; the halo rows and columns of r and p hold
    // zeros); a column past the right edge stands for the zero halo
    TI p0[RY + 2], p1[RY + 2];
    int o[RY + 2];  // (n + 2) P < 2^31 for n <= 32768
#pragma unroll
    for (int m = 0; m < RY + 2; m++) {
      o[m] = (min(j0 + m - 1, n) + 1) * P + ic + C0;
      const auto rv = ld2(rr + o[m]);
      const auto pv = ld2(pin + o[m]);
      p0[m] = in0 ? rv.x + beta * pv.x : (TI)0;
      p1[m] = in1 ? rv.y + beta * pv.y : (TI)0;
    }
#pragma unroll
    for (int m = 0; m < RY; m++) {
      // column i - 1 is the left lane's second column, column i + 2 the
      // right lane's first; the warp's edge lanes form theirs from memory
      // (the same arithmetic, same bits)
      TI pw = __shfl_up_sync(0xffffffffu, p1[m + 1], 1);
      TI pe = __shfl_down_sync(0xffffffffu, p0[m + 1], 1);
      if (lane == 0) pw = rr[o[m + 1] - 1] + beta * pin[o[m + 1] - 1];
      if (lane == TX - 1 && in1) pe = rr[o[m + 1] + 2] + beta * pin[o[m + 1] + 2];
      if (!in0 || j0 + m >= n) continue;
      const TI c0 = p0[m + 1], c1 = p1[m + 1];
      TI a0, a1;
      if (q.kind == OB2S_HEAT2D) {
        a0 = (TI)q.diag * c0 - (TI)q.off * (pw + c1 + p0[m] + p0[m + 2]);
        a1 = in1 ? (TI)q.diag * c1 - (TI)q.off * (c0 + pe + p1[m] + p1[m + 2]) : (TI)0;
      } else {
        a0 = (TI)4 * c0 - pw - c1 - p0[m] - p0[m + 2];
        a1 = in1 ? (TI)4 * c1 - c0 - pe - p1[m] - p1[m + 2] : (TI)0;
      }
      // column n (the right halo) gets zeros when i + 1 == n
      st2(pout + o[m + 1], c0, c1);
      st2(ww + o[m + 1], a0, a1);
      v[0] += (double)c0 * (double)a0 + (double)c1 * (double)a1;
    }
  }
  group_sum<1>(v, sh, g);
  if (threadIdx.x % GT == 0) q.part[NPART * t] = v[0];
}

// phase 2: x += alpha p' (FP64), r -= alpha w, (r, r); phases 0, 3:
// r = b - A x in FP64 and its (r, r).  Column n (the right halo) is written
// only with zeros: there p', w and r are zero, so x keeps its zero.
template <typename TI, int RY>
__device__ __forceinline__ void xr_tile(const Pois &q, int t, int g, double (*sh)[CTA_Y]) {
  const int lane = threadIdx.x % TX, ty = threadIdx.x % GT / TX;
  const int ph = q.phase;
  const int n = q.n, P = q.pitch;
  const int i = (t % q.tiles_x) * TXC + 2 * lane;  // columns i, i + 1
  const int j0 = (t / q.tiles_x) * (CTA_Y * RY) + ty * RY;
  double v[2] = {0.0, 0.0};
  if (i < n && j0 < n) {
    const bool in1 = i + 1 < n;
    int o[RY];  // (n + 2) P < 2^31 for n <= 32768
#pragma unroll
    for (int m = 0; m < RY; m++) o[m] = (min(j0 + m, n - 1) + 1) * P + i + C0;
    TI *rr = (TI *)q.r;
    double *x = q.x;
    if (ph == 2) {
      const TI *pn = (const TI *)(q.par ? q.p0 : q.p1);  // written by pw_tile
      const TI *ww = (const TI *)q.w;
      const double alpha64 = q.alpha;
      const TI alpha = (TI)q.alpha;
      double x0[RY], x1[RY];
      TI r0[RY], r1[RY];
#pragma unroll
      for (int m = 0; m < RY; m++) {
        const auto pv = ld2(pn + o[m]);
        const auto wv = ld2(ww + o[m]);
        const auto rv = ld2(rr + o[m]);
        const double2 xv = ld2(x + o[m]);
        x0[m] = xv.x + alpha64 * (double)pv.x;
        x1[m] = xv.y + alpha64 * (double)pv.y;
        r0[m] = rv.x - alpha * wv.x;
        r1[m] = rv.y - alpha * wv.y;
      }
#pragma unroll
      for (int m = 0; m < RY; m++) {
        if (j0 + m >= n) continue;
        st2(x + o[m], x0[m], x1[m]);
        st2(rr + o[m], r0[m], r1[m]);
        v[0] += (double)r0[m] * (double)r0[m] + (double)r1[m] * (double)r1[m];
      }
    } else {
      double *b = q.b;
      double s0[RY], s1[RY];
#pragma unroll
      for (int m = 0; m < RY; m++) {
        const int e = o[m];
        const double2 c = ld2(x + e), up = ld2(x + e - P), dn = ld2(x + e + P);
        const double xw = x[e - 1], xe = x[e + 2];
        double2 bv = ld2(b + e);
        if (q.kind == OB2S_HEAT2D) {
          if (q.newstep) {  // a new time step: its right-hand side is the last solution
            bv = c;
            if (j0 + m < n) {
              st2(b + e, bv.x, bv.y);
              v[1] += bv.x * bv.x + bv.y * bv.y;  // ||b||^2: the step's residuals are relative to it
            }
          }
          s0[m] = bv.x - (q.diag * c.x - q.off * (xw + c.y + up.x + dn.x));
          s1[m] = in1 ? bv.y - (q.diag * c.y - q.off * (c.x + xe + up.y + dn.y)) : 0.0;
        } else {
          s0[m] = bv.x - (4.0 * c.x - xw - c.y - up.x - dn.x);
          s1[m] = in1 ? bv.y - (4.0 * c.y - c.x - xe - up.y - dn.y) : 0.0;
        }
      }
#pragma unroll
      for (int m = 0; m < RY; m++) {
        if (j0 + m >= n) continue;
        st2(rr + o[m], (TI)s0[m], (TI)s1[m]);
        v[0] += s0[m] * s0[m] + s1[m] * s1[m];
      }
    }
  }
  group_sum<2>(v, sh, g);
  if (threadIdx.x % GT == 0) {
    q.part[NPART * t + 1] = v[0];
    if (ph == 0 && q.newstep) q.part[NPART * t + 2] = v[1];
  }
}

// a group's fixed-order sum of one partial column of a request (in thread 0)
__device__ __forceinline__ double request_sum(const Pois &q, int col, double (*sh)[CTA_Y], int g) {
  double v[1] = {0.0};
  for (int t = threadIdx.x % GT; t < q.tiles; t += GT) v[0] += q.part[NPART * t + col];
  group_sum<1>(v, sh, g);
  return v[0];
}

// alpha = gamma / (p', w) of a request in phase 2
__device__ __forceinline__ void form_alpha(Pois &q, double (*sh)[CTA_Y], int g) {
  if (q.done || q.phase != 2) return;  // uniform over the group
  const double pw = request_sum(q, 0, sh, g);
  if (threadIdx.x % GT != 0) return;
  if (!(pw > 0.0))  // breakdown: xr_tile computes the true residual and
    q.phase = 0;    // advance restarts from it with beta = 0
  else
    q.alpha = q.gamma / pw;
}

// the (r, r) step of a request
__device__ __forceinline__ void advance(Pois &q, double (*sh)[CTA_Y], int grp) {
  if (q.done) return;
  const int ph = q.phase;
  const bool newstep = ph == 0 && q.newstep;  // uniform over the group
  const double g = request_sum(q, 1, sh, grp);
  const double bb = newstep ? request_sum(q, 2, sh, grp) : 0.0;
  if (threadIdx.x % GT != 0) return;
  if (ph == 0 || ph == 3) {  // g = (b - A x, b - A x) in FP64
    if (newstep) {  // heat: relative to the step's right-hand side
      q.rr0 = bb;
      q.newstep = 0;
    } else if (q.outer == 0) {
      q.rr0 = g;  // Poisson starts from x = 0: (b, b)
    }
    q.outer++;
    q.rel = q.rr0 > 0.0 ? sqrt(g / q.rr0) : 0.0;
    if (q.rel <= q.tol || q.outer > q.max_outer || q.iters >= q.max_inner) {
      if (q.kind == OB2S_HEAT2D && q.rel <= q.tol && q.step + 1 < q.steps) {
        q.step++;  // next backward-Euler step, from this solution
        q.newstep = 1;
        q.outer = 0;
        q.phase = 0;
        return;
      }
      q.done = 1;
      return;
    }
    q.beta = ph == 0 ? 0.0 : g / q.gamma;
    q.gamma = g;
    q.gamma_in0 = g;
    q.phase = 2;
    return;
  }
  q.iters++;
  q.par ^= 1;
  const double drop = sqrt(g / q.gamma_in0);
  const double relr = q.rr0 > 0.0 ? sqrt(g / q.rr0) : 0.0;
  if (drop <= q.inner_tol || relr <= q.tol || q.iters >= q.max_inner || g == 0.0) {
    q.phase = 3;  // gamma stays the previous (r, r) for beta
    return;
  }
  q.beta = g / q.gamma;
  q.gamma = g;
}

// Grid barrier of a cooperative launch.  bar[0] counts arrivals for the
// engine's life (`target` is its value, modulo 2^32, when all CTAs of this
// barrier have arrived; a CTA still here sees less than a grid's arrivals
// more).  The wait is bounded: the first CTA that gives up sets bar[1] and
// adds kGaveUp to the count, which every other one finds in the word that it
// polls anyway and gives up too.  False in every thread when the barrier
// failed.
constexpr unsigned kPolls = 1u << 22;  // of some 0.5 us: seconds
constexpr unsigned kGaveUp = 1u << 30;
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned target, unsigned polls,
                                             int *ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int over = -1;  // arrivals beyond the target
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    for (unsigned k = 0; k < polls && over < 0; k++) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      over = (int)(seen - target);
    }
    if (over < 0 && atomicExch(bar + 1, 1u) == 0) atomicAdd(bar, kGaveUp);
    *ok = over >= 0 && over < (int)(kGaveUp / 2);
  }
  __syncthreads();
  return *ok != 0;
}

template <typename TI>
__device__ __forceinline__ void pw_any(const Pois &q, int t, int g, double (*sh)[CTA_Y]) {
  switch (q.ry) {  // uniform over the group
    case 1: pw_tile<TI, 1>(q, t, g, sh); break;
    case 2: pw_tile<TI, 2>(q, t, g, sh); break;
    default: pw_tile<TI, 4>(q, t, g, sh);
  }
}
template <typename TI>
__device__ __forceinline__ void xr_any(const Pois &q, int t, int g, double (*sh)[CTA_Y]) {
  switch (q.ry) {
    case 1: xr_tile<TI, 1>(q, t, g, sh); break;
    case 2: xr_tile<TI, 2>(q, t, g, sh); break;
    default: xr_tile<TI, 4>(q, t, g, sh);
  }
}

// `iters` iterations of every Poisson and heat request in one cooperative
// launch of one CTA per SM.  CTA c owns tiles [c T / G, (c + 1) T / G) of the
// work list's T, so it meets few requests; its groups take the tiles in turn.
//
// Latency-bound: the requests' vectors live in L2 and a 640^2 request's pass
// is 1 to 2 us of work, so what counts is what lies between the passes: two
// grid barriers per iteration in place of four kernel boundaries and two
// one-CTA-per-request scalar kernels.
//
// A request's partial sums of column 0 (columns 1 and 2) are written by
// pw_tile (xr_tile) before a barrier and read by form_alpha (advance) after
// it; between the reads and the next write of a column lies the iteration's
// other barrier.
template <typename TI>
__global__ void __launch_bounds__(GT * pois_groups<TI>(), 1) pois_iterate(
    const Work *__restrict__ W, Req *R, int iters, unsigned *bar, unsigned base, unsigned polls) {
  constexpr int NG = pois_groups<TI>();
  __shared__ double shs[NG][2][CTA_Y];
  __shared__ int ok;
  extern __shared__ Pois qs[];  // this CTA's requests
  const int g = threadIdx.x / GT;
  const long long total = W->pois_pref[W->npois];
  const long long t0 = total * blockIdx.x / gridDim.x, t1 = total * (blockIdx.x + 1) / gridDim.x;
  const int k0 = t1 > t0 ? find_req(W->pois_pref, W->npois, t0) : 0;
  const int nk = t1 > t0 ? find_req(W->pois_pref, W->npois, t1 - 1) - k0 + 1 : 0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    const Req &r = R[W->pois_slot[k0 + k]];
    Pois &q = qs[k];
    q.kind = r.kind; q.n = r.n; q.pitch = r.pitch; q.tiles_x = r.tiles_x; q.tiles = r.tiles;
    q.ry = r.ry; q.phase = r.phase; q.done = r.done; q.outer = r.outer; q.iters = r.iters;
    q.step = r.step; q.par = r.par; q.newstep = r.newstep; q.max_inner = r.max_inner;
    q.max_outer = r.max_outer; q.steps = r.steps; q.tol = r.tol; q.inner_tol = r.inner_tol;
    q.diag = r.diag; q.off = r.off; q.alpha = r.alpha; q.beta = r.beta; q.gamma = r.gamma;
    q.gamma_in0 = r.gamma_in0; q.rr0 = r.rr0; q.rel = r.rel; q.x = r.x; q.b = r.b;
    q.part = r.part; q.r = r.r; q.w = r.w; q.p0 = r.p0; q.p1 = r.p1;
  }
  __syncthreads();
  double(*sh)[CTA_Y] = shs[g];
  for (int it = 0; it < iters; it++) {
    for (long long u = t0 + g; u < t1; u += NG) {
      const int k = nk == 1 ? k0 : find_req(W->pois_pref, W->npois, u);
      const Pois &q = qs[k - k0];
      if (!q.done && q.phase == 2) pw_any<TI>(q, (int)(u - W->pois_pref[k]), g, sh);
    }
    base += gridDim.x;
    if (!grid_barrier(bar, base, polls, &ok)) return;
    for (int k = g; k < nk; k += NG) form_alpha(qs[k], sh, g);
    __syncthreads();
    // backwards: what pw_tile wrote last is still in L2, and the next pass
    // begins where this one ends (requests larger than L2, us per iteration:
    // 4 of 2048^2 FP64 265 -> 257, mixed 170 -> 164; 8 of 1024^2 142 -> 135
    // and 92 -> 86)
    for (long long u = t1 - 1 - (t1 - t0 + NG - 1 - g) % NG; u >= t0; u -= NG) {
      const int k = nk == 1 ? k0 : find_req(W->pois_pref, W->npois, u);
      const Pois &q = qs[k - k0];
      if (!q.done) xr_any<TI>(q, (int)(u - W->pois_pref[k]), g, sh);
    }
    base += gridDim.x;
    if (!grid_barrier(bar, base, polls, &ok)) return;
    for (int k = g; k < nk; k += NG) advance(qs[k], sh, g);
    __syncthreads();
  }
  // the CTA with a request's first tile writes its state back
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    if (W->pois_pref[k0 + k] < t0) continue;
    Req &r = R[W->pois_slot[k0 + k]];
    const Pois &q = qs[k];
    r.phase = q.phase; r.done = q.done; r.outer = q.outer; r.iters = q.iters; r.step = q.step;
    r.par = q.par; r.newstep = q.newstep; r.alpha = q.alpha; r.beta = q.beta; r.gamma = q.gamma;
    r.gamma_in0 = q.gamma_in0; r.rr0 = q.rr0; r.rel = q.rel;
  }
}

// ---------------------------------------------------------------- ADI
// grid of n^3 points including the Dirichlet boundary (adi/preproc_kernel.h):
// a = c = -lambda / 2, b = 1 + lambda inside, identity rows on the boundary.
// A line of n points is L lanes (Req::ry: 8, 16 or 32, the fewest that hold
// it) with chunks of ADI_CL points in registers, the chunk ends solved among
// the lanes (ob2_trid.cuh); a CTA of 256 threads is a unit of 256 / L lines.
// One launch per direction: one thread per line and a sequential recurrence
// took 80 to 130 us for seven requests of 32^3 to 160^3, too few threads to
// cover its latency.

// the chunk's coefficients (rows k0 .. of a line of n), then its end rows
// reduced over the line's lanes: x_last of the chunk is D, its first is
// returned in xf
template <int L>
__device__ __forceinline__ void adi_line(double (&a)[ADI_CL], double (&c)[ADI_CL],
                                         double (&d)[ADI_CL], int k0, int n, bool edge,
                                         double lambda) {
  double b[ADI_CL];
#pragma unroll
  for (int i = 0; i < ADI_CL; i++) {
    const int k = k0 + i;
    const bool in = k > 0 && k < n - 1 && !edge;
    a[i] = c[i] = in ? -0.5 * lambda : 0.0;
    b[i] = in ? 1.0 + lambda : 1.0;
  }
  chunk_reduce<ADI_CL>(a, b, c, d);
}

// right-hand side lambda * (7-point Laplacian of u), then the x solve; the
// solution in du
template <int L>
__device__ __forceinline__ void adi_x_unit(const Req &q, long long line) {
  const int n = q.n, lane = threadIdx.x % L, k0 = lane * ADI_CL;
  const bool active = line < (long long)n * n;
  const int y = active ? (int)(line % n) : 0, z = active ? (int)(line / n) : 0;
  const bool edge = y == 0 || y == n - 1 || z == 0 || z == n - 1;
  const long long sy = n, sz = (long long)n * n, o = z * sz + y * sy + k0;
  const double *u = q.u;
  const bool whole = active && k0 + ADI_CL <= n;
  double a[ADI_CL], c[ADI_CL], d[ADI_CL];
  if (whole && !edge) {
    double m[ADI_CL], n1[ADI_CL], n2[ADI_CL], n3[ADI_CL], n4[ADI_CL];
    load_chunk<double, ADI_CL>(u + o, m);
    load_chunk<double, ADI_CL>(u + o - sy, n1);
    load_chunk<double, ADI_CL>(u + o + sy, n2);
    load_chunk<double, ADI_CL>(u + o - sz, n3);
    load_chunk<double, ADI_CL>(u + o + sz, n4);
    const double lo = k0 > 0 ? u[o - 1] : 0.0, hi = k0 + ADI_CL < n ? u[o + ADI_CL] : 0.0;
#pragma unroll
    for (int i = 0; i < ADI_CL; i++) {
      const double w = i > 0 ? m[i > 0 ? i - 1 : 0] : lo, e = i < ADI_CL - 1 ? m[i < ADI_CL - 1 ? i + 1 : 0] : hi;
      d[i] = q.lambda * (w + e + n1[i] + n2[i] + n3[i] + n4[i] - 6.0 * m[i]);
      if (k0 + i == 0 || k0 + i == n - 1) d[i] = 0.0;
    }
  } else {
#pragma unroll
    for (int i = 0; i < ADI_CL; i++) {
      const int k = k0 + i;
      d[i] = 0.0;
      if (active && !edge && k > 0 && k < n - 1)
        d[i] = q.lambda * (u[o + i - 1] + u[o + i + 1] + u[o + i - sy] + u[o + i + sy] +
                           u[o + i - sz] + u[o + i + sz] - 6.0 * u[o + i]);
    }
  }
  adi_line<L>(a, c, d, k0, n, edge, q.lambda);
  double A, C, xl;
  group_reduce<L>(a[0], c[0], d[0], a[ADI_CL - 1], c[ADI_CL - 1], d[ADI_CL - 1], lane, A, C, xl);
  double xp = __shfl_up_sync(0xffffffffu, xl, 1, L);
  if (lane == 0) xp = 0.0;
  const double xf = d[0] - a[0] * xp - c[0] * xl;
  if (!active) return;
#pragma unroll
  for (int i = 0; i < ADI_CL; i++)
    d[i] = i == 0 ? xf : i == ADI_CL - 1 ? xl : d[i] - a[i] * xf - c[i] * xl;
  if (whole) {
    store_chunk<double, ADI_CL>(q.du + o, d);
  } else {
#pragma unroll
    for (int i = 0; i < ADI_CL; i++)
      if (k0 + i < n) q.du[o + i] = d[i];
  }
}

// y (DIR 1) or z (DIR 2) solve of 256 / L neighbouring lines in line-major
// order (runs of 256 / L elements along x); z adds its solution into u
template <int DIR, int L>
__device__ __forceinline__ void adi_s_unit(const Req &q, long long line0, double *sm) {
  constexpr int LPB = 256 / L, pitch = L + 1, field = LPB * pitch;
  const int n = q.n, tid = threadIdx.x, p = tid / LPB, l = tid % LPB, k0 = p * ADI_CL;
  const long long line = line0 + l, nn = (long long)n * n;
  const bool active = line < nn;
  const int x = active ? (int)(line % n) : 0, o = active ? (int)(line / n) : 0;  // o: z or y
  const bool edge = x == 0 || x == n - 1 || o == 0 || o == n - 1;
  const long long s = DIR == 1 ? n : nn;
  const long long base = (DIR == 1 ? o * nn : (long long)o * n) + x + k0 * s;
  const double *src = q.du;
  double a[ADI_CL], c[ADI_CL], d[ADI_CL];
#pragma unroll
  for (int i = 0; i < ADI_CL; i++) d[i] = active && k0 + i < n ? src[base + i * s] : 0.0;
  adi_line<L>(a, c, d, k0, n, edge, q.lambda);
  {
    double *e = sm + l * pitch + p;
    e[0] = a[0]; e[field] = c[0]; e[2 * field] = d[0];
    e[3 * field] = a[ADI_CL - 1]; e[4 * field] = c[ADI_CL - 1]; e[5 * field] = d[ADI_CL - 1];
  }
  __syncthreads();
  {
    const int lane = tid % L;
    double *e = sm + (tid / L) * pitch + lane;
    const double a0 = e[0], c0 = e[field], d0 = e[2 * field];
    double A, C, xl;
    group_reduce<L>(a0, c0, d0, e[3 * field], e[4 * field], e[5 * field], lane, A, C, xl);
    double xp = __shfl_up_sync(0xffffffffu, xl, 1, L);
    if (lane == 0) xp = 0.0;
    e[2 * field] = d0 - a0 * xp - c0 * xl;  // this lane's own slots
    e[5 * field] = xl;
  }
  __syncthreads();
  const double xf = sm[2 * field + l * pitch + p], xl = sm[5 * field + l * pitch + p];
  __syncthreads();  // the next unit overwrites the slots
  if (!active) return;
#pragma unroll
  for (int i = 0; i < ADI_CL; i++)
    if (k0 + i < n) {
      const double v = i == 0 ? xf : i == ADI_CL - 1 ? xl : d[i] - a[i] * xf - c[i] * xl;
      if (DIR == 2)
        q.u[base + i * s] = q.u[base + i * s] + v;
      else
        q.du[base + i * s] = v;
    }
}

// solve along DIR (0 x, 1 y, 2 z) of every ADI request that has a step left
// after `it` more steps than its count
template <int DIR>
__global__ void __launch_bounds__(256, 3) adi_solve(const Work *__restrict__ W, Req *R, int it) {
  __shared__ double sm[DIR ? 6 * (256 + 32) : 1];
  const long long total = W->adi_pref[W->nadi];
  for (long long un = blockIdx.x; un < total; un += gridDim.x) {
    const int k = find_req(W->adi_pref, W->nadi, un);
    const Req &q = R[W->adi_slot[k]];
    if (q.step + it >= q.steps) continue;  // uniform over the CTA
    const int L = q.ry;
    const long long line0 = (un - W->adi_pref[k]) * (256 / L);
    if (DIR == 0) {
      const long long line = line0 + threadIdx.x / L;
      if (L == 8) adi_x_unit<8>(q, line);
      else if (L == 16) adi_x_unit<16>(q, line);
      else adi_x_unit<32>(q, line);
    } else {
      constexpr int D = DIR ? DIR : 1;
      if (L == 8) adi_s_unit<D, 8>(q, line0, sm);
      else if (L == 16) adi_s_unit<D, 16>(q, line0, sm);
      else adi_s_unit<D, 32>(q, line0, sm);
    }
  }
}

// the step counts after `steps` steps of each request (or all it had left)
__global__ void adi_count(const Work *__restrict__ W, Req *R, int steps) {
  const int k = threadIdx.x;
  if (k >= W->nadi) return;
  Req &q = R[W->adi_slot[k]];
  q.step = min(q.step + steps, q.steps);
  q.iters = q.step;
  if (q.step >= q.steps) q.done = 1;
}

// ---------------------------------------------------------------- init

__global__ void pois_init(double *b, int n, int pitch, int seed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (i >= n) return;
  const double h = 1.0 / (n + 1);
  b[(long long)(j + 1) * pitch + i + C0] = h * h * (2.0 * hash_uniform(seed, i, j, 0) - 1.0);
}

// heat request: u0 ~ U(-1,1) into b and x
__global__ void heat_init(double *b, double *x, int n, int pitch, int seed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (i >= n) return;
  const double v = 2.0 * hash_uniform(seed, i, j, 3) - 1.0;
  b[(long long)(j + 1) * pitch + i + C0] = v;
  x[(long long)(j + 1) * pitch + i + C0] = v;
}

__global__ void adi_init(double *u, int n, int seed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, z = blockIdx.z;
  if (i >= n) return;
  u[((long long)z * n + j) * n + i] = 2.0 * hash_uniform(seed, i, j, z + 1) - 1.0;
}

// rows [roff, roff + n) x columns [coff, coff + n) of src into dst (n x n)
__global__ void interior_copy(const double *src, double *dst, int n, int pitch, int roff,
                              int coff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (i >= n) return;
  dst[(long long)j * n + i] = src[(long long)(j + roff) * pitch + i + coff];
}

// checksum of a request's solution in a fixed order: CTA c of kSumCtas sums
// rows [c R / G, (c + 1) R / G) of the R rows of ncols elements (element
// (i, r) at off + r pitch + i), thread-strided, then block_sum; one CTA sums
// the partials in order
constexpr int kSumCtas = 256;
__global__ void __launch_bounds__(256) sum_rows(const double *src, long long nrows, int ncols,
                                                long long pitch, long long off, double *part) {
  __shared__ double sh[1][32];
  const long long G = gridDim.x, c = blockIdx.x;
  const long long r0 = nrows * c / G, r1 = nrows * (c + 1) / G;
  double v[1] = {0.0};
  for (long long r = r0; r < r1; r++)
    for (int i = threadIdx.x; i < ncols; i += blockDim.x) v[0] += src[off + r * pitch + i];
  block_sum<1>(v, sh);
  if (threadIdx.x == 0) part[c] = v[0];
}
__global__ void __launch_bounds__(256) sum_parts(const double *part, int np, double *out) {
  __shared__ double sh[1][32];
  double v[1] = {0.0};
  for (int k = threadIdx.x; k < np; k += blockDim.x) v[0] += part[k];
  block_sum<1>(v, sh);
  if (threadIdx.x == 0) *out = v[0];
}

}  // namespace

// ---------------------------------------------------------------- host side

struct ob2s_engine {
  int mode, tile_y;
  double tol, inner_tol;
  int max_inner;
  cudaStream_t st;
  int sms;
  Req *R_d;
  Work *W_d;
  Req *R;                   // host copy, pinned (refreshed after every run); slot MAXA
                            // holds the grid barrier's words
  std::vector<int> used;    // slot in use
  std::vector<int> active;  // slot is in the work list
  std::vector<int> reported;
  std::vector<void *> mem;  // per slot allocation
  std::vector<size_t> bytes;
  bool work_dirty;
  unsigned *bar_d;     // grid barrier of pois_iterate (arrivals, failure), in R_d's last slot
  unsigned bar_base;   // arrivals before the next launch
  unsigned polls;      // of a grid barrier before it gives up
  int failed;          // error of the run whose grid barrier gave up
  long long launches;
  // the requests' memory: a pool of the engine's own that keeps freed
  // memory mapped (a request admitted after another retired reuses its
  // pages instead of mapping new ones)
  cudaMemPool_t pool;
  double *sum_d;  // checksum scratch: kSumCtas partials and the result
};

static int rc(cudaError_t e) { return (int)e; }

static size_t elem_inner(int mode) { return mode == OB2S_MIXED ? 4 : 8; }

OB2_API size_t ob2s_request_bytes(int mode, int kind, int n) {
  if (kind == OB2S_POISSON2D || kind == OB2S_HEAT2D) {
    const size_t p = (size_t)((n + 4) & ~1) * (n + 2);  // pitch x rows
    const size_t tiles = (size_t)((n + TXC - 1) / TXC) * (size_t)((n + 7) / 8);  // smallest tile
    return p * (16 + 4 * elem_inner(mode)) + 8 * NPART * tiles + 4096;
  }
  return (size_t)n * n * n * 16 + (size_t)n * 16 + 4096;
}

static size_t pois_smem() { return sizeof(Pois) * MAXA; }

// `iters` iterations of the Poisson and heat requests
static cudaError_t launch_pois(ob2s_engine *e, int iters) {
  void *args[] = {&e->W_d, &e->R_d, &iters, &e->bar_d, &e->bar_base, &e->polls};
  const bool mixed = e->mode == OB2S_MIXED;
  const void *f = mixed ? (const void *)pois_iterate<float> : (const void *)pois_iterate<double>;
  const int threads = GT * (mixed ? pois_groups<float>() : pois_groups<double>());
  const cudaError_t err =
      cudaLaunchCooperativeKernel(f, dim3(e->sms), dim3(threads), args, pois_smem(), e->st);
  if (err != cudaSuccess) return err;
  e->bar_base += 2u * (unsigned)iters * (unsigned)e->sms;
  e->launches++;
  return cudaSuccess;
}

// `steps` steps of the ADI requests
static cudaError_t launch_adi(ob2s_engine *e, int steps) {
  for (int i = 0; i < steps; i++) {
    adi_solve<0><<<e->sms * 6, 256, 0, e->st>>>(e->W_d, e->R_d, i);
    adi_solve<1><<<e->sms * 6, 256, 0, e->st>>>(e->W_d, e->R_d, i);
    adi_solve<2><<<e->sms * 6, 256, 0, e->st>>>(e->W_d, e->R_d, i);
  }
  adi_count<<<1, MAXA, 0, e->st>>>(e->W_d, e->R_d, steps);
  e->launches += 3LL * steps + 1;
  return cudaGetLastError();
}

OB2_API int ob2s_create(ob2s_engine **out, int mode, double tol, double inner_tol, int max_inner,
                        int tile_y) {
  if (mode != OB2S_FP64 && mode != OB2S_MIXED) return OB2S_ERR_BADARG;
  if (tile_y == 0) tile_y = 32;
  if (tile_y != 8 && tile_y != 16 && tile_y != 32) return OB2S_ERR_BADARG;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return rc(err);
  ob2s_engine *e = new ob2s_engine();
  e->mode = mode;
  e->tile_y = tile_y;
  e->tol = tol;
  e->inner_tol = inner_tol;
  e->max_inner = max_inner > 0 ? max_inner : 100000;
  cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev);
  if ((err = cudaStreamCreateWithFlags(&e->st, cudaStreamNonBlocking)) != cudaSuccess ||
      (err = cudaMalloc(&e->R_d, sizeof(Req) * (MAXA + 1))) != cudaSuccess ||
      (err = cudaMallocHost(&e->R, sizeof(Req) * (MAXA + 1))) != cudaSuccess ||
      (err = cudaMalloc(&e->W_d, sizeof(Work))) != cudaSuccess ||
      // cleared on the engine's stream, which every later access is ordered
      // behind (it does not wait for the default stream, whose work may be
      // long in coming)
      (err = cudaMemsetAsync(e->R_d, 0, sizeof(Req) * (MAXA + 1), e->st)) != cudaSuccess ||
      (err = cudaMemsetAsync(e->W_d, 0, sizeof(Work), e->st)) != cudaSuccess ||
      (err = cudaFuncSetAttribute(mode == OB2S_MIXED ? (const void *)pois_iterate<float>
                                                     : (const void *)pois_iterate<double>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)pois_smem())) != cudaSuccess) {
    delete e;
    return rc(err);
  }
  e->bar_d = (unsigned *)(e->R_d + MAXA);
  e->bar_base = 0;
  e->polls = kPolls;
  if (const char *v = getenv("OB2S_BARRIER_POLLS")) e->polls = (unsigned)strtoul(v, nullptr, 10);
  e->failed = 0;
  {
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = ~0ULL;  // never return freed memory to the device
    if ((err = cudaMemPoolCreate(&e->pool, &props)) != cudaSuccess) {
      cudaStreamDestroy(e->st);
      cudaFree(e->R_d);
      cudaFree(e->W_d);
      cudaFreeHost(e->R);
      delete e;
      return rc(err);
    }
    cudaMemPoolSetAttribute(e->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if ((err = cudaMalloc(&e->sum_d, sizeof(double) * (kSumCtas + 1))) != cudaSuccess) {
      cudaMemPoolDestroy(e->pool);
      cudaStreamDestroy(e->st);
      cudaFree(e->R_d);
      cudaFree(e->W_d);
      cudaFreeHost(e->R);
      delete e;
      return rc(err);
    }
  }
  memset(e->R, 0, sizeof(Req) * (MAXA + 1));
  e->used.assign(MAXA, 0);
  e->active.assign(MAXA, 0);
  e->reported.assign(MAXA, 0);
  e->mem.assign(MAXA, nullptr);
  e->bytes.assign(MAXA, 0);
  e->work_dirty = true;
  e->launches = 0;
  *out = e;
  return 0;
}

OB2_API int ob2s_reserve(ob2s_engine *e, size_t bytes) {
  if (!e) return OB2S_ERR_BADARG;
  if (bytes == 0) return 0;
  void *m = nullptr;
  cudaError_t err = cudaMallocFromPoolAsync(&m, bytes, e->pool, e->st);
  if (err != cudaSuccess) {
    cudaGetLastError();  // too large for the device: not sticky, leave no trace
    return rc(err);
  }
  err = cudaFreeAsync(m, e->st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(e->st);
  return rc(err);
}

OB2_API void ob2s_destroy(ob2s_engine *e) {
  if (!e) return;
  cudaStreamSynchronize(e->st);
  for (int k = 0; k < MAXA; k++)
    if (e->mem[k]) cudaFreeAsync(e->mem[k], e->st);
  cudaStreamSynchronize(e->st);
  cudaFree(e->R_d);
  cudaFree(e->W_d);
  cudaFreeHost(e->R);
  cudaFree(e->sum_d);
  cudaMemPoolDestroy(e->pool);
  cudaStreamDestroy(e->st);
  delete e;
}

OB2_API int ob2s_submit(ob2s_engine *e, int kind, int n, int seed, int steps, int *id) {
  const bool grid2d = kind == OB2S_POISSON2D || kind == OB2S_HEAT2D;
  if (grid2d ? (n < 1 || n > 32768 || (kind == OB2S_HEAT2D && steps < 1))
             : (kind != OB2S_ADI3D || n < 3 || n > ADI_MAX_N || steps < 1))
    return OB2S_ERR_BADARG;
  if (e->failed) return e->failed;
  int slot = -1;
  for (int k = 0; k < MAXA; k++)
    if (!e->used[k]) {
      slot = k;
      break;
    }
  if (slot < 0) return OB2S_ERR_FULL;
  const size_t nb = ob2s_request_bytes(e->mode, kind, n);
  void *m = nullptr;
  cudaError_t err = cudaMallocFromPoolAsync(&m, nb, e->pool, e->st);
  if (err != cudaSuccess) return rc(err);
  if ((err = cudaMemsetAsync(m, 0, nb, e->st)) != cudaSuccess) {
    cudaFreeAsync(m, e->st);
    return rc(err);
  }
  Req q;
  memset(&q, 0, sizeof(q));
  q.kind = kind;
  q.n = n;
  char *c = (char *)m;
  auto take = [&c](size_t b) {
    char *p = c;
    c += (b + 255) / 256 * 256;
    return (void *)p;
  };
  if (grid2d) {
    q.pitch = (n + 4) & ~1;  // even, >= n + 3: columns 0 .. n + C0
    q.tiles_x = (n + TXC - 1) / TXC;
    q.ry = e->tile_y / CTA_Y;
    q.tiles = q.tiles_x * ((n + e->tile_y - 1) / e->tile_y);
    const size_t p = (size_t)q.pitch * (n + 2);
    const size_t ei = elem_inner(e->mode);
    // the layout ob2s_request_bytes counts (seven arrays, each rounded up to
    // 256 bytes: within its 4 KB slack)
    q.x = (double *)take(p * 8);
    q.b = (double *)take(p * 8);
    q.r = take(p * ei);
    q.w = take(p * ei);
    q.p0 = take(p * ei);
    q.p1 = take(p * ei);
    q.part = (double *)take((size_t)8 * NPART * q.tiles);
    if (kind == OB2S_HEAT2D) {  // backward Euler: (1 + 4 rho) x - rho (neighbours)
      q.diag = 1.0 + 4.0 * kHeatRho;
      q.off = kHeatRho;
      q.steps = steps;
      q.newstep = 1;  // the first step's right-hand side is u0 (= x)
    }
    q.tol = e->tol;
    q.inner_tol = e->inner_tol;
    q.max_inner = e->max_inner;
    q.max_outer = 1000;
  } else {
    q.u = (double *)take((size_t)n * n * n * 8);
    q.du = (double *)take((size_t)n * n * n * 8);
    q.ry = n <= 8 * ADI_CL ? 8 : n <= 16 * ADI_CL ? 16 : 32;
  }
  if ((size_t)(c - (char *)m) > nb) {  // cannot happen: the slack covers the rounding
    cudaFreeAsync(m, e->st);
    return OB2S_ERR_BADARG;
  }
  if (kind == OB2S_POISSON2D) {
    pois_init<<<dim3((n + 127) / 128, n), 128, 0, e->st>>>(q.b, n, q.pitch, seed);
  } else if (kind == OB2S_HEAT2D) {  // u0 is the first right-hand side and guess
    heat_init<<<dim3((n + 127) / 128, n), 128, 0, e->st>>>(q.b, q.x, n, q.pitch, seed);
  } else {
    q.lambda = 1.0;
    q.steps = steps;
    adi_init<<<dim3((n + 127) / 128, n, n), 128, 0, e->st>>>(q.u, n, seed);
  }
  err = cudaMemcpyAsync(e->R_d + slot, &q, sizeof(Req), cudaMemcpyHostToDevice, e->st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(e->st);
  if (err != cudaSuccess) {
    cudaFreeAsync(m, e->st);
    return rc(err);
  }
  err = cudaGetLastError();
  if (err != cudaSuccess) return rc(err);
  e->R[slot] = q;
  e->used[slot] = 1;
  e->active[slot] = 1;
  e->reported[slot] = 0;
  e->mem[slot] = m;
  e->bytes[slot] = nb;
  e->work_dirty = true;
  *id = slot;
  return 0;
}

static int upload_work(ob2s_engine *e) {
  Work w;
  memset(&w, 0, sizeof(w));
  for (int k = 0; k < MAXA; k++) {
    if (!e->active[k]) continue;
    const Req &q = e->R[k];
    if (q.kind != OB2S_ADI3D) {
      w.pois_slot[w.npois] = k;
      w.pois_pref[w.npois + 1] = w.pois_pref[w.npois] + q.tiles;
      w.npois++;
    } else {
      const int n = q.n;
      const int a = w.nadi;
      w.adi_slot[a] = k;
      const int lpu = 256 / q.ry;  // lines per unit
      w.adi_pref[a + 1] = w.adi_pref[a] + ((long long)n * n + lpu - 1) / lpu;
      w.nadi++;
    }
  }
  cudaError_t err = cudaMemcpyAsync(e->W_d, &w, sizeof(w), cudaMemcpyHostToDevice, e->st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(e->st);  // w is a stack object
  e->work_dirty = false;
  return rc(err);
}

OB2_API int ob2s_run(ob2s_engine *e, int iters, int *ids, int cap, int *n_done) {
  if (iters < 1) return OB2S_ERR_BADARG;
  *n_done = 0;
  if (e->failed) return e->failed;
  int err;
  if (e->work_dirty && (err = upload_work(e))) return err;
  bool pois = false;
  int adi = 0;  // most steps that an ADI request has left
  for (int k = 0; k < MAXA; k++) {
    if (!e->active[k]) continue;
    if (e->R[k].kind != OB2S_ADI3D)
      pois = true;
    else
      adi = std::max(adi, e->R[k].steps - e->R[k].step);
  }
  if (pois) {
    const cudaError_t ce = launch_pois(e, iters);
    if (ce != cudaSuccess) return rc(ce);
  }
  if (adi) {
    const cudaError_t ce = launch_adi(e, std::min(adi, iters));
    if (ce != cudaSuccess) return rc(ce);
  }
  cudaError_t ce = cudaMemcpyAsync(e->R, e->R_d, sizeof(Req) * (MAXA + 1), cudaMemcpyDeviceToHost,
                                   e->st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->st);
  if (ce != cudaSuccess) return rc(ce);
  // a grid barrier gave up: the CTAs stopped in different passes, so the
  // requests' arrays do not belong together and the barrier's count is off
  if (((const unsigned *)(e->R + MAXA))[1]) return e->failed = (int)cudaErrorLaunchTimeout;
  for (int k = 0; k < MAXA; k++) {
    if (!e->used[k] || !e->R[k].done) continue;
    if (e->active[k]) {
      e->active[k] = 0;
      e->work_dirty = true;
    }
    if (!e->reported[k]) {
      e->reported[k] = 1;
      if (*n_done < cap) ids[*n_done] = k;
      (*n_done)++;
    }
  }
  return 0;
}

OB2_API int ob2s_active(ob2s_engine *e) {
  int n = 0;
  for (int k = 0; k < MAXA; k++) n += e->active[k];
  return n;
}

OB2_API int ob2s_fetch(ob2s_engine *e, int id, double *host, size_t count) {
  if (id < 0 || id >= MAXA || !e->used[id]) return OB2S_ERR_BADARG;
  const Req &q = e->R[id];
  if (!q.done) return OB2S_ERR_NOTDONE;
  const int n = q.n;
  if (q.kind != OB2S_ADI3D) {
    if (count < (size_t)n * n) return OB2S_ERR_BADARG;
    double *tmp = nullptr;
    cudaError_t ce = cudaMallocFromPoolAsync(&tmp, (size_t)n * n * 8, e->pool, e->st);
    if (ce != cudaSuccess) return rc(ce);
    interior_copy<<<dim3((n + 127) / 128, n), 128, 0, e->st>>>(q.x, tmp, n, q.pitch, 1, C0);
    ce = cudaMemcpyAsync(host, tmp, (size_t)n * n * 8, cudaMemcpyDeviceToHost, e->st);
    cudaFreeAsync(tmp, e->st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->st);
    return rc(ce);
  }
  const size_t m = (size_t)n * n * n;
  if (count < m) return OB2S_ERR_BADARG;
  cudaError_t ce = cudaMemcpyAsync(host, q.u, m * 8, cudaMemcpyDeviceToHost, e->st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->st);
  return rc(ce);
}

OB2_API int ob2s_result_of(ob2s_engine *e, int id, ob2s_result *res) {
  if (id < 0 || id >= MAXA || !e->used[id]) return OB2S_ERR_BADARG;
  const Req &q = e->R[id];
  memset(res, 0, sizeof(*res));
  res->kind = q.kind;
  res->n = q.n;
  res->done = q.done;
  res->iterations = q.iters;
  res->outer = q.outer;
  res->rel_residual = q.rel;
  if (!q.done) return 0;
  const int n = q.n;
  if (q.kind != OB2S_ADI3D)  // interior rows 1 .. n, columns C0 .. C0 + n - 1
    sum_rows<<<kSumCtas, 256, 0, e->st>>>(q.x, n, n, q.pitch, (long long)q.pitch + C0, e->sum_d);
  else
    sum_rows<<<kSumCtas, 256, 0, e->st>>>(q.u, (long long)n * n, n, n, 0, e->sum_d);
  sum_parts<<<1, 256, 0, e->st>>>(e->sum_d, kSumCtas, e->sum_d + kSumCtas);
  double s = 0.0;
  cudaError_t ce = cudaMemcpyAsync(&s, e->sum_d + kSumCtas, sizeof(double),
                                   cudaMemcpyDeviceToHost, e->st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->st);
  if (ce != cudaSuccess) return rc(ce);
  res->checksum = s;
  return 0;
}

OB2_API int ob2s_release(ob2s_engine *e, int id) {
  if (id < 0 || id >= MAXA || !e->used[id]) return OB2S_ERR_BADARG;
  cudaError_t ce = cudaStreamSynchronize(e->st);
  if (ce != cudaSuccess) return rc(ce);
  if (e->active[id]) e->work_dirty = true;
  cudaFreeAsync(e->mem[id], e->st);
  e->mem[id] = nullptr;
  e->used[id] = 0;
  e->active[id] = 0;
  e->bytes[id] = 0;
  // the slot's device state is left as is: no kernel reads a slot that is
  // not in the work list, and the work list is rebuilt before the next run
  return 0;
}

OB2_API long long ob2s_launches(ob2s_engine *e) { return e->launches; }
