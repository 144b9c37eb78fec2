// ob2_trid.cu -- batched tridiagonal solves behind ops_tridMultiDimBatch(_Inc).
//
// The reference hands these to the external tridsolver library
// (ops/c/src/tridiag/ops_tridiag_cuda.cpp:96-251).  This backend solves them
// with its own register-blocked Thomas/PCR hybrid (after the chunked scheme
// published by Laszlo, Giles and Appleyard, "Manycore algorithms for batch
// scalar and block tridiagonal solvers", ACM TOMS 42(4), 2016):
//
//   * a line is cut into segments of W chunks of CL rows (one segment for
//     lines of up to 256 points), one thread per chunk, the chunk's
//     coefficients held in FP64 registers;
//   * each thread eliminates its chunk so that every row couples only to the
//     chunk's first and last unknowns ("modified Thomas", chunk_reduce);
//   * the chunk ends form a tridiagonal system of two unknowns per chunk,
//     solved by parallel cyclic reduction (PCR) among W lanes: all of them at
//     once (pair_pcr: double storage, one segment), or the last unknowns
//     alone after the first ones are substituted (group_reduce), with the
//     couplings to the neighbouring segments carried along;
//   * several segments: the ends of each segment, two equations in the ends
//     of its neighbours, are eliminated in order by one lane (segment_ends);
//   * each thread substitutes its chunk and writes the solution (or adds it
//     to u for the _Inc form, leaving d untouched).
//
// Unit-stride lines (x): trid_x_kernel, a segment per group of W lanes, the
// segments of a line in one CTA.  Strided lines (y, z): trid_s_kernel, 256 / W
// neighbouring lines per CTA, consecutive threads on the same chunk of
// neighbouring lines so that every warp access is contiguous runs along x,
// the segments of the lines in the CTAs of a cluster.  OB2_TRID_STRIDED=0
// selects the Thomas algorithm one thread per strided line instead
// (trid_thomas_kernel).  Each coefficient is read once and the solution
// written once: the DRAM traffic is the algorithmic 5 values per point (6 for
// _Inc).  Elimination is FP64 for double and float storage.  Every register
// array is indexed with compile-time indices only (a run-time index would
// move the arrays to local memory).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>

#include "ob2_trid.cuh"
#include "ops_b200_device.h"

namespace {

namespace cg = cooperative_groups;
using namespace ob2t;

constexpr int kThreads = 256;    // CTA size
constexpr int kMaxSeg = 16;      // segments of a line: lines of up to 4096 points
constexpr int kMaxLine = 4096;

// A segment's two end equations, from lane 0 (its first chunk's first row)
// and lane W-1 (its last chunk):
//   x_first = e[2] - e[0] XL - e[1] XF,   x_last = e[5] - e[3] XL - e[4] XF.
template <int W>
__device__ __forceinline__ void put_ends(double a0, double c0, double d0, double A, double C,
                                         double D, int lane, double *e) {
  if (lane == 0) {
    e[0] = a0 - c0 * A;
    e[1] = -c0 * C;
    e[2] = d0 - c0 * D;
  }
  if (lane == W - 1) {
    e[3] = A;
    e[4] = C;
    e[5] = D;
  }
}

// Solves the ends of S segments (e[6 s + ...] as put_ends leaves them) for
// the unknowns outside segment `seg`: XL = x_last(seg - 1), XF =
// x_first(seg + 1).  Forward, x_last(s) = P - Q x_first(s + 1); f[2 s],
// f[2 s + 1] hold x_first(s) = f0 - f1 x_first(s + 1) for the way back.
__device__ __forceinline__ void segment_ends(const double *e, double *f, int S, int seg, double &XL,
                                             double &XF) {
  double P = 0.0, Q = 0.0, p0 = 0.0, q0 = 0.0;
  for (int s = 0; s < S; s++, e += 6) {
    if (s == seg) { p0 = P; q0 = Q; }
    const double inv = rcp64(1.0 - e[0] * Q);
    const double f0 = (e[2] - e[0] * P) * inv, f1 = e[1] * inv;
    f[2 * s] = f0;
    f[2 * s + 1] = f1;
    const double aq = e[3] * Q;
    P = e[5] - e[3] * P + aq * f0;
    Q = e[4] + aq * f1;
  }
  double x = 0.0;  // x_first(s + 1)
  XF = 0.0;
  for (int s = S - 1; s >= seg; s--) {
    if (s == seg) XF = x;
    x = f[2 * s] - f[2 * s + 1] * x;
  }
  XL = p0 - q0 * x;
}

// first element of line `line`; 32-bit division for fewer than 2^31 lines (a
// 64-bit one would stand before every load)
__device__ __forceinline__ long long line_base(long long line, long long nlines, int o1n,
                                               long long o1s, long long o2s) {
  if (nlines >> 31) return (line % o1n) * o1s + (line / o1n) * o2s;
  const unsigned l = (unsigned)line, q = l / (unsigned)o1n;
  return (long long)(l - q * (unsigned)o1n) * o1s + (long long)q * o2s;
}

// Unit-stride lines.  One segment (SEG 0, lines of up to W * CL points): a
// group of W lanes per line.  Several: W = 32, the S warps of a line in one
// CTA, 8 / S lines per CTA (SEG 1), or one line of 9 to 16 warps (SEG 2).
// A lane whose chunk lies inside the line loads and stores it with 16-byte
// accesses, the line's partial last chunk element by element.
//
// Latency-bound (256^3 FP64: FP64 pipe 18 %, issue slots 36 % busy, 3 CTAs per
// SM by registers).  Measured: 256^3 167 us FP64 (161 before segments and
// packed lines), 111 us FP32 (126); 300^3 269 us (715) and 246 us (537); 2048 x
// 1500 44 us FP64 (109 with the PCR of the whole line in shared memory), 35 us
// FP32 (83).
template <typename T, bool INC, int SEG, int CL, int W>
__global__ void __launch_bounds__(SEG == 2 ? 32 * kMaxSeg : kThreads, SEG == 2 ? 1 : 3) trid_x_kernel(
    int n, int S, long long nlines, int o1n, long long o1s, long long o2s, const T *__restrict__ A,
    const T *__restrict__ B, const T *__restrict__ C, T *__restrict__ D, T *__restrict__ U) {
  static_assert(!SEG || W == 32, "a segment is a warp's");
  __shared__ double sm[SEG ? kMaxSeg * (6 + 2 * kMaxSeg) : 1];
  const int lane = threadIdx.x % W;
  const int grp = threadIdx.x / W;  // this CTA's group
  const int lpc = SEG ? (int)(blockDim.x / 32) / S : (int)blockDim.x / W;
  const int l = SEG ? grp / S : grp, seg = SEG ? grp - l * S : 0;
  const long long line = (long long)blockIdx.x * lpc + l;
  const bool active = line < nlines;
  const int k0 = (seg * W + lane) * CL;
  const int len = active ? max(0, min(CL, n - k0)) : 0;
  const long long base = active ? line_base(line, nlines, o1n, o1s, o2s) + k0 : 0;
  double a[CL], b[CL], c[CL], d[CL];
  if (len == CL) {
    load_chunk<T, CL>(A + base, a);
    load_chunk<T, CL>(B + base, b);
    load_chunk<T, CL>(C + base, c);
    load_chunk<T, CL>(D + base, d);
  } else {
#pragma unroll
    for (int i = 0; i < CL; i++) {
      a[i] = 0.0; b[i] = 1.0; c[i] = 0.0; d[i] = 0.0;
      if (i < len) {
        a[i] = (double)A[base + i];
        b[i] = (double)B[base + i];
        c[i] = (double)C[base + i];
        d[i] = (double)D[base + i];
      }
    }
  }
  if (k0 == 0) a[0] = 0.0;  // no left neighbour
#pragma unroll
  for (int i = 0; i < CL; i++)
    if (k0 + i == n - 1) c[i] = 0.0;  // no right neighbour
  chunk_reduce<CL>(a, b, c, d);
  double xf, xl;
  if (SEG == 0 && sizeof(T) == 8) {
    pair_pcr<W>(a[0], c[0], d[0], a[CL - 1], c[CL - 1], d[CL - 1], lane, xf, xl);
  } else {
    double gA, gC, gD, XL = 0.0;
    group_reduce<W>(a[0], c[0], d[0], a[CL - 1], c[CL - 1], d[CL - 1], lane, gA, gC, gD);
    xl = gD;
    if (SEG) {
      double *e = sm + 6 * grp;
      put_ends<W>(a[0], c[0], d[0], gA, gC, gD, lane, e);
      __syncthreads();
      double XF = 0.0;
      if (lane == 0)
        segment_ends(sm + 6 * (l * S), sm + 6 * kMaxSeg + 2 * kMaxSeg * grp, S, seg, XL, XF);
      XL = __shfl_sync(0xffffffffu, XL, 0);
      XF = __shfl_sync(0xffffffffu, XF, 0);
      xl = gD - gA * XL - gC * XF;
    }
    double xp = __shfl_up_sync(0xffffffffu, xl, 1, W);
    if (lane == 0) xp = XL;
    xf = d[0] - a[0] * xp - c[0] * xl;
  }
  if (len <= 0) return;
  double x[CL];
#pragma unroll
  for (int i = 0; i < CL; i++)
    x[i] = (i == 0) ? xf : ((i == CL - 1) ? xl : d[i] - a[i] * xf - c[i] * xl);
  T *out = (INC ? U : D) + base;
  if (len == CL) {
    if (INC) {  // (read earlier, as trid_s_kernel does, it costs: 190 against 171 us at 256^3)
      double u[CL];
      load_chunk<T, CL>(out, u);
#pragma unroll
      for (int i = 0; i < CL; i++) x[i] += u[i];
    }
    store_chunk<T, CL>(out, x);
  } else {
#pragma unroll
    for (int i = 0; i < CL; i++)
      if (i < len) out[i] = INC ? (T)((double)out[i] + x[i]) : (T)x[i];
  }
}

// Strided lines: LPB = kThreads / W neighbouring lines per CTA in line-major
// order (consecutive threads on the same chunk of neighbouring lines, whose
// elements are contiguous: every load and store of a warp is runs of LPB
// elements), segment seg of the lines in the CTA of that rank of a cluster of
// S.  The chunk ends cross shared memory once each way; the PCR of a line
// runs in one group of W lanes.  The segments' end equations go to every CTA
// of the cluster through distributed shared memory.  32-bit element offsets
// when every offset of the batch fits (IDX32).
//
// Bound by the latency of a CTA's load, elimination and PCR phases, three CTAs
// per SM in different ones (256^3 y, FP64: 4.5 TB/s, FP64 pipe 21 %, issue
// slots 40 % busy).  The 80 registers of a thread that this takes do not hold
// an 8-row chunk in FP64 whole: 6 values spill, 13 to 20 in the _Inc forms,
// whose u is in flight during the PCR (z _Inc waits on memory 7 cycles per
// issue, y 3).  Measured, before: the same lines as 32 chunks of 8 rows
// whatever their length, lines over 256 points through shared-memory PCR.
//   256^3       y FP64 146 -> 148 us, _Inc 234 -> 208; FP32 173 -> 100, 268 -> 134
//               z FP64 201 -> 180 us, _Inc 262 -> 230; FP32 186 -> 122, 277 -> 160
//   128^3       y FP64 33 -> 23 us, _Inc 57 -> 34
//   193x131x67  z FP64 42 -> 25 us, _Inc 74 -> 33; FP32 68 -> 16, 103 -> 19
//   2048x1500   y FP64 90 -> 47 us, _Inc 183 -> 62; FP32 100 -> 40, 218 -> 49
//   1000x4096   y FP64 140 -> 78 us, _Inc 270 -> 103; FP32 154 -> 72, 345 -> 88
template <typename T, bool INC, bool IDX32, bool SEG, int CL, int W>
__global__ void __launch_bounds__(kThreads, CL > 8 ? 1 : 3) trid_s_kernel(
    int n, int S, long long nlines, long long stride, int o1n, long long o1s, long long o2s,
    const T *__restrict__ A, const T *__restrict__ B, const T *__restrict__ C,
    T *__restrict__ D, T *__restrict__ U) {
  constexpr int LPB = kThreads / W, pitch = W + 1, field = LPB * pitch;
  __shared__ double sm[6 * field];
  extern __shared__ double ends[];  // SEG: [line][segment][6], then [line][segment][2]
  // a CTA's shared memory may be written by the others once it runs: all say
  // so here and wait for one another before the first such store below
  if (SEG) cg::this_cluster().barrier_arrive();
  const int tid = threadIdx.x;
  const int p = tid / LPB, l = tid % LPB;
  const int seg = SEG ? (int)(blockIdx.x % (unsigned)S) : 0;
  const long long line = (long long)(SEG ? blockIdx.x / (unsigned)S : blockIdx.x) * LPB + l;
  const bool active = line < nlines;
  const int k0 = (seg * W + p) * CL;
  long long base = 0;
  if (active) {
    base = line_base(line, nlines, o1n, o1s, o2s);
    base = IDX32 ? (long long)((int)base + k0 * (int)stride) : base + (long long)k0 * stride;
  }
  const int len = active ? max(0, min(CL, n - k0)) : 0;
  // u is added last: its sectors are asked for in L2 with the loads below, each
  // by the lane that begins it (and the last lane, which may begin one).
  // Measured, FP64 _Inc: 333x77x300 y 131 -> 117 us, 193x131x67 z 37.1 -> 33.0,
  // 256^3 y 215 -> 206.  FP32 gets slower (256^3 y 133 -> 149 us), and the
  // segments of long lines by 1 to 2 % (2048x1500 y 61.3 -> 62.2 us).
  if (INC && !SEG && sizeof(T) == 8 && (l % 4 == 0 || l == LPB - 1)) {
#pragma unroll
    for (int i = 0; i < CL; i++)
      if (i < len)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(
            U + (IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride)));
  }
  double a[CL], b[CL], c[CL], d[CL];
  if (sizeof(T) == 8 && len == CL) {  // every load of the chunk in flight at once
#pragma unroll
    for (int i = 0; i < CL; i++) {
      const long long e = IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride;
      a[i] = (double)A[e];
      b[i] = (double)B[e];
      c[i] = (double)C[e];
      d[i] = (double)D[e];
    }
    if (k0 == 0) a[0] = 0.0;                   // no left neighbour
    if (k0 + CL == n) c[CL - 1] = 0.0;         // no right neighbour
  } else if (sizeof(T) == 8) {
#pragma unroll
    for (int i = 0; i < CL; i++) {
      a[i] = 0.0; b[i] = 1.0; c[i] = 0.0; d[i] = 0.0;
      if (i < len) {
        const long long e = IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride;
        a[i] = (k0 + i == 0) ? 0.0 : (double)A[e];
        b[i] = (double)B[e];
        c[i] = (k0 + i == n - 1) ? 0.0 : (double)C[e];
        d[i] = (double)D[e];
      }
    }
  } else {
    // every load of the chunk is issued before the first value is widened
    // (256^3 FP32, y / z: 158 / 176 -> 101 / 124 us)
    T ta[CL], tb[CL], tc[CL], td[CL];
#pragma unroll
    for (int i = 0; i < CL; i++) {
      ta[i] = tc[i] = td[i] = T(0);
      tb[i] = T(1);
      if (i < len) {
        const long long e = IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride;
        ta[i] = A[e];
        tb[i] = B[e];
        tc[i] = C[e];
        td[i] = D[e];
      }
    }
#pragma unroll
    for (int i = 0; i < CL; i++) {
      a[i] = (double)ta[i];
      b[i] = (double)tb[i];
      c[i] = k0 + i == n - 1 ? 0.0 : (double)tc[i];  // no right neighbour
      d[i] = (double)td[i];
    }
    if (k0 == 0) a[0] = 0.0;  // no left neighbour
  }
  chunk_reduce<CL>(a, b, c, d);
  // u is read here, into the registers that b held, so that it arrives while
  // the chunk ends are solved
  T u[INC ? CL : 1];
  if (INC) {
#pragma unroll
    for (int i = 0; i < CL; i++)
      if (i < len) u[i] = U[IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride];
  }
  {
    double *q = sm + l * pitch + p;
    q[0] = a[0]; q[field] = c[0]; q[2 * field] = d[0];
    q[3 * field] = a[CL - 1]; q[4 * field] = c[CL - 1]; q[5 * field] = d[CL - 1];
  }
  __syncthreads();
  {
    const int w = tid / W, lane = tid % W;  // group w reduces line w
    double *q = sm + w * pitch + lane;
    const double a0 = q[0], c0 = q[field], d0 = q[2 * field];
    double xf, xl;
    if (!SEG && sizeof(T) == 8) {
      pair_pcr<W>(a0, c0, d0, q[3 * field], q[4 * field], q[5 * field], lane, xf, xl);
    } else {
      double gA, gC, gD, XL = 0.0;
      group_reduce<W>(a0, c0, d0, q[3 * field], q[4 * field], q[5 * field], lane, gA, gC, gD);
      xl = gD;
      if (SEG) {
        cg::cluster_group cl = cg::this_cluster();
        double *mine = sm + 6 * w;  // the ends of line w, in its own rows of a spent field
        __syncthreads();            // every group has read its chunk ends
        put_ends<W>(a0, c0, d0, gA, gC, gD, lane, mine);
        __syncwarp();
        cl.barrier_wait();  // every CTA of the cluster runs
        for (int k = lane; k < 6 * S; k += W) {
          const int r = k / 6, v = k - 6 * r;
          cl.map_shared_rank(ends, r)[(w * S + seg) * 6 + v] = mine[v];
        }
        cl.sync();  // the last access to another CTA's memory
        double XF = 0.0;
        if (lane == 0)
          segment_ends(ends + 6 * S * w, ends + 6 * S * LPB + 2 * S * w, S, seg, XL, XF);
        XL = __shfl_sync(0xffffffffu, XL, 0, W);
        XF = __shfl_sync(0xffffffffu, XF, 0, W);
        xl = gD - gA * XL - gC * XF;
      }
      double xp = __shfl_up_sync(0xffffffffu, xl, 1, W);
      if (lane == 0) xp = XL;
      xf = d0 - a0 * xp - c0 * xl;
    }
    q[2 * field] = xf;  // this lane's own slots: no other lane reads them
    q[5 * field] = xl;
  }
  __syncthreads();
  if (len <= 0) return;
  const double xf = sm[2 * field + l * pitch + p], xl = sm[5 * field + l * pitch + p];
#pragma unroll
  for (int i = 0; i < CL; i++)
    if (i < len) {
      const double x = (i == 0) ? xf : ((i == CL - 1) ? xl : d[i] - a[i] * xf - c[i] * xl);
      const long long e = IDX32 ? (long long)((int)base + i * (int)stride) : base + i * stride;
      if (INC)
        U[e] = (T)((double)u[i] + x);
      else
        D[e] = (T)x;
    }
}

// Strided lines (y, z): one thread per line, neighbouring threads on
// neighbouring lines along the fastest other axis, so every load and store
// of a warp is one contiguous run.  The Thomas algorithm in FP64 with the
// operation order of the sequential restatement (c'_i = c_i m_i,
// d'_i = (d_i - a_i d'_{i-1}) m_i, m_i = 1 / (b_i - a_i c'_{i-1}), then
// x_i = d'_i - c'_i x_{i+1}), every product and difference rounded on its own
// (no contraction), so the solution equals the oracle's bit for bit.  The
// forward sweep keeps c' and d' in a device scratch array laid out
// [point][line] (coalesced too); the backward sweep reads them back, mostly
// from L2.  Traffic: the algorithmic 4 reads + 1 write per point, plus the
// scratch's 2 writes + 2 reads where it leaves L2.
template <typename T, bool INC>
__global__ void __launch_bounds__(128) trid_thomas_kernel(
    int n, long long nlines, long long stride, int o1n, long long o1s, long long o2s,
    const T *__restrict__ A, const T *__restrict__ B, const T *__restrict__ C,
    T *__restrict__ D, T *__restrict__ U, double *__restrict__ cpd) {
  for (long long line = (long long)blockIdx.x * blockDim.x + threadIdx.x; line < nlines;
       line += (long long)gridDim.x * blockDim.x) {
    const long long base = (line % o1n) * o1s + (line / o1n) * o2s;
    double *cp = cpd + line, *dp = cpd + (long long)n * nlines + line;
    double m = __ddiv_rn(1.0, (double)B[base]);
    double cprev = __dmul_rn((double)C[base], m);
    double dprev = __dmul_rn((double)D[base], m);
    cp[0] = cprev;
    dp[0] = dprev;
#pragma unroll 4
    for (int k = 1; k < n; k++) {
      const long long e = base + (long long)k * stride;
      const double a = (double)A[e], b = (double)B[e], c = (double)C[e], d = (double)D[e];
      m = __ddiv_rn(1.0, __dsub_rn(b, __dmul_rn(a, cprev)));
      cprev = __dmul_rn(c, m);
      dprev = __dmul_rn(__dsub_rn(d, __dmul_rn(a, dprev)), m);
      cp[(long long)k * nlines] = cprev;
      dp[(long long)k * nlines] = dprev;
    }
    double x = dprev;
    {
      const long long e = base + (long long)(n - 1) * stride;
      if (INC)
        U[e] = (T)__dadd_rn((double)U[e], x);
      else
        D[e] = (T)x;
    }
#pragma unroll 4
    for (int k = n - 2; k >= 0; k--) {
      x = __dsub_rn(dp[(long long)k * nlines], __dmul_rn(cp[(long long)k * nlines], x));
      const long long e = base + (long long)k * stride;
      if (INC)
        U[e] = (T)__dadd_rn((double)U[e], x);
      else
        D[e] = (T)x;
    }
  }
}

struct Lines {
  int n, o1n;
  long long nlines, stride, o1s, o2s;
};

// scratch for the Thomas kernel's c' and d' (grown on demand, kept)
double *g_cpd = nullptr;
size_t g_cpd_cap = 0;

template <typename T>
int launch_thomas(const Lines &g, const void *a, const void *b, const void *c, void *d,
                  void *u) {
  const size_t need = (size_t)2 * g.n * g.nlines * sizeof(double);
  cudaStream_t st = (cudaStream_t)ob2_dev_stream();
  if (need > g_cpd_cap) {
    if (g_cpd) {
      cudaStreamSynchronize(st);
      cudaFree(g_cpd);
      g_cpd = nullptr;
      g_cpd_cap = 0;
    }
    cudaError_t e = cudaMalloc(&g_cpd, need);
    if (e != cudaSuccess) return (int)e;
    g_cpd_cap = need;
  }
  // a persistent grid: every line in flight at once would keep 16 bytes
  // per point of scratch live, far beyond L2 for large batches
  int sms = 148;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  static int mult = -1;
  if (mult < 0) {
    const char *env = getenv("OB2_TRID_THOMAS_CTAS");
    mult = env ? atoi(env) : 4;
    if (mult < 1) mult = 1;
  }
  long long grid = std::min((g.nlines + 127) / 128, (long long)sms * mult);
  if (u)
    trid_thomas_kernel<T, true><<<(unsigned)grid, 128, 0, st>>>(
        g.n, g.nlines, g.stride, g.o1n, g.o1s, g.o2s, (const T *)a, (const T *)b, (const T *)c,
        (T *)d, (T *)u, g_cpd);
  else
    trid_thomas_kernel<T, false><<<(unsigned)grid, 128, 0, st>>>(
        g.n, g.nlines, g.stride, g.o1n, g.o1s, g.o2s, (const T *)a, (const T *)b, (const T *)c,
        (T *)d, (T *)nullptr, g_cpd);
  return (int)cudaGetLastError();
}


struct Args {
  const void *a, *b, *c;
  void *d, *u;
};

// 1: every element offset of the batch fits 32-bit arithmetic
bool offsets_fit32(const Lines &g) {
  if (g.o1s < 0 || g.o2s < 0 || g.stride < 0) return false;
  const long long d2 = (g.nlines + g.o1n - 1) / g.o1n;
  const long long mx =
      (long long)(g.o1n - 1) * g.o1s + (d2 - 1) * g.o2s + (long long)(g.n - 1) * g.stride;
  return mx < 0x7fffffffLL;
}

template <typename T, bool INC, int SEG, int CL, int W>
int launch_x(const Lines &g, int S, const Args &q) {
  const int lpc = SEG ? std::max(1, kThreads / 32 / S) : kThreads / W;
  const int threads = SEG ? lpc * S * 32 : kThreads;
  const long long grid = (g.nlines + lpc - 1) / lpc;
  if (grid > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  trid_x_kernel<T, INC, SEG, CL, W><<<(unsigned)grid, threads, 0, (cudaStream_t)ob2_dev_stream()>>>(
      g.n, S, g.nlines, g.o1n, g.o1s, g.o2s, (const T *)q.a, (const T *)q.b, (const T *)q.c,
      (T *)q.d, (T *)q.u);
  return (int)cudaGetLastError();
}

template <typename T, bool INC>
int solve_x(const Lines &g, const Args &q) {
  if constexpr (sizeof(T) == 4) {  // chunks of 6 rows where they hold the line
    if (g.n <= 8 * 6) return launch_x<T, INC, 0, 6, 8>(g, 1, q);
    if (g.n > 8 * 8 && g.n <= 16 * 6) return launch_x<T, INC, 0, 6, 16>(g, 1, q);
    if (g.n > 16 * 8 && g.n <= 32 * 6) return launch_x<T, INC, 0, 6, 32>(g, 1, q);
  }
  if (g.n <= 8 * 8) return launch_x<T, INC, 0, 8, 8>(g, 1, q);
  if (g.n <= 16 * 8) return launch_x<T, INC, 0, 8, 16>(g, 1, q);
  if (g.n <= 32 * 8) return launch_x<T, INC, 0, 8, 32>(g, 1, q);
  const int S = (g.n + 255) / 256;
  const bool few = g.n <= S * 32 * 6;
  if (S <= 8)
    return few ? launch_x<T, INC, 1, 6, 32>(g, S, q) : launch_x<T, INC, 1, 8, 32>(g, S, q);
  return few ? launch_x<T, INC, 2, 6, 32>(g, S, q) : launch_x<T, INC, 2, 8, 32>(g, S, q);
}

// CTAs of a cluster: 16 (more than the portable 8 must be asked for, and a
// device that is partitioned may not have them), OB2_TRID_CLUSTER for fewer
int cluster_limit() {
  static const int v = [] {
    const char *e = getenv("OB2_TRID_CLUSTER");
    return e ? std::max(8, std::min(kMaxSeg, atoi(e))) : kMaxSeg;
  }();
  return v;
}

// whether clusters of more than 8 CTAs of the kernel can run here
template <typename K>
bool wide_clusters(K kern, const cudaLaunchConfig_t &cfg) {
  int n = 0;
  if ((int)cfg.attrs[0].val.clusterDim.x <= cluster_limit() &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
          cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0)
    return true;
  (void)cudaGetLastError();
  return false;
}

template <typename T, bool INC, bool IDX32, bool SEG, int CL, int W>
int launch_s(const Lines &g, int S, const Args &q) {
  constexpr int LPB = kThreads / W;
  const long long grid = (g.nlines + LPB - 1) / LPB * S;
  if (grid > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  auto kern = trid_s_kernel<T, INC, IDX32, SEG, CL, W>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = (cudaStream_t)ob2_dev_stream();
  cudaLaunchAttribute at[1];
  if (SEG) {
    cfg.dynamicSmemBytes = (size_t)8 * S * LPB * sizeof(double);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // otherwise segments of twice the rows, 8 of them at most
    if constexpr (CL <= 8)
      if (S > 8 && !wide_clusters(kern, cfg))
        return launch_s<T, INC, IDX32, true, 16, W>(g, (g.n + 16 * W - 1) / (16 * W), q);
  }
  return (int)cudaLaunchKernelEx(&cfg, kern, g.n, S, g.nlines, g.stride, g.o1n, g.o1s, g.o2s,
                                 (const T *)q.a, (const T *)q.b, (const T *)q.c, (T *)q.d,
                                 (T *)q.u);
}

// CL: the fewest rows per chunk that hold the line (fewer idle lanes and
// registers); double storage in one segment keeps 8 (see pair_pcr)
template <typename T, bool INC, bool IDX32, bool SEG, int W>
int pick_s(const Lines &g, int S, const Args &q) {
  const int rows = (g.n + S * W - 1) / (S * W);  // per chunk
  if constexpr (IDX32 && (SEG || sizeof(T) == 4)) {
    if (rows <= 5) return launch_s<T, INC, true, SEG, 5, W>(g, S, q);
    if (rows <= 6) return launch_s<T, INC, true, SEG, 6, W>(g, S, q);
    if (rows <= 7) return launch_s<T, INC, true, SEG, 7, W>(g, S, q);
  }
  return launch_s<T, INC, IDX32, SEG, 8, W>(g, S, q);
}

// W: the fewest lanes whose chunks of 8 rows hold the line (more lines per CTA:
// longer runs along x, no idle lanes); segments of 256 rows beyond.  Longer
// runs through more segments do not pay (256^3 y / z FP64 with 16 lines per
// CTA and 2 segments of 128 rows: 177 / 176 us).
template <typename T, bool INC, bool IDX32>
int solve_s(const Lines &g, const Args &q) {
  if (g.n <= 64) return pick_s<T, INC, IDX32, false, 8>(g, 1, q);
  if (g.n <= 128) return pick_s<T, INC, IDX32, false, 16>(g, 1, q);
  if (g.n <= 256) return pick_s<T, INC, IDX32, false, 32>(g, 1, q);
  return pick_s<T, INC, IDX32, true, 32>(g, (g.n + 255) / 256, q);
}

// OB2_TRID_STRIDED=0: strided lines by the Thomas kernel (bit-identical to
// the sequential restatement; 256^3 FP64 y / z: 371 / 382 us)
bool use_thomas() {
  static const bool v = [] {
    const char *e = getenv("OB2_TRID_STRIDED");
    return e && atoi(e) == 0;
  }();
  return v;
}

template <typename T>
int launch(int ndim, int solvedim, const int *dims, const long long *strides, const Args &q) {
  Lines g;
  g.n = dims[solvedim];
  int o1 = -1, o2 = -1;
  for (int i = 0; i < 3; i++) {
    if (i == solvedim) continue;
    if (o1 < 0) o1 = i; else o2 = i;
  }
  const int d1 = o1 < ndim ? dims[o1] : 1;
  const int d2 = o2 < ndim ? dims[o2] : 1;
  g.o1n = d1;
  g.o1s = o1 < ndim ? strides[o1] : 0;
  g.o2s = o2 < ndim ? strides[o2] : 0;
  g.nlines = (long long)d1 * d2;
  g.stride = strides[solvedim];
  if (g.n <= 0 || g.nlines <= 0) return 0;
  const bool unit = g.stride == 1;
  if (!unit && use_thomas()) return launch_thomas<T>(g, q.a, q.b, q.c, q.d, q.u);
  if (g.n > kMaxLine) return (int)cudaErrorInvalidValue;
  if (unit) return q.u ? solve_x<T, true>(g, q) : solve_x<T, false>(g, q);
  if (offsets_fit32(g)) return q.u ? solve_s<T, true, true>(g, q) : solve_s<T, false, true>(g, q);
  return q.u ? solve_s<T, true, false>(g, q) : solve_s<T, false, false>(g, q);
}

}  // namespace

OB2_API int ob2_trid_batch(int type_size, int ndim, int solvedim, const int *dims,
                           const long long *strides, const void *a, const void *b,
                           const void *c, void *d, void *u) {
  if (ndim < 1 || ndim > 3 || solvedim < 0 || solvedim >= ndim) return (int)cudaErrorInvalidValue;
  int dd[3] = {1, 1, 1};
  long long ss[3] = {0, 0, 0};
  for (int i = 0; i < ndim; i++) {
    dd[i] = dims[i];
    ss[i] = strides[i];
  }
  if (type_size == 8) return launch<double>(ndim, solvedim, dd, ss, {a, b, c, d, u});
  if (type_size == 4) return launch<float>(ndim, solvedim, dd, ss, {a, b, c, d, u});
  return (int)cudaErrorInvalidValue;
}
