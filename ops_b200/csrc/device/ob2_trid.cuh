// ob2_trid.cuh -- register building blocks of the tridiagonal solves (ob2_trid.cu,
// the serving engine's ADI kernels): a chunk of a line per thread, its end
// rows solved among the lanes of a line.
#ifndef OB2_TRID_CUH
#define OB2_TRID_CUH

#include <cuda_runtime.h>
#include <stdint.h>

namespace ob2t {

// 1 / x for the eliminations: the Newton-Raphson iteration
// y <- y + y (1 - x y), each step doubling the correct bits, twice from the
// hardware reciprocal approximation (PTX rcp.approx.ftz.f64), with fused
// multiply-adds; zeros, infinities, NaNs and magnitudes whose reciprocal
// could leave the normal range take the IEEE division.  On the GPU the
// result equals 1.0 / x in every bit over 4M random inputs with exponents in
// [-60, 60]; it replaces a division sequence that is several times longer.
__device__ __forceinline__ double rcp64(double x) {
  // exponent outside [-1000, 1000) (integer compare: the FP64 pipe is the
  // busy one)
  const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if (ex - 23u >= 2000u) return 1.0 / x;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = __fma_rn(-x, y, 1.0);
  y = __fma_rn(y, e, y);
  e = __fma_rn(-x, y, 1.0);
  return __fma_rn(y, e, y);
}

// After chunk_reduce (all CL rows; padding rows are b = 1, a = c = d = 0),
// row i of the chunk reads
//   a_i * x_first + x_i + c_i * x_last = d_i        (0 < i < CL-1)
//   a_0 * x_prev  + x_0 + c_0 * x_last = d_0        (row 0)
//   a_{CL-1} * x_0 + x_{CL-1} + c_{CL-1} * x_next = d_{CL-1}   (last row)
// where x_prev / x_next are the end unknowns of the neighbouring chunks.
template <int CL>
__device__ __forceinline__ void chunk_reduce(double *a, const double *b, double *c, double *d) {
  {
    double r = rcp64(b[0]);
    a[0] *= r; c[0] *= r; d[0] *= r;
    r = rcp64(b[1]);
    a[1] *= r; c[1] *= r; d[1] *= r;
  }
  // forward: row i (i >= 2) loses x_{i-1}, gains x_0
#pragma unroll
  for (int i = 2; i < CL; i++) {
    const double r = rcp64(b[i] - a[i] * c[i - 1]);
    d[i] = r * (d[i] - a[i] * d[i - 1]);
    a[i] = -r * a[i] * a[i - 1];
    c[i] = r * c[i];
  }
  // backward: row i (CL-3 >= i >= 1) loses x_{i+1}, gains x_{CL-1}
#pragma unroll
  for (int i = CL - 3; i >= 1; i--) {
    d[i] = d[i] - c[i] * d[i + 1];
    a[i] = a[i] - c[i] * a[i + 1];
    c[i] = -c[i] * c[i + 1];
  }
  // row 0 loses x_1, gains x_{CL-1}
  {
    const double r = rcp64(1.0 - c[0] * a[1]);
    d[0] = r * (d[0] - c[0] * d[1]);
    a[0] = r * a[0];
    c[0] = -r * c[0] * c[1];
  }
}


// PCR over all 2 W chunk ends of a line, held two per lane (rows 2*lane and
// 2*lane+1); returns this lane's two solutions.  Rows are
// a x_{r-s} + x_r + c x_{r+s} = d at each stride s.  Twice the work of
// group_reduce; lines of double storage and one segment keep it, because
// it gives the same bits whatever W holds the line (levels past a line's own
// chunks multiply by 1 and subtract 0), so that their solutions do not depend
// on how lines are packed.
template <int W>
__device__ __forceinline__ void pair_pcr(double a0, double c0, double d0, double a1, double c1,
                                         double d1, int lane, double &xf, double &xl) {
  const unsigned full = 0xffffffffu;
  // s = 1: row 2p couples to 2p-1 (lane p-1, last) and 2p+1 (own last);
  // row 2p+1 couples to 2p (own first) and 2p+2 (lane p+1, first)
  {
    const double pa1 = __shfl_up_sync(full, a1, 1, W), pc1 = __shfl_up_sync(full, c1, 1, W),
                 pd1 = __shfl_up_sync(full, d1, 1, W);
    const double na0 = __shfl_down_sync(full, a0, 1, W), nc0 = __shfl_down_sync(full, c0, 1, W),
                 nd0 = __shfl_down_sync(full, d0, 1, W);
    const bool hasl = lane > 0, hasr = lane < W - 1;
    double k1 = hasl ? a0 : 0.0, k2 = c0;
    double inv = rcp64(1.0 - k1 * (hasl ? pc1 : 0.0) - k2 * a1);
    const double A0 = -k1 * (hasl ? pa1 : 0.0) * inv, C0 = -k2 * c1 * inv,
                 D0 = (d0 - k1 * (hasl ? pd1 : 0.0) - k2 * d1) * inv;
    k1 = a1;
    k2 = hasr ? c1 : 0.0;
    inv = rcp64(1.0 - k1 * c0 - k2 * (hasr ? na0 : 0.0));
    const double A1 = -k1 * a0 * inv, C1 = -k2 * (hasr ? nc0 : 0.0) * inv,
                 D1 = (d1 - k1 * d0 - k2 * (hasr ? nd0 : 0.0)) * inv;
    a0 = A0; c0 = C0; d0 = D0;
    a1 = A1; c1 = C1; d1 = D1;
  }
  // s = 2h rows: both rows of a lane couple to the same slot of lanes p -/+ h
#pragma unroll
  for (int h = 1; h < W; h <<= 1) {
    const bool hasl = lane >= h, hasr = lane + h < W;
    const double la0 = __shfl_up_sync(full, a0, h, W), lc0 = __shfl_up_sync(full, c0, h, W),
                 ld0 = __shfl_up_sync(full, d0, h, W);
    const double ra0 = __shfl_down_sync(full, a0, h, W), rc0 = __shfl_down_sync(full, c0, h, W),
                 rd0 = __shfl_down_sync(full, d0, h, W);
    const double la1 = __shfl_up_sync(full, a1, h, W), lc1 = __shfl_up_sync(full, c1, h, W),
                 ld1 = __shfl_up_sync(full, d1, h, W);
    const double ra1 = __shfl_down_sync(full, a1, h, W), rc1 = __shfl_down_sync(full, c1, h, W),
                 rd1 = __shfl_down_sync(full, d1, h, W);
    {
      const double k1 = hasl ? a0 : 0.0, k2 = hasr ? c0 : 0.0;
      const double inv = rcp64(1.0 - k1 * (hasl ? lc0 : 0.0) - k2 * (hasr ? ra0 : 0.0));
      const double nA = -k1 * (hasl ? la0 : 0.0) * inv, nC = -k2 * (hasr ? rc0 : 0.0) * inv;
      d0 = (d0 - k1 * (hasl ? ld0 : 0.0) - k2 * (hasr ? rd0 : 0.0)) * inv;
      a0 = nA; c0 = nC;
    }
    {
      const double k1 = hasl ? a1 : 0.0, k2 = hasr ? c1 : 0.0;
      const double inv = rcp64(1.0 - k1 * (hasl ? lc1 : 0.0) - k2 * (hasr ? ra1 : 0.0));
      const double nA = -k1 * (hasl ? la1 : 0.0) * inv, nC = -k2 * (hasr ? rc1 : 0.0) * inv;
      d1 = (d1 - k1 * (hasl ? ld1 : 0.0) - k2 * (hasr ? rd1 : 0.0)) * inv;
      a1 = nA; c1 = nC;
    }
  }
  xf = d0;
  xl = d1;
}

// Chunk ends of one line over W lanes, lane p holding chunk p: first row
//   a0 x_last(p-1) + x_first + c0 x_last(p) = d0,
// last row
//   a1 x_first + x_last + c1 x_first(p+1) = d1.
// Substituting the first rows leaves one unknown per chunk, x_last, in a
// tridiagonal system that PCR solves up to the unknowns outside the group:
// on return
//   x_last(p) = D - A XL - C XF,
// XL the unknown before the group (x_last of the chunk to the left of lane
// 0), XF the one after it (x_first of the chunk to the right of lane W-1).
// A row whose left (right) neighbour at stride h lies outside the group keeps
// its coupling to XL (XF).  Against PCR over both ends of every chunk this
// halves the FP64 work and the shuffles and needs one level less.
template <int W>
__device__ __forceinline__ void group_reduce(double a0, double c0, double d0, double a1, double c1,
                                             double d1, int lane, double &A, double &C, double &D) {
  const unsigned full = 0xffffffffu;
  const double na = __shfl_down_sync(full, a0, 1, W), nc = __shfl_down_sync(full, c0, 1, W),
               nd = __shfl_down_sync(full, d0, 1, W);
  const bool inner = lane < W - 1;
  const double ci = inner ? c1 : 0.0;
  const double inv = rcp64(1.0 - a1 * c0 - ci * na);
  A = -a1 * a0 * inv;
  C = (inner ? -c1 * nc : c1) * inv;
  D = (d1 - a1 * d0 - ci * nd) * inv;
#pragma unroll
  for (int h = 1; h < W; h <<= 1) {
    const double la = __shfl_up_sync(full, A, h, W), lc = __shfl_up_sync(full, C, h, W),
                 ld = __shfl_up_sync(full, D, h, W);
    const double ra = __shfl_down_sync(full, A, h, W), rc = __shfl_down_sync(full, C, h, W),
                 rd = __shfl_down_sync(full, D, h, W);
    const bool hl = lane >= h, hr = lane + h < W;
    const double k1 = hl ? A : 0.0, k2 = hr ? C : 0.0;
    const double v = rcp64(1.0 - k1 * lc - k2 * ra);
    D = (D - k1 * ld - k2 * rd) * v;
    A = (hl ? -k1 * la : A) * v;
    C = (hr ? -k2 * rc : C) * v;
  }
}

// CL consecutive elements at p into FP64 registers with 16-byte loads (8-byte
// ones and single elements where the alignment leaves no choice; p's
// alignment is uniform over a warp: chunks start CL elements apart, an even
// number).
template <typename T, int CL>
__device__ __forceinline__ void load_chunk(const T *p, double (&v)[CL]) {
  static_assert(CL % 2 == 0, "even chunks");
  const uintptr_t ad = (uintptr_t)p;
  if (sizeof(T) == 8) {
    const double *q = (const double *)p;
    if ((ad & 15) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 2; i++) {
        const double2 t = ((const double2 *)q)[i];
        v[2 * i] = t.x; v[2 * i + 1] = t.y;
      }
    } else {
      v[0] = q[0];
#pragma unroll
      for (int i = 0; i < CL / 2 - 1; i++) {
        const double2 t = ((const double2 *)(q + 1))[i];
        v[2 * i + 1] = t.x; v[2 * i + 2] = t.y;
      }
      v[CL - 1] = q[CL - 1];
    }
  } else {
    const float *q = (const float *)p;
    if (CL % 4 == 0 && (ad & 15) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 4; i++) {
        const float4 t = ((const float4 *)q)[i];
        v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
      }
    } else if ((ad & 7) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 2; i++) {
        const float2 t = ((const float2 *)q)[i];
        v[2 * i] = t.x; v[2 * i + 1] = t.y;
      }
    } else {  // one element, 8-byte pairs, one element
      v[0] = q[0];
#pragma unroll
      for (int i = 0; i < CL / 2 - 1; i++) {
        const float2 t = ((const float2 *)(q + 1))[i];
        v[2 * i + 1] = t.x; v[2 * i + 2] = t.y;
      }
      v[CL - 1] = q[CL - 1];
    }
  }
}

template <typename T, int CL>
__device__ __forceinline__ void store_chunk(T *p, const double (&v)[CL]) {
  const uintptr_t ad = (uintptr_t)p;
  if (sizeof(T) == 8) {
    double *q = (double *)p;
    if ((ad & 15) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 2; i++) ((double2 *)q)[i] = make_double2(v[2 * i], v[2 * i + 1]);
    } else {
      q[0] = v[0];
#pragma unroll
      for (int i = 0; i < CL / 2 - 1; i++)
        ((double2 *)(q + 1))[i] = make_double2(v[2 * i + 1], v[2 * i + 2]);
      q[CL - 1] = v[CL - 1];
    }
  } else {
    float *q = (float *)p;
    if (CL % 4 == 0 && (ad & 15) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 4; i++)
        ((float4 *)q)[i] = make_float4((float)v[4 * i], (float)v[4 * i + 1], (float)v[4 * i + 2],
                                       (float)v[4 * i + 3]);
    } else if ((ad & 7) == 0) {
#pragma unroll
      for (int i = 0; i < CL / 2; i++)
        ((float2 *)q)[i] = make_float2((float)v[2 * i], (float)v[2 * i + 1]);
    } else {
      q[0] = (float)v[0];
#pragma unroll
      for (int i = 0; i < CL / 2 - 1; i++)
        ((float2 *)(q + 1))[i] = make_float2((float)v[2 * i + 1], (float)v[2 * i + 2]);
      q[CL - 1] = (float)v[CL - 1];
    }
  }
}

}  // namespace ob2t

#endif  // OB2_TRID_CUH
