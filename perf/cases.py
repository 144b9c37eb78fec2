"""The performance cases: what programs on this framework spend their time in.

Most cases are OPS programs in the way of a user: a C++ source with kernels
written against ACC<T>, translated and compiled by ops_b200.build_app (once;
the build is kept under perf/_build), driven through a few C entry points and
the runtime's C ABI (dats set, read and exchanged through ops_dat_*).  The
serving cases go through ops_b200.serving.  Kinds:

  jacobi  explicit sweeps over one block or several blocks joined by halo
          transfers, 2D and 3D, FP64 and FP32, a max-residual at the end;
  euler   a compressible-flow step in FP64: equation of state, time-step
          reduction, boundary loops, fluxes, update (many dats per loop);
  cg      2D implicit heat conduction by conjugate gradients, plain FP64 and
          the mixed form (FP32 vectors, FP64 iterate and residual
          replacement): two reduction results on the host per iteration;
  adi3    3D ADI heat steps: coefficient set-up loop and batched tridiagonal
          solves along x, y and z, FP64 or FP32 storage;
  adi2    2D ADI steps with variable conductivity: long tridiagonal lines;
  serve   a batch of Poisson / heat / ADI requests through the serving engine,
          solutions fetched to the host;
  slab    a slab of a (multi-component) dat fetched into a packed buffer and
          set into another dat, as coupled codes and output do.
"""

from __future__ import annotations

import ctypes as C
import hashlib
import math
import os
import tempfile

import numpy as np
import torch

from ops_b200 import build_app, serving

HERE = os.path.dirname(os.path.abspath(__file__))

# --------------------------------------------------------------------------
# the program
# --------------------------------------------------------------------------

_TYPED_KERNELS = {2: r"""
void jac_$s(const ACC<$T> &u, const ACC<$T> &f, ACC<$T> &un, const $T *h2) {
  un(0, 0) = ($T)0.25 * (u(-1, 0) + u(1, 0) + u(0, -1) + u(0, 1) + h2[0] * f(0, 0));
}
void res_$s(const ACC<$T> &u, const ACC<$T> &f, const $T *h2, double *res) {
  const double r = (double)(h2[0] * f(0, 0)) -
                   (double)(($T)4.0 * u(0, 0) - u(-1, 0) - u(1, 0) - u(0, -1) - u(0, 1));
  *res = MAX(*res, fabs(r));
}
void adi2_rx_$s(const ACC<$T> &u, const ACC<$T> &ay, const ACC<$T> &by, const ACC<$T> &cy,
                ACC<$T> &d) {
  d(0, 0) = ($T)2.0 * u(0, 0) - (ay(0, 0) * u(0, -1) + by(0, 0) * u(0, 0) + cy(0, 0) * u(0, 1));
}
void adi2_ry_$s(const ACC<$T> &d, const ACC<$T> &ax, const ACC<$T> &bx, const ACC<$T> &cx,
                ACC<$T> &u) {
  u(0, 0) = ($T)2.0 * d(0, 0) - (ax(0, 0) * d(-1, 0) + bx(0, 0) * d(0, 0) + cx(0, 0) * d(1, 0));
}
""", 3: r"""
void jac_$s(const ACC<$T> &u, const ACC<$T> &f, ACC<$T> &un, const $T *h2) {
  un(0, 0, 0) = ($T)(1.0 / 6.0) * (u(-1, 0, 0) + u(1, 0, 0) + u(0, -1, 0) + u(0, 1, 0) +
                                   u(0, 0, -1) + u(0, 0, 1) + h2[0] * f(0, 0, 0));
}
void res_$s(const ACC<$T> &u, const ACC<$T> &f, const $T *h2, double *res) {
  const double r = (double)(h2[0] * f(0, 0, 0)) -
                   (double)(($T)6.0 * u(0, 0, 0) - u(-1, 0, 0) - u(1, 0, 0) - u(0, -1, 0) -
                            u(0, 1, 0) - u(0, 0, -1) - u(0, 0, 1));
  *res = MAX(*res, fabs(r));
}
void adi3_pre_$s(const ACC<$T> &u, ACC<$T> &du, ACC<$T> &ax, ACC<$T> &bx, ACC<$T> &cx,
                 ACC<$T> &ay, ACC<$T> &by, ACC<$T> &cy, ACC<$T> &az, ACC<$T> &bz,
                 ACC<$T> &cz, const int *n, const double *lambda, const int *idx) {
  double a, b, c, d;
  if (idx[0] == 0 || idx[0] == n[0] - 1 || idx[1] == 0 || idx[1] == n[1] - 1 ||
      idx[2] == 0 || idx[2] == n[2] - 1) {
    a = 0.0; b = 1.0; c = 0.0; d = 0.0;
  } else {
    d = lambda[0] * ((double)u(-1, 0, 0) + (double)u(1, 0, 0) + (double)u(0, -1, 0) +
                     (double)u(0, 1, 0) + (double)u(0, 0, -1) + (double)u(0, 0, 1) -
                     6.0 * (double)u(0, 0, 0));
    a = -0.5 * lambda[0];
    b = 1.0 + lambda[0];
    c = -0.5 * lambda[0];
  }
  du(0, 0, 0) = ($T)d;
  ax(0, 0, 0) = ($T)a; bx(0, 0, 0) = ($T)b; cx(0, 0, 0) = ($T)c;
  ay(0, 0, 0) = ($T)a; by(0, 0, 0) = ($T)b; cy(0, 0, 0) = ($T)c;
  az(0, 0, 0) = ($T)a; bz(0, 0, 0) = ($T)b; cz(0, 0, 0) = ($T)c;
}
"""}

_KERNELS = r"""
void eu_eos(const ACC<double> &rho, const ACC<double> &mx, const ACC<double> &my,
            const ACC<double> &en, ACC<double> &p, ACC<double> &c) {
  const double v = 1.0 / rho(0, 0);
  const double q = 0.4 * (en(0, 0) - 0.5 * v * (mx(0, 0) * mx(0, 0) + my(0, 0) * my(0, 0)));
  p(0, 0) = q;
  c(0, 0) = sqrt(1.4 * q * v);
}
void eu_dt(const ACC<double> &rho, const ACC<double> &mx, const ACC<double> &my,
           const ACC<double> &c, const double *h, double *dt) {
  const double v = 1.0 / rho(0, 0);
  const double sx = h[0] / (fabs(mx(0, 0) * v) + c(0, 0));
  const double sy = h[1] / (fabs(my(0, 0) * v) + c(0, 0));
  *dt = MIN(*dt, MIN(sx, sy));
}
/* Rusanov flux through the face between a cell and its left / lower one */
void eu_fx(const ACC<double> &rho, const ACC<double> &mx, const ACC<double> &my,
           const ACC<double> &en, const ACC<double> &p, const ACC<double> &c,
           ACC<double> &f0, ACC<double> &f1, ACC<double> &f2, ACC<double> &f3) {
  const double ul = mx(-1, 0) / rho(-1, 0), ur = mx(0, 0) / rho(0, 0);
  const double s = MAX(fabs(ul) + c(-1, 0), fabs(ur) + c(0, 0));
  f0(0, 0) = 0.5 * (mx(-1, 0) + mx(0, 0)) - 0.5 * s * (rho(0, 0) - rho(-1, 0));
  f1(0, 0) = 0.5 * (mx(-1, 0) * ul + p(-1, 0) + mx(0, 0) * ur + p(0, 0)) -
             0.5 * s * (mx(0, 0) - mx(-1, 0));
  f2(0, 0) = 0.5 * (my(-1, 0) * ul + my(0, 0) * ur) - 0.5 * s * (my(0, 0) - my(-1, 0));
  f3(0, 0) = 0.5 * ((en(-1, 0) + p(-1, 0)) * ul + (en(0, 0) + p(0, 0)) * ur) -
             0.5 * s * (en(0, 0) - en(-1, 0));
}
void eu_fy(const ACC<double> &rho, const ACC<double> &mx, const ACC<double> &my,
           const ACC<double> &en, const ACC<double> &p, const ACC<double> &c,
           ACC<double> &f0, ACC<double> &f1, ACC<double> &f2, ACC<double> &f3) {
  const double vl = my(0, -1) / rho(0, -1), vr = my(0, 0) / rho(0, 0);
  const double s = MAX(fabs(vl) + c(0, -1), fabs(vr) + c(0, 0));
  f0(0, 0) = 0.5 * (my(0, -1) + my(0, 0)) - 0.5 * s * (rho(0, 0) - rho(0, -1));
  f1(0, 0) = 0.5 * (mx(0, -1) * vl + mx(0, 0) * vr) - 0.5 * s * (mx(0, 0) - mx(0, -1));
  f2(0, 0) = 0.5 * (my(0, -1) * vl + p(0, -1) + my(0, 0) * vr + p(0, 0)) -
             0.5 * s * (my(0, 0) - my(0, -1));
  f3(0, 0) = 0.5 * ((en(0, -1) + p(0, -1)) * vl + (en(0, 0) + p(0, 0)) * vr) -
             0.5 * s * (en(0, 0) - en(0, -1));
}
void eu_up(ACC<double> &q, const ACC<double> &fx, const ACC<double> &fy, const double *r) {
  q(0, 0) = q(0, 0) - r[0] * (fx(1, 0) - fx(0, 0)) - r[1] * (fy(0, 1) - fy(0, 0));
}
/* reflecting walls: the halo cell mirrors its neighbour, sign -1 for the
 * momentum across the wall */
void eu_bl(ACC<double> &q, const double *sgn) { q(0, 0) = sgn[0] * q(1, 0); }
void eu_br(ACC<double> &q, const double *sgn) { q(0, 0) = sgn[0] * q(-1, 0); }
void eu_bb(ACC<double> &q, const double *sgn) { q(0, 0) = sgn[0] * q(0, 1); }
void eu_bt(ACC<double> &q, const double *sgn) { q(0, 0) = sgn[0] * q(0, -1); }

/* conjugate gradients, A u = (1 + r (faces)) u - r (neighbours), r = (rx, ry) */
void cg_copy(const ACC<double> &b, ACC<double> &u) { u(0, 0) = b(0, 0); }
void cg_res(ACC<double> &r, ACC<double> &p, const ACC<double> &Kx, const ACC<double> &Ky,
            const ACC<double> &u, const ACC<double> &b, const double *c, double *rr) {
  const double au = (1.0 + c[1] * (Ky(0, 1) + Ky(0, 0)) + c[0] * (Kx(1, 0) + Kx(0, 0))) * u(0, 0) -
                    c[1] * (Ky(0, 1) * u(0, 1) + Ky(0, 0) * u(0, -1)) -
                    c[0] * (Kx(1, 0) * u(1, 0) + Kx(0, 0) * u(-1, 0));
  const double v = b(0, 0) - au;
  r(0, 0) = v;
  p(0, 0) = v;
  *rr = *rr + v * v;
}
void cg_w(ACC<double> &w, const ACC<double> &Kx, const ACC<double> &Ky, const ACC<double> &p,
          const double *c, double *pw) {
  const double ap = (1.0 + c[1] * (Ky(0, 1) + Ky(0, 0)) + c[0] * (Kx(1, 0) + Kx(0, 0))) * p(0, 0) -
                    c[1] * (Ky(0, 1) * p(0, 1) + Ky(0, 0) * p(0, -1)) -
                    c[0] * (Kx(1, 0) * p(1, 0) + Kx(0, 0) * p(-1, 0));
  w(0, 0) = ap;
  *pw = *pw + ap * p(0, 0);
}
void cg_ur(ACC<double> &u, ACC<double> &r, const ACC<double> &p, const ACC<double> &w,
           const double *alpha, double *rnn) {
  u(0, 0) = u(0, 0) + alpha[0] * p(0, 0);
  const double v = r(0, 0) - alpha[0] * w(0, 0);
  r(0, 0) = v;
  *rnn = *rnn + v * v;
}
void cg_p(ACC<double> &p, const ACC<double> &r, const double *beta) {
  p(0, 0) = r(0, 0) + beta[0] * p(0, 0);
}
void cg_res32(ACC<float> &r, const ACC<double> &Kx, const ACC<double> &Ky,
              const ACC<double> &u, const ACC<double> &b, const double *c, double *rr) {
  const double au = (1.0 + c[1] * (Ky(0, 1) + Ky(0, 0)) + c[0] * (Kx(1, 0) + Kx(0, 0))) * u(0, 0) -
                    c[1] * (Ky(0, 1) * u(0, 1) + Ky(0, 0) * u(0, -1)) -
                    c[0] * (Kx(1, 0) * u(1, 0) + Kx(0, 0) * u(-1, 0));
  const double v = b(0, 0) - au;
  r(0, 0) = (float)v;
  *rr = *rr + v * v;
}
void cg_copy32(ACC<float> &p, const ACC<float> &r) { p(0, 0) = r(0, 0); }
void cg_w32(ACC<float> &w, const ACC<float> &Kx, const ACC<float> &Ky, const ACC<float> &p,
            const float *c, double *pw) {
  const float ap = (1.0f + c[1] * (Ky(0, 1) + Ky(0, 0)) + c[0] * (Kx(1, 0) + Kx(0, 0))) * p(0, 0) -
                   c[1] * (Ky(0, 1) * p(0, 1) + Ky(0, 0) * p(0, -1)) -
                   c[0] * (Kx(1, 0) * p(1, 0) + Kx(0, 0) * p(-1, 0));
  w(0, 0) = ap;
  *pw = *pw + (double)ap * (double)p(0, 0);
}
void cg_ur32(ACC<double> &u, ACC<float> &r, const ACC<float> &p, const ACC<float> &w,
             const double *alpha, double *rnn) {
  u(0, 0) = u(0, 0) + alpha[0] * (double)p(0, 0);
  const float v = r(0, 0) - (float)alpha[0] * w(0, 0);
  r(0, 0) = v;
  *rnn = *rnn + (double)v * (double)v;
}
void cg_p32(ACC<float> &p, const ACC<float> &r, const float *beta) {
  p(0, 0) = r(0, 0) + beta[0] * p(0, 0);
}
"""

# sweeps and steps of the kinds that exist for both value types
_TYPED_STEPS = {2: r"""
static void jac_sweep_$s(Prog *P, ops_dat *cur, ops_dat *nxt, $T h2) {
  for (size_t b = 0; b < P->blk.size(); b++)
    ops_par_loop(jac_$s, "jac_$s", P->blk[b], $D, P->in,
                 ops_arg_dat(cur[b], 1, SN, "$T", OPS_READ),
                 ops_arg_dat(P->dat[2 * P->blk.size() + b], 1, S0, "$T", OPS_READ),
                 ops_arg_dat(nxt[b], 1, S0, "$T", OPS_WRITE),
                 ops_arg_gbl(&h2, 1, "$T", OPS_READ));
}
static double jac_residual_$s(Prog *P, ops_dat *cur, $T h2) {
  for (size_t b = 0; b < P->blk.size(); b++)
    ops_par_loop(res_$s, "res_$s", P->blk[b], $D, P->in,
                 ops_arg_dat(cur[b], 1, SN, "$T", OPS_READ),
                 ops_arg_dat(P->dat[2 * P->blk.size() + b], 1, S0, "$T", OPS_READ),
                 ops_arg_gbl(&h2, 1, "$T", OPS_READ), ops_arg_reduce(RMAX, 1, "double", OPS_MAX));
  double v = 0.0;
  ops_reduction_result(RMAX, &v);
  return v;
}
static void adi2_step_$s(Prog *P) {
  ops_dat *d = P->dat.data();
  ops_par_loop(adi2_rx_$s, "adi2_rx_$s", P->blk[0], 2, P->in,
               ops_arg_dat(d[0], 1, SN, "$T", OPS_READ), ops_arg_dat(d[5], 1, S0, "$T", OPS_READ),
               ops_arg_dat(d[6], 1, S0, "$T", OPS_READ), ops_arg_dat(d[7], 1, S0, "$T", OPS_READ),
               ops_arg_dat(d[1], 1, S0, "$T", OPS_WRITE));
  ops_tridMultiDimBatch(2, 0, P->in, d[2], d[3], d[4], d[1], P->ctx);
  ops_par_loop(adi2_ry_$s, "adi2_ry_$s", P->blk[0], 2, P->in,
               ops_arg_dat(d[1], 1, SN, "$T", OPS_READ), ops_arg_dat(d[2], 1, S0, "$T", OPS_READ),
               ops_arg_dat(d[3], 1, S0, "$T", OPS_READ), ops_arg_dat(d[4], 1, S0, "$T", OPS_READ),
               ops_arg_dat(d[0], 1, S0, "$T", OPS_WRITE));
  ops_tridMultiDimBatch(2, 1, P->in, d[5], d[6], d[7], d[0], P->ctx);
}
""", 3: r"""
static void jac_sweep_$s(Prog *P, ops_dat *cur, ops_dat *nxt, $T h2) {
  for (size_t b = 0; b < P->blk.size(); b++)
    ops_par_loop(jac_$s, "jac_$s", P->blk[b], $D, P->in,
                 ops_arg_dat(cur[b], 1, SN, "$T", OPS_READ),
                 ops_arg_dat(P->dat[2 * P->blk.size() + b], 1, S0, "$T", OPS_READ),
                 ops_arg_dat(nxt[b], 1, S0, "$T", OPS_WRITE),
                 ops_arg_gbl(&h2, 1, "$T", OPS_READ));
}
static double jac_residual_$s(Prog *P, ops_dat *cur, $T h2) {
  for (size_t b = 0; b < P->blk.size(); b++)
    ops_par_loop(res_$s, "res_$s", P->blk[b], $D, P->in,
                 ops_arg_dat(cur[b], 1, SN, "$T", OPS_READ),
                 ops_arg_dat(P->dat[2 * P->blk.size() + b], 1, S0, "$T", OPS_READ),
                 ops_arg_gbl(&h2, 1, "$T", OPS_READ), ops_arg_reduce(RMAX, 1, "double", OPS_MAX));
  double v = 0.0;
  ops_reduction_result(RMAX, &v);
  return v;
}
static void adi3_step_$s(Prog *P, double lambda) {
  ops_dat *d = P->dat.data();
  ops_par_loop(adi3_pre_$s, "adi3_pre_$s", P->blk[0], 3, P->in,
               ops_arg_dat(d[0], 1, SN, "$T", OPS_READ),
               ops_arg_dat(d[1], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[2], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[3], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[4], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[5], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[6], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[7], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[8], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[9], 1, S0, "$T", OPS_WRITE),
               ops_arg_dat(d[10], 1, S0, "$T", OPS_WRITE),
               ops_arg_gbl(P->n, 3, "int", OPS_READ), ops_arg_gbl(&lambda, 1, "double", OPS_READ),
               ops_arg_idx());
  ops_tridMultiDimBatch(3, 0, P->in, d[2], d[3], d[4], d[1], P->ctx);
  ops_tridMultiDimBatch(3, 1, P->in, d[5], d[6], d[7], d[1], P->ctx);
  ops_tridMultiDimBatch_Inc(3, 2, P->in, d[8], d[9], d[10], d[1], d[0], P->ctx);
}
"""}

# further entry points of the 2D and the 3D program
_EXPORTS = {2: r"""
EXPORT double pp_euler(void *hd, int steps, double hx, double hy) {
  Prog *P = (Prog *)hd;
  ops_dat *q = P->dat.data(), p = q[4], c = q[5], *f = q + 6, *g = q + 10;
  ops_block B = P->blk[0];
  const int nx = P->n[0], ny = P->n[1];
  const double h[2] = {hx, hy};
  double t = 0.0;
  for (int s = 0; s < steps; s++) {
    int lft[] = {-1, 0, 0, ny}, rgt[] = {nx, nx + 1, 0, ny};
    int bot[] = {0, nx, -1, 0}, top[] = {0, nx, ny, ny + 1};
    for (int k = 0; k < 4; k++) {
      const double sx = k == 1 ? -1.0 : 1.0, sy = k == 2 ? -1.0 : 1.0;
      ops_par_loop(eu_bl, "eu_bl", B, 2, lft, ops_arg_dat(q[k], 1, SX, "double", OPS_RW),
                   ops_arg_gbl(&sx, 1, "double", OPS_READ));
      ops_par_loop(eu_br, "eu_br", B, 2, rgt, ops_arg_dat(q[k], 1, SL, "double", OPS_RW),
                   ops_arg_gbl(&sx, 1, "double", OPS_READ));
      ops_par_loop(eu_bb, "eu_bb", B, 2, bot, ops_arg_dat(q[k], 1, SY, "double", OPS_RW),
                   ops_arg_gbl(&sy, 1, "double", OPS_READ));
      ops_par_loop(eu_bt, "eu_bt", B, 2, top, ops_arg_dat(q[k], 1, SB, "double", OPS_RW),
                   ops_arg_gbl(&sy, 1, "double", OPS_READ));
    }
    /* one range for the interior and the walls' cells except the corners */
    int rx[] = {-1, nx + 1, 0, ny};
    ops_par_loop(eu_eos, "eu_eos", B, 2, rx, ops_arg_dat(q[0], 1, S0, "double", OPS_READ),
                 ops_arg_dat(q[1], 1, S0, "double", OPS_READ),
                 ops_arg_dat(q[2], 1, S0, "double", OPS_READ),
                 ops_arg_dat(q[3], 1, S0, "double", OPS_READ),
                 ops_arg_dat(p, 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(c, 1, S0, "double", OPS_WRITE));
    int *walls[2] = {bot, top};
    for (int w = 0; w < 2; w++)
      ops_par_loop(eu_eos, "eu_eos", B, 2, walls[w], ops_arg_dat(q[0], 1, S0, "double", OPS_READ),
                   ops_arg_dat(q[1], 1, S0, "double", OPS_READ),
                   ops_arg_dat(q[2], 1, S0, "double", OPS_READ),
                   ops_arg_dat(q[3], 1, S0, "double", OPS_READ),
                   ops_arg_dat(p, 1, S0, "double", OPS_WRITE),
                   ops_arg_dat(c, 1, S0, "double", OPS_WRITE));
    ops_par_loop(eu_dt, "eu_dt", B, 2, P->in, ops_arg_dat(q[0], 1, S0, "double", OPS_READ),
                 ops_arg_dat(q[1], 1, S0, "double", OPS_READ),
                 ops_arg_dat(q[2], 1, S0, "double", OPS_READ),
                 ops_arg_dat(c, 1, S0, "double", OPS_READ), ops_arg_gbl(h, 2, "double", OPS_READ),
                 ops_arg_reduce(RMIN, 1, "double", OPS_MIN));
    int fx[] = {0, nx + 1, 0, ny}, fy[] = {0, nx, 0, ny + 1};
    ops_par_loop(eu_fx, "eu_fx", B, 2, fx, ops_arg_dat(q[0], 1, SL, "double", OPS_READ),
                 ops_arg_dat(q[1], 1, SL, "double", OPS_READ),
                 ops_arg_dat(q[2], 1, SL, "double", OPS_READ),
                 ops_arg_dat(q[3], 1, SL, "double", OPS_READ),
                 ops_arg_dat(p, 1, SL, "double", OPS_READ),
                 ops_arg_dat(c, 1, SL, "double", OPS_READ),
                 ops_arg_dat(f[0], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(f[1], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(f[2], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(f[3], 1, S0, "double", OPS_WRITE));
    ops_par_loop(eu_fy, "eu_fy", B, 2, fy, ops_arg_dat(q[0], 1, SB, "double", OPS_READ),
                 ops_arg_dat(q[1], 1, SB, "double", OPS_READ),
                 ops_arg_dat(q[2], 1, SB, "double", OPS_READ),
                 ops_arg_dat(q[3], 1, SB, "double", OPS_READ),
                 ops_arg_dat(p, 1, SB, "double", OPS_READ),
                 ops_arg_dat(c, 1, SB, "double", OPS_READ),
                 ops_arg_dat(g[0], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(g[1], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(g[2], 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(g[3], 1, S0, "double", OPS_WRITE));
    double m = 0.0;
    ops_reduction_result(RMIN, &m);
    const double dt = 0.4 * m;
    const double r[2] = {dt / hx, dt / hy};
    for (int k = 0; k < 4; k++)
      ops_par_loop(eu_up, "eu_up", B, 2, P->in, ops_arg_dat(q[k], 1, S0, "double", OPS_RW),
                   ops_arg_dat(f[k], 1, SX, "double", OPS_READ),
                   ops_arg_dat(g[k], 1, SY, "double", OPS_READ),
                   ops_arg_gbl(r, 2, "double", OPS_READ));
    t += dt;
  }
  ops_execute();
  return t;
}

static double sum_result() {
  double v = 0.0;
  ops_reduction_result(RSUM, &v);
  return v;
}
/* solves A u = b from u = b to a relative residual tol; returns iterations */
EXPORT int pp_cg(void *hd, double rx, double ry, double tol) {
  Prog *P = (Prog *)hd;
  ops_dat b = P->dat[0], u = P->dat[1], Kx = P->dat[2], Ky = P->dat[3], r = P->dat[4],
          p = P->dat[5], w = P->dat[6];
  ops_block B = P->blk[0];
  const double c[2] = {rx, ry};
  ops_par_loop(cg_copy, "cg_copy", B, 2, P->in, ops_arg_dat(b, 1, S0, "double", OPS_READ),
               ops_arg_dat(u, 1, S0, "double", OPS_WRITE));
  ops_par_loop(cg_res, "cg_res", B, 2, P->in, ops_arg_dat(r, 1, S0, "double", OPS_WRITE),
               ops_arg_dat(p, 1, S0, "double", OPS_WRITE),
               ops_arg_dat(Kx, 1, SX, "double", OPS_READ),
               ops_arg_dat(Ky, 1, SY, "double", OPS_READ),
               ops_arg_dat(u, 1, SN, "double", OPS_READ),
               ops_arg_dat(b, 1, S0, "double", OPS_READ), ops_arg_gbl(c, 2, "double", OPS_READ),
               ops_arg_reduce(RSUM, 1, "double", OPS_INC));
  double rro = sum_result();
  const double rr0 = rro;
  int it = 0;
  while (it < 20000 && rro > 0.0 && sqrt(rro / rr0) > tol) {
    ops_par_loop(cg_w, "cg_w", B, 2, P->in, ops_arg_dat(w, 1, S0, "double", OPS_WRITE),
                 ops_arg_dat(Kx, 1, SX, "double", OPS_READ),
                 ops_arg_dat(Ky, 1, SY, "double", OPS_READ),
                 ops_arg_dat(p, 1, SN, "double", OPS_READ), ops_arg_gbl(c, 2, "double", OPS_READ),
                 ops_arg_reduce(RSUM, 1, "double", OPS_INC));
    const double alpha = rro / sum_result();
    ops_par_loop(cg_ur, "cg_ur", B, 2, P->in, ops_arg_dat(u, 1, S0, "double", OPS_RW),
                 ops_arg_dat(r, 1, S0, "double", OPS_RW),
                 ops_arg_dat(p, 1, S0, "double", OPS_READ),
                 ops_arg_dat(w, 1, S0, "double", OPS_READ),
                 ops_arg_gbl(&alpha, 1, "double", OPS_READ),
                 ops_arg_reduce(RSUM, 1, "double", OPS_INC));
    const double rnn = sum_result();
    const double beta = rnn / rro;
    ops_par_loop(cg_p, "cg_p", B, 2, P->in, ops_arg_dat(p, 1, S0, "double", OPS_RW),
                 ops_arg_dat(r, 1, S0, "double", OPS_READ),
                 ops_arg_gbl(&beta, 1, "double", OPS_READ));
    rro = rnn;
    it++;
  }
  return it;
}
/* the mixed form: r, p, w in FP32, u in FP64, the residual replaced by
 * b - A u in FP64 whenever it has dropped by 1e-2 or meets tol */
EXPORT int pp_cg_mixed(void *hd, double rx, double ry, double tol) {
  Prog *P = (Prog *)hd;
  ops_dat b = P->dat[0], u = P->dat[1], Kx = P->dat[2], Ky = P->dat[3], r = P->dat[4],
          p = P->dat[5], w = P->dat[6], Kx32 = P->dat[7], Ky32 = P->dat[8];
  ops_block B = P->blk[0];
  const double c[2] = {rx, ry};
  const float c32[2] = {(float)rx, (float)ry};
  ops_par_loop(cg_copy, "cg_copy", B, 2, P->in, ops_arg_dat(b, 1, S0, "double", OPS_READ),
               ops_arg_dat(u, 1, S0, "double", OPS_WRITE));
  double rro = 0.0, rr0 = 0.0, rtrue = 0.0, rel = 1.0;
  bool first = true, replace = true;
  int it = 0;
  while (it < 20000 && rel > tol) {
    if (replace) {
      ops_par_loop(cg_res32, "cg_res32", B, 2, P->in, ops_arg_dat(r, 1, S0, "float", OPS_WRITE),
                   ops_arg_dat(Kx, 1, SX, "double", OPS_READ),
                   ops_arg_dat(Ky, 1, SY, "double", OPS_READ),
                   ops_arg_dat(u, 1, SN, "double", OPS_READ),
                   ops_arg_dat(b, 1, S0, "double", OPS_READ),
                   ops_arg_gbl(c, 2, "double", OPS_READ),
                   ops_arg_reduce(RSUM, 1, "double", OPS_INC));
      const double rnn = sum_result();
      rtrue = rnn;
      if (first) rr0 = rnn;
      rel = rr0 > 0.0 ? sqrt(rnn / rr0) : 0.0;
      if (rel <= tol) break;
      if (first) {
        ops_par_loop(cg_copy32, "cg_copy32", B, 2, P->in,
                     ops_arg_dat(p, 1, S0, "float", OPS_WRITE),
                     ops_arg_dat(r, 1, S0, "float", OPS_READ));
      } else {
        const float beta = (float)(rnn / rro);
        ops_par_loop(cg_p32, "cg_p32", B, 2, P->in, ops_arg_dat(p, 1, S0, "float", OPS_RW),
                     ops_arg_dat(r, 1, S0, "float", OPS_READ),
                     ops_arg_gbl(&beta, 1, "float", OPS_READ));
      }
      rro = rnn;
      first = replace = false;
    }
    ops_par_loop(cg_w32, "cg_w32", B, 2, P->in, ops_arg_dat(w, 1, S0, "float", OPS_WRITE),
                 ops_arg_dat(Kx32, 1, SX, "float", OPS_READ),
                 ops_arg_dat(Ky32, 1, SY, "float", OPS_READ),
                 ops_arg_dat(p, 1, SN, "float", OPS_READ), ops_arg_gbl(c32, 2, "float", OPS_READ),
                 ops_arg_reduce(RSUM, 1, "double", OPS_INC));
    const double alpha = rro / sum_result();
    ops_par_loop(cg_ur32, "cg_ur32", B, 2, P->in, ops_arg_dat(u, 1, S0, "double", OPS_RW),
                 ops_arg_dat(r, 1, S0, "float", OPS_RW), ops_arg_dat(p, 1, S0, "float", OPS_READ),
                 ops_arg_dat(w, 1, S0, "float", OPS_READ),
                 ops_arg_gbl(&alpha, 1, "double", OPS_READ),
                 ops_arg_reduce(RSUM, 1, "double", OPS_INC));
    const double rnn = sum_result();
    it++;
    if (sqrt(rnn / rtrue) <= 1e-2 || sqrt(rnn / rr0) <= tol) {
      replace = true;
      continue;
    }
    const float beta = (float)(rnn / rro);
    ops_par_loop(cg_p32, "cg_p32", B, 2, P->in, ops_arg_dat(p, 1, S0, "float", OPS_RW),
                 ops_arg_dat(r, 1, S0, "float", OPS_READ),
                 ops_arg_gbl(&beta, 1, "float", OPS_READ));
    rro = rnn;
  }
  return it;
}

EXPORT void pp_adi2(void *hd, int steps, int type) {
  Prog *P = (Prog *)hd;
  for (int s = 0; s < steps; s++)
    if (type == 8)
      adi2_step_d(P);
    else
      adi2_step_f(P);
}
""", 3: r"""
EXPORT void pp_adi3(void *hd, int steps, int type, double lambda) {
  Prog *P = (Prog *)hd;
  for (int s = 0; s < steps; s++)
    if (type == 8)
      adi3_step_d(P, lambda);
    else
      adi3_step_f(P, lambda);
}
"""}

_PROGRAM = r"""
#include <math.h>
#include <vector>
#define OPS_$DD
#define DIM $D
#include "ops_seq_v2.h"
#include "ops_tridiag.h"
#include "perf_kernels.h"

struct Prog {
  int n[3], in[6];
  std::vector<ops_block> blk;
  std::vector<ops_dat> dat;
  ops_halo_group halo[2];  /* of the blocks' u and u2 */
  ops_tridsolver_params *ctx;
};

static ops_stencil S0, SN;  /* the point, the point and its neighbours */
#if DIM == 2
static ops_stencil SX, SY, SL, SB;  /* the point and one neighbour */
#endif
static ops_reduction RMAX, RMIN, RSUM;

static void start() {
  static bool done = false;
  if (done) return;
  done = true;
  const char *argv[] = {"perf"};
  ops_init(1, argv, 1);
#if DIM == 2
  int s0[] = {0, 0}, sn[] = {0, 0, 1, 0, -1, 0, 0, 1, 0, -1};
  int sx[] = {0, 0, 1, 0}, sy[] = {0, 0, 0, 1}, sl[] = {0, 0, -1, 0}, sb[] = {0, 0, 0, -1};
  SX = ops_decl_stencil(2, 2, sx, "00_P10");
  SY = ops_decl_stencil(2, 2, sy, "00_0P1");
  SL = ops_decl_stencil(2, 2, sl, "00_M10");
  SB = ops_decl_stencil(2, 2, sb, "00_0M1");
#else
  int s0[] = {0, 0, 0};
  int sn[] = {0, 0, 0, 1, 0, 0, -1, 0, 0, 0, 1, 0, 0, -1, 0, 0, 0, 1, 0, 0, -1};
#endif
  S0 = ops_decl_stencil(DIM, 1, s0, "0");
  SN = ops_decl_stencil(DIM, 2 * DIM + 1, sn, "neighbours");
  RMAX = ops_decl_reduction_handle(sizeof(double), "double", "max");
  RMIN = ops_decl_reduction_handle(sizeof(double), "double", "min");
  RSUM = ops_decl_reduction_handle(sizeof(double), "double", "sum");
}

static Prog *new_prog(int nx, int ny, int nz, int nblk) {
  start();
  Prog *P = new Prog();
  const int n[3] = {nx, ny, nz};
  for (int i = 0; i < 3; i++) {
    P->n[i] = n[i];
    P->in[2 * i] = 0;
    P->in[2 * i + 1] = n[i];
  }
  for (int b = 0; b < nblk; b++) P->blk.push_back(ops_decl_block(DIM, "block"));
  P->ctx = new ops_tridsolver_params(P->blk[0]);
  return P;
}
static void add_dat(Prog *P, int b, int dim, int type) {
  int base[3] = {0, 0, 0}, dm[3] = {-1, -1, -1}, dp[3] = {1, 1, 1};
  double *nd = NULL;
  float *nf = NULL;
  if (type == 8)
    P->dat.push_back(ops_decl_dat(P->blk[b], dim, P->n, base, dm, dp, nd, "double", "d"));
  else
    P->dat.push_back(ops_decl_dat(P->blk[b], dim, P->n, base, dm, dp, nf, "float", "d"));
}
/* halos of dats v[0 .. nb^dims) across every face between neighbouring blocks */
static ops_halo_group faces(Prog *P, int nb, ops_dat *v) {
  std::vector<ops_halo> h;
  int dir[] = {1, 2, 3}, step = 1;
  for (int ax = 0; ax < DIM; ax++, step *= nb)
    for (int b = 0; b < (int)P->blk.size(); b++) {
      if ((b / step) % nb == 0) continue;
      const int a = b - step;  /* the neighbour below along ax */
      int it[3] = {P->n[0], P->n[1], P->n[2]}, f[3] = {0, 0, 0}, t[3] = {0, 0, 0};
      it[ax] = 1;
      f[ax] = P->n[ax] - 1;
      t[ax] = -1;
      h.push_back(ops_decl_halo(v[a], v[b], it, f, t, dir, dir));
      f[ax] = 0;
      t[ax] = P->n[ax];
      h.push_back(ops_decl_halo(v[b], v[a], it, f, t, dir, dir));
    }
  return h.empty() ? NULL : ops_decl_halo_group((int)h.size(), h.data());
}
$STEPS
extern "C" {
#define EXPORT __attribute__((visibility("default")))
EXPORT void *pp_new(int nx, int ny, int nz, int nb, int ndat, int dim, int type) {
  int nblk = 1;
  for (int i = 0; i < DIM; i++) nblk *= nb;
  Prog *P = new_prog(nx, ny, nz, nblk);
  for (int k = 0; k < ndat; k++)
    for (int b = 0; b < nblk; b++) add_dat(P, b, dim, type);
  if (nb > 1) {
    P->halo[0] = faces(P, nb, P->dat.data());
    P->halo[1] = faces(P, nb, P->dat.data() + nblk);
  }
  return P;
}
EXPORT void pp_add(void *h, int dim, int type) { add_dat((Prog *)h, 0, dim, type); }
EXPORT void *pp_dat(void *h, int i) { return ((Prog *)h)->dat[i]; }
EXPORT void pp_free(void *h) {
  Prog *P = (Prog *)h;
  for (ops_dat d : P->dat) ops_free_dat(d);
  delete P->ctx;
  delete P;
}

/* an even number of sweeps from u to u, then the residual */
EXPORT double pp_jacobi(void *h, int sweeps, int type, double h2) {
  Prog *P = (Prog *)h;
  const size_t nb = P->blk.size();
  for (int s = 0; s < sweeps; s++) {
    ops_dat *cur = P->dat.data() + (s & 1 ? nb : 0), *nxt = P->dat.data() + (s & 1 ? 0 : nb);
    if (nb > 1) ops_halo_transfer(P->halo[s & 1]);
    if (type == 8)
      jac_sweep_d(P, cur, nxt, h2);
    else
      jac_sweep_f(P, cur, nxt, (float)h2);
  }
  if (nb > 1) ops_halo_transfer(P->halo[0]);
  return type == 8 ? jac_residual_d(P, P->dat.data(), h2)
                   : jac_residual_f(P, P->dat.data(), (float)h2);
}

$EXPORTS
}  /* extern "C" */
"""


def _typed(text: str) -> str:
    return (text.replace("$T", "double").replace("$s", "d") +
            text.replace("$T", "float").replace("$s", "f"))


def _sources(dims):
    kernels = "#ifndef PERF_KERNELS_H\n#define PERF_KERNELS_H\n" + _typed(_TYPED_KERNELS[dims]) + \
        (_KERNELS if dims == 2 else "") + "#endif\n"
    return {"perf_kernels.h": kernels,
            "perf%dd.cpp" % dims: _PROGRAM.replace("$STEPS", _typed(_TYPED_STEPS[dims]))
                                       .replace("$EXPORTS", _EXPORTS[dims])
                                       .replace("$D", str(dims))}


_DONE = "libperf_done.so"


def _build(out: str, dims: int, sources) -> str:
    """Translates and compiles the program into `out` (build_app); the name
    of the finished library is the mark of a whole build."""
    src = os.path.join(out, "src")
    os.makedirs(src, exist_ok=True)
    for name, text in sources.items():
        with open(os.path.join(src, name), "w") as f:
            f.write(text)
    if os.path.exists(os.path.join(build_app.LIBDIR, "libops_b200.so")):
        build_app.ensure_lib = lambda verbose=False: None  # the tree's own build stands
    lib = build_app.build("perf%dd" % dims, out, [os.path.join(src, "perf%dd.cpp" % dims)], [src],
                          shared=True)
    with open(os.path.join(out, "libdir"), "w") as f:
        f.write(build_app.LIBDIR)
    os.replace(lib, os.path.join(out, _DONE))
    return os.path.join(out, _DONE)


def _usable(out: str) -> bool:
    """A whole build whose run path leads to this tree's libops_b200.so."""
    try:
        with open(os.path.join(out, "libdir")) as f:
            d = f.read()
        return os.path.samefile(d, build_app.LIBDIR) and os.path.exists(os.path.join(out, _DONE))
    except OSError:
        return False


def _library(dims: int) -> str:
    sources = _sources(dims)
    h = hashlib.sha256()
    for name in sorted(sources):
        h.update(sources[name].encode())
    deps = [os.path.join(build_app.HERE, "build_app.py")]
    for d in (os.path.join(build_app.HERE, "translator"), build_app.INCLUDE):
        deps += [os.path.join(d, f) for f in sorted(os.listdir(d)) if f.endswith((".py", ".h"))]
    for p in deps:
        with open(p, "rb") as f:
            h.update(f.read())
    key = h.hexdigest()[:16]
    where = [os.path.join(HERE, "_build"),
             os.path.join(tempfile.gettempdir(), "perf_build_%d" % os.getuid())]
    # a second name for a build of the same sources in a tree elsewhere
    names = [key, key + hashlib.sha256(os.path.realpath(HERE).encode()).hexdigest()[:8]]
    for base in where:
        for n in names:
            if _usable(os.path.join(base, n)):
                return os.path.join(base, n, _DONE)
    for base in where:
        n = names[os.path.exists(os.path.join(base, names[0], _DONE))]
        try:
            os.makedirs(os.path.join(base, n), exist_ok=True)
            if os.access(os.path.join(base, n), os.W_OK):
                return _build(os.path.join(base, n), dims, sources)
        except PermissionError:
            continue
    raise RuntimeError("no place to build the program in")


_libs = {}


def _L(dims):
    if dims not in _libs:
        serving.lib()  # libops_b200.so of this tree
        L = C.CDLL(_library(dims))
        vp, i, d = C.c_void_p, C.c_int, C.c_double
        L.pp_new.restype, L.pp_new.argtypes = vp, [i] * 7
        L.pp_add.restype, L.pp_add.argtypes = None, [vp, i, i]
        L.pp_dat.restype, L.pp_dat.argtypes = vp, [vp, i]
        L.pp_free.restype, L.pp_free.argtypes = None, [vp]
        L.pp_jacobi.restype, L.pp_jacobi.argtypes = d, [vp, i, i, d]
        if dims == 2:
            L.pp_euler.restype, L.pp_euler.argtypes = d, [vp, i, d, d]
            L.pp_cg.argtypes = L.pp_cg_mixed.argtypes = [vp, d, d, d]
            L.pp_adi2.restype, L.pp_adi2.argtypes = None, [vp, i, i]
        else:
            L.pp_adi3.restype, L.pp_adi3.argtypes = None, [vp, i, i, d]
        L.ops_dat_get_raw_pointer.restype = vp
        L.ops_dat_get_raw_pointer.argtypes = [vp, i, vp, C.POINTER(i)]
        L.ops_dat_release_raw_data.argtypes = [vp, i, i]
        L.ops_dat_set_data_memspace.argtypes = [vp, i, vp, i]
        L.ops_dat_fetch_data_slab_memspace.argtypes = [vp, i, vp, C.POINTER(i), i]
        L.ops_dat_set_data_slab_memspace.argtypes = [vp, i, vp, C.POINTER(i), i]
        _libs[dims] = L
    return _libs[dims]


_HOST, _DEVICE, _READ = 1, 2, 0


class _Memory:
    """Device memory of a dat as torch takes it; keeps the program alive."""

    def __init__(self, owner, ptr, shape, strides, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "strides": strides, "typestr": kind,
                                         "data": (ptr, False), "version": 2}


class _Program:
    """One instance of the program: its block(s) and dats (one halo cell on
    every side), each dat with `dim` components of FP64 (8) or FP32 (4)."""

    def __init__(self, dims, n, nb, ndat, dim=1, ts=8):
        self.h = None
        self.dims, self.n = dims, n
        self.shape = list(reversed(n[:dims]))
        self.kinds = [(dim, ts)] * (ndat * nb ** dims)
        self.L = _L(dims)
        self.h = self.L.pp_new(n[0], n[1], n[2], nb, ndat, dim, ts)

    def __del__(self):
        if self.h:
            self.L.pp_free(self.h)

    def add(self, dim, ts):
        self.L.pp_add(self.h, dim, ts)
        self.kinds.append((dim, ts))

    def dat(self, k):
        return self.L.pp_dat(self.h, k)

    def set(self, k, t):
        """The dat's interior from a tensor on the device."""
        t = t.to(torch.float64 if self.kinds[k][1] == 8 else torch.float32).contiguous()
        torch.cuda.current_stream().synchronize()
        self.L.ops_dat_set_data_memspace(self.dat(k), 0, t.data_ptr(), _DEVICE)

    def view(self, k):
        """The dat's interior where it lies (queued loops are run first)."""
        ms = C.c_int(_DEVICE)
        d = self.dat(k)
        p = self.L.ops_dat_get_raw_pointer(d, 0, None, C.byref(ms))
        self.L.ops_dat_release_raw_data(d, 0, _READ)
        dim, ts = self.kinds[k]
        strides, s = [], dim * ts
        for i in range(self.dims):
            strides.insert(0, s)
            s *= self.n[i] + 2
        shape = list(self.shape)
        if dim > 1:
            shape.append(dim)
            strides.append(ts)
        return torch.as_tensor(_Memory(self, p, tuple(shape), tuple(strides),
                                       "<f%d" % ts), device="cuda")


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # a multi-block solver whose blocks live in L2: 2 x 2 blocks of 256^2
        # joined by halo transfers, launches and small copies count
        dict(name="jacobi2d_4x256_f64", kind="jacobi", dims=2, blocks=2, nx=256, ny=256, nz=1,
             ts=8, sweeps=100),
        # the plain streaming sweep on one large block
        dict(name="jacobi2d_4096_f64", kind="jacobi", dims=2, blocks=1, nx=4096, ny=4096, nz=1,
             ts=8, sweeps=20),
        # 3D multi-block in single precision, odd sizes
        dict(name="jacobi3d_8x_ragged_f32", kind="jacobi", dims=3, blocks=2, nx=197, ny=131,
             nz=83, ts=4, sweeps=20),
        # a small flow problem: short loops, boundary loops, one reduction a step
        dict(name="euler_240x200", kind="euler", nx=240, ny=200, steps=10),
        # a flow problem of the size of the hydrodynamics benchmark
        dict(name="euler_3840", kind="euler", nx=3840, ny=3840, steps=2),
        # implicit heat conduction, plain FP64, a mid-size odd grid
        dict(name="cg_1000x777_f64", kind="cg", nx=1000, ny=777, mixed=False),
        # the same in the mixed form at the large size
        dict(name="cg_4096_mixed", kind="cg", nx=4096, ny=4096, mixed=True),
        # 3D ADI at the standard size
        dict(name="adi3d_256_f64", kind="adi3", nx=256, ny=256, nz=256, ts=8, steps=2),
        # 3D ADI in FP32 storage, odd sizes
        dict(name="adi3d_ragged_f32", kind="adi3", nx=193, ny=131, nz=67, ts=4, steps=2),
        # 2D ADI: long lines along and across memory
        dict(name="adi2d_2048x1500_f64", kind="adi2", nx=2048, ny=1500, ts=8, steps=2),
        # a batch of requests of mixed kinds and sizes through the engine
        dict(name="serve_mixed_24", kind="serve", count=24, lo=64, hi=640, adi=7, adi_lo=32,
             adi_hi=160, heat=3, mixed=True),
        # a sub-box of a 3-component 3D dat out and into another dat
        dict(name="slab_3x200", kind="slab", nx=200, ny=180, nz=160, dim=3, ts=8, x0=3, x1=190,
             y0=0, y1=180, z0=11, z1=150, host=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jacobi", "jacobi", "euler", "cg", "adi3", "adi3", "adi2", "serve", "slab"])
    ts = rng.choice([8, 8, 4])
    if kind == "jacobi":
        dims = rng.choice([2, 3])
        blocks = rng.choice([1, 2, 3] if dims == 2 else [1, 2])
        hi = 4096 if dims == 2 else 384
        lo = 64 if dims == 2 else 24
        nx, ny = _log(rng, lo, hi) // blocks, _log(rng, lo, hi) // blocks
        nz = _log(rng, lo, hi) // blocks if dims == 3 else 1
        return dict(kind=kind, dims=dims, blocks=blocks, nx=nx, ny=ny, nz=nz, ts=ts,
                    sweeps=2 * rng.randint(2, 10))
    if kind == "euler":
        return dict(kind=kind, nx=_log(rng, 64, 3840), ny=_log(rng, 64, 3840),
                    steps=rng.randint(1, 2))
    if kind == "cg":
        return dict(kind=kind, nx=_log(rng, 128, 3000), ny=_log(rng, 128, 3000),
                    mixed=rng.random() < 0.5)
    if kind == "adi3":
        return dict(kind=kind, nx=_log(rng, 24, 256), ny=_log(rng, 24, 256),
                    nz=_log(rng, 24, 256), ts=ts, steps=rng.randint(1, 2))
    if kind == "adi2":
        return dict(kind=kind, nx=_log(rng, 100, 4096), ny=_log(rng, 100, 2048), ts=ts,
                    steps=rng.randint(1, 2))
    if kind == "serve":
        count = rng.randint(4, 32)
        return dict(kind=kind, count=count, lo=64, hi=_log(rng, 100, 640), adi=rng.randint(0, count),
                    adi_lo=32, adi_hi=_log(rng, 40, 160), heat=rng.randint(0, 3),
                    mixed=rng.random() < 0.7)
    dim = rng.choice([1, 1, 2, 3, 5])
    n = [_log(rng, 40, 256) for _ in range(3)]
    lo = [rng.randint(0, v // 4) for v in n]
    hi = [rng.randint(3 * v // 4, v) for v in n]
    return dict(kind="slab", nx=n[0], ny=n[1], nz=n[2], dim=dim, ts=ts, x0=lo[0], x1=hi[0],
                y0=lo[1], y1=hi[1], z0=lo[2], z1=hi[2], host=rng.random() < 0.25)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _inputs(case, seed):
    """The dats' first values, FP64 on the device, in the order of the dats
    (values that the program holds in FP32 are FP32 values)."""
    g, kind = _gen(seed), case["kind"]
    rnd = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    held = (lambda t: t.float().double()) if case.get("ts", 8) == 4 else (lambda t: t)
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 1)
    if kind == "jacobi":
        shape = [nz, ny, nx] if case["dims"] == 3 else [ny, nx]
        nb = case["blocks"] ** case["dims"]
        return [held(rnd(*shape)) for _ in range(nb)] + [held(2 * rnd(*shape) - 1) for _ in range(nb)]
    if kind == "euler":
        # a dense hot rectangle of 1/16 of the domain in a quiet gas, with noise
        rho = 0.2 + 0.01 * rnd(ny, nx)
        e = 1.0 + 0.01 * rnd(ny, nx)
        x0, y0 = int(rnd(1).item() * 0.75 * nx), int(rnd(1).item() * 0.75 * ny)
        box = (slice(y0, y0 + ny // 4), slice(x0, x0 + nx // 4))
        rho[box] = 1.0
        e[box] = 2.5
        mx, my = 0.05 * rho * (rnd(ny, nx) - 0.5), 0.05 * rho * (rnd(ny, nx) - 0.5)
        return [rho, mx, my, rho * e + 0.5 * (mx * mx + my * my) / rho]
    if kind == "cg":
        # conductivity 100 in a circle of radius 0.2, 0.1 outside
        c = 0.2 + 0.6 * rnd(2)
        y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) / ny - c[1]
        x = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) / nx - c[0]
        den = torch.where(y[:, None] ** 2 + x[None, :] ** 2 <= 0.04, 100.0, 0.1)
        Kx = torch.zeros(ny, nx, device="cuda", dtype=torch.float64)
        Ky = torch.zeros_like(Kx)  # zero on the domain's faces: no flux
        Kx[:, 1:] = (den[:, :-1] + den[:, 1:]) / (2 * den[:, :-1] * den[:, 1:])
        Ky[1:] = (den[:-1] + den[1:]) / (2 * den[:-1] * den[1:])
        return [rnd(ny, nx), Kx, Ky]
    if kind == "adi3":
        return [held(rnd(nz, ny, nx))]
    if kind == "adi2":
        # (1 + k_w + k_e) u - k_w u_w - k_e u_e with face conductivities in
        # (0, 2), none through the boundary
        kx, ky = 2 * rnd(ny, nx + 1), 2 * rnd(ny + 1, nx)
        kx[:, 0] = kx[:, -1] = 0
        ky[0] = ky[-1] = 0
        return [held(t) for t in (rnd(ny, nx), -kx[:, :-1], 1 + kx[:, :-1] + kx[:, 1:], -kx[:, 1:],
                                  -ky[:-1], 1 + ky[:-1] + ky[1:], -ky[1:])]
    shape = [nz, ny, nx] + ([case["dim"]] if case["dim"] > 1 else [])
    return [held(rnd(*shape)), held(rnd(*shape))]


_LAMBDA = 1.0      # adi3
_CG_DT = 4e-6
_CG_TOL = 1e-10
_ADI_STEPS, _HEAT_STEPS = 10, 5


def _h2(case):
    return 1.0 / (case["blocks"] * max(case["nx"], case["ny"]) + 1) ** 2


def _requests(case, seed):
    """(kind, n, seed, steps) of each request: sizes spread evenly over the
    logarithm of the range, largest and smallest mixed in arrival order."""
    out = []
    flat = case["count"] - case["adi"]
    for k in range(case["count"]):
        adi = (k * case["adi"]) // case["count"] != ((k + 1) * case["adi"]) // case["count"]
        j = sum(1 for o in out if (o[0] == serving.ADI3D) == adi)
        m = case["adi"] if adi else flat
        lo, hi = (case["adi_lo"], case["adi_hi"]) if adi else (case["lo"], case["hi"])
        at = ((j * 7) % m if math.gcd(7, m) == 1 else j) / max(1, m - 1)
        n = int(round(lo * (hi / lo) ** at))
        kd = serving.ADI3D if adi else serving.HEAT2D if j < case["heat"] else serving.POISSON2D
        out.append((kd, n, (seed * 1009 + k) % (1 << 20),
                    _HEAT_STEPS if kd == serving.HEAT2D else _ADI_STEPS))
    return out


class _Server:
    def __init__(self, mode):
        self.engine = serving.Engine(mode)

    def __del__(self):
        self.engine.close()


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "serve":
        st["server"] = _Server(serving.MIXED if case["mixed"] else serving.FP64)
        st["requests"] = _requests(case, seed)
        return st
    vals = _inputs(case, seed)
    n = [case["nx"], case["ny"], case.get("nz", 1)]
    if kind == "jacobi":
        nb = case["blocks"] ** case["dims"]
        p = _Program(case["dims"], n, case["blocks"], 3, ts=case["ts"])
        for b in range(nb):
            p.set(b, vals[b])
            p.set(2 * nb + b, vals[nb + b])
    elif kind == "euler":
        p = _Program(2, n, 1, 14)
        for k in range(4):
            p.set(k, vals[k])
    elif kind == "cg":
        p = _Program(2, n, 1, 4)
        for _ in range(3):
            p.add(1, 4 if case["mixed"] else 8)
        p.set(0, vals[0])
        p.set(2, vals[1])
        p.set(3, vals[2])
        if case["mixed"]:
            for k in (7, 8):
                p.add(1, 4)
                p.set(k, vals[k - 6])
    elif kind == "adi3":
        p = _Program(3, n, 1, 11, ts=case["ts"])
        p.set(0, vals[0])
    elif kind == "adi2":
        p = _Program(2, n, 1, 8, ts=case["ts"])
        p.set(0, vals[0])
        for k in range(2, 8):
            p.set(k, vals[k - 1])
    else:
        p = _Program(3, n, 1, 2, dim=case["dim"], ts=case["ts"])
        p.set(0, vals[0])
        p.set(1, vals[1])
        count = [case["z1"] - case["z0"], case["y1"] - case["y0"], case["x1"] - case["x0"]]
        shape = count + ([case["dim"]] if case["dim"] > 1 else [])
        dt = torch.float64 if case["ts"] == 8 else torch.float32
        st["buf"] = torch.zeros(shape, dtype=dt).pin_memory() if case["host"] else \
            torch.zeros(shape, dtype=dt, device="cuda")
        # out of [x0, x1) x ... of one dat, into the box at the origin of the other
        st["src"] = (C.c_int * 6)(case["x0"], case["x1"], case["y0"], case["y1"], case["z0"],
                                  case["z1"])
        st["dst"] = (C.c_int * 6)(0, count[2], 0, count[1], 0, count[0])
    st["p"] = p
    st["out"] = [p.view(k) for k in _outputs(case)]
    torch.cuda.synchronize()
    return st


def _outputs(case):
    kind = case["kind"]
    if kind == "jacobi":
        return list(range(case["blocks"] ** case["dims"]))
    return {"euler": [0, 1, 2, 3], "cg": [1], "adi3": [0, 1], "adi2": [0], "slab": [1]}[kind]


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "serve":
        reqs = [serving.Request(k, kd, n, s, 0.0, steps)
                for k, (kd, n, s, steps) in enumerate(state["requests"])]
        st = serving.serve(state["server"].engine, reqs, 2 << 30, keep_solutions=True)
        return [r.solution for r in sorted(st["done"], key=lambda r: r.idx)]
    p, L = state["p"], state["p"].L
    if kind == "jacobi":
        res = L.pp_jacobi(p.h, case["sweeps"], case["ts"], _h2(case))
        return state["out"] + [res]
    if kind == "euler":
        t = L.pp_euler(p.h, case["steps"], 1.0 / case["nx"], 1.0 / case["ny"])
        return state["out"] + [t]
    if kind == "cg":
        (L.pp_cg_mixed if case["mixed"] else L.pp_cg)(
            p.h, _CG_DT * case["nx"] ** 2, _CG_DT * case["ny"] ** 2, _CG_TOL)
    elif kind == "adi3":
        L.pp_adi3(p.h, case["steps"], case["ts"], _LAMBDA)
    elif kind == "adi2":
        L.pp_adi2(p.h, case["steps"], case["ts"])
    else:
        ms = _HOST if case["host"] else _DEVICE
        buf = state["buf"].data_ptr()
        L.ops_dat_fetch_data_slab_memspace(p.dat(0), 0, buf, state["src"], ms)
        L.ops_dat_set_data_slab_memspace(p.dat(1), 0, buf, state["dst"], ms)
        return state["out"] + [state["buf"]]
    return state["out"]


def work(case):
    """Each loop, solve and copy reads its inputs and writes its outputs
    once; the passes of an iterative solve are those it takes."""
    kind, ts = case["kind"], case.get("ts", 8)
    if kind == "serve":
        b = f = 0.0
        for kd, n, _, steps in _requests(case, 0):
            if kd == serving.ADI3D:  # coefficients are constants
                b += n ** 3 * 72.0 * steps
                f += n ** 3 * 26.0 * steps
            else:  # about 2.8 n iterations to 1e-8 for Poisson, 12 a heat step
                it = 2.8 * n if kd == serving.POISSON2D else 12.0 * steps
                b += n * n * it * (48.0 if case["mixed"] else 80.0)
                f += n * n * it * 16.0
        return {"bytes": b, "flops": f}
    pts = float(case["nx"] * case["ny"] * case.get("nz", 1))
    if kind == "jacobi":
        pts *= case["blocks"] ** case["dims"]
        return {"bytes": pts * ts * (3.0 * case["sweeps"] + 2),
                "flops": pts * (3 + 2 * case["dims"]) * case["sweeps"]}
    if kind == "euler":
        # eos 6 values, time step 4, fluxes 10 each, updates 16
        return {"bytes": pts * 8 * 46.0 * case["steps"], "flops": pts * 130.0 * case["steps"]}
    if kind == "cg":
        it = 571.0 * max(case["nx"], case["ny"]) / 4096  # 571 to 1e-10 at 4096^2
        return {"bytes": pts * it * (60.0 if case["mixed"] else 104.0), "flops": pts * it * 24.0}
    if kind == "adi3":  # set-up 11 values, solves 5 + 5 + 7 with u
        return {"bytes": pts * ts * 28.0 * case["steps"], "flops": pts * 40.0 * case["steps"]}
    if kind == "adi2":  # two loops of 5 values, two solves of 5
        return {"bytes": pts * ts * 20.0 * case["steps"], "flops": pts * 30.0 * case["steps"]}
    box = float((case["x1"] - case["x0"]) * (case["y1"] - case["y0"]) * (case["z1"] - case["z0"]))
    return {"bytes": box * case["dim"] * ts * 4, "flops": 0}


def tolerance(case):
    """About four times what the paths differ from exact() by (relative
    2-norms measured: sweeps 1.6e-16 and 5.9e-7, flow 2e-15 in the momenta,
    conjugate gradients at their stopping tolerance 1.4e-9 in FP64 and 1.3e-8
    mixed, ADI 1.9e-15 and 3.3e-7 in the right-hand side, requests 6e-8)."""
    kind, ts = case["kind"], case.get("ts", 8)
    if kind == "slab":
        return "exact"
    if kind == "jacobi":
        return {"rel": 2e-15 if ts == 8 else 2e-6}
    if kind == "euler":
        return {"rel": 1e-14}
    if kind == "cg":
        return {"rel": 6e-8 if case["mixed"] else 6e-9}
    if kind == "adi3" or kind == "adi2":
        return {"rel": 1e-14 if ts == 8 else 1.5e-6}
    return {"rel": 5e-7}


# --------------------------------------------------------------------------
# the same in 64 bits with torch and numpy
# --------------------------------------------------------------------------

def _pad(t):
    return torch.nn.functional.pad(t, [1, 1] * t.dim())


def _thomas(a, b, c, d, axis):
    """Tridiagonal solve along `axis` of equally shaped tensors."""
    a, b, c, d = (t.movedim(axis, 0) for t in (a, b, c, d))
    n = d.shape[0]
    x, cp = torch.empty_like(d), torch.empty_like(d)
    cp[0] = c[0] / b[0]
    x[0] = d[0] / b[0]
    for k in range(1, n):
        m = 1.0 / (b[k] - a[k] * cp[k - 1])
        cp[k] = c[k] * m
        x[k] = (d[k] - a[k] * x[k - 1]) * m
    for k in range(n - 2, -1, -1):
        x[k] -= cp[k] * x[k + 1]
    return x.movedim(0, axis)


def _exact_jacobi(case, vals):
    dims, nb = case["dims"], case["blocks"]
    m = nb ** dims
    shape = [case["nz"], case["ny"], case["nx"]][3 - dims:]
    h2 = _h2(case) if case["ts"] == 8 else float(np.float32(_h2(case)))

    def join(parts):
        # one array over all blocks (block b: x fastest)
        full = torch.empty([nb * s for s in shape], device="cuda", dtype=torch.float64)
        for b, t in enumerate(parts):
            full[part(b)] = t
        return full

    def part(b):
        at = [(b // nb ** i) % nb for i in range(dims)][::-1]
        return tuple(slice(k * s, (k + 1) * s) for k, s in zip(at, shape))

    def neighbours(t):
        q, s = _pad(t), 0
        for ax in range(dims):
            core = [slice(1, -1)] * dims
            for off in (slice(0, -2), slice(2, None)):
                core[ax] = off
                s = s + q[tuple(core)]
        return s

    u, f = join(vals[:m]), join(vals[m:])
    for _ in range(case["sweeps"]):
        u = (neighbours(u) + h2 * f) * (0.25 if dims == 2 else 1.0 / 6.0)
    r = (h2 * f - (2.0 * dims * u - neighbours(u))).abs().max().item()
    return [u[part(b)].contiguous() for b in range(m)] + ([r] if case["ts"] == 8 else [None])


def _exact_euler(case, vals):
    hx, hy = 1.0 / case["nx"], 1.0 / case["ny"]
    q, t = list(vals), 0.0
    for _ in range(case["steps"]):
        w = []
        for k in range(4):
            e = _pad(q[k])
            e[1:-1, 0], e[1:-1, -1] = e[1:-1, 1], e[1:-1, -2]
            e[0, 1:-1], e[-1, 1:-1] = e[1, 1:-1], e[-2, 1:-1]
            if k == 1:
                e[:, 0], e[:, -1] = -e[:, 0], -e[:, -1]
            if k == 2:
                e[0], e[-1] = -e[0], -e[-1]
            w.append(e)
        w[0][::case["ny"] + 1, ::case["nx"] + 1] = 1.0  # the unused corners
        rho, mx, my, en = w
        v = 1.0 / rho
        p = 0.4 * (en - 0.5 * v * (mx * mx + my * my))
        c = torch.sqrt(1.4 * p.clamp_min(0) * v)
        inner = (slice(1, -1), slice(1, -1))
        dt = 0.4 * min((hx / ((mx * v).abs() + c)[inner]).min().item(),
                       (hy / ((my * v).abs() + c)[inner]).min().item())
        flux = []
        for ax, m in ((1, mx), (0, my)):
            def lo(z):
                return z[1:-1, :-1] if ax == 1 else z[:-1, 1:-1]

            def hi(z):
                return z[1:-1, 1:] if ax == 1 else z[1:, 1:-1]
            ul, ur = lo(m) / lo(rho), hi(m) / hi(rho)
            s = torch.maximum(ul.abs() + lo(c), ur.abs() + hi(c))
            out = []
            for k, z in enumerate(w):
                if k == 0:
                    avg = lo(m) + hi(m)
                elif k == 3:
                    avg = (lo(z) + lo(p)) * ul + (hi(z) + hi(p)) * ur
                else:
                    avg = lo(z) * ul + hi(z) * ur
                    if (k == 1) == (ax == 1):
                        avg = avg + lo(p) + hi(p)
                out.append(0.5 * avg - 0.5 * s * (hi(z) - lo(z)))
            flux.append(out)
        for k in range(4):
            fx, fy = flux[0][k], flux[1][k]
            q[k] = q[k] - dt / hx * (fx[:, 1:] - fx[:, :-1]) - dt / hy * (fy[1:] - fy[:-1])
        t += dt
    return q + [t]


def _exact_cg(case, vals):
    b, Kx, Ky = vals
    rx, ry = _CG_DT * case["nx"] ** 2, _CG_DT * case["ny"] ** 2
    ke = torch.nn.functional.pad(Kx[:, 1:], [0, 1])
    kn = torch.nn.functional.pad(Ky[1:], [0, 0, 0, 1])
    diag = 1 + rx * (Kx + ke) + ry * (Ky + kn)

    def A(u):
        w = diag * u
        w[:, 1:] -= rx * Kx[:, 1:] * u[:, :-1]
        w[:, :-1] -= rx * Kx[:, 1:] * u[:, 1:]
        w[1:] -= ry * Ky[1:] * u[:-1]
        w[:-1] -= ry * Ky[1:] * u[1:]
        return w

    u = b.clone()
    r = b - A(u)
    p = r.clone()
    rr = rr0 = (r * r).sum().item()
    while rr > rr0 * 1e-24:
        w = A(p)
        alpha = rr / (p * w).sum().item()
        u += alpha * p
        r -= alpha * w
        rn = (r * r).sum().item()
        p = r + (rn / rr) * p
        rr = rn
    return [u]


def _adi3_steps(u, lam, steps):
    n = u.shape
    edge = torch.ones(n, device=u.device, dtype=torch.bool)
    edge[1:-1, 1:-1, 1:-1] = False
    a = torch.where(edge, 0.0, -0.5 * lam).double()
    b = torch.where(edge, 1.0, 1.0 + lam).double()
    d = None
    for _ in range(steps):
        q = _pad(u)
        lap = (q[1:-1, 1:-1, :-2] + q[1:-1, 1:-1, 2:] + q[1:-1, :-2, 1:-1] + q[1:-1, 2:, 1:-1] +
               q[:-2, 1:-1, 1:-1] + q[2:, 1:-1, 1:-1] - 6.0 * u)
        d = torch.where(edge, 0.0, lam * lap)
        d = _thomas(a, b, a, d, 2)
        d = _thomas(a, b, a, d, 1)
        u = u + _thomas(a, b, a, d, 0)
    return u, d


def _exact_adi2(case, vals):
    u, ax, bx, cx, ay, by, cy = vals
    for _ in range(case["steps"]):
        q = _pad(u)
        d = 2 * u - (ay * q[:-2, 1:-1] + by * u + cy * q[2:, 1:-1])
        d = _thomas(ax, bx, cx, d, 1)
        q = _pad(d)
        u = 2 * d - (ax * q[1:-1, :-2] + bx * d + cx * q[1:-1, 2:])
        u = _thomas(ay, by, cy, u, 0)
    return [u]


def _hash(seed, i, j, k):
    """The requests' counter-based random numbers (U[0, 1))."""
    with np.errstate(over="ignore"):
        z = (np.uint64(seed) << np.uint64(42)) ^ (i.astype(np.uint64) << np.uint64(21)) ^ \
            j.astype(np.uint64) ^ (np.asarray(k).astype(np.uint64) << np.uint64(52))
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return torch.from_numpy((z >> np.uint64(11)).astype(np.float64) / 9007199254740992.0).cuda()


def _exact_request(kd, n, seed, steps):
    i, j = np.arange(n)[None, :], np.arange(n)[:, None]
    if kd == serving.ADI3D:
        u = 2 * _hash(seed, i[None], j[None], np.arange(n)[:, None, None] + 1) - 1
        return _adi3_steps(u, 1.0, steps)[0].reshape(-1)
    # the 5-point operator with zero boundary is diagonal in sines
    k = torch.arange(1, n + 1, device="cuda", dtype=torch.float64)
    S = torch.sin(math.pi * k[:, None] * k[None, :] / (n + 1)) * math.sqrt(2.0 / (n + 1))
    lam = 2 - 2 * torch.cos(math.pi * k / (n + 1))
    lam = lam[:, None] + lam[None, :]
    if kd == serving.POISSON2D:
        f = (2 * _hash(seed, i, j, 0) - 1) / (n + 1) ** 2
        return (S @ ((S @ f @ S) / lam) @ S).reshape(-1)
    u = 2 * _hash(seed, i, j, 3) - 1
    return (S @ ((S @ u @ S) / (1 + lam) ** steps) @ S).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return [_exact_request(*r).cpu().numpy() for r in _requests(case, seed)]
    vals = _inputs(case, seed)
    if kind == "jacobi":
        return _exact_jacobi(case, vals)
    if kind == "euler":
        return _exact_euler(case, vals)
    if kind == "cg":
        return _exact_cg(case, vals)
    if kind == "adi3":
        return list(_adi3_steps(vals[0], _LAMBDA, case["steps"]))
    if kind == "adi2":
        return _exact_adi2(case, vals)
    box = vals[0][case["z0"]:case["z1"], case["y0"]:case["y1"], case["x0"]:case["x1"]]
    vals[1][:box.shape[0], :box.shape[1], :box.shape[2]] = box
    return [vals[1], box.contiguous()]
