/*
 * sweep3d: 3D loops whose kernels take several rows per thread -- 7-point
 * sweeps in double and float, a y difference that also reads the point's
 * index, and a max / count reduction over double and float dats -- over the
 * interior of one block.
 *
 * Options: -nx= -ny= -nz= (interior), -off=1 (a range that starts one point in)
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define OPS_3D
#include "ops_seq_v2.h"

#include "sweep3d_kernels.h"

static int opt(int argc, char **argv, const char *key, int def) {
  size_t n = strlen(key);
  for (int i = 1; i < argc; i++)
    if (!strncmp(argv[i], key, n)) return atoi(argv[i] + n);
  return def;
}

int main(int argc, char **argv) {
  ops_init(argc, argv, 1);
  const int nx = opt(argc, argv, "-nx=", 131), ny = opt(argc, argv, "-ny=", 97);
  const int nz = opt(argc, argv, "-nz=", 151), off = opt(argc, argv, "-off=", 0);
  ops_block g = ops_decl_block(3, "grid");
  int size[3] = {nx, ny, nz}, base[3] = {0, 0, 0}, m[3] = {-1, -1, -1}, p[3] = {1, 1, 1};
  double *dn = NULL;
  float *fn = NULL;
  ops_dat a = ops_decl_dat(g, 1, size, base, m, p, dn, "double", "a");
  ops_dat b = ops_decl_dat(g, 1, size, base, m, p, dn, "double", "b");
  ops_dat c = ops_decl_dat(g, 1, size, base, m, p, dn, "double", "c");
  ops_dat f = ops_decl_dat(g, 1, size, base, m, p, fn, "float", "f");
  ops_dat h = ops_decl_dat(g, 1, size, base, m, p, fn, "float", "h");
  int s0[3] = {0, 0, 0};
  int s7[21] = {0, 0, 0, 1, 0, 0, -1, 0, 0, 0, 1, 0, 0, -1, 0, 0, 0, 1, 0, 0, -1};
  ops_stencil S = ops_decl_stencil(3, 1, s0, "000"), S7 = ops_decl_stencil(3, 7, s7, "7pt");
  ops_reduction rx = ops_decl_reduction_handle(sizeof(double), "double", "max");
  ops_reduction rn = ops_decl_reduction_handle(sizeof(int), "int", "count");
  ops_partition("");

  int all[6] = {-1, nx + 1, -1, ny + 1, -1, nz + 1};
  int in[6] = {off, nx, off, ny, off, nz};
  ops_par_loop(sw_fill, "sw_fill", g, 3, all, ops_arg_idx(), ops_arg_dat(a, 1, S, "double", OPS_WRITE),
               ops_arg_dat(f, 1, S, "float", OPS_WRITE));
  ops_par_loop(sw_fill, "sw_fill", g, 3, all, ops_arg_idx(), ops_arg_dat(b, 1, S, "double", OPS_WRITE),
               ops_arg_dat(h, 1, S, "float", OPS_WRITE));
  for (int s = 0; s < 2; s++) {
    ops_par_loop(sw_d, "sw_d", g, 3, in, ops_arg_dat(s ? b : a, 1, S7, "double", OPS_READ),
                 ops_arg_dat(s ? a : b, 1, S, "double", OPS_WRITE));
    ops_par_loop(sw_f, "sw_f", g, 3, in, ops_arg_dat(s ? h : f, 1, S7, "float", OPS_READ),
                 ops_arg_dat(s ? f : h, 1, S, "float", OPS_WRITE));
  }
  ops_par_loop(sw_idx, "sw_idx", g, 3, in, ops_arg_idx(), ops_arg_dat(a, 1, S7, "double", OPS_READ),
               ops_arg_dat(c, 1, S, "double", OPS_WRITE));
  ops_par_loop(sw_change, "sw_change", g, 3, in, ops_arg_dat(a, 1, S, "double", OPS_READ),
               ops_arg_dat(b, 1, S, "double", OPS_READ), ops_arg_dat(f, 1, S, "float", OPS_READ),
               ops_arg_dat(h, 1, S, "float", OPS_READ), ops_arg_reduce(rx, 1, "double", OPS_MAX),
               ops_arg_reduce(rn, 1, "int", OPS_INC));
  double x;
  int n;
  ops_reduction_result(rx, &x);
  ops_reduction_result(rn, &n);
  printf("max %.17g count %d\n", x, n);
  ops_exit();
  return 0;
}
