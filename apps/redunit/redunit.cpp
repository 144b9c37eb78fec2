/*
 * redunit: how results of reductions reach the host -- handles of double,
 * float, int and complex values with one and several components, fed by one
 * loop, by several, by numbers of loops that change from result to result, by
 * a last loop with fewer components than the handle has, by loops over empty
 * ranges only, and asked for while a loop before them still runs.  Every value is a small
 * integer or a half, so sums are exact in any order.
 *
 * Options: -n= (extent, default 70), -slow= (iterations of the slow loop)
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define OPS_2D
#include "ops_seq_v2.h"

#include "redunit_kernels.h"

static int opt(int argc, char **argv, const char *key, int def) {
  size_t n = strlen(key);
  for (int i = 1; i < argc; i++)
    if (!strncmp(argv[i], key, n)) return atoi(argv[i] + n);
  return def;
}

int main(int argc, char **argv) {
  ops_init(argc, argv, 1);
  const int n = opt(argc, argv, "-n=", 70);
  int slow = opt(argc, argv, "-slow=", 3000000);
  ops_block g = ops_decl_block(2, "grid");
  int size[2] = {n, n / 2}, base[2] = {0, 0}, z[2] = {0, 0}, s0[2] = {0, 0};
  double *dn = NULL;
  float *fn = NULL;
  int *in = NULL;
  ops_dat a = ops_decl_dat(g, 1, size, base, z, z, dn, "double", "a");
  ops_dat b = ops_decl_dat(g, 1, size, base, z, z, dn, "double", "b");
  ops_dat f = ops_decl_dat(g, 1, size, base, z, z, fn, "float", "f");
  ops_dat k = ops_decl_dat(g, 1, size, base, z, z, in, "int", "k");
  ops_stencil S = ops_decl_stencil(2, 1, s0, "00");
  ops_reduction r3 = ops_decl_reduction_handle(3 * sizeof(double), "double", "r3");
  ops_reduction r1 = ops_decl_reduction_handle(sizeof(double), "double", "r1");
  ops_reduction fs = ops_decl_reduction_handle(3 * sizeof(float), "float", "fs");
  ops_reduction fx = ops_decl_reduction_handle(sizeof(float), "float", "fx");
  ops_reduction ks = ops_decl_reduction_handle(2 * sizeof(int), "int", "ks");
  ops_reduction kn = ops_decl_reduction_handle(sizeof(int), "int", "kn");
  ops_reduction zd = ops_decl_reduction_handle(sizeof(complexd), "complexd", "zd");
  ops_reduction zf = ops_decl_reduction_handle(sizeof(complexf), "complexf", "zf");
  ops_partition("");

  int all[4] = {0, size[0], 0, size[1]}, few[4] = {0, 4, 0, 2};
  ops_par_loop(ru_fill, "ru_fill", g, 2, all, ops_arg_idx(),
               ops_arg_dat(a, 1, S, "double", OPS_WRITE), ops_arg_dat(f, 1, S, "float", OPS_WRITE),
               ops_arg_dat(k, 1, S, "int", OPS_WRITE));
  ops_par_loop(ru_fill, "ru_fill", g, 2, all, ops_arg_idx(),
               ops_arg_dat(b, 1, S, "double", OPS_WRITE), ops_arg_dat(f, 1, S, "float", OPS_WRITE),
               ops_arg_dat(k, 1, S, "int", OPS_WRITE));
  double s[3];
  // numbers of loops before each result, over ranges that move
  static const int loops[] = {1, 1, 9, 9, 9, 1, 9, 1, 2, 2, 1, 1, 4, 3, 2, 1, 5};
  for (unsigned c = 0; c < sizeof loops / sizeof *loops; c++) {
    for (int j = 0; j < loops[c]; j++) {
      int part[4] = {j % 3, MAX(j % 3, size[0] - (int)c), j, MAX(j, size[1])};
      ops_par_loop(ru_one, "ru_one", g, 2, part, ops_arg_dat(a, 1, S, "double", OPS_READ),
                   ops_arg_reduce(r1, 1, "double", OPS_INC));
      ops_par_loop(ru_three, "ru_three", g, 2, part, ops_arg_dat(a, 1, S, "double", OPS_READ),
                   ops_arg_reduce(r3, 3, "double", OPS_INC));
    }
    if (c % 2)  // the last loop feeds one component of three
      ops_par_loop(ru_one, "ru_one", g, 2, few, ops_arg_dat(a, 1, S, "double", OPS_READ),
                   ops_arg_reduce(r3, 1, "double", OPS_INC));
    double one;
    ops_reduction_result(r1, &one);
    ops_reduction_result(r3, s);
    printf("sums %d %.17g : %.17g %.17g %.17g\n", (int)c, one, s[0], s[1], s[2]);
  }
  for (int c = 0; c < 3; c++) {
    for (int j = 0; j <= c; j++) {
      int part[4] = {j, size[0], 0, size[1] - c};
      ops_par_loop(ru_types, "ru_types", g, 2, part, ops_arg_dat(f, 1, S, "float", OPS_READ),
                   ops_arg_dat(k, 1, S, "int", OPS_READ), ops_arg_reduce(fs, 3, "float", OPS_INC),
                   ops_arg_reduce(fx, 1, "float", OPS_MAX), ops_arg_reduce(ks, 2, "int", OPS_INC),
                   ops_arg_reduce(kn, 1, "int", OPS_MIN));
      ops_par_loop(ru_complex, "ru_complex", g, 2, part, ops_arg_dat(a, 1, S, "double", OPS_READ),
                   ops_arg_reduce(zd, 1, "complexd", OPS_INC),
                   ops_arg_reduce(zf, 1, "complexf", OPS_INC));
    }
    float v[3], x;
    int m[2], l;
    double cd[2];
    float cf[2];
    ops_reduction_result(fs, v);
    ops_reduction_result(fx, &x);
    ops_reduction_result(ks, m);
    ops_reduction_result(kn, &l);
    ops_reduction_result(zd, (complexd *)cd);
    ops_reduction_result(zf, (complexf *)cf);
    printf("sums types %g %g %g max %g int %d %d min %d complex %g %g %g %g\n", v[0], v[1], v[2], x,
           m[0], m[1], l, cd[0], cd[1], cf[0], cf[1]);
  }
  // a result that is long in coming
  for (int c = 0; c < 3; c++) {
    ops_par_loop(ru_slow, "ru_slow", g, 2, few, ops_arg_dat(b, 1, S, "double", OPS_RW),
                 ops_arg_gbl(&slow, 1, "int", OPS_READ));
    ops_par_loop(ru_one, "ru_one", g, 2, few, ops_arg_dat(b, 1, S, "double", OPS_READ),
                 ops_arg_reduce(r1, 1, "double", OPS_INC));
    ops_reduction_result(r1, s);
    printf("sums slow %.17g\n", s[0]);
  }
  ops_exit();
  return 0;
}
