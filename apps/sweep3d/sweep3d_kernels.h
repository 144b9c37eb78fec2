/* Kernels of the sweep3d application. */
#ifndef SWEEP3D_KERNELS_H
#define SWEEP3D_KERNELS_H

void sw_fill(const int *idx, ACC<double> &a, ACC<float> &f) {
  const int h = (idx[0] * 7 + idx[1] * 13 + idx[2] * 29) % 101;
  a(0, 0, 0) = 0.01 * h;
  f(0, 0, 0) = 0.02f * (float)h;
}

void sw_d(const ACC<double> &a, ACC<double> &b) {
  b(0, 0, 0) = 0.25 * a(0, 0, 0) + 0.125 * (a(-1, 0, 0) + a(1, 0, 0) + a(0, -1, 0) + a(0, 1, 0) +
                                            a(0, 0, -1) + a(0, 0, 1));
}
void sw_f(const ACC<float> &a, ACC<float> &b) {
  b(0, 0, 0) = 0.25f * a(0, 0, 0) + 0.125f * (a(-1, 0, 0) + a(1, 0, 0) + a(0, -1, 0) +
                                              a(0, 1, 0) + a(0, 0, -1) + a(0, 0, 1));
}

void sw_idx(const int *idx, const ACC<double> &a, ACC<double> &b) {
  b(0, 0, 0) = a(0, 1, 0) - a(0, -1, 0) + 0.5 * idx[0] - idx[1] + 2.0 * idx[2];
}

void sw_change(const ACC<double> &a, const ACC<double> &b, const ACC<float> &f,
               const ACC<float> &g, double *x, int *n) {
  *x = MAX(*x, fabs(a(0, 0, 0) - b(0, 0, 0)) + fabs((double)(f(0, 0, 0) - g(0, 0, 0))));
  *n = *n + 1;
}

#endif
