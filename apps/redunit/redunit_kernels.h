/* Kernels of the redunit application. */
#ifndef REDUNIT_KERNELS_H
#define REDUNIT_KERNELS_H

void ru_fill(const int *idx, ACC<double> &a, ACC<float> &f, ACC<int> &k) {
  const int h = (idx[0] * 7 + idx[1] * 13) % 41 - 20;
  a(0, 0) = (double)h;
  f(0, 0) = 0.5f * (float)h;
  k(0, 0) = 3 * h;
}

void ru_three(const ACC<double> &a, double *s) {
  s[0] = s[0] + a(0, 0);
  s[1] = s[1] + 2.0 * a(0, 0);
  s[2] = s[2] + 1.0;
}
void ru_one(const ACC<double> &a, double *s) { s[0] = s[0] + a(0, 0); }

void ru_types(const ACC<float> &f, const ACC<int> &k, float *fs, float *fx, int *ks, int *kn) {
  fs[0] = fs[0] + f(0, 0);
  fs[1] = fs[1] + 1.0f;
  fs[2] = fs[2] + 2.0f;
  *fx = MAX(*fx, f(0, 0));
  ks[0] = ks[0] + k(0, 0);
  ks[1] = ks[1] + 1;
  *kn = MIN(*kn, k(0, 0));
}

void ru_complex(const ACC<double> &a, complexd *zd, complexf *zf) {
  *zd = *zd + complexd(a(0, 0), 1.0);
  *zf = *zf + complexf(1.0f, (float)a(0, 0));
}

/* milliseconds per point */
void ru_slow(ACC<double> &a, const int *n) {
  double x = a(0, 0);
  for (int i = 0; i < *n; i++) x = 0.5 * x + 1.0;
  a(0, 0) = x;
}

#endif
