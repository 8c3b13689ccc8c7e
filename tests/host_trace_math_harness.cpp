// Host build of the ray arithmetic of porerad_b200/csrc/pr_math.cuh next to the operations it replaces
// (g++ -ffp-contract=off).
#include "../porerad_b200/csrc/pr_math.cuh"

extern "C" {

// pr_sincos_2pi and the double-double series it has to equal
void ht_sincos(const double* x, long n, double* s, double* c, double* s_series, double* c_series) {
  for (long i = 0; i < n; ++i) {
    pr_sincos_2pi(x[i], s + i, c + i);
    pr_sincos(x[i], s_series + i, c_series + i);
  }
}

// v (n, 3) in place
void ht_unit(double* v, long n) {
  for (long i = 0; i < n; ++i) pr_unit_vector(v + 3 * i, v + 3 * i + 1, v + 3 * i + 2);
}

void ht_div(const double* a, const double* b, long n, double* q) {
  for (long i = 0; i < n; ++i) q[i] = pr_div_rcp(a[i], b[i], pr_rcp(b[i]));
}
}
