// The integer-pipe conversions (fiesta_gb300/csrc/fst_conv.cuh) on the host.
#include <cstdint>

#include "../../fiesta_gb300/csrc/fst_conv.cuh"

extern "C" void conv_check(long long n, const double* x, const float* y, float* f, double* d, float* h,
                           float* l, float* hr, float* lr) {
  for (long long i = 0; i < n; ++i) {
    f[i] = fstm::d2f(x[i]);
    d[i] = fstm::f2d(y[i]);
    const fstm::f2p p = fstm::split(x[i]), r = fstm::split<true>(x[i]);
    h[i] = p.h, l[i] = p.l, hr[i] = r.h, lr[i] = r.l;
  }
}
