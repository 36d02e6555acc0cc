// Host build of the one-correction reciprocal and reciprocal square root in csrc/df64.cuh
// (tests/test_df64_fast_host.py).  Built with -ffp-contract=off.
#include "../boccadorata-public_gb300/csrc/df64.cuh"

using namespace bd::dfm;

// op 0: 1/sqrt(a), 1: 1/a, on the double-float images of the inputs
extern "C" void bd_df64_fast(int op, const double *a, int n, double *out) {
    for (int i = 0; i < n; ++i) out[i] = to_double(op == 0 ? rsqrt2(from_double(a[i])) : rcp2(from_double(a[i])));
}
