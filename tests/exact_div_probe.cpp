// Host build of the exact fill's square root and quotients (fnec_math.cuh)
// for tests/test_exact_division.py.
#include <math.h>

#include "fnec_math.cuh"

extern "C" {
// pairs (a, x) inside the domain where sqrt(x) or a / sqrt(x) differs in any
// bit from the IEEE operations; stores the first one
long probe_sqrt_div_mismatches(const double *a, const double *x, long n, double *bad) {
    long k = 0;
    for (long i = 0; i < n; ++i) {
        if (!fnec::sqrt_recip_domain(x[i])) continue;
        const fnec::SqrtRecip sr = fnec::sqrt_recip(x[i]);
        const double r = sqrt(x[i]), q = a[i] / r;
        const double d = fnec::div_by(a[i], sr);
        if (sr.r != r || d != q || signbit(d) != signbit(q)) {
            if (k++ == 0) bad[0] = a[i], bad[1] = x[i];
        }
    }
    return k;
}
long probe_domain_count(const double *x, long n) {
    long k = 0;
    for (long i = 0; i < n; ++i) k += fnec::sqrt_recip_domain(x[i]);
    return k;
}
}
