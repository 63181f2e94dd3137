// The short sums of the likelihood's passes, compiled for the host (test_sums_cpu.py).
#include <math.h>

#include "../paragraph_gb300/csrc/pg_sums.cuh"

extern "C" double sum_values(const float* v, int n, int* holds) {
    pg::ErrSum s;
    for (int i = 0; i < n; ++i) pg::err_add(s, v[i]);
    *holds = pg::err_ranges_hold(s);
    return pg::err_value(s);
}
extern "C" double sum_products(const float* a, const float* b, int n) {
    pg::ErrSum s;
    for (int i = 0; i < n; ++i) pg::err_add_product(s, a[i], b[i]);
    return pg::err_value(s);
}
