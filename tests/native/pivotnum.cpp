// Host instantiation of the spline solves' pivot division (csrc/pivot_div.cuh) for CPU tests.
#include "pivot_div.cuh"

extern "C" {
int pn_in_range(double a) { return gkm::pivot_in_range(a) ? 1 : 0; }
void pn_quotients(const double* a, long n, double d, double r, double* q)
{
    for (long i = 0; i < n; i++) q[i] = gkm::pivot_quotient(a[i], d, r);
}
}
