// Host build of the step filter's root isolation (ccd.cuh)
#include "../../fastipc_gb300/csrc/ccd.cuh"

using namespace fipc;

extern "C" {

// per polynomial (degree n, n + 1 coefficients, highest first): the Bernstein isolation's roots and count
// (-1: left to roots01), roots01's, and whether it surely has no part of sign pos / not pos
void hc_roots(int n, int count, const double* op, double* a, int* na, double* b, int* nb, int* empty_pos, int* empty_neg) {
    for (int c = 0; c < count; ++c) {
        const double* p = op + (n + 1) * c;
        na[c] = bernstein_roots(p, n, a + 8 * c);
        nb[c] = roots01(p, n, b + 8 * c);
        empty_pos[c] = surely_empty(p, n, true);
        empty_neg[c] = surely_empty(p, n, false);
    }
}
}
