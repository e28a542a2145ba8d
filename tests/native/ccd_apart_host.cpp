// Host build of the step filter's sign test (ccd.cuh): 1 where a pair is certainly apart over the step
#include "../../fastipc_gb300/csrc/ccd.cuh"
#include "../../fastipc_gb300/csrc/geometry.cuh"

using namespace fipc;

extern "C" void hc_apart(int kind, int count, const double* x, const double* p, double eta, int* out) {
    for (int c = 0; c < count; ++c) {
        v3 X[4], Y[4];
        for (int k = 0; k < 4; ++k) {
            X[k] = load3(x + 12 * c, k);
            Y[k] = X[k] + load3(p + 12 * c, k);
        }
        const double e = eta * sqrt(kind == 0 ? pt_dist2(X[0], X[1], X[2], X[3]) : ee_dist2(X[0], X[1], X[2], X[3]));
        out[c] = kind == 0 ? vertex_face_apart(X[0], X[1], X[2], X[3], Y[0], Y[1], Y[2], Y[3], e)
                           : edge_edge_apart(X[0], X[1], X[2], X[3], Y[0], Y[1], Y[2], Y[3], e);
    }
}
