// Host build of the reciprocal of pivots (common.cuh)
#include "../../fastipc_gb300/csrc/common.cuh"

extern "C" void hc_reciprocal(int n, const double* d, double* r) {
    for (int i = 0; i < n; ++i) r[i] = fipc::reciprocal(d[i]);
}
