// Host build of the contribution lists of an aggregated pattern (mg_plan.h)
#include <cstring>

#include "../../fastipc_gb300/csrc/mg_plan.h"

using namespace fipc;

extern "C" {

// out: rp [n_coarse + 1], then ci, con_ptr (nnz + 1), src, src_row, src_col at the given capacities; calls share
// one scratch and one output pattern, as a context's do.  Returns nnz; *n_src: contributions
int hc_pattern(int n_fine, const int* rp, const int* ci, const int* agg, int n_coarse, const unsigned char* fixed, int* o_rp, int* o_ci,
               int* o_con, int* o_src, int* o_row, int* o_col, int* n_src) {
    static MgScratch scratch;
    static MgPattern p;
    mg_detail::galerkin_pattern(n_fine, rp, ci, std::vector<int>(agg, agg + n_fine), n_coarse, p, scratch, fixed);
    auto put = [](int* d, const std::vector<int>& v) { if (!v.empty()) memcpy(d, v.data(), 4 * v.size()); };
    put(o_rp, p.rp);
    put(o_ci, p.ci);
    put(o_con, p.con_ptr);
    put(o_src, p.src);
    put(o_row, p.src_row);
    put(o_col, p.src_col);
    *n_src = (int)p.src.size();
    return p.nnz();
}
}
