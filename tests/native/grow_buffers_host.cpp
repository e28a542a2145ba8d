// Host build of the broad phase's kept buffers (ctx.cuh) on an allocator that can be told to fail
#include <cstdlib>

#include "../../fastipc_gb300/csrc/ctx.cuh"

static int g_left = -1;   // allocations until one fails (-1: none does)
static size_t g_size[64];
static void* g_ptr[64];
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_left == 0) return cudaErrorMemoryAllocation;   // p stays as it was
    if (g_left > 0) --g_left;
    *p = malloc(1);
    for (int i = 0; i < 64; ++i)
        if (!g_ptr[i]) {
            g_ptr[i] = *p;
            g_size[i] = n;
            return cudaSuccess;
        }
    abort();
}
extern "C" cudaError_t cudaFree(void* p) {
    for (int i = 0; i < 64; ++i)
        if (g_ptr[i] == p) g_ptr[i] = nullptr;
    free(p);
    return cudaSuccess;
}
static size_t held(const fipc::DBuf& b) {
    for (int i = 0; i < 64; ++i)
        if (b.p && g_ptr[i] == b.p) return g_size[i];
    return 0;
}

// a table of 1024 slots for query 0, one of 4096 for query 1 whose allocation `fail` fails, then query 0 again.
// 0, or the number of the check that does not hold
extern "C" int hc_grid_after_failure(int fail) {
    g_left = -1;
    fipc::Grid g;
    if (g.ensure(1024, 0) || g.use[0] != 1024) return 1;
    g_left = fail;
    if (g.ensure(4096, 1) == fipc::FIPC_OK) return 2;
    if (g.size > held(g.hkeys) / 8 || g.size > held(g.counts) / 4 || g.size > held(g.runs) / 8 || g.size > held(g.ids) / 2) return 3;
    if (g.use[1] != 0) return 4;
    g_left = -1;
    if (g.ensure(g.use[0], 0)) return 5;
    if (held(g.hkeys) < 8 * 1024 || held(g.counts) < 4 * 1024 || held(g.runs) < 8 * 1024 || held(g.ids) < 2 * 1024) return 6;
    return 0;
}
extern "C" int hc_rows_after_failure(int fail) {
    g_left = -1;
    fipc::RowStore r;
    if (r.ensure(100) || r.cap != 100) return 1;
    g_left = fail;
    if (r.ensure(1000) == fipc::FIPC_OK) return 2;
    for (const fipc::DBuf* b : {&r.keys, &r.keys_alt, &r.all})
        if (16ull * r.cap > held(*b)) return 3;
    g_left = -1;
    if (r.ensure(100)) return 4;
    for (const fipc::DBuf* b : {&r.keys, &r.keys_alt, &r.all})
        if (16ull * r.cap > held(*b) || r.cap < 100) return 5;
    return 0;
}
