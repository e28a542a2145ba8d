// Spatial hash and the three queries built on it: constraint finding
// (NEWTON_IPC.py:181-357), the CCD step filter (NEWTON_IPC.py:377-468) and the
// intersection check (NEWTON_IPC.py:855-886).
//
// The grid keeps the reference's box conventions, with the median boundary edge as its cell.
// The reference uses the mean; enumeration is complete for any cell size, so the lists are the
// same.  What the reference appends to its sparse grid goes into an open-addressing table: count the
// entries of every occupied cell, give each cell a run of ids, fill the runs.  The order of the ids
// in a run, and of the rows found, depends on timing; nothing that is returned does.  A candidate pair whose two cell ranges overlap in several cells is
// examined only in the overlap's lowest cell (componentwise max of the two lower corners), so
// every pair is tested once without a hash set.  The narrow phase applies the reference's exact
// predicates; constraint rows are then sorted lexicographically and de-duplicated per list
// exactly like np.unique(axis=0) (NEWTON_IPC.py:348-356).
//
// A call is a chain of a few kernels and one copy to the host at its end: table sizes (of each query by itself) and row
// capacities are kept from call to call and checked on the device; a call that outgrows them is repeated with larger
// ones, and a table much larger than its query's last call needed shrinks.  Measured on a GB300 against radix-sorted grids, one sort per list and a host round trip per grid:
// constraint finding of two touching cubes (1,458 vertices) 1.16 -> 0.16 ms a call, of a pile of 180 cubes
// 5.2 -> 0.81 ms; the step filter of the cubes 2.2 -> 0.55 ms.
#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "ccd.cuh"
#include "ctx.cuh"
#include "geometry.cuh"

namespace fipc {

namespace cg = cooperative_groups;

struct C3 {
    long long x, y, z;
};

__device__ __forceinline__ C3 cell_of(v3 p, double inv_dx) {
    return C3{(long long)floor(p.x * inv_dx), (long long)floor(p.y * inv_dx), (long long)floor(p.z * inv_dx)};
}
__device__ __forceinline__ C3 cmax(C3 a, C3 b) { return C3{a.x > b.x ? a.x : b.x, a.y > b.y ? a.y : b.y, a.z > b.z ? a.z : b.z}; }
__device__ __forceinline__ unsigned long long gkey(const SceneGeo& g, int s, long long cx, long long cy, long long cz) {
    return g.vscene ? cell_key_scene(s, cx, cy, cz) : cell_key(cx, cy, cz);
}
// Box modes of stored primitives:
//  0 point [p - dh, p + dh]               (find constraints, point-triangle)
//  1 edge  [min, max]                      (find constraints, edge-edge)
//  2 moving point [min(p, p+dp) - dh, max + dh]   (CCD point-triangle)
//  3 moving edge  [min over 4 ends, max]           (CCD edge-edge)
//  4 edge  [min - dh, max + dh]            (intersection check)
__device__ __forceinline__ void stored_box(int mode, int i, const int* __restrict__ prim, const double* __restrict__ x,
                                           const double* __restrict__ p, double dh, v3* lo, v3* hi) {
    if (mode == 0 || mode == 2) {
        const v3 a = ld3(x, prim[i]);
        v3 mn = a, mx = a;
        if (mode == 2) {
            const v3 b = a + ld3(p, prim[i]);
            mn = vmin(a, b);
            mx = vmax(a, b);
        }
        *lo = mn - mk(dh, dh, dh);
        *hi = mx + mk(dh, dh, dh);
    } else {
        const v3 a = ld3(x, prim[2 * i]), b = ld3(x, prim[2 * i + 1]);
        v3 mn = vmin(a, b), mx = vmax(a, b);
        if (mode == 3) {
            const v3 a2 = a + ld3(p, prim[2 * i]), b2 = b + ld3(p, prim[2 * i + 1]);
            mn = vmin(mn, vmin(a2, b2));
            mx = vmax(mx, vmax(a2, b2));
        }
        if (mode == 4) {
            mn = mn - mk(dh, dh, dh);
            mx = mx + mk(dh, dh, dh);
        }
        *lo = mn;
        *hi = mx;
    }
}

constexpr long long MAX_CELLS_PER_PRIM = 1ll << 22;

// Candidate records of the stored primitives, built with the grid, so that the query kernels
// reject most candidates without FP64 work (GB300 issues FP64 at a small fraction of its FP32
// rate):
//  * cell: cell_of(stored lower corner), the first-cell test of the queries' pair
//    de-duplication, computed with the same FP64 expression; ext: the number of cells per axis
//    (0: not stored) and the scene, so that filling the table needs no FP64 work either;
//  * box: an FP32 box rounded outward around the FP64 box that the query's own FP64 test
//    compares against: mode 0 the point; 1 and 3 the (moving) edge box +- dh (ee_aabb,
//    ee_aabb_moving); 2 the moving point's box (pt_aabb_moving); 4 the edge box +- dh (the
//    intersection check, whose segment-triangle test cannot hit a triangle whose box is dh
//    away).  A candidate whose FP32 box misses the query's FP32 box (also rounded outward)
//    fails the FP64 test too, so the lists, steps and flags are unchanged.
__device__ __forceinline__ float4 f32_lo(v3 a) {
    return make_float4(__double2float_rd(a.x), __double2float_rd(a.y), __double2float_rd(a.z), 0.f);
}
__device__ __forceinline__ float4 f32_hi(v3 a) {
    return make_float4(__double2float_ru(a.x), __double2float_ru(a.y), __double2float_ru(a.z), 0.f);
}
__device__ __forceinline__ bool f32_overlap(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    return alo.x < bhi.x && alo.y < bhi.y && alo.z < bhi.z && blo.x < ahi.x && blo.y < ahi.y && blo.z < ahi.z;
}
__device__ __forceinline__ int clamp_cell(long long c) {
    return (int)(c < -(1ll << 30) ? -(1ll << 30) : (c > (1ll << 30) ? (1ll << 30) : c));
}

__device__ __forceinline__ void cand_record(int mode, int i, const int* __restrict__ prim, const double* __restrict__ x,
                                            const double* __restrict__ p, double dh, v3 lo, v3 hi, C3 c, int4* __restrict__ cell,
                                            float4* __restrict__ box) {
    cell[i] = make_int4(clamp_cell(c.x), clamp_cell(c.y), clamp_cell(c.z), 0);
    const v3 d = mk(dh, dh, dh);
    v3 blo = lo, bhi = hi;
    if (mode == 0) {                      // the point itself
        blo = ld3(x, prim[i]);
        bhi = blo;
    } else if (mode == 2) {               // the moving point's box, without dh
        const v3 a = ld3(x, prim[i]), b = a + ld3(p, prim[i]);
        blo = vmin(a, b);
        bhi = vmax(a, b);
    } else if (mode == 1 || mode == 3) {  // edge box +- dh, as ee_aabb(_moving) forms it
        blo = lo - d;
        bhi = hi + d;
    }
    box[2 * (size_t)i] = f32_lo(blo);
    box[2 * (size_t)i + 1] = f32_hi(bhi);
}

struct CandView {
    const int4* cell;
    const float4* box;
};
// a primitive's size, by the cells of its query box: SIZE_BIG leaves the grid, SIZE_MID may (big primitives, below)
enum : unsigned char { SIZE_GRID = 0, SIZE_MID = 1, SIZE_BIG = 2 };
constexpr int RECORD_MID = 1 << 30;   // in the records' last word
// the queries' records: the lowest cell of the query box and its cells per axis (10 bits each; 0 for a big
// primitive), the FP32 box that candidates are tested against and the scene (in box[2 i].w)
struct QueryView {
    int4* cell;
    float4* box;
    const unsigned long long* mid_pairs;   // of the queries' kind
};
__device__ __forceinline__ void query_record(const QueryView& q, int i, int sc, int size, C3 lo, C3 hi, v3 blo, v3 bhi) {
    const long long nx = hi.x - lo.x + 1, ny = hi.y - lo.y + 1, nz = hi.z - lo.z + 1;
    // at most BIG_CELLS cells unless a position is not finite
    const bool any = size != SIZE_BIG && nx > 0 && ny > 0 && nz > 0 && nx < 1024 && ny < 1024 && nz < 1024;
    q.cell[i] = make_int4(clamp_cell(lo.x), clamp_cell(lo.y), clamp_cell(lo.z),
                          any ? (int)(nx | ny << 10 | nz << 20) | (size == SIZE_MID ? RECORD_MID : 0) : 0);
    float4 l = f32_lo(blo);
    l.w = __int_as_float(sc);
    q.box[2 * (size_t)i] = l;
    q.box[2 * (size_t)i + 1] = f32_hi(bhi);
}

// The line between the grid and the pass over all partners (big primitives, below): more than BIG_CELLS cells leave
// the grid; between MID_CELLS and BIG_CELLS all of a call's primitives of a kind leave it or none, by the number of tests
// that they would take outside.
constexpr long long MID_CELLS = 64, BIG_CELLS = 256;
constexpr unsigned long long MID_PAIRS = 1ull << 23;
__device__ __forceinline__ bool mids_leave(const unsigned long long* mid_pairs) { return *mid_pairs <= MID_PAIRS; }
__device__ __forceinline__ int size_of(long long cells) { return cells > BIG_CELLS ? SIZE_BIG : (cells > MID_CELLS ? SIZE_MID : SIZE_GRID); }

// Cell table of a grid: open addressing with linear probing, load factor at most 1/2, so a query cell
// costs one or two probes.  run[slot] = (first id, ids) of the slot's cell.
constexpr unsigned long long HASH_EMPTY = ~0ull;
// the 64-bit finaliser of MurmurHash3
__device__ __forceinline__ unsigned long long mix64(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}
struct GridView {
    const unsigned long long* hk;   // table keys
    const int2* run;
    unsigned long long mask;        // table size - 1
    const int* ids;                 // primitive ids by run
    // the run of key's cell (empty when there is none; at most mask + 1 probes)
    __device__ __forceinline__ int2 find(unsigned long long key) const {
        unsigned long long h = mix64(key) & mask;
        for (unsigned long long n = 0; n <= mask; ++n) {
            const unsigned long long k = __ldg(hk + h);
            if (k == key) return __ldg(run + h);
            if (k == HASH_EMPTY) break;
            h = (h + 1) & mask;
        }
        return make_int2(0, 0);
    }
};

// A grid query: f(i, j) for query i and every stored primitive j of its cells whose FP32 box it overlaps, each
// once (in the lowest cell of the two ranges' overlap).  QG lanes per query look its cells up side by side,
// eight at a time, and then share all their candidates: a cell holds a handful of candidates and a box a few
// to BIG_CELLS cells, and each look-up and each candidate is a chain of dependent loads, so one cell after
// the other leaves lanes idle and makes a wide box the kernel's tail (a batch of 64 scenes: 1.24 ms; 0.66 so).  ORDERED: pairs within one list, only those with i < j.
constexpr int QG = 8;
template <bool ORDERED, class F>
__device__ __forceinline__ void grid_walk(int block, int n, const QueryView& qv, const SceneGeo& g, const GridView& gv, const CandView& cv, F f) {
    const int i = (block * 128 + threadIdx.x) / QG, lane = threadIdx.x % QG;
    if (i >= n) return;
    const int4 qc = __ldg(qv.cell + i);
    if (qc.w == 0 || ((qc.w & RECORD_MID) && mids_leave(qv.mid_pairs))) return;
    const float4 qlo = __ldg(qv.box + 2 * (size_t)i), qhi = __ldg(qv.box + 2 * (size_t)i + 1);
    const int sc = __float_as_int(qlo.w);
    const int nx = qc.w & 1023, ny = qc.w >> 10 & 1023, nz = qc.w >> 20 & 1023, cells = nx * ny * nz;
    const unsigned group = 0xffu << (threadIdx.x & 24);
    for (int c0 = 0; c0 < cells; c0 += QG) {
        const int c = c0 + lane, z = c % nz, y = c / nz % ny, x = c / nz / ny;
        const int2 run = c < cells ? gv.find(gkey(g, sc, (long long)qc.x + x, (long long)qc.y + y, (long long)qc.z + z)) : make_int2(0, 0);
        int upto = run.y;   // candidates in the cells up to this lane's
#pragma unroll
        for (int o = 1; o < QG; o <<= 1) {
            const int v = __shfl_up_sync(group, upto, o, QG);
            if (lane >= o) upto += v;
        }
        const int total = __shfl_sync(group, upto, QG - 1, QG), base = run.x - (upto - run.y), packed = x | y << 10 | z << 20;
        for (int q0 = 0; q0 < total; q0 += QG) {
            const int q = q0 + lane;
            int o = 0;   // the cell of candidate q: cells whose count is used up
#pragma unroll
            for (int st = QG / 2; st > 0; st >>= 1)
                if (__shfl_sync(group, upto, o + st - 1, QG) <= q) o += st;
            const int at = __shfl_sync(group, base, o, QG) + q, cell = __shfl_sync(group, packed, o, QG);
            if (q >= total) continue;
            const int j = __ldg(gv.ids + at);
            if (ORDERED && !(i < j)) continue;
            const int4 pc = __ldg(cv.cell + j);
            if (max(qc.x, pc.x) != qc.x + (cell & 1023) || max(qc.y, pc.y) != qc.y + (cell >> 10 & 1023) || max(qc.z, pc.z) != qc.z + (cell >> 20))
                continue;
            if (!f32_overlap(__ldg(cv.box + 2 * (size_t)j), __ldg(cv.box + 2 * (size_t)j + 1), qlo, qhi)) continue;
            f(i, j);
        }
    }
}

// ---------------------------------------------------------------- constraint rows
// A row as a sort key: list (3 bits) and vertex ids (21 bits each, n_verts < 2^21), so that the order of
// the keys is the lists' order and the lexicographic order within each.
struct RowKey {
    unsigned long long hi, lo;   // list, a, b;  c, d
};
__host__ __device__ __forceinline__ bool operator<(const RowKey& p, const RowKey& q) { return p.hi < q.hi || (p.hi == q.hi && p.lo < q.lo); }
__host__ __device__ __forceinline__ bool operator==(const RowKey& p, const RowKey& q) { return p.hi == q.hi && p.lo == q.lo; }
struct RowLess {
    __device__ bool operator()(const RowKey& p, const RowKey& q) const { return p < q; }
};
// device counters of a call (zeroed at its start, copied to the host at its end)
struct BroadCounters {
    int rows[N_TYPES];          // rows of each list, sorted and unique
    int flags;                  // FLAG_*
    int emitted;                // rows emitted (also past the capacity)
    int sorted;                 // rows[] holds the final counts
    int big[2], mid[2];         // triangles, edges of the sizes SIZE_BIG, SIZE_MID
    int pairs[2];               // candidate pairs of the two kinds of a query
    int work[2], doubt[2];      // step filter: pairs that pass the additive bound, the sign filter
    int cursor[2];              // ids handed out to runs (points, edges)
    unsigned long long total[2];   // grid entries (points, edges), but for those of
    unsigned long long mid_total;  // edges of SIZE_MID
    unsigned long long mid_pairs[2];   // tests that the primitives of SIZE_MID would take outside the grid (triangles, edges)
    unsigned long long alpha;   // one scene's step (bits of a double)
    int hit;                    // one scene's intersection flag
    int pad;
};
enum { FLAG_ROWS = 1, FLAG_CELLS = 2, FLAG_TABLE = 4 };
struct RowSink {
    RowKey* rows;
    BroadCounters* n;
    int cap;
};
// Warp-aggregated emission: the lanes that reach this call together reserve their rows with one
// atomicAdd.  The rows are sorted and de-duplicated afterwards, so their order does not matter.
__device__ __forceinline__ void emit(const RowSink& s, int t, int a, int b, int c, int d) {
    const cg::coalesced_group active = cg::coalesced_threads();
    int base = 0;
    if (active.thread_rank() == 0) base = atomicAdd(&s.n->emitted, (int)active.size());
    base = active.shfl(base, 0);
    const int k = base + (int)active.thread_rank();
    if (k < s.cap) s.rows[k] = RowKey{((unsigned long long)t << 42) | ((unsigned long long)a << 21) | (unsigned long long)b,
                                      ((unsigned long long)c << 21) | (unsigned long long)d};
    else atomicOr(&s.n->flags, FLAG_ROWS);
}

// attempt_PT, NEWTON_IPC.py:181-212
__device__ void attempt_pt(const double* __restrict__ x, double dh, double dh2, int p, int t0, int t1, int t2, const RowSink& s) {
    if (p == t0 || p == t1 || p == t2) return;
    const v3 P = ld3(x, p), A = ld3(x, t0), B = ld3(x, t1), C = ld3(x, t2);
    if (!pt_aabb(P, A, B, C, dh)) return;
    switch (pt_type(P, A, B, C)) {
        case 0: if (d_PP(P, A) < dh2) emit(s, T_PP, p, t0, 0, 0); break;
        case 1: if (d_PP(P, B) < dh2) emit(s, T_PP, p, t1, 0, 0); break;
        case 2: if (d_PP(P, C) < dh2) emit(s, T_PP, p, t2, 0, 0); break;
        case 3: if (d_PE(P, A, B) < dh2) emit(s, T_PE, p, t0, t1, 0); break;
        case 4: if (d_PE(P, B, C) < dh2) emit(s, T_PE, p, t1, t2, 0); break;
        case 5: if (d_PE(P, C, A) < dh2) emit(s, T_PE, p, t2, t0, 0); break;
        default: if (d_PT(P, A, B, C) < dh2) emit(s, T_PT, p, t0, t1, t2); break;
    }
}

// attempt_EE, NEWTON_IPC.py:235-312
__device__ void attempt_ee(const double* __restrict__ x, const double* __restrict__ x0, double dh, double dh2, int a0, int a1, int b0,
                           int b1, const RowSink& s) {
    if (a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1) return;
    const v3 A0 = ld3(x, a0), A1 = ld3(x, a1), B0 = ld3(x, b0), B1 = ld3(x, b1);
    if (!ee_aabb(A0, A1, B0, B1, dh)) return;
    // feature pair and its distance first; the mollifier switch (EECN2 < eps_x on the rest
    // shape) is needed only for pairs within d-hat, which is what gets emitted
    int t;
    double d2;
    switch (t = ee_type(A0, A1, B0, B1)) {
        case 0: d2 = d_PP(A0, B0); break;
        case 1: d2 = d_PP(A0, B1); break;
        case 2: d2 = d_PE(A0, B0, B1); break;
        case 3: d2 = d_PP(A1, B0); break;
        case 4: d2 = d_PP(A1, B1); break;
        case 5: d2 = d_PE(A1, B0, B1); break;
        case 6: d2 = d_PE(B0, A0, A1); break;
        case 7: d2 = d_PE(B1, A0, A1); break;
        default: d2 = d_EE(A0, A1, B0, B1); break;
    }
    if (!(d2 < dh2)) return;
    const bool m = d_EECN2(A0, A1, B0, B1) < m_threshold(ld3(x0, a0), ld3(x0, a1), ld3(x0, b0), ld3(x0, b1));
    switch (t) {
        case 0: if (m) emit(s, T_PPM, a0, a1, b0, b1); else emit(s, T_PP, a0, b0, 0, 0); break;
        case 1: if (m) emit(s, T_PPM, a0, a1, b1, b0); else emit(s, T_PP, a0, b1, 0, 0); break;
        case 2: if (m) emit(s, T_PEM, a0, a1, b0, b1); else emit(s, T_PE, a0, b0, b1, 0); break;
        case 3: if (m) emit(s, T_PPM, a1, a0, b0, b1); else emit(s, T_PP, a1, b0, 0, 0); break;
        case 4: if (m) emit(s, T_PPM, a1, a0, b1, b0); else emit(s, T_PP, a1, b1, 0, 0); break;
        case 5: if (m) emit(s, T_PEM, a1, a0, b0, b1); else emit(s, T_PE, a1, b0, b1, 0); break;
        case 6: if (m) emit(s, T_PEM, b0, b1, a0, a1); else emit(s, T_PE, b0, a0, a1, 0); break;
        case 7: if (m) emit(s, T_PEM, b1, b0, a0, a1); else emit(s, T_PE, b1, a0, a1, 0); break;
        default: if (m) emit(s, T_EEM, a0, a1, b0, b1); else emit(s, T_EE, a0, a1, b0, b1); break;
    }
}

// ---------------------------------------------------------------- candidate pairs
// The grid walks and the big-primitive passes only test FP32 boxes; the pairs that pass go to a list, one
// per kind, and the FP64 narrow phase runs over the lists with every lane on a pair.  In the walk itself one
// or two lanes of a warp would run it while the others wait, and a warp's FP64 instruction takes 19
// clocks of the SM whatever its active lanes.  A list that is full leaves its pair to the walking lane;
// the next call's is larger.
struct PairList {
    int2* w;               // [2 cap]: pairs of the first kind, then of the second
    int* count;            // [2] (may exceed cap)
    int cap;
};
// one atomic per coalesced group; false when the list is full
__device__ __forceinline__ bool pair_push(const PairList& L, int kind, int a, int b) {
    if (*(volatile int*)(L.count + kind) >= L.cap) return false;
    const cg::coalesced_group g = cg::coalesced_threads();
    int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(L.count + kind, (int)g.size());
    base = g.shfl(base, 0);
    const int k = base + (int)g.thread_rank();
    if (k >= L.cap) return false;
    L.w[(size_t)kind * L.cap + k] = make_int2(a, b);
    return true;
}
constexpr int PAIR_THREADS = 64, PAIR_BLOCKS = 16 * SMS;
// f(kind, pair) for every listed pair; a warp's pairs are of one kind
template <class F>
__device__ __forceinline__ void each_pair(const PairList& L, F f) {
    const int n0 = min(L.count[0], L.cap), n1 = min(L.count[1], L.cap), m0 = (n0 + 31) & ~31;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m0 + n1; k += gridDim.x * blockDim.x) {
        if (k < m0) {
            if (k < n0) f(0, L.w[k]);
        } else {
            f(1, L.w[(size_t)L.cap + (k - m0)]);
        }
    }
}

// the rows of point-triangle (kind 0: vertex, triangle) and edge-edge (kind 1) pairs
struct FindArgs {
    const int *bt, *be;
    const double *x, *x0;
    double dh, dh2;
};
__device__ __forceinline__ void find_pair(const FindArgs& a, int kind, int i, int j, const RowSink& s) {
    if (kind == 0) attempt_pt(a.x, a.dh, a.dh2, i, a.bt[3 * j], a.bt[3 * j + 1], a.bt[3 * j + 2], s);
    else attempt_ee(a.x, a.x0, a.dh, a.dh2, a.be[2 * i], a.be[2 * i + 1], a.be[2 * j], a.be[2 * j + 1], s);
}
__device__ __noinline__ void find_pair_call(const FindArgs& a, int kind, int i, int j, const RowSink& s) { find_pair(a, kind, i, j, s); }
__global__ void __launch_bounds__(PAIR_THREADS) k_find_pairs(FindArgs a, PairList L, RowSink s) {
    each_pair(L, [&](int kind, int2 q) { find_pair(a, kind, q.x, q.y, s); });
}

// triangles query points hashed with mode 0 (their box against pt_aabb's, the point's +- dh), edges edges
// hashed with mode 1 (query box +- dh)
__device__ __forceinline__ void find_pt(int block, int nbt, const int* __restrict__ bp, const FindArgs& a, const QueryView& qv,
                                        const SceneGeo& g, const GridView& gv, const CandView& cv, const PairList& L, const RowSink& sink) {
    grid_walk<false>(block, nbt, qv, g, gv, cv, [&](int i, int j) {
        const int p = bp[j];
        if (p == a.bt[3 * i] || p == a.bt[3 * i + 1] || p == a.bt[3 * i + 2]) return;
        if (!pair_push(L, 0, p, i)) find_pair_call(a, 0, p, i, sink);
    });
}
__device__ __forceinline__ bool edges_touch(const int* __restrict__ be, int i, int j) {
    const int a0 = be[2 * i], a1 = be[2 * i + 1], b0 = be[2 * j], b1 = be[2 * j + 1];
    return a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1;
}
__device__ __forceinline__ void find_ee(int block, int nbe, const FindArgs& a, const QueryView& qv, const SceneGeo& g, const GridView& gv,
                                        const CandView& cv, const PairList& L, const RowSink& sink) {
    grid_walk<true>(block, nbe, qv, g, gv, cv, [&](int i, int j) {
        if (edges_touch(a.be, i, j)) return;
        if (!pair_push(L, 1, i, j)) find_pair_call(a, 1, i, j, sink);
    });
}

// ---------------------------------------------------------------- CCD step filter
// A query's candidate pairs are tested in three steps of falling width, each over the list the one before
// leaves: moving boxes and the additive bound (k_ccd_pairs), the signs of the interval test's
// polynomials (k_ccd_signs), the interval test with its root finding (k_ccd_exact).  The minimum over
// pairs does not depend on where a pair's toc is computed.
struct CcdWork {
    int a, b, slot, pad;   // point-triangle: vertex, triangle; edge-edge: edge, edge; filter slot
    double d2, lb;         // current squared distance, additive lower bound
};
struct CcdList {
    CcdWork* w;            // [2 cap]: point-triangle pairs, then edge-edge pairs
    int* count;            // [2] pushes (may exceed cap: the lanes past it run the exact test themselves)
    int cap;
};

// appends e for every calling lane (one atomic per coalesced group); false when the list is full
__device__ __forceinline__ bool ccd_push(CcdWork* w, int* count, int cap, const CcdWork& e) {
    cg::coalesced_group g = cg::coalesced_threads();
    int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(count, (int)g.size());
    base = g.shfl(base, 0);
    const int k = base + (int)g.thread_rank();
    if (k >= cap) return false;
    w[k] = e;
    return true;
}

__device__ __forceinline__ void atomic_min_pos(unsigned long long* slot, double v) {
    if (v >= 0.0) atomicMin(slot, (unsigned long long)__double_as_longlong(v));
}

struct CcdArgs {
    const int *bt, *be;
    const double *x, *p;
    double dh, eta;
    const int* vscene;
    unsigned long long* alpha;
};
struct Quad {
    v3 X[4], D[4];
    int v0;
};
// a pair's vertices and directions: point, triangle (kind 0) or the two edges (kind 1)
__device__ __forceinline__ Quad quad_of(const CcdArgs& a, int kind, int i, int j) {
    int v[4];
    if (kind == 0) {
        v[0] = i;
#pragma unroll
        for (int k = 0; k < 3; ++k) v[1 + k] = a.bt[3 * j + k];
    } else {
        v[0] = a.be[2 * i];
        v[1] = a.be[2 * i + 1];
        v[2] = a.be[2 * j];
        v[3] = a.be[2 * j + 1];
    }
    Quad q;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q.X[k] = ld3(a.x, v[k]);
        q.D[k] = ld3(a.p, v[k]);
    }
    q.v0 = v[0];
    return q;
}
__device__ __forceinline__ double exact_toc(const Quad& q, int kind, double eta, double d2, double lb) {
    return kind == 0 ? pt_ccd_exact(q.X[0], q.X[1], q.X[2], q.X[3], q.D[0], q.D[1], q.D[2], q.D[3], eta, d2, lb)
                     : ee_ccd_exact(q.X[0], q.X[1], q.X[2], q.X[3], q.D[0], q.D[1], q.D[2], q.D[3], eta, d2, lb);
}
// moving boxes and the additive bound; a full work list leaves the exact test to the calling lane
__device__ __forceinline__ void ccd_pair(const CcdArgs& a, int kind, int i, int j, const CcdList& L) {
    const Quad q = quad_of(a, kind, i, j);
    double d2, lb;
    if (kind == 0) {
        if (!pt_aabb_moving(q.X[0], q.X[1], q.X[2], q.X[3], q.D[0], q.D[1], q.D[2], q.D[3], a.dh)) return;
        d2 = pt_dist2(q.X[0], q.X[1], q.X[2], q.X[3]);
        if (!pt_needs_exact(q.D[0], q.D[1], q.D[2], q.D[3], a.eta, d2, &lb)) return;
    } else {
        if (!ee_aabb_moving(q.X[0], q.X[1], q.X[2], q.X[3], q.D[0], q.D[1], q.D[2], q.D[3], a.dh)) return;
        d2 = ee_dist2(q.X[0], q.X[1], q.X[2], q.X[3]);
        if (!ee_needs_exact(q.D[0], q.D[1], q.D[2], q.D[3], a.eta, d2, &lb)) return;
    }
    const int slot = a.vscene ? a.vscene[q.v0] : 0;
    if (!ccd_push(L.w + (size_t)kind * L.cap, L.count + kind, L.cap, CcdWork{i, j, slot, 0, d2, lb}))
        atomic_min_pos(a.alpha + slot, exact_toc(q, kind, a.eta, d2, lb));
}
__device__ __noinline__ void ccd_pair_call(const CcdArgs& a, int kind, int i, int j, const CcdList& L) { ccd_pair(a, kind, i, j, L); }
__global__ void __launch_bounds__(PAIR_THREADS) k_ccd_pairs(CcdArgs a, PairList P, CcdList L) {
    each_pair(P, [&](int kind, int2 q) { ccd_pair(a, kind, q.x, q.y, L); });
}

// a pair's toc is at least its additive bound: one whose bound is not below the minimum so far cannot
// lower it
__device__ __forceinline__ bool may_lower(const CcdArgs& a, const CcdWork& e) {
    return e.lb < __longlong_as_double((long long)*(volatile unsigned long long*)(a.alpha + e.slot));
}
// pairs that the signs of the polynomials do not decide (most never come close), from L to M (as large)
__global__ void __launch_bounds__(PAIR_THREADS) k_ccd_signs(CcdArgs a, CcdList L, CcdList M) {
    const int half = gridDim.x / 2, kind = (int)blockIdx.x < half ? 0 : 1;
    const int n = min(L.count[kind], L.cap);
    for (int k = (blockIdx.x - (kind ? half : 0)) * blockDim.x + threadIdx.x; k < n; k += half * blockDim.x) {
        const CcdWork e = L.w[(size_t)kind * L.cap + k];
        if (!may_lower(a, e)) continue;
        const Quad q = quad_of(a, kind, e.a, e.b);
        const double eta = a.eta * sqrt(e.d2);
        const v3 Y[4] = {q.X[0] + q.D[0], q.X[1] + q.D[1], q.X[2] + q.D[2], q.X[3] + q.D[3]};
        if (kind == 0 ? vertex_face_apart(q.X[0], q.X[1], q.X[2], q.X[3], Y[0], Y[1], Y[2], Y[3], eta)
                      : edge_edge_apart(q.X[0], q.X[1], q.X[2], q.X[3], Y[0], Y[1], Y[2], Y[3], eta))
            continue;
        ccd_push(M.w + (size_t)kind * M.cap, M.count + kind, M.cap, e);
    }
}

// The exact test of the pairs left, eight lanes per pair: each finds the intervals of one of its four
// (point-triangle: distance, three sides) or five (edge-edge: distance, four barycentric) polynomials, all in
// the same code, and the first lane intersects them.  One thread per pair runs the root finding of its
// polynomials one after the other, a chain of dependent FP64 operations of hundreds of microseconds
// for the few hundred pairs that come this far.
constexpr int EXACT_LANES = 8;
__global__ void __launch_bounds__(PAIR_THREADS) k_ccd_exact(CcdArgs a, CcdList M) {
    __shared__ Ivl sh[PAIR_THREADS][8];
    __shared__ int sn[PAIR_THREADS];
    const int half = gridDim.x / 2, kind = (int)blockIdx.x < half ? 0 : 1;
    const int n = min(M.count[kind], M.cap);
    const int l = threadIdx.x % EXACT_LANES, t0 = threadIdx.x - l;
    constexpr int PER = PAIR_THREADS / EXACT_LANES;   // pairs per CTA and pass
    for (int k0 = (blockIdx.x - (kind ? half : 0)) * PER; k0 < n; k0 += half * PER) {
        const int k = k0 + threadIdx.x / EXACT_LANES;
        bool act = k < n;
        CcdWork e{};
        if (act) {
            e = M.w[(size_t)kind * M.cap + k];
            // one answer for the group: the minimum may move between its lanes' reads
            const int first = (int)(threadIdx.x & 31) - l;
            act = __shfl_sync(0xffu << first, (int)may_lower(a, e), first) != 0;
        }
        sn[threadIdx.x] = 0;
        Quad q{};
        double minD = 0.0;
        if (act) {
            q = quad_of(a, kind, e.a, e.b);
            minD = a.eta * sqrt(e.d2);
            minD *= minD;
            v3 V[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) V[v] = (q.X[v] + q.D[v]) - q.X[v];
            double op[7];
            int deg = 0;
            if (kind == 0) {
                if (l == 3) {
                    distance_coefficients(q.X[0] - q.X[1], q.X[2] - q.X[1], q.X[3] - q.X[1], V[0] - V[1], V[2] - V[1], V[3] - V[1], minD, op);
                    deg = 6;
                } else if (l < 3) {
                    // side l: from its first vertex the next but one and the next
                    const v3 o = l == 0 ? q.X[1] : (l == 1 ? q.X[2] : q.X[3]), u = l == 0 ? q.X[3] : (l == 1 ? q.X[1] : q.X[2]),
                             w = l == 0 ? q.X[2] : (l == 1 ? q.X[3] : q.X[1]);
                    const v3 vo = l == 0 ? V[1] : (l == 1 ? V[2] : V[3]), vu = l == 0 ? V[3] : (l == 1 ? V[1] : V[2]),
                             vw = l == 0 ? V[2] : (l == 1 ? V[3] : V[1]);
                    plane_coefficients(q.X[0] - o, cross(u - o, w - o), u - o, V[0] - vo, cross(vu - vo, vw - vo), vu - vo, op);
                    deg = 3;
                }
            } else {
                // q0, p0, q1, p1 = X[0..3]
                if (l == 4) {
                    distance_coefficients(q.X[1] - q.X[3], q.X[1] - q.X[0], q.X[3] - q.X[2], V[1] - V[3], V[1] - V[0], V[3] - V[2], minD, op);
                    deg = 6;
                } else if (l < 4) {
                    const bool second = l >= 2, flip = l & 1;   // whose parameter; from which end
                    const v3 q0 = second ? q.X[2] : q.X[0], p0 = second ? q.X[3] : q.X[1], q1 = second ? q.X[0] : q.X[2],
                             p1 = second ? q.X[1] : q.X[3];
                    const v3 vq0 = second ? V[2] : V[0], vp0 = second ? V[3] : V[1], vq1 = second ? V[0] : V[2], vp1 = second ? V[1] : V[3];
                    const v3 s = flip ? q0 : p0, f = flip ? p0 : q0, vs = flip ? vq0 : vp0, vf = flip ? vp0 : vq0;
                    bary_coefficients(p1 - q1, s - f, f - q1, vp1 - vq1, vs - vf, vf - vq1, op);
                    deg = 4;
                }
            }
            if (deg) {
                int ni;
                find_intervals(op, deg, sh[threadIdx.x], &ni, deg != 6);
                sn[threadIdx.x] = ni;
            }
        }
        __syncwarp();
        if (act && l == 0) {
            double toc = 1.0;
            bool col = true;
            for (int v = 0; v < 4 + kind; ++v) col = col && sn[t0 + v] > 0;
            if (col && kind == 0) {
                col = vertex_face_meet(sh[t0 + 3], sn[t0 + 3], sh[t0], sn[t0], sh[t0 + 1], sn[t0 + 1], sh[t0 + 2], sn[t0 + 2], &toc);
            } else if (col) {
                v3 V[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) V[v] = (q.X[v] + q.D[v]) - q.X[v];
                Ivl cp[8], par[8];
                int ncp, npar;
                split_parallel(sh[t0 + 4], sn[t0 + 4], q.X[0] - q.X[1], V[0] - V[1], q.X[2] - q.X[3], V[2] - V[3], cp, &ncp, par, &npar);
                col = edge_edge_meet(cp, ncp, par, npar, sh[t0], sn[t0], sh[t0 + 1], sn[t0 + 1], sh[t0 + 2], sn[t0 + 2], sh[t0 + 3],
                                     sn[t0 + 3], &toc);
            }
            if (col && toc < e.lb) toc = e.lb;
            if (toc < 1.0) atomic_min_pos(a.alpha + e.slot, toc);
        }
        __syncwarp();
    }
}

// compute_filter_3D_PT (NEWTON_IPC.py:377-406): triangles query their moving bbox; compute_filter_3D_EE
// (409-440): edges query moving bbox +- dh
__device__ __forceinline__ void ccd_pt(int block, int nbt, const int* __restrict__ bp, const CcdArgs& a, const QueryView& qv, const SceneGeo& g,
                                       const GridView& gv, const CandView& cv, const PairList& P, const CcdList& L) {
    grid_walk<false>(block, nbt, qv, g, gv, cv, [&](int i, int j) {
        const int p = bp[j];
        if (p == a.bt[3 * i] || p == a.bt[3 * i + 1] || p == a.bt[3 * i + 2]) return;
        if (!pair_push(P, 0, p, i)) ccd_pair_call(a, 0, p, i, L);
    });
}
__device__ __forceinline__ void ccd_ee(int block, int nbe, const CcdArgs& a, const QueryView& qv, const SceneGeo& g, const GridView& gv,
                                       const CandView& cv, const PairList& P, const CcdList& L) {
    grid_walk<true>(block, nbe, qv, g, gv, cv, [&](int i, int j) {
        if (edges_touch(a.be, i, j)) return;
        if (!pair_push(P, 1, i, j)) ccd_pair_call(a, 1, i, j, L);
    });
}

// compute_filter_3D_inversion_free (NEWTON_IPC.py:443-453)
__global__ void __launch_bounds__(128) k_ccd_inversion(int nT, const int4* __restrict__ tets, const double* __restrict__ x,
                                                       const double* __restrict__ p, double eta, SceneGeo g,
                                                       unsigned long long* __restrict__ alpha) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nT) return;
    const int4 t = tets[e];
    const v3 X[4] = {ld3(x, t.x), ld3(x, t.y), ld3(x, t.z), ld3(x, t.w)};
    const v3 P[4] = {ld3(p, t.x), ld3(p, t.y), ld3(p, t.z), ld3(p, t.w)};
    if (inversion_cannot_flip(X, P, eta)) return;
    atomic_min_pos(alpha + (g.vscene ? g.scene(t.x) : 0), inversion_free_step(X, P, eta));
}

// check_collision_3d (NEWTON_IPC.py:855-880): an edge against a triangle
struct HitArgs {
    const int *bt, *be;
    const double* x;
    const int* vscene;
    int* hit;
};
__device__ __forceinline__ void hit_pair(const HitArgs& a, int e, int t) {
    const int t0 = a.bt[3 * t], t1 = a.bt[3 * t + 1], t2 = a.bt[3 * t + 2];
    int* h = a.hit + (a.vscene ? a.vscene[t0] : 0);
    if (*(volatile int*)h) return;
    if (seg_tri(ld3(a.x, a.be[2 * e]), ld3(a.x, a.be[2 * e + 1]), ld3(a.x, t0), ld3(a.x, t1), ld3(a.x, t2))) atomicOr(h, 1);
}
__device__ __noinline__ void hit_pair_call(const HitArgs& a, int e, int t) { hit_pair(a, e, t); }
__global__ void __launch_bounds__(PAIR_THREADS) k_collision_pairs(HitArgs a, PairList P) {
    each_pair(P, [&](int, int2 q) { hit_pair(a, q.x, q.y); });
}

// an edge and a triangle of which it is no part
__device__ __forceinline__ bool edge_of_triangle(const int* __restrict__ be, const int* __restrict__ bt, int e, int t) {
    const int t0 = bt[3 * t], t1 = bt[3 * t + 1], t2 = bt[3 * t + 2], a0 = be[2 * e], a1 = be[2 * e + 1];
    return a0 == t0 || a0 == t1 || a0 == t2 || a1 == t0 || a1 == t1 || a1 == t2;
}
// triangles query bbox cells, edges hashed +- dh
__device__ __forceinline__ void collision_grid(int block, int nbt, const HitArgs& a, const QueryView& qv, const SceneGeo& g, const GridView& gv,
                                               const CandView& cv, const PairList& P) {
    grid_walk<false>(block, nbt, qv, g, gv, cv, [&](int i, int j) {
        if (edge_of_triangle(a.be, a.bt, j, i)) return;
        if (!pair_push(P, 0, j, i)) hit_pair_call(a, j, i);
    });
}

// ---------------------------------------------------------------- big primitives
// A triangle or edge whose query box covers more than BIG_CELLS cells (a ground plane meshed
// with a few large triangles next to finely meshed bodies) would enumerate, or be stored in,
// thousands of cells.  Such primitives leave the grid: each is tested against every primitive
// of its own scene with the same narrow phase, so the results are the grid's.
// Between MID_CELLS and BIG_CELLS both are possible.  A few such boxes are the tail of every walk and of filling the table
// (us in the grid / outside: pile of 180 cubes at rest, 8 edges, intersection check 636 / 522, find 759 / 726;
// 64 scenes, find 1365 / 1266; a pile of 8 cubes, the step filter 150 / 126).  But a moving box grows with its step: from
// some two cells along every axis or 14 along one, all triangles and edges of a body are such boxes, and outside the grid a
// step filter tests all pairs (180 cubes that fall by 40 cells 85 ms / 310, one of them 1.9 / 2.6).  So the line counts the
// tests outside, MID_PAIRS = 8.4M a kind.  Both sides near it: 3.8M and 8.2M pairs of edges, find 396 / 315 and 396 / 406;
// 6.1M and 13.9M pairs of a triangle and an edge, check 514 / 355 and 515 / 569; 10.8M and 29M pairs of edges, step
// filter 2169 / 1589 and 1331 / 1545.

__device__ __forceinline__ long long box_cells(v3 lo, v3 hi, double inv_dx) {
    const C3 a = cell_of(lo, inv_dx), b = cell_of(hi, inv_dx);
    return (b.x - a.x + 1) * (b.y - a.y + 1) * (b.z - a.z + 1);
}

// the partners of big primitive q of scene s are lists [off[s], off[s+1]) of its kind, in chunks of
// BIG_CHUNK: CTA (chunk, y) takes that chunk of the big primitives y, y + ny, ...  (One CTA per big
// primitive walked all its partners: on a pile of 180 cubes over a 12-triangle ground box 2 to 4 ms per
// query; the whole queries now take 0.9 to 2.2 ms.)  A partner's FP32 box (CandView; rounded outward, so equality counts as a
// touch) spares most of the FP64 tests.
struct BigArgs {
    const int *bp, *be, *bt;
    const int* off;        // [3][S+1]: points, edges, triangles
    int S;
    const unsigned char *tri_size, *edge_size;
    const int* list;       // [nbt + nbe]: triangles, then edges; of each the big ones from the front, the mid ones from the end
    const BroadCounters* n;
    int nbt, nbe, ny;
    __device__ __forceinline__ bool mids(int kind) const { return mids_leave(n->mid_pairs + kind); }
    // whether a primitive of this size is out of the grid (mids: mids(kind))
    __device__ __forceinline__ bool out(unsigned char size, bool mids) const { return size == SIZE_BIG || (size == SIZE_MID && mids); }
};
constexpr int BIG_CHUNK = 512;
__device__ __forceinline__ bool f32_touch(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    return alo.x <= bhi.x && alo.y <= bhi.y && alo.z <= bhi.z && blo.x <= ahi.x && blo.y <= ahi.y && blo.z <= ahi.z;
}
struct BoxF {
    float4 lo, hi;
};
__device__ __forceinline__ bool touches(const CandView& cv, int k, const BoxF& b) {
    return f32_touch(__ldg(cv.box + 2 * (size_t)k), __ldg(cv.box + 2 * (size_t)k + 1), b.lo, b.hi);
}
// f(i, k, box(i)) for primitive i out of the grid (kind 0: triangle, 1: edge) and its partners k in this CTA's chunk, of
// list `partners` (0 points, 1 edges, 2 triangles)
template <class BOX, class F>
__device__ __forceinline__ void big_pairs(const BigArgs& b, const SceneGeo& g, int block, int kind, int partners, BOX box, F f) {
    const int chunk = block / b.ny, big = b.n->big[kind], count = big + (b.mids(kind) ? b.n->mid[kind] : 0);
    const int first = kind ? b.nbt : 0, last = (kind ? b.nbt + b.nbe : b.nbt) - 1;
    const int* off = b.off + partners * (b.S + 1);
    for (int q = block % b.ny; q < count; q += b.ny) {
        const int i = q < big ? b.list[first + q] : b.list[last - (q - big)];
        const int sc = g.scene(kind ? b.be[2 * i] : b.bt[3 * i]);
        const int k0 = off[sc] + chunk * BIG_CHUNK, k1 = min(off[sc + 1], k0 + BIG_CHUNK);
        if (k0 >= k1) continue;
        const BoxF bx = box(i);
        for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) f(i, k, bx);
    }
}

// find_constraints: big triangles against the points, big edges against the edges of their scene (a pair
// of two big edges once, from its lower index; rows formed with the lower list index first as in the
// grid pass)
__device__ __forceinline__ BoxF triangle_box(const int* __restrict__ bt, int i, const double* __restrict__ x, double dh) {
    const v3 A = ld3(x, bt[3 * i]), B = ld3(x, bt[3 * i + 1]), C = ld3(x, bt[3 * i + 2]), d = mk(dh, dh, dh);
    return BoxF{f32_lo(vmin(vmin(A, B), C) - d), f32_hi(vmax(vmax(A, B), C) + d)};
}
__device__ __forceinline__ void find_pt_big(int block, const BigArgs& b, const FindArgs& a, const SceneGeo& g, CandView cv, const PairList& P,
                                            const RowSink& sink) {
    big_pairs(b, g, block, 0, 0, [&](int i) { return triangle_box(b.bt, i, a.x, a.dh); }, [&](int i, int k, const BoxF& bx) {
        if (!touches(cv, k, bx)) return;
        if (!pair_push(P, 0, b.bp[k], i)) find_pair_call(a, 0, b.bp[k], i, sink);
    });
}
__device__ __forceinline__ void find_ee_big(int block, const BigArgs& b, const FindArgs& a, const SceneGeo& g, CandView cv, const PairList& P,
                                            const RowSink& sink) {
    const bool mids = b.mids(1);
    big_pairs(b, g, block, 1, 1, [&](int i) {
        const v3 A0 = ld3(a.x, b.be[2 * i]), A1 = ld3(a.x, b.be[2 * i + 1]);
        return BoxF{f32_lo(vmin(A0, A1)), f32_hi(vmax(A0, A1))};
    }, [&](int i, int j, const BoxF& bx) {
        if (j == i || (j < i && b.out(b.edge_size[j], mids))) return;
        if (!touches(cv, j, bx)) return;
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        if (edges_touch(b.be, lo, hi)) return;
        if (!pair_push(P, 1, lo, hi)) find_pair_call(a, 1, lo, hi, sink);
    });
}

// CCD filter: big moving triangles against the points, big moving edges against the edges of their scene
__device__ __forceinline__ void ccd_pt_big(int block, const BigArgs& b, const CcdArgs& a, const SceneGeo& g, CandView cv, const PairList& Q,
                                           const CcdList& L) {
    big_pairs(b, g, block, 0, 0, [&](int i) {
        const int t0 = b.bt[3 * i], t1 = b.bt[3 * i + 1], t2 = b.bt[3 * i + 2];
        const v3 A = ld3(a.x, t0), B = ld3(a.x, t1), C = ld3(a.x, t2), dA = ld3(a.p, t0), dB = ld3(a.p, t1), dC = ld3(a.p, t2);
        const v3 mn = vmin(vmin(vmin(A, A + dA), vmin(B, B + dB)), vmin(C, C + dC));
        const v3 mx = vmax(vmax(vmax(A, A + dA), vmax(B, B + dB)), vmax(C, C + dC)), d = mk(a.dh, a.dh, a.dh);
        return BoxF{f32_lo(mn - d), f32_hi(mx + d)};
    }, [&](int i, int k, const BoxF& bx) {
        if (!touches(cv, k, bx)) return;
        const int pp = b.bp[k];
        if (pp == b.bt[3 * i] || pp == b.bt[3 * i + 1] || pp == b.bt[3 * i + 2]) return;
        if (!pair_push(Q, 0, pp, i)) ccd_pair_call(a, 0, pp, i, L);
    });
}
__device__ __forceinline__ void ccd_ee_big(int block, const BigArgs& b, const CcdArgs& a, const SceneGeo& g, CandView cv, const PairList& Q,
                                           const CcdList& L) {
    const bool mids = b.mids(1);
    big_pairs(b, g, block, 1, 1, [&](int i) {
        const v3 I0 = ld3(a.x, b.be[2 * i]), I1 = ld3(a.x, b.be[2 * i + 1]), dI0 = ld3(a.p, b.be[2 * i]), dI1 = ld3(a.p, b.be[2 * i + 1]);
        return BoxF{f32_lo(vmin(vmin(I0, I0 + dI0), vmin(I1, I1 + dI1))), f32_hi(vmax(vmax(I0, I0 + dI0), vmax(I1, I1 + dI1)))};
    }, [&](int i, int j, const BoxF& bx) {
        if (j == i || (j < i && b.out(b.edge_size[j], mids))) return;
        if (!touches(cv, j, bx)) return;
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        if (edges_touch(b.be, lo, hi)) return;
        if (!pair_push(Q, 1, lo, hi)) ccd_pair_call(a, 1, lo, hi, L);
    });
}

// intersection check: big triangles against the edges of their scene, big edges against the triangles of
// their scene that are in the grid (kind: which)
__device__ __forceinline__ void collision_big(int block, int kind, const BigArgs& b, const HitArgs& a, const SceneGeo& g, CandView cv,
                                              const PairList& P) {
    const bool mids = b.mids(0);
    big_pairs(b, g, block, kind, kind ? 2 : 1, [&](int i) {
        return kind ? BoxF{__ldg(cv.box + 2 * (size_t)i), __ldg(cv.box + 2 * (size_t)i + 1)} : triangle_box(b.bt, i, a.x, 0.0);
    }, [&](int i, int k, const BoxF& bx) {
        const int e = kind ? i : k, t = kind ? k : i;
        if (kind && b.out(b.tri_size[t], mids)) return;
        if (edge_of_triangle(b.be, b.bt, e, t)) return;
        if (kind) {
            const BoxF tb = triangle_box(b.bt, t, a.x, 0.0);
            if (!f32_touch(bx.lo, bx.hi, tb.lo, tb.hi)) return;
        } else if (!touches(cv, e, bx)) {
            return;
        }
        if (!pair_push(P, 0, e, t)) hit_pair_call(a, e, t);
    });
}

// ---------------------------------------------------------------- building the grids
// one grid: n stored primitives of a box mode
struct GridBuild {
    const int* prim;
    int n, mode;
    int4 *cell, *ext;
    float4* box;
    unsigned long long* hk;
    int* cnt;
    int2* run;
    int* ids;
    unsigned long long mask;   // table size - 1; the ids hold half the table size
};

// sizes and lists of the big and mid primitives (triangle boxes as queried: static or moving; edge boxes as
// queried: static or moving, +- dh), candidate records and entry counts of both grids' primitives, and
// the tables cleared.  off, S: the scenes' boundary lists (BigArgs)
__global__ void __launch_bounds__(256) k_prepare(int nbt, const int* __restrict__ bt, int nbe, const int* __restrict__ be, GridBuild gp,
                                                 GridBuild ge, const double* __restrict__ x, const double* __restrict__ p, double dh,
                                                 SceneGeo g, QueryView qt, QueryView qe, const int* __restrict__ off, int S,
                                                 unsigned char* __restrict__ tri_size, unsigned char* __restrict__ edge_size,
                                                 int* __restrict__ list, BroadCounters* __restrict__ n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
    if (k == 0) n->alpha = (unsigned long long)__double_as_longlong(1.0);
    for (unsigned long long h = k; h <= gp.mask; h += nthr) {
        gp.hk[h] = HASH_EMPTY;
        gp.cnt[h] = 0;
    }
    for (unsigned long long h = k; h <= ge.mask; h += nthr) {
        ge.hk[h] = HASH_EMPTY;
        ge.cnt[h] = 0;
    }
    const v3 d = mk(dh, dh, dh);
    const bool check = ge.mode == 4;   // the intersection check: triangles against edges, boxes without dh
    auto partners = [&](int l, int sc) { return (long long)(off[l * (S + 1) + sc + 1] - off[l * (S + 1) + sc]); };
    // entries of this thread's primitive (a point, an edge, one of SIZE_MID) and its tests outside the grid
    long long point_cells = 0, edge_cells = 0, mid_cells = 0, tri_pairs = 0, edge_pairs = 0;
    if (k < nbt) {
        const int t0 = bt[3 * k], t1 = bt[3 * k + 1], t2 = bt[3 * k + 2];
        v3 lo = vmin(vmin(ld3(x, t0), ld3(x, t1)), ld3(x, t2)), hi = vmax(vmax(ld3(x, t0), ld3(x, t1)), ld3(x, t2));
        if (p) {
            const v3 A = ld3(x, t0) + ld3(p, t0), B = ld3(x, t1) + ld3(p, t1), C = ld3(x, t2) + ld3(p, t2);
            lo = vmin(lo, vmin(vmin(A, B), C));
            hi = vmax(hi, vmax(vmax(A, B), C));
        }
        const int sc = g.scene(t0);
        const double inv_dx = g.idx(sc);
        const int size = size_of(box_cells(lo, hi, inv_dx));
        query_record(qt, k, sc, size, cell_of(lo, inv_dx), cell_of(hi, inv_dx), check ? lo : lo - d, check ? hi : hi + d);
        tri_size[k] = size;
        if (size == SIZE_BIG) list[atomicAdd(&n->big[0], 1)] = k;
        if (size == SIZE_MID) {
            list[nbt - 1 - atomicAdd(&n->mid[0], 1)] = k;
            tri_pairs = partners(check ? 1 : 0, sc);
        }
    } else if (k < nbt + nbe + gp.n) {
        const bool edge = k < nbt + nbe;
        const GridBuild& b = edge ? ge : gp;
        const int i = edge ? k - nbt : k - nbt - nbe;
        const int sv = edge ? be[2 * i] : b.prim[i];
        const int sc = g.scene(sv);
        const double inv_dx = g.idx(sc);
        int size = SIZE_GRID;
        if (edge) {
            const int a1 = be[2 * i + 1];
            v3 lo = vmin(ld3(x, sv), ld3(x, a1)), hi = vmax(ld3(x, sv), ld3(x, a1));
            if (p) {
                const v3 A = ld3(x, sv) + ld3(p, sv), B = ld3(x, a1) + ld3(p, a1);
                lo = vmin(lo, vmin(A, B));
                hi = vmax(hi, vmax(A, B));
            }
            size = size_of(box_cells(lo - d, hi + d, inv_dx));
            if (!check) query_record(qe, i, sc, size, cell_of(lo - d, inv_dx), cell_of(hi + d, inv_dx), lo, hi);
            edge_size[i] = size;
            if (size == SIZE_BIG) list[nbt + atomicAdd(&n->big[1], 1)] = i;
            if (size == SIZE_MID) {
                list[nbt + nbe - 1 - atomicAdd(&n->mid[1], 1)] = i;
                edge_pairs = partners(check ? 2 : 1, sc);
            }
        }
        v3 lo, hi;
        stored_box(b.mode, i, b.prim, x, p, dh, &lo, &hi);
        const C3 a = cell_of(lo, inv_dx), e = cell_of(hi, inv_dx);
        cand_record(b.mode, i, b.prim, x, p, dh, lo, hi, a, b.cell, b.box);
        long long c = 0;
        if (size != SIZE_BIG) {
            c = (e.x - a.x + 1) * (e.y - a.y + 1) * (e.z - a.z + 1);
            if (!(c > 0 && c <= MAX_CELLS_PER_PRIM)) {
                atomicOr(&n->flags, FLAG_CELLS);
                c = 0;
            }
        }
        b.ext[i] = c ? make_int4((int)(e.x - a.x + 1), (int)(e.y - a.y + 1), (int)(e.z - a.z + 1), sc | (size == SIZE_MID ? RECORD_MID : 0))
                     : make_int4(0, 0, 0, sc);
        if (size == SIZE_MID) mid_cells = c;
        else if (edge) edge_cells = c;
        else point_cells = c;
    }
    // totals: one add per warp
    auto add = [](long long c, unsigned long long* to) {
        if (!__any_sync(0xffffffffu, c != 0)) return;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(to, (unsigned long long)c);
    };
    add(point_cells, n->total);
    add(edge_cells, n->total + 1);
    add(mid_cells, &n->mid_total);
    add(tri_pairs, n->mid_pairs);
    add(edge_pairs, n->mid_pairs + 1);
}

// f(key, i) for every (cell, primitive) entry of both grids; four lanes share a primitive's cells.
// Nothing happens when a table is too small for its entries (the call is then repeated).
constexpr int CELL_LANES = 4;
template <class F>
__device__ __forceinline__ void each_entry(const GridBuild& gp, const GridBuild& ge, const SceneGeo& g, BroadCounters* n, F f) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) / CELL_LANES, lane = threadIdx.x % CELL_LANES;
    const bool mids = mids_leave(n->mid_pairs + 1);
    if (2 * n->total[0] > gp.mask + 1 || 2 * (n->total[1] + (mids ? 0 : n->mid_total)) > ge.mask + 1) {
        if (k == 0 && lane == 0) atomicOr(&n->flags, FLAG_TABLE);
        return;
    }
    if (k >= gp.n + ge.n) return;
    const bool edge = k >= gp.n;
    const GridBuild& b = edge ? ge : gp;
    const int i = edge ? k - gp.n : k;
    const int4 a = __ldg(b.cell + i), e = __ldg(b.ext + i);   // no cells: left to the big-primitive pass
    const int ny = e.y, nz = e.z, c = (e.w & RECORD_MID) && mids ? 0 : e.x * ny * nz, sc = e.w & ~RECORD_MID;
    for (int q = lane; q < c; q += CELL_LANES) {
        const int qz = q % nz, qy = q / nz % ny, qx = q / nz / ny;
        f(b, edge, gkey(g, sc, (long long)a.x + qx, (long long)a.y + qy, (long long)a.z + qz), i);
    }
}

// the occupied cells and their entry counts (a full table is impossible at load <= 1/2)
__global__ void __launch_bounds__(256) k_grid_insert(GridBuild gp, GridBuild ge, SceneGeo g, BroadCounters* __restrict__ n) {
    each_entry(gp, ge, g, n, [&](const GridBuild& b, bool, unsigned long long key, int) {
        unsigned long long h = mix64(key) & b.mask;
        for (unsigned long long q = 0; q <= b.mask; ++q) {
            const unsigned long long prev = atomicCAS(b.hk + h, HASH_EMPTY, key);
            if (prev == HASH_EMPTY || prev == key) {
                atomicAdd(b.cnt + h, 1);
                return;
            }
            h = (h + 1) & b.mask;
        }
    });
}

// a run of ids for every occupied cell: one atomicAdd per warp on the cursor
__global__ void __launch_bounds__(256) k_grid_runs(GridBuild gp, GridBuild ge, BroadCounters* __restrict__ n) {
    const unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool second = k > gp.mask;   // tables are multiples of 32 slots
    const GridBuild& b = second ? ge : gp;
    const unsigned long long h = second ? k - (gp.mask + 1) : k;
    const int c = h <= b.mask ? b.cnt[h] : 0;
    int sum = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    const int total = __shfl_sync(0xffffffffu, sum, 31);
    if (total == 0) return;
    int base = 0;
    if (lane == 31) base = atomicAdd(&n->cursor[second ? 1 : 0], total);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (c) b.run[h] = make_int2(base + sum - c, 0);
}

// the ids into their cells' runs; run.y counts up to the run's length
__global__ void __launch_bounds__(256) k_grid_fill(GridBuild gp, GridBuild ge, SceneGeo g, BroadCounters* __restrict__ n) {
    each_entry(gp, ge, g, n, [&](const GridBuild& b, bool, unsigned long long key, int i) {
        unsigned long long h = mix64(key) & b.mask;
        for (unsigned long long q = 0; q <= b.mask; ++q) {
            if (b.hk[h] == key) {
                const int k = b.run[h].x + atomicAdd(&b.run[h].y, 1);
                b.ids[k] = i;
                return;
            }
            h = (h + 1) & b.mask;
        }
    });
}

// ---------------------------------------------------------------- the queries' kernels
// Each query is one launch: block ranges for its grid passes and its big-primitive passes, which so run
// side by side.
struct QueryBlocks {
    int pt, ee, pt_big, ee_big;   // blocks of each pass, in this order
};
constexpr int WALK_CTAS = 8;   // per SM, of 128 threads: the walks are chains of dependent loads
__global__ void __launch_bounds__(128, WALK_CTAS) k_find(QueryBlocks nb, int nbt, const int* __restrict__ bp, int nbe, FindArgs a, QueryView qt,
                                                         QueryView qe, SceneGeo g, GridView gp, CandView cp, GridView ge, CandView ce,
                                                         BigArgs big, PairList P, RowSink sink) {
    int b = blockIdx.x;
    if (b < nb.ee) return find_ee(b, nbe, a, qe, g, ge, ce, P, sink);
    if ((b -= nb.ee) < nb.pt) return find_pt(b, nbt, bp, a, qt, g, gp, cp, P, sink);
    if ((b -= nb.pt) < nb.pt_big) return find_pt_big(b, big, a, g, cp, P, sink);
    find_ee_big(b - nb.pt_big, big, a, g, ce, P, sink);
}
__global__ void __launch_bounds__(128, WALK_CTAS) k_ccd(QueryBlocks nb, int nbt, const int* __restrict__ bp, int nbe, CcdArgs a, QueryView qt,
                                                        QueryView qe, SceneGeo g, GridView gp, CandView cp, GridView ge, CandView ce,
                                                        BigArgs big, PairList P, CcdList L) {
    int b = blockIdx.x;
    if (b < nb.ee) return ccd_ee(b, nbe, a, qe, g, ge, ce, P, L);
    if ((b -= nb.ee) < nb.pt) return ccd_pt(b, nbt, bp, a, qt, g, gp, cp, P, L);
    if ((b -= nb.pt) < nb.pt_big) return ccd_pt_big(b, big, a, g, cp, P, L);
    ccd_ee_big(b - nb.pt_big, big, a, g, ce, P, L);
}
__global__ void __launch_bounds__(128, WALK_CTAS) k_collision(QueryBlocks nb, int nbt, HitArgs a, QueryView qt, SceneGeo g, GridView ge, CandView ce,
                                                              BigArgs big, PairList P) {
    int b = blockIdx.x;
    if (b < nb.pt) return collision_grid(b, nbt, a, qt, g, ge, ce, P);
    if ((b -= nb.pt) < nb.pt_big) return collision_big(b, 0, big, a, g, ce, P);
    collision_big(b - nb.pt_big, 1, big, a, g, ce, P);
}

// ---------------------------------------------------------------- row canonicalisation
__device__ __forceinline__ int4 row_of(RowKey k) {
    const unsigned long long m = (1ull << 21) - 1;
    return make_int4((int)((k.hi >> 21) & m), (int)(k.hi & m), (int)(k.lo >> 21), (int)(k.lo & m));
}
__device__ __forceinline__ int list_of(RowKey k) { return (int)(k.hi >> 42); }

// Up to SORT_SMALL rows: sorted, made unique and written out by one CTA (bitonic in shared memory)
// right behind the queries, so that a call of a small scene needs one round trip to the host.  More
// rows go through a merge sort after that round trip (k_rows_write).  Near the line, two cubes with up to 1,900
// rows: 162 us a call against 173 through the merge sort; the CTA's stages double in number from 2,048 rows to
// 4,096, whose keys no longer fit the static shared memory.
constexpr int SORT_SMALL = 2048, SORT_THREADS = 1024;
__global__ void __launch_bounds__(SORT_THREADS) k_rows_small(const RowKey* __restrict__ in, BroadCounters* __restrict__ n, int4* __restrict__ out) {
    __shared__ RowKey k[SORT_SMALL];
    __shared__ int warp_sum[SORT_THREADS / 32], list_n[N_TYPES];
    const int total = n->emitted, t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (n->flags || total > SORT_SMALL) return;
    int size = 64;
    while (size < total) size <<= 1;
    for (int i = t; i < size; i += SORT_THREADS) k[i] = i < total ? in[i] : RowKey{~0ull, ~0ull};
    if (t < N_TYPES) list_n[t] = 0;
    __syncthreads();
    for (int len = 2; len <= size; len <<= 1)
        for (int step = len >> 1; step > 0; step >>= 1) {
            if (t < size / 2) {
                const int i = 2 * step * (t / step) + t % step, j = i + step;
                const RowKey a = k[i], b = k[j];
                if ((b < a) == ((i & len) == 0)) {
                    k[i] = b;
                    k[j] = a;
                }
            }
            __syncthreads();
        }
    // thread t: elements 2t and 2t + 1
    bool f[2] = {false, false};
    for (int q = 0; q < 2; ++q) {
        const int i = 2 * t + q;
        f[q] = i < total && (i == 0 || !(k[i] == k[i - 1]));
    }
    int sum = (int)f[0] + (int)f[1];
    const int mine = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    if (lane == 31) warp_sum[w] = sum;
    __syncthreads();
    int pos = sum - mine;
    for (int q = 0; q < w; ++q) pos += warp_sum[q];
    for (int q = 0; q < 2; ++q)
        if (f[q]) {
            const RowKey r = k[2 * t + q];
            out[pos++] = row_of(r);
            atomicAdd(&list_n[list_of(r)], 1);
        }
    __syncthreads();
    if (t < N_TYPES) n->rows[t] = list_n[t];
    if (t == 0) n->sorted = 1;
}
// the sorted, unique keys (their number in *nu) as rows, and the lists' counts
__global__ void __launch_bounds__(256) k_rows_write(const int* __restrict__ nu, const RowKey* __restrict__ in, BroadCounters* __restrict__ n,
                                                    int4* __restrict__ out) {
    __shared__ int list_n[N_TYPES];
    if (threadIdx.x < N_TYPES) list_n[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < *nu) {
        out[i] = row_of(in[i]);
        atomicAdd(&list_n[list_of(in[i])], 1);
    }
    __syncthreads();
    if (threadIdx.x < N_TYPES && list_n[threadIdx.x]) atomicAdd(&n->rows[threadIdx.x], list_n[threadIdx.x]);
}

// ---------------------------------------------------------------- host side
static inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

template <class F>
static int cub_call(fipc_ctx* c, F&& f) {
    size_t need = 0;
    if (f(nullptr, need) != cudaSuccess) return FIPC_ERR_CUDA;
    if (c->cub_tmp.ensure(need)) return FIPC_ERR_CUDA;
    size_t have = c->cub_tmp.bytes;
    if (f(c->cub_tmp.p, have) != cudaSuccess) return FIPC_ERR_CUDA;
    return FIPC_OK;
}

static SceneGeo geo(const fipc_ctx* c) {
    SceneGeo g;
    g.vscene = c->n_scenes > 1 ? c->v_scene : nullptr;
    g.inv_dx_s = c->s_hash_inv_dx;
    g.inv_dx = c->hash_inv_dx;
    return g;
}

// the queries that build grids
enum { Q_FIND = 0, Q_STEP = 1, Q_CHECK = 2 };
static unsigned long long table_size(unsigned long long entries) {
    unsigned long long size = 1024;
    while (size < 2ull * entries) size <<= 1;
    return size;
}
// for a call with this many entries: half as much again, so that a slowly growing contact does not repeat every call
static unsigned long long table_for(unsigned long long entries) { return table_size(entries < (1ull << 26) ? entries + entries / 2 : entries); }

// one call's view of the scene: grids, big primitives and counters
struct Broad {
    SceneGeo g;
    BigArgs big;
    GridBuild gp, ge;
    PairList pairs;
    QueryView qt, qe;
    BroadCounters* n;
    int query;
};

static GridView view(const GridBuild& b) { return GridView{b.hk, b.run, b.mask, b.ids}; }
static CandView cands(const GridBuild& b) { return CandView{b.cell, b.box}; }
static int big_blocks(const fipc_ctx* c, int partners, int ny) { return nblk(c->max_prims[partners], BIG_CHUNK) * ny; }

// The grids over the boundary points (mode_p < 0: none) and edges at positions x (+ direction p when
// moving), and the big primitives.  Tables start at two slots per primitive, twice over, and grow when a
// call reports that its entries need more.  Each query has a size of its own in the tables' memory: its moving boxes
// make a fast step's filter need up to hundreds of times the entries of the other queries, and clearing and scanning
// that many slots would cost every later call (find_constraints of 180 cubes 0.73 ms, 1.37 after such a filter).
constexpr long long PAIRS_MAX = 1ll << 24;
static int broad_prepare(fipc_ctx* c, const double* x, const double* p, int query, Broad* b, cudaStream_t s) {
    static const int modes_p[3] = {0, 2, -1}, modes_e[3] = {1, 3, 4};
    const int n = c->nBT + c->nBE, mode_p = modes_p[query], mode_e = modes_e[query], np = mode_p < 0 ? 0 : c->nBP;
    b->query = query;
    if (c->big_flags.ensure((size_t)n + 16) || c->big_list.ensure(4ll * n + 16) || c->broad.ensure(sizeof(BroadCounters))) return FIPC_ERR_CUDA;
    const unsigned long long slots_p = std::max(c->gp.use[query], table_size(2ull * np)), slots_e = std::max(c->ge.use[query], table_size(2ull * c->nBE));
    if (c->gp.ensure(slots_p, query) || c->ge.ensure(slots_e, query)) return FIPC_ERR_CUDA;
    if (c->gp.cell4.ensure(16ll * np + 16) || c->gp.ext4.ensure(16ll * np + 16) || c->gp.box4.ensure(32ll * np + 32) ||
        c->ge.cell4.ensure(16ll * c->nBE + 16) || c->ge.ext4.ensure(16ll * c->nBE + 16) || c->ge.box4.ensure(32ll * c->nBE + 32) ||
        c->query_cell.ensure(16ll * n + 16) || c->query_box.ensure(32ll * n + 32))
        return FIPC_ERR_CUDA;
    unsigned char* tri_size = c->big_flags.as<unsigned char>();
    b->n = c->broad.as<BroadCounters>();
    SceneGeo g = geo(c);
    auto build = [](Grid& gr, const int* prim, int np_, int mode, unsigned long long slots) {
        return GridBuild{prim, np_, mode, gr.cell4.as<int4>(), gr.ext4.as<int4>(), gr.box4.as<float4>(), gr.hkeys.as<unsigned long long>(), gr.counts.as<int>(),
                         gr.runs.as<int2>(), gr.ids.as<int>(), slots - 1};
    };
    b->gp = build(c->gp, c->bp, np, mode_p, slots_p);
    b->ge = build(c->ge, c->be, c->nBE, mode_e, slots_e);
    b->qt = QueryView{c->query_cell.as<int4>(), c->query_box.as<float4>(), b->n->mid_pairs};
    b->qe = QueryView{b->qt.cell + c->nBT, b->qt.box + 2ll * c->nBT, b->n->mid_pairs + 1};
    FIPC_CUDA(cudaMemsetAsync(b->n, 0, sizeof(BroadCounters), s));
    const long long work = (long long)n + np, slots = (long long)(slots_p + slots_e);
    const int grid = (int)std::max<long long>(nblk(work, 256), std::min<long long>(nblk(slots, 256), 8 * SMS));
    k_prepare<<<grid, 256, 0, s>>>(c->nBT, c->bt, c->nBE, c->be, b->gp, b->ge, x, p, c->dhat, g, b->qt, b->qe, c->prim_off,
                                   c->n_scenes, tri_size, tri_size + c->nBT, c->big_list.as<int>(), b->n);
    FIPC_LAUNCHED();
    b->g = g;
    // the pair lists, as long as the last calls needed
    long long want = std::min<long long>(std::max<long long>(65536ll + 2ll * n, c->pair_hint), PAIRS_MAX);
    if (c->list_limit >= 0) want = std::min<long long>(want, c->list_limit);
    if (c->pair_list.ensure(16 * want + 16)) return FIPC_ERR_CUDA;
    b->pairs = PairList{c->pair_list.as<int2>(), b->n->pairs, (int)want};
    const int entries = nblk((long long)CELL_LANES * (np + c->nBE), 256);
    if (entries > 0) {
        k_grid_insert<<<entries, 256, 0, s>>>(b->gp, b->ge, g, b->n);
        FIPC_LAUNCHED();
        k_grid_runs<<<nblk(slots, 256), 256, 0, s>>>(b->gp, b->ge, b->n);
        FIPC_LAUNCHED();
        k_grid_fill<<<entries, 256, 0, s>>>(b->gp, b->ge, g, b->n);
        FIPC_LAUNCHED();
    }
    b->big = BigArgs{c->bp, c->be, c->bt, c->prim_off, c->n_scenes, tri_size, tri_size + c->nBT, c->big_list.as<int>(), b->n, c->nBT, c->nBE,
                     c->n_scenes > 1 ? 128 : 32};
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// after the counters of a call have reached the host: FIPC_OK, an error, or RETRY with larger tables
constexpr int RETRY = -1;
static int broad_status(fipc_ctx* c, const Broad& b, const BroadCounters& h) {
    for (int k = 0; k < 2; ++k) {
        const bool out = h.mid_pairs[k] <= MID_PAIRS;
        c->broad_stats[k] = h.pairs[k];
        c->broad_stats[2 + k] = h.work[k];
        c->broad_stats[4 + k] = h.big[k] + (out ? h.mid[k] : 0);
        c->broad_stats[6 + k] = out ? 0 : h.mid[k];
        c->broad_stats[8 + k] = (k ? b.ge : b.gp).mask + 1;
    }
    c->pair_hint = std::max<long long>(c->pair_hint, std::min<long long>(2ll * std::max(h.pairs[0], h.pairs[1]), PAIRS_MAX));
    if (h.flags & FLAG_CELLS) return FIPC_ERR_CAPACITY;
    const unsigned long long entries[2] = {h.total[0], h.total[1] + (h.mid_pairs[1] <= MID_PAIRS ? 0 : h.mid_total)};
    Grid* grid[2] = {&c->gp, &c->ge};
    if (h.flags & FLAG_TABLE) {
        if (entries[0] > (1ull << 30) || entries[1] > (1ull << 30)) return FIPC_ERR_CAPACITY;
        for (int k = 0; k < 2; ++k)
            if (2 * entries[k] > grid[k]->use[b.query]) grid[k]->use[b.query] = table_for(entries[k]);
        return RETRY;
    }
    // by halves: a fast step is often followed by another
    for (int k = 0; k < 2; ++k)
        if (grid[k]->use[b.query] >= 4 * table_for(entries[k])) grid[k]->use[b.query] /= 2;
    return FIPC_OK;
}
static int broad_read(const Broad& b, BroadCounters* h, cudaStream_t s) {
    FIPC_CUDA(cudaMemcpyAsync(h, b.n, sizeof(BroadCounters), cudaMemcpyDeviceToHost, s));
    FIPC_CUDA(cudaStreamSynchronize(s));
    return FIPC_OK;
}

// sort and unique of the n emitted rows when they are too many for one CTA
static int rows_large(fipc_ctx* c, const Broad& b, int n, BroadCounters* h, cudaStream_t s) {
    RowKey* k = c->rows.keys.as<RowKey>();
    RowKey* u = c->rows.keys_alt.as<RowKey>();
    int* nu = &b.n->sorted;
    int st = cub_call(c, [&](void* t, size_t& bytes) { return cub::DeviceMergeSort::SortKeys(t, bytes, k, n, RowLess(), s); });
    if (st) return st;
    st = cub_call(c, [&](void* t, size_t& bytes) { return cub::DeviceSelect::Unique(t, bytes, k, u, nu, n, s); });
    if (st) return st;
    k_rows_write<<<nblk(n, 256), 256, 0, s>>>(nu, u, b.n, c->rows.all.as<int4>());
    FIPC_LAUNCHED();
    return broad_read(b, h, s);
}

// find_constraints (NEWTON_IPC.py:337-357) into c->rows.all / c->h_counts
int find_constraints(fipc_ctx* c, const double* x, cudaStream_t s) {
    for (int attempt = 0; attempt < 12; ++attempt) {
        Broad b;
        int st = broad_prepare(c, x, nullptr, Q_FIND, &b, s);
        if (st) return st;
        const RowSink sink{c->rows.keys.as<RowKey>(), b.n, c->rows.cap};
        QueryBlocks nb{c->nBP > 0 ? nblk((long long)QG * c->nBT, 128) : 0, nblk((long long)QG * c->nBE, 128), 0, 0};
        nb.pt_big = c->nBT > 0 && c->nBP > 0 ? big_blocks(c, 0, b.big.ny) : 0;
        nb.ee_big = c->nBE > 1 ? big_blocks(c, 1, b.big.ny) : 0;
        const int blocks = nb.pt + nb.ee + nb.pt_big + nb.ee_big;
        if (blocks > 0) {
            const FindArgs a{c->bt, c->be, x, c->x0, c->dhat, c->dhat2};
            k_find<<<blocks, 128, 0, s>>>(nb, c->nBT, c->bp, c->nBE, a, b.qt, b.qe, b.g, view(b.gp), cands(b.gp), view(b.ge), cands(b.ge), b.big, b.pairs,
                                          sink);
            FIPC_LAUNCHED();
            k_find_pairs<<<PAIR_BLOCKS, PAIR_THREADS, 0, s>>>(a, b.pairs, sink);
            FIPC_LAUNCHED();
        }
        k_rows_small<<<1, SORT_THREADS, 0, s>>>(sink.rows, b.n, c->rows.all.as<int4>());
        FIPC_LAUNCHED();
        BroadCounters h;
        st = broad_read(b, &h, s);
        if (st) return st;
        st = broad_status(c, b, h);
        if (st == RETRY) continue;
        if (st) return st;
        if (h.flags & FLAG_ROWS) {
            if (h.emitted > (1 << 29)) return FIPC_ERR_CAPACITY;
            for (int t = 0; t < N_TYPES; ++t) c->h_counts[t] = 0;   // the former lists' rows go with their buffer
            if (c->rows.ensure(2 * h.emitted)) return FIPC_ERR_CUDA;
            continue;
        }
        if (!h.sorted) {
            st = rows_large(c, b, h.emitted, &h, s);
            if (st) return st;
        }
        int off = 0;
        for (int t = 0; t < N_TYPES; ++t) {
            c->h_counts[t] = h.rows[t];
            c->h_row0[t] = off;
            off += h.rows[t];
        }
        return FIPC_OK;
    }
    return FIPC_ERR_CAPACITY;
}

// compute_intersection_free_step_size (NEWTON_IPC.py:456-468): the launches, min'd into slots (one
// double per scene, preset to 1.0 by the caller; null: the call's own)
static int ccd_launch(fipc_ctx* c, const double* x, const double* p, double eta, bool inversion, unsigned long long* slot, Broad* b,
                      cudaStream_t s) {
    int st = broad_prepare(c, x, p, Q_STEP, b, s);
    if (st) return st;
    if (!slot) slot = &b->n->alpha;
    long long cap = std::min<long long>(65536ll + c->nBE + c->nBT, 1ll << 21);
    if (c->list_limit >= 0) cap = std::min<long long>(cap, c->list_limit);
    if (c->ccd_work.ensure(4 * cap * sizeof(CcdWork) + sizeof(CcdWork))) return FIPC_ERR_CUDA;
    const CcdList L{c->ccd_work.as<CcdWork>(), b->n->work, (int)cap}, M{L.w + 2 * cap, b->n->doubt, (int)cap};
    QueryBlocks nb{c->nBP > 0 ? nblk((long long)QG * c->nBT, 128) : 0, nblk((long long)QG * c->nBE, 128), 0, 0};
    nb.pt_big = c->nBT > 0 && c->nBP > 0 ? big_blocks(c, 0, b->big.ny) : 0;
    nb.ee_big = c->nBE > 1 ? big_blocks(c, 1, b->big.ny) : 0;
    if (inversion && c->nT > 0) {
        k_ccd_inversion<<<nblk(c->nT, 128), 128, 0, s>>>(c->nT, (const int4*)c->tets, x, p, eta, b->g, slot);
        FIPC_LAUNCHED();
    }
    const int blocks = nb.pt + nb.ee + nb.pt_big + nb.ee_big;
    if (blocks > 0) {
        const CcdArgs a{c->bt, c->be, x, p, c->dhat, eta, b->g.vscene, slot};
        k_ccd<<<blocks, 128, 0, s>>>(nb, c->nBT, c->bp, c->nBE, a, b->qt, b->qe, b->g, view(b->gp), cands(b->gp), view(b->ge), cands(b->ge), b->big, b->pairs, L);
        FIPC_LAUNCHED();
        k_ccd_pairs<<<PAIR_BLOCKS, PAIR_THREADS, 0, s>>>(a, b->pairs, L);
        FIPC_LAUNCHED();
        k_ccd_signs<<<PAIR_BLOCKS, PAIR_THREADS, 0, s>>>(a, L, M);
        FIPC_LAUNCHED();
        k_ccd_exact<<<PAIR_BLOCKS, PAIR_THREADS, 0, s>>>(a, M);
        FIPC_LAUNCHED();
    }
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// one scene (slots null): the step in *alpha_h; a batch: the steps in slots
int ccd_step(fipc_ctx* c, const double* x, const double* p, double eta, bool inversion, double* alpha_h, unsigned long long* slots,
             cudaStream_t s) {
    for (int attempt = 0; attempt < 4; ++attempt) {
        Broad b;
        int st = ccd_launch(c, x, p, eta, inversion, slots, &b, s);
        if (st) return st;
        BroadCounters h;
        st = broad_read(b, &h, s);
        if (st) return st;
        st = broad_status(c, b, h);
        if (st == RETRY) continue;   // the minimum so far stays valid
        if (st) return st;
        if (alpha_h) memcpy(alpha_h, &h.alpha, 8);
        return FIPC_OK;
    }
    return FIPC_ERR_CAPACITY;
}

// check_collision_3d (NEWTON_IPC.py:881-886): one scene (hits null): the flag in *hit_h; a batch: or'd
// into hits (one int per scene, zeroed by the caller)
int check_collision(fipc_ctx* c, const double* x, int* hit_h, int* hits, cudaStream_t s) {
    for (int attempt = 0; attempt < 4; ++attempt) {
        Broad b;
        int st = broad_prepare(c, x, nullptr, Q_CHECK, &b, s);
        if (st) return st;
        int* hit = hits ? hits : &b.n->hit;
        QueryBlocks nb{c->nBE > 0 ? nblk((long long)QG * c->nBT, 128) : 0, 0, 0, 0};
        if (c->nBT > 0 && c->nBE > 0) {
            nb.pt_big = big_blocks(c, 1, b.big.ny);
            nb.ee_big = big_blocks(c, 2, b.big.ny);
        }
        const int blocks = nb.pt + nb.pt_big + nb.ee_big;
        if (blocks > 0) {
            const HitArgs a{c->bt, c->be, x, b.g.vscene, hit};
            k_collision<<<blocks, 128, 0, s>>>(nb, c->nBT, a, b.qt, b.g, view(b.ge), cands(b.ge), b.big, b.pairs);
            FIPC_LAUNCHED();
            k_collision_pairs<<<PAIR_BLOCKS, PAIR_THREADS, 0, s>>>(a, b.pairs);
            FIPC_LAUNCHED();
        }
        FIPC_CUDA(cudaGetLastError());
        BroadCounters h;
        st = broad_read(b, &h, s);
        if (st) return st;
        st = broad_status(c, b, h);
        if (st == RETRY) continue;
        if (st) return st;
        if (hit_h) *hit_h = h.hit;
        return FIPC_OK;
    }
    return FIPC_ERR_CAPACITY;
}

}  // namespace fipc
