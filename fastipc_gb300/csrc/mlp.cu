// Per-vertex MLP of the learned Newton warm start: forward, backward, MSE loss, Adam, FP32.
//
// Network: 55 inputs (padded to 64) -> 128 -> 128 -> 128 -> 3 (padded to 4), GELU after each
// hidden layer.  Rows are vertices; parameters are one flat FP32 array:
//   W1 [128][64], b1 [128], W2 [128][128], b2 [128], W3 [128][128], b3 [128], W4 [4][128], b4 [4].
// The forward pass is one kernel over tiles of rows; the backward pass alternates data-gradient
// tiles and weight-gradient chunks of rows.  FP32 FMAs throughout; every output element sums its K
// range in a fixed order, so forward and backward results are reproducible.  No counterpart in the reference: this is the
// learned warm start the task adds beside the drop-in path.
#include <cuda_runtime.h>

#include <initializer_list>

#include "ctx.cuh"

namespace fipc {

constexpr int MLP_IN = 64, MLP_H = 128, MLP_OUT = 4;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + MLP_H * MLP_IN, OFF_W2 = OFF_B1 + MLP_H, OFF_B2 = OFF_W2 + MLP_H * MLP_H,
              OFF_W3 = OFF_B2 + MLP_H, OFF_B3 = OFF_W3 + MLP_H * MLP_H, OFF_W4 = OFF_B3 + MLP_H,
              OFF_B4 = OFF_W4 + MLP_OUT * MLP_H, MLP_NPARAM = OFF_B4 + MLP_OUT;

// ---------------------------------------------------------------- tiles
// A CTA holds a tile of R rows in shared memory, k-major (Hs[k][row]), and multiplies it with a
// 128-column weight matrix whose K slices of 16 pass through a double buffer Ws.  Thread (tx, ty)
// of 16 x 16 owns R/16 consecutive rows and the columns 4 tx .. 4 tx + 3 and 64 + 4 tx ..; per k
// it loads its rows and two float4 of weights for (R/16) x 8 FMAs, two rows' in one instruction.  The
// FP32 FMA pipe binds (51% busy; the rest is waits of 4 warps per scheduler on it, on shared memory and on
// the slices' barriers): at R = 128 a k step is 32 paired FMAs per thread against 4 shared-memory loads.
// Slices of 32 hold 8 more registers in flight and spill; R = 64 and 256 are slower at 176,841 rows (0.51, 0.53
// ms against 0.45).  Rows are swizzled by the
// column group (row ^ 4 ((k / 4) % 8)) so that the transposed store of a layer's output, which
// strides by columns, meets distinct banks while the row loads stay aligned.  Every output sums
// its K range in ascending order in one FMA chain.
// R = 128 needs n >= 2 x 152 such tiles to fill the GPU; below that R = 64, then 32, keep more SMs
// busy.  Measured on a GB300, forward pass: 176,841 rows 1.19 ms as separate 64 x 64 products with
// bias and activation passes, 0.45 ms here; a training step of 8,192 rows 5.3 ms, of
// which 97% were products (the weight gradients, 128 x 128 outputs over all rows, ran on 2 to 4
// CTAs), 0.17 ms here.
constexpr int MLP_THREADS = 256, KS = 16, WLD = MLP_H + 4;

// four consecutive floats of global memory: one 16-byte access when every array of the call is
// 16-byte aligned (al), else four (callers may pass any float address)
__device__ __forceinline__ float4 ld4(const float* p, bool al) {
    return al ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
__device__ __forceinline__ void st4(float* p, float4 v, bool al) {
    if (al) {
        *reinterpret_cast<float4*>(p) = v;
    } else {
        p[0] = v.x;
        p[1] = v.y;
        p[2] = v.z;
        p[3] = v.w;
    }
}

template <int R>
__device__ __forceinline__ int hs_at(int k, int row) {
    return k * R + (row ^ (((k >> 2) & 7) << 2));
}

// rows [r0, r0 + R) of src [n][K] into Hs, zeros past n; a lane takes one row's float4 at a time
template <int R>
__device__ __forceinline__ void load_rows(float* Hs, const float* __restrict__ src, int K, int r0, int n, bool al) {
    for (int e = threadIdx.x; e < R * (K / 4); e += MLP_THREADS) {
        const int row = e % R, k = 4 * (e / R);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + row < n) v = ld4(src + (size_t)(r0 + row) * K + k, al);
        Hs[hs_at<R>(k, row)] = v.x;
        Hs[hs_at<R>(k + 1, row)] = v.y;
        Hs[hs_at<R>(k + 2, row)] = v.z;
        Hs[hs_at<R>(k + 3, row)] = v.w;
    }
}

// one K slice of the weights, held in registers between its load and its store to shared memory:
// T (transposed): W [128][K], slice[kk][c] = W[c][k0 + kk];  else W [K][128], slice[kk][c] = W[k0 + kk][c]
template <bool T>
__device__ __forceinline__ void fetch_slice(float4 (&w)[2], const float* __restrict__ W, int K, int k0, bool al) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int e = threadIdx.x + q * MLP_THREADS;
        if (T) w[q] = ld4(W + (size_t)(e % MLP_H) * K + k0 + 4 * (e / MLP_H), al);
        else w[q] = ld4(W + (size_t)(k0 + e / 32) * MLP_H + 4 * (e % 32), al);
    }
}
template <bool T>
__device__ __forceinline__ void store_slice(float* Ws, const float4 (&w)[2]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int e = threadIdx.x + q * MLP_THREADS;
        if (T) {
            float* p = Ws + 4 * (e / MLP_H) * WLD + e % MLP_H;
            p[0] = w[q].x;
            p[WLD] = w[q].y;
            p[2 * WLD] = w[q].z;
            p[3 * WLD] = w[q].w;
        } else {
            *reinterpret_cast<float4*>(Ws + (e / 32) * WLD + 4 * (e % 32)) = w[q];
        }
    }
}

// two FP32 FMAs in one instruction (each rounded as fmaf): the FMA pipe takes them in two cycles, so a k
// step's other instructions issue beside it instead of before it
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// acc[i][j] = sum_k Hs[k][row i] W(k, col j) for the thread's rows and columns; Hs complete on entry
template <int R, bool T>
__device__ __forceinline__ void tile_product(float (&acc)[R / 16][8], const float* Hs, float* Ws, const float* __restrict__ W, int K,
                                             bool al) {
    constexpr int TR = R / 16;
    const int tx = threadIdx.x % 16, row0 = (threadIdx.x / 16) * TR;
    f32x2 sum[TR / 2][8];   // pairs of rows
#pragma unroll
    for (int i = 0; i < TR / 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[i][j] = 0;
    float4 w[2];
    fetch_slice<T>(w, W, K, 0, al);
    store_slice<T>(Ws, w);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < K; k0 += KS, buf ^= 1) {
        const bool more = k0 + KS < K;
        if (more) fetch_slice<T>(w, W, K, k0 + KS, al);
        const float* Wb = Ws + buf * KS * WLD + 4 * tx;
#pragma unroll 8
        for (int kk = 0; kk < KS; ++kk) {
            const float* h = Hs + (k0 + kk) * R;
            const int s = (((k0 + kk) >> 2) & 7) << 2;
            float a[TR];
            if (TR == 2) {
                const float2 v = *reinterpret_cast<const float2*>(h + (row0 ^ s));
                a[0] = v.x;
                a[TR - 1] = v.y;
            } else {
#pragma unroll
                for (int i = 0; i + 3 < TR; i += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(h + ((row0 + i) ^ s));
                    a[i] = v.x;
                    a[i + 1] = v.y;
                    a[i + 2] = v.z;
                    a[i + 3] = v.w;
                }
            }
            const float4 b0 = *reinterpret_cast<const float4*>(Wb + kk * WLD), b1 = *reinterpret_cast<const float4*>(Wb + kk * WLD + 64);
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const f32x2 bb = pack2(b[j], b[j]);
#pragma unroll
                for (int i = 0; i < TR / 2; ++i) sum[i][j] = fma2(pack2(a[2 * i], a[2 * i + 1]), bb, sum[i][j]);
            }
        }
        if (more) store_slice<T>(Ws + (buf ^ 1) * KS * WLD, w);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TR / 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) unpack2(sum[i][j], acc[2 * i][j], acc[2 * i + 1][j]);
}
__device__ __forceinline__ int tile_col(int j) { return 4 * (threadIdx.x % 16) + (j & 3) + 64 * (j >> 2); }

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

template <int R>
constexpr int tile_smem() {
    return 4 * (MLP_H * R + 2 * KS * WLD);
}

// the whole forward pass of R rows in one CTA: the activations stay in shared memory from layer to
// layer (overwritten in place once a layer's sums are in registers); Z and A are written for the
// backward pass.  One launch instead of eight.
template <int R>
__global__ void __launch_bounds__(MLP_THREADS, 2) k_mlp_forward(int n, const float* __restrict__ X, const float* __restrict__ P,
                                                                float* __restrict__ Z, float* __restrict__ A, float* __restrict__ out, bool al) {
    extern __shared__ float4 smem4[];
    float* Hs = reinterpret_cast<float*>(smem4);
    float* Ws = Hs + MLP_H * R;
    constexpr int TR = R / 16;
    const int r0 = blockIdx.x * R, row0 = (threadIdx.x / 16) * TR;
    load_rows<R>(Hs, X, MLP_IN, r0, n, al);
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
        const int K = l == 0 ? MLP_IN : MLP_H;
        const float* W = P + (l == 0 ? OFF_W1 : (l == 1 ? OFF_W2 : OFF_W3));
        const float* bias = P + (l == 0 ? OFF_B1 : (l == 1 ? OFF_B2 : OFF_B3));
        float acc[TR][8];
        tile_product<R, true>(acc, Hs, Ws, W, K, al);
        float* Zl = Z + (size_t)l * n * MLP_H;
        float* Al = A + (size_t)l * n * MLP_H;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 bb = ld4(bias + tile_col(4 * h), al);
            const float bv[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
            for (int i = 0; i < TR; ++i) {
                float z[4], a[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    z[j] = acc[i][4 * h + j] + bv[j];
                    a[j] = gelu(z[j]);
                    acc[i][4 * h + j] = a[j];
                }
                const int r = r0 + row0 + i;
                if (r < n) {
                    const size_t o = (size_t)r * MLP_H + tile_col(4 * h);
                    st4(Zl + o, make_float4(z[0], z[1], z[2], z[3]), al);
                    st4(Al + o, make_float4(a[0], a[1], a[2], a[3]), al);
                }
            }
        }
        // tile_product ended with a barrier: every thread is done with the old activations
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (TR == 2) {
                *reinterpret_cast<float2*>(Hs + hs_at<R>(tile_col(j), row0)) = make_float2(acc[0][j], acc[TR - 1][j]);
            } else {
#pragma unroll
                for (int i = 0; i + 3 < TR; i += 4)
                    *reinterpret_cast<float4*>(Hs + hs_at<R>(tile_col(j), row0 + i)) = make_float4(acc[i][j], acc[i + 1][j], acc[i + 2][j], acc[i + 3][j]);
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < R * MLP_OUT; e += MLP_THREADS) {
        const int row = e % R, o = e / R;
        const float* w = P + OFF_W4 + o * MLP_H;
        float s = 0.f;
#pragma unroll 8
        for (int k = 0; k < MLP_H; ++k) s = fmaf(Hs[hs_at<R>(k, row)], __ldg(w + k), s);
        if (r0 + row < n) out[(size_t)(r0 + row) * MLP_OUT + o] = s + __ldg(P + OFF_B4 + o);
    }
}

// gradient of a layer's input: din = (d W) gelu'(Z), d [n][128], W [128][128]
template <int R>
__global__ void __launch_bounds__(MLP_THREADS, 2) k_mlp_data_grad(int n, const float* __restrict__ d, const float* __restrict__ W,
                                                                  const float* __restrict__ Z, float* __restrict__ din, bool al) {
    extern __shared__ float4 smem4[];
    float* Hs = reinterpret_cast<float*>(smem4);
    float* Ws = Hs + MLP_H * R;
    constexpr int TR = R / 16;
    const int r0 = blockIdx.x * R, row0 = (threadIdx.x / 16) * TR;
    load_rows<R>(Hs, d, MLP_H, r0, n, al);
    __syncthreads();
    float acc[TR][8];
    tile_product<R, false>(acc, Hs, Ws, W, MLP_H, al);
#pragma unroll
    for (int i = 0; i < TR; ++i) {
        const int r = r0 + row0 + i;
        if (r >= n) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const size_t o = (size_t)r * MLP_H + tile_col(4 * h);
            const float4 z = ld4(Z + o, al);
            st4(din + o, make_float4(acc[i][4 * h] * gelu_grad(z.x), acc[i][4 * h + 1] * gelu_grad(z.y),
                                     acc[i][4 * h + 2] * gelu_grad(z.z), acc[i][4 * h + 3] * gelu_grad(z.w)), al);
        }
    }
}

// the last layer's backward over one chunk of rows: d3 = (dout W4) gelu'(Z3) for its rows, and the
// chunk's sums of dout^T A3 [4][128] and of dout [4] into part (MLP_LAST floats per chunk).  Thread
// (c, h): column c, rows of parity h; the two halves are added at the end, rows in ascending order.
constexpr int MLP_LAST = MLP_OUT * MLP_H + MLP_OUT;
__global__ void __launch_bounds__(MLP_THREADS) k_mlp_last_grad(int n, int chunk, const float* __restrict__ dout,
                                                               const float* __restrict__ W4, const float* __restrict__ A3,
                                                               const float* __restrict__ Z3, float* __restrict__ d3,
                                                               float* __restrict__ part, bool al) {
    __shared__ float sh[MLP_OUT + 1][MLP_H];
    const int c = threadIdx.x % MLP_H, h = threadIdx.x / MLP_H;
    const int r0 = blockIdx.x * chunk, r1 = min(n, r0 + chunk);
    float w[MLP_OUT], g[MLP_OUT] = {}, b = 0.f;
#pragma unroll
    for (int o = 0; o < MLP_OUT; ++o) w[o] = __ldg(W4 + o * MLP_H + c);
#pragma unroll 4
    for (int r = r0 + h; r < r1; r += 2) {
        const float4 q = ld4(dout + (size_t)r * MLP_OUT, al);
        const float a = __ldg(A3 + (size_t)r * MLP_H + c), z = __ldg(Z3 + (size_t)r * MLP_H + c);
        g[0] = fmaf(q.x, a, g[0]);
        g[1] = fmaf(q.y, a, g[1]);
        g[2] = fmaf(q.z, a, g[2]);
        g[3] = fmaf(q.w, a, g[3]);
        if (c < MLP_OUT) b += c == 0 ? q.x : (c == 1 ? q.y : (c == 2 ? q.z : q.w));
        const float d = fmaf(q.w, w[3], fmaf(q.z, w[2], fmaf(q.y, w[1], q.x * w[0])));
        d3[(size_t)r * MLP_H + c] = d * gelu_grad(z);
    }
    if (h == 1) {
#pragma unroll
        for (int o = 0; o < MLP_OUT; ++o) sh[o][c] = g[o];
        sh[MLP_OUT][c] = b;
    }
    __syncthreads();
    if (h == 1) return;
    float* p = part + (size_t)blockIdx.x * MLP_LAST;
#pragma unroll
    for (int o = 0; o < MLP_OUT; ++o) p[o * MLP_H + c] = g[o] + sh[o][c];
    if (c < MLP_OUT) p[MLP_OUT * MLP_H + c] = b + sh[MLP_OUT][c];
}

// weight gradient of a layer over one chunk of rows: part [128][DIN] = sum_r d[r]^T in[r] and the
// bias gradient sum_r d[r] behind it (128 DIN + 128 floats per chunk).  The rows are the product's
// K range, so both operands load into shared memory as they lie.  blockIdx.y takes 64 of the 128
// output rows.
template <int DIN>
__global__ void __launch_bounds__(MLP_THREADS) k_mlp_weight_grad(int n, int chunk, const float* __restrict__ d,
                                                                 const float* __restrict__ in, float* __restrict__ part, bool al) {
    constexpr int KT = 16, TC = DIN / 16;
    __shared__ __align__(16) float Ds[2][KT][64], Is[2][KT][DIN];
    const int r0 = blockIdx.x * chunk, r1 = min(n, r0 + chunk), m0 = 64 * blockIdx.y;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][TC] = {}, bsum[4] = {};
    float4 dv, iv[DIN / 64];
    auto fetch = [&](int r) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        {
            const int q = r + threadIdx.x / 16;
            dv = q < r1 ? ld4(d + (size_t)q * MLP_H + m0 + 4 * (threadIdx.x % 16), al) : zero;
        }
#pragma unroll
        for (int k = 0; k < DIN / 64; ++k) {
            const int e = threadIdx.x + k * MLP_THREADS, q = r + e / (DIN / 4);
            iv[k] = q < r1 ? ld4(in + (size_t)q * DIN + 4 * (e % (DIN / 4)), al) : zero;
        }
    };
    auto store = [&](int b) {
        *reinterpret_cast<float4*>(&Ds[b][threadIdx.x / 16][4 * (threadIdx.x % 16)]) = dv;
#pragma unroll
        for (int k = 0; k < DIN / 64; ++k) {
            const int e = threadIdx.x + k * MLP_THREADS;
            *reinterpret_cast<float4*>(&Is[b][e / (DIN / 4)][4 * (e % (DIN / 4))]) = iv[k];
        }
    };
    fetch(r0);
    store(0);
    __syncthreads();
    for (int r = r0, buf = 0; r < r1; r += KT, buf ^= 1) {
        const bool more = r + KT < r1;
        if (more) fetch(r + KT);
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const float4 a4 = *reinterpret_cast<const float4*>(&Ds[buf][k][4 * ty]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w};
            float b[TC];
#pragma unroll
            for (int j = 0; j < TC; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&Is[buf][k][4 * tx + 16 * j]);
                b[j] = v.x;
                b[j + 1] = v.y;
                b[j + 2] = v.z;
                b[j + 3] = v.w;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bsum[i] += a[i];
#pragma unroll
                for (int j = 0; j < TC; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
        }
        if (more) store(buf ^ 1);
        __syncthreads();
    }
    float* p = part + (size_t)blockIdx.x * (MLP_H * DIN + MLP_H);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + 4 * ty + i;
#pragma unroll
        for (int j = 0; j < TC; j += 4)
            st4(p + (size_t)m * DIN + 4 * tx + 16 * j, make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]), al);
        if (tx == 0) p[MLP_H * DIN + m] = bsum[i];
    }
}

// g[e] = sum of part[q][e] over the chunks, chunks in ascending order
__global__ void k_mlp_sum_chunks(int nchunk, int size, const float* __restrict__ part, float* __restrict__ g) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= size) return;
    float s = 0.f;
#pragma unroll 8
    for (int q = 0; q < nchunk; ++q) s += __ldg(part + (size_t)q * size + e);
    g[e] = s;
}

// mean squared error over the first 3 outputs: dout = 2 (out - target) / (3 n), loss partials
__global__ void k_mse(int n, const float* __restrict__ out, const float* __restrict__ target, float* __restrict__ dout,
                      float* __restrict__ part) {
    __shared__ float sh[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.f;
    if (i < n) {
        const float s = 2.f / (3.f * (float)n);
        for (int d = 0; d < MLP_OUT; ++d) {
            const float e = d < 3 ? out[4 * (size_t)i + d] - target[4 * (size_t)i + d] : 0.f;
            dout[4 * (size_t)i + d] = s * e;
            l += e * e;
        }
    }
    sh[threadIdx.x] = l;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}
__global__ void k_mse_finish(int nb, int n, const float* __restrict__ part, float* __restrict__ loss) {
    __shared__ float sh[256];
    float a = 0.f;
    for (int i = threadIdx.x; i < nb; i += 256) a += part[i];
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = sh[0] / (3.f * (float)n);
}

// Adam with bias correction (step t >= 1)
__global__ void k_adam(int n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace fipc

// ---------------------------------------------------------------- host side
namespace fipc {
static inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// rows per tile: the largest that still gives every SM two CTAs (R = 128) or most SMs one (R = 64)
static int tile_rows(int n) { return n >= 128 * 2 * SMS ? 128 : (n >= 64 * 96 ? 64 : 32); }

template <int R>
static int launch_forward(int n, const float* X, const float* P, float* Z, float* A, float* out, bool al, cudaStream_t s) {
    FIPC_CUDA(cudaFuncSetAttribute(k_mlp_forward<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem<R>()));
    k_mlp_forward<R><<<nblk(n, R), MLP_THREADS, tile_smem<R>(), s>>>(n, X, P, Z, A, out, al);
    FIPC_LAUNCHED();
    return FIPC_OK;
}
template <int R>
static int launch_data_grad(int n, const float* d, const float* W, const float* Z, float* din, bool al, cudaStream_t s) {
    FIPC_CUDA(cudaFuncSetAttribute(k_mlp_data_grad<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem<R>()));
    k_mlp_data_grad<R><<<nblk(n, R), MLP_THREADS, tile_smem<R>(), s>>>(n, d, W, Z, din, al);
    FIPC_LAUNCHED();
    return FIPC_OK;
}

static bool aligned16(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

// weight and bias gradient of one layer.  The chunks' partial sums go to scratch (n x 128 floats,
// free at that time): a chunk takes at least 192 rows and at most 128 x 129 floats, so they fit; at
// most 152 chunks (two CTAs each).  One chunk writes the gradients directly.
template <int DIN>
static void weight_grad(int n, const float* d, const float* in, float* scratch, float* G, bool al, cudaStream_t s) {
    constexpr int size = MLP_H * DIN + MLP_H;
    int nc = n / 192;
    nc = nc < 1 ? 1 : (nc > SMS ? SMS : nc);
    const int chunk = (n + nc - 1) / nc;
    nc = nblk(n, chunk);
    k_mlp_weight_grad<DIN><<<dim3(nc, 2), MLP_THREADS, 0, s>>>(n, chunk, d, in, nc > 1 ? scratch : G, al);
    FIPC_LAUNCHED();
    if (nc > 1) {
        k_mlp_sum_chunks<<<nblk(size, 128), 128, 0, s>>>(nc, size, scratch, G);
        FIPC_LAUNCHED();
    }
}
}  // namespace fipc

using namespace fipc;

extern "C" {

int fipc_mlp_param_count(void) { return MLP_NPARAM; }

// out [n][4] for inputs X [n][64]; Z and A: scratch [3][n][128] (pre- and post-activations,
// kept for the backward pass)
int fipc_mlp_forward(int n, const float* X, const float* params, float* Z, float* A, float* out, void* stream) {
    if (n < 0 || !X || !params || !Z || !A || !out) return FIPC_ERR_ARGUMENT;
    if (n == 0) return FIPC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int R = tile_rows(n);
    const bool al = aligned16({X, params, Z, A, out});
    const int st = R == 128 ? launch_forward<128>(n, X, params, Z, A, out, al, s)
                            : (R == 64 ? launch_forward<64>(n, X, params, Z, A, out, al, s) : launch_forward<32>(n, X, params, Z, A, out, al, s));
    if (st) return st;
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// parameter gradients (grads, same layout as params) of sum(dout . out) for the forward pass
// that produced Z, A; dA: scratch [2][n][128].  One half of dA holds the current layer's output
// gradient, the other its weight gradient's partial sums until the next layer's gradient overwrites it.
int fipc_mlp_backward(int n, const float* X, const float* params, const float* Z, const float* A, const float* dout, float* grads,
                      float* dA, void* stream) {
    if (n <= 0 || !X || !params || !Z || !A || !dout || !grads || !dA) return FIPC_ERR_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t L = (size_t)n * MLP_H;
    const float* P = params;
    float* G = grads;
    float *d0 = dA, *d1 = dA + L;
    const bool al = aligned16({X, params, Z, A, dout, grads, dA});
    {   // layer 4 (linear): at least 64 rows a chunk (MLP_LAST / 64 < 8.1 floats a row)
        const int chunk = n > 64 * 2 * SMS ? nblk(n, 2 * SMS) : 64, nc = nblk(n, chunk);
        float* part = nc > 1 ? d1 : G + OFF_W4;
        k_mlp_last_grad<<<nc, MLP_THREADS, 0, s>>>(n, chunk, dout, P + OFF_W4, A + 2 * L, Z + 2 * L, d0, part, al);
        FIPC_LAUNCHED();
        if (nc > 1) {
            k_mlp_sum_chunks<<<nblk(MLP_LAST, 32), 32, 0, s>>>(nc, MLP_LAST, part, G + OFF_W4);
            FIPC_LAUNCHED();
        }
    }
    const int R = tile_rows(n);
    for (int l = 2; l >= 0; --l) {   // layers 3, 2, 1
        const int offW = l == 2 ? OFF_W3 : (l == 1 ? OFF_W2 : OFF_W1);
        if (l > 0) weight_grad<MLP_H>(n, d0, A + (l - 1) * L, d1, G + offW, al, s);
        else weight_grad<MLP_IN>(n, d0, X, d1, G + offW, al, s);
        if (l > 0) {
            const float* Zl = Z + (l - 1) * L;
            const int st = R == 128 ? launch_data_grad<128>(n, d0, P + offW, Zl, d1, al, s)
                                    : (R == 64 ? launch_data_grad<64>(n, d0, P + offW, Zl, d1, al, s) : launch_data_grad<32>(n, d0, P + offW, Zl, d1, al, s));
            if (st) return st;
            float* t = d0;
            d0 = d1;
            d1 = t;
        }
    }
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// loss = mean over n rows and 3 outputs of (out - target)^2 into *loss (device); dout its gradient;
// part: scratch of ceil(n / 256) floats
int fipc_mlp_mse(int n, const float* out, const float* target, float* dout, float* part, float* loss, void* stream) {
    if (n <= 0 || !out || !target || !dout || !part || !loss) return FIPC_ERR_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = nblk(n, 256);
    k_mse<<<nb, 256, 0, s>>>(n, out, target, dout, part);
    FIPC_LAUNCHED();
    k_mse_finish<<<1, 256, 0, s>>>(nb, n, part, loss);
    FIPC_LAUNCHED();
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// one Adam step (t counts from 1)
int fipc_mlp_adam(int n_params, float* params, const float* grads, float* m, float* v, float lr, float beta1, float beta2, float eps,
                  int t, void* stream) {
    if (n_params <= 0 || !params || !grads || !m || !v || t < 1) return FIPC_ERR_ARGUMENT;
    const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
    k_adam<<<nblk(n_params, 256), 256, 0, (cudaStream_t)stream>>>(n_params, params, grads, m, v, lr, beta1, beta2, eps, c1, c2);
    FIPC_LAUNCHED();
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

}  // extern "C"

// ---------------------------------------------------------------- per-vertex features
#include "geometry.cuh"

namespace fipc {

constexpr int MLP_NBR = 16;

__global__ void k_fill_u32(int n, unsigned* __restrict__ a, unsigned v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}

// distance of each constraint row (square root of its squared distance), min'd into its vertices
// (non-negative floats order like their bit patterns, so atomicMin on the bits is exact)
__global__ void k_row_dist(int type, int n, const int4* __restrict__ rows, const double* __restrict__ x, unsigned* __restrict__ dmin) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int4 q = rows[r];
    double d2;
    switch (type) {
        case T_PP: d2 = d_PP(ld3(x, q.x), ld3(x, q.y)); break;
        case T_PE: d2 = d_PE(ld3(x, q.x), ld3(x, q.y), ld3(x, q.z)); break;
        case T_PT: d2 = d_PT(ld3(x, q.x), ld3(x, q.y), ld3(x, q.z), ld3(x, q.w)); break;
        case T_EE: case T_EEM: d2 = d_EE(ld3(x, q.x), ld3(x, q.y), ld3(x, q.z), ld3(x, q.w)); break;
        case T_PPM: d2 = d_PP(ld3(x, q.x), ld3(x, q.z)); break;
        default: d2 = d_PE(ld3(x, q.x), ld3(x, q.z), ld3(x, q.w)); break;
    }
    const unsigned bits = __float_as_uint((float)sqrt(fmax(d2, 0.0)));
    const int nv = type_nverts(type);
    const int id[4] = {q.x, q.y, q.z, q.w};
    for (int k = 0; k < nv; ++k) atomicMin(dmin + id[k], bits);
}

// X[i] = (16 one-ring relative positions / h, v dt / h, dx_prev / h, min(dist / dhat, 1), 0 pad);
// relative positions are x_j - x_i, or (x_j - x_i) - (X_j - X_i) against the rest shape X when
// x0 is given (the one-ring's deformation)
__global__ void k_features(int nV, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ x,
                           const double* __restrict__ x0, const double* __restrict__ v, const double* __restrict__ dxp, double dt,
                           double inv_h, double inv_dhat, const unsigned* __restrict__ dmin, float* __restrict__ X) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nV) return;
    float* f = X + (size_t)i * MLP_IN;
    const v3 xi = ld3(x, i);
    const v3 Xi = x0 ? ld3(x0, i) : mk(0, 0, 0);
    int k = 0;
    for (int e = rp[i]; e < rp[i + 1] && k < MLP_NBR; ++e) {
        const int j = ci[e];
        if (j == i) continue;
        v3 d = ld3(x, j) - xi;
        if (x0) d = d - (ld3(x0, j) - Xi);
        f[3 * k] = (float)(d.x * inv_h);
        f[3 * k + 1] = (float)(d.y * inv_h);
        f[3 * k + 2] = (float)(d.z * inv_h);
        ++k;
    }
    for (; k < MLP_NBR; ++k) f[3 * k] = f[3 * k + 1] = f[3 * k + 2] = 0.f;
    const v3 vi = ld3(v, i), pi = ld3(dxp, i);
    f[48] = (float)(vi.x * dt * inv_h);
    f[49] = (float)(vi.y * dt * inv_h);
    f[50] = (float)(vi.z * dt * inv_h);
    f[51] = (float)(pi.x * inv_h);
    f[52] = (float)(pi.y * inv_h);
    f[53] = (float)(pi.z * inv_h);
    const float dm = __uint_as_float(dmin[i]);
    f[54] = fminf(dm * (float)inv_dhat, 1.f);
    for (int q = 55; q < MLP_IN; ++q) f[q] = 0.f;
}

}  // namespace fipc

extern "C" int fipc_mlp_features(fipc_ctx* c, const double* x, const double* v, const double* dx_prev, double h, int rest_relative,
                                 float* X, void* stream) {
    if (!c || !x || !v || !dx_prev || !X || !(h > 0)) return FIPC_ERR_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    if (c->mlp_dist.ensure(4ll * c->nV)) return FIPC_ERR_CUDA;
    unsigned* dmin = c->mlp_dist.as<unsigned>();
    k_fill_u32<<<nblk(c->nV, 256), 256, 0, s>>>(c->nV, dmin, 0x7f800000u);   // +inf
    FIPC_LAUNCHED();
    for (int t = 0; t < N_TYPES; ++t) {
        if (c->h_counts[t] <= 0) continue;
        k_row_dist<<<nblk(c->h_counts[t], 128), 128, 0, s>>>(t, c->h_counts[t], (const int4*)c->list_rows(t), x, dmin);
        FIPC_LAUNCHED();
    }
    k_features<<<nblk(c->nV, 128), 128, 0, s>>>(c->nV, c->row_ptr, c->col_idx, x, rest_relative ? c->x0 : nullptr, v, dx_prev, c->dt,
                                                1.0 / h, 1.0 / c->dhat, dmin, X);
    FIPC_LAUNCHED();
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}

// ---------------------------------------------------------------- smoothing of a displacement
namespace fipc {
// out_i = mean of d_j over the one-ring of i including i (the elastic block pattern); 0 on
// Dirichlet vertices
__global__ void k_ring_mean(int nV, const int* __restrict__ rp, const int* __restrict__ ci, const unsigned char* __restrict__ fixed,
                            const double* __restrict__ d, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nV) return;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (!fixed[i]) {
        for (int e = rp[i]; e < rp[i + 1]; ++e) {
            const int j = ci[e];
            s0 += d[3 * (size_t)j];
            s1 += d[3 * (size_t)j + 1];
            s2 += d[3 * (size_t)j + 2];
        }
        const double inv = 1.0 / (double)(rp[i + 1] - rp[i]);
        s0 *= inv;
        s1 *= inv;
        s2 *= inv;
    }
    out[3 * (size_t)i] = s0;
    out[3 * (size_t)i + 1] = s1;
    out[3 * (size_t)i + 2] = s2;
}
}  // namespace fipc

// passes of one-ring averaging of d [V][3] (in place, tmp: scratch [V][3]); the learned
// correction is smoothed so that its vertex-to-vertex noise does not load the elastic energy
extern "C" int fipc_mlp_smooth(fipc_ctx* c, const unsigned char* fixed, double* d, double* tmp, int passes, void* stream) {
    if (!c || !fixed || !d || !tmp || passes < 0) return FIPC_ERR_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    for (int k = 0; k < passes; ++k) {
        k_ring_mean<<<nblk(c->nV, 128), 128, 0, s>>>(c->nV, c->row_ptr, c->col_idx, fixed, d, tmp);
        FIPC_LAUNCHED();
        FIPC_CUDA(cudaMemcpyAsync(d, tmp, 24ll * c->nV, cudaMemcpyDeviceToDevice, s));
    }
    FIPC_CUDA(cudaGetLastError());
    return FIPC_OK;
}
