// Small dense layers that follow one another, and a softmax behind them, as ONE launch: x -> act(x . W + b) -> ... -> softmax.  The
// executor launches a run of such steps (a small policy network, the last layer of a value head and its softmax) this way; by
// themselves they are a launch of 3 to 5 us each whose arithmetic takes none of it.
//
// A warp takes R rows through all layers; the weights of all layers lie in shared memory (requested ahead of the dependency wait:
// they are constants).  Layers of more than eight columns give each lane a column of every 32; narrower ones give the lanes the
// reduction.  f32 multiply-adds throughout; four products are summed by themselves before they join one of two sums over every other four
// (against 64 bits, layers launched one by one 1: one running sum 1.1, of fours 1.02, two of them 1.00; 16-32-32-4, 16 networks of 4000
// rows; 128-32-8 0.78).
//
// What bounds it: one launch, the first loads, and a chain of k multiply-adds per layer.  8 rows of 16 -> 32 -> 32 -> 4 + softmax:
// four launches of 14.3 us -> one; with its copies and the host's calls 28.6 -> 22.4 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "../kernels.h"
#include "launch.cuh"

namespace kn {

namespace {

constexpr int kWarps = 4, kThreads = 32 * kWarps;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) x = fmaxf(x, __shfl_xor_sync(kFull, x, s));
    return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) x += __shfl_xor_sync(kFull, x, s);
    return x;
}

template <int R>
__global__ void __launch_bounds__(kThreads) dense_chain_kernel(const __grid_constant__ DenseChainParams p) {
    __shared__ float weights[kDenseChainWeights];
    __shared__ __align__(16) float values[kWarps][R][kDenseChainMaxK];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int l = 0; l < p.n_layers; l++) {
        const DenseLayer& d = p.layer[l];
        float* to = weights + d.at;
        if (d.n > 8) {   // [k, whole groups of four][columns, whole groups of 32], then the bias
            const int cols = (d.n + 31) & ~31, rows = (d.k + 3) & ~3;
            for (int i = threadIdx.x; i < rows * cols; i += kThreads) {
                const int k = i / cols, n = i - k * cols;
                to[i] = k < d.k && n < d.n ? __ldg(d.w + k * d.w_k + n * d.w_n) : 0.f;
            }
            for (int n = threadIdx.x; n < cols; n += kThreads) to[rows * cols + n] = d.bias && n < d.n ? __ldg(d.bias + n * d.bias_n) : 0.f;
        } else {         // [n][k], then the bias
            for (int i = threadIdx.x; i < d.n * d.k; i += kThreads) {
                const int n = i / d.k, k = i - n * d.k;
                to[i] = __ldg(d.w + k * d.w_k + n * d.w_n);
            }
            if (threadIdx.x < d.n) to[d.n * d.k + threadIdx.x] = d.bias ? __ldg(d.bias + threadIdx.x * d.bias_n) : 0.f;
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t row0 = ((int64_t)blockIdx.x * kWarps + warp) * R;
    const int k0 = p.layer[0].k, k0_padded = (k0 + 3) & ~3;
#pragma unroll
    for (int r = 0; r < R; r++)
        for (int k = lane; k < k0_padded; k += 32)
            values[warp][r][k] = k < k0 && row0 + r < p.rows ? p.in[(row0 + r) * p.in_row + k * p.in_col] : 0.f;
    __syncthreads();
    if (row0 >= p.rows) return;
    for (int l = 0; l < p.n_layers; l++) {
        const DenseLayer& d = p.layer[l];
        const float* w = weights + d.at;
        const bool last = l == p.n_layers - 1;
        if (d.n > 8) {
            const int cols = (d.n + 31) & ~31, rows = (d.k + 3) & ~3, groups = cols >> 5;
            float y[R][4], odd[R][4];   // (every other four products)
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) y[r][c] = odd[r][c] = 0.f;
            auto four = [&](float (&to)[R][4], int k) {
                float4 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = *(const float4*)&values[warp][r][k];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= groups) break;
                    const float* at = w + k * cols + c * 32 + lane;
                    const float w0 = at[0], w1 = at[cols], w2 = at[2 * cols], w3 = at[3 * cols];
#pragma unroll
                    for (int r = 0; r < R; r++) to[r][c] += fmaf(x[r].y, w1, x[r].x * w0) + fmaf(x[r].w, w3, x[r].z * w2);
                }
            };
            for (int k = 0; k < rows; k += 8) {
                four(y, k);
                if (k + 4 < rows) four(odd, k + 4);
            }
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) y[r][c] += odd[r][c];
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (row0 + r >= p.rows) continue;
                float top = -INFINITY;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= groups) break;
                    y[r][c] += w[rows * cols + c * 32 + lane];
                    if (d.relu) y[r][c] = fmaxf(y[r][c], 0.f);
                    if (c * 32 + lane < d.n) top = fmaxf(top, y[r][c]);
                }
                if (last && p.softmax) {
                    top = warp_max(top);
                    float sum = 0.f;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        if (c >= groups) break;
                        y[r][c] = expf(y[r][c] - top);
                        if (c * 32 + lane < d.n) sum += y[r][c];
                    }
                    sum = warp_sum(sum);
#pragma unroll
                    for (int c = 0; c < 4; c++) y[r][c] = y[r][c] / sum;
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= groups) break;
                    const int n = c * 32 + lane;
                    if (!last) values[warp][r][n] = n < d.n ? y[r][c] : 0.f;   // (past n: NaN where the row holds an infinity)
                    else if (n < d.n) p.out[(row0 + r) * p.out_row + n] = y[r][c];
                }
            }
        } else {
            float y[R][8];
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int n = 0; n < 8; n++) y[r][n] = 0.f;
            for (int k = lane; k < d.k; k += 32) {
                float x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = values[warp][r][k];
#pragma unroll
                for (int n = 0; n < 8; n++) {
                    if (n >= d.n) break;
                    const float v = w[n * d.k + k];
#pragma unroll
                    for (int r = 0; r < R; r++) y[r][n] = fmaf(x[r], v, y[r][n]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (row0 + r >= p.rows) continue;
                float top = -INFINITY, sum = 0.f, mine = 0.f;
#pragma unroll
                for (int n = 0; n < 8; n++) {
                    if (n >= d.n) break;
                    y[r][n] = warp_sum(y[r][n]) + w[d.n * d.k + n];
                    if (d.relu) y[r][n] = fmaxf(y[r][n], 0.f);
                    top = fmaxf(top, y[r][n]);
                }
                if (last && p.softmax) {
#pragma unroll
                    for (int n = 0; n < 8; n++) {
                        if (n >= d.n) break;
                        y[r][n] = expf(y[r][n] - top);
                        sum += y[r][n];
                    }
#pragma unroll
                    for (int n = 0; n < 8; n++) y[r][n] = y[r][n] / sum;
                }
#pragma unroll
                for (int n = 0; n < 8; n++)
                    if (n == lane) mine = y[r][n];
                if (last && lane < d.n) p.out[(row0 + r) * p.out_row + lane] = mine;
                if (!last && lane < 8) values[warp][r][lane] = lane < d.n ? mine : 0.f;
            }
        }
        __syncwarp();
    }
}

}  // namespace

int dense_chain_weights(int k, int n) {
    return n > 8 ? ((k + 3) & ~3) * ((n + 31) & ~31) + ((n + 31) & ~31) : n * k + n;
}

int launch_dense_chain(const DenseChainParams& p, cudaStream_t stream) {
    if (p.rows == 0) return 0;
    // A row per warp until the chip has several blocks an SM, then four, which share the reads of the weights; the fewer those are, the
    // later.  f32, one row -> four: 100-3 + softmax, 4096 rows 8.9 -> 12.3 us, 9000 13.7 -> 13.0; 200-8-8 3000 10.2 -> 18.4, 6000 19.1 -> 20.1;
    // 64-64 3000 17.7 -> 12.2.
    int weights = 0;
    for (int l = 0; l < p.n_layers; l++) weights += dense_chain_weights(p.layer[l].k, p.layer[l].n);
    const bool four = p.rows > 148 * kWarps * (weights <= 512 ? 15 : weights <= 2048 ? 7 : 4);
    const int64_t per_block = kWarps * (four ? 4 : 1), blocks = (p.rows + per_block - 1) / per_block;
    if (four) launch_pdl(dense_chain_kernel<4>, dim3((unsigned)blocks), dim3(kThreads), (size_t)0, stream, p);
    else launch_pdl(dense_chain_kernel<1>, dim3((unsigned)blocks), dim3(kThreads), (size_t)0, stream, p);
    return (int)cudaGetLastError();
}

}  // namespace kn
