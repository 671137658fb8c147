// out = softmax(scale * X + term) . V in f32 throughout: the second half of an attention step that keeps f32 operands (few
// rows, or a small product: plan.cpp, `try_softmax_matmul`).  X are the scores, [batch][m][n] with any strides, V is
// [batch][n][dv] with its columns contiguous; the probabilities stay in shared memory, and the result is stored with the
// heads merged where a merge follows.
//
// One CTA per 16 rows (512 threads) or 32 rows (256 threads) of a batch entry: each warp takes one or four rows' softmax (the
// whole row in shared memory), then groups of four warps share the keys of a block of 128, an eighth of the rows x 4 columns
// of the result per thread, as packed multiply-adds over column pairs, and the groups' sums meet in shared memory.  V comes
// in blocks of 128 keys through two buffers, the first two of them requested ahead of the softmax.
//
// What bounds it is latency (scores from L2, softmax, product, store; the arithmetic of 12 heads of 120 rows and keys is
// 1 us).  Softmax, product and the copy that merges the heads as three launches -> this one: 12 heads of 120 rows and keys,
// 64 columns 12.8 -> 7.1 us; 8 heads of 1024 rows, 77 keys, 80 columns 23.7 -> 11.2 us.  16 rows by 256 threads took 7.7 us
// (1 800 instructions a warp on two warps a scheduler), 32 rows by 512 threads 15.4.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../kernels.h"
#include "launch.cuh"

namespace kn {

namespace {

constexpr int kSmKeys = 128;

__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*(uint64_t*)&a), "l"(*(uint64_t*)&b), "l"(*(uint64_t*)&c));
    return *(float2*)&d;
}

struct SoftmaxMatmulParams {
    const float *x, *term, *v;   // term may be null
    float* out;
    int32_t m, n, dv, tiles;     // tiles of rows per batch entry
    int32_t v_bi;                // batch entry bt of V is at (bt % v_bi) * sv[0] + (bt / v_bi) * sv[2]
    int32_t out_heads;           // of the result at (bt / out_heads) * sc[0] + (bt % out_heads) * sc[1]
    int64_t sx[3], st[3], sv[3], sc[3];   // sv: entry, key, group of entries; sc: group of entries, entry, row
    float scale;
};

// PANELS: of 64 columns of V; RPT: rows per thread, an eighth of the CTA's; GROUPS of four warps
template <int PANELS, int RPT, int GROUPS>
__global__ void __launch_bounds__(GROUPS * 128) softmax_matmul_kernel(const __grid_constant__ SoftmaxMatmulParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kThreads = GROUPS * 128, kRows = 8 * RPT, kWarps = GROUPS * 4, kWarpRows = kRows / kWarps;
    const int blocks = (p.n + kSmKeys - 1) / kSmKeys, pitch = blocks * kSmKeys + 4, block_floats = kSmKeys * p.dv;
    float* const values = (float*)smem;                                   // up to two blocks of [128 keys][columns]
    float* const prob = values + (blocks > 1 ? 2 : 1) * block_floats;     // [rows][pitch]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned bt = blockIdx.x / (unsigned)p.tiles;
    const int row0 = (int)(blockIdx.x - bt * (unsigned)p.tiles) * kRows;
    const float* const v = p.v + (bt % (unsigned)p.v_bi) * p.sv[0] + (bt / (unsigned)p.v_bi) * p.sv[2];
    const int chunks = p.dv >> 2, v_row = tid / chunks, v_chunk = tid - v_row * chunks, row_step = kThreads / chunks, chunk_step = kThreads - row_step * chunks;
    auto load_values = [&](int block) {
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(values + (block & 1) * block_floats);
        int r = v_row, c = v_chunk;
        for (int e = tid; e < kSmKeys * chunks; e += kThreads) {
            const int key = block * kSmKeys + r;
            const bool in = key < p.n;   // (zeros after the last key)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)e * 16u), "l"(in ? v + key * p.sv[1] + c * 4 : v), "r"(in ? 16 : 0)
                         : "memory");
            r += row_step, c += chunk_step;
            if (c >= chunks) c -= chunks, r++;
        }
    };
    pdl_enter();
#pragma unroll
    for (int b = 0; b < 2; b++) {
        if (b < blocks) load_values(b);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // a warp's rows, 128 scores of each requested at a time
    float top[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) top[i] = -INFINITY;
    for (int c0 = lane; c0 < p.n; c0 += 128) {
        float x[kWarpRows][4], t[kWarpRows][4];
#pragma unroll
        for (int i = 0; i < kWarpRows; i++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int row = row0 + warp + i * kWarps, c = c0 + q * 32;
                const bool in = row < p.m && c < p.n;
                x[i][q] = in ? p.x[bt * p.sx[0] + row * p.sx[1] + c * p.sx[2]] : 0.f;
                t[i][q] = in && p.term ? p.term[bt * p.st[0] + row * p.st[1] + c * p.st[2]] : 0.f;
            }
#pragma unroll
        for (int i = 0; i < kWarpRows; i++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float s = p.scale * x[i][q] + t[i][q];
                if (c0 + q * 32 < p.n) {
                    prob[(warp + i * kWarps) * pitch + c0 + q * 32] = s;
                    top[i] = fmaxf(top[i], s);
                }
            }
    }
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], off));
    }
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) {
        float* const e = prob + (warp + i * kWarps) * pitch;
        float sum = 0.f;
#pragma unroll 4
        for (int c = lane; c < p.n; c += 32) {
            const float y = expf(e[c] - top[i]);
            e[c] = y;
            sum += y;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        // (divided here and not after the product, which would be out of range for values of V within `sum` of the largest f32)
#pragma unroll 4
        for (int c = lane; c < p.n; c += 32) e[c] /= sum;
        for (int c = p.n + lane; c < blocks * kSmKeys; c += 32) e[c] = 0.f;
    }

    // lanes 1..3 pick the row, 0 and 4 and the warp the columns (which reads are served in one pass: see contract_simt.cu)
    const int group = tid >> 7, tx = ((lane & 1) | ((lane >> 4) << 1)) + 4 * (warp & 3), ty = (lane >> 1) & 7;
    float2 acc[RPT][PANELS][2];
#pragma unroll
    for (int i = 0; i < RPT; i++)
#pragma unroll
        for (int c = 0; c < PANELS; c++) acc[i][c][0] = acc[i][c][1] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int b = 0; b < blocks; b++) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();   // (the first one: the probabilities too)
        const int block_keys = (min(kSmKeys, p.n - b * kSmKeys) + 3) & ~3, share = (block_keys + GROUPS * 4 - 1) / (GROUPS * 4) * 4;
        const int first = group * share, keys = min(share, block_keys - first);
        const float* P = prob + ty * pitch + b * kSmKeys + first;
        const float* V = values + (b & 1) * block_floats + first * p.dv + tx * 4;
#pragma unroll 4
        for (int k = 0; k < keys; k += 4) {
            float4 a[RPT];
#pragma unroll
            for (int i = 0; i < RPT; i++) a[i] = *(const float4*)(P + i * 8 * pitch + k);
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int c = 0; c < PANELS; c++) {
                    if (c * 16 + tx >= chunks) continue;
                    const float4 w = *(const float4*)(V + (k + q) * p.dv + c * 64);
#pragma unroll
                    for (int i = 0; i < RPT; i++) {
                        const float y = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
                        acc[i][c][0] = fma_pair(make_float2(y, y), make_float2(w.x, w.y), acc[i][c][0]);
                        acc[i][c][1] = fma_pair(make_float2(y, y), make_float2(w.z, w.w), acc[i][c][1]);
                    }
                }
        }
        __syncthreads();   // the block has been read
        if (b + 2 < blocks) load_values(b + 2);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float4* const others = (float4*)values;   // the other groups' sums, [group - 1][row][column / 4] (a block of V has 128 rows)
    if (group > 0) {
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int c = 0; c < PANELS; c++)
                if (c * 16 + tx < chunks)
                    others[((group - 1) * kRows + ty + i * 8) * chunks + c * 16 + tx] = make_float4(acc[i][c][0].x, acc[i][c][0].y, acc[i][c][1].x, acc[i][c][1].y);
    }
    __syncthreads();
    if (group > 0) return;
    float* const out = p.out + (bt / (unsigned)p.out_heads) * p.sc[0] + (bt % (unsigned)p.out_heads) * p.sc[1];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
        const int r = ty + i * 8;
        if (row0 + r >= p.m) continue;
#pragma unroll
        for (int c = 0; c < PANELS; c++) {
            if (c * 16 + tx >= chunks) continue;
            float4 o = make_float4(acc[i][c][0].x, acc[i][c][0].y, acc[i][c][1].x, acc[i][c][1].y);
#pragma unroll
            for (int g = 0; g < GROUPS - 1; g++) {
                const float4 t = others[(g * kRows + r) * chunks + c * 16 + tx];
                o.x += t.x, o.y += t.y, o.z += t.z, o.w += t.w;
            }
            *(float4*)(out + (int64_t)(row0 + r) * p.sc[2] + (c * 16 + tx) * 4) = o;
        }
    }
}

int shared_bytes(int64_t n, int64_t dv, int64_t rows) {
    const int64_t blocks = (n + kSmKeys - 1) / kSmKeys;
    return (int)(((blocks > 1 ? 2 : 1) * kSmKeys * dv + rows * (blocks * kSmKeys + 4)) * 4);
}

template <int PANELS, int RPT, int GROUPS>
int launch_rows(const SoftmaxMatmulParams& q, unsigned grid, cudaStream_t stream) {
    static std::mutex mu;
    static bool done[64] = {false};
    int device = 0;
    cudaGetDevice(&device);
    {   // (the opt-in to more than 48 KB is per device)
        std::lock_guard<std::mutex> lock(mu);
        if (device >= 0 && device < 64 && !done[device]) {
            cudaError_t e = cudaFuncSetAttribute(softmax_matmul_kernel<PANELS, RPT, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e != cudaSuccess) return (int)e;
            done[device] = true;
        }
    }
    launch_pdl(softmax_matmul_kernel<PANELS, RPT, GROUPS>, dim3(grid), dim3(GROUPS * 128), (size_t)shared_bytes(q.n, q.dv, 8 * RPT), stream, q);
    return (int)cudaGetLastError();
}

}  // namespace

int launch_softmax_matmul(const GemmParams& g, cudaStream_t stream) {
    SoftmaxMatmulParams q{};
    q.x = g.a;
    q.term = g.add1;
    q.v = g.b;
    q.out = g.c;
    q.m = (int32_t)g.m;
    q.n = (int32_t)g.k;
    q.dv = (int32_t)g.n;
    for (int i = 0; i < 3; i++) q.sx[i] = g.sa[i], q.st[i] = g.s1[i], q.sc[i] = g.sc[i];
    if (g.b4.enabled) {
        q.v_bi = g.b4.bi;
        q.sv[0] = g.b4.strides[2], q.sv[1] = g.b4.strides[1], q.sv[2] = g.b4.strides[3];
    } else {
        q.v_bi = (int32_t)g.batch;
        q.sv[0] = g.sb[0], q.sv[1] = g.sb[1];
    }
    q.out_heads = g.out_heads;
    q.scale = g.softmax_scale;
    // 32 rows share a pass over V where that leaves every SM a CTA (and two of them fit one SM)
    const bool wide = g.batch * ((g.m + 31) / 32) >= 148 && shared_bytes(q.n, q.dv, 32) <= 113 * 1024;
    const int rows = wide ? 32 : 16;
    q.tiles = (int32_t)((g.m + rows - 1) / rows);
    const unsigned grid = (unsigned)(g.batch * q.tiles);
    if (wide) return g.n > 64 ? launch_rows<2, 4, 2>(q, grid, stream) : launch_rows<1, 4, 2>(q, grid, stream);
    return g.n > 64 ? launch_rows<2, 2, 4>(q, grid, stream) : launch_rows<1, 2, 4>(q, grid, stream);
}

}  // namespace kn
