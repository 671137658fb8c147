// out = softmax(scale * X + term) . V in f32 throughout: the second half of an attention step that keeps f32 operands (few
// rows, or a small product: plan.cpp, `try_softmax_matmul`).  X are the scores, [batch][m][n] with any strides, V is
// [batch][n][dv] with its columns contiguous; the probabilities stay in shared memory, and the result is stored with the
// heads merged where a merge follows.
//
// One CTA per 16 rows (512 threads) or 32 rows (256 threads) of a batch entry: all of V, at most 128 keys, is requested ahead of
// the softmax; each warp takes one or four rows' softmax (the whole row in shared memory), then groups of four warps share the
// keys, an eighth of the rows x 4 columns of the result per thread, as packed multiply-adds over column pairs, and the groups'
// sums meet in shared memory.  Products of four keys are summed by themselves before they join the sum over all keys: one
// running sum is up to 1.3 times as far from 64 bits as the separate steps for rows of 128 keys.
//
// What bounds it is latency (scores and V from L2, softmax, product, store; the arithmetic of 12 heads of 120 rows and keys is
// 1 us).  Softmax, product and the copy that merges the heads as three launches -> this one: 12 heads of 120 rows and keys,
// 64 columns 9.7 -> 4.8 us; 8 heads of 1024 rows, 77 keys, 80 columns 21.3 -> 10.5 us (in a graph of eight such calls; launched by
// itself 6.2 and 11.0, kernel_bench's softmax_values_short*).  With more keys in blocks of 128, two of them in flight, it lost to the separate steps: 12 heads of 16 rows, 88 columns, 256 keys 13.6 us against 6.5, 1024 keys 49
// against 12; one CTA reads all of V, where contract_cols_kernel spreads the keys over a cluster.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../kernels.h"
#include "launch.cuh"

namespace kn {

namespace {


struct SoftmaxMatmulParams {
    const float *x, *term, *v;   // term may be null
    float* out;
    int32_t m, n, dv, tiles;     // tiles of rows per batch entry
    int32_t v_bi;                // batch entry bt of V is at (bt % v_bi) * sv[0] + (bt / v_bi) * sv[2]
    int32_t out_heads;           // of the result at (bt / out_heads) * sc[0] + (bt % out_heads) * sc[1]
    int64_t sx[3], st[3], sv[3], sc[3];   // sv: entry, key, group of entries; sc: group of entries, entry, row
    float scale;
};

// keys, and with them V and the probabilities, in steps of four (the last ones zero)
__host__ __device__ __forceinline__ int whole_keys(int n) { return (n + 3) & ~3; }

// PANELS: of 64 columns of V; RPT: rows per thread, an eighth of the CTA's; GROUPS of four warps
template <int PANELS, int RPT, int GROUPS>
__global__ void __launch_bounds__(GROUPS * 128) softmax_matmul_kernel(const __grid_constant__ SoftmaxMatmulParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kThreads = GROUPS * 128, kRows = 8 * RPT, kWarps = GROUPS * 4, kWarpRows = kRows / kWarps;
    constexpr int kPitch = (int)kSoftmaxMatmulMaxKeys + 4;
    float* const prob = (float*)smem;                 // [rows][pitch]
    float* const values = prob + kRows * kPitch;      // [keys][columns]; later the groups' sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, all_keys = whole_keys(p.n);
    const unsigned bt = blockIdx.x / (unsigned)p.tiles;
    const int row0 = (int)(blockIdx.x - bt * (unsigned)p.tiles) * kRows;
    const int chunks = p.dv >> 2;
    pdl_enter();
    {
        const float* const v = p.v + (bt % (unsigned)p.v_bi) * p.sv[0] + (bt / (unsigned)p.v_bi) * p.sv[2];
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(values);
        const int row_step = kThreads / chunks, chunk_step = kThreads - row_step * chunks;
        int r = tid / chunks, c = tid - r * chunks;
        for (int e = tid; e < all_keys * chunks; e += kThreads) {
            const bool in = r < p.n;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)e * 16u), "l"(in ? v + r * p.sv[1] + c * 4 : v), "r"(in ? 16 : 0)
                         : "memory");
            r += row_step, c += chunk_step;
            if (c >= chunks) c -= chunks, r++;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // a warp's rows, all their scores requested at once
    float s[kWarpRows][4], top[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int row = row0 + warp + i * kWarps, c = lane + q * 32;
            const bool in = row < p.m && c < p.n;
            const float x = in ? p.x[bt * p.sx[0] + row * p.sx[1] + c * p.sx[2]] : 0.f;
            const float t = in && p.term ? p.term[bt * p.st[0] + row * p.st[1] + c * p.st[2]] : 0.f;
            s[i][q] = p.scale * x + t;
        }
    }
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) {
        top[i] = -INFINITY;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (lane + q * 32 < p.n) top[i] = fmaxf(top[i], s[i][q]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], off));
    }
#pragma unroll
    for (int i = 0; i < kWarpRows; i++) {
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s[i][q] = lane + q * 32 < p.n ? expf(s[i][q] - top[i]) : 0.f;
            sum += s[i][q];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        // (divided here and not after the product, which would be out of range for values of V within `sum` of the largest f32)
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (lane + q * 32 < all_keys) prob[(warp + i * kWarps) * kPitch + lane + q * 32] = s[i][q] / sum;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // lanes 1..3 pick the row, 0 and 4 and the warp the columns (which reads are served in one pass: see contract_simt.cu)
    const int group = tid >> 7, tx = ((lane & 1) | ((lane >> 4) << 1)) + 4 * (warp & 3), ty = (lane >> 1) & 7;
    const int share = (all_keys + GROUPS * 4 - 1) / (GROUPS * 4) * 4, first = group * share, keys = min(share, all_keys - first);
    float2 acc[RPT][PANELS][2];
#pragma unroll
    for (int i = 0; i < RPT; i++)
#pragma unroll
        for (int c = 0; c < PANELS; c++) acc[i][c][0] = acc[i][c][1] = make_float2(0.f, 0.f);
    const float* const P = prob + ty * kPitch + first;
    const float* V[PANELS];   // (past the last column: that one again, not stored; a branch around these reads took half as long again)
#pragma unroll
    for (int c = 0; c < PANELS; c++) V[c] = values + first * p.dv + min(c * 16 + tx, chunks - 1) * 4;
#pragma unroll 2
    for (int k = 0; k < keys; k += 4) {
        float4 a[RPT];
#pragma unroll
        for (int i = 0; i < RPT; i++) a[i] = *(const float4*)(P + i * 8 * kPitch + k);
#pragma unroll
        for (int c = 0; c < PANELS; c++) {
            float2 part[RPT][2];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 w = *(const float4*)(V[c] + (k + q) * p.dv);
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    const float y = q == 0 ? a[i].x : q == 1 ? a[i].y : q == 2 ? a[i].z : a[i].w;
                    const float2 lo = make_float2(w.x, w.y), hi = make_float2(w.z, w.w), yy = make_float2(y, y), zero = make_float2(0.f, 0.f);
                    part[i][0] = fma_pair(yy, lo, q == 0 ? zero : part[i][0]);
                    part[i][1] = fma_pair(yy, hi, q == 0 ? zero : part[i][1]);
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; i++)
#pragma unroll
                for (int h = 0; h < 2; h++) acc[i][c][h].x += part[i][h].x, acc[i][c][h].y += part[i][h].y;
        }
    }
    __syncthreads();   // V has been read
    float4* const others = (float4*)values;   // the other groups' sums, [group - 1][row][column / 4]
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

// (V's place takes the sums of all groups but one, too)
int shared_bytes(int n, int dv, int rows, int groups) {
    return (rows * ((int)kSoftmaxMatmulMaxKeys + 4) + std::max(whole_keys(n), (groups - 1) * rows) * dv) * 4;
}

template <int PANELS, int RPT, int GROUPS>
int launch_rows(const SoftmaxMatmulParams& q, unsigned grid, cudaStream_t stream) {
    static std::mutex mu;
    static bool done[64] = {false};
    if (int e = allow_shared(softmax_matmul_kernel<PANELS, RPT, GROUPS>, 128 * 1024, done, mu)) return e;
    launch_pdl(softmax_matmul_kernel<PANELS, RPT, GROUPS>, dim3(grid), dim3(GROUPS * 128), (size_t)shared_bytes(q.n, q.dv, 8 * RPT, GROUPS), stream, q);
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
    // 32 rows share a pass over V where that leaves every SM a CTA
    const bool wide = g.batch * ((g.m + 31) / 32) >= 148;
    const int rows = wide ? 32 : 16;
    q.tiles = (int32_t)((g.m + rows - 1) / rows);
    const unsigned grid = (unsigned)(g.batch * q.tiles);
    if (wide) return g.n > 64 ? launch_rows<2, 4, 2>(q, grid, stream) : launch_rows<1, 4, 2>(q, grid, stream);
    return g.n > 64 ? launch_rows<2, 2, 4>(q, grid, stream) : launch_rows<1, 2, 4>(q, grid, stream);
}

}  // namespace kn
