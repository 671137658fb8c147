// A run of 3x3 stride-1 same-padding convolutions as ONE kernel on CTA PAIRS (sm_100a, `cta_group::2`).
//
// The same step as conv_chain.cu (whole images stay in shared memory from the first layer to the last, only filters stream in),
// with the operands the other way round: D[position = TMEM lane][output channel = column].
//   A operand  128 positions of each CTA's own images (M = 256 over the pair), per 32-channel block one 128-byte row per padded
//              position; a filter tap is the same operand started a constant number of rows further on
//   B operand  the layer's filter [output channels x 32 input channels], HALF of its rows in each CTA: a CTA fetches and stores
//              half of the filter, and every filter row read serves 256 positions
// The padding columns of 8-wide images are stepped over: an image row is one group of eight operand rows, and the distance
// between groups (the descriptor's stride byte offset) is 9 rows, so M = 128 is exactly the pixels of two 8 x 8 boards whose
// rows alternate (side by side: group 2 y + board).  Other widths take the padded image as it is (distance 8).
//
// The K loop is ordered (channel block, tap), and the layer's accumulator alternates between two sets of TMEM columns: the
// epilogue writes the next layer's operand one channel block (32 columns) after the other, in place (every MMA of the layer has
// read it), and the next layer's MMAs over block 0 run while blocks 1.. are still being written.  Of the epilogue only the first
// block and the hand-over are exposed.
//
// What bounds it: an M 256 x N 128 x K 8 instruction keeps a tensor core busy for 64 cycles and reads 4 KB of positions and
// 2 KB of filter through each SM's shared-memory pipe while the copy engine writes 2 KB: 64 wavefronts of 128 bytes, against
// 100 per instruction of 72 cycles in conv_chain_kernel, whose mainloop that pipe bound.  A layer of 128 channels takes 10 900 SM
// cycles, 9 750 of them its 144 instructions (67 each), the rest the first channel block's epilogue and the hand-over (traced:
// KN_CHAIN_TRACE=1).  33 layers + heads, 256 boards of 8 x 8: 312 -> 202 us (771 TFLOP/s); 2048 boards: 2170 -> 1435 us; 17 layers of
// 64 channels, 101 boards of 9 x 9: 89.3 -> 54.4 us.
//
// Warp roles per CTA: an elected lane of warp 0 streams its half of the filters (arriving on the LEADER's barrier), an elected
// lane of the leader's warp 1 issues the MMAs of both, warps 2.. are the epilogue (four per TMEM lane quarter, 8 columns of a
// channel block each).  Every mbarrier wait is bounded; on expiry the status word is raised and all roles leave.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>

#include "../tc.h"
#include "launch.cuh"
#include "tc_host.h"
#include "tc_ptx.cuh"

namespace kn {

namespace {

using namespace tcp;

// Epilogue warps per TMEM lane quarter (two took 208.3 us for 33 layers of 256 boards and 40.1 for 17 of 32 channels, four 206.7 and
// 37.6), and the columns of a channel block that each takes.
constexpr int kEpilogueWarps = 4, kCols = 32 / kEpilogueWarps;
constexpr int kEpilogueThreads = 128 * kEpilogueWarps, kThreads = 64 + kEpilogueThreads;
constexpr uint32_t kSleepNs = 20000u;   // suspend-time hint of the waits
// Rows of biases in shared memory.  A warp reads its first columns of a layer's row ahead of that layer's accumulator (behind the
// wait 33 layers of 256 boards take 206.7 us, ahead of it 202.4), so the row is written two layers earlier: row (l + 2) % 3 once
// accumulator l is complete, handed over with the operand of layer l + 1, which accumulator l + 1 has read.
constexpr int kBiasRows = 3;

struct ChainPairKernelParams {
    const float* in;
    float* out;
    const float* bias;
    int64_t s_in[4], s_out[4];
    int32_t n_img, c_in, k, h, w;
    int32_t n_layers, per_cta, gx, gy, wp, pitch, rows_alloc, slots, tmem_cols, blocks;
    int32_t n_trunk, n_last;     // accumulator columns of a 3x3 layer and of the pointwise last layer
    int32_t acc_cols;            // distance of the two accumulators
    int32_t out_vec;             // `out` takes four channels in one aligned store
    uint32_t slot_bytes;
    long long* trace;            // KN_CHAIN_TRACE only
    uint8_t flags[kMaxChainLayers];
    uint8_t c_blocks[kMaxChainLayers];
    uint32_t* status;
    int32_t n_heads;
    int32_t head_begin[kMaxChainHeads + 1];
    float* head_out[kMaxChainHeads];
    int64_t head_s_out[kMaxChainHeads][4];
    uint8_t head_relu[kMaxChainHeads];
};

// K-major operand, 128-byte swizzle, groups of eight rows `pitch` rows apart.  (The swizzle follows the absolute address bits,
// whatever the start row and the distance of the groups.)
__device__ __forceinline__ uint64_t smem_desc_rows(uint32_t addr, uint32_t pitch) {
    return (smem_desc_sw128(addr) & ~((uint64_t)0x3FFF << 32)) | ((uint64_t)(pitch * 8u) << 32);
}

__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*(uint64_t*)&a), "l"(*(uint64_t*)&b));
    return *(float2*)&d;
}

// rounded to TF32 (nearest, ties away): the tensor core ignores the low 13 bits
__device__ __forceinline__ uint32_t operand_bits(uint32_t u) {
    return (u & 0x7F800000u) != 0x7F800000u ? u + 0x1000u : u;
}

// TRACE: whether the first CTA stamps its phases.  PARTIAL: the trunk's last channel block has columns that are no channels, which
// are kept zero (a test of them in every variant costs 1.7 to 4 %: 157 -> 163.6 us for 17 layers of 64 channels, 101 boards of 9 x 9,
// with the copies of the call)
template <bool TRACE, bool PARTIAL>
__global__ void __launch_bounds__(kThreads, 1)
conv_chain_pair_kernel(const __grid_constant__ CUtensorMap map_trunk, const __grid_constant__ CUtensorMap map_last,
                       const __grid_constant__ ChainPairKernelParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t block_bytes = (uint32_t)p.rows_alloc * 128u;
    const uint32_t act_bytes = (uint32_t)p.blocks * block_bytes;
    const uint32_t ring_base = base + act_bytes;
    const uint32_t bias_base = ring_base + (uint32_t)p.slots * p.slot_bytes;     // kBiasRows x 128 floats
    const uint32_t bar_base = bias_base + kBiasRows * 512u;
    const uint32_t full_bar = bar_base, empty_bar = full_bar + 8u * p.slots, act_bar = empty_bar + 8u * p.slots;
    const uint32_t accum_bar = act_bar + 8u * 4u, slot_addr = accum_bar + 8u;
    float* bias_s = (float*)(gen_base + (bias_base - base));
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + (slot_addr - base));
    volatile int* abandon = (volatile int*)(gen_base + (slot_addr + 4u - base));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)(blockIdx.x >> 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.slots; s++) {
            mbar_init(full_bar + 8u * s, 1);
            mbar_init(empty_bar + 8u * s, 1);
        }
        for (int b = 0; b < 4; b++) mbar_init(act_bar + 8u * b, 2 * kEpilogueThreads / 32);   // one arrival per epilogue warp of the pair
        mbar_init(accum_bar, 1);
        *abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {   // padding positions stay zero from here on
        uint4* z = (uint4*)gen_base;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t i = threadIdx.x; i < act_bytes / 16u; i += kThreads) z[i] = zero;
    }
    if (threadIdx.x < 128 * min(2, p.n_layers)) bias_s[threadIdx.x] = p.bias[threadIdx.x];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    cluster_sync_all();   // the peer's barriers are initialised before anything is sent to them
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"((uint32_t)p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_held = tmem_base + 2u * (uint32_t)p.acc_cols;

    if (warp == 0 && elect_one()) {
        // ---------------- filter producer: three taps of a channel block per request (the pointwise layer: one), this CTA's half
        // of the rows.  Pairs begin a block at different rows of taps, so that they read different lines of L2 at a time.
        // A filter is a constant of the plan: nothing here waits for the previous kernel.
        int slot = 0, round = 0, row = 0;   // row: of 1 KB, first of the layer
        bool ok = true;
        for (int l = 0; l < p.n_layers && ok; l++) {
            const bool pointwise = (p.flags[l] & kChainFlagPointwise) != 0;
            const int tile_rows = (pointwise ? p.n_last : p.n_trunk) / 16;            // 1 KB rows of a tile's half
            const int blocks = p.c_blocks[l], per_block = pointwise ? 1 : 3;
            const int taps = pointwise ? 1 : 3;
            const uint32_t bytes = (uint32_t)(taps * tile_rows) * 1024u;
            const int half_row = row + (int)rank * blocks * per_block * taps * tile_rows;
            const int first = pointwise ? 0 : pair % 3;
            for (int cb = 0; cb < blocks && ok; cb++) {
                int r = first;
                for (int i = 0; i < per_block; i++) {
                    if (round > 0 && !mbar_wait(empty_bar + 8u * slot, (uint32_t)((round & 1) ^ 1), abandon, p.status, 11, kWaitCycles, kSleepNs)) { ok = false; break; }
                    const uint32_t bar = full_bar + 8u * slot;
                    if (rank == 0) mbar_expect_tx(bar, 2u * bytes);
                    tma_load_3d_pair(ring_base + (uint32_t)slot * p.slot_bytes, pointwise ? &map_last : &map_trunk, map_to_cta(bar, 0), 0,
                                     half_row + (cb * per_block + r) * taps * tile_rows, 0);
                    if (++r == per_block) r = 0;
                    if (++slot == p.slots) { slot = 0; round++; }
                }
            }
            row += 2 * blocks * per_block * taps * tile_rows;
        }
    } else if (warp == 1 && rank == 0 && elect_one()) {
        // ---------------- MMA issuer of the pair
        int slot = 0, round = 0;
        bool ok = true;
        const bool trace = TRACE && blockIdx.x == 0;
        const uint32_t pitch = (uint32_t)p.pitch;
        const int first = pair % 3;
        for (int l = 0; l < p.n_layers && ok; l++) {
            const bool pointwise = (p.flags[l] & kChainFlagPointwise) != 0;
            const int n = pointwise ? p.n_last : p.n_trunk;
            const uint32_t tile_bytes = (uint32_t)n * 64u;
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            const uint32_t acc = tmem_base + (uint32_t)((l & 1) * p.acc_cols);
            const int blocks = p.c_blocks[l], per_block = pointwise ? 1 : 3;
            uint32_t accumulate = 0;
            long long full_wait = 0;
            if (trace) p.trace[l * 8 + 0] = clock64();
            for (int cb = 0; cb < blocks && ok; cb++) {
                // this channel block of the layer's input is complete in both CTAs (and, block 0: the accumulator has been read out)
                ok = mbar_wait_cluster(act_bar + 8u * cb, (uint32_t)(l & 1), abandon, p.status, 12);
                if (!ok) break;
                if (trace && cb == 0) p.trace[l * 8 + 1] = clock64();
                tc_fence_after();
                const uint32_t block_rows = base + (uint32_t)cb * block_bytes;
                int r = pointwise ? 1 : first;
                for (int i = 0; i < per_block; i++) {
                    long long tw = 0;
                    if (trace) tw = clock64();
                    ok = mbar_wait(full_bar + 8u * slot, (uint32_t)(round & 1), abandon, p.status, 13);
                    if (!ok) break;
                    if (trace) full_wait += clock64() - tw;
                    tc_fence_after();
                    const uint32_t tile = ring_base + (uint32_t)slot * p.slot_bytes;
                    for (int s = pointwise ? 1 : 0; s < (pointwise ? 2 : 3); s++) {
                        const uint32_t row0 = (uint32_t)(r * p.wp + s);    // (position 0 of the operand is row wp + 1, the centre tap's)
                        const uint64_t da = smem_desc_rows(block_rows + row0 * 128u, pitch);
                        const uint64_t db = smem_desc_sw128(tile + (pointwise ? 0u : (uint32_t)s * tile_bytes));
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            mma_pair<false>(acc, da + 2u * j, db + 2u * j, idesc, accumulate);
                            accumulate = 1;
                        }
                    }
                    mma_commit_pair(empty_bar + 8u * slot);
                    if (++r == per_block) r = 0;
                    if (++slot == p.slots) { slot = 0; round++; }
                }
            }
            if (ok) mma_commit_pair(accum_bar);
            if (trace) p.trace[l * 8 + 2] = clock64(), p.trace[l * 8 + 3] = full_wait;
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: thread <-> accumulator lane <-> position of this CTA's images
        const int quarter = warp & 3;
        const int part = (warp - 2) >> 2;           // which columns of every channel block
        const int m = quarter * 32 + lane;
        const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
        const int row = p.wp + 1 + (m >> 3) * p.pitch + (m & 7);     // padded position = operand row
        int64_t img = (int64_t)blockIdx.x * p.per_cta;
        int py = 0, px = 0;
        bool real = false;
        {
            const int line = row / p.wp, col = row - line * p.wp;
            const int iy = line / (p.h + 1), ry = line - iy * (p.h + 1);
            const int ix = col / (p.w + 1), cx = col - ix * (p.w + 1);
            img += iy * p.gx + ix;
            py = ry - 1;
            px = cx - 1;
            real = cx != 0 && ry != 0 && iy < p.gy && img < p.n_img;
        }
        const uint32_t my_row = base + (uint32_t)row * 128u;
        const uint32_t phase = (uint32_t)row & 7u;
        const uint32_t leader_act = map_to_cta(act_bar, 0);
        // four channels of this position into the operand of channel block cb
        auto store_operand = [&](int cb, int chunk, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                         ::"r"(my_row + (uint32_t)cb * block_bytes + (((uint32_t)chunk ^ phase) << 4)), "r"(a), "r"(b), "r"(c), "r"(d)
                         : "memory");
        };
        auto block_done = [&](int cb) {   // this warp's share of channel block cb is in the operand buffer
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            // (no release at cluster scope, which takes 1000 cycles an arrival, 226 -> 207 us for 33 layers of 256 boards: what is handed
            // over lies in this SM's own shared memory and is read by its tensor core; the fence has completed it there)
            if (lane == 0) mbar_arrive_remote(leader_act + 8u * cb);
        };
        // layer 0's input: from global memory into the operand and the held columns
        asm volatile("griddepcontrol.wait;" ::: "memory");
        {
            const float* src = p.in + img * p.s_in[0] + (int64_t)py * p.s_in[2] + (int64_t)px * p.s_in[3];
            for (int cb = 0; cb < p.blocks; cb++) {
                const int c0 = cb * 32 + part * kCols;
                uint32_t v[kCols];
#pragma unroll
                for (int j = 0; j < kCols; j++) v[j] = real && c0 + j < p.c_in ? __float_as_uint(src[(int64_t)(c0 + j) * p.s_in[1]]) : 0u;
                if (real) {
#pragma unroll
                    for (int j = 0; j < kCols; j += 4) store_operand(cb, (part * kCols + j) / 4, operand_bits(v[j]), operand_bits(v[j + 1]), operand_bits(v[j + 2]), operand_bits(v[j + 3]));
                }
                block_done(cb);
                if (c0 < p.n_trunk) tmem_store_chunk<kCols>(tmem_held + lane_bits + (uint32_t)c0, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }

        for (int l = 0; l < p.n_layers; l++) {
            const uint32_t flags = p.flags[l];
            const bool last = l == p.n_layers - 1;
            const bool heads = last && p.n_heads > 0;
            const bool add_held = (flags & kChainFlagAddHeld) != 0;
            const bool hold = (flags & kChainFlagHold) != 0 && !last;
            const bool relu = (flags & kChainFlagRelu) != 0;
            const int n = heads ? p.n_last : p.n_trunk;
            const uint32_t acc = tmem_base + (uint32_t)((l & 1) * p.acc_cols) + lane_bits;
            const bool trace = TRACE && blockIdx.x == 0 && warp == 2 && lane == 0;
            if (trace) p.trace[l * 8 + 4] = clock64();
            // the next kernel of the stream may be scheduled once every CTA waits for its last layer: early enough to hide its
            // launch, late enough that its CTAs do not sit on this SM for the whole run
            if (last && warp == 2) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            // the bias of the layer after the next (its row was last read by the layer before this one)
            float next_bias = 0.f;
            const int et = threadIdx.x - 64;
            const bool fetch_bias = l + 2 < p.n_layers && et < 128;
            if (fetch_bias) next_bias = p.bias[(l + 2) * 128 + et];
            const float* layer_bias = bias_s + l % kBiasRows * 128;
            float4 bias[kCols / 4];   // of the columns that come next
#pragma unroll
            for (int j = 0; j < kCols; j += 4) bias[j / 4] = *(const float4*)(layer_bias + part * kCols + j);
            if (!mbar_wait(accum_bar, (uint32_t)(l & 1), abandon, p.status, 14, kWaitCycles, kSleepNs)) break;
            if (trace) p.trace[l * 8 + 5] = clock64();
            tc_fence_after();
            if (fetch_bias) bias_s[(l + 2) % kBiasRows * 128 + et] = next_bias;
            const int blocks = heads ? (n + 31) / 32 : p.blocks;
#pragma unroll 1
            for (int cb = 0; cb < blocks; cb++) {
                const int c0 = cb * 32 + part * kCols;
                uint32_t v[kCols], h[kCols];
                if (c0 < n) {
                    tmem_load_chunk_nowait<kCols>(acc + (uint32_t)c0, v);
                    if (add_held) tmem_load_chunk_nowait<kCols>(tmem_held + lane_bits + (uint32_t)c0, h);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < kCols; j += 4) {
                        const float4 b = bias[j / 4];
                        float2 x[2] = {add_pair(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), make_float2(b.x, b.y)),
                                       add_pair(make_float2(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])), make_float2(b.z, b.w))};
                        if (add_held) {
                            x[0] = add_pair(x[0], make_float2(__uint_as_float(h[j]), __uint_as_float(h[j + 1])));
                            x[1] = add_pair(x[1], make_float2(__uint_as_float(h[j + 2]), __uint_as_float(h[j + 3])));
                        }
                        const float y[4] = {x[0].x, x[0].y, x[1].x, x[1].y};
                        uint32_t r[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            v[j + i] = __float_as_uint(relu ? fmaxf(y[i], 0.f) : y[i]);
                            // (behind a ReLU there is no NaN, and infinity stays what it is without a test)
                            r[i] = relu ? (v[j + i] + 0x1000u) & 0xFFFFE000u : operand_bits(v[j + i]);
                        }
                        if (PARTIAL && c0 + kCols > p.k) {   // (what the zeros of the filter make of an infinity is NaN)
#pragma unroll
                            for (int i = 0; i < 4; i++) r[i] = c0 + j + i < p.k ? r[i] : 0u;
                        }
                        if (!last && real) store_operand(cb, (part * kCols + j) / 4, r[0], r[1], r[2], r[3]);
                    }
                } else if (PARTIAL && l == 0 && !last && real) {   // (an input wider than the trunk: its last channels are in the operand)
#pragma unroll
                    for (int j = 0; j < kCols; j += 4) store_operand(cb, (part * kCols + j) / 4, 0u, 0u, 0u, 0u);
                }
                if (!last) block_done(cb);
                if (trace && cb == 0) p.trace[l * 8 + 7] = clock64();
                if (c0 + 32 < n) {
#pragma unroll
                    for (int j = 0; j < kCols; j += 4) bias[j / 4] = *(const float4*)(layer_bias + c0 + 32 + j);
                }
                if (c0 >= n) continue;
                if (hold) tmem_store_chunk<kCols>(tmem_held + lane_bits + (uint32_t)c0, v);
                if (!real) continue;
                if (flags & kChainFlagStore) {
                    float* o = p.out + img * p.s_out[0] + (int64_t)py * p.s_out[2] + (int64_t)px * p.s_out[3];
                    if (p.out_vec) {
#pragma unroll
                        for (int j = 0; j < kCols; j += 4)
                            if (c0 + j < p.k) *(uint4*)(o + c0 + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < kCols; j++)
                            if (c0 + j < p.k) o[(int64_t)(c0 + j) * p.s_out[1]] = __uint_as_float(v[j]);
                    }
                }
                if (heads) {
#pragma unroll 1
                    for (int i = 0; i < p.n_heads; i++) {
                        const int begin = p.head_begin[i], end = p.head_begin[i + 1];
                        if (end <= c0 || begin >= c0 + kCols) continue;
                        const bool act = p.head_relu[i] != 0;
                        const int64_t s1 = p.head_s_out[i][1];
                        float* o = p.head_out[i] + img * p.head_s_out[i][0] + (int64_t)py * p.head_s_out[i][2] + (int64_t)px * p.head_s_out[i][3] + (c0 - begin) * s1;
#pragma unroll
                        for (int j = 0; j < kCols; j++) {
                            const float x = __uint_as_float(v[j]);
                            if (c0 + j >= begin && c0 + j < end) o[j * s1] = act ? fmaxf(x, 0.f) : x;
                        }
                    }
                }
            }
            if (hold) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            if (trace) p.trace[l * 8 + 6] = clock64();
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still address it
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
}

}  // namespace

// ---------------------------------------------------------------- host side
static int round_up_int(int x, int to) { return (x + to - 1) / to * to; }

// Every chain whose images fit takes this kernel: 17 to 33 layers, 7 x 7 to 9 x 9 boards, 32 to 128 channels, 20 to 2048 images ran in
// 0.45 to 0.82 of the time of conv_chain_kernel with its own best arrangement of images (one 9 x 9 board a CTA, 64 channels: 89.3 ->
// 57.1 us for 101 boards, 543 -> 388 for 1000; 128 channels, 8 x 8: 312 -> 207 us for 256 boards, 136 -> 108 for 100).
bool tc_chain_pair_geometry(int h, int w, int64_t n_img, int blocks, int k, int head_channels, ChainPairGeometry* out) {
    if (h < 1 || w < 1 || h > 126 || w > 126 || n_img < 1 || blocks < 1 || blocks > 4 || k < 1 || k > 128 || head_channels > 128) return false;
    ChainPairGeometry best{};
    for (int gx = 1; gx <= 16; gx++) {
        for (int gy = 1; gy <= 16; gy++) {
            ChainPairGeometry g{};
            g.gx = gx;
            g.gy = gy;
            g.per_cta = gx * gy;
            g.wp = gx * (w + 1);
            const int span = ((gy - 1) * (h + 1) + h - 1) * g.wp + (gx - 1) * (w + 1) + w;   // first real pixel to the last
            if (w == 8 && gy == 1 && gx * h <= 16) g.pitch = 9;      // image rows as groups of operand rows
            else if (span <= 128) g.pitch = 8;
            else break;
            g.n_trunk = round_up_int(k, 16);
            g.n_last = round_up_int(head_channels, 16);
            g.rows_alloc = round_up_int(2 * g.wp + 2 + 15 * g.pitch + 8, 8);
            g.slot_bytes = std::max(3 * g.n_trunk, g.n_last) * 64;
            const int fixed = 1024 /* alignment */ + kBiasRows * 512 + 16 * 8 + 5 * 8 + 32;
            const int act_bytes = blocks * g.rows_alloc * 128;
            g.slots = std::min(8, (227 * 1024 - fixed - act_bytes) / g.slot_bytes);
            if (g.slots < 2) break;
            g.smem_bytes = fixed + act_bytes + g.slots * g.slot_bytes;
            // the layers' time does not depend on how many images a CTA holds
            if (g.per_cta > best.per_cta) best = g;
        }
    }
    if (best.per_cta == 0) return false;
    if (out) *out = best;
    return true;
}

struct ChainPairLaunch {
    CUtensorMap map_trunk, map_last;
    ChainPairKernelParams p;
    dim3 grid;
    int smem_bytes;
};

std::shared_ptr<void> chain_pair_prepare(const ConvChainParams& c, uint32_t* status_word) {
    auto l = std::make_shared<ChainPairLaunch>();
    ChainPairKernelParams& p = l->p;
    memset(&p, 0, sizeof(p));
    int blocks = (c.k + 31) / 32;
    for (int i = 0; i < c.n_layers; i++) {
        blocks = std::max<int>(blocks, c.c_blocks[i]);
        p.flags[i] = c.flags[i];
        p.c_blocks[i] = c.c_blocks[i];
    }
    KN_CHECK(c.n_heads >= 0 && c.n_heads <= kMaxChainHeads, KN_ERR_INTERNAL, "convolution chain with too many heads");
    ChainPairGeometry g;
    KN_CHECK(tc_chain_pair_geometry(c.h, c.w, c.n, blocks, c.k, c.n_heads ? c.head_begin[c.n_heads] : 0, &g), KN_ERR_INTERNAL,
             "convolution chain does not fit a CTA pair");
    p.in = c.in;
    p.out = c.out;
    p.bias = c.bias;
    for (int i = 0; i < 4; i++) {
        p.s_in[i] = c.s_in[i];
        p.s_out[i] = c.s_out[i];
    }
    p.n_img = c.n;
    p.c_in = c.c_in;
    p.k = c.k;
    p.h = c.h;
    p.w = c.w;
    p.n_layers = c.n_layers;
    p.per_cta = g.per_cta;
    p.gx = g.gx;
    p.gy = g.gy;
    p.wp = g.wp;
    p.pitch = g.pitch;
    p.rows_alloc = g.rows_alloc;
    p.slots = g.slots;
    p.slot_bytes = (uint32_t)g.slot_bytes;
    p.blocks = blocks;
    p.n_trunk = g.n_trunk;
    p.n_last = g.n_last;
    p.acc_cols = std::max(g.n_trunk, g.n_last);
    p.tmem_cols = 32;
    while (p.tmem_cols < 2 * p.acc_cols + g.n_trunk) p.tmem_cols <<= 1;
    p.out_vec = c.s_out[1] == 1 && c.k % 4 == 0 && ((uintptr_t)c.out & 15) == 0 && c.s_out[0] % 4 == 0 && c.s_out[2] % 4 == 0 && c.s_out[3] % 4 == 0;
    p.status = status_word;
    p.n_heads = c.n_heads;
    for (int i = 0; i < c.n_heads; i++) {
        p.head_begin[i] = c.head_begin[i];
        p.head_out[i] = c.head_out[i];
        p.head_relu[i] = c.head_relu[i];
        for (int d = 0; d < 4; d++) p.head_s_out[i][d] = c.head_s_out[i][d];
    }
    p.head_begin[c.n_heads] = c.head_begin[c.n_heads];
    p.trace = chain_trace_table(c.n_layers);
    // the filters as lines of 1 KB; a request is three taps of a channel block, or one tile of the pointwise layer
    int64_t lines = 0;
    for (int i = 0; i < c.n_layers; i++)
        lines += (int64_t)((c.flags[i] & kChainFlagPointwise) ? g.n_last : 9 * g.n_trunk) * c.c_blocks[i] / 8;
    const int64_t dims[3] = {256, lines, 1}, strides[3] = {1, 256, 256 * lines};
    const int box_trunk[3] = {256, 3 * g.n_trunk / 16, 1}, box_last[3] = {256, std::max(1, g.n_last / 16), 1};
    l->map_trunk = tc_make_map(c.tiles, 3, dims, strides, box_trunk, false);
    l->map_last = tc_make_map(c.tiles, 3, dims, strides, box_last, false);
    l->grid = dim3((unsigned)(2 * ((c.n + 2 * g.per_cta - 1) / (2 * g.per_cta))), 1, 1);
    l->smem_bytes = g.smem_bytes;
    return l;
}

int chain_pair_launch(const void* launch, cudaStream_t stream) {
    const ChainPairLaunch& l = *(const ChainPairLaunch*)launch;
    static std::mutex mu;
    static bool done[4][64] = {};
    const bool trace = l.p.trace != nullptr, partial = l.p.k % 32 != 0;
    auto kernel = trace ? (partial ? conv_chain_pair_kernel<true, true> : conv_chain_pair_kernel<true, false>)
                        : (partial ? conv_chain_pair_kernel<false, true> : conv_chain_pair_kernel<false, false>);
    if (int e = allow_shared(kernel, 227 * 1024, done[2 * trace + partial], mu)) return e;
    if (l.grid.x == 0) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = l.grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)l.smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    void* args[] = {(void*)&l.map_trunk, (void*)&l.map_last, (void*)&l.p};
    return (int)cudaLaunchKernelExC(&cfg, (const void*)kernel, args);
}

}  // namespace kn
